// Fused MLP backward with several row tiles in flight per SM, for every activation, with and without biases.
//
// The backward of a 128-row tile is a chain of 2 depth + 1 short steps (recompute and park every layer's input, then
// layer by layer backwards), each a round trip "operands written -> barrier -> issue -> commit -> mbarrier -> tcgen05.ld ->
// convert -> st.shared" of about a microsecond of which the MMAs are a tenth.  Throughput is row tiles in flight over
// chain length.  ONE CTA per SM runs S independent SLOTS of 128 W threads plus one WGRAD warp:
//   * a warp of a slot issues the slot's recompute and dgrad MMAs into the slot's own accumulator columns, so that chain
//     never leaves the slot; the W warpgroups of a slot share a tile's columns (thread = tile row = TMEM lane, column half);
//   * the wgrad warp issues the weight- and bias-gradient MMAs of every slot.  MMAs of one thread execute in order, so all
//     slots accumulate into ONE shared set of TMEM columns instead of one set per tile in flight;
//   * dz of layer l - 1 is written in place over the parked input of layer l once both MMAs that read it have finished;
//   * rows come and go through a ring of buffers (features, output gradient), one more than slots where that fits, kept by ROW
//     WARPS: TMA fetches the next tile's rows while the slots work, and the input gradient, which the slot leaves in its buffer
//     as rounded rows, goes out by TMA before the buffer is filled again: one row warp; where TMA cannot describe some of the rows
//     four, which copy them.  Rows of 16 or 32 columns lie 32 or 64 bytes apart (the tensor core's 32- and 64-byte swizzles).
// The output layer's weight gradient is formed transposed, act^T . dz: an M = 64 MMA takes 27 + N / 2 cycles, and N is then the
// padded output width (16: 35 instead of 60 cycles a K step) instead of the hidden one.
// Bias gradient of a layer = column sums of dz = dz^T . ONES, a small MMA (N = 8) next to the weight gradient's.  SiLU' and
// ReLU^2' want the pre-activation: the step that needs it issues that layer's forward GEMM again into a second accumulator
// and rounds z to the storage dtype, as the forward pass did.  Biases are in the accumulators before a recompute GEMM is issued, as in
// the forward kernels: the backward opens the ReLUs that the forward opened.
//
// Measured: rows fetched and stored by the slots themselves were 22 % of a slot's time (2^21 rows 32-64-64-16; a fence for the
// tensor core also waits for the thread's own copies and stores in flight).  With the ring 0.234 -> 0.209 ms, 2^20 rows 32-4x64-16
// 0.279 -> 0.265, 300 007 rows 32-3x64-16 with biases, where the smaller row buffers make room for a third slot, 0.081 -> 0.069; with the
// issuers spread over the schedulers, their lanes elected where they issue and no load of the abort flag ahead of a wait that is over,
// 0.186, 0.220 and 0.062.
//
// Per slot three mbarriers: `ready` (one arrival: the operands of the slot's next backward step are in place), `acc` (the
// slot's own MMAs of the step are done), `wdone` (the step's wgrad is done).  The wgrad warp polls all `ready` barriers at
// once, one lane per slot, without blocking.  Every wait is bounded by the global timer and watches the CTA's abort flag;
// after an abort everybody keeps the same barrier sequence without doing work.
#include "mlp_tc_device.cuh"

#include <cstddef>

namespace th {
namespace {

constexpr int kSlotsMax = 4;
constexpr int kStepsMax = 24;  // 2 depth + 1

// Rows of at most 16, 32 or 64 columns lie 32, 64 or 128 bytes apart, in the tensor core's 32-, 64- or 128-byte swizzle.
__host__ __device__ constexpr int row_pitch(int pad) { return pad <= 16 ? 32 : (pad <= 32 ? 64 : 128); }
__host__ __device__ constexpr uint32_t desc_high(int pitch) {
    return (static_cast<uint32_t>(8 * pitch) >> 4) | (1u << 14) | ((pitch == 128 ? 2u : (pitch == 64 ? 4u : 6u)) << 29);
}
__device__ __forceinline__ uint64_t desc_of(uint32_t low, uint32_t high) {
    uint64_t d;
    asm("mov.b64 %0, {%1, %2};" : "=l"(d) : "r"(low), "r"(high));
    return d;
}

struct SlotPlan {
    int rings;           // buffers of rows: slots, or slots + 1
    int x_pitch, go_pitch;
    int ring;            // byte offset
    int ring_bytes;      // a buffer: the rows, then the output gradient
    int ones;            // byte offset of the tile of ones (biases)
    int weights;         // byte offset of the weight tiles and biases
    int tables;          // byte offset of the barriers and step table
    int total;           // dynamic shared memory
    int acc_cols;        // accumulator columns of a slot
    int tmem_cols;
    TcPlan w;            // weight and bias offsets relative to `weights`
};

// What the issuing warps need for one step of a tile, worked out once per CTA: both issue paths are on the critical chain of
// every tile, and each address or descriptor computed there is paid 2 depth + 1 times per tile.
struct __align__(16) SlotStep {
    uint32_t a_off;    // the slot's own GEMM: A operand, relative to the slot's first tile
    uint32_t b_addr;   //   B operand (a weight tile)
    uint32_t idesc;    //   instruction descriptor; 0 = the step has no GEMM of its own
    uint32_t k_steps;  //   bits 0..7: K steps of 16; bit 8: B is read MN-major
    uint32_t wa_off;   // weight gradient: A operand (dz, MN-major), relative to the slot's first tile
    uint32_t wb_off;   //   B operand (the layer's input, MN-major)
    uint32_t widesc;   //   instruction descriptor
    uint32_t dw_col;   //   bits 0..15: accumulator column; bits 16..31: the bias gradient's
    uint32_t za_off;   // pre-activation of the layer below: A operand
    uint32_t zb_addr;  //   B operand
    uint32_t z_k;      //   K steps; 0 = none
    uint32_t a_high;   // high words of the descriptors that are not a 128-byte tile's: the slot's own GEMM's A operand
    uint32_t wa_high, wb_high;  // the weight gradient's operands
    uint32_t wa_step, wb_step;  // bytes between K steps
    uint32_t flags;    // operands in the row buffer: bit 2 the weight gradient's B, 3 the pre-activation's A; 4: B is dz (transposed)
    uint32_t unused[2];
};

struct SlotTables {
    unsigned long long weights_bar;
    unsigned long long ready[kSlotsMax], acc[kSlotsMax], wdone[kSlotsMax];
    unsigned long long full[kSlotsMax + 1], empty[kSlotsMax + 1];
    uint32_t tmem_holder;
    int abort_flag;
    SlotStep steps[kStepsMax];
};

__host__ __device__ constexpr bool needs_preact(int act) { return act == TH_ACT_SILU || act == TH_ACT_RELU2; }

SlotPlan slot_plan(const MlpShape &s, int slots, int rings) {
    SlotPlan b{};
    b.rings = rings;
    b.x_pitch = row_pitch(s.ki);
    b.go_pitch = row_pitch(s.no);
    int off = slots * s.depth * kTileBytes;
    b.ring = off;
    b.ring_bytes = kTileRows * (b.x_pitch + b.go_pitch);
    off += rings * b.ring_bytes;
    b.ones = off;
    if (s.has_bias) off += kTileRows * 32;
    off = (off + 1023) & ~1023;
    b.weights = off;
    b.w = tc_plan(s, false, 0);
    off += s.has_bias ? b.w.total : b.w.bias_offset;  // the biases are the plan's last part
    b.tables = (off + 15) & ~15;
    b.total = b.tables + static_cast<int>(offsetof(SlotTables, steps)) + (2 * s.depth + 1) * static_cast<int>(sizeof(SlotStep));
    b.acc_cols = kAccCols * (needs_preact(s.act) ? 2 : 1);
    const int cols = slots * b.acc_cols + s.ki + (s.depth - 1) * s.h + s.no + (s.has_bias ? 8 * (s.depth + 1) : 0);
    int alloc = 32;
    while (alloc < cols) alloc <<= 1;
    b.tmem_cols = alloc;
    return b;
}

// 16-byte chunk c of row r lies at chunk c ^ row_swizzle_of(r, pitch)
__device__ __forceinline__ uint32_t row_swizzle_of(int r, int pitch) {
    return pitch == 128 ? (r & 7) : (pitch == 64 ? ((r >> 1) & 3) : ((r >> 2) & 1));
}

__device__ __forceinline__ bool mbar_test(uint32_t bar, uint32_t parity) {
    uint32_t done;
    asm volatile("{\n\t.reg .pred p;\n\tmbarrier.test_wait.parity.shared::cta.b64 p, [%1], %2;\n\tselp.u32 %0, 1, 0, p;\n\t}\n"
                 : "=r"(done)
                 : "r"(bar), "r"(parity)
                 : "memory");
    return done != 0;
}

__device__ __forceinline__ void mbar_init(const void *bar, uint32_t arrivals = 1) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_addr(bar)), "r"(arrivals) : "memory");
}

// This thread's columns of a row of `pad` accumulator columns (all of them, or one half of them), 8 at a time:
// fn(chunk of the row, eight values)
template <int W, typename Fn>
__device__ __forceinline__ void for_row_pieces(uint32_t taddr, int pad, int half, Fn fn) {
    if constexpr (W == 2) {
        const int n = pad / 2, first = half * (n / 8);
        for_each_piece(taddr + half * n, n, [&](int u, const uint32_t(&piece)[8]) { fn(first + u, piece); });
    } else {
        int first = 0;
#pragma unroll 1
        for (; first + 32 <= pad; first += 32)
            for_each_piece_n<32>(taddr + first, [&](int u, const uint32_t(&piece)[8]) { fn(first / 8 + u, piece); });
        if (first < pad) for_each_piece_n<16>(taddr + first, [&](int u, const uint32_t(&piece)[8]) { fn(first / 8 + u, piece); });
    }
}

// ---- rows that TMA cannot describe ----
//
// The row warps copy them, a warp its 32 rows of a tile, a thread a 16-byte chunk of a row at a time, the warp's chunks side by side, so that
// an access touches five lines.  A chunk is eight accesses at fixed distances from one address, and two chunks are in flight.  Measured, 300 007
// rows, one layer, rows off their alignment by an element, backward (a thread a row, whose accesses touch 32 lines / this): 64-64
// 350 / 200 us, 32-64 186 / 88, 32-16 114 / 61, 27-3 96 / 65.  Lanes along a row, whose addresses are worked out for every element: 230
// to 460, 188 to 290, 157, 143.

// Chunk i of the warp's 32 rows of `chunks` chunks each
struct RowChunk {
    int row, chunk;
    __device__ __forceinline__ RowChunk(int i, int chunks, int r0) {
        const int r = (i * (65536 / chunks + 1)) >> 16;  // i / chunks: i < 256, chunks <= 8
        row = r0 + r;
        chunk = i - r * chunks;
    }
    __device__ __forceinline__ uint32_t at(int pitch) const { return row * pitch + ((chunk ^ row_swizzle_of(row, pitch)) << 4); }
};

// Rows r0 .. r0 + 31 of the tile whose first row is src, `live` of the tile's rows exist -> row buffer, zero padded to `pad` columns
__device__ __forceinline__ void copy_rows_in(const unsigned short *src, long long stride, int r0, int live, int cols, int pad, int pitch, uint32_t buffer) {
    if (cols <= 8) {
        const int r = r0 + (threadIdx.x & 31);
        const uint32_t at = buffer + r * pitch, swz = row_swizzle_of(r, pitch);
        const uint4 v = gather8(src + (r < live ? r * stride : 0), 0, r < live ? cols : 0);
        for (int c = 0; c < pad / 8; ++c) st_shared_16(at + ((c ^ swz) << 4), c == 0 ? v : make_uint4(0, 0, 0, 0));
        return;
    }
    const int chunks = pad / 8;
#pragma unroll 1
    for (int i = threadIdx.x & 31; i < 32 * chunks; i += 64) {
        const RowChunk c(i, chunks, r0), e(i + 32, chunks, r0);  // an even number of chunks
        const uint4 u = gather8(src + (c.row < live ? c.row * stride : 0) + 8 * c.chunk, 8 * c.chunk, c.row < live ? cols : 0);
        const uint4 v = gather8(src + (e.row < live ? e.row * stride : 0) + 8 * e.chunk, 8 * e.chunk, e.row < live ? cols : 0);
        st_shared_16(buffer + c.at(pitch), u);
        st_shared_16(buffer + e.at(pitch), v);
    }
}

// The other way, without the padding
__device__ __forceinline__ void copy_rows_out(unsigned short *dst, long long stride, int r0, int live, int cols, int pitch, uint32_t buffer) {
    const int chunks = (cols + 7) / 8;
#pragma unroll 1
    for (int i = threadIdx.x & 31; i < 32 * chunks; i += 32) {
        const RowChunk c(i, chunks, r0);
        if (c.row < live) store_chunk_to_global(dst + c.row * stride, c.chunk, cols, ld_shared_16(buffer + c.at(pitch)), false);
    }
}

// COPIED: some rows are copied by four row warps; otherwise one asks for boxes
template <bool COPIED>
constexpr int kRowWarps = COPIED ? 4 : 1;

template <typename T, int ACT, bool BIAS, int S, int W, bool COPIED>
__global__ void __launch_bounds__(128 * S * W + 32 + 32 * kRowWarps<COPIED>, 1)
slots_mlp_bwd_tc_kernel(const MlpShape s, const MlpParams p, const __grid_constant__ WeightMaps maps, const int use_tma,
                        const __grid_constant__ CUtensorMap x_map, const __grid_constant__ CUtensorMap go_map,
                        const __grid_constant__ CUtensorMap gx_map, const int row_tma, const __grid_constant__ SlotPlan P, const T *__restrict__ x, long long x_stride, const T *__restrict__ go,
                        long long go_stride, T *__restrict__ gx, long long gx_stride, float *__restrict__ workspace, long long n_rows) {
    constexpr bool kPreact = needs_preact(ACT);
    constexpr int kSlotThreads = 128 * W;
    constexpr int bf16 = std::is_same<T, __half>::value ? 0 : 1;
    extern __shared__ __align__(1024) unsigned char smem_slots[];
    unsigned char *smem = smem_slots;
    SlotTables &tb = *reinterpret_cast<SlotTables *>(smem + P.tables);
    const int d = s.depth, n_steps = 2 * d + 1;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const bool is_wgrad_warp = warp == 4 * S * W, is_row_warp = warp > 4 * S * W;
    unsigned char *wsmem = smem + P.weights;
    volatile int *abort_now = &tb.abort_flag;

    // ---- set-up ----
    if (threadIdx.x == 0) {
        tb.abort_flag = (smem_addr(smem) & 1023u) ? 1 : 0;  // operand tiles need their alignment
        if (tb.abort_flag) g_tc_status = 1;
        mbar_init(&tb.weights_bar);
        for (int i = 0; i < S; ++i) {
            mbar_init(&tb.ready[i]);
            mbar_init(&tb.acc[i]);
            mbar_init(&tb.wdone[i]);
        }
        for (int i = 0; i < P.rings; ++i) {
            mbar_init(&tb.full[i], static_cast<uint32_t>(kRowWarps<COPIED>));
            mbar_init(&tb.empty[i]);
        }
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    // narrow networks: tiles start out as zeros, since columns a layer does not use are still read as MMA rows
    if (s.h < 64)
        for (int e = threadIdx.x; e < P.ones / 16; e += blockDim.x) reinterpret_cast<uint4 *>(smem)[e] = make_uint4(0, 0, 0, 0);
    if constexpr (BIAS) {
        // 128 rows of ones, 32 bytes apart
        const uint32_t one2 = pack_pair<T>(1.f, 1.f);
        for (int e = threadIdx.x; e < kTileRows * 2; e += blockDim.x) reinterpret_cast<uint4 *>(smem + P.ones)[e] = make_uint4(one2, one2, one2, one2);
        stage_biases<T>(wsmem, P.w, s, p);
    }
    fence_async_smem();
    if (!use_tma) {
        stage_all_weights<T>(wsmem, P.w, s, p);
        fence_async_smem();
    } else if (threadIdx.x == 0) {
        tma_issue_weights(wsmem, P.w, s, maps, &tb.weights_bar);  // awaited by the issuers, ahead of their first MMA
    }
    if (is_wgrad_warp) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_addr(&tb.tmem_holder)),
                     "r"(static_cast<uint32_t>(P.tmem_cols))
                     : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    const long long n_tiles = (n_rows + kTileRows - 1) / kTileRows;
    const long long first_tile = blockIdx.x, tile_stride = gridDim.x;
    const long long n_mine = first_tile < n_tiles ? (n_tiles - first_tile + tile_stride - 1) / tile_stride : 0;
    const uint32_t smem_base = smem_addr(smem);
    const uint32_t slot_bytes = static_cast<uint32_t>(d) * kTileBytes;
    const uint32_t go_at = static_cast<uint32_t>(kTileRows * P.x_pitch);  // the output gradient in a row buffer
    auto ring_of = [&](uint32_t b) { return smem_base + P.ring + b * P.ring_bytes; };
    auto dw_col = [&](int l) { return S * P.acc_cols + (l == 0 ? 0 : s.ki + (l - 1) * s.h); };
    auto db_col = [&](int l) { return S * P.acc_cols + s.ki + (d - 1) * s.h + s.no + 8 * l; };
    if (static_cast<int>(threadIdx.x) < n_steps) {  // steps 0 .. d - 1 recompute, step j >= d is the backward step of layer 2 d - j
        const int j = threadIdx.x;
        SlotStep st{};
        st.a_high = st.wa_high = st.wb_high = kDescHigh;
        st.wa_step = st.wb_step = 2048;
        if (j < d) {
            st.a_off = j == 0 ? 0u : static_cast<uint32_t>(j - 1) * kTileBytes;
            if (j == 0) st.a_high = desc_high(P.x_pitch);
            st.b_addr = smem_addr(weight_tile(wsmem, P.w, s, j));
            st.idesc = instr_desc(128, s.h, bf16, 0, 0);
            st.k_steps = static_cast<uint32_t>((j == 0 ? s.ki : s.h) / 16);
        } else {
            const int l = 2 * d - j;
            const int in_pad = l == 0 ? s.ki : s.h, out_pad = l == d ? s.no : s.h;
            const uint32_t dz = l == d ? go_at : static_cast<uint32_t>(l) * kTileBytes;
            if (l > 0 || gx != nullptr) {
                st.a_off = dz;
                st.b_addr = smem_addr(weight_tile(wsmem, P.w, s, l));
                st.idesc = instr_desc(128, in_pad, bf16, 0, 1);
                st.k_steps = static_cast<uint32_t>(out_pad / 16) | 256u;
            }
            st.wa_off = dz;
            st.wb_off = l == 0 ? 0u : static_cast<uint32_t>(l - 1) * kTileBytes;
            st.widesc = instr_desc(64, in_pad, bf16, 1, 1);
            if (l == d) {  // transposed: act^T . dz
                st.a_high = desc_high(P.go_pitch);
                st.wa_off = st.wb_off;
                st.wb_off = go_at;
                st.flags |= 4u | 16u;
                st.wb_high = desc_high(P.go_pitch);
                st.wb_step = 16 * P.go_pitch;
                st.widesc = instr_desc(64, out_pad, bf16, 1, 1);
            }
            if (l == 0) {
                st.flags |= 4u;
                st.wb_high = desc_high(P.x_pitch);
                st.wb_step = 16 * P.x_pitch;
            }
            st.dw_col = static_cast<uint32_t>(dw_col(l)) | (static_cast<uint32_t>(db_col(l)) << 16);
            if (kPreact && l > 0) {
                st.za_off = l == 1 ? 0u : static_cast<uint32_t>(l - 2) * kTileBytes;
                if (l == 1) st.flags |= 8u;
                st.zb_addr = smem_addr(weight_tile(wsmem, P.w, s, l - 1));
                st.z_k = static_cast<uint32_t>((l == 1 ? s.ki : s.h) / 16);
            }
        }
        tb.steps[j] = st;
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = tb.tmem_holder;

    if (is_wgrad_warp) {
        // ================= weight gradients of every slot =================
        // lane i < S keeps slot i's state: its next backward step, the tiles it still has, the parity to wait for
        int my_step = d;
        uint32_t my_buf = static_cast<uint32_t>(lane) % static_cast<uint32_t>(P.rings);
        long long my_tiles = lane < S && lane < n_mine ? (n_mine - lane + S - 1) / S : 0;
        uint32_t my_parity = 0, started = 0;
        const uint32_t my_bar = smem_addr(&tb.ready[lane < S ? lane : 0]);
        unsigned long long deadline = 0;
        unsigned idle = 0;
        const bool leader = elect_one();  // the same lane every time: MMAs of one thread execute in order
        while (__any_sync(0xffffffffu, my_tiles > 0)) {
            uint32_t mask = __ballot_sync(0xffffffffu, my_tiles > 0 && mbar_test(my_bar, my_parity));
            if (mask == 0) {
                if ((++idle & 63u) == 0) {
                    if (*abort_now) break;
                    const unsigned long long now = global_ns();
                    if (deadline == 0) deadline = now + kPipeWaitNs;
                    else if (now > deadline) {
                        *abort_now = 1;
                        g_tc_status = 1;
                        break;
                    }
                }
                continue;
            }
            idle = 0;
            deadline = 0;
            const bool mine = (mask >> lane) & 1u;
            tc_fence_after();
            while (mask) {
                const int i = __ffs(mask) - 1;
                mask &= mask - 1;
                const int j = __shfl_sync(0xffffffffu, my_step, i);
                const uint4 w = *reinterpret_cast<const uint4 *>(&tb.steps[j].wa_off);
                const uint4 h = *reinterpret_cast<const uint4 *>(&tb.steps[j].wa_high);
                const uint32_t flags = tb.steps[j].flags;
                const uint32_t tile0 = smem_base + static_cast<uint32_t>(i) * slot_bytes, rows0 = ring_of(__shfl_sync(0xffffffffu, my_buf, i));
                const bool more = (started >> (j - d)) & 1u;
                if (leader) {
                    const uint32_t a_low = desc_low(tile0 + w.x), b_low = desc_low((flags & 4u ? rows0 : tile0) + w.y);
                    for (int k = 0; k < kTileRows / 16; ++k)
                        mma_f16(tmem + (w.w & 0xffffu), desc_of(a_low + k * (h.z >> 4), h.x), desc_of(b_low + k * (h.w >> 4), h.y), w.z, more || k > 0);
                    if constexpr (BIAS) {
                        const bool from_b = flags & 16u;
                        const uint32_t dz_low = from_b ? b_low : a_low, dz_step = (from_b ? h.w : h.z) >> 4, dz_high = from_b ? h.y : h.x;
                        for (int k = 0; k < kTileRows / 16; ++k)
                            mma_f16(tmem + (w.w >> 16), desc_of(dz_low + k * dz_step, dz_high), desc_of(desc_low(smem_base + P.ones) + k * 32, desc_high(32)),
                                    instr_desc(64, 8, bf16, 1, 1), more || k > 0);
                    }
                }
                started |= 1u << (j - d);
                if (leader) mma_commit(smem_addr(&tb.wdone[i]));
            }
            __syncwarp();
            if (mine) {
                my_parity ^= 1u;
                if (++my_step == n_steps) {
                    my_step = d;
                    --my_tiles;
                    my_buf = (my_buf + S) % static_cast<uint32_t>(P.rings);
                }
            }
        }
    } else if (is_row_warp) {
        // ================= rows: the input gradient out of a buffer, the next tile's rows into it =================
        const uint32_t x_bytes = static_cast<uint32_t>(kTileRows * P.x_pitch), go_bytes = static_cast<uint32_t>(kTileRows * P.go_pitch);
        const bool x_tma = !COPIED || (row_tma & 1), go_tma = !COPIED || (row_tma & 2), gx_tma = COPIED ? (row_tma & 4) != 0 : gx != nullptr;
        const int r_warp = warp - 4 * S * W - 1;
        auto live_rows = [&](long long first) { return static_cast<int>(n_rows - first < kTileRows ? n_rows - first : kTileRows); };
        bool alive = true;  // after an abort: the same sequence of barriers, no work
        for (long long k = 0; k < n_mine + P.rings; ++k) {
            const uint32_t b = static_cast<uint32_t>(k % P.rings), rows_at = ring_of(b);
            const long long row0 = (first_tile + k * tile_stride) * kTileRows;
            if (k >= P.rings) {
                if (k - P.rings >= n_mine) continue;
                const long long old0 = row0 - P.rings * tile_stride * kTileRows;
                pipe_wait(smem_addr(&tb.empty[b]), static_cast<uint32_t>((k / P.rings - 1) & 1), &tb.abort_flag);
                alive = alive && !__any_sync(0xffffffffu, *abort_now);
                if (!alive) {
                } else if (gx_tma) {
                    if (r_warp == 0 && lane == 0) {
                        tma_store_2d(&gx_map, rows_at, 0, static_cast<int>(old0));
                        asm volatile("cp.async.bulk.wait_group.read 0;" ::: "memory");
                    }
                } else if (COPIED && gx != nullptr) {
                    copy_rows_out(reinterpret_cast<unsigned short *>(gx + old0 * gx_stride), gx_stride, 32 * r_warp, live_rows(old0), s.d_in, P.x_pitch, rows_at);
                }
                __syncwarp();
                if constexpr (COPIED) asm volatile("bar.sync 15, 128;" ::: "memory");
            }
            if (k >= n_mine || !alive) continue;
            if constexpr (COPIED) {
                if (!x_tma)
                    copy_rows_in(reinterpret_cast<const unsigned short *>(x + row0 * x_stride), x_stride, 32 * r_warp, live_rows(row0), s.d_in, s.ki, P.x_pitch, rows_at);
                if (!go_tma)
                    copy_rows_in(reinterpret_cast<const unsigned short *>(go + row0 * go_stride), go_stride, 32 * r_warp, live_rows(row0), s.d_out, s.no, P.go_pitch,
                                 rows_at + go_at);
                fence_async_smem();
                __syncwarp();
            }
            if (lane == 0) {
                const uint32_t full_bar = smem_addr(&tb.full[b]), bytes = r_warp == 0 ? (x_tma ? x_bytes : 0u) + (go_tma ? go_bytes : 0u) : 0u;
                asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(full_bar), "r"(bytes) : "memory");
                if (r_warp == 0 && x_tma) tma_load_2d(smem + P.ring + b * P.ring_bytes, &x_map, 0, static_cast<int>(row0), full_bar);
                if (r_warp == 0 && go_tma) tma_load_2d(smem + P.ring + b * P.ring_bytes + go_at, &go_map, 0, static_cast<int>(row0), full_bar);
            }
            __syncwarp();
        }
        if (lane == 0) asm volatile("cp.async.bulk.wait_group 0;" ::: "memory");
        if (*abort_now && r_warp == 0 && lane == 0) drain_copies(tb.full, P.rings);
    } else {
        // ================= slots: own MMAs, epilogues =================
        const int slot = warp / (4 * W), wq = warp & 3;
        const int tid = threadIdx.x - slot * kSlotThreads;
        const int row = tid & 127, half = W == 2 ? tid >> 7 : 0;
        const uint32_t acc = tmem + slot * P.acc_cols;
        const uint32_t taddr = acc + (static_cast<uint32_t>(32 * wq) << 16);
        const uint32_t acc_bar = smem_addr(&tb.acc[slot]), ready_bar = smem_addr(&tb.ready[slot]), wdone_bar = smem_addr(&tb.wdone[slot]);
        const uint32_t tile0 = smem_base + static_cast<uint32_t>(slot) * slot_bytes;
        auto act_addr = [&](int l) { return tile0 + static_cast<uint32_t>(l - 1) * kTileBytes; };  // input of layer l > 0
        const float *bias = reinterpret_cast<const float *>(wsmem + P.w.bias_offset);
        const uint32_t row_off = row * 128, row_swizzle = (row & 7) << 4;
        // spread over the schedulers, slots 0 to 2 on others than the wgrad warp's, which slot 3 shares (all on it: 0.261 against 0.243 ms)
        const bool issuer = (tid >> 5) == ((slot + 1) & 3);
        uint32_t acc_phase = 0, wdone_phase = 0;
        bool alive = true;
        auto slot_sync = [&]() { asm volatile("bar.sync %0, %1;" ::"r"(slot + 1), "n"(kSlotThreads) : "memory"); };
        uint32_t buf = 0, rows0 = 0, prev_buf = 0, full_phase = 0, tiles_done = 0;
        // Biases and two accumulators: the recompute steps alternate between them, the last one in the first, so that a step's biases are
        // written while the step before it waits for its MMAs (2^20 rows 64-64-64-64 SiLU 304 -> 297 us, 300 007 rows
        // 32-3x64-3 132.2 -> 130.9)
        auto recompute_col = [&](int l) { return BIAS && kPreact && ((d - 1 - l) & 1) ? kAccCols : 0; };
        // operands written -> the slot's issuing warp issues the step's own MMAs (and hands the wgrad to the wgrad warp)
        auto start_step = [&](int j) {
            fence_async_smem();
            if constexpr (BIAS) tmem_st_wait();
            tc_fence_before();
            slot_sync();
            if (issuer && alive) {
                // elected here and not ahead of the loop: 2^20 rows 32-4x64-16 0.243 -> 0.226 ms (by the time; presumably the descriptors then
                // stay in uniform registers); the weight gradients' MMAs, which the chain's wait behind, are the better for not being: 0.228
                const bool leader = elect_one();
                tc_fence_after();
                if (j == 0) {
                    // the buffer of the tile before holds its input gradient now; this tile's rows
                    if (tiles_done > 0 && leader) asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_addr(&tb.empty[prev_buf])) : "memory");
                    if (tiles_done == 0 && use_tma) pipe_wait(smem_addr(&tb.weights_bar), 0, &tb.abort_flag);
                    pipe_wait(smem_addr(&tb.full[buf]), full_phase, &tb.abort_flag);
                    __syncwarp();
                }
                if (j >= d && leader) asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(ready_bar) : "memory");
                const SlotStep &st = tb.steps[j];
                const uint4 own = *reinterpret_cast<const uint4 *>(&st.a_off);
                if (own.z != 0) {
                    if (j == 0 || j == d) {
                        if (leader) {
                            const uint32_t a_low = desc_low(rows0 + own.x), b_low = desc_low(own.y), b_step = (own.w & 256u) ? 128 : 2;
                            for (int k = 0; k < static_cast<int>(own.w & 255u); ++k)
                                mma_f16(acc + (j == 0 ? recompute_col(0) : 0), desc_of(a_low + 2 * k, st.a_high), smem_desc(b_low + k * b_step), own.z, k > 0 || (BIAS && j == 0));
                        }
                    } else {
                        issue_gemm(leader, acc + (j < d ? recompute_col(j) : 0), tile0 + own.x, 32, own.y, (own.w & 256u) ? 2048 : 32, static_cast<int>(own.w & 255u), own.z, BIAS && j < d);
                    }
                    if constexpr (kPreact) {
                        if (st.z_k) {
                            if (st.flags & 8u) {
                                if (leader)
                                    for (int k = 0; k < static_cast<int>(st.z_k); ++k)
                                        mma_f16(acc + kAccCols, desc_of(desc_low(rows0) + 2 * k, desc_high(P.x_pitch)), smem_desc(desc_low(st.zb_addr) + 2 * k), instr_desc(128, s.h, bf16, 0, 0), BIAS || k > 0);
                            } else {
                                issue_gemm(leader, acc + kAccCols, tile0 + st.za_off, 32, st.zb_addr, 32, static_cast<int>(st.z_k), instr_desc(128, s.h, bf16, 0, 0), BIAS);
                            }
                        }
                    }
                    if (leader) mma_commit(acc_bar);
                }
                __syncwarp();
            }
        };
        auto finish_step = [&](bool own, bool wgrad) {
            // every warp polls: parking three of four warps at a barrier behind the polling one measured 2-6 % slower
            if (own) alive = pipe_wait(acc_bar, acc_phase, &tb.abort_flag) && alive;
            if (wgrad) alive = pipe_wait(wdone_bar, wdone_phase, &tb.abort_flag) && alive;
            __syncwarp();
            if (own) acc_phase ^= 1u;
            if (wgrad) wdone_phase ^= 1u;
            tc_fence_after();
            return alive;
        };
        [[maybe_unused]] int read = s.h;  // BIAS: accumulator columns that the slot has read last, half of them by each warpgroup
        for (long long k = slot; k < n_mine; k += S) {
            if constexpr (BIAS) {
                if constexpr (W == 2) start_half_from_bias(taddr + recompute_col(0), half, recompute_col(0) ? s.h : read, s.h, bias);
                else start_from_bias(taddr + recompute_col(0), 0, s.h, bias);
                if (gx != nullptr) read = s.ki;
            }
            buf = static_cast<uint32_t>(k % P.rings);
            full_phase = static_cast<uint32_t>((k / P.rings) & 1);
            rows0 = ring_of(buf);
            for (int l = 0; l < d; ++l) {  // recomputed activation of layer l -> input tile of layer l + 1
                start_step(l);
                if constexpr (BIAS && kPreact) {
                    // under the step's MMAs: the other accumulator is free, for the next step or for the pre-activation of the last layer
                    const int col = l + 1 < d ? recompute_col(l + 1) : kAccCols, layer = l + 1 < d ? l + 1 : d - 1;
                    start_from_bias(taddr + col, half * (s.h / W), (half + 1) * (s.h / W), bias + layer * kMaxDim);
                }
                if (finish_step(true, false)) {
                    const uint32_t dst = act_addr(l + 1) + row_off;
                    for_row_pieces<W>(taddr + recompute_col(l), s.h, half, [&](int chunk, const uint32_t(&piece)[8]) {
                        st_shared_16(dst + ((chunk << 4) ^ row_swizzle), finish8<T, ACT, false>(piece, nullptr));
                    });
                    if (BIAS && !kPreact && l + 1 < d) start_from_bias(taddr, half * (s.h / W), (half + 1) * (s.h / W), bias + (l + 1) * kMaxDim);
                }
            }
            for (int l = d; l >= 0; --l) {
                const int in_pad = l == 0 ? s.ki : s.h;
                start_step(2 * d - l);
                const bool ok = finish_step(l > 0 || gx != nullptr, true);
                if (l > 0 && ok) {  // dz of the layer below = dy * act', in place over that layer's parked output
                    const uint32_t parked = act_addr(l) + row_off;
                    if constexpr (kPreact) {
#pragma unroll 1
                        for (int u = 0; u < in_pad / (8 * W); ++u) {
                            const int chunk = half * (in_pad / 16) + u;
                            uint32_t dy[8], zz[8];
                            tmem_ld8(taddr + 8 * chunk, dy);
                            tmem_ld8(taddr + kAccCols + 8 * chunk, zz);
                            tmem_ld_wait();
                            float g[8];
#pragma unroll
                            for (int e = 0; e < 8; ++e) {
                                const float z = to_float<T>(from_float<T>(__uint_as_float(zz[e])));  // the forward pass stored z rounded
                                g[e] = activate_grad(ACT, z, __uint_as_float(dy[e]));
                            }
                            st_shared_16(parked + ((chunk << 4) ^ row_swizzle),
                                         make_uint4(pack_pair<T>(g[0], g[1]), pack_pair<T>(g[2], g[3]), pack_pair<T>(g[4], g[5]), pack_pair<T>(g[6], g[7])));
                        }
                        if (BIAS && l > 1) start_from_bias(taddr + kAccCols, half * (s.h / W), (half + 1) * (s.h / W), bias + (l - 2) * kMaxDim);
                    } else {
                        for_row_pieces<W>(taddr, in_pad, half, [&](int chunk, const uint32_t(&piece)[8]) {
                            const uint32_t off = (chunk << 4) ^ row_swizzle;
                            uint4 gq = finish8<T, TH_ACT_NONE, false>(piece, nullptr);
                            if constexpr (ACT == TH_ACT_RELU) {
                                const uint4 a = ld_shared_16(parked + off);
                                gq.x = keep_where_positive<T>(gq.x, a.x);
                                gq.y = keep_where_positive<T>(gq.y, a.y);
                                gq.z = keep_where_positive<T>(gq.z, a.z);
                                gq.w = keep_where_positive<T>(gq.w, a.w);
                            }
                            st_shared_16(parked + off, gq);
                        });
                    }
                } else if (ok && gx != nullptr) {
                    // into the tile's row buffer, whose readers are done: the row warps send it off
                    const uint32_t at = rows0 + row * P.x_pitch, swz = row_swizzle_of(row, P.x_pitch);
                    for_row_pieces<W>(taddr, in_pad, half, [&](int chunk, const uint32_t(&piece)[8]) {
                        st_shared_16(at + ((chunk ^ swz) << 4), finish8<T, TH_ACT_NONE, false>(piece, nullptr));
                    });
                    tc_fence_before();
                }
            }
            prev_buf = buf;
            ++tiles_done;
        }
        fence_async_smem();
        slot_sync();
        if (tiles_done > 0 && issuer && elect_one()) asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_addr(&tb.empty[prev_buf])) : "memory");
    }

    // ---- flush the weight gradients (M = 64 layout: lanes 0..15 of warp quarter q hold rows 16 q ..); a warpgroup per layer ----
    // (the slots have waited for every weight gradient; the row warps may still be sending the last rows off)
    if (!is_wgrad_warp && !is_row_warp) {
        tc_fence_before();
        asm volatile("bar.sync 14, %0;" ::"n"(128 * S * W) : "memory");
        tc_fence_after();
    }
    if (!tb.abort_flag && n_mine > 0 && !is_wgrad_warp && !is_row_warp) {
        const MlpGradWorkspace G = grad_workspace_layout(s, workspace);
        const int wq = warp & 3;
        const uint32_t lane_base = static_cast<uint32_t>(32 * wq) << 16;
        for (int l = warp >> 2; l <= d; l += S * W) {
            const int in_pad = l == 0 ? s.ki : s.h;
            const int in_dim = l == 0 ? s.d_in : s.d_hid, out_dim = l == d ? s.d_out : s.d_hid;
            float *dst = G.base + (l == 0 ? G.w_in : (l == d ? G.w_out : G.w_hid + (l - 1) * s.d_hid * s.d_hid));
            const int o = 16 * wq + lane;  // gradient row this lane holds
            if (l == d) {  // transposed: this lane holds input 16 wq + lane, a column an output
                for (int first = 0; first < s.no; first += 16) {
                    uint32_t raw[32];
                    tmem_ld16(tmem + lane_base + dw_col(l) + first, raw);
                    tmem_ld_wait();
                    if (lane < 16 && o < in_dim) {
#pragma unroll
                        for (int c = 0; c < 16; ++c)
                            if (first + c < out_dim) atomicAdd(dst + (first + c) * in_dim + o, __uint_as_float(raw[c]));
                    }
                }
            }
            const bool quads = in_dim % 4 == 0 && (reinterpret_cast<uintptr_t>(dst) & 15) == 0;
            for (int first = 0; l < d && first < in_pad; first += 16) {
                uint32_t raw[32];
                tmem_ld16(tmem + lane_base + dw_col(l) + first, raw);
                tmem_ld_wait();
                if (lane < 16 && o < out_dim) {
#pragma unroll
                    for (int c = 0; c < 16; c += 4) {
                        if (quads) {
                            if (first + c < in_dim)
                                asm volatile("red.global.add.v4.f32 [%0], {%1, %2, %3, %4};" ::"l"(dst + o * in_dim + first + c), "f"(__uint_as_float(raw[c])),
                                             "f"(__uint_as_float(raw[c + 1])), "f"(__uint_as_float(raw[c + 2])), "f"(__uint_as_float(raw[c + 3]))
                                             : "memory");
                        } else {
#pragma unroll
                            for (int e = 0; e < 4; ++e)
                                if (first + c + e < in_dim) atomicAdd(dst + o * in_dim + first + c + e, __uint_as_float(raw[c + e]));
                        }
                    }
                }
            }
            if constexpr (BIAS) {
                float *bdst = G.base + (l == 0 ? G.b_in : (l == d ? G.b_out : G.b_hid + (l - 1) * s.d_hid));
                uint32_t raw[8];
                tmem_ld8(tmem + lane_base + db_col(l), raw);
                tmem_ld_wait();
                if (lane < 16 && o < out_dim) atomicAdd(bdst + o, __uint_as_float(raw[0]));
            }
        }
    }
    if (tb.abort_flag && use_tma && threadIdx.x == 0) drain_copies(&tb.weights_bar, 1);
    tc_fence_before();
    __syncthreads();
    if (is_wgrad_warp)
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(static_cast<uint32_t>(P.tmem_cols)) : "memory");
}

bool one_slot_only() {
    static const bool off = [] {
        const char *v = getenv("TH_MLP_NO_SLOTS");
        return v && v[0] == '1';
    }();
    return off;
}

// A matrix of rows as boxes of 128 rows of a row buffer: `pitch` bytes of every row (zeros past the last column)
bool make_rows_map(CUtensorMap *map, const void *base, long long rows, int cols, int pitch, long long row_stride) {
    EncodeTiledFn encode = encode_tiled_fn();
    memset(map, 0, sizeof(*map));
    if (!encode || !base || cols % 8 != 0 || row_stride % 8 != 0 || !aligned_to(base, 16) || rows >= (1ll << 31) - kTileRows) return false;
    const cuuint64_t dims[2] = {static_cast<cuuint64_t>(cols), static_cast<cuuint64_t>(rows)};
    const cuuint64_t strides[1] = {static_cast<cuuint64_t>(row_stride) * 2};
    const cuuint32_t box[2] = {static_cast<cuuint32_t>(pitch / 2), kTileRows};
    const cuuint32_t elem[2] = {1, 1};
    return encode(map, CU_TENSOR_MAP_DATA_TYPE_UINT16, 2, const_cast<void *>(base), dims, strides, box, elem, CU_TENSOR_MAP_INTERLEAVE_NONE,
                  pitch == 128 ? CU_TENSOR_MAP_SWIZZLE_128B : (pitch == 64 ? CU_TENSOR_MAP_SWIZZLE_64B : CU_TENSOR_MAP_SWIZZLE_32B),
                  CU_TENSOR_MAP_L2_PROMOTION_L2_128B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

// S slots of W warpgroups and `rings` row buffers, if that fits one SM.
template <typename T, int ACT, bool BIAS, int S, int W>
int launch_slots(int rings, const MlpShape &s, const MlpParams &p, const void *x, int64_t x_stride, const void *go, int64_t go_stride,
                 void *gx, int64_t gx_stride, float *workspace, int64_t rows, cudaStream_t stream) {
    const SlotPlan P = slot_plan(s, S, rings);
    if (P.total > kSmemBudget || P.tmem_cols > 512 || 2 * s.depth + 1 > kStepsMax) return kTcNotApplicable;
    CUtensorMap x_map, go_map, gx_map;
    memset(&gx_map, 0, sizeof(gx_map));
    const bool x_tma = make_rows_map(&x_map, x, rows, s.d_in, P.x_pitch, x_stride), go_tma = make_rows_map(&go_map, go, rows, s.d_out, P.go_pitch, go_stride);
    const bool gx_tma = gx != nullptr && make_rows_map(&gx_map, gx, rows, s.d_in, P.x_pitch, gx_stride);
    // three slots of two warpgroups leave registers for one row warp
    constexpr bool kMayCopy = S * W <= 4;
    const bool copied = !(x_tma && go_tma && (gx_tma || gx == nullptr));
    if (copied && !kMayCopy) return kTcNotApplicable;
    int smem = P.total;
    if (smem < kSmemBudget / 2 + 1024) smem = kSmemBudget / 2 + 1024;  // one CTA per SM
    WeightMaps maps;
    const int use_tma = make_weight_maps(maps, s, p);
    auto kernel = slots_mlp_bwd_tc_kernel<T, ACT, BIAS, S, W, false>;
    if constexpr (kMayCopy)
        if (copied) kernel = slots_mlp_bwd_tc_kernel<T, ACT, BIAS, S, W, true>;
    if (int rc = cuda_status(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, smem),
                             "cudaFuncSetAttribute(slots_mlp_bwd_tc_kernel)")) return rc;
    const long long tiles = (rows + kTileRows - 1) / kTileRows;
    const long long cap = sm_count();
    kernel<<<static_cast<unsigned>(tiles < cap ? tiles : cap), 128 * S * W + 32 + 32 * (copied ? kRowWarps<true> : kRowWarps<false>), smem, stream>>>(
        s, p, maps, use_tma, x_map, go_map, gx_map, (x_tma ? 1 : 0) | (go_tma ? 2 : 0) | (gx_tma ? 4 : 0), P, static_cast<const T *>(x), x_stride,
        static_cast<const T *>(go), go_stride, static_cast<T *>(gx), gx_stride, workspace, rows);
    return launch_status("slots_mlp_bwd_tc_kernel launch");
}

// The most slots that fit are the fastest, two warpgroups per slot when there are threads left, and then one row buffer more than
// slots (B200, ms; with / without the spare buffer, before the issuers were spread): 2^21 rows 32-64-64-16 4 x 1 0.209 / 0.231, 3 x 2
// 0.250; 2^20 rows 32-4x64-16 2 x 2 0.265 / 0.293; 300 007 rows 32-3x64-16 with biases 3 x 2 0.069, 2 x 2 0.081; 2^18 rows 32-64-64-16
// with biases 4 x 1 0.043, 3 x 2 0.048.  Tried: dz in a tile of its own so that the chain waits for a weight gradient one step late (0.287
// at 32-4x64-16: MMAs run in the order of issue, and the next step's queue behind the weight gradient's all the same); the chain's A
// operands in tensor memory (0.304; the epilogue writes both places); unrolled loops over 32 columns (2^21 rows: 0.280 against 0.234).
template <typename T, int ACT, bool BIAS>
int launch_any_slots(const MlpShape &s, const MlpParams &p, const void *x, int64_t x_stride, const void *go, int64_t go_stride, void *gx,
                     int64_t gx_stride, float *workspace, int64_t rows, cudaStream_t stream) {
    // One or two tiles per CTA: two warpgroups walk a tile's chain faster than one, and there is nothing for more slots to do (2^14
    // rows 32-64-64-16 with biases: 13.6 us as 1 x 2, 14.6 as 2 x 2; two tiles, 18 945 to 37 888 rows, 2 x 2 against the most slots that
    // fit with rows fetched by the slots: 32-64-16 12.4 to 13.6 / 14.2 to 15.4, 32-64-64-16 16.8 / 19.1, 32-3x64-16 18.2 / 20.5).
    const int64_t tiles_per_cta = ((rows + kTileRows - 1) / kTileRows + sm_count() - 1) / sm_count();
#define TH_SLOTS(S, W)                                                                                                                        \
    for (int rings = S + 1; rings >= S; --rings)                                                                                              \
        if (const int rc = launch_slots<T, ACT, BIAS, S, W>(rings, s, p, x, x_stride, go, go_stride, gx, gx_stride, workspace, rows, stream); \
            rc != kTcNotApplicable)                                                                                                           \
            return rc;
    if (!one_slot_only() && tiles_per_cta > 1) {
        if (tiles_per_cta > 2) {
            TH_SLOTS(4, 1)
            TH_SLOTS(3, 2)
        }
        TH_SLOTS(2, 2)
    }
    TH_SLOTS(1, 2)
#undef TH_SLOTS
    return kTcNotApplicable;
}

template <typename T>
int launch_slots_act(const MlpShape &s, const MlpParams &p, const void *x, int64_t x_stride, const void *go, int64_t go_stride, void *gx,
                     int64_t gx_stride, float *workspace, int64_t rows, cudaStream_t stream) {
#define TH_SLOTS_ACT(A)                                                                                                      \
    (s.has_bias ? launch_any_slots<T, A, true>(s, p, x, x_stride, go, go_stride, gx, gx_stride, workspace, rows, stream)     \
                : launch_any_slots<T, A, false>(s, p, x, x_stride, go, go_stride, gx, gx_stride, workspace, rows, stream))
    switch (s.act) {
        case TH_ACT_RELU: return TH_SLOTS_ACT(TH_ACT_RELU);
        case TH_ACT_SILU: return TH_SLOTS_ACT(TH_ACT_SILU);
        case TH_ACT_RELU2: return TH_SLOTS_ACT(TH_ACT_RELU2);
        default: return TH_SLOTS_ACT(TH_ACT_NONE);
    }
#undef TH_SLOTS_ACT
}

}  // namespace

int mlp_bwd_slots(const MlpShape &s, const MlpParams &p, const void *x, int64_t x_stride, const void *go, int64_t go_stride, void *gx,
                  int64_t gx_stride, float *workspace, int64_t rows, int dtype, cudaStream_t stream) {
    switch (dtype) {
        case TH_F16: return launch_slots_act<__half>(s, p, x, x_stride, go, go_stride, gx, gx_stride, workspace, rows, stream);
        case TH_BF16: return launch_slots_act<__nv_bfloat16>(s, p, x, x_stride, go, go_stride, gx, gx_stride, workspace, rows, stream);
        default: return kTcNotApplicable;
    }
}

int mlp_bwd_slots_status() {
    int status = 0;
    if (cudaMemcpyFromSymbol(&status, g_tc_status, sizeof(int)) != cudaSuccess) return -1;
    return status;
}

}  // namespace th
