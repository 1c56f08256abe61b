// Fully fused MLP on the 5th-generation tensor cores (tcgen05.mma, accumulators in TMEM).
//
// A 128-row tile of the batch is the unit of work (M = 128 = the TMEM lanes; a thread that reads an
// accumulator reads the TMEM lanes of its warp quarter, thread = lane = tile row).  Every operand
// tile lives in shared memory in ONE layout: rows 128 bytes apart (64 16-bit features), 16-byte
// chunk c of row r stored at chunk position c ^ (r & 7), tile base 1024-byte aligned.  That is the
// canonical 128-byte-swizzle layout of the tensor core, and the same bytes can be described to it
// two ways:
//   K-major  (the row index is M or N, features are K)  - forward GEMMs, the A side of dgrad;
//   MN-major (the row index is K, features are M or N)  - wgrad (K = the tile's 128 rows) and
//            the weight side of dgrad (K = a layer's outputs, N = its inputs),
// so neither activations nor weights are ever transposed or stored twice.
//
//   forward : ACC[128 x out] = ACT_l[128 x in] . W_l^T        A K-major, B K-major
//   dgrad   : ACC[128 x in]  = DZ_l[128 x out] . W_l          A K-major, B MN-major
//   wgrad   : DW_l[out x in] += DZ_l^T[out x 128] . ACT_l     A, B MN-major, M = 64
//
// An elected lane issues the MMAs and commits them to an mbarrier; the epilogue threads read their
// part of the accumulator row with tcgen05.ld, apply bias / activation / ReLU mask on packed 16-bit
// pairs and write the next operand tile straight back to shared memory (fence.proxy.async before
// the tensor core reads it).  Weight gradients stay in TMEM columns for the whole life of the CTA
// (wgrad MMAs accumulate tile after tile) and leave once, at the end, as red.global.add.f32.
//
// The forward kernels are here, the backward in fused_mlp_bwd.cu:
//   mlp_fwd_tc_kernel   one tile per CTA of 256 threads, several CTAs per SM; the forward for rows
//                       TMA cannot describe
//   mlp_fwd_pipe_kernel one CTA per SM, up to five independent 128-thread slots with a tile each in
//                       flight, sharing the weights; input tiles by TMA - the usual forward
//
// Weights reach shared memory by TMA (cp.async.bulk.tensor.2d, one box per layer, 128-byte swizzle:
// the box lands directly in the operand-tile layout, zero filled where a layer is narrower than its
// padded tile); arrays TMA cannot describe (inner dimension not a multiple of 8 elements) are staged
// with plain loads instead.  No multicast: every CTA loads its own copy.
//
// Every wait is bounded: a stuck mbarrier sets a device-side status word and the CTA frees its
// TMEM and returns.  tcgen05.alloc cannot block for good because the launcher sizes shared
// memory so that the CTAs resident on one SM never ask for more than its 512 TMEM columns.
#include "mlp_tc_device.cuh"

namespace th {
namespace {

// ---- forward -----------------------------------------------------------------------------------
template <typename T, int ACT, bool BIAS>
__global__ void __launch_bounds__(kTcThreads, 3)
mlp_fwd_tc_kernel(const MlpShape s, const MlpParams p, const __grid_constant__ WeightMaps maps, const int use_tma,
                  const T *__restrict__ x, long long x_stride, T *__restrict__ y, long long y_stride, long long n_rows,
                  int x_vec, int y_vec) {
    extern __shared__ unsigned char smem_raw[];
    unsigned char *smem = reinterpret_cast<unsigned char *>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
    __shared__ uint32_t tmem_holder;
    __shared__ __align__(8) unsigned long long mbar;
    __shared__ int abort_flag;
    const TcPlan P = tc_plan(s, false);
    constexpr int bf16 = std::is_same<T, __half>::value ? 0 : 1;

    __shared__ __align__(8) unsigned long long wbar;
    if (threadIdx.x == 0) abort_flag = 0;
    stage_biases<T>(smem, P, s, p);
    bool weights_ok = true;
    if (use_tma) weights_ok = tma_stage_weights(smem, P, s, maps, &wbar);
    else stage_all_weights<T>(smem, P, s, p);
    const uint32_t tmem = cta_setup(&tmem_holder, &mbar, P.tmem_cols);
    if (!weights_ok) {  // the bytes never arrived: report and leave (after the barrier inside cta_setup)
        abort_flag = 1;
        g_tc_status = 1;
    }
    __syncthreads();
    const uint32_t bar = smem_addr(&mbar);
    const float *bias = reinterpret_cast<const float *>(smem + P.bias_offset);
    const Seat seat;
    const uint32_t taddr = tmem + seat.lane_base;
    if constexpr (BIAS) {
        start_half_from_bias(taddr, seat.group, s.h, s.h, bias);
        tmem_st_wait();
    }
    uint32_t phase = 0;
    const long long n_tiles = (n_rows + kTileRows - 1) / kTileRows;

    // Input tiles alternate between two buffers: while tile t runs through its layers in place in
    // buffer t & 1, tile t + 1 streams into the other one.
    auto start_input = [&](long long t, int b) {
        unsigned char *dst = smem + b * kTileBytes;
        if (x_vec) {
            async_tile_load<T>(dst, x, x_stride, t * kTileRows, n_rows, s.d_in, s.ki);
        } else {
            TileRegs regs;
            fetch_tile<T>(regs, x, x_stride, t * kTileRows, n_rows, s.d_in, s.ki, false);
            commit_tile(dst, regs, s.ki);
        }
    };
    int cur = 0;
    if (static_cast<long long>(blockIdx.x) < n_tiles) start_input(blockIdx.x, 0);
    for (long long tile = blockIdx.x; tile < n_tiles; tile += gridDim.x, cur ^= 1) {
        const long long row0 = tile * kTileRows;
        unsigned char *act_tile = smem + cur * kTileBytes;
        const uint32_t act_addr = smem_addr(act_tile);
        async_tile_wait();
        fence_async_smem();
        tc_fence_before();
        __syncthreads();
        if (abort_flag) break;
        // the other buffer is free (its tile finished before the barrier above): start the next input
        if (tile + gridDim.x < n_tiles) start_input(tile + gridDim.x, cur ^ 1);
        for (int l = 0; l <= s.depth; ++l) {
            const int in_pad = l == 0 ? s.ki : s.h;
            const int out_pad = l == s.depth ? s.no : s.h;
            if (threadIdx.x < 32) {
                const bool leader = elect_one();
                tc_fence_after();
                issue_gemm(leader, tmem, act_addr, 32, smem_addr(weight_tile(smem, P, s, l)), 32, in_pad / 16,
                           instr_desc(128, out_pad, bf16, 0, 0), BIAS);
                if (leader) mma_commit(bar);
                __syncwarp();
            }
            const bool ok = cta_wait_mma(bar, phase, &abort_flag);
            if (!ok) {
                g_tc_status = 1;
            } else if (l < s.depth) {
                hidden_epilogue<T, ACT>(taddr, seat, out_pad, act_tile);
            } else {
                const bool live = row0 + seat.row < n_rows;
                output_epilogue<T>(taddr, seat, out_pad, y + (live ? row0 + seat.row : 0) * y_stride, s.d_out, live, y_vec);
            }
            if constexpr (BIAS) {  // of the next layer, or of the next tile's first one
                const int next = l == s.depth ? 0 : l + 1;
                start_half_from_bias(taddr, seat.group, out_pad, next == s.depth ? s.no : s.h, bias + next * kMaxDim);
                tmem_st_wait();
            }
            if (l < s.depth) {
                fence_async_smem();
                tc_fence_before();
                __syncthreads();
                if (abort_flag) break;
            }
        }
        tc_fence_before();
        if (abort_flag) break;
    }
    cta_teardown(tmem, P.tmem_cols);
}

// ---- forward, several row tiles per CTA ------------------------------------------------------------
//
// The kernel above keeps one row tile per CTA in flight and every thread walks the same chain
// (issue, wait, epilogue, barrier); only co-resident CTAs overlap, and each of them needs its own
// copy of the weights.  Here one CTA per SM runs S independent "slots" of 128 threads (4 warps).
// A slot is what a CTA is above - it owns 64 TMEM columns (96 with its hidden activations there), one operand tile (two
// where those stay in shared memory) and its mbarriers, and walks its row tiles layer by layer - but the slots share the weights, and they never meet at a
// CTA-wide barrier after set-up, so one slot's MMAs run under the other slots' epilogues:
//
//   its issuing warp    : fetches the slot's next input tile by TMA (a box of 64 columns x 128 rows
//                         lands in the operand-tile layout; rows past the end and columns past
//                         d_in arrive as zeros), waits for the current one, issues each layer's
//                         GEMM, commits it to `acc_full` and polls that barrier;
//   all 4 warps         : meet at the slot's named barrier (the three other warps park there while
//                         the MMAs run), turn their accumulator rows (thread = tile row =
//                         TMEM lane) into the next layer's operand rows in place, or into output
//                         rows in global memory, and meet at the slot's named barrier.
//
// The prefetch of a slot's next tile lands in its one buffer once the first layer has read it, or (two buffers) in the other.
// Every mbarrier wait is bounded and watches a shared abort flag; after an abort a slot keeps the
// SAME sequence of named barriers (doing no work) so nobody is left waiting at one.

constexpr int kMaxSlots = 5;

// Wide output rows leave through shared memory: a warp rounds its 32 rows, 32 columns at a time, into 2 KB of staging and one TMA
// store writes the box.  Written by the threads, a row each, one instruction touches 32 lines for 16 bytes of each (2^18 rows, ten
// 64-wide layers: 5 000 cycles a tile for the output against 1 500; 0.0387 -> 0.0313 ms).  Rows of up to 32 bytes are whole
// sectors of neighbouring lines either way, and the staging costs more than it saves (2^20 rows 32-4x64-16: 0.0531 against 0.0517).
constexpr int kStageCols = 32;
constexpr int kStageBytes = 32 * kStageCols * 2;

// Shared memory of the multi-slot kernel: the TcPlan's tiles and weights, then the biases and the output staging.
struct PipePlan {
    TcPlan w;
    int bias;      // BIAS_MMA: operand tiles, four layers each; otherwise fp32 [(depth + 1)][64]
    int staging;   // kStageBytes per warp
    int total;     // excluding the 1 KB alignment slack
};

__host__ __device__ inline PipePlan pipe_plan(const MlpShape &s, int tiles, int slots, bool bias_mma, bool staged) {
    PipePlan p{};
    p.w = tc_plan(s, false, tiles);
    p.bias = p.w.bias_offset;
    p.staging = p.bias;
    if (s.has_bias) p.staging += bias_mma ? (s.depth / 4 + 1) * 64 * 128 : (s.depth + 1) * kMaxDim * 4;
    p.staging = (p.staging + 1023) & ~1023;
    p.total = p.staging + (staged ? slots * 4 * kStageBytes : 0);
    return p;
}

// How a kernel's output rows are written: element by element, in 16-byte chunks, or through the staging
constexpr int kRowsStaged = 2;

struct SlotBarriers {
    unsigned long long in_full[kMaxSlots][2];
    unsigned long long acc_full[kMaxSlots];
};

__device__ __forceinline__ void slot_barrier(int slot) {
    asm volatile("bar.sync %0, 128;" ::"r"(slot + 1) : "memory");
}

// TA: hidden activations go back to the tensor core through tensor memory (32 more columns per slot) instead of
// the operand tile in shared memory; the first layer still reads the TMA-fetched input tile.
// H64: the hidden width (padded) is 64 at compile time: one form of the hidden layers' epilogue and of their GEMMs' issue
// (2^20 rows 32-4x64-16: 0.058 -> 0.054 ms; 2^21 rows 32-64-64-16: 0.070 -> 0.065).
// BM: a layer's bias is one more K step of its GEMM, ahead of the others: A is a constant in tensor memory (element 0 of every row
// is one), B an operand tile whose element 16 (l % 4) of row n is b_l[n].  The elements beside it are zeros, so that no other layer's
// bias (it may be infinite) is multiplied by anything.  The additions in the epilogue it replaces cost 64 instructions and 16
// shared loads a row and layer, 600 of 2 900 cycles (2^18 rows, ten 64-wide layers: 0.0434 -> 0.0339 ms).  Without BM the epilogue
// of the layer before writes the biases into the accumulator.
template <typename T, int ACT, bool BIAS, int S, bool MSE, bool TA, bool H64, bool BM>
__global__ void __launch_bounds__(128 * S, 1)
mlp_fwd_pipe_kernel(const MlpShape shape, const MlpParams p, const __grid_constant__ WeightMaps maps,
                    const __grid_constant__ CUtensorMap x_map, const __grid_constant__ CUtensorMap y_map, T *__restrict__ y,
                    long long y_stride, long long n_rows, int y_vec, const MseArgs mse) {
    MlpShape s = shape;
    if constexpr (H64) s.h = 64;
    extern __shared__ unsigned char smem_raw[];
    unsigned char *smem = reinterpret_cast<unsigned char *>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
    __shared__ uint32_t tmem_holder;
    __shared__ int abort_flag;
    __shared__ __align__(8) unsigned long long wbar;
    __shared__ __align__(8) SlotBarriers bars;
    // TA: the input tile is free as soon as the first layer has read it, and the next one is fetched into it under the others:
    // one tile per slot, so that deep networks keep five slots too (2^18 rows, ten 64-wide layers: four slots 0.058 ms, five 0.051)
    constexpr int kBuffers = TA ? 1 : 2;
    constexpr bool kBiasMma = BIAS && BM;  // the epilogues have no bias to add
    static_assert(!BM || TA, "the bias step takes its A operand from tensor memory");
    const PipePlan plan = pipe_plan(s, kBuffers * S, S, BM, y_vec == kRowsStaged);
    const TcPlan &P = plan.w;
    constexpr int bf16 = std::is_same<T, __half>::value ? 0 : 1;
    constexpr uint32_t kTmemCols = S * (kAccCols + (TA ? 32 : 0)) + (kBiasMma ? 8 : 0) <= 256 ? 256 : 512;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;

    // ---- set-up: barriers, biases, weights, TMEM ----
    if (threadIdx.x == 0) {
        abort_flag = 0;
        for (int i = 0; i < S; ++i) {
            asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_addr(&bars.in_full[i][0])), "r"(1u) : "memory");
            asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_addr(&bars.in_full[i][1])), "r"(1u) : "memory");
            asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_addr(&bars.acc_full[i])), "r"(1u) : "memory");
        }
    }
    if constexpr (kBiasMma) {
        for (int e = threadIdx.x; e < (s.depth / 4 + 1) * 64 * 8; e += blockDim.x) {
            const int r = (e >> 3) & 63, c = (e & 7) ^ (r & 7), l = (e >> 9) * 4 + (c >> 1);  // 16-byte chunk c of row r holds K elements 8 c ..
            unsigned short v = 0;
            if ((c & 1) == 0 && l <= s.depth && r < (l == s.depth ? s.d_out : s.d_hid)) {
                const void *b = l == 0 ? p.b_in : (l == s.depth ? p.b_out : p.b_hid);
                v = static_cast<const unsigned short *>(b)[l == 0 || l == s.depth ? r : (l - 1) * s.d_hid + r];
            }
            reinterpret_cast<uint4 *>(smem + plan.bias)[e] = make_uint4(v, 0, 0, 0);
        }
        fence_async_smem();
    } else if constexpr (BIAS) {
        float *bias = reinterpret_cast<float *>(smem + plan.bias);
        for (int e = threadIdx.x; e < (s.depth + 1) * kMaxDim; e += blockDim.x) {
            const int layer = e / kMaxDim, c = e % kMaxDim;
            float v = 0.f;
            if (layer == 0) {
                if (c < s.d_hid) v = to_float<T>(static_cast<const T *>(p.b_in)[c]);
            } else if (layer < s.depth) {
                if (c < s.d_hid) v = to_float<T>(static_cast<const T *>(p.b_hid)[(layer - 1) * s.d_hid + c]);
            } else if (c < s.d_out) {
                v = to_float<T>(static_cast<const T *>(p.b_out)[c]);
            }
            bias[e] = v;
        }
    }
    if (threadIdx.x == 0) {
        asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_addr(&wbar)), "r"(1u) : "memory");
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        tma_issue_weights(smem, P, s, maps, &wbar);  // awaited by the issuers, ahead of their first MMA
    }
    if (warp == 0) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_addr(&tmem_holder)),
                     "r"(kTmemCols)
                     : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = tmem_holder;
    const float *bias = reinterpret_cast<const float *>(smem + plan.bias);
    const uint32_t one_tmem = tmem + S * (kAccCols + 32);
    if constexpr (kBiasMma) {
        if (warp < 4) {
            const uint32_t one[8] = {pack_pair<T>(1.f, 0.f), 0, 0, 0, 0, 0, 0, 0};
            tmem_st8(one_tmem + (static_cast<uint32_t>(32 * warp) << 16), one);
            tmem_st_wait();
        }
    } else if constexpr (BIAS) {
        start_from_bias(tmem + (warp >> 2) * kAccCols + (static_cast<uint32_t>(32 * (warp & 3)) << 16), 0, s.h, bias);
        tmem_st_wait();
    }
    if constexpr (BIAS) {
        tc_fence_before();
        __syncthreads();
        tc_fence_after();
    }

    const long long n_tiles = (n_rows + kTileRows - 1) / kTileRows;
    const long long first_tile = blockIdx.x;
    const long long n_mine = first_tile < n_tiles ? (n_tiles - first_tile + gridDim.x - 1) / gridDim.x : 0;

    // ---- the slot's life; nothing below depends on other slots ----
    const int slot = warp >> 2;
    // The issuing warps of the slots spread over the schedulers (the fifth shares the first's), and the lane that issues elected where it
    // issues: 2^20 rows 32-4x64-16 0.0497 -> 0.0477 ms; with the lane elected once, ahead of the loop, 0.0514 and 0.0560 (by the time;
    // presumably the descriptors then miss the uniform registers).
    const bool issuer = (warp & 3) == (slot & 3);
    const int row = 32 * (warp & 3) + lane;
    const uint32_t stage = smem_addr(smem + plan.staging) + static_cast<uint32_t>(warp) * kStageBytes;
    const uint32_t acc = tmem + slot * kAccCols;
    const uint32_t taddr = acc + (static_cast<uint32_t>(32 * (warp & 3)) << 16);
    const uint32_t act_tmem = tmem + S * kAccCols + slot * 32;  // TA: the slot's hidden activations, 16-bit pairs
    const uint32_t act_taddr = act_tmem + (static_cast<uint32_t>(32 * (warp & 3)) << 16);
    const uint32_t acc_bar = smem_addr(&bars.acc_full[slot]);
    unsigned char *buffers = smem + kBuffers * slot * kTileBytes;
    const uint32_t weights = smem_addr(smem + P.w_offset[0]);  // H64: every layer's tile 8 KB after the one before
    uint32_t acc_phase = 0;  // tracked by the issuer warp
    const bool early_target = MSE && s.no == 16 && !mse.target_f32;
    float loss = 0.f;        // MSE: this thread's share of sum (prediction - target)^2

    auto fetch_input = [&](int b, long long k) {  // by the issuer warp
        if (elect_one()) {
            const uint32_t bar = smem_addr(&bars.in_full[slot][b]);
            asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(static_cast<uint32_t>(kTileBytes))
                         : "memory");
            tma_load_2d(buffers + b * kTileBytes, &x_map, 0, static_cast<int>((first_tile + k * gridDim.x) * kTileRows), bar);
        }
        __syncwarp();
    };
    if (issuer && slot < n_mine) {
        fetch_input(0, slot);
        pipe_wait(smem_addr(&wbar), 0, &abort_flag);
    }

    for (long long k = slot, q = 0; k < n_mine; k += S, ++q) {
        const int b = TA ? 0 : static_cast<int>(q & 1);
        const long long row0 = (first_tile + k * gridDim.x) * kTileRows;
        unsigned char *tile = buffers + b * kTileBytes;
        const uint32_t tile_addr = smem_addr(tile);
        const uint32_t row_addr = tile_addr + row * 128, row_swizzle = (row & 7) << 4;  // chunk c of the row: row_addr + ((c << 4) ^ row_swizzle)
        if (issuer) {
            // the other buffer's last reader was the previous tile of this slot: finished
            if (!TA && k + S < n_mine && !*reinterpret_cast<volatile int *>(&abort_flag)) fetch_input(b ^ 1, k + S);
            pipe_wait(smem_addr(&bars.in_full[slot][b]), static_cast<uint32_t>((TA ? q : q >> 1) & 1), &abort_flag);
        }
        // MSE: this row's target.  Sixteen 16-bit columns are fetched here, ahead of the layers, so that the access (a random one where
        // the rows are ordered) is over when the output layer's epilogue needs it; of wider rows over an order a prefetch asks for the
        // first sector (2^21 rows with 16 targets, ordered: 0.119 with the prefetch, 0.088 with the loads).
        long long target_at = 0;
        uint4 target[2];
        if constexpr (MSE) {
            const long long r = row0 + row < n_rows ? row0 + row : 0;
            target_at = mse.order ? static_cast<long long>(__float_as_uint(__ldg(&mse.order[r].w))) : r;
            target[0] = target[1] = make_uint4(0, 0, 0, 0);
            if (early_target) {
                const uint4 *at = reinterpret_cast<const uint4 *>(static_cast<const T *>(mse.target) + target_at * mse.target_stride);
                target[0] = __ldcs(at);
                if (s.d_out > 8) target[1] = __ldcs(at + 1);
            }
        }
        for (int l = 0; l <= s.depth; ++l) {
            const int in_pad = l == 0 ? s.ki : s.h;
            const int out_pad = l == s.depth ? s.no : s.h;
            if constexpr (MSE) {
                if (l == 1 && mse.order && !early_target) {
                    const char *at = static_cast<const char *>(mse.target) + target_at * mse.target_stride * (mse.target_f32 ? 4 : 2);
                    asm volatile("prefetch.global.L2 [%0];" ::"l"(at));
                }
            }
            // Only the issuer warp polls the mbarrier; the slot's other warps park at the named barrier,
            // which costs no issue slots (all four polling: 2^21 rows 0.069 against 0.067 ms).  A wait that gives up raises
            // the abort flag; everybody reads it a step late, where the load costs nothing: work stops, the barrier sequence goes on.
            const int given_up = *reinterpret_cast<volatile int *>(&abort_flag);
            if (issuer) {
                if (__all_sync(0xffffffffu, !given_up)) {
                    const bool leader = elect_one();
                    tc_fence_after();
                    const uint32_t idesc = instr_desc(128, out_pad, bf16, 0, 0);
                    const uint32_t w_addr = H64 ? weights + static_cast<uint32_t>(l) * 64 * 128 : smem_addr(weight_tile(smem, P, s, l));
                    if constexpr (kBiasMma) {
                        if (leader) mma_f16_ta(acc, one_tmem, smem_desc(desc_low(smem_addr(smem + plan.bias) + (l >> 2) * 64 * 128) + 2 * (l & 3)), idesc, 0);
                    }
                    if (TA && l > 0)
                        issue_gemm_ta(leader, acc, act_tmem, w_addr, 32, H64 ? 4 : in_pad / 16, idesc, BIAS);
                    else
                        issue_gemm(leader, acc, tile_addr, 32, w_addr, 32, in_pad / 16, idesc, BIAS);
                    if (leader) mma_commit(acc_bar);
                    __syncwarp();
                    pipe_wait(acc_bar, acc_phase, &abort_flag);
                    acc_phase ^= 1u;
                    if (TA && l == 0 && k + S < n_mine && !*reinterpret_cast<volatile int *>(&abort_flag)) fetch_input(0, k + S);
                }
            }
            slot_barrier(slot);
            if (!given_up) {
                tc_fence_after();
                if (l < s.depth) {
                    if constexpr (TA) {
                        drain_row<T, ACT>(taddr, H64 ? 64 : out_pad, [&](int chunk, uint4 packed) { tmem_st4(act_taddr + 4 * chunk, packed); });
                        tmem_st_wait();
                    } else {
                        drain_row<T, ACT>(taddr, out_pad, [&](int chunk, uint4 packed) {
                            st_shared_16(row_addr + ((chunk << 4) ^ row_swizzle), packed);
                        });
                        fence_async_smem();
                    }
                } else {
                    const bool live = row0 + row < n_rows;
                    if constexpr (MSE) {
                        // d_out is a multiple of 8 and all rows are 16-byte aligned here (checked by the launcher)
                        const long long r = live ? row0 + row : 0;
                        const T *target_row = static_cast<const T *>(mse.target) + target_at * mse.target_stride;
                        const float *target_row_f32 = static_cast<const float *>(mse.target) + target_at * mse.target_stride;
                        T *grad_row = static_cast<T *>(mse.grad) + r * mse.grad_stride;
                        T *out_row = y ? y + r * y_stride : nullptr;
                        drain_row<T, TH_ACT_NONE>(taddr, out_pad, [&](int chunk, uint4 packed) {
                            if (live && 8 * chunk < s.d_out) {
                                if (out_row) __stcs(reinterpret_cast<uint4 *>(out_row + 8 * chunk), packed);
                                uint4 g;
                                if (mse.target_f32)
                                    g = mse_chunk_f32<T>(packed, target_row_f32 + 8 * chunk, mse.grad_scale, loss);
                                else
                                    g = mse_chunk<T>(packed, early_target ? (chunk == 0 ? target[0] : target[1]) : __ldcs(reinterpret_cast<const uint4 *>(target_row + 8 * chunk)),
                                                     mse.grad_scale, loss);
                                __stcs(reinterpret_cast<uint4 *>(grad_row + 8 * chunk), g);
                            }
                        });
                    } else {
                        T *out_row = y + (live ? row0 + row : 0) * y_stride;
                        if (y_vec == kRowsStaged) {
                            const uint32_t stage_row = stage + lane * (kStageCols * 2), stage_swizzle = ((lane >> 1) & 3) << 4;
#pragma unroll 1
                            for (int first = 0; first < out_pad; first += kStageCols) {
                                if (lane == 0) asm volatile("cp.async.bulk.wait_group.read 0;" ::: "memory");  // the box before has been read
                                __syncwarp();
                                uint32_t raw[32];
                                tmem_ld32(taddr + first, raw);  // (columns past out_pad are the slot's own and are not stored)
                                tmem_ld_wait();
#pragma unroll
                                for (int u = 0; u < 4; ++u)
                                    st_shared_16(stage_row + ((u << 4) ^ stage_swizzle), finish8<T, TH_ACT_NONE, false>(raw + 8 * u, nullptr));
                                fence_async_smem();
                                __syncwarp();
                                if (lane == 0 && row0 + 32 * (warp & 3) < n_rows) tma_store_2d(&y_map, stage, first, static_cast<int>(row0) + 32 * (warp & 3));
                            }
                        } else {
                            drain_row<T, TH_ACT_NONE>(taddr, out_pad, [&](int chunk, uint4 packed) {
                                if (live) store_chunk_to_global<T>(out_row, chunk, s.d_out, packed, y_vec);
                            });
                        }
                    }
                }
                if constexpr (BIAS && !BM) {  // of the next layer, or of the next tile's first one
                    const int next = l == s.depth ? 0 : l + 1;
                    start_from_bias(taddr, 0, next == s.depth ? s.no : s.h, bias + next * kMaxDim);
                    tmem_st_wait();
                }
                tc_fence_before();
            }
            slot_barrier(slot);
        }
    }

    if constexpr (MSE) {
        // one atomic per warp for the whole kernel
        for (int off = 16; off > 0; off >>= 1) loss += __shfl_xor_sync(0xffffffffu, loss, off);
        if ((threadIdx.x & 31) == 0 && mse.loss_sum) atomicAdd(mse.loss_sum, loss * mse.loss_scale);
    }

    // ---- teardown ----
    if (lane == 0) asm volatile("cp.async.bulk.wait_group 0;" ::: "memory");
    if (abort_flag && (threadIdx.x & 127) == 0) {
        drain_copies(bars.in_full[slot], 2);
        if (threadIdx.x == 0) drain_copies(&wbar, 1);
    }
    tc_fence_before();
    __syncthreads();
    if (warp == 0)
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(kTmemCols) : "memory");
}

constexpr int kPipeSmem = kSmemBudget - static_cast<int>(sizeof(SlotBarriers)) - 64;  // dynamic; the rest is the kernel's static shared memory

// One warp's box of an output matrix: 32 rows x 32 columns, 64-byte swizzle (16-byte chunk c of row r at c ^ (r / 2 % 4))
bool make_store_map(CUtensorMap *map, void *base, long long rows, int cols, long long row_stride) {
    EncodeTiledFn encode = encode_tiled_fn();
    if (!encode || cols % 8 != 0 || row_stride % 8 != 0 || !aligned_to(base, 16)) return false;
    const cuuint64_t dims[2] = {static_cast<cuuint64_t>(cols), static_cast<cuuint64_t>(rows)};
    const cuuint64_t strides[1] = {static_cast<cuuint64_t>(row_stride) * 2};
    const cuuint32_t box[2] = {kStageCols, 32};
    const cuuint32_t elem[2] = {1, 1};
    return encode(map, CU_TENSOR_MAP_DATA_TYPE_UINT16, 2, base, dims, strides, box, elem, CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_64B,
                  CU_TENSOR_MAP_L2_PROMOTION_NONE, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

bool pipe_disabled() {
    static const bool off = [] {
        const char *v = getenv("TH_MLP_NO_PIPE");
        return v && v[0] == '1';
    }();
    return off;
}

bool tmem_a_enabled() {
    static const bool on = [] {
        const char *v = getenv("TH_MLP_NO_TMEM_A");
        return !(v && v[0] == '1');
    }();
    return on;
}

template <typename T, int ACT, bool BIAS, int S, bool MSE, bool TA, bool BM = TA && BIAS>
int launch_fwd_pipe(const MlpShape &s, const MlpParams &p, const void *x, int64_t x_stride, void *y, int64_t y_stride,
                    int64_t rows, cudaStream_t stream, const MseArgs &mse = MseArgs{}) {
    CUtensorMap y_map;
    memset(&y_map, 0, sizeof(y_map));
    int y_vec = y ? rows_vector_ok(y, y_stride, s.d_out) : 0;
    if (!MSE && y_vec && s.no > 16 && pipe_plan(s, (TA ? 1 : 2) * S, S, BM, true).total + 1024 <= kPipeSmem && make_store_map(&y_map, y, rows, s.d_out, y_stride))
        y_vec = kRowsStaged;
    const int smem = pipe_plan(s, (TA ? 1 : 2) * S, S, BM, y_vec == kRowsStaged).total + 1024;
    if (smem > kPipeSmem || pipe_disabled()) return kTcNotApplicable;
    if (rows >= (1ll << 31) - kTileRows) return kTcNotApplicable;  // TMA coordinates are 32-bit
    WeightMaps maps;
    CUtensorMap x_map;
    if (!make_weight_maps(maps, s, p)) return kTcNotApplicable;
    if (!make_map(&x_map, x, rows, s.d_in, kTileRows, x_stride)) return kTcNotApplicable;
    if (S * (kAccCols + (TA ? 32 : 0)) > 512) return kTcNotApplicable;
    auto kernel = TA && BM == BIAS && s.h == 64 ? mlp_fwd_pipe_kernel<T, ACT, BIAS, S, MSE, TA, TA && BM == BIAS, BM> : mlp_fwd_pipe_kernel<T, ACT, BIAS, S, MSE, TA, false, BM>;
    if (int rc = cuda_status(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, smem),
                             "cudaFuncSetAttribute(mlp_fwd_pipe_kernel)")) return rc;
    const long long tiles = (rows + kTileRows - 1) / kTileRows;
    const long long cap = sm_count();
    kernel<<<static_cast<unsigned>(tiles < cap ? tiles : cap), 128 * S, smem, stream>>>(
        s, p, maps, x_map, y_map, static_cast<T *>(y), y_stride, rows, y_vec, mse);
    return launch_status("mlp_fwd_pipe_kernel launch");
}

// Slots per CTA, measured (2^21 rows, 32-64-64-16, with the loss; 2^20 rows, 32-4x64-16):
//   activations through shared memory: 3 slots 0.136 ms, 4: 0.122 / 0.083, 5: 0.127 / 0.098, 6: 0.153 - MMA operand reads and
//     epilogue stores share the SM's shared-memory bandwidth, and beyond four tiles in flight they only queue up;
//   activations through tensor memory: 3 slots 0.128 / 0.088, 4: 0.104 / 0.069, 5: 0.092 / 0.064 - five slots x 96 columns are
//     what tensor memory holds.
// TH_MLP_SLOTS=n lowers the cap (0 = never), TH_MLP_NO_TMEM_A=1 keeps the activations in shared memory.
template <typename T, int ACT, bool BIAS, bool MSE>
int launch_fwd_slots(const MlpShape &s, const MlpParams &p, const void *x, int64_t x_stride, void *y, int64_t y_stride,
                     int64_t rows, cudaStream_t stream, const MseArgs &mse) {
    static const int cap = [] {
        const char *v = getenv("TH_MLP_SLOTS");
        return v ? atoi(v) : 5;
    }();
    int rc = kTcNotApplicable;
    if (tmem_a_enabled()) {
        if (cap >= 5) rc = launch_fwd_pipe<T, ACT, BIAS, 5, MSE, true>(s, p, x, x_stride, y, y_stride, rows, stream, mse);
        if (rc == kTcNotApplicable && cap >= 4) rc = launch_fwd_pipe<T, ACT, BIAS, 4, MSE, true>(s, p, x, x_stride, y, y_stride, rows, stream, mse);
        if (rc == kTcNotApplicable && cap >= 3) rc = launch_fwd_pipe<T, ACT, BIAS, 3, MSE, true>(s, p, x, x_stride, y, y_stride, rows, stream, mse);
        // networks of 18 layers and more, whose weights leave no room for the biases' operand tiles
        if constexpr (BIAS)
            if (rc == kTcNotApplicable && cap >= 3) rc = launch_fwd_pipe<T, ACT, BIAS, 3, MSE, true, false>(s, p, x, x_stride, y, y_stride, rows, stream, mse);
        return rc;
    }
    if (cap >= 4) rc = launch_fwd_pipe<T, ACT, BIAS, 4, MSE, false>(s, p, x, x_stride, y, y_stride, rows, stream, mse);
    if (rc == kTcNotApplicable && cap >= 3) rc = launch_fwd_pipe<T, ACT, BIAS, 3, MSE, false>(s, p, x, x_stride, y, y_stride, rows, stream, mse);
    return rc;
}

template <typename T, int ACT, bool BIAS>
int launch_fwd_t(const MlpShape &s, const MlpParams &p, const void *x, int64_t x_stride, void *y, int64_t y_stride,
                 int64_t rows, cudaStream_t stream) {
    {
        const int rc = launch_fwd_slots<T, ACT, BIAS, false>(s, p, x, x_stride, y, y_stride, rows, stream, MseArgs{});
        if (rc != kTcNotApplicable) return rc;
    }
    const TcPlan P = tc_plan(s, false);
    int ctas = 0;
    const int smem = occupancy_plan(P, &ctas);
    if (ctas < 1) return kTcNotApplicable;
    auto kernel = mlp_fwd_tc_kernel<T, ACT, BIAS>;
    if (int rc = cuda_status(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, smem),
                             "cudaFuncSetAttribute(mlp_fwd_tc_kernel)")) return rc;
    const long long tiles = (rows + kTileRows - 1) / kTileRows;
    const long long cap = static_cast<long long>(sm_count()) * ctas;
    WeightMaps maps;
    const int use_tma = make_weight_maps(maps, s, p);
    kernel<<<static_cast<unsigned>(tiles < cap ? tiles : cap), kTcThreads, smem, stream>>>(
        s, p, maps, use_tma, static_cast<const T *>(x), x_stride, static_cast<T *>(y), y_stride, rows,
        rows_vector_ok(x, x_stride, s.d_in), rows_vector_ok(y, y_stride, s.d_out));
    return launch_status("mlp_fwd_tc_kernel launch");
}

template <typename T, bool BIAS>
int launch_fwd_act(const MlpShape &s, const MlpParams &p, const void *x, int64_t x_stride, void *y, int64_t y_stride,
                   int64_t rows, cudaStream_t stream) {
    switch (s.act) {
        case TH_ACT_RELU: return launch_fwd_t<T, TH_ACT_RELU, BIAS>(s, p, x, x_stride, y, y_stride, rows, stream);
        case TH_ACT_SILU: return launch_fwd_t<T, TH_ACT_SILU, BIAS>(s, p, x, x_stride, y, y_stride, rows, stream);
        case TH_ACT_RELU2: return launch_fwd_t<T, TH_ACT_RELU2, BIAS>(s, p, x, x_stride, y, y_stride, rows, stream);
        default: return launch_fwd_t<T, TH_ACT_NONE, BIAS>(s, p, x, x_stride, y, y_stride, rows, stream);
    }
}

template <typename T>
int launch_fwd(const MlpShape &s, const MlpParams &p, const void *x, int64_t x_stride, void *y, int64_t y_stride,
               int64_t rows, cudaStream_t stream) {
    return s.has_bias ? launch_fwd_act<T, true>(s, p, x, x_stride, y, y_stride, rows, stream)
                      : launch_fwd_act<T, false>(s, p, x, x_stride, y, y_stride, rows, stream);
}

// ---- forward with the fused MSE epilogue: only the multi-slot kernel has it ----

template <typename T, bool BIAS>
int launch_fwd_mse_act(const MlpShape &s, const MlpParams &p, const void *x, int64_t x_stride, void *y, int64_t y_stride,
                       const MseArgs &mse, int64_t rows, cudaStream_t stream) {
    switch (s.act) {
        case TH_ACT_RELU: return launch_fwd_slots<T, TH_ACT_RELU, BIAS, true>(s, p, x, x_stride, y, y_stride, rows, stream, mse);
        case TH_ACT_SILU: return launch_fwd_slots<T, TH_ACT_SILU, BIAS, true>(s, p, x, x_stride, y, y_stride, rows, stream, mse);
        case TH_ACT_RELU2: return launch_fwd_slots<T, TH_ACT_RELU2, BIAS, true>(s, p, x, x_stride, y, y_stride, rows, stream, mse);
        default: return launch_fwd_slots<T, TH_ACT_NONE, BIAS, true>(s, p, x, x_stride, y, y_stride, rows, stream, mse);
    }
}

template <typename T>
int launch_fwd_mse(const MlpShape &s, const MlpParams &p, const void *x, int64_t x_stride, void *y, int64_t y_stride,
                   const MseArgs &mse, int64_t rows, cudaStream_t stream) {
    return s.has_bias ? launch_fwd_mse_act<T, true>(s, p, x, x_stride, y, y_stride, mse, rows, stream)
                      : launch_fwd_mse_act<T, false>(s, p, x, x_stride, y, y_stride, mse, rows, stream);
}

}  // namespace

int mlp_fwd_mse_tc(const MlpShape &s, const MlpParams &p, const void *x, int64_t x_stride, void *y, int64_t y_stride,
                   const MseArgs &mse, int64_t rows, int dtype, cudaStream_t stream) {
    if (tc_disabled() || rows <= 0) return kTcNotApplicable;
    if (s.h != 16 && s.h != 32 && s.h != 64) return kTcNotApplicable;
    // whole 16-byte chunks of every row: prediction (if kept), target and gradient
    const bool target_ok = mse.target_f32 ? aligned_to(mse.target, 16) && mse.target_stride % 4 == 0
                                          : rows_vector_ok(mse.target, mse.target_stride, s.d_out);
    if (s.d_out % 8 != 0 || !target_ok ||
        !rows_vector_ok(mse.grad, mse.grad_stride, s.d_out) || (y && !rows_vector_ok(y, y_stride, s.d_out)))
        return kTcNotApplicable;
    switch (dtype) {
        case TH_F16: return launch_fwd_mse<__half>(s, p, x, x_stride, y, y_stride, mse, rows, stream);
        case TH_BF16: return launch_fwd_mse<__nv_bfloat16>(s, p, x, x_stride, y, y_stride, mse, rows, stream);
        default: return kTcNotApplicable;
    }
}

int mlp_fwd_tc(const MlpShape &s, const MlpParams &p, const void *x, int64_t x_stride, void *y, int64_t y_stride,
               int64_t rows, int dtype, cudaStream_t stream) {
    if (tc_disabled() || rows <= 0) return kTcNotApplicable;
    if (s.h != 16 && s.h != 32 && s.h != 64) return kTcNotApplicable;
    switch (dtype) {
        case TH_F16: return launch_fwd<__half>(s, p, x, x_stride, y, y_stride, rows, stream);
        case TH_BF16: return launch_fwd<__nv_bfloat16>(s, p, x, x_stride, y, y_stride, rows, stream);
        default: return kTcNotApplicable;
    }
}

int mlp_bwd_tc(const MlpShape &s, const MlpParams &p, const void *x, int64_t x_stride, const void *go, int64_t go_stride,
               void *gx, int64_t gx_stride, float *workspace, int64_t rows, int dtype, cudaStream_t stream) {
    if (tc_disabled() || rows <= 0) return kTcNotApplicable;
    if (s.h != 16 && s.h != 32 && s.h != 64) return kTcNotApplicable;
    return mlp_bwd_slots(s, p, x, x_stride, go, go_stride, gx, gx_stride, workspace, rows, dtype, stream);
}

}  // namespace th


// 1 when tensor maps can be built in this process (the driver exposes cuTensorMapEncodeTiled), i.e.
// when the tensor-core MLP kernels load their weights by TMA; 0 when they fall back to plain loads.
extern "C" int th_mlp_tma_available(void) { return th::encode_tiled_fn() != nullptr ? 1 : 0; }

namespace th {
int field_tc_status_word();  // neural_field.cu: the fused encoding + MLP kernels' copy of the status word
}

// Device-side status of the tcgen05 kernels: 0 = fine, non-zero = a bounded wait ran out.  Synchronises.
extern "C" int th_mlp_tc_status(void) {
    int status = 0;
    if (cudaMemcpyFromSymbol(&status, th::g_tc_status, sizeof(int)) != cudaSuccess) return -1;
    const int field = th::field_tc_status_word(), slots = th::mlp_bwd_slots_status();
    if (field < 0 || slots < 0) return -1;
    return status | ((field & 1) << 1) | (slots << 2);
}
