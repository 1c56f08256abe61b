// Reversible (additive coupling) fused MLP on the 5th-generation tensor cores.
//
// The residual stream of a 128-row tile lives in TENSOR MEMORY as fp32 for the whole stack:
// x1 in one 64-column accumulator, x2 in another.  A branch y = x + W2 . act(W1 . u) is two GEMMs,
// and the second one simply accumulates into the stream's own columns (enable-input-d), so the
// residual add costs nothing; the backward pass undoes a branch with the same GEMM and the
// A operand negated (x = y - W2 . act(W1 . u)), and the gradient stream (also fp32 in TMEM)
// receives its dgrad the same way.  Only what the tensor core must read as an operand is rounded
// to 16 bits and written to a shared-memory operand tile by the epilogue threads.
//
//   forward, per branch:   HID = U . W1^T                       U = 16-bit copy of the input stream
//                          OUT += act(HID) . W2^T               OUT = the other stream, in TMEM
//   backward, per branch:  HID = U . W1^T ,  DH = DY . W2       (one commit: recompute + dgrad)
//                          OUT += (-act(HID)) . W2^T            reconstruct the branch's input side
//                          IN_D += DZ . W1                      gradient into the input stream
//                          DW2 = DY^T . act(HID) , DW1 = DZ^T . U     (M = 64, K = the 128 rows)
//
// Weights (4 matrices per block) stream block by block through a two-stage cp.async ring in the
// operand-tile layout; the same tile is read K-major by the forward GEMMs and MN-major by dgrad.
// Weight gradients of a (tile, block, branch) leave TMEM for staging in shared memory and from there as bulk reductions
// (cp.reduce.async.bulk, 4 KB each) for the CTA's own fp32 accumulators in global memory, carried out by four extra warps while
// the other eight are already in the next branch; a reduction kernel sums the CTAs' copies.  As vector reductions of the four warps they
// shared the load / store pipe with the chain's stores: 32 KB a branch, 17 % of the kernel (2^19 rows, eight blocks of 64 -> 64 -> 64:
// 0.872 -> 0.757 ms, 0.72 with no reductions at all).  An accumulator has one owner, whose first tile writes it and whose later ones add
// to it in order, so the weight gradients are the same bits at every call.  (Sixteen copies that all CTAs add to in the order of
// arrival: 1 to 6 % less time from 20 000 rows on, up to 11 % at ten blocks, for the shorter sum over the copies; gradients that vary from
// call to call.  Cleared copies, only added to: 3 to 34 % more.)
//
// The chain's A operands (U and DY, h and dz) lie in 64 TMEM columns besides their tiles, which the weight gradients read: an MMA
// then takes 43 cycles instead of 76.  The two weight-gradient accumulators (M = 64) share 64 columns, one in lanes 0..15 and one in
// lanes 16..31 of every quarter.  Backward 512 columns, one CTA per SM; forward 192 (256 allocated), two.
//
// Bias gradients are column sums of the DY and DZ tiles, formed by the flush warps while the chain goes on (in the chain's
// epilogues they cost 2 us a pass): tensor memory has no columns left for the MMA with ones that the fused MLP uses.
//
// Measured, backward: with biases and SiLU, 2^17 rows, six blocks of 64 -> 64 -> 64 0.397 -> 0.360 ms; without biases, ReLU, eight
// blocks, 2^19 rows 0.885 -> 0.731 ms, 5 003 rows 34 us (graph replays, the sum over the copies included).
//
// Covered here: float16 / bfloat16, 16-byte-aligned rows.  Everything else stays on the mma.sync kernels.
#include "rev_shape.cuh"
#include "tc_tiles.cuh"

#include <cstdlib>
#include <cstring>
#include <type_traits>

namespace th {
namespace {

constexpr int kWTileBytes = 64 * 128;            // one weight matrix as an operand tile
constexpr int kStageBytes = 4 * kWTileBytes;     // [f1 | f2 | g1 | g2]
// TMEM columns
constexpr int kS1 = 0, kS2 = 64;                 // the stream
constexpr int kFwdHid = 128;                     // forward: hidden pre-activation
constexpr int kFwdAU = 192, kFwdAH = 224;        // forward: 16-bit A operands (the branch's input, its hidden activation), 32 columns each
constexpr int kD1 = 128, kD2 = 192, kZ = 256, kDH = 320, kDW1 = 384, kDW2 = 384 + (16 << 16), kA0 = 448, kA1 = 480;  // backward; kDW2: lanes 16..31

struct RevTcPlan {
    int tiles;     // operand tiles before the weight ring (2 forward, 8 backward)
    int ring;      // byte offset of the ring (2 stages)
    int bias;      // fp32 [2 stages][4][64]
    int stage;     // backward: 8 KB of weight gradients per flush warp
    int total;
    int tmem_cols;
};

__host__ __device__ constexpr RevTcPlan rev_tc_plan(bool backward) {
    RevTcPlan p{};
    p.tiles = backward ? 8 : 2;
    p.ring = p.tiles * kTileBytes;
    p.bias = p.ring + 2 * kStageBytes;
    p.stage = p.bias + 2 * 4 * kMaxDim * 4;
    p.total = p.stage + (backward ? 32768 : 0);
    p.tmem_cols = backward ? 512 : 256;
    return p;
}
// one backward CTA per SM, two forward ones, beside 1 KB of the kernels' static variables each
static_assert(rev_tc_plan(true).total + 1024 <= kSmemBudget && 2 * (rev_tc_plan(false).total + 1024) <= kSmemBudget);

// Operand tiles need their alignment, which the shared memory's declaration asks for: should the base be another one, all threads leave
// before anything is set up, with the status word raised.
__device__ __forceinline__ bool misplaced(const unsigned char *smem) {
    if ((smem_addr(smem) & 1023u) == 0) return false;
    g_tc_status = 1;
    return true;
}

// Queue block k's four weight matrices into ring stage `stage` (cp.async, operand-tile layout).
// A call, not inlined: the kernels live on their instruction cache and almost never come here.
template <typename T>
__device__ __noinline__ void prefetch_weights(unsigned char *smem, const RevTcPlan &P, const RevShape &s, const RevParams &p, int k,
                                 int stage) {
    const T *src[4] = {static_cast<const T *>(p.w_f1), static_cast<const T *>(p.w_f2), static_cast<const T *>(p.w_g1),
                       static_cast<const T *>(p.w_g2)};
#pragma unroll
    for (int m = 0; m < 4; ++m) {
        const int rows = (m & 1) ? s.half : s.hid, cols = (m & 1) ? s.hid : s.half;
        unsigned char *tile = smem + P.ring + stage * kStageBytes + m * kWTileBytes;
        const T *g = src[m] + static_cast<size_t>(k) * rows * cols;
        const int chunks = cols / 8;
        for (int id = threadIdx.x; id < rows * chunks; id += kTcThreads) {
            const int r = id / chunks, c = id - r * chunks;
            asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(smem_addr(chunk_ptr(tile, r, c))),
                         "l"(g + r * cols + 8 * c)
                         : "memory");
        }
    }
    if (s.has_bias) {
        float *bias = reinterpret_cast<float *>(smem + P.bias) + stage * 4 * kMaxDim;
        const T *bsrc[4] = {static_cast<const T *>(p.b_f1), static_cast<const T *>(p.b_f2), static_cast<const T *>(p.b_g1),
                            static_cast<const T *>(p.b_g2)};
        for (int e = threadIdx.x; e < 4 * kMaxDim; e += kTcThreads) {
            const int m = e / kMaxDim, c = e % kMaxDim;
            const int width = (m & 1) ? s.half : s.hid;
            bias[e] = c < width ? to_float<T>(bsrc[m][k * width + c]) : 0.f;
        }
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
}

// The same by TMA: one 64-column box per matrix lands in the operand-tile layout, issued by one thread
// and counted on the ring stage's mbarrier (the cp.async version above keeps every thread busy for
// ~1 800 cycles per block).  Biases, when present, still come with plain loads.
struct RevWeightMaps {
    CUtensorMap m[4];  // w_f1, w_f2, w_g1, w_g2: [blocks * rows][cols], 16-bit
};

// What a kernel knows of the widths at compile time, and the form of its code that goes with it:
//   <64, 64>  everything: one form of every epilogue and of every GEMM's issue remains (2^20 rows, eight blocks, forward
//             0.63 -> 0.50 ms, backward 1.97 -> 1.69)
//   <h, 0>    the half: the hidden layer's epilogue and issue keep a form per width
//   <0, 0>    nothing: rolled loops
// 2^17 rows, eight float16 blocks of 32 -> 32 -> 32, ReLU without biases: <0, 0> forward 78, backward 248 us, <32, 0> 62 and 211;
// 16 -> 16 -> 16: 66 and 240, 57 and 193; 48 -> 48 -> 48: 88 and 307, 71 and 253.
template <int HALF, int HID>
__device__ __forceinline__ RevShape known_widths(RevShape s) {
    if constexpr (HALF > 0) s.half = HALF;
    if constexpr (HID > 0) s.hid = HID;
    return s;
}

// The row tiles of the backward pass, a column half of y or of the output gradient each: [rows][half], box = 128 rows
struct RevRowMaps {
    CUtensorMap y1, y2, go1, go2;
};

template <typename T, bool BIAS>
__device__ __forceinline__ void prefetch_weights_tma(unsigned char *smem, const RevTcPlan &P, const RevShape &s, const RevParams &p,
                                     const RevWeightMaps &maps, unsigned long long *ring_bars, int k, int stage, volatile int *abort_now = nullptr) {
    if (threadIdx.x == 64 && !(abort_now && *abort_now)) {  // not warp 0, which is about to issue MMAs
        const uint32_t bar = smem_addr(&ring_bars[stage]);
        const uint32_t bytes = static_cast<uint32_t>(2 * (s.hid + s.half) * 128);  // four boxes of 64 columns
        asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(bytes) : "memory");
#pragma unroll
        for (int m = 0; m < 4; ++m) {
            const int rows = (m & 1) ? s.half : s.hid;
            tma_load_2d(smem + P.ring + stage * kStageBytes + m * kWTileBytes, &maps.m[m], 0, k * rows, bar);
        }
    }
    if constexpr (BIAS) {
        float *bias = reinterpret_cast<float *>(smem + P.bias) + stage * 4 * kMaxDim;
        const T *bsrc[4] = {static_cast<const T *>(p.b_f1), static_cast<const T *>(p.b_f2), static_cast<const T *>(p.b_g1),
                            static_cast<const T *>(p.b_g2)};
        for (int e = threadIdx.x; e < 4 * kMaxDim; e += kTcThreads) {
            const int m = e / kMaxDim, c = e % kMaxDim;
            const int width = (m & 1) ? s.half : s.hid;
            bias[e] = c < width ? to_float<T>(bsrc[m][k * width + c]) : 0.f;
        }
    }
}

// Warp 0 waits (bounded) for the ring stage used by running step `step`; the CTA barrier that follows
// in the caller hands the result to everybody.
__device__ __forceinline__ void ring_wait(unsigned long long *ring_bars, int step, int *abort_flag) {
    if (threadIdx.x < 32 && !mbar_wait(smem_addr(&ring_bars[step & 1]), static_cast<uint32_t>((step >> 1) & 1))) *abort_flag = 1;
}

// This thread's pieces of a 16-bit operand tile row -> fp32 in TMEM (stream initialisation)
template <typename T>
__device__ __forceinline__ void tile_row_to_tmem(unsigned char *tile, const Seat &seat, int width, uint32_t taddr) {
    const int count = width / (8 * kGroups), first = seat.group * count;
#pragma unroll
    for (int u = 0; u < kMaxChunks; ++u) {
        if (u < count) {
            uint32_t wide[8];
            widen_chunk<T>(*reinterpret_cast<const uint4 *>(chunk_ptr(tile, seat.row, first + u)), wide);
            tmem_st8(taddr + 8 * (first + u), wide);
        }
    }
}

// This thread's pieces of an fp32 TMEM accumulator -> (optional bias, written back) -> rounded into an
// operand tile and / or a global row.
template <typename T, bool BIAS, bool ROLLED>
__device__ __forceinline__ void stream_epilogue(uint32_t taddr, const Seat &seat, int width, const float *bias,
                                                unsigned char *tile, T *global_row, bool live) {
    const int n = width / kGroups, first = seat.group * (n / 8);  // this thread's columns / first 8-column piece
    const uint32_t row_addr = (tile ? smem_addr(tile) : 0u) + seat.row * 128, row_swizzle = (seat.row & 7) << 4;
    for_each_piece<ROLLED>(taddr + seat.group * n, n, [&](int u, const uint32_t(&piece)[8]) {
        uint32_t v[8];
#pragma unroll
        for (int k = 0; k < 8; ++k) v[k] = piece[k];
        if constexpr (BIAS) {
#pragma unroll
            for (int k = 0; k < 8; ++k) v[k] = __float_as_uint(__uint_as_float(v[k]) + bias[8 * (first + u) + k]);
            tmem_st8(taddr + 8 * (first + u), v);
        }
        const uint4 packed = finish8<T, TH_ACT_NONE, false>(v, nullptr);
        if (tile) st_shared_16(row_addr + (((first + u) << 4) ^ row_swizzle), packed);
        if (global_row && live) __stcs(reinterpret_cast<uint4 *>(global_row + 8 * (first + u)), packed);
    });
    if constexpr (BIAS) tmem_st_wait();
}

// The same with the rounded copy going to a 16-bit A operand in tensor memory (4 columns per 16-byte chunk).
template <typename T, bool BIAS, bool ROLLED>
__device__ __forceinline__ void stream_epilogue_ta(uint32_t taddr, const Seat &seat, int width, const float *bias, uint32_t a_taddr,
                                                   T *global_row, bool live) {
    const int n = width / kGroups, first = seat.group * (n / 8);
    for_each_piece<ROLLED>(taddr + seat.group * n, n, [&](int u, const uint32_t(&piece)[8]) {
        uint32_t v[8];
#pragma unroll
        for (int k = 0; k < 8; ++k) v[k] = piece[k];
        if constexpr (BIAS) {
#pragma unroll
            for (int k = 0; k < 8; ++k) v[k] = __float_as_uint(__uint_as_float(v[k]) + bias[8 * (first + u) + k]);
            tmem_st8(taddr + 8 * (first + u), v);
        }
        const uint4 packed = finish8<T, TH_ACT_NONE, false>(v, nullptr);
        tmem_st4(a_taddr + 4 * (first + u), packed);
        if (global_row && live) __stcs(reinterpret_cast<uint4 *>(global_row + 8 * (first + u)), packed);
    });
    tmem_st_wait();
}

__device__ __forceinline__ bool commit_and_wait(bool leader, uint32_t bar, uint32_t &phase, int *abort_flag) {
    if (threadIdx.x < 32) {
        if (leader) mma_commit(bar);
        __syncwarp();
    }
    return cta_wait_mma(bar, phase, abort_flag);
}

__device__ __forceinline__ void publish(bool to_async_proxy) {
    if (to_async_proxy) fence_async_smem();
    tc_fence_before();
    __syncthreads();
}

// ---- forward -----------------------------------------------------------------------------------

// TA: the two A operands of a branch (the 16-bit copy of its input stream, its hidden activation) live in tensor
// memory and never touch shared memory; the operand tiles only stage the rows as they arrive.
template <typename T, int ACT, bool BIAS, bool TA, int HALF, int HID>
__global__ void __launch_bounds__(kTcThreads, 2)
rev_fwd_tc_kernel(const RevShape shape, const RevParams p, const __grid_constant__ RevWeightMaps maps, const int use_tma,
                  const T *__restrict__ x, long long x_stride, T *__restrict__ y, long long y_stride, long long n_rows) {
    constexpr bool kRolled = HALF == 0, kLines = HALF > 0 && HID == 0;
    const RevShape s = known_widths<HALF, HID>(shape);
    extern __shared__ __align__(1024) unsigned char smem_raw[];
    unsigned char *smem = smem_raw;
    if (misplaced(smem)) return;
    __shared__ uint32_t tmem_holder;
    __shared__ __align__(8) unsigned long long mbar;
    __shared__ int abort_flag;
    const RevTcPlan P = rev_tc_plan(false);
    constexpr int bf16 = std::is_same<T, __half>::value ? 0 : 1;
    unsigned char *u_tile = smem, *h_tile = smem + kTileBytes;

    __shared__ __align__(8) unsigned long long ring_bars[2];
    if (threadIdx.x == 0) {
        abort_flag = 0;
        asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_addr(&ring_bars[0])), "r"(1u) : "memory");
        asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_addr(&ring_bars[1])), "r"(1u) : "memory");
    }
    const long long n_tiles = (n_rows + kTileRows - 1) / kTileRows;
    if (!use_tma && static_cast<long long>(blockIdx.x) < n_tiles) prefetch_weights<T>(smem, P, shape, p, 0, 0);
    const uint32_t tmem = cta_setup(&tmem_holder, &mbar, P.tmem_cols);  // publishes the barrier inits
    if (use_tma && static_cast<long long>(blockIdx.x) < n_tiles) {
        prefetch_weights_tma<T, BIAS>(smem, P, s, p, maps, ring_bars, 0, 0);  // awaited behind the first rows
    }
    // With the A operands in tensor memory and the weights by TMA nothing that an MMA reads is written by a thread, and the fence
    // between the two proxies, which waits for the row loads and stores in flight, is left out (2^19 rows, eight blocks: 0.250 -> 0.229 ms)
    const bool needs_fence = !TA || !use_tma;
    const uint32_t bar = smem_addr(&mbar);
    const Seat seat;
    const uint32_t taddr = tmem + seat.lane_base;
    uint32_t phase = 0;
    int step = 0;  // running (tile, block) counter: ring stage = step & 1
    const uint32_t idesc_hid = instr_desc(128, s.hid, bf16, 0, 0), idesc_half = instr_desc(128, s.half, bf16, 0, 0);

    for (long long tile = blockIdx.x; tile < n_tiles && !abort_flag; tile += gridDim.x) {
        const long long row0 = tile * kTileRows;
        const bool live = row0 + seat.row < n_rows;
        T *y_row = y + (live ? row0 + seat.row : 0) * y_stride;
        // x1 -> scratch tile, x2 -> the first branch's operand tile; then both into the fp32 stream in TMEM
        async_tile_load<T>(h_tile, x, x_stride, row0, n_rows, s.half, s.half);
        async_tile_load<T>(u_tile, x + s.half, x_stride, row0, n_rows, s.half, s.half);
        async_tile_wait();  // also the weights queued for this step
        if (use_tma && step == 0) ring_wait(ring_bars, 0, &abort_flag);
        __syncthreads();
        tile_row_to_tmem<T>(h_tile, seat, s.half, taddr + kS1);
        tile_row_to_tmem<T>(u_tile, seat, s.half, taddr + kS2);
        if constexpr (TA) {  // x2 as the first branch's A operand
            const int count = s.half / (8 * kGroups), first = seat.group * count;
            for (int u = 0; u < count; ++u)
                tmem_st4(taddr + kFwdAU + 4 * (first + u), *reinterpret_cast<const uint4 *>(chunk_ptr(u_tile, seat.row, first + u)));
        }
        tmem_st_wait();
        publish(needs_fence);

        for (int k = 0; k < s.blocks && !abort_flag; ++k, ++step) {
            const int stage = step & 1;
            // the other stage was last read by the previous block, whose GEMMs have all completed
            const bool more = k + 1 < s.blocks || tile + gridDim.x < n_tiles;
            if (more) {
                if (use_tma) prefetch_weights_tma<T, BIAS>(smem, P, s, p, maps, ring_bars, (k + 1) % s.blocks, stage ^ 1);
                else prefetch_weights<T>(smem, P, shape, p, (k + 1) % s.blocks, stage ^ 1);
            }
            const unsigned char *w = smem + P.ring + stage * kStageBytes;
            const float *bias = reinterpret_cast<const float *>(smem + P.bias) + stage * 4 * kMaxDim;
#pragma unroll 1
            for (int branch = 0; branch < 2; ++branch) {
                // branch 0: x1 += F(x2) (U holds x2), branch 1: x2 += G(x1) (U holds x1)
                const uint32_t w1 = smem_addr(w + (2 * branch) * kWTileBytes), w2 = smem_addr(w + (2 * branch + 1) * kWTileBytes);
                const uint32_t out_col = branch == 0 ? kS1 : kS2;
                bool leader = false;
                if (threadIdx.x < 32) {
                    leader = elect_one();
                    tc_fence_after();
                    if constexpr (TA) issue_gemm_ta<kLines>(leader, tmem + kFwdHid, tmem + kFwdAU, w1, 32, s.half / 16, idesc_hid, false);
                    else issue_gemm<kLines>(leader, tmem + kFwdHid, smem_addr(u_tile), 32, w1, 32, s.half / 16, idesc_hid, false);
                }
                commit_and_wait(leader, bar, phase, &abort_flag);
                {
                    const int n = s.hid / kGroups, first = seat.group * (n / 8);
                    const uint32_t row_addr = smem_addr(h_tile) + seat.row * 128, row_swizzle = (seat.row & 7) << 4;
                    const float *layer_bias = bias + (2 * branch) * kMaxDim;
                    for_each_piece<kRolled>(taddr + kFwdHid + seat.group * n, n, [&](int u, const uint32_t(&piece)[8]) {
                        const uint4 packed = finish8<T, ACT, BIAS>(piece, layer_bias + 8 * (first + u));
                        if constexpr (TA) tmem_st4(taddr + kFwdAH + 4 * (first + u), packed);
                        else st_shared_16(row_addr + (((first + u) << 4) ^ row_swizzle), packed);
                    });
                    if constexpr (TA) tmem_st_wait();
                }
                publish(needs_fence);
                if (threadIdx.x < 32) {
                    leader = elect_one();
                    tc_fence_after();
                    if constexpr (TA) issue_gemm_ta<kLines>(leader, tmem + out_col, tmem + kFwdAH, w2, 32, s.hid / 16, idesc_half, true);
                    else issue_gemm<kLines>(leader, tmem + out_col, smem_addr(h_tile), 32, w2, 32, s.hid / 16, idesc_half, true);
                }
                commit_and_wait(leader, bar, phase, &abort_flag);
                // the updated stream: rounded copy for the next branch, and the output after the last block
                const bool last = k == s.blocks - 1;
                if constexpr (TA)
                    stream_epilogue_ta<T, BIAS, kRolled>(taddr + out_col, seat, s.half, bias + (2 * branch + 1) * kMaxDim, taddr + kFwdAU,
                                                last ? y_row + branch * s.half : nullptr, live);
                else
                    stream_epilogue<T, BIAS, kRolled>(taddr + out_col, seat, s.half, bias + (2 * branch + 1) * kMaxDim, u_tile,
                                             last ? y_row + branch * s.half : nullptr, live);
                if (branch == 1) {  // next block's weights have landed
                    if (!use_tma) async_tile_wait();
                    else if (more) ring_wait(ring_bars, step + 1, &abort_flag);
                }
                publish(needs_fence);
            }
        }
    }
    if (abort_flag) {
        g_tc_status = 1;
        if (use_tma && threadIdx.x == 64) drain_copies(ring_bars, 2);
    }
    cta_teardown(tmem, P.tmem_cols);
}

// ---- backward ----------------------------------------------------------------------------------

// An accumulator matrix is stored [row / 16][column / 4][row % 16][column % 4]: what one flush warp holds of it is contiguous.
constexpr int kWgradIssuer = 2;  // the flush warp that issues the weight gradients: on another scheduler than the chain's issuer

// The backward kernel runs 256 "main" threads (the chain: issue, wait, epilogue) and 128 "flush" threads
// that carry the weight gradients of a pass out of TMEM while the main threads are already in the next pass.
constexpr int kRevFlushThreads = 128;

// CTA barrier of the main threads only
__device__ __forceinline__ void main_sync() { asm volatile("bar.sync 1, 256;" ::: "memory"); }

__device__ __forceinline__ void main_publish() {
    fence_async_smem();
    tc_fence_before();
    main_sync();
}

// Bounded wait that also gives up when somebody else has: false = do not go on.
__device__ __forceinline__ bool rev_wait(uint32_t bar, uint32_t parity, int *abort_flag) {
    for (int poll = 0; poll < kWaitPolls; ++poll) {
        uint32_t done;
        asm volatile(
            "{\n\t.reg .pred p;\n\tmbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\tselp.u32 %0, 1, 0, p;\n\t}\n"
            : "=r"(done)
            : "r"(bar), "r"(parity)
            : "memory");
        if (done) return true;
        if ((poll & 63) == 63 && *reinterpret_cast<volatile int *>(abort_flag)) return false;
    }
    *reinterpret_cast<volatile int *>(abort_flag) = 1;
    return false;
}

// The MMAs committed to `mbar` are done.  Every main warp polls: with one polling and the others parked at a barrier behind it
// 0.805 against 0.757 ms (2^19 rows, eight blocks).
__device__ __forceinline__ void main_wait_mma(uint32_t mbar, uint32_t &phase, int *abort_flag) {
    rev_wait(mbar, phase, abort_flag);
    __syncwarp();
    phase ^= 1;
    tc_fence_after();
}

// One flush warp's share of both accumulators: TMEM lanes 32 q .. 32 q + 15 hold rows 16 q .. of the first matrix, the other sixteen
// those of the second; the matrices have n1 and n2 rows, n2 and n1 columns, and only those leave (2^19 rows, four blocks of 16 -> 16 ->
// 16, backward: whole 64 x 64 matrices 371 us, this 355; 32 -> 32 -> 32 405, 393).  The accumulators are free once they are in
// registers.  `first`: nothing has been written to dst yet.
__device__ __forceinline__ void flush_dw_pair(uint32_t tmem, int q, uint32_t stage, float *dst, int n1, int n2, uint32_t flushed, bool first) {
    const int lane = threadIdx.x & 31;
    const uint32_t taddr = tmem + (static_cast<uint32_t>(32 * q) << 16) + kDW1;
    uint32_t lo[32], hi[32];
    tmem_ld32(taddr, lo);
    tmem_ld32(taddr + 32, hi);
    tmem_ld_wait();
    tc_fence_before();
    if (lane == 0) asm volatile("cp.async.bulk.wait_group.read 0;" ::: "memory");  // the reductions before have been read
    __syncwarp();
    if (lane == 0) asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(flushed) : "memory");
    const uint32_t at = stage + (lane >> 4) * 4096 + (lane & 15) * 16;
#pragma unroll
    for (int h = 0; h < 8; ++h) st_shared_16(at + h * 256, make_uint4(lo[4 * h], lo[4 * h + 1], lo[4 * h + 2], lo[4 * h + 3]));
#pragma unroll
    for (int h = 0; h < 8; ++h) st_shared_16(at + 2048 + h * 256, make_uint4(hi[4 * h], hi[4 * h + 1], hi[4 * h + 2], hi[4 * h + 3]));
    fence_async_smem();
    __syncwarp();
    if (lane == 0) {
        // Bulk copies and reductions in flight together arrive in no order.  The next ones to the same addresses are two passes or more
        // away (the other branch lies between), so these are sent once all but the last pass's have been performed.
        asm volatile("cp.async.bulk.wait_group 1;" ::: "memory");
        // The copies (0.5 MB per CTA) are revisited once per row tile while a gigabyte of rows streams through L2: ask it to keep them
        unsigned long long keep;
        asm volatile("createpolicy.fractional.L2::evict_last.b64 %0, 1.0;" : "=l"(keep));
#pragma unroll
        for (int m = 0; m < 2; ++m) {
            float *at_dst = dst + m * kMatFloats + q * 1024;
            if (16 * q >= (m == 0 ? n1 : n2)) continue;
            const uint32_t bytes = (m == 0 ? n2 : n1) * 64;  // 16 rows of the columns there are, quads of columns one after the other
            if (first)
                asm volatile("cp.async.bulk.global.shared::cta.bulk_group.L2::cache_hint [%0], [%1], %2, %3;" ::"l"(at_dst), "r"(stage + m * 4096), "r"(bytes),
                             "l"(keep)
                             : "memory");
            else
                asm volatile("cp.reduce.async.bulk.global.shared::cta.bulk_group.L2::cache_hint.add.f32 [%0], [%1], %2, %3;" ::"l"(at_dst),
                             "r"(stage + m * 4096), "r"(bytes), "l"(keep)
                             : "memory");
        }
        asm volatile("cp.async.bulk.commit_group;" ::: "memory");
    }
}

// Column sums of a 128 x 64 operand tile by the 128 flush threads, added to dst: a thread sums eight rows of one 16-byte chunk,
// the four threads of a warp with the same chunk meet in two shuffles.
template <typename T>
__device__ __forceinline__ void add_tile_column_sums(uint32_t tile, int width, float *dst) {
    const int t = threadIdx.x & 127, chunk = t & 7, row0 = (t >> 3) * 8;
    float v[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
#pragma unroll
    for (int r = 0; r < 8; ++r) {
        const uint4 q = ld_shared_16(tile + (row0 + r) * 128 + ((chunk ^ r) << 4));
        const uint32_t w[4] = {q.x, q.y, q.z, q.w};
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            const float2 f = unpack_pair<T>(w[k]);
            v[2 * k] += f.x;
            v[2 * k + 1] += f.y;
        }
    }
#pragma unroll
    for (int k = 0; k < 8; ++k) {
        v[k] += __shfl_xor_sync(0xffffffffu, v[k], 8);
        v[k] += __shfl_xor_sync(0xffffffffu, v[k], 16);
    }
    if ((t & 31) < 8 && 8 * chunk < width) {
#pragma unroll
        for (int k = 0; k < 8; k += 4)
            asm volatile("red.global.add.v4.f32 [%0], {%1, %2, %3, %4};" ::"l"(dst + 8 * chunk + k), "f"(v[k]), "f"(v[k + 1]), "f"(v[k + 2]), "f"(v[k + 3])
                         : "memory");
    }
}

template <typename T, int ACT, bool BIAS, int HALF, int HID>
__global__ void __launch_bounds__(kTcThreads + kRevFlushThreads, 1)
rev_bwd_tc_kernel(const RevShape shape, const RevParams p, const __grid_constant__ RevWeightMaps maps,
                  const __grid_constant__ RevRowMaps row_maps, const int use_tma,
                  const T *__restrict__ y, long long y_stride,
                  const T *__restrict__ go, long long go_stride, T *__restrict__ gx, long long gx_stride,
                  T *__restrict__ x_rec, long long xr_stride, float *__restrict__ workspace, long long n_rows) {
    constexpr bool kRolled = HALF == 0, kLines = HALF > 0 && HID == 0;
    const RevShape s = known_widths<HALF, HID>(shape);
    extern __shared__ __align__(1024) unsigned char smem_raw[];
    unsigned char *smem = smem_raw;
    if (misplaced(smem)) return;
    __shared__ uint32_t tmem_holder;
    __shared__ __align__(8) unsigned long long mbar;
    __shared__ int abort_flag;
    const RevTcPlan P = rev_tc_plan(true);
    constexpr int bf16 = std::is_same<T, __half>::value ? 0 : 1;
    // U (the branch's input, 16-bit) and DY (the gradient of its output) alternate between two tiles each: the
    // epilogue of a pass writes the next pass's copies while this pass's weight-gradient MMAs still read theirs
    unsigned char *u_tiles = smem, *h_tile = smem + 2 * kTileBytes, *dy_tiles = smem + 3 * kTileBytes, *dz_tile = smem + 5 * kTileBytes;
    unsigned char *y2_tile = smem + 6 * kTileBytes, *go1_tile = smem + 7 * kTileBytes;  // the next row tile's, on their way to tensor memory
    const bool is_flush = threadIdx.x >= kTcThreads;

    __shared__ __align__(8) unsigned long long ring_bars[2];
    // wgrad_bar: the weight-gradient MMAs of a pass are done (one commit per pass); flushed_bar: the flush warps
    // have read them out (one arrival per flush warp), so the next pass may overwrite the accumulators
    // operands_bar: h and dz of a pass are in place and the chain's MMAs on them issued (one arrival)
    // BIAS - summed_bar: the flush warps have summed the columns of dz and dy
    // rows_bar: the four TMA boxes of a row tile have landed
    // the main threads' copy of the abort flag: written before a barrier of theirs and read behind it, so that all of them leave together
    __shared__ int stop_flag;
    __shared__ __align__(8) unsigned long long wgrad_bar, flushed_bar, operands_bar, summed_bar, rows_bar;
    if (threadIdx.x == 0) {
        abort_flag = stop_flag = 0;
        asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_addr(&ring_bars[0])), "r"(1u) : "memory");
        asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_addr(&ring_bars[1])), "r"(1u) : "memory");
        asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_addr(&wgrad_bar)), "r"(1u) : "memory");
        asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_addr(&operands_bar)), "r"(1u) : "memory");
        asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_addr(&rows_bar)), "r"(1u) : "memory");
        asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_addr(&summed_bar)), "r"(static_cast<uint32_t>(kRevFlushThreads / 32)) : "memory");
        asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_addr(&flushed_bar)), "r"(static_cast<uint32_t>(kRevFlushThreads / 32)) : "memory");
    }
    for (int e = threadIdx.x; e < P.tiles * kTileBytes / 16; e += blockDim.x) reinterpret_cast<uint4 *>(smem)[e] = make_uint4(0, 0, 0, 0);
    const long long n_tiles = (n_rows + kTileRows - 1) / kTileRows;
    if (!is_flush && !use_tma && static_cast<long long>(blockIdx.x) < n_tiles) prefetch_weights<T>(smem, P, shape, p, s.blocks - 1, 0);
    const uint32_t tmem = cta_setup(&tmem_holder, &mbar, P.tmem_cols);  // publishes the barrier inits
    float *cta_acc = workspace + static_cast<size_t>(blockIdx.x) * rev_cta_floats(s);
    const uint32_t wgrad_addr = smem_addr(&wgrad_bar), flushed_addr = smem_addr(&flushed_bar);
    const uint32_t operands_addr = smem_addr(&operands_bar), summed_addr = smem_addr(&summed_bar);

    if (is_flush) {
        // ================= weight gradients out of TMEM, one pass behind the main threads =================
        const int q = (threadIdx.x >> 5) & 3;
        const uint32_t stage = smem_addr(smem + P.stage) + q * 8192;
        const uint32_t id_dw2 = instr_desc(64, s.hid, bf16, 1, 1), id_dw1 = instr_desc(64, s.half, bf16, 1, 1);  // both operands MN-major, M = 64
        uint32_t n = 0;  // passes flushed so far
        bool alive = true;
        for (long long tile = blockIdx.x; alive && tile < n_tiles; tile += gridDim.x) {
            for (int k = s.blocks - 1; alive && k >= 0; --k) {
                float *block_acc = cta_acc + static_cast<size_t>(k) * 4 * kMatFloats;
                for (int pass = 0; pass < 2; ++pass, ++n) {
                    const uint32_t dy_cur = smem_addr(dy_tiles + (n & 1u) * kTileBytes);
                    if (BIAS || q == kWgradIssuer) {
                        alive = __all_sync(0xffffffffu, rev_wait(operands_addr, n & 1u, &abort_flag));
                        // the accumulators hold the previous pass's sums until all four flush warps have read them
                        if (q == kWgradIssuer && alive && n > 0) alive = __all_sync(0xffffffffu, rev_wait(flushed_addr, (n - 1) & 1u, &abort_flag));
                        if (!alive) break;
                    }
                    if (q == kWgradIssuer) {
                        const bool leader = elect_one();
                        tc_fence_after();
                        const uint32_t u_cur = smem_addr(u_tiles + (n & 1u) * kTileBytes);
                        issue_gemm<kLines>(leader, tmem + kDW2, dy_cur, 2048, smem_addr(h_tile), 2048, kTileRows / 16, id_dw2, false);
                        issue_gemm<kLines>(leader, tmem + kDW1, smem_addr(dz_tile), 2048, u_cur, 2048, kTileRows / 16, id_dw1, false);
                        if (leader) mma_commit(wgrad_addr);
                        __syncwarp();
                    }
                    if constexpr (BIAS) {
                        float *sums = cta_acc + static_cast<size_t>(s.blocks) * 4 * kMatFloats + (static_cast<size_t>(k) * 4 + (pass == 0 ? 2 : 0)) * kMaxDim;
                        add_tile_column_sums<T>(smem_addr(dz_tile), s.hid, sums);
                        add_tile_column_sums<T>(dy_cur, s.half, sums + kMaxDim);
                        __syncwarp();
                        if ((threadIdx.x & 31) == 0) asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(summed_addr) : "memory");
                    }
                    alive = __all_sync(0xffffffffu, rev_wait(wgrad_addr, n & 1u, &abort_flag));
                    if (!alive) break;
                    tc_fence_after();
                    const int m1 = pass == 0 ? 2 : 0;
                    flush_dw_pair(tmem, q, stage, block_acc + m1 * kMatFloats, s.hid, s.half, flushed_addr, tile == blockIdx.x);
                }
            }
        }
        if ((threadIdx.x & 31) == 0) asm volatile("cp.async.bulk.wait_group 0;" ::: "memory");
    } else {
        // ================= the chain =================
        if (use_tma && static_cast<long long>(blockIdx.x) < n_tiles) {
            prefetch_weights_tma<T, BIAS>(smem, P, s, p, maps, ring_bars, s.blocks - 1, 0);
            ring_wait(ring_bars, 0, &abort_flag);
        }
        const uint32_t bar = smem_addr(&mbar);
        const Seat seat;
        const uint32_t taddr = tmem + seat.lane_base;
        uint32_t phase = 0;
        int step = 0;
        uint32_t n = 0;  // passes started so far; pass n reads U / DY copy n & 1 and writes copy (n + 1) & 1
        // instruction descriptors: forward-type, dgrad (B MN-major), reconstruction (A negated)
        const uint32_t id_z = instr_desc(128, s.hid, bf16, 0, 0);
        const uint32_t id_dh = instr_desc(128, s.hid, bf16, 0, 1);
        const uint32_t id_undo = instr_desc(128, s.half, bf16, 0, 0) | (1u << 13);
        const uint32_t id_din = instr_desc(128, s.half, bf16, 0, 1);
        volatile int *abort_now = &abort_flag;

        // A row tile: y1 -> U (input of the last G), go2 -> DY (gradient of G's output), the other halves -> scratch.  Fetched
        // during the last pass of the tile before, whose epilogue leaves its U / DY copies free.
        const uint32_t rows_addr = smem_addr(&rows_bar);
        auto fetch_rows = [&](long long row0, uint32_t copy) {
            unsigned char *u_in = u_tiles + copy * kTileBytes, *dy_in = dy_tiles + copy * kTileBytes;
            if (use_tma) {
                if (threadIdx.x == 64 && !*abort_now) {
                    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(rows_addr), "r"(4u * kTileBytes) : "memory");
                    const int at = static_cast<int>(row0);
                    tma_load_2d(u_in, &row_maps.y1, 0, at, rows_addr);
                    tma_load_2d(dy_in, &row_maps.go2, 0, at, rows_addr);
                    tma_load_2d(y2_tile, &row_maps.y2, 0, at, rows_addr);
                    tma_load_2d(go1_tile, &row_maps.go1, 0, at, rows_addr);
                }
            } else {
                async_tile_load<T>(u_in, y, y_stride, row0, n_rows, s.half, s.half);
                async_tile_load<T>(y2_tile, y + s.half, y_stride, row0, n_rows, s.half, s.half);
                async_tile_load<T>(go1_tile, go, go_stride, row0, n_rows, s.half, s.half);
                async_tile_load<T>(dy_in, go + s.half, go_stride, row0, n_rows, s.half, s.half);
            }
        };
        uint32_t rows_phase = 0;
        if (static_cast<long long>(blockIdx.x) < n_tiles) fetch_rows(static_cast<long long>(blockIdx.x) * kTileRows, 0);

        volatile int *stop = &stop_flag;
        for (long long tile = blockIdx.x; tile < n_tiles && !*stop; tile += gridDim.x) {
            const long long row0 = tile * kTileRows;
            const bool live = row0 + seat.row < n_rows;
            unsigned char *u_in = u_tiles + (n & 1u) * kTileBytes, *dy_in = dy_tiles + (n & 1u) * kTileBytes;
            if (use_tma) {
                rev_wait(rows_addr, rows_phase, &abort_flag);
                rows_phase ^= 1;
            } else {
                async_tile_wait();
                main_sync();
            }
            tile_row_to_tmem<T>(u_in, seat, s.half, taddr + kS1);
            tile_row_to_tmem<T>(y2_tile, seat, s.half, taddr + kS2);
            tile_row_to_tmem<T>(go1_tile, seat, s.half, taddr + kD1);
            tile_row_to_tmem<T>(dy_in, seat, s.half, taddr + kD2);
            {
                const int count = s.half / (8 * kGroups), first = seat.group * count;
                for (int u = 0; u < count; ++u) {
                    tmem_st4(taddr + kA0 + 4 * (first + u), *reinterpret_cast<const uint4 *>(chunk_ptr(u_in, seat.row, first + u)));
                    tmem_st4(taddr + kA1 + 4 * (first + u), *reinterpret_cast<const uint4 *>(chunk_ptr(dy_in, seat.row, first + u)));
                }
            }
            tmem_st_wait();
            main_publish();

            for (int k = s.blocks - 1; k >= 0 && !*stop; --k, ++step) {
                const int stage = step & 1;
                const bool more = k > 0 || tile + gridDim.x < n_tiles;
                if (more) {
                    if (use_tma) prefetch_weights_tma<T, BIAS>(smem, P, s, p, maps, ring_bars, k > 0 ? k - 1 : s.blocks - 1, stage ^ 1, abort_now);
                    else prefetch_weights<T>(smem, P, shape, p, k > 0 ? k - 1 : s.blocks - 1, stage ^ 1);
                }
                const unsigned char *w = smem + P.ring + stage * kStageBytes;
                const float *block_bias = reinterpret_cast<const float *>(smem + P.bias) + stage * 4 * kMaxDim;
#pragma unroll 1
                for (int pass = 0; pass < 2; ++pass, ++n) {
                    // pass 0 undoes y2 = x2 + G(y1): input stream S1, output stream S2, gradient flows D2 -> D1
                    // pass 1 undoes y1 = x1 + F(x2): input stream S2, output stream S1, gradient flows D1 -> D2
                    const int m1 = pass == 0 ? 2 : 0, m2 = m1 + 1;
                    const uint32_t w1 = smem_addr(w + m1 * kWTileBytes), w2 = smem_addr(w + m2 * kWTileBytes);
                    const uint32_t out_col = pass == 0 ? kS2 : kS1, in_d_col = pass == 0 ? kD1 : kD2;
                    const uint32_t u_cur = smem_addr(u_tiles + (n & 1u) * kTileBytes), dy_cur = smem_addr(dy_tiles + (n & 1u) * kTileBytes);
                    unsigned char *u_next = u_tiles + ((n + 1) & 1u) * kTileBytes, *dy_next = dy_tiles + ((n + 1) & 1u) * kTileBytes;
                    // step A: z = U . W1^T and dh = DY . W2 together
                    if (threadIdx.x < 32) {
                        const bool leader = elect_one();
                        tc_fence_after();
                        issue_gemm_ta<kLines>(leader, tmem + kZ, tmem + kA0, w1, 32, s.half / 16, id_z, false);
                        issue_gemm_ta<kLines>(leader, tmem + kDH, tmem + kA1, w2, 2048, s.half / 16, id_dh, false);
                        if (leader) mma_commit(bar);
                        __syncwarp();
                    }
                    if constexpr (BIAS) {
                        // under those MMAs: the branch's second bias comes off the stream that step B takes the rest from; and the
                        // flush warps must have summed the previous pass's dz before it is overwritten below
                        const int nh = s.half / kGroups, first_h = seat.group * (nh / 8);
                        const float *bias2 = block_bias + m2 * kMaxDim;
                        for_each_piece<kRolled>(taddr + out_col + seat.group * nh, nh, [&](int u, const uint32_t(&piece)[8]) {
                            uint32_t v[8];
#pragma unroll
                            for (int e = 0; e < 8; ++e) v[e] = __float_as_uint(__uint_as_float(piece[e]) - bias2[8 * (first_h + u) + e]);
                            tmem_st8(taddr + out_col + seat.group * nh + 8 * u, v);
                        });
                        tmem_st_wait();
                        if (n > 0) rev_wait(summed_addr, (n - 1) & 1u, &abort_flag);
                    }
                    // the previous pass's weight-gradient MMAs read the h and dz tiles the epilogue below overwrites
                    if (n > 0) rev_wait(wgrad_addr, (n - 1) & 1u, &abort_flag);
                    main_wait_mma(bar, phase, &abort_flag);
                    const bool last = k == 0 && pass == 1;
                    if (last && tile + gridDim.x < n_tiles) fetch_rows(row0 + static_cast<long long>(gridDim.x) * kTileRows, (n + 1) & 1u);
                    {
                        // h = act(z) first (also the ReLU mask), then dz = dh where h > 0
                        const int nn = s.hid / kGroups, first = seat.group * (nn / 8);
                        const uint32_t row_off = seat.row * 128, row_swizzle = (seat.row & 7) << 4;
                        const uint32_t h_row = smem_addr(h_tile) + row_off, dz_row = smem_addr(dz_tile) + row_off;
                        const float *bias1 = block_bias + m1 * kMaxDim;
                        auto store_h = [&](int u, uint4 q) {
                            st_shared_16(h_row + (((first + u) << 4) ^ row_swizzle), q);
                            tmem_st4(taddr + kA0 + 4 * (first + u), q);
                        };
                        auto store_dz = [&](int u, uint4 g) {
                            st_shared_16(dz_row + (((first + u) << 4) ^ row_swizzle), g);
                            tmem_st4(taddr + kA1 + 4 * (first + u), g);
                        };
                        if constexpr (HALF == 64 && HID == 64 && (ACT == TH_ACT_RELU || ACT == TH_ACT_NONE)) {
                            // both accumulators in flight together, the mask from registers
                            uint32_t zz[32], dh[32];
                            tmem_ld32(taddr + kZ + seat.group * 32, zz);
                            tmem_ld32(taddr + kDH + seat.group * 32, dh);
                            tmem_ld_wait();
#pragma unroll
                            for (int u = 0; u < 4; ++u) {
                                const uint4 h = finish8<T, ACT, BIAS>(zz + 8 * u, bias1 + 8 * (first + u));
                                store_h(u, h);
                                uint4 g = finish8<T, TH_ACT_NONE, false>(dh + 8 * u, nullptr);
                                if constexpr (ACT == TH_ACT_RELU) {
                                    g.x = keep_where_positive<T>(g.x, h.x);
                                    g.y = keep_where_positive<T>(g.y, h.y);
                                    g.z = keep_where_positive<T>(g.z, h.z);
                                    g.w = keep_where_positive<T>(g.w, h.w);
                                }
                                store_dz(u, g);
                            }
                        } else {
                            for_each_piece<kRolled>(taddr + kZ + seat.group * nn, nn, [&](int u, const uint32_t(&piece)[8]) {
                                store_h(u, finish8<T, ACT, BIAS>(piece, bias1 + 8 * (first + u)));
                            });
                            if constexpr (ACT == TH_ACT_SILU || ACT == TH_ACT_RELU2) {
                                // the derivative is taken at the pre-activation rounded to the storage type
#pragma unroll 1
                                for (int u = 0; u < nn / 8; ++u) {
                                    uint32_t dh[8], zz[8];
                                    tmem_ld8(taddr + kDH + seat.group * nn + 8 * u, dh);
                                    tmem_ld8(taddr + kZ + seat.group * nn + 8 * u, zz);
                                    tmem_ld_wait();
                                    float g[8];
#pragma unroll
                                    for (int e = 0; e < 8; ++e) {
                                        float z = __uint_as_float(zz[e]);
                                        if constexpr (BIAS) z += bias1[8 * (first + u) + e];
                                        z = to_float<T>(from_float<T>(z));
                                        g[e] = activate_grad(ACT, z, __uint_as_float(dh[e]));
                                    }
                                    store_dz(u, make_uint4(pack_pair<T>(g[0], g[1]), pack_pair<T>(g[2], g[3]), pack_pair<T>(g[4], g[5]), pack_pair<T>(g[6], g[7])));
                                }
                            } else {
                                for_each_piece<kRolled>(taddr + kDH + seat.group * nn, nn, [&](int u, const uint32_t(&piece)[8]) {
                                    uint4 g = finish8<T, TH_ACT_NONE, false>(piece, nullptr);
                                    if constexpr (ACT == TH_ACT_RELU) {
                                        const uint4 h = ld_shared_16(h_row + (((first + u) << 4) ^ row_swizzle));  // this thread's own store above
                                        g.x = keep_where_positive<T>(g.x, h.x);
                                        g.y = keep_where_positive<T>(g.y, h.y);
                                        g.z = keep_where_positive<T>(g.z, h.z);
                                        g.w = keep_where_positive<T>(g.w, h.w);
                                    }
                                    store_dz(u, g);
                                });
                            }
                        }
                        tmem_st_wait();
                    }
                    main_publish();
                    // step B: undo the branch and push the gradient through.  Then the flush warps may issue the two weight gradients:
                    // MMAs execute in the order of issue and an issuing thread is held while the queue is full, so sixteen more
                    // of them here would keep the chain waiting until most of them have run.
                    if (threadIdx.x < 32) {
                        const bool leader = elect_one();
                        tc_fence_after();
                        issue_gemm_ta<kLines>(leader, tmem + out_col, tmem + kA0, w2, 32, s.hid / 16, id_undo, true);
                        issue_gemm_ta<kLines>(leader, tmem + in_d_col, tmem + kA1, w1, 2048, s.hid / 16, id_din, true);
                        if (leader) mma_commit(bar);
                        if (leader) asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(operands_addr) : "memory");
                        __syncwarp();
                    }
                    main_wait_mma(bar, phase, &abort_flag);
                    // next pass: its input is the stream just reconstructed, its output gradient the one just updated
                    if (!last) {
                        if constexpr (HALF == 64) {
                            uint32_t su[32], sd[32];
                            tmem_ld32(taddr + out_col + seat.group * 32, su);
                            tmem_ld32(taddr + in_d_col + seat.group * 32, sd);
                            tmem_ld_wait();
                            const uint32_t row_off = seat.row * 128, row_swizzle = (seat.row & 7) << 4;
                            const uint32_t u_row = smem_addr(u_next) + row_off, dy_row = smem_addr(dy_next) + row_off;
#pragma unroll
                            for (int u = 0; u < 4; ++u) {
                                const int c = 4 * seat.group + u;
                                const uint4 a = finish8<T, TH_ACT_NONE, false>(su + 8 * u, nullptr), g = finish8<T, TH_ACT_NONE, false>(sd + 8 * u, nullptr);
                                st_shared_16(u_row + ((c << 4) ^ row_swizzle), a);
                                st_shared_16(dy_row + ((c << 4) ^ row_swizzle), g);
                                tmem_st4(taddr + kA0 + 4 * c, a);
                                tmem_st4(taddr + kA1 + 4 * c, g);
                            }
                            tmem_st_wait();
                        } else {
                            auto both = [&](uint32_t from, unsigned char *tile, uint32_t a_col) {
                                const int n8 = s.half / kGroups, first = seat.group * (n8 / 8);
                                const uint32_t row_addr = smem_addr(tile) + seat.row * 128, row_swizzle = (seat.row & 7) << 4;
                                for_each_piece<kRolled>(taddr + from + seat.group * n8, n8, [&](int u, const uint32_t(&piece)[8]) {
                                    const uint4 q = finish8<T, TH_ACT_NONE, false>(piece, nullptr);
                                    st_shared_16(row_addr + (((first + u) << 4) ^ row_swizzle), q);
                                    tmem_st4(taddr + a_col + 4 * (first + u), q);
                                });
                            };
                            both(out_col, u_next, kA0);
                            both(in_d_col, dy_next, kA1);
                            tmem_st_wait();
                        }
                    }
                    if (pass == 1) {  // next block's weights have landed
                        if (!use_tma) async_tile_wait();
                        else if (more) ring_wait(ring_bars, step + 1, &abort_flag);
                        if (threadIdx.x == 0) *stop = *abort_now;
                    }
                    main_publish();
                }
            }
            // the stream is now the reconstructed input, the gradient stream the input gradient
            if (!*stop) {
#pragma unroll 1
                for (int q = 0; q < 4; ++q) {
                    // q: 0 = dx1 (D1), 1 = dx2 (D2), 2 = x1 (S1), 3 = x2 (S2)
                    T *base = q < 2 ? gx : x_rec;
                    const long long stride = q < 2 ? gx_stride : xr_stride;
                    const uint32_t col = q == 0 ? kD1 : (q == 1 ? kD2 : (q == 2 ? kS1 : kS2));
                    if (base != nullptr)
                        stream_epilogue<T, false, kRolled>(taddr + col, seat, s.half, nullptr, nullptr,
                                                  base + (live ? row0 + seat.row : 0) * stride + (q & 1) * s.half, live);
                }
            }
        }
    }
    if (abort_flag) {
        g_tc_status = 1;
        if (use_tma && threadIdx.x == 64) {
            drain_copies(ring_bars, 2);
            drain_copies(&rows_bar, 1);
        }
    }
    cta_teardown(tmem, P.tmem_cols);
}

// Sum the accumulators ([CTA][block][matrix][row / 16][column / 4][row % 16][column % 4], then [block][4][64] bias sums) into the
// gradient tensors: a thread sums one quad of every 8th copy, the block's eight shares meet in shared memory in a fixed order.
constexpr int kReduceQuads = 32, kReduceShares = 8;
template <typename T>
__global__ void __launch_bounds__(kReduceQuads * kReduceShares)
rev_grad_reduce_tc_kernel(const RevShape s, const float *__restrict__ workspace, int copies, T *dw_f1, T *dw_f2, T *dw_g1,
                                          T *dw_g2, T *db_f1, T *db_f2, T *db_g1, T *db_g2) {
    const size_t per_cta = rev_cta_floats(s), mat_total = static_cast<size_t>(s.blocks) * 4 * kMatFloats, total = s.has_bias ? per_cta : mat_total;
    const int lane = threadIdx.x % kReduceQuads, share = threadIdx.x / kReduceQuads;
    const size_t e = (static_cast<size_t>(blockIdx.x) * kReduceQuads + lane) * 4;
    __shared__ float4 part[kReduceShares][kReduceQuads];
    float4 sum = make_float4(0.f, 0.f, 0.f, 0.f);
    T *dst = nullptr;
    if (e < mat_total) {
        const int k = static_cast<int>(e / (4 * kMatFloats)), m = static_cast<int>((e / kMatFloats) % 4);
        const int at = static_cast<int>(e % kMatFloats), row = at / 1024 * 16 + at / 4 % 16, col = at / 64 % 16 * 4;
        const int out_dim = (m & 1) ? s.half : s.hid, in_dim = (m & 1) ? s.hid : s.half;
        T *dw = m == 0 ? dw_f1 : (m == 1 ? dw_f2 : (m == 2 ? dw_g1 : dw_g2));
        if (dw && row < out_dim && col < in_dim) dst = dw + (static_cast<size_t>(k) * out_dim + row) * in_dim + col;
    } else if (e < total) {
        const int b = static_cast<int>(e - mat_total), k = b / 256, m = (b / 64) % 4, c = b % 64;
        const int width = (m & 1) ? s.half : s.hid;
        T *db = m == 0 ? db_f1 : (m == 1 ? db_f2 : (m == 2 ? db_g1 : db_g2));
        if (db && c < width) dst = db + static_cast<size_t>(k) * width + c;
    }
    if (dst) {
#pragma unroll 4
        for (int c = share; c < copies; c += kReduceShares) {
            const float4 v = __ldcs(reinterpret_cast<const float4 *>(workspace + c * per_cta + e));
            sum.x += v.x;
            sum.y += v.y;
            sum.z += v.z;
            sum.w += v.w;
        }
    }
    part[share][lane] = sum;
    __syncthreads();
    if (share == 0 && dst) {
#pragma unroll
        for (int i = 1; i < kReduceShares; ++i) {
            const float4 v = part[i][lane];
            sum.x += v.x;
            sum.y += v.y;
            sum.z += v.z;
            sum.w += v.w;
        }
        dst[0] = from_float<T>(sum.x);
        dst[1] = from_float<T>(sum.y);
        dst[2] = from_float<T>(sum.z);
        dst[3] = from_float<T>(sum.w);
    }
}

// ---- host side ---------------------------------------------------------------------------------

bool rev_tc_disabled() {
    static const bool off = [] {
        const char *v = getenv("TH_MLP_LEGACY");
        return v && v[0] == '1';
    }();
    return off;
}

bool rows16_ok(const void *p, int64_t stride) { return p && stride % 8 == 0 && aligned_to(p, 16); }

// Dynamic shared memory to request so that no more than `ctas` CTAs share an SM.
int smem_request(const RevTcPlan &P, int ctas) {
    const int need = P.total;
    const int floor_bytes = kSmemBudget / (ctas + 1) + 1;
    return need > floor_bytes ? need : floor_bytes;
}

// Tensor maps of the four stacked weight arrays (box = 64 columns x one block's rows); 0 when one of
// them cannot be described (then the kernels stage the weights with cp.async) or TH_MLP_NO_TMA=1.
int make_rev_maps(RevWeightMaps &maps, const RevShape &s, const RevParams &p) {
    memset(&maps, 0, sizeof(maps));
    static const bool off = [] {
        const char *v = getenv("TH_MLP_NO_TMA");
        return v && v[0] == '1';
    }();
    if (off) return 0;
    const void *w[4] = {p.w_f1, p.w_f2, p.w_g1, p.w_g2};
    for (int m = 0; m < 4; ++m) {
        const int rows = (m & 1) ? s.half : s.hid, cols = (m & 1) ? s.hid : s.half;
        if (!make_map(&maps.m[m], w[m], static_cast<long long>(s.blocks) * rows, cols, rows)) return 0;
    }
    return 1;
}

// TH_MLP_NO_TMEM_A=1 keeps the A operands of the forward GEMMs in shared memory (for A/B runs).
bool rev_tmem_a_enabled() {
    static const bool on = [] {
        const char *v = getenv("TH_MLP_NO_TMEM_A");
        return !(v && v[0] == '1');
    }();
    return on;
}

template <typename T, int ACT, bool BIAS, bool TA>
int launch_rev_fwd_ta(const RevShape &s, const RevParams &p, const void *x, int64_t x_stride, void *y, int64_t y_stride,
                      int64_t rows, cudaStream_t stream) {
    const RevTcPlan P = rev_tc_plan(false);
    const int ctas = 2;  // 256 of the 512 TMEM columns each
    const int smem = smem_request(P, ctas);
    auto kernel = rev_fwd_tc_kernel<T, ACT, BIAS, TA, 0, 0>;
    if constexpr (TA) {
        if (s.half == 64 && s.hid == 64) kernel = rev_fwd_tc_kernel<T, ACT, BIAS, TA, 64, 64>;
        else if (s.half == 64) kernel = rev_fwd_tc_kernel<T, ACT, BIAS, TA, 64, 0>;
        else if (s.half == 48) kernel = rev_fwd_tc_kernel<T, ACT, BIAS, TA, 48, 0>;
        else if (s.half == 32) kernel = rev_fwd_tc_kernel<T, ACT, BIAS, TA, 32, 0>;
        else kernel = rev_fwd_tc_kernel<T, ACT, BIAS, TA, 16, 0>;
    }
    if (int rc = cuda_status(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, smem),
                             "cudaFuncSetAttribute(rev_fwd_tc_kernel)")) return rc;
    const long long tiles = (rows + kTileRows - 1) / kTileRows;
    const long long cap = static_cast<long long>(sm_count()) * ctas;
    RevWeightMaps maps;
    const int use_tma = make_rev_maps(maps, s, p);
    kernel<<<static_cast<unsigned>(tiles < cap ? tiles : cap), kTcThreads, smem, stream>>>(
        s, p, maps, use_tma, static_cast<const T *>(x), x_stride, static_cast<T *>(y), y_stride, rows);
    return launch_status("rev_fwd_tc_kernel launch");
}

template <typename T, int ACT, bool BIAS>
int launch_rev_fwd_t(const RevShape &s, const RevParams &p, const void *x, int64_t x_stride, void *y, int64_t y_stride,
                     int64_t rows, cudaStream_t stream) {
    return rev_tmem_a_enabled() ? launch_rev_fwd_ta<T, ACT, BIAS, true>(s, p, x, x_stride, y, y_stride, rows, stream)
                                : launch_rev_fwd_ta<T, ACT, BIAS, false>(s, p, x, x_stride, y, y_stride, rows, stream);
}

template <typename T, bool BIAS>
int launch_rev_fwd_act(const RevShape &s, const RevParams &p, const void *x, int64_t x_stride, void *y, int64_t y_stride,
                       int64_t rows, cudaStream_t stream) {
    switch (s.act) {
        case TH_ACT_RELU: return launch_rev_fwd_t<T, TH_ACT_RELU, BIAS>(s, p, x, x_stride, y, y_stride, rows, stream);
        case TH_ACT_SILU: return launch_rev_fwd_t<T, TH_ACT_SILU, BIAS>(s, p, x, x_stride, y, y_stride, rows, stream);
        case TH_ACT_RELU2: return launch_rev_fwd_t<T, TH_ACT_RELU2, BIAS>(s, p, x, x_stride, y, y_stride, rows, stream);
        default: return launch_rev_fwd_t<T, TH_ACT_NONE, BIAS>(s, p, x, x_stride, y, y_stride, rows, stream);
    }
}

template <typename T>
int launch_rev_fwd(const RevShape &s, const RevParams &p, const void *x, int64_t x_stride, void *y, int64_t y_stride,
                   int64_t rows, cudaStream_t stream) {
    return s.has_bias ? launch_rev_fwd_act<T, true>(s, p, x, x_stride, y, y_stride, rows, stream)
                      : launch_rev_fwd_act<T, false>(s, p, x, x_stride, y, y_stride, rows, stream);
}

template <typename T, int ACT, bool BIAS>
int launch_rev_bwd_t(const RevShape &s, const RevParams &p, const void *y, int64_t y_stride, const void *go,
                     int64_t go_stride, void *gx, int64_t gx_stride, void *x_rec, int64_t xr_stride, void *const dw[4],
                     void *const db[4], float *workspace, int n_ctas, int64_t rows, cudaStream_t stream) {
    const RevTcPlan P = rev_tc_plan(true);
    const int smem = smem_request(P, 1);  // all 512 TMEM columns: one CTA per SM
    auto kernel = s.half == 64 && s.hid == 64 ? rev_bwd_tc_kernel<T, ACT, BIAS, 64, 64> : rev_bwd_tc_kernel<T, ACT, BIAS, 0, 0>;
    if constexpr (!BIAS && (ACT == TH_ACT_RELU || ACT == TH_ACT_NONE)) {
        if (s.half == 64 && s.hid != 64) kernel = rev_bwd_tc_kernel<T, ACT, BIAS, 64, 0>;
        else if (s.half == 48) kernel = rev_bwd_tc_kernel<T, ACT, BIAS, 48, 0>;
        else if (s.half == 32) kernel = rev_bwd_tc_kernel<T, ACT, BIAS, 32, 0>;
        else if (s.half == 16) kernel = rev_bwd_tc_kernel<T, ACT, BIAS, 16, 0>;
    }
    if (int rc = cuda_status(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, smem),
                             "cudaFuncSetAttribute(rev_bwd_tc_kernel)")) return rc;
    RevWeightMaps maps;
    RevRowMaps row_maps;
    memset(&row_maps, 0, sizeof(row_maps));
    const T *y_rows = static_cast<const T *>(y), *go_rows = static_cast<const T *>(go);
    const int use_tma = rows < (1ll << 31) - kTileRows && make_rev_maps(maps, s, p) && make_map(&row_maps.y1, y_rows, rows, s.half, kTileRows, y_stride) &&
                        make_map(&row_maps.y2, y_rows + s.half, rows, s.half, kTileRows, y_stride) &&
                        make_map(&row_maps.go1, go_rows, rows, s.half, kTileRows, go_stride) &&
                        make_map(&row_maps.go2, go_rows + s.half, rows, s.half, kTileRows, go_stride);
    // the matrices are written by a CTA's first tile (it has one: n_ctas is at most the number of tiles), the bias sums only added to
    if constexpr (BIAS) {
        const size_t pitch = sizeof(float) * rev_cta_floats(s), sums = sizeof(float) * s.blocks * 4 * kMaxDim;
        if (int rc = cuda_status(cudaMemset2DAsync(reinterpret_cast<unsigned char *>(workspace) + pitch - sums, pitch, 0, sums, n_ctas, stream),
                                 "cudaMemset2DAsync(workspace)")) return rc;
    }
    kernel<<<n_ctas, kTcThreads + kRevFlushThreads, smem, stream>>>(s, p, maps, row_maps, use_tma, static_cast<const T *>(y), y_stride,
                                                static_cast<const T *>(go), go_stride, static_cast<T *>(gx), gx_stride,
                                                static_cast<T *>(x_rec), xr_stride, workspace, rows);
    if (int rc = launch_status("rev_bwd_tc_kernel launch")) return rc;
    rev_grad_reduce_tc_kernel<T><<<static_cast<unsigned>((rev_cta_floats(s) / 4 + kReduceQuads - 1) / kReduceQuads), kReduceQuads * kReduceShares, 0, stream>>>(
        s, workspace, n_ctas, static_cast<T *>(dw[0]), static_cast<T *>(dw[1]), static_cast<T *>(dw[2]),
        static_cast<T *>(dw[3]), static_cast<T *>(db[0]), static_cast<T *>(db[1]), static_cast<T *>(db[2]), static_cast<T *>(db[3]));
    return launch_status("rev_grad_reduce_tc_kernel launch");
}

}  // namespace

int rev_fwd_tc(const RevShape &s, const RevParams &p, const void *x, int64_t x_stride, void *y, int64_t y_stride,
               int64_t rows, int dtype, cudaStream_t stream) {
    if (rev_tc_disabled() || rows <= 0) return kRevTcNotApplicable;
    if (!rows16_ok(x, x_stride) || !rows16_ok(y, y_stride)) return kRevTcNotApplicable;
    switch (dtype) {
        case TH_F16: return launch_rev_fwd<__half>(s, p, x, x_stride, y, y_stride, rows, stream);
        case TH_BF16: return launch_rev_fwd<__nv_bfloat16>(s, p, x, x_stride, y, y_stride, rows, stream);
        default: return kRevTcNotApplicable;
    }
}

int rev_bwd_tc(const RevShape &s, const RevParams &p, const void *y, int64_t y_stride, const void *go, int64_t go_stride,
               void *gx, int64_t gx_stride, void *x_rec, int64_t xr_stride, void *const dw[4], void *const db[4], float *workspace,
               int n_ctas, int64_t rows, int dtype, cudaStream_t stream) {
    if (rev_tc_disabled() || rows <= 0) return kRevTcNotApplicable;
    // Biased batches that do not fill one tile stay with the mma.sync kernel, which agrees with the storage-rounded oracle in more
    // single rows (1.1 against 0.6 % of the rows of eight float16 blocks differ by a switched ReLU; a few rows are compared one by
    // one).  Against float64 neither is the more exact: ratio of the errors of eight and ten biased ReLU blocks, 128 .. 30 011 rows,
    // 0.995 float16, 1.0004 bfloat16.  In time the tensor core would gain (127 rows, eight blocks of 64: 115 -> 53 us).
    if (s.has_bias && rows < kTileRows) return kRevTcNotApplicable;
    if (!rows16_ok(y, y_stride) || !rows16_ok(go, go_stride) || (gx && !rows16_ok(gx, gx_stride)) ||
        (x_rec && !rows16_ok(x_rec, xr_stride)))
        return kRevTcNotApplicable;
#define TH_REV_BWD(T, A)                                                                                                              \
    (s.has_bias ? launch_rev_bwd_t<T, A, true>(s, p, y, y_stride, go, go_stride, gx, gx_stride, x_rec, xr_stride, dw, db, workspace,  \
                                               n_ctas, rows, stream)                                                                  \
                : launch_rev_bwd_t<T, A, false>(s, p, y, y_stride, go, go_stride, gx, gx_stride, x_rec, xr_stride, dw, db, workspace, \
                                                n_ctas, rows, stream))
#define TH_REV_BWD_ACT(T)                                          \
    switch (s.act) {                                               \
        case TH_ACT_RELU: return TH_REV_BWD(T, TH_ACT_RELU);       \
        case TH_ACT_SILU: return TH_REV_BWD(T, TH_ACT_SILU);       \
        case TH_ACT_RELU2: return TH_REV_BWD(T, TH_ACT_RELU2);     \
        default: return TH_REV_BWD(T, TH_ACT_NONE);                \
    }
    if (dtype == TH_F16) { TH_REV_BWD_ACT(__half) }
    if (dtype == TH_BF16) { TH_REV_BWD_ACT(__nv_bfloat16) }
    return kRevTcNotApplicable;
#undef TH_REV_BWD_ACT
#undef TH_REV_BWD
}

}  // namespace th

// Device-side status of the reversible tensor-core kernels: 0 = fine, 1 = a bounded wait ran out.
extern "C" int th_rev_tc_status(void) {
    int status = 0;
    if (cudaMemcpyFromSymbol(&status, th::g_tc_status, sizeof(int)) != cudaSuccess) return -1;
    return status;
}

