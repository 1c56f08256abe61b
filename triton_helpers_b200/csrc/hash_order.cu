// Spatial ordering of a batch of points, for the encoding kernels.
//
// What it buys: the encoding is bound by requests from the SMs to L2, one per corner row (pair).  Neighbours in
// space share corner rows on every level whose cells hold more than one point, so a batch walked along a Morton
// curve finds its rows in L1 (forward) and sums its gradients in registers before they go out (backward); the
// order of the points in memory is the caller's and usually random.
//
// A counting sort into cubic buckets, about one bucket per point (at most 2^21), in four launches:
//   clear     counters (one uint32 per bucket)
//   count     bucket of every point; the atomic that counts it returns the point's rank in its bucket
//   offsets   a CTA scans 2048 counters and takes its range of the output with ONE atomic on a cursor: ranges of
//             different CTAs follow each other in no fixed order, which costs nothing (2048 buckets are a compact
//             region of space) and saves the passes of a global scan
//   scatter   {x, y, z, row} of every point, one 16-byte store
// Points of one bucket keep no order among themselves.  Bound by random 4- and 16-byte accesses that stay in L2.
//
// The backward pass over an ordered batch is here too (hash_bwd_tile_kernel); the forward pass is hash_fwd_kernel.
#include "hash_device.cuh"

namespace th {
namespace {

constexpr int kScanThreads = 512;
constexpr int kScanItems = 4;  // counters per thread
constexpr int kScanTile = kScanThreads * kScanItems;

// Morton (Z-order) code by the usual halving masks: bit j of axis d goes to bit j * D + d.
template <int D>
__device__ __forceinline__ uint32_t spread(uint32_t v) {
    if constexpr (D == 1) return v;
    if constexpr (D == 2) {
        v &= 0xffffu;
        v = (v | (v << 8)) & 0x00ff00ffu;
        v = (v | (v << 4)) & 0x0f0f0f0fu;
        v = (v | (v << 2)) & 0x33333333u;
        return (v | (v << 1)) & 0x55555555u;
    }
    v &= 0x3ffu;
    v = (v | (v << 16)) & 0x030000ffu;
    v = (v | (v << 8)) & 0x0300f00fu;
    v = (v | (v << 4)) & 0x030c30c3u;
    return (v | (v << 2)) & 0x09249249u;
}

template <int D>
__device__ __forceinline__ uint32_t bucket_of(const float (&x)[D], int bits) {
    const float cells = static_cast<float>(1u << bits);
    uint32_t key = 0;
#pragma unroll
    for (int d = 0; d < D; ++d) {
        // saturating conversion (NaN and negative -> 0): coordinates outside the unit range end up in border buckets
        const uint32_t c = min(static_cast<uint32_t>(x[d] * cells), (1u << bits) - 1u);
        key |= spread<D>(c) << d;
    }
    return key;
}

template <int D>
__device__ __forceinline__ void read_point(const CoordView &cv, float scale, long long i, float (&x)[D]) {
    load_coords_strided<D>(cv, i, x);
    if (scale != 1.f) {
#pragma unroll
        for (int d = 0; d < D; ++d) x[d] = __fdiv_rn(x[d], scale);
    }
}

template <int D>
__global__ void __launch_bounds__(kThreads)
order_count_kernel(const CoordView cv, float scale, long long n, int bits, uint32_t *__restrict__ counters, uint32_t *__restrict__ rank) {
    const long long i = static_cast<long long>(blockIdx.x) * kThreads + threadIdx.x;
    if (i >= n) return;
    float x[D];
    read_point<D>(cv, scale, i, x);
    rank[i] = atomicAdd(counters + bucket_of<D>(x, bits), 1u);
}

// counters -> first output position of every bucket; counters[buckets] is the cursor
__global__ void __launch_bounds__(kScanThreads)
order_offsets_kernel(uint32_t *__restrict__ counters, uint32_t *__restrict__ cursor) {
    __shared__ uint32_t warp_sums[kScanThreads / 32];
    __shared__ uint32_t base;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    uint4 *mine = reinterpret_cast<uint4 *>(counters + static_cast<size_t>(blockIdx.x) * kScanTile) + threadIdx.x;
    const uint4 c = *mine;
    const uint32_t total = c.x + c.y + c.z + c.w;
    uint32_t sum = total;  // inclusive over the warp
#pragma unroll
    for (int d = 1; d < 32; d *= 2) {
        const uint32_t v = __shfl_up_sync(0xffffffffu, sum, d);
        if (lane >= d) sum += v;
    }
    if (lane == 31) warp_sums[warp] = sum;
    __syncthreads();
    if (warp == 0) {
        const uint32_t own = lane < kScanThreads / 32 ? warp_sums[lane] : 0u;
        uint32_t s = own;
#pragma unroll
        for (int d = 1; d < 32; d *= 2) {
            const uint32_t v = __shfl_up_sync(0xffffffffu, s, d);
            if (lane >= d) s += v;
        }
        if (lane < kScanThreads / 32) warp_sums[lane] = s - own;
        if (lane == 31) base = s ? atomicAdd(cursor, s) : 0u;
    }
    __syncthreads();
    uint4 first;
    first.x = base + warp_sums[warp] + sum - total;
    first.y = first.x + c.x;
    first.z = first.y + c.y;
    first.w = first.z + c.z;
    *mine = first;
}

template <int D>
__global__ void __launch_bounds__(kThreads)
order_scatter_kernel(const CoordView cv, float scale, long long n, int bits, const uint32_t *__restrict__ first,
                     const uint32_t *__restrict__ rank, float4 *__restrict__ order) {
    const long long i = static_cast<long long>(blockIdx.x) * kThreads + threadIdx.x;
    if (i >= n) return;
    float x[D];
    read_point<D>(cv, scale, i, x);
    float4 p = make_float4(x[0], 0.f, 0.f, __uint_as_float(static_cast<uint32_t>(i)));
    if constexpr (D > 1) p.y = x[1];
    if constexpr (D > 2) p.z = x[2];
    order[first[bucket_of<D>(x, bits)] + __ldcs(rank + i)] = p;
}

// Bits per axis: about one bucket per point, 2^21 (three axes) or 2^20 at most - finer buckets than points order
// nothing more on uniform points, and clustered ones (whose buckets are the fuller ones) still get the finest.
int order_bits(int64_t n, int dims) {
    int log2n = 11;  // the scan works on whole tiles of 2048 counters
    while ((1ll << log2n) < n && log2n < 21) ++log2n;
    int bits = log2n / dims;
    while (bits * dims < 11) ++bits;
    return bits;
}

template <int D>
int launch_order(const CoordView &cv, float scale, int64_t n, float4 *order, uint32_t *scratch, cudaStream_t stream) {
    const int bits = order_bits(n, D);
    const size_t buckets = static_cast<size_t>(1) << (bits * D);
    uint32_t *counters = scratch, *cursor = scratch + buckets, *rank = cursor + 4;
    if (int rc = cuda_status(cudaMemsetAsync(scratch, 0, (buckets + 4) * sizeof(uint32_t), stream), "cudaMemsetAsync(order counters)")) return rc;
    const unsigned grid = static_cast<unsigned>((n + kThreads - 1) / kThreads);
    order_count_kernel<D><<<grid, kThreads, 0, stream>>>(cv, scale, n, bits, counters, rank);
    if (int rc = launch_status("order_count_kernel launch")) return rc;
    order_offsets_kernel<<<static_cast<unsigned>(buckets / kScanTile), kScanThreads, 0, stream>>>(counters, cursor);
    if (int rc = launch_status("order_offsets_kernel launch")) return rc;
    order_scatter_kernel<D><<<grid, kThreads, 0, stream>>>(cv, scale, n, bits, counters, rank, order);
    return launch_status("order_scatter_kernel launch");
}

// ---- backward over an ordered batch --------------------------------------------------------------
//
// A CTA takes a tile of 1024 consecutive points, a compact piece of space; a thread keeps four of them in registers.
// On a level whose cells hold several points the tile is sorted by cell in shared memory (a counting sort: integer
// atomics, one scan; what is sorted are records of the fractional position, the packed cell and the gradient), every
// lane pair walks eight records and keeps the sums of its 2^(D-1) corners in registers while the cell stays the same,
// and pairs that stop in the cell their neighbours work on are summed across the warp.  A cell then costs one
// reduction per corner and tile instead of one per corner and point; sums are formed in float32 whatever the table's
// type.  On the first level that shows fewer than 1.5 points per cell the CTA goes over to one reduction per corner
// and point, as hash_bwd_kernel, for that level and all finer ones: sorting costs about as many instructions as it
// would save requests there.  The choice is the tile's own, so clustered batches keep sorting on levels where uniform
// ones do not.
//
// Bound by the SMs' requests to L2 (request path 68 % busy, L2 68 %, a third of the issue slots used: 22 warps per SM that wait for
// memory most of the time); CTAs that sort and CTAs on the fine levels overlap.  Against hash_bwd_kernel + hash_bwd_coarse_kernel
// on unordered points: 2^21 uniform points, 16 levels, 2 x float16: 0.65 against 0.77 ms (gradients in order; 0.70 in the caller's);
// 2^22 points in 8 clusters, 4 x float32, 681 MB: 2.31 against 4.12 ms.

constexpr int kTileBins = 2048;

// A cell's coordinates in one word, exact for cells up to kMask: grids up to kMaxSortedRes with coordinates in the unit range.
// Finer levels are not sorted, nor is a tile whose points could reach past cell kMask (coordinates above the range are accepted
// and hashed as they are: a clamped cell would send their gradients to other rows than their values come from).
template <int D>
struct CellKey {
    static constexpr int kBits = 32 / D;  // 32, 16, 10
    static constexpr uint32_t kMask = D == 1 ? 0xffffffffu : (1u << kBits) - 1u;
    static constexpr uint32_t kMaxSortedRes = kMask;

    static __device__ __forceinline__ uint32_t pack(const uint32_t (&cell)[D]) {
        uint32_t key = 0;
#pragma unroll
        for (int d = 0; d < D; ++d) key |= (D == 1 ? cell[d] : min(cell[d], kMask)) << (d * kBits % 32);
        return key;
    }
    // Whether the cells of points up to `top` fit their fields on every grid that is sorted: locate()'s product, which grows with
    // the coordinate and the grid.
    static __device__ __forceinline__ bool fits(float top) {
        return D == 1 || !(__fmul_rn(top, static_cast<float>(kMaxSortedRes)) >= static_cast<float>(kMask) + 1.f);
    }
    static __device__ __forceinline__ void unpack(uint32_t key, uint32_t (&cell)[D]) {
#pragma unroll
        for (int d = 0; d < D; ++d) cell[d] = (key >> (d * kBits % 32)) & kMask;
    }
    // Bin of a cell: its low coordinate bits, so that the cells of a compact region fall into different bins (two cells
    // in one bin only break a run).
    static __device__ __forceinline__ uint32_t bin(uint32_t key) {
        if constexpr (D == 1) return key & 2047u;
        if constexpr (D == 2) return (key & 63u) | ((key >> 10) & (31u << 6));
        return (key & 15u) | ((key >> 6) & (15u << 4)) | ((key >> 12) & (7u << 8));
    }
};

// blockIdx.y: the pass (range of levels).  Passes are the slower grid index, so that the CTAs resident at one time mostly
// update the rows of one pass.
template <typename T, int D, int F>
__global__ void __launch_bounds__(kThreads, 3)
hash_bwd_tile_kernel(const __grid_constant__ LevelParams P, const __grid_constant__ LevelPasses passes, const float4 *__restrict__ order,
                     const T *__restrict__ grad_out, long long go_stride, int keep_order, int row_vector_ok, int group_vector_ok,
                     T *__restrict__ grad_table, long long n_points) {
    constexpr int kSide = 1 << (D - 1);
    constexpr int kGroup = F * sizeof(T) >= 16 ? 1 : 16 / (F * sizeof(T));  // levels in 16 bytes of a gradient row
    constexpr int kTilePoints = kPointsPerTile<F>;
    constexpr int kOwn = kTilePoints / kThreads;        // points per thread while sorting
    constexpr int kRun = kTilePoints / (kThreads / 2);  // records per lane pair while summing
    using Key = CellKey<D>;
    __shared__ __align__(16) float4 where[kTilePoints];  // fractional position, packed cell
    __shared__ __align__(16) float grads[kTilePoints * F];
    __shared__ __align__(16) uint32_t bins[kTileBins];
    __shared__ uint32_t warp_points[kThreads / 32], warp_bins[kThreads / 32];
    __shared__ float warp_low[kThreads / 32][D], warp_high[kThreads / 32][D];
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, side = tid & 1, pair = tid >> 1;
    const long long first = static_cast<long long>(blockIdx.x) * kTilePoints;
    const int count = n_points - first < kTilePoints ? static_cast<int>(n_points - first) : kTilePoints;
    const int level_end = passes.end[blockIdx.y];
    int level = passes.begin[blockIdx.y];

    // ---- levels with several points per cell ----
    if (P.res[level] <= Key::kMaxSortedRes) {
        float x[kOwn][D];
        uint32_t row[kOwn];
#pragma unroll
        for (int j = 0; j < kOwn; ++j) {
            const int id = tid + j * kThreads;
            row[j] = 0;
#pragma unroll
            for (int d = 0; d < D; ++d) x[j][d] = 0.f;
            if (id < count) {
                row[j] = load_ordered<D>(order, first + id, x[j]);
                if (keep_order) row[j] = static_cast<uint32_t>(first + id);
            }
        }
        // the tile's bounding box: a level on which it has far more cells than the tile has points is not worth a look (infinite, and no
        // level is, where a cell would not fit its key)
        float extent[D];
#pragma unroll
        for (int d = 0; d < D; ++d) {
            float low = __FLT_MAX__, high = -__FLT_MAX__;
#pragma unroll
            for (int j = 0; j < kOwn; ++j) {
                if (tid + j * kThreads < count) {
                    low = fminf(low, x[j][d]);
                    high = fmaxf(high, x[j][d]);
                }
            }
#pragma unroll
            for (int step = 16; step > 0; step /= 2) {
                low = fminf(low, __shfl_xor_sync(0xffffffffu, low, step));
                high = fmaxf(high, __shfl_xor_sync(0xffffffffu, high, step));
            }
            if (lane == 0) {
                warp_low[warp][d] = low;
                warp_high[warp][d] = high;
            }
        }
        __syncthreads();
#pragma unroll
        for (int d = 0; d < D; ++d) {
            float low = warp_low[0][d], high = warp_high[0][d];
#pragma unroll
            for (int w = 1; w < kThreads / 32; ++w) {
                low = fminf(low, warp_low[w][d]);
                high = fmaxf(high, warp_high[w][d]);
            }
            extent[d] = Key::fits(high) ? high - low : __int_as_float(0x7f800000);
        }
        for (; level < level_end && P.res[level] <= Key::kMaxSortedRes; ++level) {
            const uint32_t res = P.res[level];
            float box = 1.f;
#pragma unroll
            for (int d = 0; d < D; ++d) box *= __fmaf_rn(extent[d], static_cast<float>(res), 1.f);
            if (box > 4.f * count) break;
            float go[kOwn][F];
#pragma unroll
            for (int j = 0; j < kOwn; ++j)
                if (tid + j * kThreads < count) load_elems_checked<T, F>(grad_out + row[j] * go_stride + level * F, go[j], row_vector_ok);
            reinterpret_cast<uint4 *>(bins)[tid] = make_uint4(0, 0, 0, 0);
            reinterpret_cast<uint4 *>(bins)[tid + kThreads] = make_uint4(0, 0, 0, 0);
            __syncthreads();
            uint32_t key[kOwn], rank[kOwn];
            float t[kOwn][D];
#pragma unroll
            for (int j = 0; j < kOwn; ++j) {
                uint32_t cell[D];
                locate<D>(x[j], res, cell, t[j]);
                key[j] = Key::pack(cell);
                if (tid + j * kThreads < count) rank[j] = atomicAdd(bins + Key::bin(key[j]), 1u);
            }
            __syncthreads();
            constexpr int kPer = kTileBins / kThreads;  // bins per thread
            uint32_t c[kPer], total = 0, used = 0;
#pragma unroll
            for (int k = 0; k < kPer; k += 4) {
                const uint4 four = reinterpret_cast<const uint4 *>(bins)[tid * (kPer / 4) + k / 4];
                c[k] = four.x;
                c[k + 1] = four.y;
                c[k + 2] = four.z;
                c[k + 3] = four.w;
            }
#pragma unroll
            for (int k = 0; k < kPer; ++k) {
                total += c[k];
                used += c[k] ? 1u : 0u;
            }
            uint32_t sum = total;  // inclusive over the warp
#pragma unroll
            for (int d = 1; d < 32; d *= 2) {
                const uint32_t v = __shfl_up_sync(0xffffffffu, sum, d);
                if (lane >= d) sum += v;
            }
            used = __reduce_add_sync(0xffffffffu, used);
            if (lane == 31) {
                warp_points[warp] = sum;
                warp_bins[warp] = used;
            }
            __syncthreads();
            uint32_t at_bin = sum - total, all_used = 0;
#pragma unroll
            for (int w = 0; w < kThreads / 32; ++w) {
                if (w < warp) at_bin += warp_points[w];
                all_used += warp_bins[w];
            }
            if (3 * all_used > 2 * static_cast<uint32_t>(count)) break;  // the same for every thread
#pragma unroll
            for (int k = 0; k < kPer; ++k) {
                const uint32_t n = c[k];
                c[k] = at_bin;
                at_bin += n;
            }
#pragma unroll
            for (int k = 0; k < kPer; k += 4)
                reinterpret_cast<uint4 *>(bins)[tid * (kPer / 4) + k / 4] = make_uint4(c[k], c[k + 1], c[k + 2], c[k + 3]);
            __syncthreads();
#pragma unroll
            for (int j = 0; j < kOwn; ++j) {
                if (tid + j * kThreads < count) {
                    // record r goes to slot (r % kRun, r / kRun): the k-th records of neighbouring pairs are neighbours in memory
                    const uint32_t r = bins[Key::bin(key[j])] + rank[j];
                    const uint32_t at = (r % kRun) * (kThreads / 2) + r / kRun;
                    where[at] = make_float4(t[j][0], D > 1 ? t[j][D > 1 ? 1 : 0] : 0.f, D > 2 ? t[j][D > 2 ? 2 : 0] : 0.f, __uint_as_float(key[j]));
                    if constexpr (F == 2) {
                        reinterpret_cast<float2 *>(grads)[at] = make_float2(go[j][0], go[j][1]);
                    } else if constexpr (F % 4 == 0) {
#pragma unroll
                        for (int f = 0; f < F; f += 4)
                            reinterpret_cast<float4 *>(grads)[at * (F / 4) + f / 4] = make_float4(go[j][f], go[j][f + 1], go[j][f + 2], go[j][f + 3]);
                    } else {
                        grads[at] = go[j][0];
                    }
                }
            }
            __syncthreads();

            // walk the records, eight per lane pair
            T *base = grad_table + P.offset[level] * F;
            const int here = min(count - pair * kRun, kRun);
            uint32_t at = 0;
            float acc[kSide][F];
#pragma unroll
            for (int k = 0; k < kSide; ++k)
#pragma unroll
                for (int f = 0; f < F; ++f) acc[k][f] = 0.f;
            auto flush = [&]() {
                uint32_t cell[D], idx[kSide];
                Key::unpack(at, cell);
                side_indices<D>(cell, P, level, side, idx);
#pragma unroll
                for (int k = 0; k < kSide; ++k) red_add_row<F>(base + static_cast<size_t>(idx[k]) * F, acc[k]);
            };
#pragma unroll
            for (int k = 0; k < kRun; ++k) {
                if (k >= here) break;
                const float4 q = where[k * (kThreads / 2) + pair];
                float g[F], pos[D], w[kSide];
                if constexpr (F == 2) {
                    const float2 v = reinterpret_cast<const float2 *>(grads)[k * (kThreads / 2) + pair];
                    g[0] = v.x;
                    g[1] = v.y;
                } else if constexpr (F % 4 == 0) {
#pragma unroll
                    for (int f = 0; f < F; f += 4) {
                        const float4 v = reinterpret_cast<const float4 *>(grads)[(k * (kThreads / 2) + pair) * (F / 4) + f / 4];
                        g[f] = v.x;
                        g[f + 1] = v.y;
                        g[f + 2] = v.z;
                        g[f + 3] = v.w;
                    }
                } else {
                    g[0] = grads[k * (kThreads / 2) + pair];
                }
                pos[0] = q.x;
                if constexpr (D > 1) pos[1] = q.y;
                if constexpr (D > 2) pos[2] = q.z;
                const uint32_t cell_key = __float_as_uint(q.w);
                if (cell_key != at || k == 0) {
                    if (k > 0) flush();
                    at = cell_key;
#pragma unroll
                    for (int j = 0; j < kSide; ++j)
#pragma unroll
                        for (int f = 0; f < F; ++f) acc[j][f] = 0.f;
                }
                side_weights<D>(pos, side, w);
#pragma unroll
                for (int j = 0; j < kSide; ++j)
#pragma unroll
                    for (int f = 0; f < F; ++f) acc[j][f] = __fmaf_rn(w[j], g[f], acc[j][f]);
            }
            __syncwarp();
            // pairs next to each other that stopped in one cell: the first of them takes the others' sums
            const bool head = __shfl_up_sync(0xffffffffu, at, 2) != at || lane < 2 || here <= 0;
            const uint32_t heads = __ballot_sync(0xffffffffu, head) & 0x55555555u;
            if (heads != 0x55555555u) {
                const uint32_t later = heads & ~((2u << (lane & 30)) - 1u);
                const int end = later ? __ffs(later) - 1 : 32;  // first lane of the next cell
#pragma unroll
                for (int step = 2; step < 32; step *= 2) {
                    const bool inside = lane + step < end;
                    if (!__any_sync(0xffffffffu, inside)) break;
#pragma unroll
                    for (int k = 0; k < kSide; ++k)
#pragma unroll
                        for (int f = 0; f < F; ++f) {
                            const float other = __shfl_down_sync(0xffffffffu, acc[k][f], step);
                            if (inside) acc[k][f] += other;
                        }
                }
            }
            if (head && here > 0) flush();
        }
    }
    if (level >= level_end) return;

    // ---- finer levels: one reduction per corner and point ----
    // (in a launch of its own this part fills the SMs better and is still slower together with the sorting, 0.80 against
    //  0.70 ms at 2^21 points: here tiles that sort and tiles that wait for the request path share an SM.  Fetching the
    //  gradients of several points of a pair ahead: 0.76 ms, spills.)
    for (int id = pair; id < count; id += kThreads / 2) {
        float x[D];
        const uint32_t row = load_ordered<D>(order, first + id, x);
        const T *go_row = grad_out + (keep_order ? first + id : static_cast<long long>(row)) * go_stride;
        auto scatter = [&](int l, const float *go) {
            uint32_t cell[D], idx[kSide];
            float t[D], w[kSide];
            locate<D>(x, P.res[l], cell, t);
            side_weights<D>(t, side, w);
            side_indices<D>(cell, P, l, side, idx);
            T *base = grad_table + P.offset[l] * F;
#pragma unroll
            for (int k = 0; k < kSide; ++k) {
                float v[F];
#pragma unroll
                for (int f = 0; f < F; ++f) v[f] = __fmul_rn(w[k], go[f]);
                red_add_row<F>(base + static_cast<size_t>(idx[k]) * F, v);
            }
        };
        int l = level;
        while (l < level_end) {
            if (kGroup > 1 && l % kGroup == 0 && l + kGroup <= level_end) {
                float go[kGroup * F];
                load_elems_checked<T, kGroup * F>(go_row + l * F, go, group_vector_ok);
#pragma unroll
                for (int j = 0; j < kGroup; ++j) scatter(l + j, go + j * F);
                l += kGroup;
            } else {
                float go[F];
                load_elems_checked<T, F>(go_row + l * F, go, row_vector_ok);
                scatter(l, go);
                ++l;
            }
        }
    }
}

template <typename T, int D, int F>
int launch_bwd_ordered(const LevelParams &P, const float4 *order, int keep_order, const void *go, int64_t go_stride, void *grad_table,
                       int64_t n, int l0, int l1, cudaStream_t stream) {
    constexpr int kRow = F * sizeof(T) < 16 ? F * sizeof(T) : 16;
    const int row_vec = aligned_to(go, kRow) && (go_stride * sizeof(T)) % kRow == 0;
    const int group_vec = aligned_to(go, 16) && (go_stride * sizeof(T)) % 16 == 0;
    LevelPasses passes = plan_level_passes(P, n, l0, l1, F * sizeof(T));
    const long long tiles = (n + kPointsPerTile<F> - 1) / kPointsPerTile<F>;
    // Small batches: less than two waves of tiles (three CTAs per SM) are split over the levels as well, in pieces of a
    // multiple of four (200 003 points in two dimensions, 16 levels: one piece 71 us, two 52).
    if (passes.count == 1) {
        int pieces = 1;
        while (pieces < 4 && (l1 - l0) % (8 * pieces) == 0 && l0 % 4 == 0 && tiles * pieces < 6ll * sm_count()) pieces *= 2;
        passes.count = pieces;
        for (int p = 0; p < pieces; ++p) {
            passes.begin[p] = l0 + (l1 - l0) / pieces * p;
            passes.end[p] = passes.begin[p] + (l1 - l0) / pieces;
        }
    }
    const dim3 grid(static_cast<unsigned>(tiles), static_cast<unsigned>(passes.count), 1);
    hash_bwd_tile_kernel<T, D, F><<<grid, kThreads, 0, stream>>>(P, passes, order, static_cast<const T *>(go), go_stride, keep_order, row_vec, group_vec,
                                                                 static_cast<T *>(grad_table), n);
    return launch_status("hash_bwd_tile_kernel launch");
}

}  // namespace
}  // namespace th

using namespace th;

// Where the order pays: time with it, sorting included, over time without (B200; 2, 4, 8 or 16 levels, tables of 2^14 .. 2^22 rows per
// level, finest grids of 512 .. 4096, 1 .. 8 features of 2 or 4 bytes, points uniform or in eight clusters, which the host cannot tell
// apart).  A form is ordered where none of these is more than a few hundredths above 1:
//   forward + backward, three dimensions, 16 levels: 2^19 0.40-0.99, 2^20 0.40-0.96, 2^21 0.41-0.97, 2^23 0.78-1.01; eight levels share
//     the cost of sorting: 2^19 0.40-1.04, 2^20 0.45-1.01, 2^21 0.46-0.94; four: 2^19 0.50-1.35, 2^21 0.42-1.16.  Left out: tables with
//     more than twelve rows a point (0.42-1.24), past 24 M rows with rows below 16 bytes (2^22 0.98-1.05), past 8 M rows with
//     eight levels (2^21 up to 1.13) or rows of 8 x 16 bit (up to 1.05; less 0.41-1.00), rows of one 16-bit element (single-element
//     atomics, 0.25-1.3).
//   two dimensions, 4 x float32, 16 levels: 2^16 0.99, 2^17 0.63-0.91, 2^19 0.62-0.95, 2^20 0.66-1.00, 2^21 0.78-1.14 (the ordered
//     forward writes whole rows in random order, and loses once all of them are past twice the L2); eight: 2^17 0.75-0.99, 2^20
//     0.65-0.93; four: up to 1.14; 8 x 16 bit 0.56-1.02, 2^21 up to 1.05, one dimension up to 1.16.  8 x float32 in one or two: 16 levels
//     2^17 0.33-0.86, 2^21 0.62-0.95, four 2^17 0.55-0.98, two up to 1.24.  Narrower rows: two dimensions 0.80-1.35, one 0.74-1.94.
//   forward alone, three dimensions, 16 levels, up to four features, outputs up to 512 MB (more: up to 1.25), tables up to 24 M rows
//     (more: 0.73-1.22): rows of 8 and 16 bytes 2^19 0.65-1.15, 2^20 0.59-1.04, 2^21 0.55-1.03; of 4 bytes 2^20 0.62-1.12, 2^21
//     0.55-0.94, 2^23 0.77-0.91; eight levels 2^21 0.66-1.54; eight features 0.81-2.2; two dimensions 0.69-3.9; one 1.16-3.5.
extern "C" int th_hash_order_pays(int64_t n_points, int n_dims, int n_feats, int n_levels, int row_bytes, int64_t table_rows, int backward) {
    if (n_points >= (1ll << 31) || row_bytes < 4) return 0;
    const int64_t outputs = n_points * n_levels * row_bytes;
    const bool large = table_rows > (24ll << 20);
    if (!backward) return n_dims >= 3 && n_feats <= 4 && n_levels >= 16 && n_points >= (row_bytes >= 8 ? 1 << 20 : 1 << 21) && outputs <= (1ll << 29) && !large;
    if (n_dims >= 3) {
        if (n_points < (1 << 19) || 12 * n_points < table_rows || (large && row_bytes < 16)) return 0;
        if (n_feats == 8 && row_bytes < 32 && table_rows > (8ll << 20)) return 0;
        return n_levels >= 16 || (n_levels >= 8 && n_points >= (1 << 20) && outputs <= (1ll << 28) && table_rows <= (8ll << 20));
    }
    if (n_points < (1 << 17)) return 0;
    if (row_bytes >= 32) return n_levels >= 4;
    return n_dims == 2 && row_bytes == 16 && n_levels >= 8 && outputs <= (1ll << 28);
}

extern "C" int64_t th_hash_order_scratch_bytes(int64_t n_points, int n_dims) {
    if (n_points < 0 || n_points >= (1ll << 31) || n_dims < 1 || n_dims > TH_MAX_DIMS) return -1;
    return static_cast<int64_t>(((static_cast<size_t>(1) << (order_bits(n_points, n_dims) * n_dims)) + 4 + static_cast<size_t>(n_points)) * sizeof(uint32_t));
}

extern "C" int th_hash_order(const void *coords_dev, int64_t coord_stride_n, int64_t coord_stride_d, int coord_dtype, int64_t n_points,
                             int n_dims, float scale, void *order_dev, void *scratch_dev, int64_t scratch_bytes, void *stream) {
    if (n_points < 0 || n_points >= (1ll << 31)) return fail(TH_ERR_BAD_ARG, "n_points %lld outside [0, 2^31)", (long long)n_points);
    if (n_dims < 1 || n_dims > TH_MAX_DIMS) return fail(TH_ERR_UNSUPPORTED, "n_dims %d outside [1, %d]", n_dims, TH_MAX_DIMS);
    if (!(scale > 0.f)) return fail(TH_ERR_BAD_ARG, "scale must be positive");
    if (n_points == 0) return TH_OK;
    CoordView cv;
    if (int rc = make_coord_view(cv, coords_dev, coord_stride_n, coord_stride_d, coord_dtype, n_dims)) return rc;
    if (!order_dev || !scratch_dev) return fail(TH_ERR_BAD_ARG, "null order or scratch");
    if (!aligned_to(order_dev, 16) || !aligned_to(scratch_dev, 16)) return fail(TH_ERR_ALIGNMENT, "order and scratch must be 16-byte aligned");
    const int64_t need = th_hash_order_scratch_bytes(n_points, n_dims);
    if (scratch_bytes < need) return fail(TH_ERR_WORKSPACE, "scratch of %lld bytes needed, %lld given", (long long)need, (long long)scratch_bytes);
    cudaStream_t s = static_cast<cudaStream_t>(stream);
    float4 *order = static_cast<float4 *>(order_dev);
    uint32_t *scratch = static_cast<uint32_t *>(scratch_dev);
    switch (n_dims) {
        case 1: return launch_order<1>(cv, scale, n_points, order, scratch, s);
        case 2: return launch_order<2>(cv, scale, n_points, order, scratch, s);
        default: return launch_order<3>(cv, scale, n_points, order, scratch, s);
    }
}

extern "C" int th_hash_bwd_ordered(const void *order_dev, int keep_order, const void *grad_out_dev, int64_t go_stride_n, void *grad_table_dev,
                                   int table_dtype, int64_t n_points, int n_dims, int n_feats, int n_levels, const int32_t *level_res_host,
                                   const int64_t *level_rows_host, const int64_t *level_offset_host, const int64_t *primes_host, int level_begin,
                                   int level_end, void *stream) {
    if (n_points < 0) return fail(TH_ERR_BAD_ARG, "negative n_points");
    LevelParams P;
    if (int rc = fill_params(P, n_dims, n_levels, level_res_host, level_rows_host, level_offset_host, primes_host, 1.f)) return rc;
    if (!level_offset_host) return fail(TH_ERR_BAD_ARG, "null level offsets");
    if (int rc = check_range(n_levels, level_begin, level_end)) return rc;
    if (n_points == 0) return TH_OK;
    if (!order_dev || !grad_out_dev || !grad_table_dev) return fail(TH_ERR_BAD_ARG, "null order or gradient pointer");
    const size_t row_bytes = n_feats * dtype_bytes(table_dtype);
    if (!aligned_to(order_dev, 16)) return fail(TH_ERR_ALIGNMENT, "the order must be 16-byte aligned");
    if (!aligned_to(grad_table_dev, row_bytes < 16 ? row_bytes : 16)) return fail(TH_ERR_ALIGNMENT, "table rows must be aligned to min(row bytes, 16)");
    if (go_stride_n < static_cast<int64_t>(n_levels) * n_feats) return fail(TH_ERR_BAD_ARG, "go_stride_n smaller than n_levels * n_feats");
    const float4 *order = static_cast<const float4 *>(order_dev);
    cudaStream_t s = static_cast<cudaStream_t>(stream);
#define TH_CALL_BWD(T, D, F) launch_bwd_ordered<T, D, F>(P, order, keep_order, grad_out_dev, go_stride_n, grad_table_dev, n_points, level_begin, level_end, s)
    TH_DISPATCH(TH_CALL_BWD)
#undef TH_CALL_BWD
}
