// The two element-wise steps either side of the fused operators in a neural-field training
// step: the scaled MSE gradient that feeds the MLP backward, and an Adam update for 16-bit
// parameters with fp32 moments.  triton_helpers has no counterpart (its benchmarks stop at
// forward/backward, triton_helpers/benchmark.py:175-187); these exist so the data-parallel
// training step never leaves hand-written kernels between the forward and the next step.
//
// Both are pure streaming kernels: 128-bit loads and stores, grid-stride over 8-element packets.
#include "common.cuh"

namespace th {
namespace {

constexpr int kOptThreads = 256;

template <typename T>
struct Vec8 {
    T v[8];
};
template <>
struct __align__(16) Vec8<__half> {
    __half v[8];
};
template <>
struct __align__(16) Vec8<__nv_bfloat16> {
    __nv_bfloat16 v[8];
};
template <>
struct __align__(32) Vec8<float> {
    float v[8];
};

// grad = (pred - target) * grad_scale ;  *loss_sum += sum (pred - target)^2
template <typename T>
__global__ void __launch_bounds__(kOptThreads)
mse_grad_kernel(const T *__restrict__ pred, const T *__restrict__ target, T *__restrict__ grad,
                float *__restrict__ loss_sum, long long n, float grad_scale) {
    float local = 0.f;
    const long long packets = n / 8;
    for (long long i = static_cast<long long>(blockIdx.x) * blockDim.x + threadIdx.x; i < packets;
         i += static_cast<long long>(gridDim.x) * blockDim.x) {
        const Vec8<T> p = reinterpret_cast<const Vec8<T> *>(pred)[i];
        const Vec8<T> t = reinterpret_cast<const Vec8<T> *>(target)[i];
        Vec8<T> g;
#pragma unroll
        for (int k = 0; k < 8; ++k) {
            const float d = to_float<T>(p.v[k]) - to_float<T>(t.v[k]);
            local += d * d;
            g.v[k] = from_float<T>(d * grad_scale);
        }
        reinterpret_cast<Vec8<T> *>(grad)[i] = g;
    }
    // ragged tail
    for (long long i = packets * 8 + static_cast<long long>(blockIdx.x) * blockDim.x + threadIdx.x; i < n;
         i += static_cast<long long>(gridDim.x) * blockDim.x) {
        const float d = to_float<T>(pred[i]) - to_float<T>(target[i]);
        local += d * d;
        grad[i] = from_float<T>(d * grad_scale);
    }
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) local += __shfl_xor_sync(0xffffffffu, local, off);
    __shared__ float warp_sum[kOptThreads / 32];
    if ((threadIdx.x & 31) == 0) warp_sum[threadIdx.x >> 5] = local;
    __syncthreads();
    if (threadIdx.x == 0) {
        float total = 0.f;
#pragma unroll
        for (int w = 0; w < kOptThreads / 32; ++w) total += warp_sum[w];
        if (loss_sum) atomicAdd(loss_sum, total);
    }
}

struct AdamScalars {
    float lr, beta1, beta2, eps;
    float bias1, bias2_sqrt;  // 1 - beta1^t, sqrt(1 - beta2^t)
    float grad_scale;         // multiplies the stored gradient (1 / loss scale / world size)
    int zero_grad;            // write zeros back into the gradient buffer
};

// One element.  A gradient that is not finite (a 16-bit sum that overflowed, a NaN from upstream)
// leaves the parameter and both moments as they were and is counted in `skipped`: one bad element
// must not turn into inf / inf = NaN in the parameter and poison every later step.
template <typename T>
__device__ __forceinline__ T adam_one(T p, T g_in, float &m, float &v, const AdamScalars &a, int &skipped) {
    const float g = to_float<T>(g_in) * a.grad_scale;
    if (!isfinite(g)) {
        ++skipped;
        return p;
    }
    m = a.beta1 * m + (1.f - a.beta1) * g;
    v = a.beta2 * v + (1.f - a.beta2) * g * g;
    const float denom = sqrtf(v) / a.bias2_sqrt + a.eps;
    return from_float<T>(to_float<T>(p) - (a.lr / a.bias1) * (m / denom));
}

// Elements of a parameter in one 16-byte packet, and the matching moments (float32: four, for twice the threads and half their
// registers of eight: 3.3 M parameters 34.2 -> 26.4 us)
template <typename T>
constexpr int kPacket = 16 / sizeof(T);
template <typename T>
struct __align__(16) Packet16 {
    T v[kPacket<T>];
};
template <int N>
struct __align__(16) Moments {
    float v[N];
};

// The same update for several tensors of one dtype in one launch: a small network's tensors are a few blocks each, and
// a launch per tensor (seven for a table and a biased MLP: 43 us of kernels and 100 us of host time in a training step)
// costs more than the update.  Every block walks every tensor with the whole grid's stride.
constexpr int kMaxTensors = 16;

struct AdamTensors {
    void *param[kMaxTensors], *grad[kMaxTensors];
    float *exp_avg[kMaxTensors], *exp_avg_sq[kMaxTensors];
    long long n[kMaxTensors];
    float grad_scale[kMaxTensors];
    int zero_grad[kMaxTensors];
    int count;
};

template <typename T>
__device__ __forceinline__ int adam_walk(T *__restrict__ param, T *__restrict__ grad, float *__restrict__ exp_avg, float *__restrict__ exp_avg_sq,
                                         long long n, const AdamScalars &a) {
    constexpr int N = kPacket<T>;
    int skipped = 0;
    const long long packets = n / N;
    for (long long i = static_cast<long long>(blockIdx.x) * blockDim.x + threadIdx.x; i < packets;
         i += static_cast<long long>(gridDim.x) * blockDim.x) {
        Packet16<T> p = reinterpret_cast<Packet16<T> *>(param)[i];
        const Packet16<T> g = reinterpret_cast<const Packet16<T> *>(grad)[i];
        Moments<N> m = reinterpret_cast<Moments<N> *>(exp_avg)[i];
        Moments<N> v = reinterpret_cast<Moments<N> *>(exp_avg_sq)[i];
#pragma unroll
        for (int k = 0; k < N; ++k) p.v[k] = adam_one<T>(p.v[k], g.v[k], m.v[k], v.v[k], a, skipped);
        reinterpret_cast<Packet16<T> *>(param)[i] = p;
        reinterpret_cast<Moments<N> *>(exp_avg)[i] = m;
        reinterpret_cast<Moments<N> *>(exp_avg_sq)[i] = v;
        if (a.zero_grad) {
            Packet16<T> z;
#pragma unroll
            for (int k = 0; k < N; ++k) z.v[k] = from_float<T>(0.f);
            reinterpret_cast<Packet16<T> *>(grad)[i] = z;
        }
    }
    for (long long i = packets * N + static_cast<long long>(blockIdx.x) * blockDim.x + threadIdx.x; i < n;
         i += static_cast<long long>(gridDim.x) * blockDim.x) {
        param[i] = adam_one<T>(param[i], grad[i], exp_avg[i], exp_avg_sq[i], a, skipped);
        if (a.zero_grad) grad[i] = from_float<T>(0.f);
    }
    return skipped;
}

template <typename T>
__global__ void __launch_bounds__(kOptThreads)
adam_many_kernel(const __grid_constant__ AdamTensors t, AdamScalars a, int *__restrict__ skipped_total) {
    int skipped = 0;
    for (int k = 0; k < t.count; ++k) {
        a.grad_scale = t.grad_scale[k];
        a.zero_grad = t.zero_grad[k];
        skipped += adam_walk<T>(static_cast<T *>(t.param[k]), static_cast<T *>(t.grad[k]), t.exp_avg[k], t.exp_avg_sq[k], t.n[k], a);
    }
    if (skipped_total && skipped) atomicAdd(skipped_total, skipped);
}

struct CastTensors {
    const void *src[kMaxTensors];
    void *dst[kMaxTensors];
    long long n[kMaxTensors];
    int count;
};

// dst = src in another type, several tensors in one launch; 8 elements per access where both are 32-byte aligned
template <typename S, typename T>
__global__ void __launch_bounds__(kOptThreads)
cast_many_kernel(const __grid_constant__ CastTensors t) {
    const long long first = static_cast<long long>(blockIdx.x) * blockDim.x + threadIdx.x, stride = static_cast<long long>(gridDim.x) * blockDim.x;
    for (int k = 0; k < t.count; ++k) {
        const S *src = static_cast<const S *>(t.src[k]);
        T *dst = static_cast<T *>(t.dst[k]);
        const long long n = t.n[k];
        const bool vec = ((reinterpret_cast<unsigned long long>(src) | reinterpret_cast<unsigned long long>(dst)) & 31ull) == 0;
        const long long packets = vec ? n / 8 : 0;
        for (long long i = first; i < packets; i += stride) {
            const Vec8<S> in = reinterpret_cast<const Vec8<S> *>(src)[i];
            Vec8<T> out;
#pragma unroll
            for (int e = 0; e < 8; ++e) out.v[e] = from_float<T>(to_float<S>(in.v[e]));
            reinterpret_cast<Vec8<T> *>(dst)[i] = out;
        }
        for (long long i = packets * 8 + first; i < n; i += stride) dst[i] = from_float<T>(to_float<S>(src[i]));
    }
}

// dst[i] = round(src[i] * scale): the float32 sums a backward pass left in its workspace, normalised
// and rounded into a 16-bit (or float32) gradient buffer.
template <typename T>
__global__ void __launch_bounds__(kOptThreads)
scale_cast_kernel(const float *__restrict__ src, T *__restrict__ dst, long long n, float scale) {
    for (long long i = static_cast<long long>(blockIdx.x) * blockDim.x + threadIdx.x; i < n;
         i += static_cast<long long>(gridDim.x) * blockDim.x)
        dst[i] = from_float<T>(src[i] * scale);
}

unsigned stream_grid(long long n, int packet = 8, int per_sm = 8) {
    const long long blocks = (n / packet + kOptThreads - 1) / kOptThreads + 1;
    const long long cap = static_cast<long long>(sm_count()) * per_sm;
    return static_cast<unsigned>(blocks < cap ? blocks : cap);
}

}  // namespace
}  // namespace th

using namespace th;

extern "C" int th_mse_grad(const void *pred_dev, const void *target_dev, void *grad_dev, float *loss_sum_dev,
                           int64_t n_elems, float grad_scale, int dtype, void *stream) {
    if (n_elems < 0) return fail(TH_ERR_BAD_ARG, "negative element count");
    if (n_elems == 0) return TH_OK;
    if (!pred_dev || !target_dev || !grad_dev) return fail(TH_ERR_BAD_ARG, "null tensor pointer");
    if (!aligned_to(pred_dev, 32) || !aligned_to(target_dev, 32) || !aligned_to(grad_dev, 32))
        return fail(TH_ERR_ALIGNMENT, "tensors must be 32-byte aligned");
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    const unsigned grid = stream_grid(n_elems);
    switch (dtype) {
        case TH_F32:
            mse_grad_kernel<float><<<grid, kOptThreads, 0, st>>>(static_cast<const float *>(pred_dev), static_cast<const float *>(target_dev),
                                                                  static_cast<float *>(grad_dev), loss_sum_dev, n_elems, grad_scale);
            break;
        case TH_F16:
            mse_grad_kernel<__half><<<grid, kOptThreads, 0, st>>>(static_cast<const __half *>(pred_dev), static_cast<const __half *>(target_dev),
                                                                   static_cast<__half *>(grad_dev), loss_sum_dev, n_elems, grad_scale);
            break;
        case TH_BF16:
            mse_grad_kernel<__nv_bfloat16><<<grid, kOptThreads, 0, st>>>(static_cast<const __nv_bfloat16 *>(pred_dev), static_cast<const __nv_bfloat16 *>(target_dev),
                                                                          static_cast<__nv_bfloat16 *>(grad_dev), loss_sum_dev, n_elems, grad_scale);
            break;
        default: return fail(TH_ERR_BAD_ARG, "unknown dtype %d", dtype);
    }
    return launch_status("mse_grad_kernel launch");
}

extern "C" int th_adam_steps(int n_tensors, void *const *param_dev, void *const *grad_dev, float *const *exp_avg_dev,
                             float *const *exp_avg_sq_dev, const int64_t *n_elems, const float *grad_scale, const int *zero_grad, float lr,
                             float beta1, float beta2, float eps, int step, int dtype, int *skipped_dev, void *stream) {
    if (n_tensors < 0 || n_tensors > kMaxTensors) return fail(TH_ERR_BAD_ARG, "%d tensors outside [0, %d]", n_tensors, kMaxTensors);
    if (step < 1) return fail(TH_ERR_BAD_ARG, "step counts from 1");
    AdamTensors t{};
    long long most = 0;
    for (int k = 0; k < n_tensors; ++k) {
        if (n_elems[k] < 0) return fail(TH_ERR_BAD_ARG, "negative element count");
        if (n_elems[k] == 0) continue;
        if (!param_dev[k] || !grad_dev[k] || !exp_avg_dev[k] || !exp_avg_sq_dev[k]) return fail(TH_ERR_BAD_ARG, "null tensor pointer");
        if (!aligned_to(param_dev[k], 32) || !aligned_to(grad_dev[k], 32) || !aligned_to(exp_avg_dev[k], 32) || !aligned_to(exp_avg_sq_dev[k], 32))
            return fail(TH_ERR_ALIGNMENT, "tensors must be 32-byte aligned");
        t.param[t.count] = param_dev[k];
        t.grad[t.count] = grad_dev[k];
        t.exp_avg[t.count] = exp_avg_dev[k];
        t.exp_avg_sq[t.count] = exp_avg_sq_dev[k];
        t.n[t.count] = n_elems[k];
        t.grad_scale[t.count] = grad_scale[k];
        t.zero_grad[t.count++] = zero_grad[k];
        most = n_elems[k] > most ? n_elems[k] : most;
    }
    if (t.count == 0) return TH_OK;
    AdamScalars a{lr, beta1, beta2, eps, 0.f, 0.f, 1.f, 0};
    a.bias1 = static_cast<float>(1.0 - pow(static_cast<double>(beta1), step));
    a.bias2_sqrt = static_cast<float>(sqrt(1.0 - pow(static_cast<double>(beta2), step)));
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    const unsigned grid = dtype == TH_F32 ? stream_grid(most, 4, 24) : stream_grid(most);
    switch (dtype) {
        case TH_F32: adam_many_kernel<float><<<grid, kOptThreads, 0, st>>>(t, a, skipped_dev); break;
        case TH_F16: adam_many_kernel<__half><<<grid, kOptThreads, 0, st>>>(t, a, skipped_dev); break;
        case TH_BF16: adam_many_kernel<__nv_bfloat16><<<grid, kOptThreads, 0, st>>>(t, a, skipped_dev); break;
        default: return fail(TH_ERR_BAD_ARG, "unknown dtype %d", dtype);
    }
    return launch_status("adam_many_kernel launch");
}

extern "C" int th_adam_step(void *param_dev, void *grad_dev, float *exp_avg_dev, float *exp_avg_sq_dev, int64_t n_elems,
                            float lr, float beta1, float beta2, float eps, int step, float grad_scale, int zero_grad,
                            int dtype, int *skipped_dev, void *stream) {
    return th_adam_steps(1, &param_dev, &grad_dev, &exp_avg_dev, &exp_avg_sq_dev, &n_elems, &grad_scale, &zero_grad, lr, beta1, beta2, eps, step,
                         dtype, skipped_dev, stream);
}

extern "C" int th_cast(int n_tensors, const void *const *src_dev, void *const *dst_dev, const int64_t *n_elems, int src_dtype, int dst_dtype,
                       void *stream) {
    if (n_tensors < 0 || n_tensors > kMaxTensors) return fail(TH_ERR_BAD_ARG, "%d tensors outside [0, %d]", n_tensors, kMaxTensors);
    if ((src_dtype == TH_F32) == (dst_dtype == TH_F32)) return fail(TH_ERR_BAD_ARG, "one side of a cast is float32");
    CastTensors t{};
    long long most = 0;
    for (int k = 0; k < n_tensors; ++k) {
        if (n_elems[k] < 0) return fail(TH_ERR_BAD_ARG, "negative element count");
        if (n_elems[k] == 0) continue;
        if (!src_dev[k] || !dst_dev[k]) return fail(TH_ERR_BAD_ARG, "null tensor pointer");
        t.src[t.count] = src_dev[k];
        t.dst[t.count] = dst_dev[k];
        t.n[t.count++] = n_elems[k];
        most = n_elems[k] > most ? n_elems[k] : most;
    }
    if (t.count == 0) return TH_OK;
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    const unsigned grid = stream_grid(most);
    switch (src_dtype * 4 + dst_dtype) {
        case TH_F32 * 4 + TH_F16: cast_many_kernel<float, __half><<<grid, kOptThreads, 0, st>>>(t); break;
        case TH_F32 * 4 + TH_BF16: cast_many_kernel<float, __nv_bfloat16><<<grid, kOptThreads, 0, st>>>(t); break;
        case TH_F16 * 4 + TH_F32: cast_many_kernel<__half, float><<<grid, kOptThreads, 0, st>>>(t); break;
        case TH_BF16 * 4 + TH_F32: cast_many_kernel<__nv_bfloat16, float><<<grid, kOptThreads, 0, st>>>(t); break;
        default: return fail(TH_ERR_BAD_ARG, "unknown dtypes %d, %d", src_dtype, dst_dtype);
    }
    return launch_status("cast_many_kernel launch");
}

extern "C" int th_scale_cast(const float *src_dev, void *dst_dev, int64_t n_elems, float scale, int dtype, void *stream) {
    if (n_elems < 0) return fail(TH_ERR_BAD_ARG, "negative element count");
    if (n_elems == 0) return TH_OK;
    if (!src_dev || !dst_dev) return fail(TH_ERR_BAD_ARG, "null tensor pointer");
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    const long long blocks = (n_elems + kOptThreads - 1) / kOptThreads;
    const long long cap = static_cast<long long>(sm_count()) * 8;
    const unsigned grid = static_cast<unsigned>(blocks < cap ? blocks : cap);
    switch (dtype) {
        case TH_F32: scale_cast_kernel<float><<<grid, kOptThreads, 0, st>>>(src_dev, static_cast<float *>(dst_dev), n_elems, scale); break;
        case TH_F16: scale_cast_kernel<__half><<<grid, kOptThreads, 0, st>>>(src_dev, static_cast<__half *>(dst_dev), n_elems, scale); break;
        case TH_BF16: scale_cast_kernel<__nv_bfloat16><<<grid, kOptThreads, 0, st>>>(src_dev, static_cast<__nv_bfloat16 *>(dst_dev), n_elems, scale); break;
        default: return fail(TH_ERR_BAD_ARG, "unknown dtype %d", dtype);
    }
    return launch_status("scale_cast_kernel launch");
}
