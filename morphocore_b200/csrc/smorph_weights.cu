// Small kernels around the smorph and dilation / erosion kernels: the re-parametrisation of smorph's structuring element
// with its gradient, and the zeroing of gradient buffers. All are bound by launch latency at the sizes that occur (a
// structuring element of 64 x 64 x 11 x 11 is 2 MB): what counts is that each is one launch.
#include "zero.cuh"

namespace mc
{

namespace
{

struct ZeroArgs
{
    ZeroRange range[4];
};

__global__ void __launch_bounds__(THREADS) zero_kernel(const ZeroArgs a)
{
    const ZeroRange r = a.range[blockIdx.y];
    const size_t first = static_cast<size_t>(blockIdx.x) * THREADS + threadIdx.x, step = static_cast<size_t>(gridDim.x) * THREADS;
    size_t done = 0;
    if (reinterpret_cast<uintptr_t>(r.p) % 16 == 0)
    {
        const size_t vectors = r.bytes / 16;
        for (size_t i = first; i < vectors; i += step) static_cast<uint4*>(r.p)[i] = make_uint4(0u, 0u, 0u, 0u);
        done = vectors * 4;
    }
    for (size_t i = done + first; i < r.bytes / 4; i += step) static_cast<uint32_t*>(r.p)[i] = 0u;
}

__device__ __forceinline__ float tanh_of(float v) { return tanhf(v); }
__device__ __forceinline__ double tanh_of(double v) { return tanh(v); }

/// w~ = t * ((1 - t) / 2 * flip(w) + (1 + t) / 2 * w), t = tanh(alpha of the pair): one thread per element.
template <typename T>
__global__ void __launch_bounds__(THREADS) reparametrise_kernel(const T* __restrict__ w, const T* __restrict__ alpha, T* __restrict__ out, int taps, int64_t n)
{
    for (int64_t e = static_cast<int64_t>(blockIdx.x) * THREADS + threadIdx.x; e < n; e += static_cast<int64_t>(gridDim.x) * THREADS)
    {
        const int64_t pair = e / taps;
        const int k = static_cast<int>(e - pair * taps);
        const T t = tanh_of(__ldg(alpha + pair));
        const T straight = (T(1) + t) * T(0.5), mirrored = (T(1) - t) * T(0.5);
        out[e] = t * (mirrored * __ldg(w + pair * taps + taps - 1 - k) + straight * __ldg(w + e));
    }
}

/// Gradient of the above: with G the gradient of w~ and s_k = (1 - t) / 2 w[flip k] + (1 + t) / 2 w[k],
///   grad w[k]   = t (1 + t) / 2 G[k] + t (1 - t) / 2 G[flip k]
///   grad alpha += (1 - t^2) sum_k G[k] (s_k + t (w[k] - w[flip k]) / 2),
/// the sum over k also for the alpha gradient the kernel already holds (that of the operator itself). One warp per pair.
template <typename T>
__global__ void __launch_bounds__(THREADS) reparametrise_backward_kernel(const T* __restrict__ w, const T* __restrict__ alpha, const T* __restrict__ grad,
                                                                         T* __restrict__ gw, T* __restrict__ galpha, int taps, int64_t pairs)
{
    const int lane = threadIdx.x & 31;
    const int64_t warps = static_cast<int64_t>(gridDim.x) * (THREADS / 32);
    for (int64_t pair = static_cast<int64_t>(blockIdx.x) * (THREADS / 32) + (threadIdx.x >> 5); pair < pairs; pair += warps)
    {
        const T t = tanh_of(__ldg(alpha + pair));
        const T straight = (T(1) + t) * T(0.5), mirrored = (T(1) - t) * T(0.5);
        const T *wp = w + pair * taps, *gp = grad + pair * taps;
        T sum = T(0);
        for (int k = lane; k < taps; k += 32)
        {
            const T wk = __ldg(wp + k), wf = __ldg(wp + taps - 1 - k), gk = __ldg(gp + k), gf = __ldg(gp + taps - 1 - k);
            gw[pair * taps + k] = t * (straight * gk + mirrored * gf);
            sum += gk * (mirrored * wf + straight * wk + t * T(0.5) * (wk - wf));
        }
#pragma unroll
        for (int d = 16; d > 0; d >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, d);
        if (lane == 0) galpha[pair] += (T(1) - t * t) * sum;
    }
}

/// Buffers above this size are zeroed by a memset of their own: on 35 MB it takes 7.1 us where the kernel takes 14.2, on
/// 4.7 MB the one launch for all buffers still wins (3.4 us against 2.1 + 1.3 us and a launch more).
constexpr size_t MEMSET_FROM = 6u << 20;

unsigned blocks_for(int64_t items, int64_t per_block) { return static_cast<unsigned>(std::min<int64_t>((items + per_block - 1) / per_block, 148 * 16)); }

}  // namespace

int zero_buffers(std::initializer_list<ZeroRange> ranges, cudaStream_t stream)
{
    ZeroArgs a{};
    unsigned count = 0;
    size_t most = 0;
    for (const ZeroRange& r : ranges)
    {
        if (r.bytes == 0) continue;
        if (r.bytes > MEMSET_FROM)
        {
            const cudaError_t err = cudaMemsetAsync(r.p, 0, r.bytes, stream);
            if (err != cudaSuccess)
            {
                set_last_error("cudaMemsetAsync: %s", cudaGetErrorString(err));
                return MC_ERR_CUDA;
            }
            continue;
        }
        a.range[count++] = r;
        most = std::max(most, r.bytes);
    }
    if (count == 0) return MC_OK;
    zero_kernel<<<dim3(blocks_for(static_cast<int64_t>(most / 16 + 1), 4 * THREADS), count), THREADS, 0, stream>>>(a);
    return check_launch("zero_kernel");
}

template <typename T> int smorph_reparametrise(const mc_desc& d, const T* w, const T* alpha, T* out, cudaStream_t stream)
{
    const int taps = d.kH * d.kW;
    const int64_t n = static_cast<int64_t>(d.Co) * (d.merge == MC_MERGE_IDENTITY ? 1 : d.Ci) * taps;
    reparametrise_kernel<T><<<blocks_for(n, THREADS), THREADS, 0, stream>>>(w, alpha, out, taps, n);
    return check_launch("reparametrise_kernel");
}

template <typename T> int smorph_reparametrise_backward(const mc_desc& d, const T* w, const T* alpha, const T* grad, T* gw, T* galpha, cudaStream_t stream)
{
    const int64_t pairs = static_cast<int64_t>(d.Co) * (d.merge == MC_MERGE_IDENTITY ? 1 : d.Ci);
    reparametrise_backward_kernel<T><<<blocks_for(pairs, THREADS / 32), THREADS, 0, stream>>>(w, alpha, grad, gw, galpha, d.kH * d.kW, pairs);
    return check_launch("reparametrise_backward_kernel");
}

template int smorph_reparametrise<float>(const mc_desc&, const float*, const float*, float*, cudaStream_t);
template int smorph_reparametrise<double>(const mc_desc&, const double*, const double*, double*, cudaStream_t);
template int smorph_reparametrise_backward<float>(const mc_desc&, const float*, const float*, const float*, float*, float*, cudaStream_t);
template int smorph_reparametrise_backward<double>(const mc_desc&, const double*, const double*, const double*, double*, double*, cudaStream_t);

}  // namespace mc
