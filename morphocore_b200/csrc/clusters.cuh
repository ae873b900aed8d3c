// Thread block clusters whose members divide the input channels of a tile.
#pragma once
#include <algorithm>

#include "common.cuh"
#include "shares.cuh"

namespace mc
{

/// Barrier over the thread blocks of a cluster: what they wrote to shared memory before it is visible to the others after it.
__device__ __forceinline__ void cluster_sync()
{
    asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}
/// Reads of the shared memory of the cluster's block `rank`, at the place that `address` has in the reader's own.
__device__ __forceinline__ float4 load_cluster_float4(uint32_t address, int rank)
{
    float4 v;
    asm volatile("{\n\t.reg .b32 a;\n\tmapa.shared::cluster.u32 a, %4, %5;\n\tld.shared::cluster.v4.f32 {%0, %1, %2, %3}, [a];\n\t}"
                 : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "r"(address), "r"(rank) : "memory");
    return v;
}
template <typename T> __device__ __forceinline__ T load_cluster(uint32_t address, int rank)
{
    T v;
    if constexpr (sizeof(T) == 4)
        asm volatile("{\n\t.reg .b32 a;\n\tmapa.shared::cluster.u32 a, %1, %2;\n\tld.shared::cluster.f32 %0, [a];\n\t}"
                     : "=f"(v) : "r"(address), "r"(rank) : "memory");
    else
        asm volatile("{\n\t.reg .b32 a;\n\tmapa.shared::cluster.u32 a, %1, %2;\n\tld.shared::cluster.f64 %0, [a];\n\t}"
                     : "=d"(v) : "r"(address), "r"(rank) : "memory");
    return v;
}

/// CTAs of a cluster that divide the input channels of an item (a tile and a group of output channels) in the smorph forward
/// kernels: the fewest waves of `per_sm` CTAs per SM, each as long as the channels a CTA walks plus its fixed work (barriers,
/// first copy, the exchange of the sums) in units of one channel. 3 x 3, 32 items of 28 x 28 maps with 8 channels: 20.9 us with
/// one CTA an item, 14.4 with a cluster; one 224 x 224 image, 64 -> 64 channels (448 items on 296 places): 515 and 465 us;
/// 5 x 5 on (4, 16, 96, 96) -> 16: 120 and 90 us.
inline int cluster_size(int64_t items, int channels, int per_sm)
{
    constexpr int MOST = 8;
    const int64_t places = 148 * per_sm;
    int best = 1;
    double best_cost = 0.0;
    for (int s = 1; s <= std::min(channels, MOST) && items * s <= 0x7fffffffLL; s++)
    {
        const double cost = static_cast<double>((items * s + places - 1) / places) * ((channels + s - 1) / s + (s == 1 ? 1.0 : 2.0));
        if (s == 1 || cost < 0.95 * best_cost)
        {
            best = s;
            best_cost = cost;
        }
    }
    return best;
}

/// Launches `items` clusters of `cluster` thread blocks.
template <typename Kernel, typename... Args>
inline int launch_clusters(Kernel kernel, int cluster, int64_t items, size_t smem, cudaStream_t stream, const char* name, const Args&... args)
{
    cudaLaunchAttribute attribute{};
    attribute.id = cudaLaunchAttributeClusterDimension;
    attribute.val.clusterDim.x = static_cast<unsigned>(cluster);
    attribute.val.clusterDim.y = attribute.val.clusterDim.z = 1;
    cudaLaunchConfig_t config{};
    config.gridDim = dim3(static_cast<unsigned>(items * cluster));
    config.blockDim = dim3(THREADS);
    config.dynamicSmemBytes = smem;
    config.stream = stream;
    config.attrs = &attribute;
    config.numAttrs = cluster > 1 ? 1 : 0;
    cudaLaunchKernelEx(&config, kernel, args...);
    return check_launch(name);
}

}  // namespace mc
