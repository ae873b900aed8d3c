// Thread block clusters whose members divide the input channels of a tile.
#pragma once
#include <algorithm>

#include "common.cuh"
#include "shares.cuh"
#include "tma.cuh"

namespace mc
{

/// Barrier over the thread blocks of a cluster: what they wrote to shared memory before it is visible to the others after it.
__device__ __forceinline__ void cluster_sync()
{
    __syncwarp();   // .aligned: the warp arrives as one
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

// A wait on a copy that runs out must not keep the other CTAs of the cluster at its barriers. Threads time their waits one by
// one, and where the copy lands just then some of them give up and others do not: so the CTA decides as one (cta_gave_up), in
// place of the barrier that follows the wait, and then leaves the kernel as one (leave_cluster), through the same two cluster
// barriers as its peers, which learn of it at the first (cluster_complete) and store nothing.

__device__ __forceinline__ bool cta_gave_up(bool landed) { return __syncthreads_or(!landed) != 0; }

/// The barrier between writing the parts and merging them; true where every CTA of the cluster has written its own. `gave_up`:
/// a word of shared memory. A second cluster_sync follows when the parts have been read.
__device__ __forceinline__ bool cluster_complete(uint32_t* gave_up, int cluster)
{
    if (threadIdx.x == 0) *gave_up = 0;
    cluster_sync();
    const int rank = threadIdx.x & 31;
    uint32_t flag = 0;
    if (rank < cluster)
        asm volatile("{\n\t.reg .b32 a;\n\tmapa.shared::cluster.u32 a, %1, %2;\n\tld.shared::cluster.u32 %0, [a];\n\t}"
                     : "=r"(flag) : "r"(smem_addr(gave_up)), "r"(rank) : "memory");
    return !__any_sync(0xffffffffu, flag != 0);
}

/// What a CTA that gave up does instead of writing and merging parts; it returns afterwards. Thread 0 counts it and waits, once
/// more with a limit, for the `copies` copies still in flight (on barriers with copy n's on full[n & 1], from copy `first` on),
/// so that the shared memory they write is not given back before they have landed.
__device__ __forceinline__ void leave_cluster(uint32_t* gave_up, uint64_t* full, int first, int copies, unsigned int* errors, uint64_t limit_ns)
{
    if (threadIdx.x == 0) *gave_up = 1;
    cluster_sync();
    cluster_sync();
    if (threadIdx.x != 0) return;
    if (errors != nullptr) atomicAdd(errors, 1u);
    for (int n = first; n < first + copies; n++) mbar_wait(full + (n & 1), (n >> 1) & 1, limit_ns > 1000000000ull ? limit_ns : 1000000000ull);
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
