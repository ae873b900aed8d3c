// Zeroing of the gradient buffers that the backward kernels build up with atomic adds.
#pragma once
#include <initializer_list>

#include "common.cuh"

namespace mc
{

struct ZeroRange
{
    void* p;
    size_t bytes;   // a multiple of 4
};

/// Queues one kernel that zeroes up to four buffers, and a memset for a large one (a backward pass has two to four of them, most of a few KiB: a memset
/// each costs about 2 us of host time and 1.7 us of device time in a chain of dependent launches). MC_OK or MC_ERR_CUDA.
int zero_buffers(std::initializer_list<ZeroRange> ranges, cudaStream_t stream);

}  // namespace mc
