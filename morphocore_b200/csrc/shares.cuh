// Division of the channels of a tile among thread blocks.
#pragma once
#include <algorithm>
#include <cstdint>

namespace mc
{

/// First of `count` channels that belongs to share `i` of `n`.
__host__ __device__ __forceinline__ int share_begin(int count, int i, int n) { return static_cast<int>(static_cast<int64_t>(count) * i / n); }

/// In how many shares the output channels that a thread block would have to walk are divided among thread blocks. With one
/// share a small batch leaves SMs without a block, or a last wave nearly empty. The estimate counts waves of the `per_sm`
/// blocks an SM holds, times the channels a block walks plus its fixed work (staging its window, flushing its results) in
/// units of one channel; a block that has its SM to itself, in the last wave too, takes 0.6 of the time of one that shares it.
inline int channel_shares(int64_t blocks, int channels, int per_sm, int fixed)
{
    constexpr int SMS = 148, MOST = 16;
    int best = 1;
    double best_cost = 0.0;
    for (int s = 1; s <= std::min(channels, MOST) && blocks * s <= 0x7fffffffLL; s++)
    {
        const int64_t n = blocks * s;
        const int64_t places = static_cast<int64_t>(SMS) * per_sm, rest = n % places;
        double last = rest == 0 ? 0.0 : 1.0;
        if (rest > 0 && per_sm > 1) last = rest <= SMS ? 0.6 : 0.6 + 0.4 * static_cast<double>(rest - SMS) / static_cast<double>(places - SMS);
        const double waves = static_cast<double>(n / places) + last;
        const double cost = waves * ((channels + s - 1) / s + fixed);
        if (s == 1 || cost < 0.97 * best_cost)
        {
            best = s;
            best_cost = cost;
        }
    }
    return best;
}

}  // namespace mc
