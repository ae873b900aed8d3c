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
/// units of one channel. Its constants were fitted to the backward kernels of dilation and erosion (20 to 592 tiles, 2 to 21
/// channels, up to 16 shares):
///   - `alone`: time of one block on each of the 148 SMs, of that of two on each, measured 0.65 - 0.8. A higher figure divides
///     more often: 0.7 is 3 % faster over the float kernels that compute four channels together, but loses up to 18 % against one
///     share in the 5 x 5 kernel, where 0.6 loses nowhere more than 2 %;
///   - `group`: a kernel that computes that many channels together saves little where some of them do not exist. Two of four
///     cost 0.73 (7 x 7), 0.88 (9 x 9) and 0.89 (11 x 11) of four, one of two in double 0.8. With partial groups at their
///     channels' price 104 tiles of four channels became two shares of two: 71.0 against 53.6 us at 9 x 9, 81.1 against 63.5 at
///     11 x 11. Shares of whole groups only lose as well (12 channels on 20 tiles at 9 x 9: 59.4 us, two channels a share 51.2).
inline int channel_shares(int64_t blocks, int channels, int per_sm, int fixed, int group = 1, double alone = 0.6)
{
    constexpr int SMS = 148, MOST = 16;
    constexpr double PARTIAL = 0.75;   // of a group's price that its first channel costs
    int best = 1;
    double best_cost = 0.0;
    for (int s = 1; s <= std::min(channels, MOST) && blocks * s <= 0x7fffffffLL; s++)
    {
        const int64_t n = blocks * s;
        const int64_t places = static_cast<int64_t>(SMS) * per_sm, rest = n % places;
        double last = rest == 0 ? 0.0 : 1.0;
        if (rest > 0 && per_sm > 1) last = rest <= SMS ? alone : alone + (1.0 - alone) * static_cast<double>(rest - SMS) / static_cast<double>(places - SMS);
        const double waves = static_cast<double>(n / places) + last;
        const int most = (channels + s - 1) / s, partial = most % group;   // channels of the largest share, and of its last group
        const double work = most - partial + (partial == 0 ? 0.0 : PARTIAL * group + (1.0 - PARTIAL) * partial);
        const double cost = waves * (work + fixed);
        if (s == 1 || cost < 0.97 * best_cost)
        {
            best = s;
            best_cost = cost;
        }
    }
    return best;
}

}  // namespace mc
