// Which channels and linear pieces of a view the distance-driven grad's tiles
// stage, shared by the kernel and its host check (tests/cpp/dd_window_check.cc).
// A tile's positions lie within `e` channels of the window's centre channel, a
// footprint reaches `reach` channels to either side.
#pragma once

#if defined(__CUDACC__)
#define CTR_DD_HD __host__ __device__ __forceinline__
#else
#define CTR_DD_HD inline
#endif

namespace ctr {

constexpr int kDgHalf = 64;  // channels staged on either side of the window's centre

// Tiles with a larger window go pixel by pixel.
CTR_DD_HD bool dg_fits(float e, float reach) { return e + reach < kDgHalf - 3; }
// Channels staged on either side.
CTR_DD_HD int dg_need(float e, float reach) { return static_cast<int>(e + reach) + 2; }
// Whole channels between a footprint's ends: a piece i is formed from the
// staged channels i - m .. i + 1 (channel 0 is kDgHalf before the centre).
// `two`: twice the reach, 32.32 fixed point.
CTR_DD_HD int dg_spread(long long two)
{
    const long long m = two >> 32;
    return static_cast<int>(m < 2 * kDgHalf ? m : 2 * kDgHalf);
}
// Pieces are formed from here to kDgHalf + need - 1: the ones before are past
// no tile's position, and would read in front of the channels.
CTR_DD_HD int dg_first_piece(int need, int m) { return kDgHalf - need > m ? kDgHalf - need : m; }

}  // namespace ctr
