// The single-view backprojector's walk: the shared address of the channel after
// the one numbered by the bits of a float near 1.5 * 2^23 (built for the host by
// tests/cpp/sv_walk_check.cc).  `at0` is the address less that of the number
// itself, so that the sum wraps around to the channel's: unsigned throughout.
#pragma once

#if defined(__CUDACC__)
#define CTR_SV_HD __host__ __device__ __forceinline__
#else
#define CTR_SV_HD inline
#endif

namespace ctr {

constexpr unsigned kSvMagicBits = 0x4B400000u;  // of 1.5 * 2^23

// at: the row's first channel; i: the channel before the reference position (its
// successor for a walk downwards); dir4: bytes to the next channel, 4 or -4.
CTR_SV_HD unsigned sv_base(unsigned at, int i, int dir4)
{
    const unsigned d = static_cast<unsigned>(dir4);
    return at + 4u * static_cast<unsigned>(i) + d - kSvMagicBits * d;
}
CTR_SV_HD unsigned sv_address(unsigned at0, int num, int dir4)
{
    return at0 + static_cast<unsigned>(num) * static_cast<unsigned>(dir4);
}

}  // namespace ctr
