// How many latent pixels a run of texels can touch: what decides whether its footprint fits a staging buffer.
#pragma once

#include <stdint.h>

namespace ntcb
{

// Most latent pixels, of a grid of `grid` pixels, that texels x .. x + span of an axis of `extent` texels read: the last tap's index minus
// the first's, plus the second tap of each end.
//
// The positions of the first and the last texel are span * grid / extent apart, so their floors differ by at most that, rounded down, plus 1.
// But the kernels work the positions out in binary32 (AxisTap), and each may be off by the roundings of the coordinate (at most 2 ulp of an
// approximate division: 4 * 2^-24 of it) and of the multiply-add (2^-24 of the position), together 5 * 2^-24 * grid.  From 2^22 texels or latent
// pixels on the conversions and the half that is added round too (at most 4 * 2^-24 more).  (Without that term the bound of a
// 23953-wide mip over a grid of 7984 was 7 columns where some tiles have 8: their last pixels were staged past the buffer.)
constexpr long long FootprintPixels(int grid, int extent, int span)
{
    const long long units = grid > (1 << 22) || extent > (1 << 22) ? 20 : 10; // both positions, in 2^-24 of the grid
    // (span + extent * units / 2^24) * grid / extent
    const long long slack = (long long)extent * units;
    return (long long)((__int128)grid * (((long long)span << 24) + slack) / ((long long)extent << 24)) + 3;
}

} // namespace ntcb
