// How much of mip 0 a texture set decodes in a launch of its own, under the upload that is still under way or ahead of the host's copies.
#pragma once

#include <algorithm>
#include <stddef.h>

namespace ntcb
{

constexpr int kBandMinRows = 512;

// Texels a nanosecond that the kernels decode, as far as the split of a streamed upload cares.  Exact accumulation with Int8 weights is the slow one:
// a decompress of 2048 x 2048 (8 features at scale 1) takes 628 us at 18 and 657 at 27, its 8-bit pixels 655 and 685, 4096 x 4096
// (8 features at scale 2) 1335 and 1367.  The others decode 23 to 34, and 27 is as good for them as 22 or 34 (FP8, the same two sets: 561 and 974
// us, with 22 568 and 1002; Int8 in reference numerics 580 and 1069, 578 and 1081).
inline float DecodeRate(bool exactNumerics, bool int8Weights)
{
    return exactNumerics && int8Weights ? 18.f : 27.f;
}

// Rows of mip 0 that are decoded in a launch of their own, 0: none.
//
// For a host read of texels of `hostTexelBytes` bytes (0: the texels stay on the device): copying the first band should take
// as long as decoding everything else does, so that the copies never wait again.  The kernels decode about 20 Gtexel/s, the
// host link takes about 57 GB/s: copying a texel of n bytes takes 0.35 n times as long as decoding it, and the band's share of
// the work is 1 / (1 + 0.35 n).  (Four equal bands and the other mips apart took five launches, each with a ramp at both
// ends: 326 us for a 2048 x 2048 set that decodes in 250.)
//
// `streamedBytes`, an upload beside the decode (0: none): decoding the first band should take as long as the rest of the upload does, at
// `texelsPerNanosecond` and what many copies get of the host link.
inline int FirstBandRows(int width, int height, size_t hostTexelBytes, size_t streamedBytes, float texelsPerNanosecond)
{
    if (height < kBandMinRows)
        return 0;
    float share = hostTexelBytes ? 1.f / (1.f + 0.35f * float(hostTexelBytes)) : 0.f;
    if (streamedBytes)
    {
        const float upload = float(streamedBytes) / 50.f, decode = float(width) * float(height) / texelsPerNanosecond; // nanoseconds
        share = std::max(share, upload / (upload + decode));
    }
    return std::min(height, (int(float(height) * share) + 15) & ~15);
}

} // namespace ntcb
