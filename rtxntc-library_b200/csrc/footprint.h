// Runs of tiles and their footprints: how many latent pixels one can touch, and whether its buffers in shared memory hold them.
#pragma once

#include <stdint.h>

namespace ntcb
{

constexpr int kChainTileWidth = 16;
constexpr int kChainTileHeight = 8;
constexpr int kMaxRunTiles = 4; // tiles of a run, see KernelMip::runTiles

// Shared memory of a chain for the latents of a run of tiles, in the high-res and the low-res grid, and what a latent pixel takes of it: eight bytes per
// layer, either side by side without gaps, where two layers of a tap are one load of 16 bytes (GatherTexel), or padded to an odd multiple of eight, so
// that 8-byte loads of neighbouring pixels fall into different banks.
// Wide loads are taken where they pay: 16 features, Int8, 2048 x 2048, 228.5 us instead of 231.1, 1920 x 1080 at a grid of a half 139.6 instead of
// 142.7; 8 features, FP8, 143.5 instead of 145.1, at a half 153.7 instead of 157.6.  With 16 features and FP8 weights (166.9 instead of 161.7) or with exact
// accumulation (8 features 256 instead of 249, 16 features 288 instead of 279) the kernels run out of registers.
struct FootprintBuffers
{
    int hiBytes, loBytes;
    int pixelBytes[5]; // by layers
};
// What a tile covers at a grid-to-mip ratio of 1 (high-res: 18 x 10 pixels of 24 bytes) and 1/2 (low-res: 10 x 6), or a run of tiles at a smaller
// one.  The FP8 kernels have room for runs of two at a ratio of 1 with two latent layers (34 x 10 pixels of 16 bytes), and of four at 1/2 with three
// (34 x 6 of 24) or at 1/3 with four (24 x 5 of 40).  (With the Int8 kernels' buffers: 1920 x 1080, 8 features at scale 1, 101.3 us instead of 93.8; 3000 x 2000, 12
// features at scale 2, 262 instead of 253, 16 features at scale 3, 284 instead of 261.)
inline constexpr FootprintBuffers kRefFp8Footprint{5440, 2080, {0, 8, 16, 24, 40}};
inline constexpr FootprintBuffers kRefInt8Footprint{4352, 1440, {0, 8, 16, 24, 32}}; // (all that the CTA has left)
// The exact-accumulation kernels have room for a tile at a ratio of 4/5 with four latent layers (15 x 8 pixels of 40 bytes, 9 x 5).  (With the FP8
// kernels' buffers mips at 4/5 and 2/3 were read tap by tap: mip 1 of a 3000 x 4000 Int8 set of 16 features at scale 3 took 224 us, now
// 196, FP8 162 and 135; mip 2 of 4096 x 4096 at scale 5 79.5 and 72.6.  With 6144 and 2432 bytes more runs would be longer, some for the worse:
// 3000 x 2000 Int8, 12 features, 445 and 455 us.)
inline constexpr FootprintBuffers kExactFootprint{4800, 1808, {0, 8, 24, 24, 40}};

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
    // (span + extent * units / 2^24) * grid / extent, where `units` is what both positions may be off, in 2^-24 of the grid
    if (grid <= (1 << 22) && extent <= (1 << 22))
        return (long long)grid * (((long long)span << 24) + (long long)extent * 10) / ((long long)extent << 24) + 3; // (below 2^53)
    return (long long)((__int128)grid * (((long long)span << 24) + (long long)extent * 20) / ((long long)extent << 24)) + 3;
}

// Tiles side by side, a power of two up to `most`, whose footprints in both grids fit the buffers; 0: not even those of one do, and texels read their
// taps from global memory, as they do where a footprint has more pixels than its texels have taps.  (Mip 1 of a 4096 x 4096 set of 4 features at
// scale 1, 33 x 17 pixels for 128 texels, exact accumulation: staged 301 us Int8 and 233 FP8, read directly 237 and 167.)  A run is no longer than its
// mip is wide.
constexpr int StagedTiles(int hiWidth, int hiHeight, int loWidth, int loHeight, int width, int height, int pixelBytes, FootprintBuffers buffers,
    int most)
{
    int tiles = 0;
    for (int next = 1; next <= most && (next == 1 || (next / 2) * kChainTileWidth < width); next *= 2)
    {
        const int columns = next * kChainTileWidth - 1, rows = kChainTileHeight - 1;
        const long long hiPixels = FootprintPixels(hiWidth, width, columns) * FootprintPixels(hiHeight, height, rows);
        if (hiPixels > 4 * next * kChainTileWidth * kChainTileHeight || hiPixels > buffers.hiBytes / pixelBytes ||
            FootprintPixels(loWidth, width, columns) * FootprintPixels(loHeight, height, rows) > buffers.loBytes / pixelBytes)
            break;
        tiles = next;
    }
    return tiles;
}

} // namespace ntcb
