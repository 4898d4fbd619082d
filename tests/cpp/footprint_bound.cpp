// Walks every run of tiles of the mips on standard input (lines of `extent grid`) with the kernels' binary32 tap arithmetic and prints the
// runs that read more latent pixels than FootprintPixels allows: `extent grid columns bound pixels`.
#include <algorithm>
#include <cmath>
#include <cstdio>

#include "../../rtxntc-library_b200/csrc/footprint.h"

// AxisTap: `ulps` is how far the quotient lies from the rounded one (an approximate division: up to 2).
static long long Tap(int texel, int extent, int grid, bool division, int ulps)
{
    const float centre = float(texel) + 0.5f;
    float u = division ? centre / float(extent) : centre * (1.0f / float(extent));
    for (; ulps > 0; --ulps)
        u = std::nextafterf(u, 2.0f);
    for (; ulps < 0; ++ulps)
        u = std::nextafterf(u, -1.0f);
    return (long long)std::floor(std::fmaf(u, float(grid), -0.5f));
}

int main()
{
    int extent, grid;
    while (std::scanf("%d %d", &extent, &grid) == 2)
        for (int columns : {8, 16, 32, 64}) // rows of a tile, columns of a run
        {
            long long most = 0;
            for (int x = 0; x < extent; x += columns)
            {
                const int last = std::min(x + columns, extent) - 1;
                most = std::max(most, Tap(last, extent, grid, false, 0) - Tap(x, extent, grid, false, 0) + 2);
                most = std::max(most, Tap(last, extent, grid, true, 2) - Tap(x, extent, grid, true, -2) + 2);
            }
            const long long bound = ntcb::FootprintPixels(grid, extent, columns - 1);
            if (most > bound)
                std::printf("%d %d %d %lld %lld\n", extent, grid, columns, bound, most);
        }
    return 0;
}
