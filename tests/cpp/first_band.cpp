// Per line of standard input, `width height hostTexelBytes streamedBytes exact int8`: the rows of mip 0 that are decoded first.
#include <cstdio>

#include "../../rtxntc-library_b200/csrc/first_band.h"

int main()
{
    int width, height, exact, int8;
    size_t hostTexelBytes, streamedBytes;
    while (std::scanf("%d %d %zu %zu %d %d", &width, &height, &hostTexelBytes, &streamedBytes, &exact, &int8) == 6)
        std::printf("%d\n", ntcb::FirstBandRows(width, height, hostTexelBytes, streamedBytes, ntcb::DecodeRate(exact != 0, int8 != 0)));
    return 0;
}
