// What the block-compression kernels share: the description of the source mip and of the block
// rectangle, and the texel loads (block_compress.cu: BC1 - BC5; block_compress_bc7.cu: BC7).
#pragma once

#include <cuda_fp16.h>
#include <stdint.h>

#include "ntcb.h"

namespace ntcb
{

struct BlockCompressArguments
{
    const __half* texels;
    int layout, width, height, channels, firstChannel;
    int srcLeft, srcTop, widthInBlocks, heightInBlocks, formatChannels;
    bool pairs; // see ChannelPairs
    uint8_t* blocks;
    size_t rowPitch;
};

// Whether channel firstChannel and those two, four ... after it can be loaded with the next one as an aligned 32-bit word (LoadPair): in
// both layouts when the mip starts on such a word, the channel is even and so is their count.  `texels` may be any address of halves.
inline bool ChannelPairs(const BlockCompressArguments& args)
{
    return !(reinterpret_cast<uintptr_t>(args.texels) & 3) && !(args.firstChannel & 1) && !(args.channels & 1);
}

// Whether a texel lies inside the mip.  (Unsigned: a position that has passed 2^31 - a window far outside - counts as outside.)
__device__ __forceinline__ bool Inside(const BlockCompressArguments& args, int x, int y)
{
    return unsigned(x) < unsigned(args.width) && unsigned(y) < unsigned(args.height);
}

__device__ __forceinline__ __half LoadHalf(const BlockCompressArguments& args, int x, int y, int channel)
{
    const size_t w = size_t(args.width), c = size_t(args.channels);
    const size_t index = args.layout == NTCB_LAYOUT_INTERLEAVED
        ? (size_t(y) * w + size_t(x)) * c + size_t(channel)
        : size_t(y) * w * c + size_t(channel & ~1) * w + 2 * size_t(x) + size_t(channel & 1);
    return args.texels[index];
}

// Channels `channel` and `channel + 1` of one texel as one word (args.pairs).
__device__ __forceinline__ uint32_t LoadPair(const BlockCompressArguments& args, int x, int y, int channel)
{
    const size_t w = size_t(args.width), c = size_t(args.channels);
    const size_t index = args.layout == NTCB_LAYOUT_INTERLEAVED ? (size_t(y) * w + size_t(x)) * c + size_t(channel)
                                                                 : size_t(y) * w * c + size_t(channel) * w + 2 * size_t(x);
    return *reinterpret_cast<const uint32_t*>(args.texels + index);
}

// Sixteen indices of kBits bits, one per nibble, moved together (a loop over the pixels with a 64-bit shift each cost more
// than finding the indices).
template <int kBits>
__device__ __forceinline__ uint64_t JoinIndices(uint64_t x)
{
    if (kBits == 4)
        return x;
    constexpr int kGap = 4 - kBits; // every step joins two fields, whose gap doubles
    constexpr uint64_t kField = (1u << kBits) - 1u;
    constexpr uint64_t kNibbles = kField * 0x0101010101010101ull;
    x = (x & kNibbles) | ((x >> kGap) & (kNibbles << kBits));
    constexpr uint64_t kBytes = ((1u << (2 * kBits)) - 1u) * 0x0001000100010001ull;
    x = (x & kBytes) | ((x >> (2 * kGap)) & (kBytes << (2 * kBits)));
    constexpr uint64_t kShorts = ((1u << (4 * kBits)) - 1u) * 0x0000000100000001ull;
    x = (x & kShorts) | ((x >> (4 * kGap)) & (kShorts << (4 * kBits)));
    constexpr uint64_t kWord = (1ull << (8 * kBits)) - 1ull;
    return (x & kWord) | ((x >> (8 * kGap)) & (kWord << (8 * kBits)));
}

// Calls launch(part, first row of blocks, grid) for the block rectangle in rows of as many CTAs of `width` x `height` blocks as a grid may have
// (an image of a million and more texel rows takes several launches).
template <typename Launch>
inline void ForEachGrid(const BlockCompressArguments& args, int width, int height, Launch&& launch)
{
    for (int top = 0, rows = 0; top < args.heightInBlocks; top += rows)
    {
        rows = args.heightInBlocks - top < 65535 * height ? args.heightInBlocks - top : 65535 * height;
        BlockCompressArguments part = args;
        part.srcTop = args.srcTop + 4 * top;
        part.heightInBlocks = rows;
        part.blocks = args.blocks + size_t(top) * args.rowPitch;
        launch(part, top, dim3(unsigned(part.widthInBlocks + width - 1) / width, unsigned(part.heightInBlocks + height - 1) / height));
    }
}

// The BC7 half of ntcb_block_compress (block_compress_bc7.cu); `params` has passed the checks common to all formats.
int LaunchBlockCompressBc7(const NtcbBlockCompressParams& params, const BlockCompressArguments& args, cudaStream_t stream);

} // namespace ntcb
