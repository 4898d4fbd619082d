// The converting epilogue of the decode kernels: the thread's decoded channels (eight binary16
// pairs) become the pixel in the client's channel format and are stored.  `Context` is the
// kernel's per-thread tile context: `out` is the address of the thread's pixel, `outStepWords` the
// pixel's linear index in its mip (the dither seed), `rowChunk` the thread's 16-byte slot in chunk 0
// of its chain's A operand (chunks are 2048 bytes apart).
#pragma once

#include <cuda_fp16.h>
#include <stdint.h>

#include "kernel_parts.cuh"
#include "output_convert.cuh"

namespace ntcb
{
namespace
{

// Stores `bytes` bytes of a pixel held in `words` (little endian) at `pixel`, whose address and
// size are both multiples of the widest store used.
template <int kMaxWords>
__device__ __forceinline__ void StorePixel(unsigned char* pixel, const uint32_t (&words)[kMaxWords], int bytes)
{
    if ((bytes & 15) == 0 && kMaxWords >= 4)
    {
#pragma unroll
        for (int w = 0; w + 3 < kMaxWords; w += 4)
            if (w * 4 < bytes)
                *reinterpret_cast<uint4*>(pixel + w * 4) = make_uint4(words[w], words[w + 1], words[w + 2], words[w + 3]);
    }
    else if ((bytes & 7) == 0 && kMaxWords >= 2)
    {
#pragma unroll
        for (int w = 0; w + 1 < kMaxWords; w += 2)
            if (w * 4 < bytes)
                *reinterpret_cast<uint2*>(pixel + w * 4) = make_uint2(words[w], words[w + 1]);
    }
    else if ((bytes & 3) == 0)
    {
#pragma unroll
        for (int w = 0; w < kMaxWords; ++w)
            if (w * 4 < bytes)
                *reinterpret_cast<uint32_t*>(pixel + w * 4) = words[w];
    }
    else if ((bytes & 1) == 0)
    {
#pragma unroll
        for (int h = 0; h < kMaxWords * 2; ++h)
            if (h * 2 < bytes)
                *reinterpret_cast<uint16_t*>(pixel + h * 2) = uint16_t(words[h >> 1] >> (16 * (h & 1)));
    }
    else
    {
#pragma unroll
        for (int b = 0; b < kMaxWords * 4; ++b)
            if (b < bytes)
                pixel[b] = (unsigned char)(words[b >> 2] >> (8 * (b & 3)));
    }
}

// max(0, min(limit, roundf(x))) for an integer limit below 2^16, as RoundToCode, from a sum that rounds down: of x + 2^15 + 0.5
// bits 8 to 15 are the integer part (8-bit codes), of x + 2^16 + 0.5 bits 7 to 22 (16-bit codes).
__device__ __forceinline__ uint32_t RoundToByte1(float x)
{
    return __float_as_uint(__fadd_rd(fmaxf(fminf(x, 255.f), 0.f), 32768.5f));
}
__device__ __forceinline__ uint32_t RoundTo16Bits(float x)
{
    return (__float_as_uint(__fadd_rd(fmaxf(fminf(x, 65535.f), 0.f), 65536.5f)) >> 7) & 0xFFFFu;
}

// SrgbEncode clamped to [0, 1].  (The value is finite, so no NaN reaches the clamp.)
__device__ __forceinline__ float SrgbEncodeSaturated(float linear)
{
    float low, high;
    asm("mul.ftz.sat.f32 %0, %1, %2;" : "=f"(low) : "f"(linear), "f"(12.92f));
    asm("fma.rn.ftz.sat.f32 %0, %1, %2, %3;" : "=f"(high) : "f"(1.055f), "f"(ApproxPow(linear, 1.0f / 2.4f)), "f"(-0.055f));
    return linear <= 0.0031308f ? low : high;
}

// Two linear channels; codes of 16 bits in the low bits, with anything above.
template <int kFormat>
__device__ __forceinline__ void LinearPair(uint32_t pair, uint32_t& lo, uint32_t& hi)
{
    if (kFormat == kFormatUnorm16)
    {
        // the sums round down: x + 0.5 to a grid that holds the integers, then to the integers
        const float2 v = __half22float2(__hmul2_sat(AsHalf2(pair), __float2half2_rn(1.f)));
        lo = __float_as_uint(__fadd_rd(__fadd_rd(MulFtz(v.x, 65535.f), 0.5f), 8388608.f));
        hi = __float_as_uint(__fadd_rd(__fadd_rd(MulFtz(v.y, 65535.f), 0.5f), 8388608.f));
    }
    else if (kFormat == kFormatFloat16)
    {
        lo = pair; // finite binary16 values as they are
        hi = pair >> 16;
    }
    else
    {
        const float2 v = __half22float2(AsHalf2(pair));
        lo = QuantizeComponent(kFormat, v.x, 0.f);
        hi = QuantizeComponent(kFormat, v.y, 0.f);
    }
}

// An undithered component that is a channel in colour spaces, or a default (0; component 3: 1).
template <int kFormat>
__device__ __forceinline__ uint32_t UnditheredComponent(const OutputConversion& conversion, int numChannels, int c, uint32_t half)
{
    if (c >= numChannels)
    {
        constexpr uint32_t kOneCode = kFormat == kFormatUnorm8 ? 255u : kFormat == kFormatUnorm16 ? 65535u : kFormat == kFormatFloat16 ? 0x3c00u
                                    : kFormat == kFormatFloat32 ? 0x3f800000u : 1u;
        return c == 3 ? kOneCode : 0u;
    }
    const uint32_t kind = (conversion.componentKinds >> (2 * c)) & 3u;
    if (kFormat == kFormatFloat16 && kind == kKindLinear)
        return half; // finite binary16 values as they are
    float value = __half2float(__ushort_as_half((unsigned short)half));
    if (kind != kKindLinear)
    {
        const int srcSpace = (conversion.srcSpaces >> (2 * c)) & 3, dstSpace = (conversion.dstSpaces >> (2 * c)) & 3;
        value = EncodeColorSpace(dstSpace, DecodeColorSpace(srcSpace, value));
    }
    if (kFormat == kFormatUnorm8)
        return __byte_perm(RoundToByte1(MulFtz(value, 255.f)), 0u, 0x4441);
    if (kFormat == kFormatUnorm16)
        return RoundTo16Bits(MulFtz(value, 65535.f));
    return QuantizeComponent(kFormat, value, 0.f);
}

// Two linear channels as 8-bit codes in bytes 0 and 2: round(clamp(v) * 255).  In binary16 the sum v * 255 + 1024 lies in
// [1024, 1279], where the spacing is 1, and the fused multiply-add rounds it once; the only tie, v = 0.5, goes to 1152 - to
// even and away from zero - so the low byte is the reference's roundf() result.  (Decoded texels are finite.)
__device__ __forceinline__ uint32_t LinearCodes(uint32_t pair)
{
    const __half2 clamped = __hmul2_sat(AsHalf2(pair), __float2half2_rn(1.f));
    return AsU32(__hfma2(clamped, __float2half2_rn(255.f), __float2half2_rn(1024.f)));
}

// The kConvertUnorm8 epilogue: word by word, four linear channels in six instructions, then the bytes of the channels that are
// encoded to sRGB.  What a word takes is the same for every pixel.  (With one sRGB texture in a 12-channel set all channels
// went through the general quantiser: 500 us more on a 4096 x 4096 chain than fp16 texels; now about 115.)
template <typename Context>
__device__ __forceinline__ void ConvertUnorm8Pixel(const OutputConversion& conversion, const Context& ctx, const uint32_t (&pairs)[8])
{
    uint32_t words[4] = {0, 0, 0, 0};
#pragma unroll
    for (int w = 0; w < 4; ++w)
    {
        if (4 * w < conversion.dstChannels)
        {
            uint32_t word = __byte_perm(LinearCodes(pairs[2 * w]), LinearCodes(pairs[2 * w + 1]), 0x6420);
            if ((conversion.srgb >> (4 * w)) & 15u)
            {
#pragma unroll
                for (int k = 0; k < 4; ++k)
                {
                    if ((conversion.srgb >> (4 * w + k)) & 1u)
                    {
                        const __half2 pair = AsHalf2(pairs[2 * w + (k >> 1)]);
                        const float value = (k & 1) ? __high2float(pair) : __low2float(pair);
                        constexpr uint32_t kInsert[4] = {0x3215u, 0x3250u, 0x3510u, 0x5210u}; // byte 1 of the second operand as byte k
                        word = __byte_perm(word, RoundToByte1(MulFtz(SrgbEncodeSaturated(value), 255.f)), kInsert[k]);
                    }
                }
            }
            words[w] = (word & conversion.keep[w]) | conversion.ones[w];
        }
    }
    StorePixel<4>(reinterpret_cast<unsigned char*>(ctx.out), words, conversion.dstChannels);
}

// Converting epilogue for one channel format: pairs[j] holds the requested channels 2j and 2j + 1
// as (scrubbed) binary16; the pixel goes to ctx.out.  What ITextureSet::ReadChannels would produce
// from the stored texels (src/TextureSet.cpp:915-985, src/ImageProcessing.cu:220-266).
template <int kFormat, typename Context>
__device__ __forceinline__ void ConvertPixel(const OutputConversion& conversion, int numChannels, const Context& ctx,
    const uint32_t (&pairs)[8])
{
    constexpr int kBytes = kFormat == kFormatUnorm8 ? 1 : (kFormat == kFormatUnorm16 || kFormat == kFormatFloat16) ? 2 : 4;
    constexpr int kPerWord = 4 / kBytes;
    constexpr int kMaxWords = 16 / kPerWord;
    const int components = conversion.dstChannels;
    uint32_t words[kMaxWords];
#pragma unroll
    for (int w = 0; w < kMaxWords; ++w)
        words[w] = 0;

    if (!conversion.dither)
    {
#pragma unroll
        for (int j = 0; j < 8; ++j)
        {
            if (2 * j < components)
            {
                uint32_t lo, hi;
                if (((conversion.componentKinds >> (4 * j)) & 15u) == kKindLinear * 5u)
                    LinearPair<kFormat>(pairs[j], lo, hi);
                else
                {
                    lo = UnditheredComponent<kFormat>(conversion, numChannels, 2 * j, pairs[j] & 0xFFFFu);
                    hi = 2 * j + 1 < components ? UnditheredComponent<kFormat>(conversion, numChannels, 2 * j + 1, pairs[j] >> 16) : 0u;
                }
                if (kBytes == 4)
                {
                    words[(2 * j) % kMaxWords] = lo;
                    words[(2 * j + 1) % kMaxWords] = hi;
                }
                else if (kBytes == 2)
                    words[j % kMaxWords] = __byte_perm(lo, hi, 0x5410);
                else
                    words[(j >> 1) % kMaxWords] |= (lo | hi << 8) << (16 * (j & 1));
            }
        }
    }
    else
    {
        const uint32_t seed = DitherSeed(ctx.outStepWords);
#pragma unroll
        for (int c = 0; c < 16; ++c)
        {
            if (c < components)
            {
                const __half2 pair = AsHalf2(pairs[c >> 1]);
                float value = __half2float((c & 1) ? __high2half(pair) : __low2half(pair));
                const uint32_t kind = (conversion.componentKinds >> (2 * c)) & 3u;
                if (kind == kKindSrgbEncode)
                    value = SrgbEncode(value);
                else if (kind == kKindOther)
                    value = EncodeColorSpace((conversion.dstSpaces >> (2 * c)) & 3, DecodeColorSpace((conversion.srcSpaces >> (2 * c)) & 3, value));
                else if (kind == kKindDefault)
                    value = c == 3 ? 1.f : 0.f;
                const float dither = DitherDraw(seed, uint32_t(c) + 1u);
                uint32_t component;
                if (kFormat == kFormatUnorm8)
                    component = __byte_perm(RoundToByte1(MulFtz(AddFtz(value, ApproxDivide(dither, 255.f)), 255.f)), 0u, 0x4441);
                else if (kFormat == kFormatUnorm16)
                    component = RoundTo16Bits(MulFtz(AddFtz(value, ApproxDivide(dither, 65535.f)), 65535.f));
                else
                    component = QuantizeComponent(kFormat, value, dither);
                words[c / kPerWord] |= component << (8 * kBytes * (c % kPerWord));
            }
        }
    }
    StorePixel<kMaxWords>(reinterpret_cast<unsigned char*>(ctx.out), words, components * kBytes);
}

// Converting epilogue: the thread's (scrubbed) fp16 channel pairs -> the pixel in the client's
// format, stored at ctx.out.
template <int kConvert, typename Context>
__device__ __forceinline__ void StoreConverted(const OutputConversion& conversion, int firstChannel, int numChannels,
    const Context& ctx, uint32_t (&bits)[8])
{
    if (firstChannel != 0)
    {
        // Re-base the channels so that the first requested one sits in bits[0]: park them in the
        // thread's own slots of the A operand, which the tensor core has finished reading (layer 3's
        // MMA has completed), and read them back from the shifted position.
        uint4* slot = ctx.rowChunk;
        slot[0] = make_uint4(bits[0], bits[1], bits[2], bits[3]);
        slot[128] = make_uint4(bits[4], bits[5], bits[6], bits[7]);
        const unsigned char* parked = reinterpret_cast<const unsigned char*>(slot);
#pragma unroll
        for (int j = 0; j < 8; ++j)
        {
            const int c0 = firstChannel + 2 * j, c1 = c0 + 1;
            const uint32_t lo = c0 < 16 ? *reinterpret_cast<const uint16_t*>(parked + (c0 >> 3) * 2048 + (c0 & 7) * 2) : 0u;
            const uint32_t hi = c1 < 16 ? *reinterpret_cast<const uint16_t*>(parked + (c1 >> 3) * 2048 + (c1 & 7) * 2) : 0u;
            bits[j] = lo | (hi << 16);
        }
    }
    if (kConvert == kConvertUnorm8)
    {
        ConvertUnorm8Pixel(conversion, ctx, bits);
        return;
    }
    switch (conversion.format)
    {
    case kFormatUnorm8: ConvertPixel<kFormatUnorm8>(conversion, numChannels, ctx, bits); break;
    case kFormatUnorm16: ConvertPixel<kFormatUnorm16>(conversion, numChannels, ctx, bits); break;
    case kFormatFloat16: ConvertPixel<kFormatFloat16>(conversion, numChannels, ctx, bits); break;
    case kFormatFloat32: ConvertPixel<kFormatFloat32>(conversion, numChannels, ctx, bits); break;
    default: ConvertPixel<kFormatUint32>(conversion, numChannels, ctx, bits); break;
    }
}

} // namespace
} // namespace ntcb
