// Building blocks shared by the decode kernels (decode_kernel.cu: exact accumulation;
// decode_kernel_ref.cu: the reference's binary16 accumulation): PTX wrappers for mbarriers, tensor
// memory and the TMA bulk copy, the shared-memory matrix descriptor, and the bilinear tap setup.
#pragma once

#include <cuda_fp16.h>
#include <cuda_runtime.h>
#include <stdint.h>

#include "decode_kernel.h"

namespace ntcb
{
namespace
{

__device__ __forceinline__ uint32_t SharedAddress(const void* p)
{
    return static_cast<uint32_t>(__cvta_generic_to_shared(p));
}

// Start of the kernel's dynamic shared memory: a constant, so what is computed from it is visibly the same in every thread.
__device__ __forceinline__ uint32_t DynamicSharedBase()
{
    extern __shared__ __align__(128) unsigned char dynamicShared[];
    return SharedAddress(dynamicShared);
}

__device__ __forceinline__ void MbarrierInit(uint32_t bar, uint32_t count)
{
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(bar), "r"(count) : "memory");
}

__device__ __forceinline__ void FenceBarrierInit()
{
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
}

// One poll of a barrier phase.  The instruction may suspend the thread until the phase completes, and gives up by itself after 1.4 us.
// (With a suspend-time hint a poll is three instructions, one of them a sleep: 4096 x 4096 FP8 647 us instead of 640, 2048 x 2048 of 8 features 163
// instead of 153, 8192 x 8192 Int8 3612 instead of 3572, 16.7 M queries 643 instead of 634.)
__device__ __forceinline__ bool MbarrierTryWait(uint32_t bar, uint32_t parity)
{
    uint32_t done;
    asm volatile(
        "{\n\t"
        ".reg .pred p;\n\t"
        "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t"
        "}"
        : "=r"(done)
        : "r"(bar), "r"(parity)
        : "memory");
    return done != 0;
}

// Announces `bytes` of asynchronous copies that will complete on the barrier, and arrives on it.
__device__ __forceinline__ void MbarrierArriveExpectTx(uint32_t bar, uint32_t bytes)
{
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(bytes) : "memory");
}

// TMA bulk copy global -> shared memory of this CTA (addresses and size multiples of 16 bytes);
// completion is signalled on the barrier.
__device__ __forceinline__ void BulkCopyToShared(uint32_t dstShared, const void* srcGlobal, uint32_t bytes, uint32_t bar)
{
    asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];"
                 ::"r"(dstShared), "l"(srcGlobal), "r"(bytes), "r"(bar)
                 : "memory");
}

// Bounded wait: returns false when the barrier did not complete within `limit` polls.
__device__ __forceinline__ bool MbarrierWaitBounded(uint32_t bar, uint32_t parity, uint32_t limit = kSpinLimit)
{
    if (limit != 0 && MbarrierTryWait(bar, parity))
        return true;
    // (not unrolled: with the scrub below 4096 x 4096 texels take 832 us instead of 851, in instructions and their fetches)
#pragma unroll 1
    for (uint32_t spin = 1; spin < limit; ++spin)
    {
        if (MbarrierTryWait(bar, parity))
            return true;
    }
    return false;
}

// Records an expired wait in the status words.  The first thread of the grid to report claims word 0
// and alone writes the tile and layer, so the three words always describe one and the same wait.
__device__ __noinline__ void ReportTimeout(uint32_t* status, uint32_t tile, uint32_t layer)
{
    if (atomicCAS(&status[0], 0u, kStatusBarrierTimeout) == 0u)
    {
        status[1] = tile;
        status[2] = layer;
    }
}

// Programmatic dependent launch: the decode kernels are launched so that the next one in the stream may start once all
// CTAs of this one are running and hold their tensor memory (LaunchOverlapped).  Until GridDependencyWait returns - everything
// before this kernel in the stream has completed and is visible - a CTA touches nothing in global memory; it sets up barriers,
// constant tables and tensor memory meanwhile.
//
// GridDependencyLaunch comes after the barrier that follows the CTA's TmemAlloc, never before: a CTA of the next kernel takes its
// columns and keeps them while it waits for this kernel to end, so a CTA of this kernel that had not allocated by then
// could wait for those columns for good.
__device__ __forceinline__ void GridDependencyWait()
{
    asm volatile("griddepcontrol.wait;" ::: "memory");
}
__device__ __forceinline__ void GridDependencyLaunch()
{
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
}

__device__ __forceinline__ void FenceProxyAsyncShared()
{
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
}

__device__ __forceinline__ void TcgenFenceBeforeSync()
{
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
}

__device__ __forceinline__ void TcgenFenceAfterSync()
{
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
}

__device__ __forceinline__ void TmemAlloc(uint32_t sharedSlot, uint32_t columns)
{
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(sharedSlot), "r"(columns)
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
}

__device__ __forceinline__ void TmemFree(uint32_t address, uint32_t columns)
{
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(address), "r"(columns) : "memory");
}

__device__ __forceinline__ void UmmaCommit(uint32_t bar)
{
    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(bar) : "memory");
}

// ... by a converged warp, from the lane that elect.sync picks.
__device__ __forceinline__ void UmmaCommitElected(uint32_t bar)
{
    asm volatile(
        "{\n\t"
        ".reg .pred q;\n\t"
        "elect.sync _|q, 0xFFFFFFFF;\n\t"
        "@q tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];\n\t"
        "}" ::"r"(bar)
        : "memory");
}

// 16 consecutive 32-bit columns of this thread's TMEM lane.
__device__ __forceinline__ void TmemLoad16(uint32_t address, uint32_t (&r)[16])
{
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x16.b32 "
        "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, [%16];"
        : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]),
          "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
        : "r"(address)
        : "memory");
}

// Four consecutive 32-bit columns of this thread's TMEM lane, written.
__device__ __forceinline__ void TmemStore4(uint32_t address, uint32_t a, uint32_t b, uint32_t c, uint32_t d)
{
    asm volatile("tcgen05.st.sync.aligned.32x32b.x4.b32 [%0], {%1, %2, %3, %4};" ::"r"(address), "r"(a), "r"(b), "r"(c), "r"(d)
                 : "memory");
}

// Eight, sixteen.
__device__ __forceinline__ void TmemStore8(uint32_t address, const uint32_t* w)
{
    asm volatile("tcgen05.st.sync.aligned.32x32b.x8.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8};" ::"r"(address), "r"(w[0]), "r"(w[1]),
                 "r"(w[2]), "r"(w[3]), "r"(w[4]), "r"(w[5]), "r"(w[6]), "r"(w[7])
                 : "memory");
}

__device__ __forceinline__ void TmemStore16(uint32_t address, const uint32_t* w)
{
    asm volatile("tcgen05.st.sync.aligned.32x32b.x16.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, %16};"
                 ::"r"(address), "r"(w[0]), "r"(w[1]), "r"(w[2]), "r"(w[3]), "r"(w[4]), "r"(w[5]), "r"(w[6]), "r"(w[7]), "r"(w[8]), "r"(w[9]),
                 "r"(w[10]), "r"(w[11]), "r"(w[12]), "r"(w[13]), "r"(w[14]), "r"(w[15])
                 : "memory");
}

__device__ __forceinline__ void TmemStoreWait()
{
    asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
}

__device__ __forceinline__ void TmemLoadWait()
{
    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
}

// Shared-memory matrix descriptor, K-major, no swizzle: 8x16-byte core matrices; `leadingBytes`
// separates core matrices along K, `strideBytes` separates 8-row groups along M/N.  As its two words: the high one is a constant, the low one
// holds the address in units of 16 bytes (DescriptorAddress), so operands at constant distances are one 32-bit addition apart.
__host__ __device__ constexpr uint32_t DescriptorLow(uint32_t leadingBytes)
{
    return (leadingBytes >> 4) << 16;
}
__host__ __device__ constexpr uint32_t DescriptorHigh(uint32_t strideBytes)
{
    return (strideBytes >> 4) | 1u << 14; // bit 46: descriptor version of this architecture; base offset 0, layout type 0 (no swizzle)
}
__device__ __forceinline__ uint32_t DescriptorAddress(uint32_t sharedAddress)
{
    return (sharedAddress & 0x3FFFF) >> 4;
}

__device__ __forceinline__ uint32_t AsU32(__half2 v)
{
    return *reinterpret_cast<uint32_t*>(&v);
}

__device__ __forceinline__ __half2 AsHalf2(uint32_t v)
{
    return *reinterpret_cast<__half2*>(&v);
}

// Clamped HGELU in binary16 (src/tin/tin_activation.h:88-92).
__device__ __forceinline__ __half2 ClampedHgelu(__half2 x)
{
    const __half2 t = __hfma2_sat(__float2half2_rn(1 / 3.f), x, __float2half2_rn(0.5f));
    return __hmul2_rn(__hmin2(x, __float2half2_rn(3.f)), t);
}

// Two pairs of values -> four e4m3 codes (round to nearest even, saturating).  The conversions fill the two halves of one register, which
// leaves nothing to extend or to join (with 16-bit results widened and joined by a multiply-add a texel of an FP8 network took 987
// instructions instead of 891: 4096 x 4096 779 -> 719 us, 16.7 M queries 692 -> 648).
// No value may be converted twice where the compiler can see that it is the same, in the other half or in another word: ptxas 12.9 then shares one
// conversion between them and leaves bytes undefined - for E4m3Codes(x, x), also of constants, and E4m3Codes(x, y) beside E4m3Codes(y, x); without
// optimisation all are right.  (Joining 16-bit results by a shift, a permutation or a multiply-add has no such fault.)  The callers convert
// accumulators, blended features and encoded positions, once each.
__device__ __forceinline__ uint32_t E4m3Codes(__half2 first, __half2 second)
{
    uint32_t codes;
    asm("{\n\t"
        ".reg .b16 low, high;\n\t"
        "cvt.rn.satfinite.e4m3x2.f16x2 low, %1;\n\t"
        "cvt.rn.satfinite.e4m3x2.f16x2 high, %2;\n\t"
        "mov.b32 %0, {low, high};\n\t"
        "}"
        : "=r"(codes)
        : "r"(AsU32(first)), "r"(AsU32(second)));
    return codes;
}

// Inf / NaN -> 0 in the channel pairs of one texel (src/Inference.cu:125-126, src/CudaUtils.h:30-35).
// The largest magnitude of all pairs, a NaN counting as largest, shows whether anything has to be done at all.  (Sums of products with zero show it
// in as many instructions, but on the packed-fp16 pipe, the busiest: 8192 x 8192 Int8 3468 us instead of 3448, 4096 x 4096 FP8 592.7 instead of 589.5.)
__device__ __forceinline__ void ScrubSpecials(uint32_t (&bits)[8], int channelPairs)
{
    uint32_t largest = bits[0];
#pragma unroll
    for (int j = 1; j < 8; ++j) // (all pairs: a special value in a pair beyond the channels only leads to the check of each)
        asm("max.NaN.xorsign.abs.f16x2 %0, %1, %2;" : "=r"(largest) : "r"(largest), "r"(bits[j]));
    if (((largest & 0x7C007C00u) + 0x04000400u) & 0x80008000u)
    {
        // rare, so kept off the common path
#pragma unroll
        for (int j = 0; j < 8; ++j)
        {
            if (j < channelPairs)
            {
                if ((bits[j] & 0x7C00u) == 0x7C00u) bits[j] &= 0xFFFF0000u;
                if ((bits[j] & 0x7C000000u) == 0x7C000000u) bits[j] &= 0x0000FFFFu;
            }
        }
    }
}

// Stores the channel pairs of one texel.  Pixel-interleaved layout: the pairs are consecutive words
// and go out as 16-, 8- or 4-byte stores, whatever `vectorBytes` (the alignment every texel of the
// mip has) allows; planar-pair layout: `stepWords` words apart, one word each.
__device__ __forceinline__ void StoreTexel(uint32_t* out, uint32_t stepWords, int vectorBytes, const uint32_t (&bits)[8],
    int channelPairs)
{
    if (vectorBytes == 16)
    {
#pragma unroll
        for (int j = 0; j < 8; j += 4)
            if (j < channelPairs)
                *reinterpret_cast<uint4*>(out + j) = make_uint4(bits[j], bits[j + 1], bits[j + 2], bits[j + 3]);
    }
    else if (vectorBytes == 8)
    {
#pragma unroll
        for (int j = 0; j < 8; j += 2)
            if (j < channelPairs)
                *reinterpret_cast<uint2*>(out + j) = make_uint2(bits[j], bits[j + 1]);
    }
    else
    {
#pragma unroll
        for (int j = 0; j < 8; ++j)
            if (j < channelPairs)
                out[j * stepWords] = bits[j];
    }
}

// Latent codes to binary16 without a table.  A code n (0 .. 15) in bits 5-8 of a binary16 is the subnormal number z = n * 2^-19;
// times 2^19 / 15 it becomes the value the reference's fp16(float(n) * (1.f / 15.f)) has (src/Quantizer.cu:490-495).  The factor's nearest binary16
// number, 34944, gives all sixteen but 9 and 13, which it puts on a tie that goes the wrong way; one z more moves the ties up and nothing else
// (compared): z * 34944 + z, one operation on two codes at a time.  (As the sum of two products with factors of a code in bits 4-7:
// 16.7 M queries 616 us instead of 591,
// 1920 x 1080 with 16 features read directly 169 instead of 159.)  (Looked up in a table of all bytes in shared memory, the 32 unrelated bytes of a warp
// fell on 3.5 deep banks on average, 48 times per query of inference on sample, whose bound was the L1's data pipe: 16.7 M
// queries 0.97 -> 0.84 ms without.)
__device__ __forceinline__ __half2 CodesToHalves(uint32_t codes)
{
    const __half2 z = AsHalf2(codes & 0x01E001E0u);
    return __hfma2(z, __float2half2_rn(34944.f), z);
}

// A latent pixel of one layer (four 4-bit features in the low 16 bits) -> features (0, 1) and (2, 3).
__device__ __forceinline__ void UnpackPixel(uint32_t pixel, __half2& first, __half2& second)
{
    // a byte's low code to bits 5-8, its high code to bits 21-24
    first = CodesToHalves((pixel & 0xFFu) * 0x20020u);
    second = CodesToHalves(__byte_perm(pixel, 0u, 0x4441) * 0x20020u);
}

// Two layers of a latent pixel side by side in one word -> per feature the values of (first layer, second layer).
__device__ __forceinline__ void UnpackTwoLayers(uint32_t word, __half2 (&features)[4])
{
    features[0] = CodesToHalves(word << 5);
    features[1] = CodesToHalves(word << 1);
    features[2] = CodesToHalves(word >> 3);
    features[3] = CodesToHalves(word >> 7);
}

struct GridTaps
{
    int o00, o01, o10, o11;
    __half2 w00, w01, w10, w11;
};

// Bilinear footprint of one texel in one latent grid (src/FeatureGridDevice.h:33-58).
__device__ __forceinline__ void SetupTaps(float u, float v, int w, int h, GridTaps& taps)
{
    float px = __fmaf_rn(u, float(w), -0.5f);
    float py = __fmaf_rn(v, float(h), -0.5f);
    float xbf = floorf(px), ybf = floorf(py);
    float dx = __fsub_rn(px, xbf), dy = __fsub_rn(py, ybf);
    float dxn = __fsub_rn(1.f, dx), dyn = __fsub_rn(1.f, dy);
    int xb = int(xbf), yb = int(ybf);
    // wrap addressing; the sample position is < size - 0.5, so only -1 needs folding
    int x0 = xb < 0 ? xb + w : xb;
    int y0 = yb < 0 ? yb + h : yb;
    int x1 = (x0 + 1 == w) ? 0 : x0 + 1;
    int y1 = (y0 + 1 == h) ? 0 : y0 + 1;
    taps.o00 = y0 * w + x0;
    taps.o01 = y0 * w + x1;
    taps.o10 = y1 * w + x0;
    taps.o11 = y1 * w + x1;
    taps.w00 = __half2half2(__float2half_rn(__fmul_rn(dxn, dyn)));
    taps.w01 = __half2half2(__float2half_rn(__fmul_rn(dx, dyn)));
    taps.w10 = __half2half2(__float2half_rn(__fmul_rn(dxn, dy)));
    taps.w11 = __half2half2(__float2half_rn(__fmul_rn(dx, dy)));
}

__device__ __forceinline__ float Frac(float t)
{
    return __fsub_rn(t, floorf(t));
}

// Normalised sample coordinate of a texel, (texel + 0.5) / extent (src/Inference.cu:52-53).  The
// reference is built with --use_fast_math, so its division is the approximate one
// (div.approx.ftz.f32: the operand times the hardware's reciprocal approximation, which for extents
// that are not powers of two can differ from the correctly rounded reciprocal in the last bit, and
// with it - rarely - a bilinear weight).  The reference-numerics kernels issue the same instruction;
// the exact-accumulation kernels keep the multiplication by the correctly rounded reciprocal that
// their CPU restatement uses.
template <bool kReferenceDivision>
__device__ __forceinline__ float TexelCoordinate(int texel, int extent, float invExtent)
{
    const float centre = __fadd_rn(float(texel), 0.5f);
    if (kReferenceDivision)
    {
        float u;
        asm("div.approx.ftz.f32 %0, %1, %2;" : "=f"(u) : "f"(centre), "f"(float(extent)));
        return u;
    }
    return __fmul_rn(centre, invExtent);
}

// One axis of the bilinear footprint (src/FeatureGridDevice.h:35-45): base tap index (before
// wrapping) and the fractional offset of a texel coordinate in a latent grid of `size` pixels.
template <bool kReferenceDivision>
__device__ __forceinline__ void AxisTap(int texel, int extent, float invExtent, int size, int& base, float& frac)
{
    const float u = TexelCoordinate<kReferenceDivision>(texel, extent, invExtent);
    const float p = __fmaf_rn(u, float(size), -0.5f);
    const float b = floorf(p);
    base = int(b);
    frac = __fsub_rn(p, b);
}

// Nonzero in exactly one lane of the (converged) warp.
__device__ __forceinline__ uint32_t ElectOne()
{
    uint32_t elected;
    asm volatile(
        "{\n\t"
        ".reg .pred p;\n\t"
        "elect.sync _|p, 0xFFFFFFFF;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t"
        "}"
        : "=r"(elected));
    return elected;
}

// The same value of a warp's first lane in all of its lanes, visibly so: what is computed from it stays in uniform registers, and branches on it
// need no reconvergence.
__device__ __forceinline__ uint32_t Uniform(uint32_t value)
{
    return __shfl_sync(0xFFFFFFFFu, value, 0);
}

// All 128 threads of a chain.
__device__ __forceinline__ void ChainBarrier(int chain)
{
    asm volatile("bar.sync %0, 128;" ::"r"(chain + 1) : "memory");
}

// The barrier before a layer's matrix products.  The operand rows, tables and footprints of a
// chain are written by the chain's own 128 threads, and only they read its accumulators, so a chain meets in a named barrier of
// its own and the chains of a CTA, up to eight, drift apart instead of waiting for each other.
//
// Giving up: a thread whose wait expired sets the chain's give-up word for the tile, of which there are two in turn, and goes on; in
// the next tile's layer 0, after the barrier, all threads read it.  The words alternate, so a word that some thread may still
// be reading is not written before that thread has met the others again, and all take the same decision.  (A barrier that
// reduces a predicate, bar.red, says the same at once but costs more than the barrier alone: inference on sample became
// 6 % faster with half as many of them.)  Returns nonzero when the chain is to leave.
__device__ __forceinline__ void SetGiveUp(uint32_t word)
{
    asm volatile("st.volatile.shared.u32 [%0], 1;" ::"r"(word) : "memory");
}

template <int kLayer>
__device__ __forceinline__ uint32_t LayerBarrier(int chain, uint32_t& giveUp)
{
    ChainBarrier(chain);
    if (kLayer != 0)
        return 0;
    uint32_t word;
    asm volatile("ld.volatile.shared.u32 %0, [%1];" : "=r"(word) : "r"(giveUp) : "memory");
    giveUp ^= 4u; // the two words share an aligned pair
    return word;
}

// Launches a kernel that calls GridDependencyWait before it touches global memory, so that its start overlaps the end of
// the kernel before it in the stream: when it came, a 96 x 40 set decoded back to back in 6.3 us instead
// of 8.2, mip 0 of a 1024 x 1024 one in 58.8 instead of 61.6 (now 4.3 and 40.9).
template <typename Kernel, typename Params>
cudaError_t LaunchOverlapped(Kernel kernel, int ctas, int threads, size_t sharedBytes, cudaStream_t stream, const Params& params)
{
    cudaLaunchConfig_t config{};
    config.gridDim = dim3(unsigned(ctas));
    config.blockDim = dim3(unsigned(threads));
    config.dynamicSmemBytes = sharedBytes;
    config.stream = stream;
    cudaLaunchAttribute attribute{};
    attribute.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attribute.val.programmaticStreamSerializationAllowed = 1;
    config.attrs = &attribute;
    config.numAttrs = 1;
    return cudaLaunchKernelEx(&config, kernel, params);
}

} // namespace
} // namespace ntcb
