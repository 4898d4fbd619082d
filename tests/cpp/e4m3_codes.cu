// E4m3Codes against single conversions, for every binary16 number in each of the four places and for a few literals: prints what differs.
#include <cstdio>
#include <cstring>
#include <vector>

#include <cuda_fp8.h>

#include "kernel_parts.cuh"

using namespace ntcb;

constexpr int kWords = 65536, kLiterals = 8;

// The four numbers of word `i`: each place sees all 65536.
__host__ __device__ inline uint2 Operands(uint32_t i)
{
    return make_uint2((i * 0x9E35u & 0xFFFFu) << 16 | i, ((i ^ 0x5A5Au) & 0xFFFFu) << 16 | ((i * 0x6A95u + 0x1234u) & 0xFFFFu));
}

__global__ void Words(uint32_t* words)
{
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    const uint2 operands = Operands(i);
    words[i] = E4m3Codes(AsHalf2(operands.x), AsHalf2(operands.y));
}

// Literals, no two of the same value in one word.
constexpr uint32_t kLiteral[kLiterals][2] = {{0u, 0x3C003C00u}, {0x3C003C00u, 0u}, {0x80008000u, 0x80000000u}, {0x7C00FC00u, 0x7E000001u},
                                             {0x12345678u, 0x9ABCDEF0u}, {0x5F005F80u, 0x00010000u}, {0x00003C00u, 0x3C000000u}, {0x3800B800u, 0x34000000u}};

template <uint32_t kFirst, uint32_t kSecond>
__global__ void Literal(uint32_t* word)
{
    *word = E4m3Codes(AsHalf2(kFirst), AsHalf2(kSecond));
}

template <int kIndex = 0>
void LaunchLiterals(uint32_t* words)
{
    Literal<kLiteral[kIndex][0], kLiteral[kIndex][1]><<<1, 1>>>(words + kIndex);
    if constexpr (kIndex + 1 < kLiterals)
        LaunchLiterals<kIndex + 1>(words);
}

__global__ void Single(const uint2* operands, uint8_t* codes) // a thread per number
{
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    const uint32_t word = (i & 2) ? operands[i >> 2].y : operands[i >> 2].x;
    __half_raw half;
    half.x = uint16_t((i & 1) ? word >> 16 : word);
    codes[i] = __nv_cvt_halfraw_to_fp8(half, __NV_SATFINITE, __NV_E4M3);
}

int main()
{
    constexpr int kAll = kWords + 256; // the literals are the last ones, padded with zeros
    std::vector<uint2> operands(kAll, make_uint2(0, 0));
    for (int i = 0; i < kWords; ++i)
        operands[i] = Operands(uint32_t(i));
    for (int i = 0; i < kLiterals; ++i)
        operands[kWords + i] = make_uint2(kLiteral[i][0], kLiteral[i][1]);
    uint2* deviceOperands = nullptr;
    uint32_t* words = nullptr;
    uint8_t* codes = nullptr;
    if (cudaMalloc(&deviceOperands, kAll * sizeof(uint2)) != cudaSuccess || cudaMalloc(&words, kAll * 4) != cudaSuccess ||
        cudaMalloc(&codes, kAll * 4) != cudaSuccess)
        return 2;
    cudaMemcpy(deviceOperands, operands.data(), kAll * sizeof(uint2), cudaMemcpyHostToDevice);
    Words<<<kWords / 256, 256>>>(words);
    LaunchLiterals(words + kWords);
    Single<<<kAll * 4 / 256, 256>>>(deviceOperands, codes);
    std::vector<uint32_t> got(kAll), expected(kAll);
    cudaMemcpy(got.data(), words, kAll * 4, cudaMemcpyDeviceToHost);
    cudaMemcpy(expected.data(), codes, kAll * 4, cudaMemcpyDeviceToHost);
    if (cudaDeviceSynchronize() != cudaSuccess)
        return 2;
    int different = 0;
    for (int i = 0; i < kWords + kLiterals; ++i)
        if (got[i] != expected[i] && ++different <= 10)
            std::printf("%08x %08x: %08x, expected %08x\n", operands[i].x, operands[i].y, got[i], expected[i]);
    return different != 0;
}
