// Packed binary32 arithmetic (add / mul / fma .f32x2): two IEEE operations per instruction and issue slot, on an aligned
// pair of registers.  Used where a kernel is bound by instruction issue and has two independent values at hand.
#pragma once

namespace ntcb
{
namespace
{

struct Pair
{
    unsigned long long bits;
};

__device__ __forceinline__ Pair MakePair(float first, float second)
{
    Pair r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r.bits) : "f"(first), "f"(second));
    return r;
}
__device__ __forceinline__ Pair Both(float v) { return MakePair(v, v); }
__device__ __forceinline__ void Split(Pair p, float& first, float& second)
{
    asm("mov.b64 {%0, %1}, %2;" : "=f"(first), "=f"(second) : "l"(p.bits));
}
__device__ __forceinline__ Pair operator*(Pair a, Pair b)
{
    Pair r;
    asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r.bits) : "l"(a.bits), "l"(b.bits));
    return r;
}
__device__ __forceinline__ Pair MultiplyAdd(Pair a, Pair b, Pair c)
{
    Pair r;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r.bits) : "l"(a.bits), "l"(b.bits), "l"(c.bits));
    return r;
}
// ... rounded down
__device__ __forceinline__ Pair MultiplyAddDown(Pair a, Pair b, Pair c)
{
    Pair r;
    asm("fma.rm.f32x2 %0, %1, %2, %3;" : "=l"(r.bits) : "l"(a.bits), "l"(b.bits), "l"(c.bits));
    return r;
}
__device__ __forceinline__ Pair Negate(Pair a)
{
    float x, y;
    Split(a, x, y);
    return MakePair(-x, -y);
}
// a + b where neither is a product, or where the sum is exact
__device__ __forceinline__ Pair PlainAdd(Pair a, Pair b)
{
    Pair r;
    asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r.bits) : "l"(a.bits), "l"(b.bits));
    return r;
}
// Other sums are multiply-adds with factors of 1 and -1 (an exact product: one rounding, the sum's).  The factors come from
// constant memory, so that they are not known at compile time: written as add.rn.f32x2, a sum is fused with the packed
// multiplication before it, whatever --fmad says, and comes out with another rounding.
__constant__ float2 kOne = {1.f, 1.f};
__constant__ float2 kMinusOne = {-1.f, -1.f};
__device__ __forceinline__ Pair operator+(Pair a, Pair b) { return MultiplyAdd(a, MakePair(kOne.x, kOne.y), b); }
__device__ __forceinline__ Pair operator-(Pair a, Pair b) { return MultiplyAdd(b, MakePair(kMinusOne.x, kMinusOne.y), a); }

} // namespace
} // namespace ntcb
