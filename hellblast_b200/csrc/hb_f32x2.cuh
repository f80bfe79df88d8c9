// Packed FP32 pairs (fma.rn.f32x2 and its kin): each half is an ordinary IEEE operation, so a packed
// computation gives the bits of the two scalar ones.  Measured on this GPU: the same FMA rate as
// scalar instructions (122 per clock and SM) at half the issue slots; 83 to 102 when the three
// operands are all different registers, as in scalar code.
#pragma once
namespace hb {
using f32x2 = unsigned long long;
__device__ __forceinline__ f32x2 pk(float a, float b) {
    f32x2 r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(a), "f"(b));
    return r;
}
__device__ __forceinline__ void unpk(f32x2 v, float &a, float &b) { asm("mov.b64 {%0, %1}, %2;" : "=f"(a), "=f"(b) : "l"(v)); }
__device__ __forceinline__ f32x2 dup2(float a) { return pk(a, a); }
__device__ __forceinline__ f32x2 fma2(f32x2 a, f32x2 b, f32x2 c) {
    f32x2 r;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
    return r;
}
__device__ __forceinline__ f32x2 mul2(f32x2 a, f32x2 b) {
    f32x2 r;
    asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}
__device__ __forceinline__ f32x2 add2(f32x2 a, f32x2 b) {
    f32x2 r;
    asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}
// OR of bit patterns, and whether any of the ORed values can be past 2^32 in magnitude (no false
// negatives: the OR's exponent field is at least every value's)
__device__ __forceinline__ unsigned bits_or(unsigned acc, f32x2 v) { return acc | (unsigned)v | (unsigned)(v >> 32); }
__device__ __forceinline__ bool maybe_big(unsigned acc) { return (acc & 0x7f800000u) >= 0x4f800000u; }
constexpr float F32_UP = 4294967296.0f;                 // 2^32: a state past this moves to the next exponent
constexpr float F32_DOWN = 5.42101086242752217e-20f;    // 2^-64: one exponent step
// (north, south) coefficients of a ring pair, as two 8-byte accesses: F and G are the caller's, complex64, and need
// no more alignment than that
__device__ __forceinline__ float4 load_ns(const float2 *p) {
    const float2 n = p[0], s = p[1];
    return make_float4(n.x, n.y, s.x, s.y);
}
__device__ __forceinline__ void put_ns(float2 *p, float nr, float ni, float sr, float si) {
    p[0] = make_float2(nr, ni);
    p[1] = make_float2(sr, si);
}
// factor that takes sums in units of 2^(64 e0) to units of 2^(64 e1).  Exponents rise from block to block, but for a
// first block's e1 < 0 against the 0 of empty sums: one step up is then as good as any, and stays finite.
__device__ __forceinline__ float sums_to_unit(int e0, int e1) {
    return e0 == e1 ? 1.f : ldexpf(1.f, 64 * max(-3, min(1, e0 - e1)));
}
}  // namespace hb
