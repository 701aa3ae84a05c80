// Two f32 operations per instruction (packed f32x2): IEEE round-to-nearest in each half, the same results as two scalar
// instructions (measured on 4 M random operands). One trap: the assembler contracts a mul2 whose only use is a packed add into
// a fused multiply-add, -fmad=false or not (36 % of the results change). Kernels that need the product rounded write the sum
// as fma2(product, one, sum) with a 1.0 that arrives as a kernel argument, which it cannot see through, or add in scalars.
#pragma once

namespace bk {

#ifdef __CUDACC__
using f32x2 = unsigned long long;
__device__ __forceinline__ f32x2 pack2(float a, float b) { f32x2 r; asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(a), "f"(b)); return r; }
__device__ __forceinline__ f32x2 pack2(int a, int b) { f32x2 r; asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "r"(a), "r"(b)); return r; }
__device__ __forceinline__ f32x2 pack2(unsigned a, unsigned b) { return pack2(int(a), int(b)); }
__device__ __forceinline__ void unpack2(f32x2 v, float& a, float& b) { asm("mov.b64 {%0, %1}, %2;" : "=f"(a), "=f"(b) : "l"(v)); }
__device__ __forceinline__ f32x2 sub2(f32x2 a, f32x2 b) { f32x2 r; asm("sub.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b)); return r; }
__device__ __forceinline__ f32x2 mul2(f32x2 a, f32x2 b) { f32x2 r; asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b)); return r; }
__device__ __forceinline__ f32x2 fma2(f32x2 a, f32x2 b, f32x2 c) { f32x2 r; asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c)); return r; }
#endif

}  // namespace bk
