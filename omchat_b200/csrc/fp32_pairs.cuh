// Packed fp32 pairs (sm_100: one instruction, two IEEE fp32 operations) and the quotients behind sigmoids that are made of them.
#pragma once
#include <cuda_runtime.h>

namespace omc {

typedef unsigned long long f32x2;
__device__ __forceinline__ f32x2 pack2(float lo, float hi) {
  f32x2 r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(lo), "f"(hi));
  return r;
}
__device__ __forceinline__ void unpack2(f32x2 v, float& lo, float& hi) { asm("mov.b64 {%0, %1}, %2;" : "=f"(lo), "=f"(hi) : "l"(v)); }
__device__ __forceinline__ f32x2 fma2(f32x2 a, f32x2 b, f32x2 c) {
  f32x2 d;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(d) : "l"(a), "l"(b), "l"(c));
  return d;
}
__device__ __forceinline__ f32x2 mul2(f32x2 a, f32x2 b) {
  f32x2 d;
  asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
  return d;
}

// x[i] / y[i] for neg[i] = -x[i], 1 <= y <= 2^64 and x zero or of a magnitude from 2^-60 to 2^100 (smaller too where y is 2, as behind exp(-x)), rounded as a division is (P. Markstein, Computation of elementary functions on
// the IBM RISC System/6000 processor, IBM J. Res. Dev. 34, 1990): a reciprocal with one Newton step, the quotient, and its remainder, which an fma has exactly. NaN in, NaN
// out. For pairs without one sign to turn: with R = -1 / y, q = -x R, and x / y = q + R (y q - x).
__device__ __forceinline__ void quotients2(float neg0, float neg1, float y0, float y1, float& q0, float& q1) {
  float r0, r1;
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r0) : "f"(-y0));
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r1) : "f"(-y1));
  const f32x2 neg = pack2(neg0, neg1), y = pack2(y0, y1), one = pack2(1.f, 1.f);
  f32x2 r = pack2(r0, r1);
  r = fma2(r, fma2(y, r, one), r);
  const f32x2 q = mul2(neg, r);
  unpack2(fma2(r, fma2(y, q, neg), q), q0, q1);
}

}  // namespace omc
