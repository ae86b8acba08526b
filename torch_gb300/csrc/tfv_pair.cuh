// Packed single precision: two floats in a 64-bit register pair, one
// instruction for both (add / sub / mul / fma .f32x2, sm_100 and later).  Each
// half rounds as the scalar operation does (flush-to-zero like the units that
// use it).  The step kernels are bound by instruction issue, not by the FMA
// pipe, so a packed instruction saves an issue slot; packing costs nothing
// where the halves are results that the compiler can place side by side: the
// two sides of a face, a cell's upper and lower predicted states.  3D step 256^3
// 51.8 -> 49.0 warp instructions a cell, 986 -> 966 us a step; 32 2D grids of
// 64^2 to 1024^2 499 -> 485 us.  Limited slopes of two components packed
// (min / max have no packed form) were slower by 0.6%.
#pragma once

#include <cuda_runtime.h>

namespace tfv {

struct Pair {
  unsigned long long v;
};
__device__ __forceinline__ Pair pk(float lo, float hi) {
  Pair r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r.v) : "f"(lo), "f"(hi));
  return r;
}
__device__ __forceinline__ Pair pk(float x) { return pk(x, x); }
__device__ __forceinline__ void unpk(Pair p, float& lo, float& hi) {
  asm("mov.b64 {%0, %1}, %2;" : "=f"(lo), "=f"(hi) : "l"(p.v));
}
__device__ __forceinline__ float lo_(Pair p) {
  float a, b;
  unpk(p, a, b);
  return a;
}
__device__ __forceinline__ float hi_(Pair p) {
  float a, b;
  unpk(p, a, b);
  return b;
}
__device__ __forceinline__ Pair operator+(Pair a, Pair b) {
  Pair r;
  asm("add.rn.ftz.f32x2 %0, %1, %2;" : "=l"(r.v) : "l"(a.v), "l"(b.v));
  return r;
}
__device__ __forceinline__ Pair operator-(Pair a, Pair b) {
  Pair r;
  asm("sub.rn.ftz.f32x2 %0, %1, %2;" : "=l"(r.v) : "l"(a.v), "l"(b.v));
  return r;
}
__device__ __forceinline__ Pair operator*(Pair a, Pair b) {
  Pair r;
  asm("mul.rn.ftz.f32x2 %0, %1, %2;" : "=l"(r.v) : "l"(a.v), "l"(b.v));
  return r;
}
__device__ __forceinline__ Pair fma2(Pair a, Pair b, Pair c) {
  Pair r;
  asm("fma.rn.ftz.f32x2 %0, %1, %2, %3;" : "=l"(r.v) : "l"(a.v), "l"(b.v), "l"(c.v));
  return r;
}

}  // namespace tfv
