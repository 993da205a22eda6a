// Packed FP32x2 arithmetic for sm_100a stencils (internal).  F2 holds the
// values of two neighbouring grid points in one 64-bit register pair, so that
// it goes through packed arithmetic, 64-bit loads and stores without the
// moves a struct of two floats costs (with one, a fifth of k_force's and
// k_scalars' instructions were moves).  Every operator is one packed
// instruction (add/sub/mul/fma.rn.f32x2) that rounds each lane exactly as the
// scalar instruction would, so a formula written over F2 gives each point
// the value the scalar formula gives it.  Scalars (per-level constants)
// broadcast to both lanes.
#pragma once
#include <cuda_runtime.h>
#include <cstdint>

namespace cress {

struct F2 {
  uint64_t b;
  __device__ __forceinline__ float x() const { return __uint_as_float((uint32_t)b); }
  __device__ __forceinline__ float y() const { return __uint_as_float((uint32_t)(b >> 32)); }
};

__device__ __forceinline__ F2 f2(float a, float b) {
  F2 r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r.b) : "f"(a), "f"(b));
  return r;
}
__device__ __forceinline__ F2 f2(float a) { return f2(a, a); }

__device__ __forceinline__ F2 operator+(F2 a, F2 b) {
  F2 r;
  asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r.b) : "l"(a.b), "l"(b.b));
  return r;
}
__device__ __forceinline__ F2 operator*(F2 a, F2 b) {
  F2 r;
  asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r.b) : "l"(a.b), "l"(b.b));
  return r;
}
__device__ __forceinline__ F2 operator-(F2 a, F2 b) {
  F2 r;
  asm("sub.rn.f32x2 %0, %1, %2;" : "=l"(r.b) : "l"(a.b), "l"(b.b));
  return r;
}
__device__ __forceinline__ F2 fma2(F2 a, F2 b, F2 c) {
  F2 r;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r.b) : "l"(a.b), "l"(b.b), "l"(c.b));
  return r;
}
__device__ __forceinline__ F2 operator*(float s, F2 b) { return f2(s) * b; }
__device__ __forceinline__ F2 operator*(F2 a, float s) { return a * f2(s); }
__device__ __forceinline__ F2 operator+(F2 a, float s) { return a + f2(s); }
__device__ __forceinline__ F2 operator+(float s, F2 b) { return f2(s) + b; }
__device__ __forceinline__ F2 operator-(F2 a, float s) { return a - f2(s); }
__device__ __forceinline__ F2 operator-(float s, F2 b) { return f2(s) - b; }
__device__ __forceinline__ F2 fmax2(F2 a, float s) { return f2(fmaxf(a.x(), s), fmaxf(a.y(), s)); }

// Per-point choice: the lanes whose bit is set in mask (bit 0 the first
// point, bit 1 the second) take a, the others b.  The float overload serves
// one-point code (bit 0).
__device__ __forceinline__ F2 sel2(int mask, F2 a, F2 b) {
  return f2((mask & 1) ? a.x() : b.x(), (mask & 2) ? a.y() : b.y());
}
__device__ __forceinline__ float sel2(int mask, float a, float b) { return (mask & 1) ? a : b; }

// Two consecutive floats at an 8-byte aligned address (generic, or global
// memory the kernel does not write), and their store.
__device__ __forceinline__ F2 ld2(const float* p) { return F2{*reinterpret_cast<const uint64_t*>(p)}; }
__device__ __forceinline__ F2 gld2(const float* p) {
  return F2{__ldg(reinterpret_cast<const unsigned long long*>(p))};
}
__device__ __forceinline__ void st2(float* p, F2 v) { *reinterpret_cast<uint64_t*>(p) = v.b; }

// The pair between two aligned neighbouring pairs.
__device__ __forceinline__ F2 mid2(F2 a, F2 b) { return f2(a.y(), b.x()); }

// The pair (p[dx], p[dx+1]) for a compile-time dx, from aligned pairs only
// (p itself 8-byte aligned): an odd dx combines the halves of the aligned
// pairs on either side.
__device__ __forceinline__ F2 pair_at(const float* p, int dx) {
  if ((dx & 1) == 0) return ld2(p + dx);
  return mid2(ld2(p + dx - 1), ld2(p + dx + 1));
}

// The same pair kept as two floats and, through the intrinsics, open to the fusing
// of a multiply with an add: for k_scalars, whose separate terms (the reference's
// parenthesisation) the compiler schedules better in it, and k_hevi2.  512 x 512 x 64
// scalars, without and with the eddy mixing: 1193 and 1403 us, in F2 1257 and 1496; a
// substep of tile 11 at 256 x 256 x 60: 162 us, in F2 168.
struct V2 {
  float2 v;
  __device__ __forceinline__ float x() const { return v.x; }
  __device__ __forceinline__ float y() const { return v.y; }
};

__device__ __forceinline__ V2 v2(float a, float b) { return V2{make_float2(a, b)}; }
__device__ __forceinline__ V2 v2(float a) { return v2(a, a); }
__device__ __forceinline__ V2 operator+(V2 a, V2 b) { return V2{__fadd2_rn(a.v, b.v)}; }
__device__ __forceinline__ V2 operator*(V2 a, V2 b) { return V2{__fmul2_rn(a.v, b.v)}; }
__device__ __forceinline__ V2 operator-(V2 a, V2 b) {
  const F2 d = f2(a.x(), a.y()) - f2(b.x(), b.y());
  V2 r;
  asm("mov.b64 {%0, %1}, %2;" : "=f"(r.v.x), "=f"(r.v.y) : "l"(d.b));
  return r;
}
__device__ __forceinline__ V2 operator*(float s, V2 b) { return v2(s) * b; }
__device__ __forceinline__ V2 operator*(V2 a, float s) { return a * v2(s); }
__device__ __forceinline__ V2 operator-(V2 a, float s) { return a - v2(s); }
__device__ __forceinline__ V2 fmax2(V2 a, float s) { return v2(fmaxf(a.x(), s), fmaxf(a.y(), s)); }
__device__ __forceinline__ V2 sel2(int mask, V2 a, V2 b) {
  return v2((mask & 1) ? a.x() : b.x(), (mask & 2) ? a.y() : b.y());
}
__device__ __forceinline__ V2 ldv2(const float* p) { return V2{*reinterpret_cast<const float2*>(p)}; }
__device__ __forceinline__ void st2(float* p, V2 a) { *reinterpret_cast<float2*>(p) = a.v; }
__device__ __forceinline__ V2 vpair_at(const float* p, int dx) {
  if ((dx & 1) == 0) return ldv2(p + dx);
  return v2(ldv2(p + dx - 1).y(), ldv2(p + dx + 1).x());
}

}  // namespace cress
