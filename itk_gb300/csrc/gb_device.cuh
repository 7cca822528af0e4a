// gb_device.cuh -- device-side building blocks of the registration-metric kernels.
//
// GB300 issues FP64 at a small fraction of its FP32 rate, so nothing in the
// per-sample loops is FP64.  Positions are mapped in double-float arithmetic:
// the per-evaluation affine map (virtual point -> moving continuous index) is
// computed once in FP64 and split into FP32 hi/lo pairs; each sample's
// (exactly representable, float) coordinates are multiplied with error-free
// FMA products and summed with two-sum, giving the continuous index to ~1e-12
// voxel, i.e. the reference's double arithmetic for every practical input,
// including points that fall exactly on a buffer edge.
#pragma once

#include <cstdint>
#include <cuda_runtime.h>

namespace gb {

constexpr int kWarp = 32;

// FP64 multiply / add that are never fused into an FMA: positions computed in
// FP64 must round exactly like the reference's separate operations (a fused
// product-sum turns an exact cancellation into a 1e-20 residue, which moves
// points off exact buffer-edge ties).  Host code is built with -ffp-contract=off.
__host__ __device__ __forceinline__ double dmul(double a, double b) {
#ifdef __CUDA_ARCH__
  return __dmul_rn(a, b);
#else
  return a * b;
#endif
}
__host__ __device__ __forceinline__ double dadd(double a, double b) {
#ifdef __CUDA_ARCH__
  return __dadd_rn(a, b);
#else
  return a + b;
#endif
}

// ---------------------------------------------------------------------------
// Programmatic dependent launch.  The kernels of one evaluation run back to
// back on a stream; each one after the first is launched with programmatic
// stream serialization, so its blocks may be scheduled while its predecessor
// drains.  griddep_wait() blocks until the predecessor grids have completed
// and their memory writes are visible (a no-op for a normal launch); nothing
// before it may touch global memory that a predecessor reads or writes.
// griddep_launch_dependents() lets the next kernel's blocks be scheduled.
__device__ __forceinline__ void griddep_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
__device__ __forceinline__ void griddep_launch_dependents() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }

// ---------------------------------------------------------------------------
// Kahan-compensated FP32 accumulator (the reference's CompensatedSummation,
// Core/Common/include/itkCompensatedSummation.hxx:38-48, at FP32).
struct KahanF {
  float s, c;
  __device__ __forceinline__ void zero() { s = 0.f; c = 0.f; }
  __device__ __forceinline__ void add(float x) {
    const float y = __fsub_rn(x, c);
    const float t = __fadd_rn(s, y);
    c = __fsub_rn(__fsub_rn(t, s), y);  // _rn intrinsics are never contracted or reassociated
    s = t;
  }
  __device__ __forceinline__ float value() const { return s - c; }
};

__device__ __forceinline__ float warp_sum(float v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}

__device__ __forceinline__ double warp_sum_d(double v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}

__device__ __forceinline__ unsigned warp_sum_u(unsigned v) { return __reduce_add_sync(0xffffffffu, v); }

// ---------------------------------------------------------------------------
// Cubic B-spline Parzen window (order 3).  With the window starting at bin
// pdfm = midx - 1 and t = term - midx in [0, 1], the four arguments are
// -1-t, -t, 1-t, 2-t; BSplineKernelFunction<3> (Core/Common/include/itkBSplineKernelFunction.h:152-169)
// and BSplineDerivativeKernelFunction<3> (itkBSplineDerivativeKernelFunction.h:156-180)
// evaluated there are the uniform cubic B-spline basis polynomials below.

// 6 * beta3(arg_k), k = 0..3 (integer coefficients: no rounding of 1/6)
__device__ __forceinline__ void parzen6(float t, float w6[4]) {
  const float u = 1.f - t;
  const float t2 = t * t, t3 = t2 * t;
  w6[0] = u * u * u;
  w6[1] = fmaf(3.f, t3, fmaf(-6.f, t2, 4.f));
  w6[2] = fmaf(-3.f, t3, fmaf(3.f, t2, fmaf(3.f, t, 1.f)));
  w6[3] = t3;
}

// beta3'(arg_k), k = 0..3
__device__ __forceinline__ void parzen_deriv(float t, float d[4]) {
  const float u = 1.f - t;
  d[0] = 0.5f * u * u;
  d[1] = t * fmaf(-1.5f, t, 2.f);
  d[2] = u * fmaf(1.5f, u, -2.f);
  d[3] = -0.5f * t * t;
}

// ---------------------------------------------------------------------------
// A continuous index as its nearest integer b = floor(cidx + 0.5) and the
// centred remainder f = cidx - b in [-0.5, 0.5).  Positions close to a voxel
// centre keep full relative precision in f, and the buffer test becomes exact.
struct CIdx {
  int b[3];
  float f[3];
};

// ImageFunction::IsInsideBuffer: cidx in [-0.5, n - 0.5) per axis, NaN outside
// (Core/ImageFunction/include/itkImageFunction.h:157-169).  With b the
// round-half-up index, cidx >= -0.5 <=> b >= 0 and cidx < n - 0.5 <=> b <= n - 1.
__device__ __forceinline__ bool ci_inside(const CIdx& c, int nx, int ny, int nz) {
  const float any = __fadd_rn(__fadd_rn(c.f[0], c.f[1]), c.f[2]);  // NaN if one is (|f| <= 1/2 otherwise)
  return any == any && (unsigned)c.b[0] < (unsigned)nx && (unsigned)c.b[1] < (unsigned)ny &&
         (unsigned)c.b[2] < (unsigned)nz;
}

// Corner indices and weights of LinearInterpolateImageFunction's 3-D path
// (Core/ImageFunction/include/itkLinearInterpolateImageFunction.h:227-470):
// trilinear interpolation with neighbours clamped to the buffer, an axis with
// distance <= 0 below the start contributing the start voxel only.  Measured
// from the nearest voxel b, the second corner is b + sign(f) with weight |f|.
struct Stencil {
  int x0, x1, y0, y1, z0, z1;
  float dx, dy, dz;
};

__device__ __forceinline__ void stencil_axis(int b, float f, int n, int& i0, int& i1, float& w) {
  i0 = b;
  int j = f > 0.f ? b + 1 : (f < 0.f ? b - 1 : b);
  j = j < 0 ? 0 : (j > n - 1 ? n - 1 : j);
  i1 = j;
  w = fabsf(f);
}

__device__ __forceinline__ Stencil make_stencil(const CIdx& c, int nx, int ny, int nz) {
  Stencil s;
  stencil_axis(c.b[0], c.f[0], nx, s.x0, s.x1, s.dx);
  stencil_axis(c.b[1], c.f[1], ny, s.y0, s.y1, s.dy);
  stencil_axis(c.b[2], c.f[2], nz, s.z0, s.z1, s.dz);
  return s;
}

__device__ __forceinline__ float lerp(float a, float b, float t) { return fmaf(b - a, t, a); }

// Two FP32 values in a register pair, and one instruction on both (each rounded as its
// scalar form, so results do not depend on which form computed them).  The FP32 units take
// two cycles for a pair, but the warp issues one instruction instead of two: the per-sample
// loops are bound by issue (430 to 870 instructions a sample at the start, a third to half
// of them FP32), and the slots go to their integer and memory instructions.
typedef unsigned long long f32x2;
__device__ __forceinline__ f32x2 pair(float a, float b) {
  f32x2 r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(a), "f"(b));
  return r;
}
__device__ __forceinline__ f32x2 pair(float a) { return pair(a, a); }
__device__ __forceinline__ void unpair(f32x2 v, float& a, float& b) { asm("mov.b64 {%0, %1}, %2;" : "=f"(a), "=f"(b) : "l"(v)); }
__device__ __forceinline__ f32x2 add2(f32x2 a, f32x2 b) {
  f32x2 r;
  asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
  return r;
}
__device__ __forceinline__ f32x2 sub2(f32x2 a, f32x2 b) {
  f32x2 r;
  asm("sub.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
  return r;
}
__device__ __forceinline__ f32x2 mul2(f32x2 a, f32x2 b) {
  f32x2 r;
  asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
  return r;
}
__device__ __forceinline__ f32x2 fma2(f32x2 a, f32x2 b, f32x2 c) {
  f32x2 r;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
  return r;
}
__device__ __forceinline__ f32x2 lerp2(f32x2 a, f32x2 b, f32x2 t) { return fma2(sub2(b, a), t, a); }
// lerp of four values held as two pairs
__device__ __forceinline__ ulonglong2 lerp4(ulonglong2 a, ulonglong2 b, f32x2 t) {
  return make_ulonglong2(lerp2(a.x, b.x, t), lerp2(a.y, b.y, t));
}

// KahanF on a pair of sums.
struct KahanF2 {
  f32x2 s, c;
  __device__ __forceinline__ void zero() { s = c = 0ull; }
  __device__ __forceinline__ void add(f32x2 x) {
    const f32x2 y = sub2(x, c);
    const f32x2 t = add2(s, y);
    c = sub2(sub2(t, s), y);
    s = t;
  }
  __device__ __forceinline__ void split(KahanF& a, KahanF& b) const {
    unpair(s, a.s, b.s);
    unpair(c, a.c, b.c);
  }
};

// Trilinear gather of the packed (value, gx, gy, gz) moving image.
__device__ __forceinline__ float4 gather4(const float4* __restrict__ img, const Stencil& s, int nx, int ny) {
  // 32-bit offsets: volumes are limited to 2^31 voxels at set-up
  const unsigned sy = (unsigned)nx, sz = (unsigned)nx * (unsigned)ny;
  const unsigned r00 = s.z0 * sz + s.y0 * sy, r10 = s.z0 * sz + s.y1 * sy;
  const unsigned r01 = s.z1 * sz + s.y0 * sy, r11 = s.z1 * sz + s.y1 * sy;
  const ulonglong2* q = reinterpret_cast<const ulonglong2*>(img);  // (value, gx), (gy, gz)
  const ulonglong2 v000 = __ldg(q + r00 + s.x0), v100 = __ldg(q + r00 + s.x1);
  const ulonglong2 v010 = __ldg(q + r10 + s.x0), v110 = __ldg(q + r10 + s.x1);
  const ulonglong2 v001 = __ldg(q + r01 + s.x0), v101 = __ldg(q + r01 + s.x1);
  const ulonglong2 v011 = __ldg(q + r11 + s.x0), v111 = __ldg(q + r11 + s.x1);
  const f32x2 dx = pair(s.dx), dy = pair(s.dy), dz = pair(s.dz);
  const ulonglong2 x00 = lerp4(v000, v100, dx), x10 = lerp4(v010, v110, dx);
  const ulonglong2 x01 = lerp4(v001, v101, dx), x11 = lerp4(v011, v111, dx);
  const ulonglong2 xx0 = lerp4(x00, x10, dy), xx1 = lerp4(x01, x11, dy);
  const ulonglong2 r = lerp4(xx0, xx1, dz);
  float4 o;
  unpair(r.x, o.x, o.y);
  unpair(r.y, o.z, o.w);
  return o;
}

// Trilinear gather of a scalar image.
__device__ __forceinline__ float gather1(const float* __restrict__ img, const Stencil& s, int nx, int ny) {
  const unsigned sy = (unsigned)nx, sz = (unsigned)nx * (unsigned)ny;
  const unsigned r00 = s.z0 * sz + s.y0 * sy, r10 = s.z0 * sz + s.y1 * sy;
  const unsigned r01 = s.z1 * sz + s.y0 * sy, r11 = s.z1 * sz + s.y1 * sy;
  const float v000 = __ldg(img + r00 + s.x0), v100 = __ldg(img + r00 + s.x1);
  const float v010 = __ldg(img + r10 + s.x0), v110 = __ldg(img + r10 + s.x1);
  const float v001 = __ldg(img + r01 + s.x0), v101 = __ldg(img + r01 + s.x1);
  const float v011 = __ldg(img + r11 + s.x0), v111 = __ldg(img + r11 + s.x1);
  const float x00 = lerp(v000, v100, s.dx), x10 = lerp(v010, v110, s.dx);
  const float x01 = lerp(v001, v101, s.dx), x11 = lerp(v011, v111, s.dx);
  const float xx0 = lerp(x00, x10, s.dy), xx1 = lerp(x01, x11, s.dy);
  return lerp(xx0, xx1, s.dz);
}

// ---------------------------------------------------------------------------
// double-float helpers

__device__ __forceinline__ void two_sum(float a, float b, float& s, float& e) {
  s = __fadd_rn(a, b);
  const float bb = __fsub_rn(s, a);
  e = __fadd_rn(__fsub_rn(a, __fsub_rn(s, bb)), __fsub_rn(b, bb));
}

// A position as unevaluated sums hi + lo per axis (|lo| <= ulp(hi) / 2).
struct DFPos {
  float hi[3], lo[3];
};

// Affine map virtual point -> moving continuous index, as FP32 hi/lo pairs:
// cidx_k = sum_j (hi + lo)(k, j) x_j + (bhi + blo)(k).  Rows 0 and 1 lie in pairs, six
// 16-byte words in all: (hi0j, hi1j, lo0j, lo1j) for j = 0..2, (bhi0, bhi1, blo0, blo1),
// (hi20, lo20, hi21, lo21), (hi22, lo22, bhi2, blo2).
struct __align__(16) AffineDF {
  float v[24];
  static constexpr int kHi(int k, int j) { return k < 2 ? 4 * j + k : 16 + 2 * j; }
  static constexpr int kLo(int k, int j) { return k < 2 ? 4 * j + 2 + k : 17 + 2 * j; }
  static constexpr int kBhi(int k) { return k < 2 ? 12 + k : 22; }
  static constexpr int kBlo(int k) { return k < 2 ? 14 + k : 23; }
  __host__ __device__ float& hi(int k, int j) { return v[kHi(k, j)]; }
  __host__ __device__ float& lo(int k, int j) { return v[kLo(k, j)]; }
  __host__ __device__ float& bhi(int k) { return v[kBhi(k)]; }
  __host__ __device__ float& blo(int k) { return v[kBlo(k)]; }
  __host__ __device__ float hi(int k, int j) const { return v[kHi(k, j)]; }
  __host__ __device__ float lo(int k, int j) const { return v[kLo(k, j)]; }
  __host__ __device__ float bhi(int k) const { return v[kBhi(k)]; }
  __host__ __device__ float blo(int k) const { return v[kBlo(k)]; }
};

__device__ __forceinline__ void two_sum2(f32x2 a, f32x2 b, f32x2& s, f32x2& e) {
  s = add2(a, b);
  const f32x2 bb = sub2(s, a);
  e = add2(sub2(a, sub2(s, bb)), sub2(b, bb));
}

// Unevaluated sums s + err per axis, renormalized.
__device__ __forceinline__ DFPos df_renorm(f32x2 s01, f32x2 e01, float s2, float e2) {
  DFPos r;
  const f32x2 hi = add2(s01, e01);
  unpair(hi, r.hi[0], r.hi[1]);
  unpair(sub2(e01, sub2(hi, s01)), r.lo[0], r.lo[1]);
  r.hi[2] = __fadd_rn(s2, e2);
  r.lo[2] = __fsub_rn(e2, __fsub_rn(r.hi[2], s2));
  return r;
}

// Continuous index of one float point to ~1e-12 voxel: products by FMA error
// terms, sums by two-sum.  K in shared memory.
__device__ __forceinline__ DFPos map_pos(const AffineDF& K, float x, float y, float z) {
  const ulonglong2* q = reinterpret_cast<const ulonglong2*>(K.v);
  const float4* w = reinterpret_cast<const float4*>(K.v);
  const float xs[3] = {x, y, z};
  const ulonglong2 b01 = q[3];
  const float4 r0 = w[4], r1 = w[5];
  const float hi2[3] = {r0.x, r0.z, r1.x}, lo2[3] = {r0.y, r0.w, r1.y};
  f32x2 s01 = b01.x, e01 = b01.y;
  float s2 = r1.z, e2 = r1.w;
#pragma unroll
  for (int j = 0; j < 3; ++j) {
    const ulonglong2 A = q[j];
    const f32x2 X = pair(xs[j]), nX = pair(-xs[j]);
    const f32x2 p = mul2(A.x, X);
    const f32x2 npe = fma2(A.x, nX, p);  // exact product error, negated
    f32x2 t, e;
    two_sum2(s01, p, t, e);
    s01 = t;
    e01 = add2(e01, sub2(e, fma2(A.y, nX, npe)));
    const float p2 = __fmul_rn(hi2[j], xs[j]);
    const float pe2 = __fmaf_rn(hi2[j], xs[j], -p2);
    float t2, u2;
    two_sum(s2, p2, t2, u2);
    s2 = t2;
    e2 = __fadd_rn(e2, __fadd_rn(u2, __fmaf_rn(lo2[j], xs[j], pe2)));
  }
  return df_renorm(s01, e01, s2, e2);
}

// Nearest integer b = floor(hi + lo + 0.5) and the remainder hi + lo - b.  hi - rint(hi)
// is exact; lo, at most half an ulp of hi, decides the ties and the crossings next to them
// (the differences from 1/2 are exact there).
__device__ __forceinline__ void split_nearest(float hi, float lo, int& b, float& f) {
  const float r = rintf(hi);
  const float d = __fsub_rn(hi, r);
  const float adj = lo >= __fsub_rn(0.5f, d) ? 1.f : (lo < __fsub_rn(-0.5f, d) ? -1.f : 0.f);
  b = (int)__fadd_rn(r, adj);  // saturates for huge values: outside any buffer
  f = __fadd_rn(__fsub_rn(d, adj), lo);
}

__device__ __forceinline__ CIdx to_cidx(const DFPos& p) {
  CIdx c;
#pragma unroll
  for (int k = 0; k < 3; ++k) split_nearest(p.hi[k], p.lo[k], c.b[k], c.f[k]);
  return c;
}

__device__ __forceinline__ CIdx map_df(const AffineDF& K, float x, float y, float z) {
  return to_cidx(map_pos(K, x, y, z));
}

// p + (dhi + dlo) per axis, renormalized.
__device__ __forceinline__ DFPos df_offset(const DFPos& p, const float* dhi, const float* dlo, float sign) {
  DFPos r;
#pragma unroll
  for (int k = 0; k < 3; ++k) {
    float s, e;
    two_sum(p.hi[k], sign * dhi[k], s, e);
    e = __fadd_rn(e, __fadd_rn(p.lo[k], sign * dlo[k]));
    r.hi[k] = __fadd_rn(s, e);
    r.lo[k] = __fsub_rn(e, __fsub_rn(r.hi[k], s));
  }
  return r;
}

// A double as an unevaluated float pair hi + lo by integer operations only (no
// FP64 instruction): hi is the double truncated to 24 significant bits, lo the
// remaining 29 bits rounded to float, so hi + lo = x within 2^-47 |x|.
// |x| < 2^-126 gives 0 (lo is 0 below 2^-74); |x| >= 2^128, inf and NaN give NaN.
__device__ __forceinline__ void split_double_bits(double x, float& hi, float& lo) {
  const unsigned long long b = (unsigned long long)__double_as_longlong(x);
  const unsigned w1 = (unsigned)(b >> 32), w0 = (unsigned)b;
  const unsigned sign = w1 & 0x80000000u;
  const int e = (int)((w1 >> 20) & 0x7ffu);  // biased exponent
  if (e < 897) {
    hi = 0.f;
    lo = 0.f;
    return;
  }
  if (e > 1150) {
    hi = __int_as_float(0x7fc00000);
    lo = 0.f;
    return;
  }
  hi = __uint_as_float(sign | ((unsigned)(e - 896) << 23) | ((w1 & 0xfffffu) << 3) | (w0 >> 29));
  lo = e < 949 ? 0.f : __uint2float_rn(w0 & 0x1fffffffu) * __uint_as_float(sign | ((unsigned)(e - 948) << 23));
}

// p + A u for a double-float matrix A (in shared memory) and a double-float vector u
// (products with FMA error terms, sums by two-sum), renormalized.
__device__ __forceinline__ DFPos df_add_matvec(const DFPos& p, const AffineDF& K, const float uhi[3],
                                               const float ulo[3]) {
  const ulonglong2* q = reinterpret_cast<const ulonglong2*>(K.v);
  const float4* w = reinterpret_cast<const float4*>(K.v);
  const float4 r0 = w[4];
  const float2 r1 = *reinterpret_cast<const float2*>(K.v + 20);
  const float hi2[3] = {r0.x, r0.z, r1.x}, lo2[3] = {r0.y, r0.w, r1.y};
  f32x2 s01 = pair(p.hi[0], p.hi[1]), e01 = pair(p.lo[0], p.lo[1]);
  float s2 = p.hi[2], e2 = p.lo[2];
#pragma unroll
  for (int j = 0; j < 3; ++j) {
    const ulonglong2 A = q[j];
    const f32x2 U = pair(uhi[j]), nU = pair(-uhi[j]), nL = pair(-ulo[j]);
    const f32x2 v = mul2(A.x, U);
    const f32x2 nve = fma2(A.x, nU, v);  // exact product error, negated
    f32x2 t, e;
    two_sum2(s01, v, t, e);
    s01 = t;
    e01 = add2(e01, sub2(e, add2(nve, fma2(A.y, nU, mul2(A.x, nL)))));
    const float v2 = __fmul_rn(hi2[j], uhi[j]);
    const float ve2 = __fmaf_rn(hi2[j], uhi[j], -v2);
    float t2, u2;
    two_sum(s2, v2, t2, u2);
    s2 = t2;
    e2 = __fadd_rn(e2, __fadd_rn(u2, __fadd_rn(ve2, __fmaf_rn(lo2[j], uhi[j], __fmul_rn(hi2[j], ulo[j])))));
  }
  return df_renorm(s01, e01, s2, e2);
}

// ---------------------------------------------------------------------------
// Ordered-int encodings of floats for atomic min/max.
__device__ __forceinline__ int float_to_ordered(float f) {
  int i = __float_as_int(f);
  return i >= 0 ? i : i ^ 0x7fffffff;
}
__device__ __forceinline__ float ordered_to_float(int i) {
  return __int_as_float(i >= 0 ? i : i ^ 0x7fffffff);
}

// 21-bit-per-axis Morton interleave (x fastest bit).
__device__ __forceinline__ uint64_t morton_spread(uint64_t v) {
  v &= 0x1fffff;
  v = (v | v << 32) & 0x1f00000000ffffULL;
  v = (v | v << 16) & 0x1f0000ff0000ffULL;
  v = (v | v << 8) & 0x100f00f00f00f00fULL;
  v = (v | v << 4) & 0x10c30c30c30c30c3ULL;
  v = (v | v << 2) & 0x1249249249249249ULL;
  return v;
}
__device__ __forceinline__ uint64_t morton3(uint32_t x, uint32_t y, uint32_t z) {
  return morton_spread(x) | (morton_spread(y) << 1) | (morton_spread(z) << 2);
}

}  // namespace gb
