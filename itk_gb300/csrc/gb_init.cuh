// gb_init.cuh -- Initialize()-time kernels: image ranges, the device sample
// list (fixed values / fixed Parzen bins in FP64), packing of the moving image.
#pragma once

#include <cfloat>

#include "gb_device.cuh"

namespace gb {

// FP64 trilinear interpolation with the reference's clamps
// (Core/ImageFunction/include/itkLinearInterpolateImageFunction.h:227-470);
// used once per Initialize for the fixed image, so its value equals the
// reference's double interpolation rounded to float.
__device__ __forceinline__ double interp_d(const float* __restrict__ img, const int64_t n[3], const double ci[3]) {
  int64_t b0[3], b1[3];
  double d[3];
#pragma unroll
  for (int k = 0; k < 3; ++k) {
    int64_t f = __double2ll_rd(ci[k]);
    if (f < 0) f = 0;
    double dist = ci[k] - (double)f;
    b0[k] = f;
    b1[k] = f + 1 <= n[k] - 1 ? f + 1 : f;
    if (!(dist > 0.0)) { dist = 0.0; b1[k] = f; }
    d[k] = dist;
  }
  const int64_t nx = n[0], nxy = n[0] * n[1];
#define GBPIX(x, y, z) ((double)img[(x) + (y) * nx + (z) * nxy])
  const double v000 = GBPIX(b0[0], b0[1], b0[2]), v100 = GBPIX(b1[0], b0[1], b0[2]);
  const double v010 = GBPIX(b0[0], b1[1], b0[2]), v110 = GBPIX(b1[0], b1[1], b0[2]);
  const double v001 = GBPIX(b0[0], b0[1], b1[2]), v101 = GBPIX(b1[0], b0[1], b1[2]);
  const double v011 = GBPIX(b0[0], b1[1], b1[2]), v111 = GBPIX(b1[0], b1[1], b1[2]);
#undef GBPIX
  if (d[0] <= 0.0 && d[1] <= 0.0 && d[2] <= 0.0) return v000;
  // a + (b - a) d with separate roundings, as the reference computes it
#define GBLERP(a, b, t) dadd((a), dmul(dadd((b), -(a)), (t)))
  const double x00 = GBLERP(v000, v100, d[0]);
  const double x10 = GBLERP(v010, v110, d[0]);
  const double x01 = GBLERP(v001, v101, d[0]);
  const double x11 = GBLERP(v011, v111, d[0]);
  const double xx0 = GBLERP(x00, x10, d[1]);
  const double xx1 = GBLERP(x01, x11, d[1]);
  return GBLERP(xx0, xx1, d[2]);
#undef GBLERP
}

struct DGeom {
  int64_t n[3];
  double origin[3];
  double i2p[9];
  double p2i[9];
  int diag;  // both matrices are diagonal
};

// Initialize's kernels are bound by FP64 (about 1.7 operations per SM and clock), so an
// axis-aligned grid's products with exact zeros are left out (the same sums).
__device__ __forceinline__ void d_point_to_cindex(const DGeom& g, const double p[3], double ci[3]) {
  double v[3];
#pragma unroll
  for (int k = 0; k < 3; ++k) v[k] = dadd(p[k], -g.origin[k]);
  if (g.diag) {
#pragma unroll
    for (int i = 0; i < 3; ++i) ci[i] = dmul(g.p2i[4 * i], v[i]);
    return;
  }
#pragma unroll
  for (int i = 0; i < 3; ++i) {
    double s = 0.0;
    for (int j = 0; j < 3; ++j) s = dadd(s, dmul(g.p2i[3 * i + j], v[j]));
    ci[i] = s;
  }
}

__device__ __forceinline__ bool d_inside(const DGeom& g, const double ci[3]) {
#pragma unroll
  for (int k = 0; k < 3; ++k)
    if (!(ci[k] >= -0.5 && ci[k] < (double)(g.n[k] - 1) + 0.5)) return false;
  return true;
}

// TransformPhysicalPointToIndex (round half up) + inside test, itkImageBase.h:463-479
__device__ __forceinline__ bool d_nearest_of(const DGeom& g, const double ci[3], int64_t idx[3]) {
  bool inside = true;
#pragma unroll
  for (int i = 0; i < 3; ++i) {
    idx[i] = __double2ll_rd(dadd(ci[i], 0.5));
    if (idx[i] < 0 || idx[i] >= g.n[i]) inside = false;
  }
  return inside;
}
__device__ __forceinline__ bool d_nearest_index(const DGeom& g, const double p[3], int64_t idx[3]) {
  double ci[3];
  d_point_to_cindex(g, p, ci);
  return d_nearest_of(g, ci, idx);
}

// Physical point -> continuous index with every coefficient as an FP32 pair.
struct DFMap {
  float hi[9], lo[9], bhi[3], blo[3];
  float size[3];  // sum of |coefficient * origin|, at least |b|
  float unit;     // error of an index / (size + sum of |coefficient * point|)
  int n[3];
};

// One point's continuous index c in FP32 pairs.  An FP64 instruction of a warp takes some 19
// cycles of its SM, an FP32 one a quarter of a cycle, so Initialize takes the point's index
// and value this way and leaves to FP64 only the points whose result could differ: `sure`
// says that floor, rounding and the buffer test are those of the FP64 index, whose distance
// from this one is at most err.  NaN and infinity are never sure.
//
// With u = 2^-24, B the sum of |coefficient * origin| and A the |coefficient * point| in order:
// the coefficients' pairs lose u^2 (B + A1 + A2 + A3), the products' errors 2 u^2 (A1 + A2 + A3),
// the additions u + qe and then to e (|e| reaches u (4B + 5A1 + 4A2 + 3A3)) u^2 (12B + 17A1 + 11A2
// + 6A3), the last pair u |e| (where e exceeds s), and t and its pair 3 u^2: below 2^-43 of the
// sum.  With one product to a row those are 4B + 9A1, 2B + 3A1 and 3: below 2^-44.
struct DFIndex {
  int floor[3], nearest[3];
  float t[3], tl[3];  // c - floor in [0, 1], as a pair
  float err[3];
  bool sure;
};

__device__ __forceinline__ DFIndex df_index(const DFMap& M, const float p[3]) {
  DFIndex c;
  c.sure = true;
#pragma unroll
  for (int r = 0; r < 3; ++r) {
    float s = M.bhi[r], e = M.blo[r], size = M.size[r];
#pragma unroll
    for (int k = 0; k < 3; ++k) {
      const float q = __fmul_rn(M.hi[3 * r + k], p[k]);
      const float qe = __fmaf_rn(M.lo[3 * r + k], p[k], __fmaf_rn(M.hi[3 * r + k], p[k], -q));
      float sum, u;
      two_sum(s, q, sum, u);
      s = sum;
      e = __fadd_rn(e, __fadd_rn(u, qe));
      size += fabsf(q);
    }
    const float err = size * M.unit;
    const float hi = __fadd_rn(s, e), lo = __fsub_rn(e, __fsub_rn(hi, s));
    const float f = floorf(hi);
    float t, tl, d, dl;
    two_sum(hi, -f, d, dl);  // not exact between -1 and 0 without its error
    two_sum(d, __fadd_rn(lo, dl), t, tl);
    const bool below = t < 0.f;  // hi is whole and lo negative
    if (below) {
      float u;
      two_sum(1.f, t, t, u);
      tl += u;
    }
    c.floor[r] = (int)f - (below ? 1 : 0);
    const float half = __fadd_rn(__fsub_rn(t, 0.5f), tl);
    c.nearest[r] = c.floor[r] + (half >= 0.f ? 1 : 0);
    c.t[r] = t;
    c.tl[r] = tl;
    c.err[r] = err;
    c.sure = c.sure && fabsf(hi) < 4194304.f && t > 2.f * err &&
             __fsub_rn(__fsub_rn(1.f, t), tl) > 2.f * err && fabsf(half) > 2.f * err;
  }
  return c;
}

__device__ __forceinline__ bool df_inside(const DFMap& M, const DFIndex& c) {
  return (unsigned)c.nearest[0] < (unsigned)M.n[0] && (unsigned)c.nearest[1] < (unsigned)M.n[1] &&
         (unsigned)c.nearest[2] < (unsigned)M.n[2];
}

struct DFVal {
  float h, l;
};
__device__ __forceinline__ DFVal df_lerp(const DFVal& a, const DFVal& b, float t, float tl) {
  float d, dl, s, e;
  two_sum(b.h, -a.h, d, dl);
  dl = __fadd_rn(dl, __fsub_rn(b.l, a.l));
  const float q = __fmul_rn(d, t);
  const float qe = __fadd_rn(__fmaf_rn(d, t, -q), __fmaf_rn(d, tl, __fmul_rn(dl, t)));
  two_sum(a.h, q, s, e);
  e = __fadd_rn(e, __fadd_rn(qe, a.l));
  const float h = __fadd_rn(s, e);
  return {h, __fsub_rn(e, __fsub_rn(h, s))};
}

// interp_d rounded to float; false if the pairs' error leaves the rounding open.  The
// interpolation is linear along each axis, so an index's error moves the value by at most err
// times the largest difference along that axis; the interpolations themselves lose 26 u^2 of
// the largest corner along x and 53 u^2 each along y and z (u = 2^-24; 2^-40 is 256).
__device__ __forceinline__ bool df_interp(const float* __restrict__ img, const DFMap& M, const DFIndex& c, float& out) {
  int b0[3], b1[3];
  float t[3], tl[3];
#pragma unroll
  for (int k = 0; k < 3; ++k) {
    const bool low = c.floor[k] < 0;
    b0[k] = low ? 0 : c.floor[k];
    b1[k] = low ? 0 : min(b0[k] + 1, M.n[k] - 1);
    t[k] = low ? 0.f : c.t[k];
    tl[k] = low ? 0.f : c.tl[k];
  }
  const int64_t nx = M.n[0], nxy = nx * M.n[1];
  float v[8], lo = FLT_MAX, hi = -FLT_MAX;
#pragma unroll
  for (int k = 0; k < 8; ++k) {
    v[k] = img[(k & 1 ? b1[0] : b0[0]) + (k & 2 ? b1[1] : b0[1]) * nx + (k & 4 ? b1[2] : b0[2]) * nxy];
    lo = fminf(lo, v[k]);
    hi = fmaxf(hi, v[k]);
  }
  const DFVal x00 = df_lerp({v[0], 0.f}, {v[1], 0.f}, t[0], tl[0]), x10 = df_lerp({v[2], 0.f}, {v[3], 0.f}, t[0], tl[0]);
  const DFVal x01 = df_lerp({v[4], 0.f}, {v[5], 0.f}, t[0], tl[0]), x11 = df_lerp({v[6], 0.f}, {v[7], 0.f}, t[0], tl[0]);
  const DFVal xx0 = df_lerp(x00, x10, t[1], tl[1]), xx1 = df_lerp(x01, x11, t[1], tl[1]);
  const DFVal r = df_lerp(xx0, xx1, t[2], tl[2]);
  const float range = hi - lo, big = fmaxf(fabsf(lo), fabsf(hi));
  float e = 0x1p-40f * big;
#pragma unroll
  for (int r = 0; r < 3; ++r) {
    const int x = 1 << r, y = r == 0 ? 2 : 1, z = r == 2 ? 2 : 4;  // this axis, the others
    const float slope = fmaxf(fmaxf(fabsf(v[x] - v[0]), fabsf(v[x + y] - v[y])),
                              fmaxf(fabsf(v[x + z] - v[z]), fabsf(v[x + y + z] - v[y + z])));
    e = fmaf(c.err[r], slope, e);
  }
  out = __fadd_rn(r.h, __fadd_rn(r.l, e));
  const bool flat = range == 0.f;  // eight equal values (a background): that value
  if (flat) out = __fadd_rn(v[0], 0.f);
  return (flat && r.h == r.h) || (out == __fadd_rn(r.h, __fsub_rn(r.l, e)) && big > 1e-25f && big < 1e30f);
}

struct BuildArgs {
  const float* points;  // sampled points (xyz) or nullptr for the dense virtual grid
  int64_t n;            // candidates
  int points_virtual;
  DGeom virt, fixed;
  DFMap virt_df, fixed_df;
  int same_grid;  // virt and fixed are one grid
  int cell_shift;  // sort keys: B-spline cell above this bit, spatial order below it
  const float* fixed_img;
  // B-spline support (transform kinds 1, 2)
  int bspline;
  int64_t grid[3];
  double g_origin[3];
  double g_p2i[9];
  uint64_t* keys;
  uint32_t* vals;
  float4* recs;
  float4* sup;  // B-spline support record per candidate (null without a B-spline)
  uint32_t* voff;  // nearest virtual voxel per candidate, ~0u outside (displacement field on a point set; else null)
  unsigned long long* nvalid;
};

__device__ __forceinline__ int64_t dbl_ulp_order(double x) {
  long long i = __double_as_longlong(x);
  if (i < 0) i = (long long)0x8000000000000000LL - i;
  return i;
}

// BSplineTransform::InsideValidRegion, Core/Transform/include/itkBSplineTransform.hxx:478-507
__device__ __forceinline__ bool d_bspline_inside(const int64_t grid[3], double ci[3]) {
  const double minLimit = 1.0;
#pragma unroll
  for (int j = 0; j < 3; ++j) {
    const double maxLimit = (double)grid[j] - 1.0 - 1.0;
    bool almost = fabs(ci[j] - maxLimit) <= 0.1 * DBL_EPSILON;
    if (!almost && (signbit(ci[j]) == signbit(maxLimit))) {
      long long d = dbl_ulp_order(ci[j]) - dbl_ulp_order(maxLimit);
      if (d < 0) d = -d;
      almost = d <= 4;
    }
    if (almost) ci[j] = __longlong_as_double(__double_as_longlong(maxLimit) - 6);
    else if (ci[j] >= maxLimit) return false;
    else if (ci[j] < minLimit) return false;
  }
  return true;
}

// One candidate sample: virtual point -> fixed value (FP64 interpolation,
// TransformAndEvaluateFixedPoint, itkImageToImageMetricv4.hxx:290-322).  Invalid candidates
// get a key of ones and sort last.
//
// Bound by FP64 before (327k points 84 us); points go through FP32 pairs now, with the same
// floats and keys (22 us).  The dense grid's points are whole indices, next to every
// threshold, and stay with FP64.
__device__ __forceinline__ bool build_sample(const BuildArgs& b, int64_t i) {
  double vp[3];
  float pt[3] = {0.f, 0.f, 0.f};
  bool ok = true, sure = false;
  float fval = 0.f;
  int64_t vi[3];  // nearest virtual voxel
  if (b.points) {
#pragma unroll
    for (int k = 0; k < 3; ++k) {
      pt[k] = b.points[3 * i + k];
      vp[k] = 0.0;
    }
    const DFIndex f = df_index(b.fixed_df, pt);
    DFIndex v = f;
    if (!b.same_grid) v = df_index(b.virt_df, pt);
    sure = f.sure && v.sure;
    if (sure) {
      ok = df_inside(b.fixed_df, f) && (b.points_virtual || df_inside(b.virt_df, v));
      if (ok) sure = df_interp(b.fixed_img, b.fixed_df, f, fval);
#pragma unroll
      for (int k = 0; k < 3; ++k) vi[k] = v.nearest[k];
    }
    if (!sure || b.bspline || b.voff)
#pragma unroll
      for (int k = 0; k < 3; ++k) vp[k] = pt[k];
  }
  if (!sure) {
    ok = true;
    if (b.points) {
      // MapFixedSampledPointSetToVirtual keeps points whose nearest virtual index is inside, .hxx:594-607
      if (!b.points_virtual) ok = d_nearest_index(b.virt, vp, vi);
    } else {
      const int64_t nx = b.virt.n[0], ny = b.virt.n[1];
      const double idx[3] = {(double)(i % nx), (double)((i / nx) % ny), (double)(i / (nx * ny))};
#pragma unroll
      for (int r = 0; r < 3; ++r) {
        double p = b.virt.origin[r];
        if (b.virt.diag) p = dadd(p, dmul(b.virt.i2p[4 * r], idx[r]));
        else
          for (int c = 0; c < 3; ++c) p = dadd(p, dmul(b.virt.i2p[3 * r + c], idx[c]));
        vp[r] = p;
      }
    }
    if (ok) {
      double ci[3];
      d_point_to_cindex(b.fixed, vp, ci);
      ok = d_inside(b.fixed, ci);
      if (ok) {
        fval = (float)interp_d(b.fixed_img, b.fixed.n, ci);
        if (b.same_grid) d_nearest_of(b.virt, ci, vi);
        else d_nearest_index(b.virt, vp, vi);
      }
    }
  }
  // B-spline support of the virtual point (BSplineTransform::TransformPoint,
  // itkBSplineTransform.hxx:510-591): in-cell positions t = ci - start - 1 in
  // [0, 1] and the start node packed as sx | sy << 10 | sz << 20 | valid << 30;
  // cell = 1 + start's linear node index (0: outside the valid region).
  float4 sup = make_float4(0.f, 0.f, 0.f, 0.f);
  uint64_t cell = 0;
  if (ok && b.bspline) {
    double gi[3], v[3];
#pragma unroll
    for (int k = 0; k < 3; ++k) v[k] = dadd(vp[k], -b.g_origin[k]);
#pragma unroll
    for (int r = 0; r < 3; ++r) {
      double s = 0.0;
      for (int j = 0; j < 3; ++j) s = dadd(s, dmul(b.g_p2i[3 * r + j], v[j]));
      gi[r] = s;
    }
    if (d_bspline_inside(b.grid, gi)) {
      int st[3];
      float t[3];
#pragma unroll
      for (int k = 0; k < 3; ++k) {
        st[k] = (int)floor(dadd(dadd(gi[k], 0.5), -1.5));  // BSplineInterpolationWeightFunction start index
        t[k] = (float)dadd(dadd(gi[k], -(double)st[k]), -1.0);
      }
      const unsigned packed = (unsigned)st[0] | ((unsigned)st[1] << 10) | ((unsigned)st[2] << 20) | (1u << 30);
      sup = make_float4(t[0], t[1], t[2], __uint_as_float(packed));
      cell = 1 + (uint64_t)st[0] + (uint64_t)b.grid[0] * ((uint64_t)st[1] + (uint64_t)b.grid[1] * (uint64_t)st[2]);
    }
  }
  uint64_t key = ~0ull;
  if (ok) {
    const uint32_t x = (uint32_t)(vi[0] < 0 ? 0 : vi[0]);
    const uint32_t y = (uint32_t)(vi[1] < 0 ? 0 : vi[1]);
    const uint32_t z = (uint32_t)(vi[2] < 0 ? 0 : vi[2]);
    // 8 x 2 x 2 bricks of the virtual grid in Morton order, scan order inside a
    // brick: a warp's samples cover long x runs over few (y, z) rows, so the
    // trilinear gathers of one load instruction touch few 128-byte lines
    const uint64_t brick = morton3((x >> 3) & 0xfff, (y >> 1) & 0xfff, (z >> 1) & 0xfff) & ((1ull << 36) - 1);
    key = (brick << 5) | ((uint64_t)(z & 1) << 4) | ((uint64_t)(y & 1) << 3) | (uint64_t)(x & 7) |
          (cell << b.cell_shift);
  }
  b.keys[i] = key;
  b.vals[i] = (uint32_t)i;
  // domain coordinates: the point for a point set, the exact grid index for the dense domain
  if (b.points) b.recs[i] = make_float4(pt[0], pt[1], pt[2], fval);
  else b.recs[i] = make_float4((float)(i % b.virt.n[0]), (float)((i / b.virt.n[0]) % b.virt.n[1]),
                               (float)(i / (b.virt.n[0] * b.virt.n[1])), fval);
  if (b.sup) b.sup[i] = sup;
  if (b.voff) {
    // the derivative block's voxel: TransformPhysicalPointToIndex of the point
    // (ImageToImageMetricv4GetValueAndDerivativeThreader.hxx:58), with
    // ComputeParameterOffsetFromVirtualIndex (itkObjectToObjectMetric.hxx:332-343)
    const bool in = d_nearest_index(b.virt, vp, vi);
    b.voff[i] = in ? (uint32_t)(vi[0] + b.virt.n[0] * (vi[1] + b.virt.n[1] * vi[2])) : 0xffffffffu;
  }
  return ok;
}

__global__ void __launch_bounds__(kBlock) k_build_samples(const __grid_constant__ BuildArgs b) {
  const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  const bool ok = i < b.n && build_sample(b, i);
  const int valid = __syncthreads_count(ok);
  if (threadIdx.x == 0 && valid) atomicAdd(b.nvalid, (unsigned long long)valid);
}

// The samples in sorted order; for Mattes, the fixed value's Parzen bin takes its place
// (ComputeSingleFixedImageParzenWindowIndex, Mattes...v4.hxx:571-597).
struct FixedBins {
  int bins;  // 0: keep the value
  double bs, normmin;
  float inv_bs_f, normmin_f;
};
__device__ __forceinline__ int fixed_bin(const FixedBins& b, float fval) {
  // the integer part by FP32, or by the reference's FP64 division where an integer is near:
  // the FP32 error is below 2^-23 of |fval / bs| + |normmin|, rounded twice
  const float q = fval * b.inv_bs_f;
  const float term = q - b.normmin_f;
  const float err = 0x1p-21f * (fabsf(q) + fabsf(b.normmin_f));
  long long p;
  if (fabsf(term) < 65536.f && fabsf(term - rintf(term)) > err) p = (long long)term;
  else p = (long long)((double)fval / b.bs - b.normmin);
  if (p < 2) p = 2;
  else if (p > b.bins - 3) p = b.bins - 3;
  return (int)p;
}

__global__ void k_gather_samples(const uint32_t* __restrict__ perm, int64_t n, const float4* __restrict__ recs,
                                 float4* __restrict__ out, const float4* __restrict__ sup_in,
                                 float4* __restrict__ sup_out, const uint32_t* __restrict__ voff_in,
                                 uint32_t* __restrict__ voff_out, FixedBins fb) {
  const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const uint32_t j = perm[i];
  float4 r = recs[j];
  if (fb.bins) r.w = __int_as_float(fixed_bin(fb, r.w));
  out[i] = r;
  if (sup_out) sup_out[i] = sup_in[j];
  if (voff_out) voff_out[i] = voff_in[j];
}

// Initialize's small results: two min / max pairs as ordered integers, the valid samples.
struct InitStats {
  int range[4];  // fixed min, max, moving min, max
  unsigned long long nvalid;
};
__global__ void k_init_stats(InitStats* s) {
  if (threadIdx.x < 4) s->range[threadIdx.x] = float_to_ordered(threadIdx.x & 1 ? -FLT_MAX : FLT_MAX);
  if (threadIdx.x == 4) s->nvalid = 0;
}

// A block's min / max into out[0], out[1] (one pair of atomics to the block: from every warp
// they queued on the two words).
__device__ __forceinline__ void minmax_block(float lo, float hi, int* out) {
  __shared__ int s_mm[2];
  if (threadIdx.x == 0) {
    s_mm[0] = float_to_ordered(FLT_MAX);
    s_mm[1] = float_to_ordered(-FLT_MAX);
  }
  __syncthreads();
  const int l = __reduce_min_sync(0xffffffffu, float_to_ordered(lo));
  const int h = __reduce_max_sync(0xffffffffu, float_to_ordered(hi));
  if ((threadIdx.x & 31) == 0) {
    atomicMin(&s_mm[0], l);
    atomicMax(&s_mm[1], h);
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    atomicMin(&out[0], s_mm[0]);
    atomicMax(&out[1], s_mm[1]);
  }
}

// min / max over a float buffer: out[0] = min, out[1] = max.  16-byte loads where the buffer
// starts on such a boundary.
__global__ void k_minmax(const float* __restrict__ img, int64_t n, int* out) {
  float lo = FLT_MAX, hi = -FLT_MAX;
  const int64_t first = (int64_t)blockIdx.x * blockDim.x + threadIdx.x, step = (int64_t)gridDim.x * blockDim.x;
  const int64_t n4 = (reinterpret_cast<uintptr_t>(img) & 15) == 0 ? n / 4 : 0;
  const float4* q = reinterpret_cast<const float4*>(img);
#pragma unroll 4
  for (int64_t i = first; i < n4; i += step) {
    const float4 v = __ldg(q + i);
    lo = fminf(fminf(fminf(lo, v.x), fminf(v.y, v.z)), v.w);
    hi = fmaxf(fmaxf(fmaxf(hi, v.x), fmaxf(v.y, v.z)), v.w);
  }
  for (int64_t i = 4 * n4 + first; i < n; i += step) {
    const float v = img[i];
    lo = fminf(lo, v);
    hi = fmaxf(hi, v);
  }
  minmax_block(lo, hi, out);
}

// Mattes fixed range over the sampled points (nearest-index pixel values),
// itkMattesMutualInformationImageToImageMetricv4.hxx:99-153
__global__ void k_minmax_points(const float* __restrict__ pts, int64_t n, const __grid_constant__ DGeom fixed,
                                const __grid_constant__ DFMap fixed_df, const float* __restrict__ img, int* out) {
  float lo = FLT_MAX, hi = -FLT_MAX;
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
    const float pt[3] = {pts[3 * i], pts[3 * i + 1], pts[3 * i + 2]};
    const DFIndex c = df_index(fixed_df, pt);
    int64_t idx[3] = {c.nearest[0], c.nearest[1], c.nearest[2]};
    bool in = df_inside(fixed_df, c);
    if (!c.sure) {
      const double p[3] = {pt[0], pt[1], pt[2]};
      in = d_nearest_index(fixed, p, idx);
    }
    if (in) {
      const float v = img[idx[0] + fixed.n[0] * (idx[1] + fixed.n[1] * idx[2])];
      lo = fminf(lo, v);
      hi = fmaxf(hi, v);
    }
  }
  minmax_block(lo, hi, out);
}

// (value, gx, gy, gz) packing of the moving image and its gradient image
// (CovariantVector<double,3> voxels, rounded to FP32).
__global__ void k_pack_moving(const float* __restrict__ mov, const double* __restrict__ grad, int64_t n,
                              float4* __restrict__ out) {
  const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  float4 v = make_float4(mov[i], 0.f, 0.f, 0.f);
  if (grad) {
    v.y = (float)grad[3 * i];
    v.z = (float)grad[3 * i + 1];
    v.w = (float)grad[3 * i + 2];
  }
  out[i] = v;
}

}  // namespace gb
