// gb_filters.cu -- device forms of the per-level image filters of the
// registration method and of the metric's default moving-gradient filter:
// recursive-Gaussian smoothing, recursive-Gaussian gradient, shrink geometry.
//
// Reference semantics (paths relative to ITK's Modules/):
//   RecursiveGaussianImageFilter coefficients   Filtering/Smoothing/include/itkRecursiveGaussianImageFilter.hxx:56-300
//   RecursiveSeparableImageFilter line filter   Filtering/ImageFilterBase/include/itkRecursiveSeparableImageFilter.hxx:60-150
//   SmoothingRecursiveGaussianImageFilter       Filtering/Smoothing/include/itkSmoothingRecursiveGaussianImageFilter.hxx
//   GradientRecursiveGaussianImageFilter        Filtering/ImageGradient/include/itkGradientRecursiveGaussianImageFilter.hxx:160-270
//   ShrinkImageFilter geometry                  Filtering/ImageGrid/include/itkShrinkImageFilter.hxx:230-290
//   metric's default gradient filter settings   Registration/Metricsv4/include/itkImageToImageMetricv4.hxx:488-503
//
// A 1-D pass keeps whole image lines in shared memory: a block copies a tile of
// lines in once, runs the causal and the anticausal recursion of each line side by
// side (they start at opposite ends) and writes their sum, so a pass reads and
// writes the image once.  Passes that share their input share the copy, and the
// gradient's last axis forms all three components and the direction product in one
// kernel.  The coefficients come from FP64 on the host; the recursions run in FP32
// (the reference filters in double and, for float images, stores float between the
// smoothing passes).
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <cstring>
#include <type_traits>

#include "gb_device.cuh"
#include "gb_internal.h"

namespace gb {

// IIR coefficients of one pass: N0..N3, D1..D4, M1..M4, BN1..BN4, BM1..BM4.
struct RGCoef {
  double n[4], d[4], m[4], bn[4], bm[4];
};
// The same in FP32 as one recursion that runs in either direction:
//   o_s = sum_{k=0..3} a_k u_{s-k} - sum_{k=1..4} d_k o_{s-k},
// u the inputs in the direction's order (causal), or those one element behind (anticausal).
// Before the line, u is its first element, and an output that is not there yet enters as
// that element times b_k.
struct RGTaps {
  float a[4], d[4], b[4];
};
struct RGCoefF {
  RGTaps dir[2];  // causal, anticausal
};

// Deriche-style recursive Gaussian with the parameters of Farneback and
// Westin ("Improving Deriche-style recursive Gaussian filters", Table 3) and
// the reference's normalizations: order 0 (smoothing) or 1 (first derivative).
static int rg_setup(double sigma, double spacing, int order, bool normalize_across_scale, RGCoef& c) {
  double direction = 1.0;
  if (spacing < 0.0) {
    direction = -1.0;
    spacing = -spacing;
  }
  if (spacing < 1e-8 || !(sigma > 0.0) || (order != 0 && order != 1)) return GB_ERR_BAD_ARG;
  const double sd = sigma / spacing;  // sigma in voxels
  // exponential-series parameters: A, B per order, W, L per pair
  const double A1 = order == 0 ? 1.3530 : -0.6724, B1 = order == 0 ? 1.8151 : -3.4327;
  const double A2 = order == 0 ? -0.3531 : 0.6724, B2 = order == 0 ? 0.0902 : 0.6100;
  const double W1 = 0.6681, L1 = -1.3932, W2 = 2.0787, L2 = -1.3732;
  const double cos1 = std::cos(W1 / sd), cos2 = std::cos(W2 / sd);
  const double sin1 = std::sin(W1 / sd), sin2 = std::sin(W2 / sd);
  const double e1 = std::exp(L1 / sd), e2 = std::exp(L2 / sd);
  // denominator: poles of the two second-order sections
  c.d[3] = e1 * e1 * e2 * e2;
  c.d[2] = -2 * cos1 * e1 * e2 * e2;
  c.d[2] += -2 * cos2 * e2 * e1 * e1;
  c.d[1] = 4 * cos2 * cos1 * e1 * e2;
  c.d[1] += e1 * e1 + e2 * e2;
  c.d[0] = -2 * (e2 * cos2 + e1 * cos1);
  const double SD = 1.0 + c.d[0] + c.d[1] + c.d[2] + c.d[3];
  const double DD = c.d[0] + 2 * c.d[1] + 3 * c.d[2] + 4 * c.d[3];
  // numerator of the causal part
  c.n[0] = A1 + A2;
  c.n[1] = e2 * (B2 * sin2 - (A2 + 2 * A1) * cos2);
  c.n[1] += e1 * (B1 * sin1 - (A1 + 2 * A2) * cos1);
  c.n[2] = (A1 + A2) * cos2 * cos1;
  c.n[2] -= B1 * cos2 * sin1 + B2 * cos1 * sin2;
  c.n[2] *= 2 * e1 * e2;
  c.n[2] += A2 * e1 * e1 + A1 * e2 * e2;
  c.n[3] = e2 * e1 * e1 * (B2 * sin2 - A2 * cos2);
  c.n[3] += e1 * e2 * e2 * (B1 * sin1 - A1 * cos1);
  const double SN = c.n[0] + c.n[1] + c.n[2] + c.n[3];
  const double DN = c.n[1] + 2 * c.n[2] + 3 * c.n[3];
  // normalization: unit gain (order 0) / unit slope response (order 1, times sigma across scales)
  double alpha;
  double scale = 1.0;
  if (order == 0) {
    alpha = 2 * SN / SD - c.n[0];
  } else {
    if (normalize_across_scale) scale = sigma;
    alpha = 2 * (SN * DD - DN * SD) / (SD * SD) * direction;
  }
  for (int k = 0; k < 4; ++k) c.n[k] *= scale / alpha;
  // anticausal numerator: symmetric for order 0, antisymmetric for order 1
  const double sgn = order == 0 ? 1.0 : -1.0;
  c.m[0] = sgn * (c.n[1] - c.d[0] * c.n[0]);
  c.m[1] = sgn * (c.n[2] - c.d[1] * c.n[0]);
  c.m[2] = sgn * (c.n[3] - c.d[2] * c.n[0]);
  c.m[3] = sgn * (-c.d[3] * c.n[0]);
  // edge extension
  const double sn = c.n[0] + c.n[1] + c.n[2] + c.n[3];
  const double sm = c.m[0] + c.m[1] + c.m[2] + c.m[3];
  const double sdd = 1.0 + c.d[0] + c.d[1] + c.d[2] + c.d[3];
  for (int k = 0; k < 4; ++k) {
    c.bn[k] = c.d[k] * sn / sdd;
    c.bm[k] = c.d[k] * sm / sdd;
  }
  return GB_OK;
}

static RGCoefF to_float(const RGCoef& c) {
  RGCoefF f;
  for (int k = 0; k < 4; ++k) {
    f.dir[0].a[k] = (float)c.n[k];
    f.dir[1].a[k] = (float)c.m[k];
    f.dir[0].d[k] = f.dir[1].d[k] = (float)c.d[k];
    f.dir[0].b[k] = (float)c.bn[k];
    f.dir[1].b[k] = (float)c.bm[k];
  }
  return f;
}

__device__ __forceinline__ void copy_async4(float* dst, const float* src) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"((unsigned)__cvta_generic_to_shared(dst)), "l"(src)
               : "memory");
}
__device__ __forceinline__ void copy_async16(float* dst, const float* src) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"((unsigned)__cvta_generic_to_shared(dst)), "l"(src)
               : "memory");
}
// n copies from src, src + hop, ... to dst, dst + inc, ..., their addresses formed ahead in
// groups (a copy holds its address register until it has been read).
template <bool WIDE>
__device__ __forceinline__ void copy_async_rows(float* dst, int inc, const float* src, int64_t hop, int n) {
  constexpr int kGroup = 8;
  for (; n >= kGroup; n -= kGroup) {
    const float* p[kGroup];
#pragma unroll
    for (int u = 0; u < kGroup; ++u) p[u] = src + u * hop;
#pragma unroll
    for (int u = 0; u < kGroup; ++u) WIDE ? copy_async16(dst + u * inc, p[u]) : copy_async4(dst + u * inc, p[u]);
    src += kGroup * hop;
    dst += kGroup * inc;
  }
  for (; n > 0; --n, src += hop, dst += inc) WIDE ? copy_async16(dst, src) : copy_async4(dst, src);
}
__device__ __forceinline__ void copy_async_wait() { asm volatile("cp.async.wait_all;" ::: "memory"); }

// The recursion's state, advanced one element at a time: the last inputs and outputs.  Sums
// and roundings are written out, so that a line's values do not depend on which kernel runs
// it or on what the compiler fuses there.
struct RGLine {
  float p;               // the element behind (anticausal input)
  float u1, u2, u3;      // the last inputs
  float o1, o2, o3, o4;  // the last outputs
  // a0 u + a1 u1 + a2 u2 + a3 u3 (repeated: the first two elements are one, their terms
  // added the other way round)
  __device__ __forceinline__ float inputs(const RGTaps& c, float u, bool repeated) const {
    const float s = repeated ? fmaf(u, c.a[0], __fmul_rn(u1, c.a[1])) : fmaf(u1, c.a[1], __fmul_rn(u, c.a[0]));
    return fmaf(u3, c.a[3], fmaf(u2, c.a[2], s));
  }
  __device__ __forceinline__ float next(float u, float in, float t) {
    const float o = __fsub_rn(in, t);
    u3 = u2;
    u2 = u1;
    u1 = u;
    o4 = o3;
    o3 = o2;
    o2 = o1;
    o1 = o;
    return o;
  }
  // back: whether the recursion is anticausal
  template <typename Back>
  __device__ __forceinline__ float step(const RGTaps& c, float x, Back back) {
    const float u = back ? p : x;
    p = x;
    const float t = fmaf(o4, c.d[3], fmaf(o3, c.d[2], fmaf(o1, c.d[0], __fmul_rn(o2, c.d[1]))));
    return next(u, inputs(c, u, false), t);
  }
  // the line's first four elements
  template <typename Back>
  __device__ __forceinline__ void start(const RGTaps& c, const float (&x)[4], float (&o)[4], Back back) {
    const float v = x[0], x1 = back ? x[0] : x[1], x2 = back ? x[1] : x[2], x3 = back ? x[2] : x[3];
    u1 = u2 = u3 = v;
    o1 = o2 = o3 = o4 = 0.f;
    o[0] = next(v, inputs(c, v, true),
                fmaf(v, c.b[3], fmaf(v, c.b[2], fmaf(v, c.b[0], __fmul_rn(v, c.b[1])))));
    o[1] = next(x1, inputs(c, x1, back), fmaf(v, c.b[3], fmaf(v, c.b[2], fmaf(v, c.b[1], __fmul_rn(o1, c.d[0])))));
    o[2] = next(x2, inputs(c, x2, false),
                fmaf(v, c.b[3], fmaf(v, c.b[2], fmaf(o2, c.d[1], __fmul_rn(o1, c.d[0])))));
    o[3] = next(x3, inputs(c, x3, false),
                fmaf(v, c.b[3], fmaf(o3, c.d[2], fmaf(o2, c.d[1], __fmul_rn(o1, c.d[0])))));
    p = x[3];
  }
};

// `count` elements of one line: x walks the shared-memory input by inc floats; put(outputs)
// takes them in the same order, in groups of kRGRun and then one by one, after put.fetch has
// requested what it adds to the next ones.  The next group of inputs is requested before the present one's outputs are stored (the compiler cannot
// move a load above a store to shared memory).
constexpr int kRGRun = 8;
template <typename Back, typename Put>
__device__ __forceinline__ void rg_run(RGLine& l, const RGTaps& c, Back back, const float*& x, int inc, int count,
                                       Put& put) {
  float v[kRGRun];
  if (count >= kRGRun) {
#pragma unroll
    for (int u = 0; u < kRGRun; ++u) v[u] = x[u * inc];
    put.fetch(kRGRun);
    x += kRGRun * inc;
    for (count -= kRGRun; count >= kRGRun; count -= kRGRun) {
      float w[kRGRun];
#pragma unroll
      for (int u = 0; u < kRGRun; ++u) w[u] = x[u * inc];
      x += kRGRun * inc;
#pragma unroll
      for (int u = 0; u < kRGRun; ++u) v[u] = l.step(c, v[u], back);
      put(v);
      put.fetch(kRGRun);
#pragma unroll
      for (int u = 0; u < kRGRun; ++u) v[u] = w[u];
    }
#pragma unroll
    for (int u = 0; u < kRGRun; ++u) v[u] = l.step(c, v[u], back);
    put(v);
  }
  for (; count > 0; --count, x += inc) {
    put.fetch(1);
    float one[1] = {l.step(c, *x, back)};
    put(one);
  }
}

// The first `count` (>= 4) elements, from the line's start.
template <typename Back, typename Put>
__device__ __forceinline__ void rg_begin(RGLine& l, const RGTaps& c, Back back, const float*& x, int inc, int count,
                                         Put& put) {
  float v[4], o[4];
#pragma unroll
  for (int u = 0; u < 4; ++u) v[u] = x[u * inc];
  l.start(c, v, o, back);
  put(o);
  x += 4 * inc;
  rg_run(l, c, back, x, inc, count - 4, put);
}

// put of a recursion's first half: parked in shared memory.
struct RGPark {
  float* sum;
  int inc;
  __device__ __forceinline__ void fetch(int) {}
  template <int N>
  __device__ __forceinline__ void operator()(const float (&v)[N]) {
#pragma unroll
    for (int u = 0; u < N; ++u) sum[u * inc] = v[u];
    sum += N * inc;
  }
};
// put of its second half: the other recursion's parked part added and scaled, in place.
struct RGAdd {
  float* sum;
  int inc;
  float scale;
  float e[kRGRun];
  __device__ __forceinline__ void fetch(int n) {
#pragma unroll
    for (int u = 0; u < kRGRun; ++u)
      if (u < n) e[u] = sum[u * inc];
  }
  template <int N>
  __device__ __forceinline__ void operator()(const float (&v)[N]) {
#pragma unroll
    for (int u = 0; u < N; ++u) sum[u * inc] = (e[u] + v[u]) * scale;
    sum += N * inc;
  }
};
// The same, written to the output image.
struct RGStore {
  const float* sum;
  int inc;
  float scale;
  float* dst;
  int64_t step;
  bool live;
  float e[kRGRun];
  __device__ __forceinline__ void fetch(int n) {
#pragma unroll
    for (int u = 0; u < kRGRun; ++u)
      if (u < n) e[u] = sum[u * inc];
    sum += n * inc;
  }
  template <int N>
  __device__ __forceinline__ void operator()(const float (&v)[N]) {
#pragma unroll
    for (int u = 0; u < N; ++u)
      if (live) dst[u * step] = (e[u] + v[u]) * scale;
    dst += N * step;
  }
};

// One pass along an axis with NOUT outputs of the same input (NOUT pairs of warps: the
// causal and the anticausal recursion of each output, a thread per line).  A block owns
// kRGLines consecutive lines; line l starts at (l % n1) * s1 + (l / n1) * s2 and has ln
// elements `step` apart.  X: the lines run along x (l * ln, step 1) and lie in shared
// memory at an odd pitch, else element i of the tile's lines is row i: both without bank
// conflicts.  The first `half` outputs of each recursion are parked in shared memory;
// past that the other one has left its part there, and the sum is final.
// One read and NOUT writes of the image; bound by the tiles in flight (8 or 12 bytes of
// shared memory an element: two to four blocks per SM, each copying, filtering and storing
// in turn).  Measured at 256x256x200 (one output along z, x, y; two outputs along x, y):
// 33, 39, 28; 63, 49 us, where one thread per line through global memory took 141, 303,
// 185; 605, 357 us.  A row of 32 lines is copied in 16-byte pieces where the lines come in
// aligned groups of four: 4-byte copies took twice as long to issue.
constexpr int kRGLines = 32;
struct RGOut {
  float* p;
  float scale;
  RGCoefF c;
};
struct RGPass {
  const float* in;
  RGOut out[2];
  int64_t lines, step, n1, s1, s2;
  int ln;
  int wide;  // lines in groups of four at 16-byte boundaries (axes other than x)
};
__host__ __device__ inline int rg_pitch(int ln) { return ln | 1; }  // odd: a column of lines hits every bank
static size_t rg_tile_bytes(bool x, int ln) { return sizeof(float) * kRGLines * (size_t)(x ? rg_pitch(ln) : ln); }

// The recursion DIR (1 causal, -1 anticausal) of output o of the tile's lines, in two halves:
// the block's barrier between them stands in the kernel, where every warp meets it (the
// directions are two branches, and a barrier in either would be one of its own).
struct RGHalf {
  RGLine s;
  const float* x;
  float* sum;
};
template <bool X, int DIR>
__device__ __forceinline__ void rg_first_half(const RGPass& a, float* tile, int o, RGHalf& h) {
  constexpr int kInc = X ? DIR : DIR * kRGLines;
  const int ln = a.ln, lane = threadIdx.x & 31;
  const int pitch = rg_pitch(ln), size = X ? kRGLines * pitch : kRGLines * ln;
  const RGTaps c = a.out[o].c.dir[DIR < 0];
  const int half = DIR < 0 ? ln / 2 : (ln + 1) / 2;
  const int first = X ? lane * pitch + (DIR < 0 ? ln - 1 : 0) : lane + (DIR < 0 ? (ln - 1) * kRGLines : 0);
  h.x = tile + first;
  h.sum = tile + (1 + o) * size + first;
  const std::integral_constant<bool, (DIR < 0)> back{};
  RGPark park{h.sum, kInc};
  rg_begin(h.s, c, back, h.x, kInc, half, park);
  h.sum += half * kInc;
}
template <bool X, int DIR>
__device__ __forceinline__ void rg_second_half(const RGPass& a, int o, RGHalf& h, int64_t base, bool live) {
  constexpr int kInc = X ? DIR : DIR * kRGLines;
  const int ln = a.ln;
  const RGTaps c = a.out[o].c.dir[DIR < 0];
  const float scale = a.out[o].scale;
  const int half = DIR < 0 ? ln / 2 : (ln + 1) / 2;
  const std::integral_constant<bool, (DIR < 0)> back{};
  if (X) {
    RGAdd add{h.sum, kInc, scale};
    rg_run(h.s, c, back, h.x, kInc, ln - half, add);
  } else {
    RGStore store{h.sum, kInc, scale, a.out[o].p + base + (DIR < 0 ? ln - 1 - half : half) * a.step,
                  DIR * a.step, live};
    rg_run(h.s, c, back, h.x, kInc, ln - half, store);
  }
}

template <bool X, int NOUT>
__global__ void __launch_bounds__(64 * NOUT) k_rg_pass(RGPass a) {
  extern __shared__ __align__(16) float tile[];
  const int ln = a.ln, lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int64_t l0 = (int64_t)blockIdx.x * kRGLines, l = l0 + lane;
  const bool live = l < a.lines;
  const int pitch = rg_pitch(ln);
  const int size = X ? kRGLines * pitch : kRGLines * ln;
  const int64_t base = X ? l * ln : (l % a.n1) * a.s1 + (l / a.n1) * a.s2;
  if (X) {
    const int rows = (int)min((int64_t)kRGLines, a.lines - l0);
    for (int r = warp; r < rows; r += 2 * NOUT) {
      const float* src = a.in + (l0 + r) * ln;
      float* dst = tile + r * pitch;
#pragma unroll 4
      for (int i = lane; i < ln; i += 32) copy_async4(dst + i, src + i);
    }
  } else if (a.wide) {  // four lines at a time: a warp copies four rows
    const int64_t w = l0 + 4 * (lane & 7);
    const int i = 4 * warp + (lane >> 3);
    if (w < a.lines && i < ln)
      copy_async_rows<true>(tile + i * kRGLines + 4 * (lane & 7), 8 * NOUT * kRGLines,
                            a.in + (w % a.n1) * a.s1 + (w / a.n1) * a.s2 + i * a.step, 8 * NOUT * a.step,
                            (ln - i + 8 * NOUT - 1) / (8 * NOUT));
  } else if (live && warp < ln) {
    copy_async_rows<false>(tile + warp * kRGLines + lane, 2 * NOUT * kRGLines, a.in + base + warp * a.step,
                           2 * NOUT * a.step, (ln - warp + 2 * NOUT - 1) / (2 * NOUT));
  }
  copy_async_wait();
  __syncthreads();
  // even warps causal, odd ones anticausal; past the middle each adds what the other parked
  RGHalf h;
  if (warp & 1) rg_first_half<X, -1>(a, tile, warp >> 1, h);
  else rg_first_half<X, 1>(a, tile, warp >> 1, h);
  __syncthreads();
  if (warp & 1) rg_second_half<X, -1>(a, warp >> 1, h, base, live);
  else rg_second_half<X, 1>(a, warp >> 1, h, base, live);
  if (X) {
    // rows leave in order
    __syncthreads();
    const int o = warp >> 1, rows = (int)min((int64_t)kRGLines, a.lines - l0);
    const float* sum = tile + (1 + o) * size;
    for (int r = warp & 1; r < rows; r += 2) {
      float* dst = a.out[o].p + (l0 + r) * ln;
      const float* src = sum + r * pitch;
#pragma unroll 4
      for (int i = lane; i < ln; i += 32) dst[i] = src[i];
    }
  }
}

// The same for lines too long for a tile, or too short to meet past both starts (under
// kRGShort elements): one thread per line, the causal part through the output image.
constexpr int kRGShort = 8;
__global__ void __launch_bounds__(128) k_rg_long(RGPass a) {
  const int64_t id = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (id >= a.lines) return;
  const int64_t base = (id % a.n1) * a.s1 + (id / a.n1) * a.s2;
  const float* x = a.in + base;
  float* y = a.out[0].p + base;
  const RGCoefF& c = a.out[0].c;
  RGLine s;
  float v[4], o[4];
  for (int u = 0; u < 4; ++u) v[u] = __ldg(x + u * a.step);
  s.start(c.dir[0], v, o, false);
  for (int u = 0; u < 4; ++u) y[u * a.step] = o[u];
  for (int64_t i = 4; i < a.ln; ++i) y[i * a.step] = s.step(c.dir[0], __ldg(x + i * a.step), false);
  const int64_t last = a.ln - 1;
  for (int u = 0; u < 4; ++u) v[u] = __ldg(x + (last - u) * a.step);
  s.start(c.dir[1], v, o, true);
  for (int u = 0; u < 4; ++u) y[(last - u) * a.step] = (y[(last - u) * a.step] + o[u]) * a.out[0].scale;
  for (int64_t i = last - 4; i >= 0; --i)
    y[i * a.step] = (y[i * a.step] + s.step(c.dir[1], __ldg(x + i * a.step), true)) * a.out[0].scale;
}

// Largest dynamic shared memory of a block.
constexpr size_t kRGMaxShared = 227 * 1024;

// The axis's lines: element step and count, and where line l = (j1, j2) starts; the two
// other axes, the faster-varying one first (x whenever it is not the filtered axis).
static RGPass rg_lines(const float* in, const int64_t size[3], int axis) {
  RGPass a;
  memset(&a, 0, sizeof(a));
  a.in = in;
  a.ln = (int)size[axis];
  a.step = axis == 0 ? 1 : (axis == 1 ? size[0] : size[0] * size[1]);
  const int a1 = axis == 0 ? 1 : 0, a2 = axis == 2 ? 1 : 2;
  a.n1 = size[a1];
  a.s1 = a1 == 0 ? 1 : size[0];
  a.s2 = a2 == 1 ? size[0] : size[0] * size[1];
  a.lines = size[a1] * size[a2];
  a.wide = axis != 0 && size[0] % 4 == 0 && (reinterpret_cast<uintptr_t>(in) & 15) == 0 ? 1 : 0;
  return a;
}

template <bool X, int NOUT>
static cudaError_t rg_launch(cudaStream_t st, const RGPass& a, size_t shared) {
  // the same limit on every call: threads filtering images of different sizes share it
  const cudaError_t e =
      cudaFuncSetAttribute(k_rg_pass<X, NOUT>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kRGMaxShared);
  if (e != cudaSuccess) return e;
  k_rg_pass<X, NOUT><<<(unsigned)((a.lines + kRGLines - 1) / kRGLines), 64 * NOUT, shared, st>>>(a);
  return cudaGetLastError();
}

// nout (1 or 2) filters of one image along an axis.
static cudaError_t rg_pass(cudaStream_t st, const float* in, const int64_t size[3], int axis, const RGOut* out,
                           int nout) {
  RGPass a = rg_lines(in, size, axis);
  const size_t shared = (1 + nout) * rg_tile_bytes(axis == 0, a.ln);
  if (shared > kRGMaxShared || a.ln < kRGShort) {
    if (nout == 2) {
      const cudaError_t e = rg_pass(st, in, size, axis, out, 1);
      return e != cudaSuccess ? e : rg_pass(st, in, size, axis, out + 1, 1);
    }
    a.out[0] = out[0];
    k_rg_long<<<(unsigned)((a.lines + 127) / 128), 128, 0, st>>>(a);
    return cudaGetLastError();
  }
  for (int k = 0; k < nout; ++k) a.out[k] = out[k];
  if (axis == 0) return nout == 1 ? rg_launch<true, 1>(st, a, shared) : rg_launch<true, 2>(st, a, shared);
  return nout == 1 ? rg_launch<false, 1>(st, a, shared) : rg_launch<false, 2>(st, a, shared);
}

// SmoothingRecursiveGaussianImageFilter: zero order along z, then x, then y.
// t1, t2: scratch images of the same size (in may equal out).
int smooth_rg_device(cudaStream_t st, const float* in, float* out, float* t1, float* t2, const int64_t size[3],
                     const double spacing[3], const double sigma[3]) {
  for (int d = 0; d < 3; ++d)
    if (size[d] < 4)
      return fail(GB_ERR_BAD_ARG, "The number of pixels along dimension " + std::to_string(d) +
                                      " is less than 4. This filter requires a minimum of four pixels along the "
                                      "dimension to be processed.");
  RGCoef c;
  const int order[3] = {2, 0, 1};
  const float* src = in;
  float* dst[3] = {t1, t2, out};
  for (int p = 0; p < 3; ++p) {
    const int ax = order[p];
    if (rg_setup(sigma[ax], spacing[ax], 0, false, c) != GB_OK) return fail(GB_ERR_BAD_ARG, "sigma must be > 0");
    const RGOut o{dst[p], 1.f, to_float(c)};
    cudaError_t e = rg_pass(st, src, size, ax, &o, 1);
    if (e != cudaSuccess) return fail(GB_ERR_CUDA, std::string("smoothing pass: ") + cudaGetErrorString(e));
    src = dst[p];
  }
  return GB_OK;
}

// The direction matrix applied to a gradient.
struct RGMatrix {
  float m[9];
  __device__ __forceinline__ float row(int r, float a, float b, float c) const {
    return fmaf(m[3 * r], a, fmaf(m[3 * r + 1], b, m[3 * r + 2] * c));
  }
};

// (value, D (gx, gy, gz)) per voxel, the gradient in physical units.
__global__ void k_pack_gradient(const float* __restrict__ v, const float* __restrict__ gx,
                                const float* __restrict__ gy, const float* __restrict__ gz, int64_t n, RGMatrix m,
                                float4* __restrict__ out4, float* __restrict__ out3) {
  const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const float a = gx[i], b = gy[i], c = gz[i];
  if (out4) out4[i] = make_float4(v[i], m.row(0, a, b, c), m.row(1, a, b, c), m.row(2, a, b, c));
  if (out3)
    for (int r = 0; r < 3; ++r) out3[3 * i + r] = m.row(r, a, b, c);
}

// The gradient's last axis (z), its direction product and its packing in one kernel: the
// three components' lines of a tile of kRGzLines lines, one warp per component (lanes
// 0-15 the causal, 16-31 the anticausal recursion of the tile's lines), then float4
// (value, gradient) or xyz triplets, each voxel's output written once.  Kept apart, the
// three passes would write 12 and read 12 bytes a voxel more.  Element k from a line's
// start lies in row 2k and element k from its end in row 2k + 1: both recursions walk
// rows upwards to the middle and downwards past it by the same stride, in different banks.
// 12 (with the value 16) bytes read and 12 or 16 written per voxel; bound as k_rg_pass is.
// Measured at 256x256x200: 118 us (triplets), where three passes and the packing took 485.
constexpr int kRGzLines = 16;
struct RGGradZ {
  const float* in[3];
  const float* v;
  RGOut out[3];  // p unused
  RGMatrix m;
  int64_t lines, step;
  int ln;
  int wide;  // lines in groups of four at 16-byte boundaries
  float4* out4;
  float* out3;
};
static size_t rgz_array(int ln) { return (size_t)kRGzLines * (size_t)ln; }

__global__ void __launch_bounds__(96) k_rg_grad_z(RGGradZ a) {
  extern __shared__ __align__(16) float tile[];
  constexpr int kInc = 2 * kRGzLines;
  const int ln = a.ln, lane = threadIdx.x & 31, comp = threadIdx.x >> 5;
  const int line = lane & (kRGzLines - 1), back = lane >> 4;
  const int size = kRGzLines * ln, half = ln / 2;
  const int64_t l0 = (int64_t)blockIdx.x * kRGzLines;
  const int64_t dir = back ? -a.step : a.step;                               // this lane's way along its line
  const int64_t begin = l0 + line + (back ? (int64_t)(ln - 1) * a.step : 0);
  const int mine = half + ((ln & 1) && !back ? 1 : 0);                       // rows of this parity
  float* const xs = tile + 2 * comp * size + lane;
  if (a.wide) {  // four lines at a time: a warp copies eight rows, the same way along each line
    const int p = lane >> 2, w = 4 * (lane & 3);
    const int64_t hop = (p & 1) ? -4 * a.step : 4 * a.step;
    const int64_t from = l0 + w + ((p & 1) ? ln - 1 - (p >> 1) : p >> 1) * a.step;
    if (l0 + w < a.lines && p < ln) {
      copy_async_rows<true>(tile + 2 * comp * size + p * kRGzLines + w, 8 * kRGzLines, a.in[comp] + from, hop,
                            (ln - p + 7) / 8);
      if (a.out4 && p + 8 * comp < ln)
        copy_async_rows<true>(tile + 6 * size + (p + 8 * comp) * kRGzLines + w, 24 * kRGzLines,
                              a.v + from + comp * hop, 3 * hop, (ln - p - 8 * comp + 23) / 24);
    }
  } else if (l0 + line < a.lines) {
    copy_async_rows<false>(xs, kInc, a.in[comp] + begin, dir, mine);
    if (a.out4 && comp < mine)
      copy_async_rows<false>(tile + 6 * size + lane + comp * kInc, 3 * kInc, a.v + begin + comp * dir, 3 * dir,
                             (mine - comp + 2) / 3);
  }
  copy_async_wait();
  __syncwarp();  // a warp's recursions read what the same warp has copied
  RGTaps c;  // this lane's direction, by selection: no divergent copies
#pragma unroll
  for (int k = 0; k < 4; ++k) {
    c.a[k] = back ? a.out[comp].c.dir[1].a[k] : a.out[comp].c.dir[0].a[k];
    c.b[k] = back ? a.out[comp].c.dir[1].b[k] : a.out[comp].c.dir[0].b[k];
    c.d[k] = a.out[comp].c.dir[0].d[k];
  }
  const float scale = a.out[comp].scale;
  const float* x = xs;
  RGLine s;
  RGPark park{xs + size, kInc};
  rg_begin(s, c, back != 0, x, kInc, half, park);
  __syncwarp();
  if (ln & 1) {  // the middle element, the last row, for both
    float* m = xs - lane + size + (ln - 1) * kRGzLines + line;
    const float v = s.step(c, xs[(ln - 1) * kRGzLines - lane + line], back != 0);
    if (!back) *m = v;
    __syncwarp();
    if (back) *m = (*m + v) * scale;
  }
  // past the middle: the other recursion's rows, from the last one down
  const int last = (half - 1) * kInc - lane + (lane ^ kRGzLines);
  x = xs + last;
  RGAdd add{xs + size + last, -kInc, scale};
  rg_run(s, c, back != 0, x, -kInc, half, add);
  __syncthreads();
  const float *g0 = tile + size, *g1 = tile + 3 * size, *g2 = tile + 5 * size, *v0 = tile + 6 * size;
  constexpr int kOut = 8;  // rows read together
  if (a.out4 && l0 + line < a.lines) {  // thread t: line t % 16 of every sixth row from t / 16
    const int p = threadIdx.x >> 4;
    const int64_t hop = (p & 1) ? -3 * a.step : 3 * a.step;
    float4* dst = a.out4 + l0 + line + ((p & 1) ? ln - 1 - (p >> 1) : p >> 1) * a.step;
    for (int q = threadIdx.x; q < size; q += 96 * kOut, dst += kOut * hop) {
      float4 o[kOut];
#pragma unroll
      for (int u = 0; u < kOut; ++u)
        if (q + 96 * u < size) o[u] = make_float4(v0[q + 96 * u], g0[q + 96 * u], g1[q + 96 * u], g2[q + 96 * u]);
#pragma unroll
      for (int u = 0; u < kOut; ++u)
        if (q + 96 * u < size)
          dst[u * hop] = make_float4(o[u].x, a.m.row(0, o[u].y, o[u].z, o[u].w), a.m.row(1, o[u].y, o[u].z, o[u].w),
                                     a.m.row(2, o[u].y, o[u].z, o[u].w));
    }
  }
  if (a.out3) {  // a row's 48 floats in order: thread t % 48 writes component t % 3 of line t / 3
    const int p = threadIdx.x / (3 * kRGzLines), t = threadIdx.x % (3 * kRGzLines), r = t % 3, w = t / 3;
    const float m0 = a.m.m[3 * r], m1 = a.m.m[3 * r + 1], m2 = a.m.m[3 * r + 2];
    const int64_t hop = p ? -3 * a.step : 3 * a.step;
    float* dst = a.out3 + 3 * (l0 + (p ? (int64_t)(ln - 1) * a.step : 0)) + t;
    if (l0 + w < a.lines)
      for (int q = p * kRGzLines + w; q < size; q += kInc * kOut, dst += kOut * hop) {
        float o[kOut];
#pragma unroll
        for (int u = 0; u < kOut; ++u)
          if (q + kInc * u < size) o[u] = fmaf(m0, g0[q + kInc * u], fmaf(m1, g1[q + kInc * u], m2 * g2[q + kInc * u]));
#pragma unroll
        for (int u = 0; u < kOut; ++u)
          if (q + kInc * u < size) dst[u * hop] = o[u];
      }
  }
}

// GradientRecursiveGaussianImageFilter: component d = first order along d and
// zero order along the other axes, / spacing[d], then the direction matrix.
// The zero-order x pass and the y passes are shared between components.
// Writes float4 (value, gradient) and/or xyz float triplets.
int gradient_rg_device(cudaStream_t st, const float* in, const int64_t size[3], const double spacing[3],
                       const double direction[9], double sigma, bool normalize_across_scale, bool use_direction,
                       float4* out4, float* out3) {
  for (int d = 0; d < 3; ++d)
    if (size[d] < 4)
      return fail(GB_ERR_BAD_ARG, "The number of pixels along dimension " + std::to_string(d) +
                                      " is less than 4. This filter requires a minimum of four pixels along the "
                                      "dimension to be processed.");
  const int64_t n = size[0] * size[1] * size[2];
  float* buf = nullptr;
  cudaError_t e = cudaMallocAsync(reinterpret_cast<void**>(&buf), sizeof(float) * 5 * (size_t)n, st);
  if (e != cudaSuccess) return fail(GB_ERR_OUT_OF_MEMORY, "gradient filter scratch: out of device memory");
  float *A = buf, *B = buf + n, *C = buf + 2 * n, *D = buf + 3 * n, *E = buf + 4 * n;
  RGCoefF s[3], dv[3];
  int rc = GB_OK;
  for (int k = 0; k < 3 && rc == GB_OK; ++k) {
    RGCoef c;
    rc = rg_setup(sigma, spacing[k], 0, normalize_across_scale, c);
    s[k] = to_float(c);
    if (rc == GB_OK) rc = rg_setup(sigma, spacing[k], 1, normalize_across_scale, c);
    dv[k] = to_float(c);
  }
  if (rc != GB_OK) {
    cudaFreeAsync(buf, st);
    return fail(GB_ERR_BAD_ARG, "sigma must be > 0");
  }
  const float inv[3] = {(float)(1.0 / spacing[0]), (float)(1.0 / spacing[1]), (float)(1.0 / spacing[2])};
  RGMatrix m{{1, 0, 0, 0, 1, 0, 0, 0, 1}};
  if (use_direction)
    for (int k = 0; k < 9; ++k) m.m[k] = (float)direction[k];
  // x: A = Dx I, B = Sx I; y: C = Sy A, D = Dy B, E = Sy B;
  // z: gx = Sz C / sx, gy = Sz D / sy, gz = Dz E / sz
  const RGOut ox[2] = {{A, 1.f, dv[0]}, {B, 1.f, s[0]}};
  const RGOut oy[3] = {{C, 1.f, s[1]}, {D, 1.f, dv[1]}, {E, 1.f, s[1]}};
  e = rg_pass(st, in, size, 0, ox, 2);
  if (e == cudaSuccess) e = rg_pass(st, A, size, 1, oy, 1);
  if (e == cudaSuccess) e = rg_pass(st, B, size, 1, oy + 1, 2);
  const size_t shared = sizeof(float) * rgz_array((int)size[2]) * (out4 ? 7 : 6);
  if (shared <= kRGMaxShared && size[2] >= kRGShort) {
    RGGradZ z;
    memset(&z, 0, sizeof(z));
    z.in[0] = C;
    z.in[1] = D;
    z.in[2] = E;
    z.v = in;
    for (int k = 0; k < 3; ++k) z.out[k] = RGOut{nullptr, inv[k], k < 2 ? s[2] : dv[2]};
    z.m = m;
    z.lines = size[0] * size[1];
    z.step = z.lines;
    z.ln = (int)size[2];
    z.wide = n % 4 == 0 && z.lines % 4 == 0 && (reinterpret_cast<uintptr_t>(in) & 15) == 0 ? 1 : 0;
    z.out4 = out4;
    z.out3 = out3;
    if (e == cudaSuccess)
      e = cudaFuncSetAttribute(k_rg_grad_z, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kRGMaxShared);
    if (e == cudaSuccess) {
      k_rg_grad_z<<<(unsigned)((z.lines + kRGzLines - 1) / kRGzLines), 96, shared, st>>>(z);
      e = cudaGetLastError();
    }
  } else {
    const RGOut oz[3] = {{A, inv[0], s[2]}, {B, inv[1], s[2]}, {C, inv[2], dv[2]}};
    const float* iz[3] = {C, D, E};  // C is read before it is written
    for (int k = 0; k < 3; ++k)
      if (e == cudaSuccess) e = rg_pass(st, iz[k], size, 2, oz + k, 1);
    if (e == cudaSuccess) {
      k_pack_gradient<<<(unsigned)((n + 255) / 256), 256, 0, st>>>(in, A, B, C, n, m, out4, out3);
      e = cudaGetLastError();
    }
  }
  cudaFreeAsync(buf, st);
  if (e != cudaSuccess) return fail(GB_ERR_CUDA, std::string("gradient filter: ") + cudaGetErrorString(e));
  return GB_OK;
}

// ShrinkImageFilter::GenerateOutputInformation (start index 0): output spacing
// spacing * f, size floor(size / f) (at least 1), origin moved so that the
// image centre stays put.
void shrink_geometry(const int64_t size[3], const double spacing[3], const double origin[3], const double dir[9],
                     const int64_t factors[3], int64_t out_size[3], double out_spacing[3], double out_origin[3]) {
  double in_c[3], out_c[3];
  for (int i = 0; i < 3; ++i) {
    const int64_t f = factors[i] < 1 ? 1 : factors[i];
    out_spacing[i] = spacing[i] * (double)f;
    out_size[i] = std::max<int64_t>(1, (int64_t)std::floor((double)size[i] / (double)f));
    in_c[i] = (double)(size[i] - 1) / 2.0;
    out_c[i] = (double)(out_size[i] - 1) / 2.0;
  }
  for (int r = 0; r < 3; ++r) {
    double s_in = 0.0, s_out = 0.0;  // continuous index -> point: the sum, then the origin
    for (int c = 0; c < 3; ++c) {
      s_in += dir[r * 3 + c] * spacing[c] * in_c[c];
      s_out += dir[r * 3 + c] * out_spacing[c] * out_c[c];
    }
    out_origin[r] = origin[r] + ((s_in + origin[r]) - (s_out + origin[r]));
  }
}

}  // namespace gb

using namespace gb;

extern "C" int gb_smooth_recursive_gaussian(gb_ctx* ctx, uint64_t stream, const float* d_in, float* d_out,
                                            const int64_t size[3], const double spacing[3], const double sigma[3]) {
  if (!ctx || !d_in || !d_out || !size || !spacing || !sigma) return fail(GB_ERR_BAD_ARG, "null argument");
  if (cudaSetDevice(ctx->device) != cudaSuccess) return fail(GB_ERR_CUDA, "cudaSetDevice failed");
  cudaStream_t st = reinterpret_cast<cudaStream_t>(static_cast<uintptr_t>(stream));
  const int64_t n = size[0] * size[1] * size[2];
  float* tmp = nullptr;
  if (cudaMallocAsync(reinterpret_cast<void**>(&tmp), sizeof(float) * 2 * (size_t)n, st) != cudaSuccess)
    return fail(GB_ERR_OUT_OF_MEMORY, "smoothing scratch: out of device memory");
  const int rc = smooth_rg_device(st, d_in, d_out, tmp, tmp + n, size, spacing, sigma);
  cudaFreeAsync(tmp, st);
  return rc;
}

extern "C" int gb_gradient_recursive_gaussian(gb_ctx* ctx, uint64_t stream, const float* d_in, float* d_out_xyz,
                                              const int64_t size[3], const double spacing[3],
                                              const double direction[9], double sigma, int normalize_across_scale,
                                              int use_image_direction) {
  if (!ctx || !d_in || !d_out_xyz || !size || !spacing || !direction) return fail(GB_ERR_BAD_ARG, "null argument");
  if (cudaSetDevice(ctx->device) != cudaSuccess) return fail(GB_ERR_CUDA, "cudaSetDevice failed");
  cudaStream_t st = reinterpret_cast<cudaStream_t>(static_cast<uintptr_t>(stream));
  return gradient_rg_device(st, d_in, size, spacing, direction, sigma, normalize_across_scale != 0,
                            use_image_direction != 0, nullptr, d_out_xyz);
}

// Host-buffer forms: copy in, run the device filter, copy out (synchronous).
extern "C" int gb_smooth_recursive_gaussian_host(gb_ctx* ctx, const float* in, float* out, const int64_t size[3],
                                                 const double spacing[3], const double sigma[3]) {
  if (!ctx || !in || !out || !size || !spacing || !sigma) return fail(GB_ERR_BAD_ARG, "null argument");
  if (cudaSetDevice(ctx->device) != cudaSuccess) return fail(GB_ERR_CUDA, "cudaSetDevice failed");
  const int64_t n = size[0] * size[1] * size[2];
  DevBuf<float> d;
  if (d.alloc(3 * (size_t)n) != cudaSuccess) return fail(GB_ERR_OUT_OF_MEMORY, "smoothing: out of device memory");
  if (cudaMemcpy(d.p, in, sizeof(float) * n, cudaMemcpyHostToDevice) != cudaSuccess)
    return fail(GB_ERR_CUDA, "smoothing: copy in failed");
  int rc = smooth_rg_device(0, d.p, d.p, d.p + n, d.p + 2 * n, size, spacing, sigma);
  if (rc == GB_OK && cudaMemcpy(out, d.p, sizeof(float) * n, cudaMemcpyDeviceToHost) != cudaSuccess)
    rc = fail(GB_ERR_CUDA, "smoothing: copy out failed");
  return rc;
}

extern "C" int gb_gradient_recursive_gaussian_host(gb_ctx* ctx, const float* in, float* out_xyz,
                                                   const int64_t size[3], const double spacing[3],
                                                   const double direction[9], double sigma,
                                                   int normalize_across_scale, int use_image_direction) {
  if (!ctx || !in || !out_xyz || !size || !spacing || !direction) return fail(GB_ERR_BAD_ARG, "null argument");
  if (cudaSetDevice(ctx->device) != cudaSuccess) return fail(GB_ERR_CUDA, "cudaSetDevice failed");
  const int64_t n = size[0] * size[1] * size[2];
  DevBuf<float> d;
  if (d.alloc(4 * (size_t)n) != cudaSuccess) return fail(GB_ERR_OUT_OF_MEMORY, "gradient: out of device memory");
  if (cudaMemcpy(d.p, in, sizeof(float) * n, cudaMemcpyHostToDevice) != cudaSuccess)
    return fail(GB_ERR_CUDA, "gradient: copy in failed");
  int rc = gradient_rg_device(0, d.p, size, spacing, direction, sigma, normalize_across_scale != 0,
                              use_image_direction != 0, nullptr, d.p + n);
  if (rc == GB_OK && cudaMemcpy(out_xyz, d.p + n, sizeof(float) * 3 * n, cudaMemcpyDeviceToHost) != cudaSuccess)
    rc = fail(GB_ERR_CUDA, "gradient: copy out failed");
  return rc;
}

extern "C" int gb_shrink_geometry(const int64_t size[3], const double spacing[3], const double origin[3],
                                  const double direction[9], const int64_t factors[3], int64_t out_size[3],
                                  double out_spacing[3], double out_origin[3]) {
  if (!size || !spacing || !origin || !direction || !factors || !out_size || !out_spacing || !out_origin)
    return fail(GB_ERR_BAD_ARG, "null argument");
  shrink_geometry(size, spacing, origin, direction, factors, out_size, out_spacing, out_origin);
  return GB_OK;
}
