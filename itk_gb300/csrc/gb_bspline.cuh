// gb_bspline.cuh -- B-spline (order 3) and [affine, B-spline] composite moving transforms.
//
// Reference semantics (paths relative to ITK's Modules/):
//   BSplineTransform::TransformPoint / Jacobian   Core/Transform/include/itkBSplineTransform.hxx:478-652
//   BSplineInterpolationWeightFunction::Evaluate  Core/Common/include/itkBSplineInterpolationWeightFunction.hxx:43-93
//   CompositeTransform point and chain rule        Core/Transform/include/itkCompositeTransform.hxx:60-70,466-580
//
// Each sample's support (first node, in-cell fractions, valid-region flag) is
// fixed by its virtual point, so Initialize computes it once in FP64 with the
// reference's InsideValidRegion rules.  Per evaluation a sample needs the 64
// tensor weights and the displacement sum over the coefficients (staged in
// shared memory when they fit).  The Jacobian has 192 nonzeros per sample,
//   (J^T g)[n_k + d * nper] = W_k (M^T g)_d,
// M the composite's initial affine (identity for a plain B-spline).  Samples
// are sorted by B-spline cell; a chunk kernel sums W_k a_s over chunks of
// same-cell samples (a lane keeps a plane of the support's nodes), and a gather kernel adds,
// for every parameter, the chunk sums of the cells whose support holds its
// node -- in a fixed order, with no atomics.
#pragma once

#include "gb_kernels.cuh"

namespace gb {

constexpr int kChunkBatch = 256;   // samples staged at a time by the chunk kernel; its block size
constexpr int kChunkLen = 2048;    // samples per chunk (at most)
constexpr int kChunkSlices = 64;   // the chunk kernel's partial sums of a batch
constexpr int kFoldBatches = 4;    // batches to a slice's sum: 16 plain FP32 additions, then pairwise
static_assert(kFoldBatches * kChunkBatch <= 16 * kChunkSlices, "additions that a slice loses bits in");
constexpr int kParamsBlock = 256;  // k_bspline_params: 8 nodes per block (warp form) or 1 (block form)

__device__ __forceinline__ void unpack_support(float w, int& sx, int& sy, int& sz, bool& valid) {
  const unsigned u = __float_as_uint(w);
  sx = (int)(u & 1023u);
  sy = (int)((u >> 10) & 1023u);
  sz = (int)((u >> 20) & 1023u);
  valid = ((u >> 30) & 1u) != 0u;
}

// Weights of the 4 nodes along one axis at in-cell position t in [0, 1]:
// BSplineKernelFunction<3> at t+1, t, t-1, t-2; 1/6 applied as hi + lo parts.
__device__ __forceinline__ void bspline_basis(float t, float* w) {
  constexpr float c_hi = 0.16666667163372039795f;  // nearest float to 1/6
  constexpr float c_lo = -4.96705373e-09f;         // 1/6 - c_hi
  float w6[4];
  parzen6(t, w6);
#pragma unroll
  for (int k = 0; k < 4; ++k) w[k] = fmaf(w6[k], c_hi, w6[k] * c_lo);
}

// One coefficient node (c_x, c_y, c_z, 0) from the FP64 parameters
// (BSplineTransform's parameter layout: all x coefficients, then y, then z).
__device__ __forceinline__ float4 node_from_params(const double* __restrict__ p, int nper, int n) {
  return make_float4((float)__ldg(p + n), (float)__ldg(p + nper + n), (float)__ldg(p + 2 * nper + n), 0.f);
}

#ifndef GB_KERNELS_HELPERS_ONLY
// Float4 node array from device-resident parameters (the host call converts on
// the host and uploads the nodes); one conversion per node per evaluation,
// rather than one per node in every block of the sample pass.
__global__ void k_prepare_bspline(EvalArgs a) {
  griddep_wait();
  if (halted(a)) return;
  griddep_launch_dependents();
  if (a.clear_acc) clear_accumulators(a);
  const int n = blockIdx.x * blockDim.x + threadIdx.x;
  if (n < a.nper) a.nodes[n] = node_from_params(a.params, a.nper, n);
}
#endif  // GB_KERNELS_HELPERS_ONLY

// The nodes in shared memory (SMEM), else the global array.  A compile-time
// choice, so node reads compile to shared-memory loads rather than generic ones.
template <bool SMEM>
__device__ __forceinline__ const float4* stage_nodes(const EvalArgs& a, float4* sh) {
  if constexpr (SMEM) {
    for (int k = threadIdx.x; k < a.nper; k += blockDim.x) sh[k] = __ldcg(a.nodes + k);
    return sh;
  } else {
    return a.nodes;
  }
}

// Displacements of R samples in one cell (start node sx, sy, sz; in-cell positions in su),
// axis by axis, x and y components in pairs.
//
// A warp's 16-byte loads of one node take four cycles of the SM's 128-byte shared-memory path
// whatever the lanes read: 256 cycles for the 64 nodes against some 150 for all of a sample's
// instructions.  Two samples to a thread share them (173x181x149, 20 %, mesh 8: MeanSquares 46.1
// -> 42.0 us; 256x256x200, 40 %, mesh 3: 177 -> 150 us); what remains is the moving image's gathers.
template <int R>
__device__ __forceinline__ void bspline_displacements(const float4* nodes, const EvalArgs& a, int sx, int sy, int sz,
                                                      const float4 su[R], float u[R][3]) {
  float wx[R][4], wy[R][4], wz[R][4];
#pragma unroll
  for (int r = 0; r < R; ++r) {
    bspline_basis(su[r].x, wx[r]);
    bspline_basis(su[r].y, wy[r]);
    bspline_basis(su[r].z, wz[r]);
  }
  f32x2 uxy[R];
#pragma unroll
  for (int kz = 0; kz < 4; ++kz) {
    f32x2 pxy[R];
    float pz[R];
#pragma unroll
    for (int ky = 0; ky < 4; ++ky) {
      const ulonglong2* row =
          reinterpret_cast<const ulonglong2*>(nodes + (sx + a.gx * ((sy + ky) + a.gy * (sz + kz))));
      f32x2 rxy[R];
      float rz[R];
#pragma unroll
      for (int kx = 0; kx < 4; ++kx) {
        const ulonglong2 c = row[kx];  // (x, y), (z, 0)
        float cz, none;
        unpair(c.y, cz, none);
#pragma unroll
        for (int r = 0; r < R; ++r) {
          const f32x2 w = pair(wx[r][kx]);
          rxy[r] = kx == 0 ? mul2(w, c.x) : fma2(w, c.x, rxy[r]);
          rz[r] = kx == 0 ? wx[r][kx] * cz : fmaf(wx[r][kx], cz, rz[r]);
        }
      }
#pragma unroll
      for (int r = 0; r < R; ++r) {
        const f32x2 w = pair(wy[r][ky]);
        pxy[r] = ky == 0 ? mul2(w, rxy[r]) : fma2(w, rxy[r], pxy[r]);
        pz[r] = ky == 0 ? wy[r][ky] * rz[r] : fmaf(wy[r][ky], rz[r], pz[r]);
      }
    }
#pragma unroll
    for (int r = 0; r < R; ++r) {
      const f32x2 w = pair(wz[r][kz]);
      uxy[r] = kz == 0 ? mul2(w, pxy[r]) : fma2(w, pxy[r], uxy[r]);
      u[r][2] = kz == 0 ? wz[r][kz] * pz[r] : fmaf(wz[r][kz], pz[r], u[r][2]);
    }
  }
#pragma unroll
  for (int r = 0; r < R; ++r) unpair(uxy[r], u[r][0], u[r][1]);
}

// Moving continuous indices of R samples under the B-spline (+ initial affine):
// cidx = A x + b + P2I M u, A x + b in double-float, the displacement u in FP32.
// has_jac: inside the B-spline valid region (else the transform is the identity
// there and its Jacobian is zero, itkBSplineTransform.hxx:519-523,610-616).
template <int R>
__device__ __forceinline__ void bspline_positions(const EvalConsts& K, const float4* nodes, const EvalArgs& a,
                                                  const float4 s[R], const float4 su[R], DFPos p[R],
                                                  bool has_jac[R]) {
  float u[R][3];
  int sx, sy, sz;
  unpack_support(su[0].w, sx, sy, sz, has_jac[0]);
  bool together = R > 1;
#pragma unroll
  for (int r = 1; r < R; ++r) together = together && __float_as_uint(su[r].w) == __float_as_uint(su[0].w);
  if (together) {
#pragma unroll
    for (int r = 1; r < R; ++r) has_jac[r] = has_jac[0];
    if (has_jac[0]) bspline_displacements<R>(nodes, a, sx, sy, sz, su, u);
  } else {
#pragma unroll
    for (int r = 0; r < R; ++r) {
      unpack_support(su[r].w, sx, sy, sz, has_jac[r]);
      if (has_jac[r]) bspline_displacements<1>(nodes, a, sx, sy, sz, su + r, u + r);
    }
  }
#pragma unroll
  for (int r = 0; r < R; ++r) {
    p[r] = map_pos(K.map, s[r].x, s[r].y, s[r].z);
    if (!has_jac[r]) continue;
#pragma unroll
    for (int k = 0; k < 3; ++k) {
      const float corr = fmaf(K.Pm[3 * k], u[r][0], fmaf(K.Pm[3 * k + 1], u[r][1], K.Pm[3 * k + 2] * u[r][2]));
      float hs, he;
      two_sum(p[r].hi[k], corr, hs, he);
      he = __fadd_rn(he, p[r].lo[k]);
      p[r].hi[k] = __fadd_rn(hs, he);
      p[r].lo[k] = __fsub_rn(he, __fsub_rn(p[r].hi[k], hs));
    }
  }
}

__device__ __forceinline__ DFPos bspline_position(const EvalConsts& K, const float4* nodes, const EvalArgs& a,
                                                  const float4& s, const float4& su, bool& has_jac) {
  DFPos p;
  bspline_positions<1>(K, nodes, a, &s, &su, &p, &has_jac);
  return p;
}

__device__ __forceinline__ float3 grad_map(const EvalConsts& K, float3 g) {
  return make_float3(fmaf(K.Mg[0], g.x, fmaf(K.Mg[1], g.y, K.Mg[2] * g.z)),
                     fmaf(K.Mg[3], g.x, fmaf(K.Mg[4], g.y, K.Mg[5] * g.z)),
                     fmaf(K.Mg[6], g.x, fmaf(K.Mg[7], g.y, K.Mg[8] * g.z)));
}

#ifndef GB_KERNELS_HELPERS_ONLY
// MeanSquares, B-spline: value sum and count; per sample a = 2 (f - m) M^T g in the cache.
// R samples to a thread, 32 apart, so that a warp's 32 R consecutive samples mostly lie in one
// cell.
template <int GRAD, bool SMEM, int R>
__global__ void __launch_bounds__(kBlock, SMEM && R == 1 ? 4 : 3) k_msq_bspline(EvalArgs a) {
  extern __shared__ float4 nodes_sh[];
  __shared__ EvalConsts K;
  __shared__ float red[kBlock / 32][1];
  __shared__ double blk[1], fin[1];
  griddep_wait();
  if (halted(a)) return;
  griddep_launch_dependents();
  load_consts(a.consts, K);
  const float4* nodes = stage_nodes<SMEM>(a, nodes_sh);
  __syncthreads();
  KahanF acc[1];
  acc[0].zero();
  unsigned nv = 0;
  const int64_t stride = (int64_t)gridDim.x * kBlock * R;
  const int64_t first = (int64_t)blockIdx.x * kBlock * R + (threadIdx.x >> 5) * 32 * R + (threadIdx.x & 31);
  for (int64_t i0 = first; i0 < a.n; i0 += stride) {
    float4 s[R], su[R];
#pragma unroll
    for (int r = 0; r < R; ++r) {
      const bool live = r == 0 || i0 + 32 * r < a.n;
      s[r] = live ? __ldcs(a.samples + i0 + 32 * r) : make_float4(0.f, 0.f, 0.f, 0.f);
      su[r] = live ? __ldcs(a.sup + i0 + 32 * r) : make_float4(0.f, 0.f, 0.f, 0.f);
    }
    DFPos p[R];
    bool has_jac[R];
    bspline_positions<R>(K, nodes, a, s, su, p, has_jac);
#pragma unroll
    for (int r = 0; r < R; ++r) {
      const int64_t i = i0 + 32 * r;
      if (r > 0 && i >= a.n) break;
      float m;
      float3 g;
      float4 cache = make_float4(0.f, 0.f, 0.f, 0.f);
      if (eval_moving<GRAD>(a, p[r], a.with_derivative != 0 && has_jac[r], m, g)) {
        const float diff = s[r].w - m;  // MeanSquares...Threader.hxx:46
        acc[0].add(diff * diff);
        ++nv;
        if (has_jac[r]) {
          const float3 gm = grad_map(K, g);
          const float t = 2.f * diff;
          cache = make_float4(t * gm.x, t * gm.y, t * gm.z, 1.f);
        }
      }
      if (a.with_derivative) __stcs(a.cache + i, cache);
    }
  }
  block_count(nv, a.acc_n);
  block_sums<1>(acc, red, blk);
  if (!grid_sums<1>(blk, a.part, a.grp, a.tickets + kTicketMain, fin)) return;
  if (threadIdx.x == 0) {
    const unsigned long long N = __ldcg(a.acc_n);
    a.out[1] = (double)N;
    if (N == 0) {
      a.out[0] = DBL_MAX;
      *a.status = GB_ERR_NO_VALID_POINTS;
    } else {
      a.out[0] = fin[0] / (double)N;
      *a.status = GB_OK;
    }
  }
}

// Dynamic shared memory of the B-spline Mattes pass 1: histogram, column sums,
// fixed counts, then (16-byte aligned) the nodes.
__host__ __device__ inline size_t mattes_bspline_node_offset(int B) {
  return (mattes_hist_bytes(B) + 15) / 16 * 16;
}

// Mattes pass 1, B-spline: as k_mattes_pass1_affine, caching (term, M^T g).
template <int GRAD, bool SMEM, int R>
__global__ void __launch_bounds__(kBlock, SMEM && R == 1 ? 4 : 3) k_mattes_pass1_bspline(EvalArgs a) {
  extern __shared__ __align__(16) unsigned smem_hist[];
  const int B = a.bins;
  __shared__ unsigned long long warp_total[kBlock / 32];
  const MattesHist h(smem_hist, warp_total, B);
  float4* nodes_sh = reinterpret_cast<float4*>(reinterpret_cast<unsigned char*>(smem_hist) + mattes_bspline_node_offset(B));
  __shared__ EvalConsts K;
  mattes_hist_clear(h, B);
  griddep_wait();
  if (halted(a)) return;
  griddep_launch_dependents();
  load_consts(a.consts, K);
  const float4* nodes = stage_nodes<SMEM>(a, nodes_sh);
  __syncthreads();
  // 32-bit sample indices (a handle holds at most 2^31 - 1)
  const unsigned n = (unsigned)a.n, stride = (unsigned)(gridDim.x * kBlock * R);
  const float4 zero = make_float4(0.f, 0.f, 0.f, 0.f);
  const unsigned mine = (threadIdx.x >> 5) * 32 * R + (threadIdx.x & 31);  // then 32 apart
  unsigned base = (unsigned)(blockIdx.x * kBlock * R);
  for (;;) {
    int left = kHistSamples / (kBlock * R);
    for (; left > 0 && base < n; base += stride, --left) {
      const unsigned i0 = base + mine;
      float4 s[R], su[R];
#pragma unroll
      for (int r = 0; r < R; ++r) {
        const unsigned i = i0 + 32 * r;
        s[r] = i < n ? __ldcs(a.samples + i) : zero;
        su[r] = i < n ? __ldcs(a.sup + i) : zero;
        if (i + stride < n) {  // the next iteration's records towards L2 (held in registers they cost 16)
          asm volatile("prefetch.global.L2 [%0];" ::"l"(a.samples + i + stride));
          asm volatile("prefetch.global.L2 [%0];" ::"l"(a.sup + i + stride));
        }
      }
      DFPos p[R];
      bool has_jac[R];
      bspline_positions<R>(K, nodes, a, s, su, p, has_jac);
#pragma unroll
      for (int r = 0; r < R; ++r) {
        const unsigned i = i0 + 32 * r;
        const bool live = i < n;
        float m = 0.f;
        float3 g = make_float3(0.f, 0.f, 0.f);
        bool ok = false;
        if (live) {
          ok = eval_moving<GRAD>(a, p[r], a.with_derivative != 0 && has_jac[r], m, g);
          ok = ok && !(m < a.mmin) && !(m > a.mmax);  // Mattes...Threader.hxx:238-245
        }
        const float term = fmaf(m - a.mmin, a.m_inv_bs, 2.f);
        if (a.with_derivative && live) {
          const float3 gm = has_jac[r] ? grad_map(K, g) : make_float3(0.f, 0.f, 0.f);
          __stcs(a.cache + i, ok ? make_float4(term, gm.x, gm.y, gm.z)
                                 : make_float4(__int_as_float(0x7fc00000), 0.f, 0.f, 0.f));
        }
        int pdfm = 0;
        unsigned q[4] = {0u, 0u, 0u, 0u};
        const int fidx = __float_as_int(s[r].w);
        if (ok) {
          float t, w6[4];
          parzen_window(term, B, pdfm, t);
          parzen6(t, w6);
#pragma unroll
          for (int k = 0; k < 4; ++k) q[k] = (__float2uint_rn(w6[k] * kQScale) + 3u) / 6u;
        }
        hist_add_aggregated(ok, fidx * B + pdfm, fidx, q, h.bins, h.fm);
      }
    }
    __syncthreads();
    mattes_hist_flush(a, h, hw_grid());
    if (base >= n) break;
    mattes_hist_restart(a, h);
  }
  mattes_pass1_epilogue(a, h);
}

// The sums of a_s W_k over chunks of same-cell samples, for the cell's 64 support nodes k and
// three components (a 64 x samples by samples x 3 product).  A team of TEAM threads forms a
// chunk: a block (chunks chunk_first[b] .. chunk_first[b + 1], laid out at Initialize so that the
// blocks of one wave hold equal numbers of samples and a long cell is cut where a block ends) or,
// where the cells are small and many, a warp (warp w of block b: b + w G, then every 8 G-th).
//
// Load phase, TEAM samples at a time: thread j stages sample j's 12 axis weights and its
// 3-vector a_s = 2 (f - m) M^T g (MeanSquares) or w(term) M^T g (Mattes,
// w = sum_k log(p/pm)[f][m_k] beta3'(m_k - term)); the next samples' inputs travel meanwhile.
// Sum phase: lane (kz, slice) holds the 16 nodes of plane kz, 48 sums in registers, over the
// samples of its slice (kChunkSlices of a block's: 8 to a warp).  After kFoldBatches batches, and at a
// chunk's end, the 8 slices of a warp are added by halving exchanges; a block's 8 warps follow,
// compensated.
//
// A sum's last additions are its largest, so a chunk of 2048 samples summed plainly to its end loses
// more than eight of 256 do: roundings of 23 (u S)^2 in the mean square against 17 (S the chunk's
// sum, u = 2^-24), with the fold and the compensation 13.  The derivative's error against 64 bits
// over 320 inputs of six kinds (the samples' own arithmetic is 0.98 of it): 0.998 +- 0.006 of
// that of plainly summed 256-sample chunks, without the fold 1.02 at 933k samples in 512 cells.
// The fold costs 1 us in 80 to 90 of a call; chunks of 1024 instead cost 2 to 4 (more entries).
//
// The sum phase is bound by its shared-memory reads and its FMAs alike: a sample costs 13
// wavefronts and 8 x 63 FMAs to eight lanes.  With a row of 4 nodes to a thread it cost 40
// wavefronts, and a sum over the slices and one set of partial sums for each 256 samples.  933k
// samples in 512 cells: 28.3 -> 22.1 us (23 with the fold), the parameters (k_bspline_params)
// 14.3 -> 10.2 us; 5.2M in 27: 120 -> 93 and 59 -> 12.3 us.
//
// A block spends 2 us on a chunk whatever its size.  546k samples, by blocks and by warps: 21,952
// cells 86 and 22.5 us, 8000 36.5 and 18.2; MeanSquares calls 282 and 224 us, 142 and 124, 4096 cells 105
// and 101, 2744 90 and 88; 1728 cells alike, 512 22 us more (a warp needs 8 times as long for a
// cell).  Hence the rule: chunks of less than kWarpChunk samples in the mean, and at least
// kWarpChunks of them to a block.
constexpr int kWarpChunk = 256, kWarpChunks = 6;
template <bool MATTES, int TEAM>
__global__ void __launch_bounds__(kChunkBatch, 3) k_bspline_chunks(EvalArgs a) {
  extern __shared__ float pr_sh[];  // Mattes: the log(p / pm) table
  __shared__ __align__(16) float W1[kChunkBatch][12];
  __shared__ float4 AV[kChunkBatch];
  __shared__ __align__(16) float qs[kChunkBatch / 32][192];
  griddep_wait();
  if (halted(a)) return;
  const int B = a.bins;
  constexpr bool kWarps = TEAM == 32;
  const int t = threadIdx.x % TEAM, w0 = threadIdx.x - t;  // in the team, its first staging row
  if (MATTES) {
    mattes_value_groups(a);  // the value's group partials (blocks b, b + G, ...) and their sum
    for (int k = threadIdx.x; k < B * B; k += blockDim.x) pr_sh[k] = __ldcg(a.pratio + k);
  }
  // this thread's inputs of one batch: the sample's support, cache and fixed bin
  struct In {
    float4 su, c;
    int fbin;
  };
  auto fetch = [&](int pos, int end) {
    In in;
    in.su = in.c = make_float4(0.f, 0.f, 0.f, 0.f);
    in.fbin = 0;
    if (t < end - pos) {
      const int64_t i = (int64_t)pos + t;
      in.su = __ldg(a.sup + i);
      in.c = __ldcg(a.cache + i);
      if (MATTES) in.fbin = __float_as_int(__ldg(&a.samples[i].w));
    }
    return in;
  };
  const bool mine = (int)blockIdx.x < a.chunk_blocks;
  const int next_chunk = kWarps ? (int)gridDim.x * (kChunkBatch / TEAM) : 1;
  int c = kWarps ? (int)(blockIdx.x + gridDim.x * (threadIdx.x / TEAM)) : mine ? __ldg(a.chunk_first + blockIdx.x) : 0;
  const int c1 = kWarps ? __ldg(a.chunk_first + a.chunk_blocks) : mine ? __ldg(a.chunk_first + blockIdx.x + 1) : 0;
  auto sync = [] {
    if (kWarps) __syncwarp();
    else __syncthreads();
  };
  int2 run = c < c1 ? __ldg(a.chunks + c) : make_int2(0, 0);
  In cur = fetch(run.x, run.y);
  __syncthreads();  // the staged table
  const int lane = t & 31, warp = threadIdx.x >> 5, kz = lane >> 3, slice = (t >> 5) * 8 + (lane & 7);
  f32x2 acc[4][3][2];  // [ky][component][kx pair]
#pragma unroll
  for (int k = 0; k < 24; ++k) (&acc[0][0][0])[k] = 0ull;
  int batch = 0;  // of the chunk
  while (c < c1) {
    const int len = min(TEAM, run.y - run.x);
    int cn = c;
    int2 next = make_int2(run.x + TEAM, run.y);
    if (next.x >= next.y) {
      cn += next_chunk;
      next = cn < c1 ? __ldg(a.chunks + cn) : make_int2(0, 0);
    }
    if (t < len) {
      float4 av = make_float4(0.f, 0.f, 0.f, 0.f);
      if (MATTES) {
        const float4 c4 = cur.c;
        if (c4.x == c4.x) {
          int pdfm;
          float tt, d[4];
          parzen_window(c4.x, B, pdfm, tt);
          parzen_deriv(tt, d);
          const float* row = pr_sh + cur.fbin * B + pdfm;
          const float w = row[0] * d[0] + row[1] * d[1] + row[2] * d[2] + row[3] * d[3];
          av = make_float4(w * c4.y, w * c4.z, w * c4.w, 0.f);
        }
      } else {
        av = make_float4(cur.c.x, cur.c.y, cur.c.z, 0.f);
      }
      float w4[12];
      bspline_basis(cur.su.x, w4);
      bspline_basis(cur.su.y, w4 + 4);
      bspline_basis(cur.su.z, w4 + 8);
#pragma unroll
      for (int k = 0; k < 3; ++k)
        *reinterpret_cast<float4*>(&W1[w0 + t][4 * k]) = make_float4(w4[4 * k], w4[4 * k + 1], w4[4 * k + 2], w4[4 * k + 3]);
      AV[w0 + t] = av;
    }
    cur = fetch(next.x, next.y);  // in flight while this batch is summed
    sync();
    for (int j = slice; j < len; j += kChunkSlices / (kChunkBatch / TEAM)) {
      const ulonglong2 wx = *reinterpret_cast<const ulonglong2*>(&W1[w0 + j][0]);
      const float4 wy = *reinterpret_cast<const float4*>(&W1[w0 + j][4]);
      const float wz = W1[w0 + j][8 + kz];
      const float4 v = AV[w0 + j];
      const float vz[3] = {v.x * wz, v.y * wz, v.z * wz}, wys[4] = {wy.x, wy.y, wy.z, wy.w};
#pragma unroll
      for (int ky = 0; ky < 4; ++ky)
#pragma unroll
        for (int d = 0; d < 3; ++d) {
          const f32x2 p = pair(vz[d] * wys[ky]);
          acc[ky][d][0] = fma2(wx.x, p, acc[ky][d][0]);
          acc[ky][d][1] = fma2(wx.y, p, acc[ky][d][1]);
        }
    }
    // a warp's eight slices are added at the chunk's end, and after every kFoldBatches batches
    if (cn != c || batch % kFoldBatches == kFoldBatches - 1) {
      // halving exchanges over the slice bits: lane bits 2 and 1 choose the ky kept, bit 0 the kx pair
      auto halve = [&](f32x2 low, f32x2 high, int bit) {
        const bool up = (lane & bit) != 0;
        return add2(up ? high : low, __shfl_xor_sync(0xffffffffu, up ? low : high, bit));
      };
#pragma unroll
      for (int d = 0; d < 3; ++d) {
        f32x2 h[2];
#pragma unroll
        for (int x = 0; x < 2; ++x)
          h[x] = halve(halve(acc[0][d][x], acc[2][d][x], 4), halve(acc[1][d][x], acc[3][d][x], 4), 2);
        const f32x2 sum = halve(h[0], h[1], 1);
        const int node = 2 * (lane & 1) + 4 * (2 * ((lane >> 2) & 1) + ((lane >> 1) & 1)) + 16 * kz;
        f32x2* const mine = reinterpret_cast<f32x2*>(&qs[warp][64 * d + node]);
        *mine = batch < kFoldBatches ? sum : add2(*mine, sum);
      }
#pragma unroll
      for (int k = 0; k < 24; ++k) (&acc[0][0][0])[k] = 0ull;
    }
    ++batch;
    if (cn != c) {
      batch = 0;
      sync();
      if (kWarps) {  // two nodes to a lane
        const float* q = qs[warp];
#pragma unroll
        for (int node = lane; node < 64; node += 32)
          a.chunk_part[(size_t)c * 64 + node] = make_float4(q[node], q[64 + node], q[128 + node], 0.f);
      } else if (t < 192) {
        KahanF sum;
        sum.zero();
#pragma unroll
        for (int q = 0; q < kChunkBatch / 32; ++q) sum.add(qs[q][t]);
        reinterpret_cast<float*>(a.chunk_part)[((size_t)c * 64 + (t & 63)) * 4 + (t >> 6)] = sum.value();
      }
    }
    sync();  // the next batch overwrites W1, AV and qs
    c = cn;
    run = next;
  }
  griddep_launch_dependents();
}

// For each node n and its three parameters (n + d * nper): the sum of the
// chunk sums of every cell whose 4x4x4 support holds n, listed at Initialize in
// node_entries (chunk * 64 + support position).  Compensated FP32 over the
// list, fixed XOR trees, FP64 only for the metric's scale (1/N for MeanSquares,
// -1/(binsize N) for Mattes, MeanSquares...Threader.hxx:71-79,
// Mattes...Threader.hxx:446-457).  BLOCK = false: one warp per node (lane-strided
// list); BLOCK = true, for coarse grids whose nodes hold thousands of entries:
// one block per node (thread-strided list, warps added in fixed order), so the
// few hundred nodes still spread over every SM.
template <bool MATTES, bool BLOCK>
__global__ void __launch_bounds__(kParamsBlock) k_bspline_params(EvalArgs a) {
  const int n = BLOCK ? (int)blockIdx.x : (int)((blockIdx.x * blockDim.x + threadIdx.x) >> 5);
  const int lane = threadIdx.x & 31;
  // the list is Initialize's: its first entries are read before the wait for the chunk sums
  const int first = BLOCK ? (int)threadIdx.x : lane;
  const int step = BLOCK ? (int)blockDim.x : 32;
  int e = 0, e1 = 0, entry = 0;
  if (n < a.nper) {
    e = __ldg(a.node_first + n) + first;
    e1 = __ldg(a.node_first + n + 1);
    if (e < e1) entry = __ldg(a.node_entries + e);
  }
  griddep_wait();
  if (halted(a)) return;
  griddep_launch_dependents();
  // MeanSquares: the status of the value pass, scale 1 / N; Mattes: the scale formed by
  // the table kernel (0 unless the status is OK), and block 0 writes the value summed by
  // the chunk kernel's last group warp, the count and the status
  const unsigned long long N = __ldcg(a.acc_n);
  const double table_scale = MATTES ? __ldcg(&a.marg[2]) : 0.0;
  const int status = MATTES ? GB_OK : __ldcg(a.status);
  if (blockIdx.x == 0 && threadIdx.x == 0) {
    a.out[1] = (double)N;
    if (MATTES) {
      const int st = mattes_status(a);
      *a.status = st;
      a.out[0] = st == GB_OK ? -1.0 * __ldcg(&a.part[kPartValue]) : 0.0;
    }
  }
  if (n >= a.nper) return;
  KahanF s0, s1, s2;
  s0.zero();
  s1.zero();
  s2.zero();
  auto add = [&](const float4& q) {
    s0.add(q.x);
    s1.add(q.y);
    s2.add(q.z);
  };
  if (e < e1) add(__ldcg(a.chunk_part + entry));
#pragma unroll 4
  for (e += step; e < e1; e += step) add(__ldcg(a.chunk_part + __ldg(a.node_entries + e)));
  float t0 = warp_sum(s0.value()), t1 = warp_sum(s1.value()), t2 = warp_sum(s2.value());
  if (BLOCK) {
    __shared__ float wsum[kParamsBlock / 32][3];
    const int w = threadIdx.x >> 5;
    if (lane == 0) {
      wsum[w][0] = t0;
      wsum[w][1] = t1;
      wsum[w][2] = t2;
    }
    __syncthreads();
    if (threadIdx.x != 0) return;
    KahanF b0, b1, b2;
    b0.zero();
    b1.zero();
    b2.zero();
    for (int k = 0; k < (int)(blockDim.x >> 5); ++k) {
      b0.add(wsum[k][0]);
      b1.add(wsum[k][1]);
      b2.add(wsum[k][2]);
    }
    t0 = b0.value();
    t1 = b1.value();
    t2 = b2.value();
  }
  if (lane == 0) {
    const double scale = MATTES ? table_scale : status == GB_OK && N > 0 ? 1.0 / (double)N : 0.0;
    a.out[2 + n] = (double)t0 * scale;
    a.out[2 + a.nper + n] = (double)t1 * scale;
    a.out[2 + 2 * a.nper + n] = (double)t2 * scale;
  }
}
#endif  // GB_KERNELS_HELPERS_ONLY

}  // namespace gb
