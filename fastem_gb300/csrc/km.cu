// km.cu -- Lloyd k-means iteration (NaiveKMA::ComputeMSEAndCorrect,
// Clust/KMAlgorithm.cpp:205-255) and the k-means half of the C-ABI.
//
// Assignment must equal an FP64 difference-form argmin over centroids in
// index order with strict '<' (Clust/KMAlgorithm.cpp:226-234).  Candidate
// distances are computed fast (FP32 here, BF16 tensor cores in km_tc.cu)
// together with a rigorous error bound; a row whose best candidate is not
// separated from the runner-up by the bounds is re-decided in FP64 with
// the reference's summation order.  Centroid sums are accumulated exactly
// in 64-bit fixed point (x * 2^shift is an integer for every float the
// data holds), so they are order independent; the fit uses
//   sum_i ||x_i - c_l(i)||^2 = sum_i ||x_i - g||^2
//        - 2 sum_j (c_j - g).(S_j - n_j g) + sum_j n_j ||c_j - g||^2
// with the exact cluster sums S_j and the data mean g.
#include <algorithm>
#include <cfloat>
#include <climits>
#include <cmath>
#include <cstring>
#include <new>
#include <sstream>
#include <string>
#include <vector>

#include "fem_internal.cuh"
#include "km_kernels.cuh"

using namespace fem;

namespace fem {

__device__ __forceinline__ double warp_sum_d(double v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
  return v;
}

// ----------------------------------------------------------- data stats
// One pass over X for the data mean g, max |x| and sum_i ||x_i - g||^2: per
// CTA and column, S1 = sum t and S2 = sum t^2 in FP64 with t = x - c (c = the
// dataset's first row: x - c is exact in FP64 for FP32 data, and c lies inside
// the data, so S2 - S1^2 / n below does not cancel), plus max |x|.  The host
// merges the CTAs: g = c + S1 / n, sum ||x - g||^2 = sum_q (S2_q - S1_q^2 / n).
// Threads own (row group, column) pairs, so a warp reads whole rows.
__global__ void __launch_bounds__(256)
k_km_stats(const float *__restrict__ X, int64_t n, int d, int64_t rows_per_block, const float *__restrict__ c,
           double *__restrict__ s1, double *__restrict__ s2, float *__restrict__ amax) {
  __shared__ double r1[256], r2[256];
  __shared__ float rm[256];
  const int64_t r0 = (int64_t)blockIdx.x * rows_per_block, r1e = min(n, r0 + rows_per_block);
  const bool narrow = d <= 256;
  const int groups = narrow ? 256 / d : 1;       // row groups a pass covers
  const int tid = threadIdx.x;
  float mx = 0.f;
  for (int q0 = 0; q0 < d; q0 += 256) {
    const int q = q0 + (narrow ? tid % d : tid), g = narrow ? tid / d : 0;
    const int cols = narrow ? d : min(256, d - q0);
    double a = 0.0, b = 0.0;
    if (g < groups && q < d) {
      const double cq = (double)c[q];
      for (int64_t i = r0 + g; i < r1e; i += groups) {
        const float x = X[i * d + q];
        const double t = (double)x - cq;
        a += t;
        b = fma(t, t, b);
        mx = fmaxf(mx, fabsf(x));
      }
    }
    r1[tid] = a, r2[tid] = b;
    __syncthreads();
    // column q0 + tid's row groups sit at tid + cols g: summed in group order
    if (tid < cols) {
      double sa = 0.0, sb = 0.0;
      for (int gg = 0; gg < groups; gg++) sa += r1[tid + gg * cols], sb += r2[tid + gg * cols];
      s1[(size_t)blockIdx.x * d + q0 + tid] = sa;
      s2[(size_t)blockIdx.x * d + q0 + tid] = sb;
    }
    __syncthreads();
  }
  rm[tid] = mx;
  __syncthreads();
  if (tid == 0) {
    float m = 0.f;
    for (int t = 0; t < 256; t++) m = fmaxf(m, rm[t]);
    amax[blockIdx.x] = m;
  }
}

// The screens' frame: a centre amid the data (per column the median of a sample of
// rows) and the power of two that brings the data's spread around it (mean of the
// sampled rows' largest difference, the farthest rows left out) to 1/2..1.  Not the
// mean and the maximum: rows far out would move the one and widen the other, and
// with them every row's bound.  The sample's rows are drawn by a hash, so that
// sorted or periodic data are sampled as any other; 256 rows, 4 left out.  About 15
// us an upload.
constexpr int kFrameRows = 256, kFrameFar = 4;

__device__ __forceinline__ int64_t frame_row(int s, int64_t n) {
  uint64_t v = (uint64_t)(s + 1) * 0x9E3779B97F4A7C15ull;     // splitmix64
  v = (v ^ (v >> 30)) * 0xBF58476D1CE4E5B9ull;
  v = (v ^ (v >> 27)) * 0x94D049BB133111EBull;
  return (int64_t)__umul64hi(v ^ (v >> 31), (uint64_t)n);
}

// ascending bitonic sort of kFrameRows values, one per thread
__device__ void frame_sort(float *v) {
#pragma unroll 1
  for (int k = 2; k <= kFrameRows; k *= 2)
#pragma unroll 1
    for (int j = k / 2; j > 0; j /= 2) {
      __syncthreads();
      const int i = threadIdx.x, o = i ^ j;
      const float a = v[i], b = v[o];
      __syncthreads();
      v[i] = (i < o) == ((i & k) == 0) ? fminf(a, b) : fmaxf(a, b);
    }
  __syncthreads();
}

__global__ void __launch_bounds__(kFrameRows)
k_km_centre(const float *__restrict__ X, int64_t n, int d, float *__restrict__ gs) {
  __shared__ float v[kFrameRows];
  const float x = X[frame_row(threadIdx.x, n) * d + blockIdx.x];
  v[threadIdx.x] = isfinite(x) ? x : 0.f;
  frame_sort(v);
  if (threadIdx.x == 0) gs[blockIdx.x] = 0.5f * v[kFrameRows / 2 - 1] + 0.5f * v[kFrameRows / 2];
}

__global__ void __launch_bounds__(kFrameRows)
k_km_spread(const float *__restrict__ X, int64_t n, int d, const float *__restrict__ gs, float *__restrict__ xscale) {
  __shared__ float v[kFrameRows];
  const float *x = X + frame_row(threadIdx.x, n) * d;
  float m = 0.f, big = 0.f;
#pragma unroll 16
  for (int q = 0; q < d; q++) {
    const float g = gs[q], t = fabsf(x[q] - g);
    m = t <= m ? m : t;                       // NaN stays
    big = fmaxf(big, fabsf(g));
  }
  v[threadIdx.x] = m < INFINITY ? m : INFINITY;
  frame_sort(v);
  if (threadIdx.x < 32) {
    float s = 0.f;
    for (int i = threadIdx.x; i < kFrameRows - kFrameFar; i += 32) s += v[i] * (1.f / (kFrameRows - kFrameFar));
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
    // no less than FP32 resolves at the centre
    s = fmaxf(s, fmaxf(big * 5.9604645e-8f, 1e-32f));
    if (threadIdx.x == 0) *xscale = ldexpf(1.f, -1 - min(ilogbf(s), 125));
  }
}

// centroids -> float copy and norm, and for the FP32 path the copy around g (as
// float) and half its squared norm; one warp per centroid.  Clears the range of
// norms that the tensor-core path's preparation collects.
__global__ void __launch_bounds__(128)
k_km_prep(const double *__restrict__ cent, const float *__restrict__ g, int K, int d, float *__restrict__ centf,
          float *__restrict__ cnorm, float *__restrict__ centg, float *__restrict__ hnorm, int *__restrict__ range) {
  if (blockIdx.x == 0 && threadIdx.x < 2) range[threadIdx.x] = 0;
  const int j = blockIdx.x * 4 + (threadIdx.x >> 5), lane = threadIdx.x & 31;
  if (j >= K) return;
  double s = 0.0, h = 0.0;
  for (int q = lane; q < d; q += 32) {
    const double c = cent[(size_t)j * d + q];
    centf[(size_t)j * d + q] = (float)c;
    s = fma(c, c, s);
    if (centg) {
      const double cg = c - (double)g[q];
      centg[(size_t)j * d + q] = (float)cg;
      h = fma(cg, cg, h);
    }
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1)
    s += __shfl_xor_sync(0xffffffffu, s, o), h += __shfl_xor_sync(0xffffffffu, h, o);
  if (lane == 0) {
    cnorm[j] = (float)sqrt(s);
    if (centg) hnorm[j] = (float)(0.5 * h);
  }
}

// FP64 difference form in column order, no contraction: bit-identical to
// `for q: t = c[q] - x[q]; s += t*t;` compiled without FMA.
__device__ __forceinline__ double dist64(const double *__restrict__ c, const float *x, int d) {
  double s = 0.0;
  for (int q = 0; q < d; q++) {
    const double t = __dsub_rn(c[q], (double)x[q]);
    s = __dadd_rn(s, __dmul_rn(t, t));
  }
  return s;
}

// bound on |fp32 difference-form distance - exact distance| (x2 safety)
__device__ __forceinline__ float bound_f32(float s, float cn, int d) {
  const float u = 5.9604645e-8f;  // 2^-24
  return 2.f * ((float)(d + 4) * u * s + 2.01f * u * sqrtf(fmaxf(s, 0.f)) * cn + u * u * cn * cn) +
         1e-30f;
}

// =================================================== FP32 assignment
// Every warp takes its own share of the rows, 32 R at a time (R rows per
// lane, in registers), and screens all centroids by
//   w_j = ||c'_j||^2 / 2 - x'.c'_j     (x' = x - g, c' = c - g, g amid the data;
//                                       ||x - c||^2 = ||x'||^2 + 2 w_j),
// D products per (row, centroid) where the difference form takes 2 D
// operations, keeping the two smallest.  With u = 2^-24 and N = ||c'_j|| the computed
// w_j is within
//   B(N) = 1.05 (D + 6) u (||x'|| N + N^2 / 2)
// of the exact one (rounding of x', c', ||c'||^2 and the D-term sum).  A row's
// nearest centroid is no farther from g than L = l + 2 ||x'||, l the smallest
// ||c'||; one beyond 1.01 L, at N, has w_j at least 0.0049 N^2 above the one at l,
// more than B(N) and B(1.01 L) together, so it is never the smallest.  A row whose
// two smallest differ by more than 2 B(min(||c'||max, 1.01 L)) is therefore decided
// (with ||c'||max alone one centroid at 10^4 opened every row of unit blobs: N =
// 1000003, D = 64, K = 100 43 ms an iteration, without it 0.62).  Where several
// of a warp's 32 rows stay open (centroids close together, far from g) each lane first
// tries its own in the difference form: with D >= 32 that costs as much as deciding
// two rows, with 8 and 16 about five (20 centroids in each of 5 blobs, D = 64: 13.2 ->
// 1.3 ms, one row per thread 1.8; D = 2, K = 700 0.42 -> 0.53, so not there).  The
// others, few, go through the difference form by the whole warp (lane = centroid): FP32 with
// the bound of bound_f32, then the reference's FP64 sums among the centroids
// that remain, lowest index on ties.  Rows are added to exact fixed-point sums
// in shared memory (a float times 2^shift is exact), so the order is free.
// Bound by the FP32 pipe, and by the broadcast loads of the centroids where R <
// 4 (R = 4 loads 16 bytes per 16 products).  N = 1000003, D = 16, K = 100 on
// the GB300: 442 -> 128 us an iteration (difference form, one row per thread).
template <int D>
struct KmShape {
  static constexpr int R = D <= 32 ? 4 : 2;               // rows per lane
  static constexpr int kThreads = D <= 16 ? 512 : 256;
};

__device__ __forceinline__ float2 km_ffma2(float2 a, float2 b, float2 c) { return __ffma2_rn(a, b, c); }

// two smallest w and the first's index for NR rows per lane
template <int D, int NR>
__device__ __forceinline__ void km_screen(const float2 (*x)[D / 2], const float *sC, const float *sH, int K, float *m1,
                                          float *m2, int *j1) {
#pragma unroll
  for (int r = 0; r < NR; r++) m1[r] = INFINITY, m2[r] = INFINITY, j1[r] = -1;
#pragma unroll 1
  for (int j = 0; j < K; j++) {
    const float *c = sC + j * D;
    float2 w[NR];
    const float h = sH[j];
#pragma unroll
    for (int r = 0; r < NR; r++) w[r] = make_float2(h, 0.f);
    if constexpr (D >= 4) {
#pragma unroll
      for (int q = 0; q < D / 4; q++) {
        const float4 c4 = reinterpret_cast<const float4 *>(c)[q];
#pragma unroll
        for (int r = 0; r < NR; r++) {
          w[r] = km_ffma2(x[r][2 * q], make_float2(c4.x, c4.y), w[r]);
          w[r] = km_ffma2(x[r][2 * q + 1], make_float2(c4.z, c4.w), w[r]);
        }
      }
    } else {
      const float2 c2 = *reinterpret_cast<const float2 *>(c);
#pragma unroll
      for (int r = 0; r < NR; r++) w[r] = km_ffma2(x[r][0], c2, w[r]);
    }
#pragma unroll
    for (int r = 0; r < NR; r++) {
      const float v = w[r].x + w[r].y;
      m2[r] = fminf(m2[r], fmaxf(m1[r], v));
      if (v < m1[r]) j1[r] = j;
      m1[r] = fminf(m1[r], v);
    }
  }
}

// a lane's own row in the difference form over all centroids around g: the nearest,
// and whether FP32 tells it from every other.  q: ||x'|| plus the largest ||c'|| that
// counts (km_screen's callers); x' and c' are rounded, so a distance is off by what
// bound_f32 says with q for ||c||, and farther centroids are out of reach of theirs.
template <int D>
__device__ __forceinline__ bool km_differences(const float2 (&x)[D / 2], const float *sC, int K, float q, int *j1) {
  constexpr float u = 5.9604645e-8f;  // 2^-24
  const float e1 = 2.f * 2.01f * u * q, e0 = 2.f * (u * q) * (u * q) + 1e-30f;
  float U = INFINITY, l1 = INFINITY, l2 = INFINITY;
  *j1 = -1;
#pragma unroll 1
  for (int j = 0; j < K; j++) {
    const float2 *c = reinterpret_cast<const float2 *>(sC + j * D);     // -c'
    float2 s2 = make_float2(0.f, 0.f);
#pragma unroll
    for (int p = 0; p < D / 2; p++) {
      const float2 t = __fadd2_rn(x[p], c[p]);
      s2 = km_ffma2(t, t, s2);
    }
    const float s = s2.x + s2.y, e = fmaf(2.f * (D + 4) * u, s, fmaf(e1, sqrtf(s), e0)), lb = s - e;
    U = fminf(U, s + e);
    if (lb < l1)
      l2 = l1, l1 = lb, *j1 = j;
    else
      l2 = fminf(l2, lb);
  }
  return l2 > U;
}

// the reference's choice for one row, by the whole warp: -1 when no centroid
// compares (a row with NaN); *fp64 when FP64 had to decide
template <int D>
__device__ int km_decide(const float *__restrict__ x, const float *__restrict__ centf, const float *__restrict__ cnorm,
                         const double *__restrict__ cent, int K, bool *fp64) {
  const int lane = threadIdx.x & 31;
  float xr[D];
#pragma unroll
  for (int q = 0; q < D; q++) xr[q] = x[q];
  // 16 bytes a load where the registers allow it: the lanes' rows lie a row apart
  auto dist = [&](int j) {
    float s = 0.f;
    if constexpr (D >= 32) {
      const float4 *c = reinterpret_cast<const float4 *>(centf + (size_t)j * D);
#pragma unroll
      for (int q = 0; q < D / 4; q++) {
        const float4 v = __ldg(c + q);
        const float t0 = xr[4 * q] - v.x, t1 = xr[4 * q + 1] - v.y, t2 = xr[4 * q + 2] - v.z, t3 = xr[4 * q + 3] - v.w;
        s = fmaf(t3, t3, fmaf(t2, t2, fmaf(t1, t1, fmaf(t0, t0, s))));
      }
    } else {
#pragma unroll
      for (int q = 0; q < D; q++) {
        const float t = xr[q] - centf[(size_t)j * D + q];
        s = fmaf(t, t, s);
      }
    }
    return s;
  };
  float U = INFINITY;
  for (int j = lane; j < K; j += 32) {
    const float s = dist(j);
    U = fminf(U, s + bound_f32(s, cnorm[j], D));
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) U = fminf(U, __shfl_xor_sync(0xffffffffu, U, o));
  double best = DBL_MAX;
  int lab = INT_MAX, cand = 0, only = INT_MAX;
  for (int j = lane; j < K; j += 32) {
    const float s = dist(j);
    if (s - bound_f32(s, cnorm[j], D) <= U) cand++, only = min(only, j);
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    cand += __shfl_xor_sync(0xffffffffu, cand, o);
    only = min(only, __shfl_xor_sync(0xffffffffu, only, o));
  }
  *fp64 = cand > 1;
  if (cand <= 1) return cand == 1 ? only : -1;
  for (int j = lane; j < K; j += 32) {
    const float s = dist(j);
    if (s - bound_f32(s, cnorm[j], D) <= U) {
      const double s64 = dist64(cent + (size_t)j * D, xr, D);
      if (s64 < best) best = s64, lab = j;       // a lane's centroids come in index order
    }
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    const double ob = __shfl_xor_sync(0xffffffffu, best, o);
    const int ol = __shfl_xor_sync(0xffffffffu, lab, o);
    if (ob < best || (ob == best && ol < lab)) best = ob, lab = ol;
  }
  return lab == INT_MAX ? -1 : lab;
}

template <int D>
__global__ void __launch_bounds__(KmShape<D>::kThreads)
k_km_assign_f32(const float *__restrict__ X, int64_t n, int K, const float *__restrict__ gs,
                const float *__restrict__ centg, const float *__restrict__ hnorm, const float *__restrict__ centf,
                const float *__restrict__ cnorm, const double *__restrict__ cent, int32_t *__restrict__ labels,
                long long *__restrict__ accg, int *__restrict__ cntg, float scale, DevStatus *st) {
  constexpr int R = KmShape<D>::R, T = KmShape<D>::kThreads;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  long long *sAcc = (long long *)smem_raw;              // K x D
  float *sC = (float *)(sAcc + (size_t)K * D);          // K x D, around g
  float *sH = sC + (size_t)K * D;                       // K
  int *sCnt = (int *)(sH + K);                          // K
  __shared__ __align__(16) float sG[D < 4 ? 4 : D];
  __shared__ float sMax[T / 32], sMin[T / 32];
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  float hmax = 0.f, hmin = INFINITY;
  for (int e = tid; e < K * D; e += T) {
    sAcc[e] = 0;
    sC[e] = -centg[e];                                  // w = h + x'.(-c')
  }
  for (int j = tid; j < K; j += T) {
    const float h = hnorm[j];
    sCnt[j] = 0;
    sH[j] = h;
    hmax = fmaxf(hmax, h), hmin = fminf(hmin, h);
  }
  if (tid < D) sG[tid] = gs[tid];
#pragma unroll
  for (int o = 16; o > 0; o >>= 1)
    hmax = fmaxf(hmax, __shfl_xor_sync(0xffffffffu, hmax, o)), hmin = fminf(hmin, __shfl_xor_sync(0xffffffffu, hmin, o));
  if (lane == 0) sMax[warp] = hmax, sMin[warp] = hmin;
  __syncthreads();
#pragma unroll
  for (int w = 0; w < T / 32; w++) hmax = fmaxf(hmax, sMax[w]), hmin = fminf(hmin, sMin[w]);
  const float cmax = sqrtf(2.f * hmax) * 1.00001f, clo = sqrtf(2.f * hmin) * 1.0101f;   // ||c'||max, 1.01 l
  const bool track = st->track_changes;
  constexpr float kU = 5.9604645e-8f * 1.05f * (D + 6);
  int64_t rechecks = 0;
  bool changed = false;
  // this warp's rows: an even share, in whole groups of 32
  const int64_t nw = (int64_t)gridDim.x * (T / 32), gw = (int64_t)blockIdx.x * (T / 32) + warp;
  const int64_t groups = (n + 31) / 32;
  const int64_t r0 = gw * groups / nw * 32, r1 = min(n, (gw + 1) * groups / nw * 32);
  for (int64_t base = r0; base < r1; base += 32 * R) {
    float2 x[R][D / 2];
    float xn[R], m1[R], m2[R];
    int j1[R];
#pragma unroll
    for (int r = 0; r < R; r++) {
      const int64_t row = base + 32 * r + lane;
      const float *xr = X + (row < r1 ? row : r0) * D;
      float ss = 0.f;
      if constexpr (D >= 4) {
#pragma unroll
        for (int q = 0; q < D / 4; q++) {
          const float4 v = __ldg(reinterpret_cast<const float4 *>(xr) + q);
          const float4 g4 = reinterpret_cast<const float4 *>(sG)[q];
          x[r][2 * q] = make_float2(v.x - g4.x, v.y - g4.y);
          x[r][2 * q + 1] = make_float2(v.z - g4.z, v.w - g4.w);
        }
      } else {
        x[r][0] = make_float2(xr[0] - sG[0], xr[1] - sG[1]);
      }
#pragma unroll
      for (int q = 0; q < D / 2; q++) ss = fmaf(x[r][q].x, x[r][q].x, fmaf(x[r][q].y, x[r][q].y, ss));
      xn[r] = sqrtf(ss) * 1.00001f;
    }
    const int live = (int)min((int64_t)R, (r1 - base + 31) / 32);   // row groups of this pass
    if (live == R)
      km_screen<D, R>(x, sC, sH, K, m1, m2, j1);
    else if (R > 2 && live == 3)
      km_screen<D, R - 1>(x, sC, sH, K, m1, m2, j1);
    else if (R > 2 && live == 2)
      km_screen<D, 2>(x, sC, sH, K, m1, m2, j1);
    else
      km_screen<D, 1>(x, sC, sH, K, m1, m2, j1);
#pragma unroll
    for (int r = 0; r < R; r++) {
      if (r >= live) break;
      const int64_t row = base + 32 * r + lane;
      const bool in = row < r1;
      // the last term covers the reference's own FP64 rounding
      const float cn = fminf(cmax, fmaf(2.02f, xn[r], clo));
      const float B = fmaf(kU, fmaf(xn[r], cn, 0.5f * cn * cn), 1e-13f * fmaf(xn[r], xn[r], cn * cn)) + 1e-30f;
      int lab = j1[r];
      unsigned open = __ballot_sync(0xffffffffu, in && !(m2[r] - m1[r] > 2.1f * B));
      if constexpr (D >= 8) {
        if (__popc(open) >= (D >= 32 ? 2 : 5)) {
          int l;
          const bool told = km_differences<D>(x[r], sC, K, xn[r] + cn, &l);
          if (told && (open >> lane & 1)) lab = l;
          open &= ~__ballot_sync(0xffffffffu, told);
        }
      }
      while (open) {
        const int b = __ffs(open) - 1;
        open &= open - 1;
        bool fp64 = false;
        const int l = km_decide<D>(X + (base + 32 * r + b) * D, centf, cnorm, cent, K, &fp64);
        if (lane == b) {
          lab = l;
          if (fp64) rechecks++;
        }
      }
      if (in) {
        if (track && labels[row] != lab) changed = true;
        labels[row] = lab;
        if (lab >= 0) atomicAdd(&sCnt[lab], 1);
      } else {
        lab = -1;
      }
      // exact sums: the 32 rows again, lanes along the dimensions
#pragma unroll 4
      for (int i = lane; i < 32 * D; i += 32) {
        const int p = i / D, l = __shfl_sync(0xffffffffu, lab, p);
        if (l >= 0) {
          const float xv = __ldg(X + (base + 32 * r) * D + i);
          atomicAdd((unsigned long long *)&sAcc[l * D + i % D], (unsigned long long)__float2ll_rn(xv * scale));
        }
      }
    }
  }
  if (changed) st->changed = 1;
  if (rechecks) atomicAdd((unsigned long long *)&st->rechecked, (unsigned long long)rechecks);
  __syncthreads();
  for (int e = tid; e < K * D; e += T) accg[(size_t)blockIdx.x * K * D + e] = sAcc[e];
  for (int j = tid; j < K; j += T) cntg[(size_t)blockIdx.x * K + j] = sCnt[j];
}

// sums the per-CTA partials (exact), forms the new centroids and the fit terms
// (one CTA per centroid, the CTAs' partials split over its 8 warps: the sums
// are integers, so their order is free)
__global__ void __launch_bounds__(256)
k_km_final(const long long *__restrict__ accg, const int *__restrict__ cntg, int G, int K, int d, double inv_scale,
           const double *__restrict__ cent, const double *__restrict__ g, double *__restrict__ out) {
  const int j = blockIdx.x, lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  __shared__ long long red[8][32], s_n[8];
  long long c = 0;
  for (int b = threadIdx.x; b < G; b += 256) c += cntg[(size_t)b * K + j];
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) c += __shfl_xor_sync(0xffffffffu, c, o);
  if (lane == 0) s_n[w] = c;
  __syncthreads();
  long long nj = 0;
#pragma unroll
  for (int q = 0; q < 8; q++) nj += s_n[q];
  double term = 0.0;
  for (int q0 = 0; q0 < d; q0 += 32) {
    const int q = q0 + lane;
    long long S = 0;
    if (q < d) {
#pragma unroll 4
      for (int b = w; b < G; b += 8) S += accg[((size_t)b * K + j) * d + q];
    }
    __syncthreads();
    red[w][lane] = S;
    __syncthreads();
    if (w == 0 && q < d) {
#pragma unroll
      for (int u = 1; u < 8; u++) S += red[u][lane];
      const double sum = (double)S * inv_scale;
      out[(size_t)j * d + q] = nj > 0 ? sum * (1.0 / (double)nj) : 0.0;
      const double cg = cent[(size_t)j * d + q] - g[q];
      term += -2.0 * cg * (sum - (double)nj * g[q]) + (double)nj * cg * cg;
    }
  }
  if (w == 0) {
    term = warp_sum_d(term);
    if (lane == 0) {
      out[(size_t)K * d + j] = (double)nj;
      out[(size_t)K * d + K + j] = term;
    }
  }
}

int km_launch_assign_f32(fem_km *h) {
  const int D = h->d, K = h->k;
  const size_t sm = (size_t)K * D * 12 + (size_t)K * 8;
#define FEM_KA(DD)                                                                                             \
  case DD:                                                                                                     \
    FEM_CUDA(allow_dyn_smem(k_km_assign_f32<DD>, sm));                                                         \
    k_km_assign_f32<DD><<<h->grid, KmShape<DD>::kThreads, sm, h->stream>>>(                                    \
        h->X, h->n, K, h->gs, h->centg, h->hnorm, h->centf, h->cnorm, h->cent, h->labels, h->acc, h->cnt,       \
        ldexpf(1.f, h->shift), h->dstat);                                                                      \
    break;
  switch (D) {
    FEM_KA(2)
    FEM_KA(4)
    FEM_KA(8)
    FEM_KA(16)
    FEM_KA(32)
    FEM_KA(64)
    default:
      set_error("k-means FP32 path supports d in {2,4,8,16,32,64} (got %d)", D);
      return FEM_ERR_UNSUPPORTED;
  }
#undef FEM_KA
  FEM_CUDA(cudaGetLastError());
  return FEM_OK;
}

size_t km_assign_smem(int K, int D) {
  return (size_t)K * D * 12 + (size_t)K * 8 + 1024 + (size_t)256 * (D + 1) * 4;
}

}  // namespace fem

// =============================================================== C-ABI
namespace {

int check(fem_km *h) {
  if (!h) {
    set_error("null k-means handle");
    return FEM_ERR_BAD_ARG;
  }
  return FEM_OK;
}

void free_km(fem_km *h) {
  dfree(h->X);
  dfree(h->labels);
  dfree(h->cent);
  dfree(h->centf);
  dfree(h->centg);
  dfree(h->hnorm);
  dfree(h->cnorm);
  dfree(h->acc);
  dfree(h->cnt);
  dfree(h->g);
  dfree(h->gs);
  dfree(h->xscale);
  dfree(h->range);
  dfree(h->out);
  dfree(h->dstat);
  km_tc_destroy(h);
  if (h->hout) cudaFreeHost(h->hout);
  if (h->hstat) cudaFreeHost(h->hstat);
  if (h->hg) delete[] h->hg;
  h->hout = nullptr;
  h->hstat = nullptr;
  h->hg = nullptr;
  for (auto &e : h->ev)
    if (e) cudaEventDestroy(e), e = nullptr;
  if (h->stream) cudaStreamDestroy(h->stream);
  h->stream = nullptr;
}

int upload_km(fem_km *h, const float *X, int64_t ld, cudaMemcpyKind kind) {
  FEM_TRY(check(h));
  if (!X || ld < h->d) {
    set_error("bad dataset pointer or ld");
    return FEM_ERR_BAD_ARG;
  }
  const int d = h->d;
  const int64_t n = h->n;
  FEM_CUDA(cudaSetDevice(h->cfg.device));
  FEM_CUDA(cudaMemcpy2DAsync(h->X, (size_t)d * 4, X, (size_t)ld * 4, (size_t)d * 4, (size_t)n, kind,
                             h->stream));
  // data mean, max |x| -> fixed-point shift, sum ||x - g||^2, in one pass
  const int G = (int)std::min<int64_t>(4 * (int64_t)sm_count(), (n + 255) / 256);
  const int64_t rpb = (n + G - 1) / G;
  double *s1 = nullptr, *s2 = nullptr;
  float *amax = nullptr;
  FEM_TRY(dalloc(&s1, (size_t)G * d));
  FEM_TRY(dalloc(&s2, (size_t)G * d));
  FEM_TRY(dalloc(&amax, G));
  k_km_stats<<<G, 256, 0, h->stream>>>(h->X, n, d, rpb, h->X, s1, s2, amax);
  k_km_centre<<<d, kFrameRows, 0, h->stream>>>(h->X, n, d, h->gs);
  k_km_spread<<<1, kFrameRows, 0, h->stream>>>(h->X, n, d, h->gs, h->xscale);
  std::vector<double> h1((size_t)G * d), h2((size_t)G * d);
  std::vector<float> hm(G), c(d);
  cudaMemcpyAsync(c.data(), h->X, (size_t)d * 4, cudaMemcpyDeviceToHost, h->stream);
  cudaMemcpyAsync(h1.data(), s1, h1.size() * 8, cudaMemcpyDeviceToHost, h->stream);
  cudaMemcpyAsync(h2.data(), s2, h2.size() * 8, cudaMemcpyDeviceToHost, h->stream);
  cudaMemcpyAsync(hm.data(), amax, hm.size() * 4, cudaMemcpyDeviceToHost, h->stream);
  cudaError_t e = cudaStreamSynchronize(h->stream);
  dfree(s1);
  dfree(s2);
  dfree(amax);
  if (e != cudaSuccess) {
    set_error("dataset statistics failed: %s", cudaGetErrorString(e));
    return FEM_ERR_CUDA;
  }
  float mx = 0.f;
  for (int b = 0; b < G; b++) mx = std::max(mx, hm[b]);
  h->xg2 = 0.0;
  for (int q = 0; q < d; q++) {
    double a = 0.0, b2 = 0.0;
    for (int b = 0; b < G; b++) a += h1[(size_t)b * d + q], b2 += h2[(size_t)b * d + q];
    h->hg[q] = (double)c[q] + a / (double)n;
    h->xg2 += b2 - a * a / (double)n;
  }
  // |x| * 2^shift * n < 2^62: the per-CTA and the final int64 sums cannot overflow
  const double lg = std::log2((double)std::max(mx, 1e-30f)) + std::log2((double)n);
  h->xmax = mx;
  h->shift = (int)std::min(40.0, std::floor(61.0 - std::ceil(lg)));
  FEM_CUDA(cudaMemcpyAsync(h->g, h->hg, d * 8, cudaMemcpyHostToDevice, h->stream));
  h->have_data = true;
  return FEM_OK;
}

}  // namespace

extern "C" {

void fem_km_config_default(fem_km_config *cfg) {
  if (!cfg) return;
  cfg->precision = FEM_PREC_MIXED;
  cfg->device = 0;
  cfg->seed = 0;
  cfg->repair = FEM_KM_REPAIR_RANDOM;
}

int fem_km_create(int d, int64_t n, int k, const fem_km_config *cfg, fem_km **out) {
  if (!out) {
    set_error("out is NULL");
    return FEM_ERR_BAD_ARG;
  }
  *out = nullptr;
  fem_km_config c;
  if (cfg)
    c = *cfg;
  else
    fem_km_config_default(&c);
  if (d < 1 || n < 1 || k < 1 || k > 1024) {
    set_error("bad sizes d=%d n=%lld k=%d", d, (long long)n, k);
    return FEM_ERR_BAD_ARG;
  }
  if (c.precision != FEM_PREC_FP32 && c.precision != FEM_PREC_MIXED) {
    set_error("k-means precision must be FEM_PREC_FP32 or FEM_PREC_MIXED");
    return FEM_ERR_BAD_ARG;
  }
  if (c.repair != FEM_KM_REPAIR_NONE && c.repair != FEM_KM_REPAIR_RANDOM && c.repair != FEM_KM_REPAIR_NEXT) {
    set_error("repair must be FEM_KM_REPAIR_NONE, FEM_KM_REPAIR_RANDOM or FEM_KM_REPAIR_NEXT");
    return FEM_ERR_BAD_ARG;
  }
  if (c.precision == FEM_PREC_FP32 && !(d == 2 || d == 4 || d == 8 || d == 16 || d == 32 || d == 64)) {
    set_error("k-means FP32 path supports d in {2,4,8,16,32,64}");
    return FEM_ERR_UNSUPPORTED;
  }
  if (c.precision == FEM_PREC_MIXED && !km_tc_supported(d, k)) {
    set_error("k-means mixed (tensor-core) path supports d = 32 and k <= 256 (got d=%d k=%d)", d, k);
    return FEM_ERR_UNSUPPORTED;
  }
  if (km_assign_smem(k, d) > 220 * 1024 && c.precision == FEM_PREC_FP32) {
    set_error("k*d too large for the shared-memory centroid table");
    return FEM_ERR_UNSUPPORTED;
  }
  FEM_TRY(select_device(c.device));
  fem_km *h = new (std::nothrow) fem_km();
  if (!h) return FEM_ERR_BAD_ARG;
  h->d = d;
  h->n = n;
  h->k = k;
  h->cfg = c;
  h->rng.seed((unsigned)c.seed);
  h->hg = new double[d];
  auto fail = [&](int st) {
    free_km(h);
    delete h;
    return st;
  };
  if (cudaStreamCreateWithFlags(&h->stream, cudaStreamNonBlocking) != cudaSuccess) return fail(FEM_ERR_CUDA);
  for (auto &e : h->ev)
    if (cudaEventCreate(&e) != cudaSuccess) return fail(FEM_ERR_CUDA);
  h->grid = sm_count();
  int st;
  if ((st = dalloc(&h->X, (size_t)n * d)) || (st = dalloc(&h->labels, n)) ||
      (st = dalloc(&h->cent, (size_t)k * d)) || (st = dalloc(&h->centf, (size_t)k * d)) ||
      (st = dalloc(&h->cnorm, k)) || (st = dalloc(&h->acc, (size_t)h->grid * k * d)) ||
      (st = dalloc(&h->cnt, (size_t)h->grid * k)) || (st = dalloc(&h->g, d)) ||
      (st = dalloc(&h->gs, d)) || (st = dalloc(&h->xscale, 1)) || (st = dalloc(&h->range, 2)) ||
      (st = dalloc(&h->out, (size_t)k * d + 2 * k)) || (st = dalloc(&h->dstat, 1)))
    return fail(st);
  if (cudaMallocHost(&h->hout, ((size_t)k * d + 2 * k) * 8) != cudaSuccess ||
      cudaMallocHost(&h->hstat, sizeof(DevStatus)) != cudaSuccess)
    return fail(FEM_ERR_CUDA);
  if (c.precision == FEM_PREC_FP32 && ((st = dalloc(&h->centg, (size_t)k * d)) || (st = dalloc(&h->hnorm, k))))
    return fail(st);
  if (c.precision == FEM_PREC_MIXED && (st = km_tc_create(h))) return fail(st);
  FEM_CUDA(cudaMemsetAsync(h->labels, 0, n * 4, h->stream));
  *out = h;
  return FEM_OK;
}

void fem_km_destroy(fem_km *h) {
  if (!h) return;
  if (h->stream) cudaStreamSynchronize(h->stream);
  free_km(h);
  delete h;
}

int fem_km_upload(fem_km *h, const float *X, int64_t ld) { return upload_km(h, X, ld, cudaMemcpyHostToDevice); }

int fem_km_upload_device(fem_km *h, const float *dX, int64_t ld) {
  return upload_km(h, dX, ld, cudaMemcpyDeviceToDevice);
}

int fem_km_init_data_structures(fem_km *h) {
  FEM_TRY(check(h));
  FEM_CUDA(cudaMemsetAsync(h->labels, 0, h->n * 4, h->stream));
  FEM_CUDA(cudaStreamSynchronize(h->stream));
  return FEM_OK;
}

int fem_km_seed(fem_km *h, uint64_t seed) {
  FEM_TRY(check(h));
  h->rng.seed((unsigned)seed);
  h->uni.reset();
  return FEM_OK;
}

int fem_km_set_rng_state(fem_km *h, const char *state) {
  FEM_TRY(check(h));
  std::mt19937_64 r;
  std::istringstream in(state ? state : "");
  if (!state || !(in >> r)) {
    set_error("fem_km_set_rng_state: not an mt19937_64 state");
    return FEM_ERR_BAD_ARG;
  }
  h->rng = r;
  h->uni.reset();
  return FEM_OK;
}

int fem_km_get_rng_state(fem_km *h, char *buf, size_t len) {
  FEM_TRY(check(h));
  std::ostringstream out;
  out << h->rng;
  const std::string t = out.str();
  if (!buf || len < t.size() + 1) {
    set_error("fem_km_get_rng_state: %zu bytes needed", t.size() + 1);
    return FEM_ERR_BAD_ARG;
  }
  std::memcpy(buf, t.c_str(), t.size() + 1);
  return FEM_OK;
}

// one Lloyd iteration (NaiveKMA::ComputeMSEAndCorrect / CorrectWithoutMSE,
// Clust/KMAlgorithm.cpp:148-255): labels, fixed-point sums, divide or repair;
// with `changed` the kernels also report whether any label moved
static int km_iterate(fem_km *h, double *centroids, double *fit, int64_t *counts, int *changed) {
  FEM_TRY(check(h));
  if (!h->have_data || !centroids) {
    set_error("k-means iteration needs an uploaded dataset and centroids");
    return FEM_ERR_STATE;
  }
  FEM_CUDA(cudaSetDevice(h->cfg.device));
  const int K = h->k, d = h->d;
  const size_t kd = (size_t)K * d;
  DevStatus z{};
  z.track_changes = changed != nullptr;
  *h->hstat = z;
  FEM_CUDA(cudaMemcpyAsync(h->dstat, h->hstat, sizeof(DevStatus), cudaMemcpyHostToDevice, h->stream));
  FEM_CUDA(cudaMemcpyAsync(h->cent, centroids, kd * 8, cudaMemcpyHostToDevice, h->stream));
  k_km_prep<<<(K + 3) / 4, 128, 0, h->stream>>>(h->cent, h->gs, K, d, h->centf, h->cnorm, h->centg, h->hnorm, h->range);
  FEM_CUDA(cudaGetLastError());
  FEM_CUDA(cudaEventRecord(h->ev[0], h->stream));
  if (h->cfg.precision == FEM_PREC_MIXED)
    FEM_TRY(km_tc_assign(h));
  else
    FEM_TRY(km_launch_assign_f32(h));
  FEM_CUDA(cudaEventRecord(h->ev[1], h->stream));
  k_km_final<<<K, 256, 0, h->stream>>>(h->acc, h->cnt, h->grid, K, d, ldexp(1.0, -h->shift), h->cent,
                                      h->g, h->out);
  FEM_CUDA(cudaGetLastError());
  FEM_CUDA(cudaEventRecord(h->ev[2], h->stream));
  FEM_CUDA(cudaMemcpyAsync(h->hout, h->out, (kd + 2 * K) * 8, cudaMemcpyDeviceToHost, h->stream));
  FEM_CUDA(cudaMemcpyAsync(h->hstat, h->dstat, sizeof(DevStatus), cudaMemcpyDeviceToHost, h->stream));
  FEM_CUDA(cudaStreamSynchronize(h->stream));
  if (h->hstat->timeout) {
    set_error("a bounded device wait timed out in the tensor-core k-means kernel");
    return FEM_ERR_TIMEOUT;
  }
  float a = 0, b = 0;
  cudaEventElapsedTime(&a, h->ev[0], h->ev[1]);
  cudaEventElapsedTime(&b, h->ev[1], h->ev[2]);
  h->t_assign = a;
  h->t_update = b;
  double total = h->xg2;
  for (int j = 0; j < K; j++) total += h->hout[kd + K + j];
  if (fit) *fit = total / (double)h->n;
  // NaiveKMA: divide, or CentroidRandomRepair in index order
  for (int j = 0; j < K; j++) {
    const int64_t nj = (int64_t)h->hout[kd + j];
    if (counts) counts[j] = nj;
    if (nj > 0) {
      for (int q = 0; q < d; q++) centroids[(size_t)j * d + q] = h->hout[(size_t)j * d + q];
    } else if (h->cfg.repair != FEM_KM_REPAIR_NONE) {
      int64_t src;
      if (h->cfg.repair == FEM_KM_REPAIR_RANDOM) {
        src = (int64_t)(h->uni(h->rng) * (double)h->n);
      } else {
        src = h->next_repair;
        if (++h->next_repair == h->n) h->next_repair = 0;
      }
      std::vector<float> row(d);
      FEM_CUDA(cudaMemcpy(row.data(), h->X + src * d, d * 4, cudaMemcpyDeviceToHost));
      for (int q = 0; q < d; q++) centroids[(size_t)j * d + q] = (double)row[q];
    }
  }
  if (changed) *changed = h->hstat->changed;
  return FEM_OK;
}

int fem_km_compute_mse_and_correct(fem_km *h, double *centroids, double *fit, int64_t *counts) {
  return km_iterate(h, centroids, fit, counts, nullptr);
}

int fem_km_correct_without_mse(fem_km *h, double *centroids, int *changed) {
  if (!changed) {
    set_error("fem_km_correct_without_mse: null output");
    return FEM_ERR_BAD_ARG;
  }
  return km_iterate(h, centroids, nullptr, nullptr, changed);
}

int fem_km_run(fem_km *h, double *centroids, double min_rel, int max_iter, double *best_fit, int *iters) {
  FEM_TRY(check(h));
  double best = DBL_MAX;
  FEM_TRY(fem_km_init_data_structures(h));
  if (max_iter == 0) {
    if (best_fit) *best_fit = 0.0;
    if (iters) *iters = 0;
    return FEM_OK;
  }
  int i;
  for (i = 1;; i++) {
    double fit = 0.0;
    FEM_TRY(fem_km_compute_mse_and_correct(h, centroids, &fit, nullptr));
    const double rel = (best - fit) / best;
    if (fit < std::nextafter(fit, best))
      best = fit;
    else
      break;
    if (min_rel > 0.0 && min_rel > rel) break;
    if (max_iter > 0 && i == max_iter - 1) break;
  }
  if (best_fit) *best_fit = best;
  if (iters) *iters = i;
  return FEM_OK;
}

int fem_km_get_assignment(fem_km *h, int32_t *labels) {
  FEM_TRY(check(h));
  if (!labels) return FEM_ERR_BAD_ARG;
  FEM_CUDA(cudaMemcpyAsync(labels, h->labels, h->n * 4, cudaMemcpyDeviceToHost, h->stream));
  FEM_CUDA(cudaStreamSynchronize(h->stream));
  return FEM_OK;
}

int fem_km_stats(fem_km *h, int64_t *rechecked_rows, double *assign_ms, double *update_ms) {
  FEM_TRY(check(h));
  if (rechecked_rows) *rechecked_rows = h->hstat ? h->hstat->rechecked : 0;
  if (assign_ms) *assign_ms = h->t_assign;
  if (update_ms) *update_ms = h->t_update;
  return FEM_OK;
}

}  // extern "C"
