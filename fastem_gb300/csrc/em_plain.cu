// em_plain.cu -- CUDA-core EM sweep in FP32 or FP64 (the "plain" precision
// forms), plus the FP64 per-component factorisation shared by every form.
//
// One sweep = SimpleMatrixEM::PrecomputeDensityMatrix + MStep + the
// RegularizeCovariances / InitDensities that TrainNoCopy runs after it
// (EM2/MatrixEM.cpp:275-378, EM2/EMAlgorithm.cpp:139-191).
//
// Layout in HBM: X is n x d float rows; posteriors R are component-major
// (k rows, post_ld(n) apart) so every per-component pass streams contiguous memory; the
// inverse Cholesky factors are stored as W_j = L_j^-1 (lower, row-major), so
// the Mahalanobis term of point x is ||W_j (x - mu_j)||^2 (the reference
// multiplies by CholInvC = W_j^T from the right, EM2/MatrixEM.cpp:76).
#include <cfloat>
#include <cmath>
#include <cstring>

#include "fem_internal.cuh"
#include "em_kernels.cuh"
#include "em_factor.cuh"
#include "em_tri.cuh"

namespace fem {

// ------------------------------------------------------------ reductions
__device__ __forceinline__ double warp_sum(double v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
  return v;
}

// deterministic block sum (fixed shuffle tree, fixed warp order); result in thread 0
template <int NT>
__device__ double block_sum(double v, double *red) {
  v = warp_sum(v);
  const int w = threadIdx.x >> 5, l = threadIdx.x & 31;
  __syncthreads();
  if (l == 0) red[w] = v;
  __syncthreads();
  double s = 0.0;
  if (threadIdx.x == 0)
    for (int i = 0; i < NT / 32; i++) s += red[i];
  return s;
}

template <typename T> __device__ __forceinline__ T t_exp(T x);
template <> __device__ __forceinline__ float t_exp(float x) { return expf(x); }
template <> __device__ __forceinline__ double t_exp(double x) { return exp(x); }
template <typename T> __device__ __forceinline__ T t_log(T x);
template <> __device__ __forceinline__ float t_log(float x) { return logf(x); }
template <> __device__ __forceinline__ double t_log(double x) { return log(x); }

// online log-sum-exp step (max-shifted), -inf entries contribute nothing
template <typename T>
__device__ __forceinline__ void lse_push(T l, T &mx, T &se) {
  if (l > mx) {
    se = se * t_exp(mx - l) + T(1);
    mx = l;
  } else if (l > -INFINITY) {
    se += t_exp(l - mx);
  }
}

// ================================================================ E-step
// MatrixEMBase::BlockDensities + PostProcessDensityMatrix
// (EM2/MatrixEM.cpp:39-51,69-81) for d <= D (columns d..D-1 are zero in the
// rows and the factors).  A CTA takes 128 P points, P per thread; the factors'
// lower triangles, means and log coefficients of KC components are copied
// asynchronously one group ahead.  Per component a thread centres its points,
// forms ||W_j (x - mu_j)||^2 and writes l_ij to R.
// FP32 is bound by the FMA pipe and the 16-byte broadcast loads of the factor,
// which serve P points; columns are multiplied in pairs (em_tri.cuh) and the
// log-sum-exp takes one exponential and no branch.  Against one point per
// thread, one component at a time and a branch (GB300): 250007 x 16 x 200
// 893 -> 548 us, 400000 x 32 x 40 808 -> 501, 300000 x 4 x 200 276 -> 228; where
// the dimension had no kernel of its own, 250007 x 13 x 135 1590 -> 445,
// 200000 x 40 x 60 5264 -> 726.
// FP64: 100000 x 8 x 10 231 -> 167 us, 100000 x 13 x 10 375 -> 332,
// 20000 x 4 x 5 29 -> 19.
constexpr int kEPThreads = 128;

template <typename T, int D, int KC>
struct EstepBuf {
  static constexpr int TRI = tri_off(D);
  static constexpr int CB = KC * (TRI + D + 4);     // elements (log coefficients at the end)
};

template <typename T, int BYTES>
__device__ __forceinline__ void ep_copy(T *dst, const T *src, bool valid) {
  const uint32_t da = static_cast<uint32_t>(__cvta_generic_to_shared(dst));
  asm volatile("cp.async.ca.shared.global [%0], [%1], %2, %3;\n" ::"r"(da), "l"(src), "n"(BYTES), "r"(valid ? BYTES : 0)
               : "memory");
}

// components [j0, j0 + kc) into buf; rows of the triangle from d on and columns
// from d on become zero.  16-byte copies when a row of the factors is a
// multiple of 16 bytes.
template <typename T, int D, int KC>
__device__ __forceinline__ void ep_stage(T *buf, const T *__restrict__ mu, const T *__restrict__ W,
                                         const T *__restrict__ logc, int d, int j0, int kc) {
  constexpr int TRI = tri_off(D), V = 16 / sizeof(T);
  T *m = buf + KC * TRI, *l = m + KC * D;
  const int tid = threadIdx.x;
  const T *Wj = W + (size_t)j0 * d * d, *mj = mu + (size_t)j0 * d;
  auto copy = [&](auto vec) {
    constexpr int E = decltype(vec)::value, Q = D / E;
    for (int e = tid; e < kc * D * Q; e += kEPThreads) {
      const int jj = e / (D * Q), r = (e / Q) % D, c = E * (e % Q);
      if (c >= tri_row(r)) continue;
      const bool v = r < d && c < d;
      ep_copy<T, E * (int)sizeof(T)>(buf + jj * TRI + tri_off(r) + c, Wj + (v ? (jj * d + r) * d + c : 0), v);
    }
    for (int e = tid; e < kc * Q; e += kEPThreads) {
      const int jj = e / Q, q = E * (e % Q);
      ep_copy<T, E * (int)sizeof(T)>(m + jj * D + q, mj + (q < d ? jj * d + q : 0), q < d);
    }
  };
  if (d % V == 0)
    copy(std::integral_constant<int, V>());
  else
    copy(std::integral_constant<int, 1>());
  for (int e = tid; e < kc; e += kEPThreads) ep_copy<T, (int)sizeof(T)>(l + e, logc + j0 + e, true);
  asm volatile("cp.async.commit_group;\n" ::: "memory");
}

// FP32, with an online log-sum-exp; a second pass turns R into exp(l - LSE).
// Rows in registers, or (XS) as columns of pairs in shared memory.
template <int D, int P, bool XS, int KC>
__global__ void __launch_bounds__(kEPThreads)
k_estep_f32(const float *__restrict__ X, int64_t n, int d, int K, const float *__restrict__ mu,
            const float *__restrict__ W, const float *__restrict__ logc, float *__restrict__ R,
            double *__restrict__ part) {
  using S = EstepBuf<float, D, KC>;
  constexpr int TRI = S::TRI, PS = kEPThreads * P + 1;
  extern __shared__ __align__(16) float esm[];
  __shared__ double red[kEPThreads / 32];
  float *cbuf = esm;
  uint64_t *sx = reinterpret_cast<uint64_t *>(esm + 2 * S::CB) + threadIdx.x;
  const int tid = threadIdx.x;
  const int64_t p0 = (int64_t)blockIdx.x * kEPThreads * P;
  ep_stage<float, D, KC>(cbuf, mu, W, logc, d, 0, min(KC, K));
  uint64_t x[P][XS ? 1 : D / 2];
  bool live[P];
#pragma unroll
  for (int p = 0; p < P; p++) live[p] = p0 + tid + p * kEPThreads < n;
  if constexpr (XS) {
    float *sf = esm + 2 * S::CB;
    const int np = (int)min((int64_t)kEPThreads * P, n - p0);
    const float *src = X + (size_t)p0 * d;
#pragma unroll 8
    for (int e = tid; e < kEPThreads * P * D; e += kEPThreads) {
      const int pt = e / D, q = e % D;
      sf[2 * ((q / 2) * PS + pt) + (q & 1)] = (pt < np && q < d) ? __ldg(src + pt * d + q) : 0.f;
    }
  } else {
#pragma unroll
    for (int p = 0; p < P; p++) {
      const float *xr = X + (live[p] ? p0 + tid + p * kEPThreads : 0) * d;
      if (d == D) {
#pragma unroll
        for (int q = 0; q < D / 4; q++) {
          const ulonglong2 v = __ldg(reinterpret_cast<const ulonglong2 *>(xr) + q);
          x[p][2 * q] = v.x, x[p][2 * q + 1] = v.y;
        }
      } else {
#pragma unroll
        for (int q = 0; q < D / 2; q++)
          x[p][q] = f2_pack(2 * q < d ? __ldg(xr + 2 * q) : 0.f, 2 * q + 1 < d ? __ldg(xr + 2 * q + 1) : 0.f);
      }
    }
  }
  float mx[P], se[P];
#pragma unroll
  for (int p = 0; p < P; p++) mx[p] = -INFINITY, se[p] = 0.f;
  int b = 0;
  for (int j0 = 0; j0 < K; j0 += KC, b ^= 1) {
    const int kc = min(KC, K - j0);
    if (j0 + KC < K)
      ep_stage<float, D, KC>(cbuf + (b ^ 1) * S::CB, mu, W, logc, d, j0 + KC, min(KC, K - j0 - KC));
    else
      asm volatile("cp.async.commit_group;\n" ::: "memory");   // keeps the wait count uniform
    asm volatile("cp.async.wait_group 1;\n" ::: "memory");
    __syncthreads();
    const float *sW = cbuf + b * S::CB, *sm = sW + KC * TRI, *sl = sm + KC * D;
    float *Rj = R + (size_t)j0 * post_ld(n) + p0 + tid;
#pragma unroll 1
    for (int jj = 0; jj < kc; jj++, Rj += post_ld(n)) {
      const uint64_t *m = reinterpret_cast<const uint64_t *>(sm + jj * D);
      uint64_t t[P][D / 2];
#pragma unroll
      for (int q = 0; q < D / 2; q++) {
        const uint64_t mq = m[q];
#pragma unroll
        for (int p = 0; p < P; p++) t[p][q] = f2_sub(XS ? sx[q * PS + p * kEPThreads] : x[p][XS ? 0 : q], mq);
      }
      float s[P];
      tri_norms<D, P>(t, sW + jj * TRI, s);
      const float lc = sl[jj];
#pragma unroll
      for (int p = 0; p < P; p++) {
        const float l = lc - 0.5f * s[p];
        if (live[p]) Rj[p * kEPThreads] = l;
        lse_add(l, mx[p], se[p]);
      }
    }
    __syncthreads();
  }
  double v = 0.0;
  float lse[P];
#pragma unroll
  for (int p = 0; p < P; p++) {
    lse[p] = mx[p] + logf(se[p]);
    if (live[p]) v += (double)lse[p];
  }
  float *Rt = R + p0 + tid;
#pragma unroll 4
  for (int j = 0; j < K; j++)
#pragma unroll
    for (int p = 0; p < P; p++)
      if (live[p]) {
        float *q = Rt + (size_t)j * post_ld(n) + p * kEPThreads;
        *q = expf(*q - lse[p]);
      }
  const double s = block_sum<kEPThreads>(v, red);
  if (tid == 0) part[blockIdx.x] = s;
}

// FP64 is bound by its pipe, of which an exponential takes half a d = 8
// component's share: the maximum only is kept and each exponential is taken
// once.  R holds l, then exp(l - max), then that over its sum.
template <int D, int P, int KC>
__global__ void __launch_bounds__(kEPThreads)
k_estep_f64(const float *__restrict__ X, int64_t n, int d, int K, const double *__restrict__ mu,
            const double *__restrict__ W, const double *__restrict__ logc, double *__restrict__ R,
            double *__restrict__ part) {
  using S = EstepBuf<double, D, KC>;
  constexpr int TRI = S::TRI;
  extern __shared__ __align__(16) double dsm[];
  __shared__ double red[kEPThreads / 32];
  const int tid = threadIdx.x;
  const int64_t p0 = (int64_t)blockIdx.x * kEPThreads * P;
  ep_stage<double, D, KC>(dsm, mu, W, logc, d, 0, min(KC, K));
  float x[P][D];
  bool live[P];
  double mx[P], se[P];
#pragma unroll
  for (int p = 0; p < P; p++) {
    live[p] = p0 + tid + p * kEPThreads < n;
    mx[p] = -INFINITY, se[p] = 0.0;
    const float *xr = X + (live[p] ? p0 + tid + p * kEPThreads : 0) * d;
#pragma unroll
    for (int q = 0; q < D; q++) x[p][q] = q < d ? __ldg(xr + q) : 0.f;
  }
  double *Rt = R + p0 + tid;
  int b = 0;
  for (int j0 = 0; j0 < K; j0 += KC, b ^= 1) {
    const int kc = min(KC, K - j0);
    if (j0 + KC < K)
      ep_stage<double, D, KC>(dsm + (b ^ 1) * S::CB, mu, W, logc, d, j0 + KC, min(KC, K - j0 - KC));
    else
      asm volatile("cp.async.commit_group;\n" ::: "memory");
    asm volatile("cp.async.wait_group 1;\n" ::: "memory");
    __syncthreads();
    const double *sW = dsm + b * S::CB, *sm = sW + KC * TRI, *sl = sm + KC * D;
    for (int jj = 0; jj < kc; jj++) {
      double t[P][D], s[P];
#pragma unroll
      for (int q = 0; q < D; q++) {
        const double mq = sm[jj * D + q];
#pragma unroll
        for (int p = 0; p < P; p++) t[p][q] = (double)x[p][q] - mq;
      }
      tri_norms<D, P>(t, sW + jj * TRI, s);
      const double lc = sl[jj];
#pragma unroll
      for (int p = 0; p < P; p++) {
        const double l = lc - 0.5 * s[p];
        if (live[p]) Rt[(size_t)(j0 + jj) * post_ld(n) + p * kEPThreads] = l;
        mx[p] = l > mx[p] ? l : mx[p];
      }
    }
    __syncthreads();
  }
#pragma unroll 4
  for (int j = 0; j < K; j++)
#pragma unroll
    for (int p = 0; p < P; p++)
      if (live[p]) {
        double *q = Rt + (size_t)j * post_ld(n) + p * kEPThreads;
        const double l = *q, e = exp(l - mx[p]);
        if (l > -INFINITY) se[p] += e;
        *q = e;
      }
  double v = 0.0, c[P];
#pragma unroll
  for (int p = 0; p < P; p++) {
    c[p] = 1.0 / se[p];
    if (live[p]) v += mx[p] + log(se[p]);
  }
#pragma unroll 4
  for (int j = 0; j < K; j++)
#pragma unroll
    for (int p = 0; p < P; p++)
      if (live[p]) Rt[(size_t)j * post_ld(n) + p * kEPThreads] *= c[p];
  const double s = block_sum<kEPThreads>(v, red);
  if (tid == 0) part[blockIdx.x] = s;
}

// d = 64: one point per thread, components one at a time.  The unrolled triangle
// of the kernels above no longer fits the instruction cache (FP32, 20000 rows,
// 10 components: 108 us against 75 here) or, in FP64, the registers (30000 rows,
// 10 components: 3446 us against 1458; k_estep_plain_generic takes 1776).
template <typename T>
__global__ void __launch_bounds__(128)
k_estep_64(const float *__restrict__ X, int64_t n, int K, const T *__restrict__ mu,
              const T *__restrict__ W, const T *__restrict__ logc, T *__restrict__ R,
              double *__restrict__ part) {
  constexpr int D = 64;
  __shared__ __align__(16) T sW[D * D];
  __shared__ __align__(16) T smu[D];
  __shared__ double red[4];
  const int tid = threadIdx.x;
  const int64_t i = (int64_t)blockIdx.x * 128 + tid;
  const bool valid = i < n;
  float x[D];
#pragma unroll
  for (int q = 0; q < D; q++) x[q] = valid ? X[i * D + q] : 0.f;
  T mx = -INFINITY, se = T(0);
  for (int j = 0; j < K; j++) {
    __syncthreads();
    for (int e = tid; e < D * D; e += 128) sW[e] = W[(size_t)j * D * D + e];
    if (tid < D) smu[tid] = mu[(size_t)j * D + tid];
    __syncthreads();
    T t[D];
#pragma unroll
    for (int q = 0; q < D; q++) t[q] = (T)x[q] - smu[q];
    T s = T(0);
#pragma unroll
    for (int kk = 0; kk < D; kk++) {
      T y = T(0);
#pragma unroll
      for (int m = 0; m <= kk; m++) y = fma(t[m], sW[kk * D + m], y);
      s = fma(y, y, s);
    }
    const T l = logc[j] - T(0.5) * s;
    if (valid) R[(size_t)j * post_ld(n) + i] = l;
    lse_push(l, mx, se);
  }
  const T lse = mx + t_log(se);
  if (valid)
    for (int j = 0; j < K; j++) {
      T *p = R + (size_t)j * post_ld(n) + i;
      *p = t_exp(*p - lse);
    }
  double s = block_sum<128>(valid ? (double)lse : 0.0, red);
  if (tid == 0) part[blockIdx.x] = s;
}

// runtime dimension: centred point in shared memory, factor read through L1
template <typename T>
__global__ void __launch_bounds__(64)
k_estep_plain_generic(const float *__restrict__ X, int64_t n, int d, int K,
                      const T *__restrict__ mu, const T *__restrict__ W,
                      const T *__restrict__ logc, T *__restrict__ R, double *__restrict__ part) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  T *sT = (T *)smem_raw;  // 64 x (d+1)
  __shared__ double red[2];
  const int tid = threadIdx.x;
  const int64_t i = (int64_t)blockIdx.x * 64 + tid;
  const bool valid = i < n;
  T *t = sT + (size_t)tid * (d + 1);
  T mx = -INFINITY, se = T(0);
  for (int j = 0; j < K; j++) {
    const T *mj = mu + (size_t)j * d;
    const T *Wj = W + (size_t)j * d * d;
    for (int q = 0; q < d; q++) t[q] = valid ? ((T)X[i * d + q] - mj[q]) : T(0);
    T s = T(0);
    for (int kk = 0; kk < d; kk++) {
      const T *wr = Wj + (size_t)kk * d;
      T y = T(0);
      for (int m = 0; m <= kk; m++) y = fma(t[m], wr[m], y);
      s = fma(y, y, s);
    }
    const T l = logc[j] - T(0.5) * s;
    if (valid) R[(size_t)j * post_ld(n) + i] = l;
    lse_push(l, mx, se);
  }
  const T lse = mx + t_log(se);
  if (valid)
    for (int j = 0; j < K; j++) {
      T *p = R + (size_t)j * post_ld(n) + i;
      *p = t_exp(*p - lse);
    }
  double s = block_sum<64>(valid ? (double)lse : 0.0, red);
  if (tid == 0) part[blockIdx.x] = s;
}

// register-tiled form for d > 64: a CTA of 256 threads takes P = 32 PT
// points.  Per component the centred points are staged once, transposed
// (sT[m][p], pitch P + 1), and L^-1 is streamed through 64 x 64 chunks
// (sW[m][o], pitch 68) up to the diagonal: output chunk o0 needs columns
// m < o0 + 64 only (the factor's upper triangle is stored as zeros, so the
// diagonal chunk needs no mask).  Thread (tp, to) = (tid / 8, tid % 8)
// holds y for points tp + 32 i (i < PT) and outputs o0 + 8 to + (0..7): per
// column m, PT broadcast loads of t and one 8-wide load of W feed 8 PT FMAs.
// s = ||y||^2 is summed per thread over its outputs, then over the 8 threads
// of a point group by a fixed shuffle tree (run-to-run reproducible).
constexpr int kETileOC = 64;              // outputs per chunk
constexpr int kETileMC = 64;              // factor columns per chunk
constexpr int kETileWP = kETileOC + 4;    // sW pitch (16-byte rows)
constexpr size_t kMaxDynSmem = 232448;    // opt-in shared memory per CTA (227 KB)

// 8 consecutive elements from a 16-byte-aligned shared-memory address
__device__ __forceinline__ void load8(const float *p, float (&v)[8]) {
  const float4 a = reinterpret_cast<const float4 *>(p)[0], b = reinterpret_cast<const float4 *>(p)[1];
  v[0] = a.x, v[1] = a.y, v[2] = a.z, v[3] = a.w, v[4] = b.x, v[5] = b.y, v[6] = b.z, v[7] = b.w;
}
__device__ __forceinline__ void load8(const double *p, double (&v)[8]) {
#pragma unroll
  for (int q = 0; q < 4; q++) {
    const double2 a = reinterpret_cast<const double2 *>(p)[q];
    v[2 * q] = a.x, v[2 * q + 1] = a.y;
  }
}

template <typename T, int PT>
constexpr size_t estep_tiled_smem(int d) {
  return ((size_t)((d + 63) & ~63) * (32 * PT + 1) + (size_t)kETileMC * kETileWP + 32 * PT) * sizeof(T);
}

template <typename T, int PT>
__global__ void __launch_bounds__(256)
k_estep_plain_tiled(const float *__restrict__ X, int64_t n, int d, int K, const T *__restrict__ mu,
                    const T *__restrict__ W, const T *__restrict__ logc, T *__restrict__ R,
                    double *__restrict__ part) {
  constexpr int P = 32 * PT, TP = P + 1;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const int dpad = (d + 63) & ~63;
  T *sW = (T *)smem_raw;                       // kETileMC x kETileWP (first: 16-byte aligned rows)
  T *sT = sW + kETileMC * kETileWP;            // dpad x TP
  T *sLse = sT + (size_t)dpad * TP;            // P
  __shared__ double red[8];
  const int tid = threadIdx.x, to = tid & 7, tp = tid >> 3;
  const int64_t i0 = (int64_t)blockIdx.x * P;
  T mx[PT], se[PT];
#pragma unroll
  for (int i = 0; i < PT; i++) mx[i] = -INFINITY, se[i] = T(0);
  for (int j = 0; j < K; j++) {
    const T *mj = mu + (size_t)j * d;
    const T *Wj = W + (size_t)j * d * d;
    __syncthreads();                           // the previous component's reads of sT are done
    // coalesced rows of X (column fastest); pitch TP puts consecutive
    // columns of one point in consecutive banks
    for (int e = tid; e < P * dpad; e += 256) {
      const int p = e / dpad, m = e - p * dpad;
      T t = T(0);
      if (m < d && i0 + p < n) t = (T)X[(i0 + p) * d + m] - mj[m];
      sT[(size_t)m * TP + p] = t;
    }
    T s[PT];
#pragma unroll
    for (int i = 0; i < PT; i++) s[i] = T(0);
    for (int o0 = 0; o0 < dpad; o0 += kETileOC) {
      T y[PT][8];
#pragma unroll
      for (int i = 0; i < PT; i++)
#pragma unroll
        for (int o = 0; o < 8; o++) y[i][o] = T(0);
      for (int m0 = 0; m0 <= o0; m0 += kETileMC) {
        __syncthreads();                       // sW free (and sT staged, on the first chunk)
        for (int e = tid; e < kETileOC * kETileMC; e += 256) {
          const int o = e / kETileMC, m = e - o * kETileMC;
          const int go = o0 + o, gm = m0 + m;
          sW[m * kETileWP + o] = (go < d && gm < d) ? Wj[(size_t)go * d + gm] : T(0);
        }
        __syncthreads();
        const T *tcol = sT + (size_t)m0 * TP + tp;
        const T *wrow = sW + to * 8;
#pragma unroll 4
        for (int m = 0; m < kETileMC; m++) {
          T tv[PT], wv[8];
#pragma unroll
          for (int i = 0; i < PT; i++) tv[i] = tcol[(size_t)m * TP + 32 * i];
          load8(wrow + m * kETileWP, wv);
#pragma unroll
          for (int i = 0; i < PT; i++)
#pragma unroll
            for (int o = 0; o < 8; o++) y[i][o] = fma(tv[i], wv[o], y[i][o]);
        }
      }
#pragma unroll
      for (int i = 0; i < PT; i++)
#pragma unroll
        for (int o = 0; o < 8; o++) s[i] = fma(y[i][o], y[i][o], s[i]);
    }
    // the 8 threads of a point group are 8 consecutive lanes
#pragma unroll
    for (int i = 0; i < PT; i++) {
      s[i] += __shfl_xor_sync(0xffffffffu, s[i], 1);
      s[i] += __shfl_xor_sync(0xffffffffu, s[i], 2);
      s[i] += __shfl_xor_sync(0xffffffffu, s[i], 4);
    }
    if (to == 0) {
      const T lc = logc[j];
#pragma unroll
      for (int i = 0; i < PT; i++) {
        const int64_t pi = i0 + tp + 32 * i;
        const T l = lc - T(0.5) * s[i];
        if (pi < n) R[(size_t)j * post_ld(n) + pi] = l;
        lse_push(l, mx[i], se[i]);
      }
    }
  }
  double v = 0.0;
  if (to == 0)
#pragma unroll
    for (int i = 0; i < PT; i++) {
      const T lse = mx[i] + t_log(se[i]);
      sLse[tp + 32 * i] = lse;
      if (i0 + tp + 32 * i < n) v += (double)lse;
    }
  __syncthreads();                             // sLse and every l_ij of this CTA written
  for (int e = tid; e < K * P; e += 256) {
    const int j = e / P, p = e - j * P;
    if (i0 + p < n) {
      T *q = R + (size_t)j * post_ld(n) + i0 + p;
      *q = t_exp(*q - sLse[p]);
    }
  }
  const double ls = block_sum<256>(v, red);
  if (tid == 0) part[blockIdx.x] = ls;
}

// single-block deterministic sum of the per-block log-likelihood partials
__global__ void __launch_bounds__(1024) k_reduce_logl(const double *part, int64_t np, DevStatus *st) {
  __shared__ double red[32];
  double v = 0.0;
  for (int64_t b = threadIdx.x; b < np; b += 1024) v += part[b];
  double s = block_sum<1024>(v, red);
  if (threadIdx.x == 0) st->logl = s;
}

// PosteriorSum, Means = MeanSums / PosteriorSum, Probs = PosteriorSum / N
// (EM2/MatrixEM.cpp:341-343,375); one block per component, blocks summed in order
// and split over the 8 warps of its CTA (lane = column 0, the posterior sum,
// or 1 + dimension), combined in warp order
template <typename T>
__global__ void __launch_bounds__(256)
k_final_means(const double *__restrict__ part, int G, int K, int d, int64_t n, double *__restrict__ mu,
              double *__restrict__ pi, double *__restrict__ psum, T *__restrict__ muT) {
  const int j = blockIdx.x, lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  __shared__ double red[8][32], s1;
  for (int c0 = 0; c0 <= d; c0 += 32) {
    const int c = c0 + lane;
    double s = 0.0;
    if (c <= d) {
#pragma unroll 8
      for (int g = w; g < G; g += 8) s += part[((size_t)g * K + j) * (d + 1) + c];
    }
    red[w][lane] = s;
    __syncthreads();
    if (w == 0 && c <= d) {
#pragma unroll
      for (int q = 1; q < 8; q++) s += red[q][lane];
      red[0][lane] = s;
      if (c == 0) {
        s1 = s;
        psum[j] = s;
        pi[j] = s / (double)n;
      }
    }
    __syncthreads();
    if (w == 0 && c >= 1 && c <= d) {
      const double m = red[0][lane] / s1;
      mu[(size_t)j * d + c - 1] = m;
      muT[(size_t)j * d + c - 1] = (T)m;
    }
  }
}

// ======================================================= factorisation
// EMAlgorithm::RegularizeCovariances + NormalDensity::Init + CalcLogCoeffs
// (EM2/EMAlgorithm.cpp:237-244, EM2/NormalDensity.cpp:43-65,
// EM2/MatrixEM.cpp:83-87) in FP64, one CTA per component: symmetric copy of
// the lower triangle, right-looking Cholesky (a pivot <= 0 fails, as in
// Eigen's LLT), log det = 2 sum log L_ii, W = L^-1, log coefficient
// log pi_j - d/2 log 2pi - 1/2 log det, and an upper bound of the condition
// number lambda_max / lambda_min folded into st->cond_bound: lambda_max <=
// ||Sigma||_F and 1 / lambda_min = ||L^-1||_2^2 <= ||L^-1||_F^2, at most d^1.5
// times the true value; the caller runs the exact eigenvalues
// (block_jacobi_cond) only when the bound does not settle a test.
constexpr double kLog2Pi = 1.8378770664093454835606594728112;   // log(2 pi)

// Up to d = kFactorSmemD both matrices live in shared memory (k_factor_smem);
// above it the Cholesky runs blocked over matrices in L2 (k_factor) and L^-1 by
// column blocks on SMs of their own (k_factor_inverse).
template <typename T, int NS>
__global__ void __launch_bounds__(kFactorThreads)
k_factor_smem(int K, int d, double reg, int regularize, double *__restrict__ sigma, const double *__restrict__ pi,
              const double *__restrict__ mu, double *__restrict__ work, double *__restrict__ linv,
              double *__restrict__ logdet, double *__restrict__ logc, T *__restrict__ muT, T *__restrict__ linvT,
              T *__restrict__ logcT, DevStatus *st) {
  const int j = blockIdx.x, tid = threadIdx.x, ld = factor_ld(d);
  extern __shared__ double fsm[];
  __shared__ double red[3 * kFactorThreads / 32];
  __shared__ double s_logpi;
  double *A = fsm, *W = A + d * ld, *piv = W + d * ld, *rd = piv + d, *m = rd + d;
  double *S = sigma + (size_t)j * d * d;
  double add = 0.0;
  const bool rg = regularize && reg != 0.0;
  if (rg) {
    // (1 - reg) S + (reg tr(S) / d) I
    double t[1] = {tid < d ? S[(size_t)tid * d + tid] : 0.0};
    block_sums(t, red);
    add = reg * t[0] / (double)d;
  }
  double sums[3] = {0.0, 0.0, 0.0};      // ||Sigma||_F^2, ||L^-1||_F^2, log det
  for (int e = tid; e < d * d; e += kFactorThreads) {
    const int r = e / d, c = e - r * d;
    double v = S[e];
    if (rg) {
      v = v * (1.0 - reg) + (r == c ? add : 0.0);
      S[e] = v;
    }
    if (c <= r) {
      A[r * ld + c] = v;
      sums[0] = fma(c == r ? v : 2.0 * v, v, sums[0]);
    }
  }
  for (int q = tid; q < d; q += kFactorThreads) muT[(size_t)j * d + q] = (T)mu[(size_t)j * d + q];
  __syncthreads();
  if (!block_factor_smem<NS>(A, W, piv, rd, m, d, ld)) {
    if (tid == 0) atomicMin(&st->chol_failed, j);
    return;
  }
  if (tid < d) sums[2] = log(piv[tid]);
  if (tid == kFactorThreads - 1) s_logpi = log(pi[j]);
  for (int e = tid; e < d * d; e += kFactorThreads) {
    const int r = e / d, c = e - r * d;
    const double w = c > r ? 0.0 : (c == r ? rd[r] : W[r * ld + c] * rd[r]);
    sums[1] = fma(w, w, sums[1]);
    linv[(size_t)j * d * d + e] = w;
    linvT[(size_t)j * d * d + e] = (T)w;
    // the wide E-step keeps L
    if (d > 64) work[(size_t)j * d * d + e] = c > r ? 0.0 : (c == r ? sqrt(piv[r]) : A[r * ld + c] * rd[c]);
  }
  block_sums(sums, red);
  if (tid == 0) {
    // non-negative doubles order like their bit patterns
    atomicMax(reinterpret_cast<unsigned long long *>(&st->cond_bound),
              (unsigned long long)__double_as_longlong(sqrt(sums[0]) * sums[1]));
    logdet[j] = sums[2];
    const double lc = s_logpi - 0.5 * (double)d * kLog2Pi - 0.5 * sums[2];
    logc[j] = lc;
    logcT[j] = (T)lc;
  }
}

constexpr int kInvThreads = 128;
// fpart, doubles per component: ||L^-1||_F^2 of each column block, ||Sigma||_F^2
// (negative: no factor)
constexpr int kFactorParts = kFactorMaxD / 32 + 1;

template <typename T>
__global__ void __launch_bounds__(kFactorThreads)
k_factor(int K, int d, double reg, int regularize, double *__restrict__ sigma,
         const double *__restrict__ pi, const double *__restrict__ mu, double *__restrict__ work,
         double *__restrict__ fpart, double *__restrict__ logdet, double *__restrict__ logc,
         T *__restrict__ muT, T *__restrict__ logcT, DevStatus *st) {
  const int j = blockIdx.x, tid = threadIdx.x, nt = blockDim.x;
  double *S = sigma + (size_t)j * d * d;
  double *A = work + (size_t)j * d * d;
  double *part = fpart + (size_t)j * kFactorParts;
  extern __shared__ double fsm[];
  __shared__ double red[kFactorThreads / 32];
  if (regularize && reg != 0.0) block_regularize(S, d, reg);
  if (!block_cholesky_panels(S, d, A, fsm)) {
    if (tid == 0) {
      atomicMin(&st->chol_failed, j);
      part[kFactorParts - 1] = -1.0;
    }
    return;
  }
  const double ld = block_chol_logdet(A, d);
  const double fs = block_frob2(S, d, red);
  if (tid == 0) {
    part[kFactorParts - 1] = fs;
    logdet[j] = ld;
    const double lc = log(pi[j]) - 0.5 * (double)d * log(2.0 * M_PI) - 0.5 * ld;
    logc[j] = lc;
    logcT[j] = (T)lc;
  }
  for (int q = tid; q < d; q += nt) muT[(size_t)j * d + q] = (T)mu[(size_t)j * d + q];
}

// Columns 32 b .. 32 b + 31 of W_j = L_j^-1 (lower, row-major; lane = column),
// j = blockIdx.x % K and b = blockIdx.x / K, so the blocks with the most rows
// start first.  The columns of an inverse are independent, and one SM's FP64
// pipe (2 lanes per clock) is the limit of a whole matrix: spread like this
// K = 64 components of d = 256 use every SM.  By blocks of 32 rows: the rows of
// L are staged in shared memory, the terms of the rows above the block are a
// product over W's own column, 8 rows per warp, and one warp solves the block's
// triangle, each new entry at once taken off all later rows (32 independent
// chains; a running sum per row would wait for the FP64 latency at every term).
// Against one CTA per component for factor and inverse, with running sums (GB300):
// d = 256, K = 64 3438 -> 1317 + 757 us, d = 128, K = 64 877 -> 367 + 195,
// d = 119, K = 5 919 -> 328 + 187.
template <typename T>
__global__ void __launch_bounds__(kInvThreads)
k_factor_inverse(int K, int d, const double *__restrict__ work, double *linv, T *__restrict__ linvT,
                 double *__restrict__ fpart) {
  extern __shared__ double fsm[];                   // 32 rows of L from column c0 on
  __shared__ double s_acc[32][33], s_rd[32];
  const int j = blockIdx.x % K, b = blockIdx.x / K, tid = threadIdx.x, w = tid >> 5, lane = tid & 31;
  const int c0 = 32 * b, c = c0 + lane;
  const double *A = work + (size_t)j * d * d;
  double *Wi = linv + (size_t)j * d * d, *part = fpart + (size_t)j * kFactorParts;
  T *Wt = linvT + (size_t)j * d * d;
  if (part[kFactorParts - 1] < 0.0) return;
  for (int r = w; r < c0; r += kInvThreads / 32)
    if (c < d) {
      Wi[(size_t)r * d + c] = 0.0;
      Wt[(size_t)r * d + c] = T(0);
    }
  double fw = 0.0;
  for (int r0 = c0; r0 < d; r0 += 32) {
    const int rb = min(32, d - r0), mp = r0 - c0, mw = mp + rb;
    __syncthreads();                                // the previous block's rows are used up, its W is written
#pragma unroll 4
    for (int rr = w; rr < 32; rr += kInvThreads / 32)
      for (int m = lane; m < mw; m += 32) fsm[rr * mw + m] = rr < rb ? A[(size_t)(r0 + rr) * d + c0 + m] : 0.0;
    if (tid < rb) s_rd[tid] = 1.0 / A[(size_t)(r0 + tid) * d + r0 + tid];
    __syncthreads();
    double acc[8];
#pragma unroll
    for (int i = 0; i < 8; i++) acc[i] = 0.0;
    if (c < d) {
      const double *Lw = fsm + 8 * w * mw;
#pragma unroll 4
      for (int m = 0; m < mp; m++) {
        const double wm = Wi[(size_t)(c0 + m) * d + c];   // zero above the diagonal
#pragma unroll
        for (int i = 0; i < 8; i++) acc[i] = fma(-Lw[i * mw + m], wm, acc[i]);
      }
    }
#pragma unroll
    for (int i = 0; i < 8; i++) s_acc[8 * w + i][lane] = acc[i];
    __syncthreads();
    if (w == 0) {
      double s[32];
#pragma unroll
      for (int rr = 0; rr < 32; rr++) s[rr] = r0 + rr == c ? 1.0 : s_acc[rr][lane];
#pragma unroll
      for (int rr = 0; rr < 32; rr++) {
        if (rr >= rb) break;
        const double v = r0 + rr < c ? 0.0 : s[rr] * s_rd[rr];
#pragma unroll
        for (int q = rr + 1; q < 32; q++) s[q] = fma(-fsm[q * mw + mp + rr], v, s[q]);
        if (c < d) {
          Wi[(size_t)(r0 + rr) * d + c] = v;
          Wt[(size_t)(r0 + rr) * d + c] = (T)v;
          fw = fma(v, v, fw);
        }
      }
    }
  }
  if (w == 0) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) fw += __shfl_xor_sync(0xffffffffu, fw, o);
    if (lane == 0) part[b] = fw;
  }
}

__global__ void __launch_bounds__(256)
k_factor_bound(int K, int nb, const double *__restrict__ fpart, DevStatus *st) {
  for (int j = threadIdx.x; j < K; j += 256) {
    const double *part = fpart + (size_t)j * kFactorParts;
    if (part[kFactorParts - 1] < 0.0) continue;
    double s = 0.0;
    for (int b = 0; b < nb; b++) s += part[b];
    atomicMax(reinterpret_cast<unsigned long long *>(&st->cond_bound),
              (unsigned long long)__double_as_longlong(sqrt(part[kFactorParts - 1]) * s));
  }
}

// =========================================================== launchers
// P points per thread once there are two CTAs of that many per SM; below that
// one, which spreads the rows over more SMs.  With one point the rows are in
// registers up to D = 32 (20000 x 24 x 20: 37 us, in shared memory 39).
template <int D, int P, bool XS, int KC>
static int estep_f32(fem_em *h, int64_t *nb) {
  constexpr bool XS1 = XS && D > 32;
  const bool wide = P > 1 && h->n >= (int64_t)2 * sm_count() * kEPThreads * P;
  const int pw = wide ? P : 1, pts = kEPThreads * pw;
  const size_t sm = (2 * (size_t)EstepBuf<float, D, KC>::CB + ((wide ? XS : XS1) ? (size_t)D * (kEPThreads * pw + 1) : 0)) * sizeof(float);
  *nb = (h->n + pts - 1) / pts;
  auto launch = [&](auto kern) -> int {
    FEM_CUDA(allow_dyn_smem(kern, sm));
    kern<<<(unsigned)*nb, kEPThreads, sm, h->stream>>>(h->X, h->n, h->d, h->k, (const float *)h->muT, (const float *)h->linvT,
                                                       (const float *)h->logcT, (float *)h->R, h->logl_part);
    return FEM_OK;
  };
  return wide ? launch(k_estep_f32<D, P, XS, KC>) : launch(k_estep_f32<D, 1, XS1, KC>);
}

template <int D, int P, int KC>
static int estep_f64(fem_em *h, int64_t *nb) {
  const bool wide = P > 1 && h->n >= (int64_t)2 * sm_count() * kEPThreads * P;
  const int pts = kEPThreads * (wide ? P : 1);
  const size_t sm = 2 * (size_t)EstepBuf<double, D, KC>::CB * sizeof(double);
  *nb = (h->n + pts - 1) / pts;
  auto launch = [&](auto kern) -> int {
    FEM_CUDA(allow_dyn_smem(kern, sm));
    kern<<<(unsigned)*nb, kEPThreads, sm, h->stream>>>(h->X, h->n, h->d, h->k, (const double *)h->muT, (const double *)h->linvT,
                                                       (const double *)h->logcT, (double *)h->R, h->logl_part);
    return FEM_OK;
  };
  return wide ? launch(k_estep_f64<D, P, KC>) : launch(k_estep_f64<D, 1, KC>);
}

template <typename T>
static int estep_plain_t(fem_em *h) {
  const int64_t n = h->n;
  const int d = h->d, K = h->k;
  const T *mu = (const T *)h->muT, *W = (const T *)h->linvT, *lc = (const T *)h->logcT;
  T *R = (T *)h->R;
  int64_t nb = 0;
  int st = FEM_OK;
  bool done = true;
  // FP32 below 64 columns: the next D.  P, rows in registers or shared memory and
  // KC by measurement: D = 16 in registers P = 2, 3, 4: 609, 548, 619 us
  // (250007 x 16 x 200), in shared memory P = 4: 636; D = 32 in shared memory
  // P = 2, 3, 4: 554, 517, 633 (400000 x 32 x 40), one point in registers 808.
  // FP64 up to 16 and at 32 (60000 x 32 x 10: 833 us, generic form 873): from 17
  // on the generic form, which has no padding, is the faster one (60000 x 20 x 10:
  // 394 against 495 us padded to 24).
  if constexpr (sizeof(T) == 4) {
    if (d <= 4)
      st = estep_f32<4, 4, false, 16>(h, &nb);
    else if (d <= 8)
      st = estep_f32<8, 4, false, 8>(h, &nb);
    else if (d <= 12)
      st = estep_f32<12, 3, false, 4>(h, &nb);
    else if (d <= 16)
      st = estep_f32<16, 3, false, 4>(h, &nb);
    else if (d <= 20)
      st = estep_f32<20, 2, true, 2>(h, &nb);
    else if (d <= 24)
      st = estep_f32<24, 2, true, 2>(h, &nb);
    else if (d <= 28)
      st = estep_f32<28, 3, true, 2>(h, &nb);
    else if (d <= 32)
      st = estep_f32<32, 3, true, 2>(h, &nb);
    else if (d <= 40)
      st = estep_f32<40, 2, true, 2>(h, &nb);
    else if (d <= 48)
      st = estep_f32<48, 2, true, 2>(h, &nb);
    else if (d < 64)
      st = estep_f32<64, 2, true, 1>(h, &nb);
    else
      done = false;
  } else {
    if (d <= 4)
      st = estep_f64<4, 2, 8>(h, &nb);
    else if (d <= 6)
      st = estep_f64<6, 2, 8>(h, &nb);
    else if (d <= 8)
      st = estep_f64<8, 2, 8>(h, &nb);
    else if (d <= 10)
      st = estep_f64<10, 1, 8>(h, &nb);
    else if (d <= 12)
      st = estep_f64<12, 1, 8>(h, &nb);
    else if (d <= 14)
      st = estep_f64<14, 1, 8>(h, &nb);
    else if (d <= 16)
      st = estep_f64<16, 1, 8>(h, &nb);
    else if (d == 32)
      st = estep_f64<32, 1, 2>(h, &nb);
    else
      done = false;
  }
  FEM_TRY(st);
  if (!done) {
    constexpr int PT = sizeof(T) == 4 ? 4 : 2;   // 128 FP32 or 64 FP64 points per CTA
    const size_t smt = estep_tiled_smem<T, PT>(d);
    if (d > 64 && smt <= kMaxDynSmem) {
      nb = (n + 32 * PT - 1) / (32 * PT);
      FEM_CUDA(allow_dyn_smem(k_estep_plain_tiled<T, PT>, smt));
      k_estep_plain_tiled<T, PT><<<(unsigned)nb, 256, smt, h->stream>>>(h->X, n, d, K, mu, W, lc, R, h->logl_part);
    } else if (d == 64) {
      nb = (n + 127) / 128;
      k_estep_64<T><<<(unsigned)nb, 128, 0, h->stream>>>(h->X, n, K, mu, W, lc, R, h->logl_part);
    } else {
      nb = (n + 63) / 64;
      const size_t sm = (size_t)64 * (d + 1) * sizeof(T);
      FEM_CUDA(allow_dyn_smem(k_estep_plain_generic<T>, sm));
      k_estep_plain_generic<T><<<(unsigned)nb, 64, sm, h->stream>>>(h->X, n, d, K, mu, W, lc, R, h->logl_part);
    }
  }
  FEM_CUDA(cudaGetLastError());
  k_reduce_logl<<<1, 1024, 0, h->stream>>>(h->logl_part, nb, h->dstat);
  FEM_CUDA(cudaGetLastError());
  h->launches += 2;
  return FEM_OK;
}

int em_plain_estep(fem_em *h) {
  return h->cfg.precision == FEM_PREC_FP64 ? estep_plain_t<double>(h) : estep_plain_t<float>(h);
}

size_t em_factor_parts(int d, int k) { return d > kFactorSmemD ? (size_t)k * kFactorParts : 0; }

int64_t em_plain_logl_blocks(int64_t n, int d) { (void)d; return (n + 63) / 64; }

template <typename T>
static int mstep_plain_t(fem_em *h) {
  const int d = h->d, K = h->k;
  const int64_t n = h->n;
  // the form's limit: components times 4-, 8-, 16- or 32-column chunks
  const int C = d <= 4 ? 4 : (d <= 8 ? 8 : (d <= 16 ? 16 : 32));
  if (K * ((d + C - 1) / C) > 1024) {
    set_error("plain M-step: k*d too large (k=%d d=%d)", K, d);
    return FEM_ERR_UNSUPPORTED;
  }
  FEM_TRY(em_means_plain(h));
  k_final_means<T><<<K, 256, 0, h->stream>>>(h->mpart, h->means.chunks, K, d, n, h->mu, h->pi, h->psum,
                                             (T *)h->muT);
  FEM_CUDA(cudaGetLastError());
  FEM_TRY(em_cov_plain(h));
  h->launches += 4;
  return FEM_OK;
}

int em_plain_mstep(fem_em *h) {
  return h->cfg.precision == FEM_PREC_FP64 ? mstep_plain_t<double>(h) : mstep_plain_t<float>(h);
}

constexpr size_t kJacobiSmem = 96 * 1024;

// NormalDensity::ComputeConditionNumber (EM2/NormalDensity.cpp:67-71), one
// CTA per component on a symmetric copy of Sigma_j (block_jacobi_cond); the
// largest cond_j is folded into *out (non-negative doubles order like their bits).
__global__ void __launch_bounds__(256)
k_cond_jacobi(const double *__restrict__ sigma, int d, double *__restrict__ work, unsigned long long *out) {
  extern __shared__ double smem_jac[];
  const int j = blockIdx.x, tid = threadIdx.x, nt = blockDim.x;
  // the matrix lives in shared memory when it fits (d <= 110), else in `work`
  double *A = (size_t)d * d * sizeof(double) <= kJacobiSmem ? smem_jac : work + (size_t)j * d * d;
  const double *S = sigma + (size_t)j * d * d;
  for (int e = tid; e < d * d; e += nt) {
    const int r = e / d, c = e - r * d;
    A[e] = (c <= r) ? S[e] : S[(size_t)c * d + r];
  }
  __syncthreads();
  const double cond = block_jacobi_cond(A, d);
  if (tid == 0) atomicMax(out, (unsigned long long)__double_as_longlong(cond));
}

int em_max_cond(fem_em *h, double *cond) {
  if (h->d > 256) {
    set_error("condition check supports d <= 256 (got %d)", h->d);
    return FEM_ERR_UNSUPPORTED;
  }
  unsigned long long *dout = nullptr;
  FEM_TRY(dalloc(&dout, 1));
  FEM_CUDA(cudaMemsetAsync(dout, 0, sizeof(unsigned long long), h->stream));
  const size_t sm = (size_t)h->d * h->d * sizeof(double) <= kJacobiSmem ? (size_t)h->d * h->d * sizeof(double) : 0;
  FEM_CUDA(allow_dyn_smem(k_cond_jacobi, sm));
  k_cond_jacobi<<<h->k, 256, sm, h->stream>>>(h->sigma, h->d, h->work, dout);
  cudaError_t e = cudaGetLastError();
  unsigned long long bits = 0;
  if (e == cudaSuccess) e = cudaMemcpyAsync(&bits, dout, sizeof(bits), cudaMemcpyDeviceToHost, h->stream);
  if (e == cudaSuccess) e = cudaStreamSynchronize(h->stream);
  dfree(dout);
  if (e != cudaSuccess) {
    set_error("condition-number kernel failed: %s", cudaGetErrorString(e));
    return FEM_ERR_CUDA;
  }
  std::memcpy(cond, &bits, sizeof(double));
  h->launches += 1;
  return FEM_OK;
}

template <typename T>
static int factor_t(fem_em *h, bool regularize) {
  const int K = h->k, d = h->d;
  const size_t sm = factor_smem_bytes(d);
#define FEM_FK(KERNEL)                                                                                                \
  do {                                                                                                                \
    FEM_CUDA(allow_dyn_smem(KERNEL, sm));                                                                             \
    KERNEL<<<K, kFactorThreads, sm, h->stream>>>(K, d, h->cfg.reg_coef, regularize, h->sigma, h->pi, h->mu, h->work,  \
                                                 h->linv, h->logdet, h->logc, (T *)h->muT, (T *)h->linvT,             \
                                                 (T *)h->logcT, h->dstat);                                            \
  } while (0)
  if (d <= 32)
    FEM_FK((k_factor_smem<T, 1>));
  else if (d <= 64)
    FEM_FK((k_factor_smem<T, 2>));
  else if (d <= kFactorSmemD)
    FEM_FK((k_factor_smem<T, 4>));
  else {
    FEM_CUDA(allow_dyn_smem(k_factor<T>, sm));
    k_factor<T><<<K, kFactorThreads, sm, h->stream>>>(K, d, h->cfg.reg_coef, regularize, h->sigma, h->pi, h->mu, h->work,
                                                      h->fpart, h->logdet, h->logc, (T *)h->muT, (T *)h->logcT, h->dstat);
    FEM_CUDA(cudaGetLastError());
    const int nb = (d + 31) / 32;
    const size_t si = (size_t)32 * d * sizeof(double);
    FEM_CUDA(allow_dyn_smem(k_factor_inverse<T>, si));
    k_factor_inverse<T><<<K * nb, kInvThreads, si, h->stream>>>(K, d, h->work, h->linv, (T *)h->linvT, h->fpart);
    FEM_CUDA(cudaGetLastError());
    k_factor_bound<<<1, 256, 0, h->stream>>>(K, nb, h->fpart, h->dstat);
    h->launches += 2;
  }
#undef FEM_FK
  FEM_CUDA(cudaGetLastError());
  h->launches += 1;
  return FEM_OK;
}

int em_factor(fem_em *h, bool regularize) {
  return h->cfg.precision == FEM_PREC_FP64 ? factor_t<double>(h, regularize) : factor_t<float>(h, regularize);
}

// ------------------------------------------------ posteriors read-back
template <typename T>
__global__ void k_post_rows(const T *__restrict__ R, int64_t n, int K, int64_t r0, int64_t rows,
                            double *__restrict__ out) {
  const int64_t e = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (e >= rows * K) return;
  const int64_t i = e / K;
  const int j = (int)(e - i * K);
  out[e] = (double)R[(size_t)j * post_ld(n) + r0 + i];
}

// EMAlgorithm::RetrieveClasses: first index of the largest posterior
template <typename T>
__global__ void k_classes(const T *__restrict__ R, int64_t n, int K, int32_t *__restrict__ cls) {
  const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  double best = -1.0;
  int bj = -1;
  for (int j = 0; j < K; j++) {
    const double v = (double)R[(size_t)j * post_ld(n) + i];
    if (v > best) {
      best = v;
      bj = j;
    }
  }
  cls[i] = bj;
}

int em_post_rows(fem_em *h, int64_t r0, int64_t rows, double *dout) {
  const int64_t tot = rows * h->k;
  const unsigned nb = (unsigned)((tot + 255) / 256);
  if (h->cfg.precision == FEM_PREC_FP64)
    k_post_rows<double><<<nb, 256, 0, h->stream>>>((const double *)h->R, h->n, h->k, r0, rows, dout);
  else
    k_post_rows<float><<<nb, 256, 0, h->stream>>>((const float *)h->R, h->n, h->k, r0, rows, dout);
  FEM_CUDA(cudaGetLastError());
  return FEM_OK;
}

int em_classes(fem_em *h, int32_t *dcls) {
  const unsigned nb = (unsigned)((h->n + 255) / 256);
  if (h->cfg.precision == FEM_PREC_FP64)
    k_classes<double><<<nb, 256, 0, h->stream>>>((const double *)h->R, h->n, h->k, dcls);
  else
    k_classes<float><<<nb, 256, 0, h->stream>>>((const float *)h->R, h->n, h->k, dcls);
  FEM_CUDA(cudaGetLastError());
  return FEM_OK;
}

}  // namespace fem
