// em_factor.cuh -- block-wide FP64 steps on one d x d covariance matrix,
// shared by the single-fit kernels (em_plain.cu) and the batched engine
// (em_batch.cu).  Every thread of the block calls each function; matrices are
// row-major d x d in global or shared memory.
#pragma once

#include <cmath>

namespace fem {

// EMAlgorithm::RegularizeCovariances (EM2/EMAlgorithm.cpp:237-244):
// S <- (1 - reg) S + (reg tr(S) / d) I, in place.
__device__ inline void block_regularize(double *S, int d, double reg) {
  __shared__ double s_add;
  if (threadIdx.x == 0) {
    double tr = 0.0;
    for (int q = 0; q < d; q++) tr += S[(size_t)q * d + q];
    s_add = reg * tr / (double)d;
  }
  __syncthreads();
  const double add = s_add;
  for (int e = threadIdx.x; e < d * d; e += blockDim.x) {
    const int r = e / d, c = e - r * d;
    S[e] = S[e] * (1.0 - reg) + (r == c ? add : 0.0);
  }
  __syncthreads();
}

constexpr int kFactorMaxD = 256;   // largest d of the block factorisation helpers
constexpr int kFactorThreads = 256;

// N sums over the block in a fixed order; the values in every thread.  red:
// N doubles per warp
template <int N>
__device__ inline void block_sums(double (&v)[N], double *red) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1)
#pragma unroll
    for (int q = 0; q < N; q++) v[q] += __shfl_xor_sync(0xffffffffu, v[q], o);
  __syncthreads();
  if ((threadIdx.x & 31) == 0)
#pragma unroll
    for (int q = 0; q < N; q++) red[(threadIdx.x >> 5) * N + q] = v[q];
  __syncthreads();
#pragma unroll
  for (int q = 0; q < N; q++) {
    v[q] = red[q];
    for (int w = 1; w < (int)blockDim.x / 32; w++) v[q] += red[w * N + q];
  }
}

// u / p for N values of u: the hardware's approximate reciprocal y (relative
// error below 2^-20) and a third-order correction, u y (1 + e + e^2) with
// e = 1 - p y (Schulz / Householder iteration): three dependent FP64
// operations to within 2^-60 before rounding
template <int N>
__device__ __forceinline__ void factor_divide(double (&u)[N], double p) {
  const int ex = (__double2hiint(p) >> 20) & 0x7ff;
  if (ex < 64 || ex > 1983) {                    // the approximation flushes subnormal results
#pragma unroll
    for (int s = 0; s < N; s++) u[s] = u[s] / p;
    return;
  }
  double y;
  asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(p));
  const double e = fma(-p, y, 1.0), e2 = fma(e, e, e);
#pragma unroll
  for (int s = 0; s < N; s++) {
    const double t = u[s] * y;
    u[s] = fma(t, e2, t);
  }
}

// NormalDensity::Init (EM2/NormalDensity.cpp:43-65) with both matrices in
// shared memory, as L D L^T: A (row stride ld, lower triangle = the
// covariance) ends as L sqrt(D) columns before their scaling, W as the rows of
// the unit inverse, piv[k] = D_k and rd[k] = 1 / sqrt(D_k), so that
//   L_rc = A[r][c] rd[c] (r > c), L_rr = sqrt(piv[r]),
//   (L^-1)_rc = W[r][c] rd[r] (r > c), (L^-1)_rr = rd[r]
// (the upper triangles and the diagonal of W are not written).  A pivot <= 0
// fails, as Eigen's LLT reports (the pivots are the same); the answer is the
// same in every thread.  m: 2 d doubles of scratch.  d <= 32 NS.
//
// FP64 runs at 2 lanes per clock and SM with a long latency, so the form is
// chosen for its chain: per column one barrier, and between two barriers warp
// 0 (lane = row) forms column k + 1, the reciprocal of its pivot and its
// multipliers, 6 dependent operations where a Cholesky column's square root
// and divisions are ~25; the square roots wait for the end.  Meanwhile the
// other warps (warp = row, lane = column) apply column k: row i takes the
// inverse's columns 0..k and the factor's k + 2..i in one pass.
// Against one thread per column over matrices in L2 (GB300, the whole kernel):
// d = 24, K = 21 73 -> 21 us; d = 64, K = 128 263 -> 95 us; d = 99, K = 23
// 593 -> 284 us.  From d = 48 on the updates' shared-memory round trips and the
// FP64 pipe set the time; batching 2 or 4 rows per warp to overlap them was
// slower (d = 99: 335, 369 us: warp 0's chain waits behind the bursts).
template <int NS>
__device__ inline bool block_factor_smem(double *A, double *W, double *piv, double *rd, double *m, int d, int ld) {
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, nu = (blockDim.x >> 5) - 1;
  // by column parity: warp 0 may be in the next column, and set its flag, before
  // the slowest warp has read this one's behind the column's only barrier
  __shared__ int s_fail[2];
  if (threadIdx.x < 2) s_fail[threadIdx.x] = 0;
  __syncthreads();
  bool ok = true;
  for (int k = -1; k < d - 1; k++) {
    const double *mk = m + (k & 1) * d;
    if (warp == 0) {
      const int c = k + 1;
      double u[NS];
      const double uc = k >= 0 ? -A[c * ld + k] : 0.0;
#pragma unroll
      for (int s = 0; s < NS; s++) {
        const int r = c + lane + 32 * s;
        u[s] = 0.0;
        if (r < d) u[s] = k >= 0 ? fma(mk[r], uc, A[r * ld + c]) : A[r * ld + c];
      }
      const double p = __shfl_sync(0xffffffffu, u[0], 0);
      const long long pb = __double_as_longlong(p);
      if (pb <= 0 || pb > 0x7ff0000000000000LL) {    // !(p > 0), without waiting for the FP64 pipe
        if (lane == 0) s_fail[k & 1] = 1;
      } else {
        double *mc = m + (c & 1) * d;
#pragma unroll
        for (int s = 0; s < NS; s++) {
          const int r = c + lane + 32 * s;
          if (r < d) A[r * ld + c] = u[s];
        }
        factor_divide(u, p);
#pragma unroll
        for (int s = 0; s < NS; s++) {
          const int r = c + lane + 32 * s;
          if (r < d) mc[r] = u[s];
        }
        if (lane == 0) piv[c] = p;
      }
    } else if (k >= 0) {
      double v[NS];
      double *col[NS];                    // column c of the inverse's or the factor's rows
#pragma unroll
      for (int s = 0; s < NS; s++) {
        const int c = lane + 32 * s;
        v[s] = c < k ? W[k * ld + c] : (c > k + 1 && c < d ? A[c * ld + k] : 0.0);
        col[s] = (c <= k ? W : A) + c;
      }
      for (int i = k + warp; i < d; i += nu) {
        const double mi = -mk[i];
#pragma unroll
        for (int s = 0; s < NS; s++) {
          const int c = lane + 32 * s;
          if (c > i || c == k + 1) continue;
          double *t = col[s] + i * ld;
          *t = c == k ? mi : fma(mi, v[s], *t);
        }
      }
    }
    __syncthreads();
    if (s_fail[k & 1]) {
      ok = false;
      break;
    }
  }
  if (ok)
    for (int q = threadIdx.x; q < d; q += blockDim.x) rd[q] = 1.0 / sqrt(piv[q]);
  __syncthreads();
  return ok;
}

// ------------------------------------------------------------------------
// Blocked Cholesky for one CTA of kFactorThreads threads (kFactorSmemD < d <=
// kFactorMaxD).  The matrix stays in global memory (L2); the panel being
// factored sits in shared memory, the trailing updates are 4 x 4 register
// tiles, and the FP64 pipe is the limit (d^3 / 6 fused multiply-adds).
constexpr int kPanel = 32;                // columns per Cholesky panel
constexpr int kPanelLd = kPanel + 1;      // panel row stride (doubles)
// block_factor_smem holds both matrices in shared memory up to this d
constexpr int kFactorSmemD = 118;
__host__ __device__ constexpr int factor_ld(int d) { return d | 1; }

// dynamic shared memory: both matrices and block_factor_smem's vectors up to
// kFactorSmemD, else the panel
__host__ __device__ constexpr size_t factor_smem_bytes(int d) {
  return (d <= kFactorSmemD ? (size_t)2 * d * factor_ld(d) + 4 * d : (size_t)d * kPanelLd) * sizeof(double);
}

// Right-looking Cholesky of sym(lower(S)) by panels of kPanel columns, the
// trailing lower triangle updated as 4 x 4 tiles.  The upper triangle of A keeps
// the symmetric copy of S.  In a panel (rows k0 .. d-1) thread i holds row
// k0 + i in registers, and the panel's own triangle is warp 0, lane = row: per
// column the warp divides the column by its pivot (L D L^T; the square roots
// wait for the end of the panel) and one barrier later every row takes the
// column off.  With the panel in shared memory, a square root and a division per
// column and two barriers, the kernel took 1391 us at d = 256 and 350 at d = 119,
// here 1317 and 330; the trailing updates, at the FP64 pipe's rate, are the rest.
// P: factor_smem_bytes(d) of shared memory.  Returns true on success, the
// same in every thread.
__device__ inline bool block_cholesky_panels(const double *S, int d, double *A, double *P) {
  __shared__ double s_m[2][kPanel], s_piv[kPanel], s_rd[kPanel];
  const int tid = threadIdx.x, nt = blockDim.x;
  for (int e = tid; e < d * d; e += nt) {
    const int r = e / d, c = e - r * d;
    A[e] = (c <= r) ? S[e] : S[(size_t)c * d + r];
  }
  __syncthreads();
  for (int k0 = 0; k0 < d; k0 += kPanel) {
    const int w = min(kPanel, d - k0), m = d - k0;
    for (int e = tid; e < m * w; e += nt) {
      const int i = e / w, q = e - i * w;
      P[i * kPanelLd + q] = A[(size_t)(k0 + i) * d + k0 + q];
    }
    __syncthreads();
    const int i = tid;                    // panel row owned by this thread
    double x[kPanel];
#pragma unroll
    for (int q = 0; q < kPanel; q++) x[q] = i < m && q < w ? P[i * kPanelLd + q] : 0.0;
#pragma unroll
    for (int q = 0; q < kPanel; q++) {
      if (q >= w) break;
      int bad = 0;
      if (tid < 32) {
        const double p = __shfl_sync(0xffffffffu, x[q], q);
        if (!(p > 0.0)) {
          bad = 1;
        } else {
          double u[1] = {x[q]};
          factor_divide(u, p);
          s_m[q & 1][tid] = u[0];
          if (tid == q) s_piv[q] = p;
        }
      }
      if (__syncthreads_or(bad)) return false;     // the same in every thread
      // the entries right of a row's own diagonal are never used
#pragma unroll
      for (int c = q + 1; c < kPanel; c++) x[c] = fma(-x[q], s_m[q & 1][c], x[c]);
    }
    if (tid < w) s_rd[tid] = 1.0 / sqrt(s_piv[tid]);
    __syncthreads();
    if (i < m) {
#pragma unroll
      for (int q = 0; q < kPanel; q++)
        if (q < w) P[i * kPanelLd + q] = i == q ? sqrt(s_piv[q]) : x[q] * s_rd[q];
    }
    __syncthreads();
    for (int e = tid; e < m * w; e += nt) {
      const int r = e / w, q = e - r * w;
      if (q <= r) A[(size_t)(k0 + r) * d + k0 + q] = P[r * kPanelLd + q];
    }
    // trailing update: A[r][c] -= sum_q L[r][q] L[c][q], w <= c <= r < m
    // (panel-relative), over 4 x 4 tiles of the lower triangle
    const int n2 = m - w;
    if (n2 > 0) {
      const int T = (n2 + 3) >> 2;
      const int ntile = T * (T + 1) / 2;
      for (int t = tid; t < ntile; t += nt) {
        int ti = (int)((sqrt(8.0 * (double)t + 1.0) - 1.0) * 0.5);
        while ((ti + 1) * (ti + 2) / 2 <= t) ti++;
        while (ti * (ti + 1) / 2 > t) ti--;
        const int tc = t - ti * (ti + 1) / 2;
        const int rb = w + 4 * ti, cb = w + 4 * tc;
        double acc[4][4];
#pragma unroll
        for (int u = 0; u < 4; u++)
#pragma unroll
          for (int v = 0; v < 4; v++) {
            const int r = rb + u, c = cb + v;
            acc[u][v] = (r < m && c <= r) ? A[(size_t)(k0 + r) * d + k0 + c] : 0.0;
          }
        for (int q = 0; q < w; q++) {
          double a[4], b[4];
#pragma unroll
          for (int u = 0; u < 4; u++) {
            a[u] = (rb + u < m) ? P[(rb + u) * kPanelLd + q] : 0.0;
            b[u] = (cb + u < m) ? P[(cb + u) * kPanelLd + q] : 0.0;
          }
#pragma unroll
          for (int u = 0; u < 4; u++)
#pragma unroll
            for (int v = 0; v < 4; v++) acc[u][v] = fma(-a[u], b[v], acc[u][v]);
        }
#pragma unroll
        for (int u = 0; u < 4; u++)
#pragma unroll
          for (int v = 0; v < 4; v++) {
            const int r = rb + u, c = cb + v;
            if (r < m && c <= r) A[(size_t)(k0 + r) * d + k0 + c] = acc[u][v];
          }
      }
    }
    __syncthreads();
  }
  return true;
}

// log det = 2 sum log L_ii (L in the lower triangle of A): the logarithms in
// parallel, summed in index order by one thread; the value in every thread.
// d <= kFactorMaxD.
__device__ inline double block_chol_logdet(const double *A, int d) {
  __shared__ double s_log[kFactorMaxD];
  __shared__ double s_ld;
  for (int q = threadIdx.x; q < d; q += blockDim.x) s_log[q] = log(A[(size_t)q * d + q]);
  __syncthreads();
  if (threadIdx.x == 0) {
    double ld = 0.0;
    for (int q = 0; q < d; q++) ld += s_log[q];
    s_ld = 2.0 * ld;
  }
  __syncthreads();
  const double v = s_ld;
  __syncthreads();
  return v;
}

// ||sym(lower(S))||_F^2, in every thread.  red: a double per warp.
__device__ inline double block_frob2(const double *S, int d, double *red) {
  double v[1] = {0.0};
  for (int e = threadIdx.x; e < d * d; e += blockDim.x) {
    const int r = e / d, c = e - r * d;
    if (c <= r) v[0] = fma(c == r ? S[e] : 2.0 * S[e], S[e], v[0]);
  }
  block_sums(v, red);
  return v[0];
}

// NormalDensity::ComputeConditionNumber (EM2/NormalDensity.cpp:67-71): the
// eigenvalues of the symmetric matrix in A (overwritten) by cyclic Jacobi in
// FP64.  Each sweep runs the n - 1 rounds of a round-robin schedule; a round
// rotates n / 2 disjoint (p, q) pairs at once (columns, then rows).  Sweeps
// stop when the off-diagonal mass is below 1e-30 of the diagonal's, or after
// 100.  Returns |max eig / min eig| in every thread.  blockDim.x <= 256,
// d <= 256.
__device__ inline double block_jacobi_cond(double *A, int d) {
  const int tid = threadIdx.x, nt = blockDim.x;
  const int n = d + (d & 1);          // players of the round robin (a dummy when d is odd)
  const int np = n / 2;
  __shared__ double sc[128], ss[128];
  __shared__ int sp[128], sq[128];
  __shared__ double red_off[256], red_diag[256];
  __shared__ int done;
  __shared__ double s_cond;
  for (int sweep = 0; sweep < 100; sweep++) {
    double off = 0.0, dg = 0.0;
    for (int e = tid; e < d * d; e += nt) {
      const int r = e / d, c = e - r * d;
      const double v = A[e];
      if (c > r) off += v * v;
      else if (c == r) dg += v * v;
    }
    red_off[tid] = off;
    red_diag[tid] = dg;
    __syncthreads();
    if (tid == 0) {
      double o = 0.0, g = 0.0;
      for (int t = 0; t < nt; t++) o += red_off[t], g += red_diag[t];
      done = !(o > 1e-30 * g);
    }
    __syncthreads();
    if (done) break;
    for (int round = 0; round < n - 1; round++) {
      for (int i = tid; i < np; i += nt) {
        // position m holds player 0 (m = 0) or 1 + (m - 1 + round) mod (n - 1)
        const int m1 = i, m2 = n - 1 - i;
        const int p0 = m1 == 0 ? 0 : 1 + (m1 - 1 + round) % (n - 1);
        const int q0 = 1 + (m2 - 1 + round) % (n - 1);
        const int p = min(p0, q0), q = max(p0, q0);
        double c = 1.0, s = 0.0;
        if (q < d) {
          const double apq = A[(size_t)p * d + q];
          if (apq != 0.0) {
            const double app = A[(size_t)p * d + p], aqq = A[(size_t)q * d + q];
            const double th = (aqq - app) / (2.0 * apq);
            const double t = (th >= 0 ? 1.0 : -1.0) / (fabs(th) + sqrt(th * th + 1.0));
            c = 1.0 / sqrt(t * t + 1.0);
            s = t * c;
          }
        }
        sc[i] = c, ss[i] = s, sp[i] = p, sq[i] = q;
      }
      __syncthreads();
      for (int e = tid; e < d * np; e += nt) {     // columns p, q of every row
        const int i = e / d, r = e - i * d;
        const int p = sp[i], q = sq[i];
        if (q < d && ss[i] != 0.0) {
          const double arp = A[(size_t)r * d + p], arq = A[(size_t)r * d + q];
          A[(size_t)r * d + p] = sc[i] * arp - ss[i] * arq;
          A[(size_t)r * d + q] = ss[i] * arp + sc[i] * arq;
        }
      }
      __syncthreads();
      for (int e = tid; e < d * np; e += nt) {     // rows p, q of every column
        const int i = e / d, r = e - i * d;
        const int p = sp[i], q = sq[i];
        if (q < d && ss[i] != 0.0) {
          const double apr = A[(size_t)p * d + r], aqr = A[(size_t)q * d + r];
          A[(size_t)p * d + r] = sc[i] * apr - ss[i] * aqr;
          A[(size_t)q * d + r] = ss[i] * apr + sc[i] * aqr;
        }
      }
      __syncthreads();
    }
  }
  if (tid == 0) {
    double mn = A[0], mx = A[0];
    for (int p = 1; p < d; p++) {
      mn = fmin(mn, A[(size_t)p * d + p]);
      mx = fmax(mx, A[(size_t)p * d + p]);
    }
    s_cond = fabs(mx / mn);
  }
  __syncthreads();
  const double cond = s_cond;
  __syncthreads();
  return cond;
}

}  // namespace fem
