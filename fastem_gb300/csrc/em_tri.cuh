// em_tri.cuh -- ||W t||^2 for a lower-triangular W in shared memory and several
// points per thread, and the online log-sum-exp, shared by the single-fit and
// batched E-steps (MatrixEMBase::BlockDensities and PostProcessDensityMatrix,
// EM2/MatrixEM.cpp:39-51,69-81), and the addition of point groups' sums in the
// M-steps (EM2/MatrixEM.cpp:309-378).
#pragma once

#include <cmath>
#include <cstdint>

namespace fem {

// padded lower triangle: row kk holds kk + 1 entries in 4 * ceil((kk + 1) / 4)
__host__ __device__ constexpr int tri_row(int kk) { return 4 * ((kk + 4) / 4); }
__host__ __device__ constexpr int tri_off(int kk) {
  int s = 0;
  for (int r = 0; r < kk; r++) s += tri_row(r);
  return s;
}

// ---- FP32: two columns per instruction.  A packed operation takes the FMA pipe
// as long as two single ones but one issue slot, and the pair (even, odd column)
// is what a 16-byte load of a row delivers.
__device__ __forceinline__ uint64_t f2_sub(uint64_t a, uint64_t b) {
  uint64_t r;
  asm("sub.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
  return r;
}
__device__ __forceinline__ uint64_t f2_mul(uint64_t a, uint64_t b) {
  uint64_t r;
  asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
  return r;
}
__device__ __forceinline__ uint64_t f2_fma(uint64_t a, uint64_t b, uint64_t c) {
  uint64_t r;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
  return r;
}
__device__ __forceinline__ uint64_t f2_pack(float x, float y) {
  uint64_t r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(x), "f"(y));
  return r;
}
__device__ __forceinline__ void f2_unpack(uint64_t v, float &x, float &y) {
  asm("mov.b64 {%0, %1}, %2;" : "=f"(x), "=f"(y) : "l"(v));
}

// s_p += (row r of W . t_p)^2 for r = KK..D-1, t_p packed by column pairs, RB
// rows side by side (their chains are independent); rows by compile-time
// recursion so every column bound is a constant.  Nothing right of the diagonal
// is multiplied (a non-finite centred value stays out of the rows above its own).
template <int D, int P, int RB, int KK>
__device__ __forceinline__ void tri_rows(const uint64_t (&t)[P][D / 2], const float *__restrict__ w, float (&s)[P]) {
  uint64_t y[RB][P];
  float z[RB][P];
#pragma unroll
  for (int m4 = 0; m4 <= (KK + RB - 1) / 4; m4++) {
#pragma unroll
    for (int r = 0; r < RB; r++) {
      const int kk = KK + r;
      if (4 * m4 > kk) continue;
      const ulonglong2 v = *reinterpret_cast<const ulonglong2 *>(w + tri_off(kk) + 4 * m4);
#pragma unroll
      for (int h = 0; h < 2; h++) {
        const int c = 4 * m4 + 2 * h;
        const uint64_t we = h ? v.y : v.x;
        if (c + 1 <= kk) {
#pragma unroll
          for (int p = 0; p < P; p++) y[r][p] = c == 0 ? f2_mul(t[p][0], we) : f2_fma(t[p][c / 2], we, y[r][p]);
          if (c + 1 == kk) {
#pragma unroll
            for (int p = 0; p < P; p++) {
              float lo, hi;
              f2_unpack(y[r][p], lo, hi);
              z[r][p] = lo + hi;
            }
          }
        } else if (c == kk) {
          float w0, w1;
          f2_unpack(we, w0, w1);
#pragma unroll
          for (int p = 0; p < P; p++) {
            float t0, t1, lo = 0.f, hi = 0.f;
            f2_unpack(t[p][c / 2], t0, t1);
            if (c) f2_unpack(y[r][p], lo, hi);
            z[r][p] = c ? fmaf(t0, w0, lo) + hi : t0 * w0;
          }
        }
      }
    }
  }
#pragma unroll
  for (int r = 0; r < RB; r++)
#pragma unroll
    for (int p = 0; p < P; p++) s[p] = KK + r ? fmaf(z[r][p], z[r][p], s[p]) : z[r][p] * z[r][p];
  if constexpr (KK + RB < D) tri_rows<D, P, RB, KK + RB>(t, w, s);
}

// s_p = ||W t_p||^2
template <int D, int P>
__device__ __forceinline__ void tri_norms(const uint64_t (&t)[P][D / 2], const float *__restrict__ w, float (&s)[P]) {
  tri_rows<D, P, 2, 0>(t, w, s);
}

// ---- FP64
template <int D, int P>
__device__ __forceinline__ void tri_norms(const double (&t)[P][D], const double *__restrict__ w, double (&s)[P]) {
#pragma unroll
  for (int p = 0; p < P; p++) s[p] = 0.0;
#pragma unroll
  for (int kk = 0; kk < D; kk++) {
    double y[P];
#pragma unroll
    for (int p = 0; p < P; p++) y[p] = 0.0;
#pragma unroll
    for (int m = 0; m <= kk; m += 2) {
      const double2 v = *reinterpret_cast<const double2 *>(w + tri_off(kk) + m);
#pragma unroll
      for (int p = 0; p < P; p++) {
        y[p] = fma(t[p][m], v.x, y[p]);
        if (m + 1 <= kk) y[p] = fma(t[p][m + 1], v.y, y[p]);
      }
    }
#pragma unroll
    for (int p = 0; p < P; p++) s[p] = fma(y[p], y[p], s[p]);
  }
}

// Online log-sum-exp without a branch: one exponential whichever of l and the
// maximum is larger.  l = -infinity and NaN leave the sum as it is.
__device__ __forceinline__ void lse_add(float l, float &mx, float &se) {
  const float e = expf(fminf(l, mx) - fmaxf(l, mx));
  const float a = l > mx ? fmaf(se, e, 1.f) : se + e;
  se = l > -INFINITY ? a : se;
  mx = fmaxf(l, mx);
}

// sum of n FP32 values `stride` apart, in order, to FP64: the rounding errors of
// the FP32 additions are carried along exactly (two-sum), so three FP64
// operations suffice instead of 2 n, which the FP64 pipe's rate would make a
// tenth of a covariance item's time
__device__ __forceinline__ double group_sum(const float *v, int n, int stride) {
  float hi = v[0], lo = 0.f;
  for (int g = 1; g < n; g++) {
    const float x = v[g * stride], t = __fadd_rn(hi, x), b = __fsub_rn(t, hi);
    lo = __fadd_rn(lo, __fadd_rn(__fsub_rn(hi, __fsub_rn(t, b)), __fsub_rn(x, b)));
    hi = t;
  }
  // an infinite sum has no error term (inf - inf above)
  return isfinite(hi) ? (double)hi + (double)lo : (double)hi;
}
__device__ __forceinline__ double group_sum(const double *v, int n, int stride) {
  double s = v[0];
  for (int g = 1; g < n; g++) s += v[g * stride];
  return s;
}

}  // namespace fem
