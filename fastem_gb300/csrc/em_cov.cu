// em_cov.cu -- the CUDA-core covariance sums of the EM sweep (FP32, FP64, and
// FP32 from the mixed path's FP16 hi/lo posteriors).
//
// MatrixEMBase::ComputeWeightedTempDataset + BlockCovariances
// (EM2/MatrixEM.cpp:53-67,90-99): CovSum_j += r_ij (x_i - mu_j)(x_i - mu_j)^T
// over the upper triangle, then Covs_j = CovSum_j / PosteriorSum_j
// (EM2/MatrixEM.cpp:363-375).
//
// A thread owns one TB x TB block of one component (a "unit") and keeps its
// sums in registers while the CTA's rows stream past; x - mu and r (x - mu)
// are formed in registers from the staged rows, so nothing per component is
// written to shared memory and a tile costs one barrier.  Bound by the
// FP32 pipe: 64 of the 88 FP32 operations per point and unit are the products
// (16 subtractions and 8 multiplications by r beside them) and, at 77 % of its
// rate, by the 128-bit shared-memory loads; in FP64 by the FP64 pipe (2 per
// clock and SM).  On the GB300, against a kernel that wrote sqrt(r) (x - mu)
// of every component to shared memory and used one thread per block:
//   N = 2^20, d = 64, K = 128, FP32 from FP16 hi/lo   82.9 -> 20.7 ms
//   N = 250007, d = 16, K = 200, FP32                  8.20 -> 0.89 ms
//   N = 200003, d = 24, K = 21, FP32 from FP16 hi/lo   0.75 -> 0.14 ms
//   N = 100000, d = 8, K = 10, FP64                    1.52 -> 0.14 ms
#include <algorithm>
#include <cmath>

#include "em_kernels.cuh"
#include "fem_internal.cuh"

namespace fem {

namespace {

constexpr int kCvThreads = 256;
constexpr int kCvRows = 2048;              // rows an FP32 sum may span before it is added into FP64
constexpr int kCvMaxGroups = 64;
constexpr size_t kCvMaxSmem = 232448;

__device__ __forceinline__ void cv_copy4(void *dst, const void *src, bool valid) {
  const uint32_t da = static_cast<uint32_t>(__cvta_generic_to_shared(dst));
  asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;\n" ::"r"(da), "l"(src), "r"(valid ? 4 : 0) : "memory");
}
__device__ __forceinline__ void cv_copy8(void *dst, const void *src, bool valid) {
  const uint32_t da = static_cast<uint32_t>(__cvta_generic_to_shared(dst));
  asm volatile("cp.async.ca.shared.global [%0], [%1], 8, %2;\n" ::"r"(da), "l"(src), "r"(valid ? 8 : 0) : "memory");
}
__device__ __forceinline__ void cv_copy16(void *dst, const void *src, bool valid) {
  const uint32_t da = static_cast<uint32_t>(__cvta_generic_to_shared(dst));
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;\n" ::"r"(da), "l"(src), "r"(valid ? 16 : 0) : "memory");
}

// ------------------------------------------------------- posterior sources
// A source stages rows t0 .. t0 + TP - 1 of cj components into shared memory
// (rows past `end` as zero) and reads one of them back.  `pitch` is the
// number of elements between two components there.

// component-major array of T, rows n apart (any alignment)
template <typename T>
struct PostTyped {
  const T *R;
  int64_t ld;
  static constexpr size_t kBytes = sizeof(T);
  __device__ void stage(unsigned char *buf, int pitch, int j0, int cj, int64_t t0, int TP, int64_t end) const {
    T *s = reinterpret_cast<T *>(buf);
    for (int e = threadIdx.x; e < cj * TP; e += kCvThreads) {
      const int j = e / TP, p = e - j * TP;
      const bool v = t0 + p < end;
      const T *src = R + (size_t)(j0 + j) * ld + (v ? t0 + p : 0);
      if (sizeof(T) == 4)
        cv_copy4(s + j * pitch + p, src, v);
      else
        cv_copy8(s + j * pitch + p, src, v);
    }
  }
  __device__ __forceinline__ T get(const unsigned char *buf, int o, int) const {
    return reinterpret_cast<const T *>(buf)[o];
  }
};

// the mixed path's FP16 hi + lo arrays: rows on 128-byte boundaries and
// padded to 64 points, so 8 points are copied at a time (TP and t0 are
// multiples of 8); lo follows hi in the stage, cj pitch elements behind
struct PostHiLo {
  const __half *Rh, *Rl;
  int64_t ld;
  static constexpr size_t kBytes = 2 * sizeof(__half);
  __device__ void stage(unsigned char *buf, int pitch, int j0, int cj, int64_t t0, int TP, int64_t end) const {
    __half *s = reinterpret_cast<__half *>(buf);
    const int c8 = TP / 8;
    for (int e = threadIdx.x; e < 2 * cj * c8; e += kCvThreads) {
      const int half = e / (cj * c8), r = e - half * cj * c8, j = r / c8, p = 8 * (r - j * c8);
      // the last copy may bring posteriors of the padding behind row n, which are not summed
      const bool v = t0 + p < end;
      const __half *src = (half ? Rl : Rh) + (size_t)(j0 + j) * ld + (v ? t0 + p : 0);
      cv_copy16(s + (half * cj + j) * pitch + p, src, v);
    }
  }
  __device__ __forceinline__ float get(const unsigned char *buf, int o, int lo) const {
    const __half *s = reinterpret_cast<const __half *>(buf);
    return __half2float(s[o]) + __half2float(s[o + lo]);
  }
};

// position of dimension q inside a staged row: 4-float groups of the TB = 8
// blocks are split into even and odd halves, so lanes that read consecutive
// blocks' first (or second) groups read consecutive 16-byte words
template <int TB>
__device__ __forceinline__ int cv_pos(int q, int nb) {
  if (TB == 4) return q;
  return ((q >> 2) & 1) * (4 * nb) + (q >> 3) * 4 + (q & 3);
}

template <int TB>
__device__ __forceinline__ void cv_load(const float *row, int b, int nb, float (&v)[TB]) {
  const float4 a = *reinterpret_cast<const float4 *>(row + 4 * b);
  v[0] = a.x, v[1] = a.y, v[2] = a.z, v[3] = a.w;
  if constexpr (TB == 8) {
    const float4 c = *reinterpret_cast<const float4 *>(row + 4 * nb + 4 * b);
    v[4] = c.x, v[5] = c.y, v[6] = c.z, v[7] = c.w;
  }
}

constexpr int cv_ne(int TB, bool TRI) { return TRI ? TB * (TB + 1) / 2 : TB * TB; }

// The (component, upper block) units u0 = blockIdx.x upc .. + upc - 1, rows of
// chunk blockIdx.y.  Thread t owns unit u0 + t % upc for the points p = t /
// upc, t / upc + G, ... of every tile (G = groups), so fits with few units
// still use every thread.  TRI: one block covers all dimensions (d <= TB) and
// only its upper triangle is summed.  part[chunk][element][unit], FP64.
template <typename T, int TB, bool TRI, class Src>
__global__ void __launch_bounds__(kCvThreads, sizeof(T) == 4 ? 2 : 1)
k_cov_units(const float *__restrict__ X, int64_t n, int d, int K, Src R, const T *__restrict__ mu, int mu_ld,
            double *__restrict__ part, int nb, int nblk, int64_t rows_per_chunk, int upc, int G, int TP, int xpitch,
            int rpitch, int cjmax) {
  constexpr int NE = cv_ne(TB, TRI);
  extern __shared__ __align__(16) unsigned char cv_smem[];
  const int tid = threadIdx.x;
  const int units = K * nblk;
  const int u0 = blockIdx.x * upc;
  const int j_lo = u0 / nblk, cj = min(K - 1, (u0 + upc - 1) / nblk) - j_lo + 1;
  const int g = tid / upc, ul = tid - g * upc, unit = u0 + ul;
  const bool act = g < G && unit < units;
  const size_t xbytes = (size_t)TP * xpitch * sizeof(float);
  const size_t rbytes = ((size_t)cjmax * rpitch * Src::kBytes + 15) & ~(size_t)15;
  const size_t buf_bytes = xbytes + rbytes;
  int j = j_lo, bi = 0, bj = 0;
  if (act) {
    j = unit / nblk;
    int b = unit - j * nblk;
    // upper-triangular enumeration of nb x nb blocks: row bi has nb - bi blocks
    while (b >= nb - bi) {
      b -= nb - bi;
      bi++;
    }
    bj = bi + b;
  }
  T ma[TB], mb[TB];
#pragma unroll
  for (int a = 0; a < TB; a++) {
    const int qa = bi * TB + a, qb = bj * TB + a;
    ma[a] = act && qa < d ? mu[(size_t)j * mu_ld + qa] : T(0);
    mb[a] = act && qb < d ? mu[(size_t)j * mu_ld + qb] : T(0);
  }
  T acc[NE];
#pragma unroll
  for (int e = 0; e < NE; e++) acc[e] = T(0);

  const int64_t c0 = (int64_t)blockIdx.y * rows_per_chunk, c1 = min(n, c0 + rows_per_chunk);
  // dimensions d .. nb TB - 1 of every staged row stay zero
  const int dp = nb * TB;
  if (d < dp)
    for (int e = tid; e < 2 * TP * (dp - d); e += kCvThreads) {
      const int row = e / (dp - d), q = d + e - row * (dp - d);
      float *sx = reinterpret_cast<float *>(cv_smem + (row >= TP ? buf_bytes : 0));
      sx[(row >= TP ? row - TP : row) * xpitch + cv_pos<TB>(q, nb)] = 0.f;
    }
  auto stage = [&](int buf, int64_t t0) {
    float *sx = reinterpret_cast<float *>(cv_smem + buf * buf_bytes);
    if ((d & 3) == 0) {
      const int d4 = d >> 2;
      for (int e = tid; e < TP * d4; e += kCvThreads) {
        const int p = e / d4, q = 4 * (e - p * d4);
        const bool v = t0 + p < c1;
        cv_copy16(sx + p * xpitch + cv_pos<TB>(q, nb), X + (v ? (t0 + p) * d + q : 0), v);
      }
    } else {
      for (int e = tid; e < TP * d; e += kCvThreads) {
        const int p = e / d, q = e - p * d;
        const bool v = t0 + p < c1;
        cv_copy4(sx + p * xpitch + cv_pos<TB>(q, nb), X + (v ? (t0 + p) * d + q : 0), v);
      }
    }
    R.stage(cv_smem + buf * buf_bytes + xbytes, rpitch, j_lo, cj, t0, TP, c1);
    asm volatile("cp.async.commit_group;\n" ::: "memory");
  };

  bool first = true;
  // adds the FP32 sums into this CTA's FP64 partials (or stores them); the
  // groups' sums of a unit are added in T first, in group order
  auto flush = [&](bool more) {
    double *o = part + (size_t)blockIdx.y * NE * units + u0;
    if (G == 1) {
      if (act) {
        o += ul;
        if (first) {
#pragma unroll
          for (int e = 0; e < NE; e++, o += units) *o = (double)acc[e];
        } else {
#pragma unroll
          for (int e = 0; e < NE; e++, o += units) *o += (double)acc[e];
        }
      }
    } else {
      T *red = reinterpret_cast<T *>(cv_smem);   // NE x 256, over the tiles
      asm volatile("cp.async.wait_group 0;\n" ::: "memory");
      __syncthreads();
#pragma unroll
      for (int e = 0; e < NE; e++) red[e * kCvThreads + tid] = acc[e];
      __syncthreads();
      const int live = min(upc, units - u0);
      for (int i = tid; i < live * NE; i += kCvThreads) {
        const int e = i / live, u = i - e * live;
        T s = red[e * kCvThreads + u];
        for (int q = 1; q < G; q++) s += red[e * kCvThreads + q * upc + u];
        double *p = o + (size_t)e * units + u;
        *p = first ? (double)s : *p + (double)s;
      }
      __syncthreads();
    }
    first = false;
    if (more) {
#pragma unroll
      for (int e = 0; e < NE; e++) acc[e] = T(0);
    }
  };

  stage(0, c0);
  int buf = 0, rows = 0;
  const int tile_rows = TP / G;
  const int roff = (j - j_lo) * rpitch, rlo = cj * rpitch;
  for (int64_t t0 = c0; t0 < c1; t0 += TP, buf ^= 1) {
    if (t0 + TP < c1)
      stage(buf ^ 1, t0 + TP);
    else
      asm volatile("cp.async.commit_group;\n" ::: "memory");   // keeps the wait count uniform
    asm volatile("cp.async.wait_group 1;\n" ::: "memory");
    __syncthreads();
    const float *sx = reinterpret_cast<const float *>(cv_smem + buf * buf_bytes);
    const unsigned char *sr = cv_smem + buf * buf_bytes + xbytes;
    if (act) {
      const int live = (int)min((int64_t)TP, c1 - t0);
#pragma unroll(TRI ? 2 : 1)
      for (int p = g; p < live; p += G) {
        const T r = R.get(sr, roff + p, rlo);
        float xa[TB];
        cv_load<TB>(sx + p * xpitch, bi, nb, xa);
        T ua[TB];
#pragma unroll
        for (int a = 0; a < TB; a++) ua[a] = (T)xa[a] - ma[a];
        if constexpr (TRI) {
          int e = 0;
#pragma unroll
          for (int a = 0; a < TB; a++) {
            const T w = r * ua[a];
#pragma unroll
            for (int b = a; b < TB; b++) acc[e] = fma(w, ua[b], acc[e]), e++;
          }
        } else {
          float xb[TB];
          cv_load<TB>(sx + p * xpitch, bj, nb, xb);
          T ub[TB];
#pragma unroll
          for (int b = 0; b < TB; b++) ub[b] = (T)xb[b] - mb[b];
#pragma unroll
          for (int a = 0; a < TB; a++) {
            const T w = r * ua[a];
#pragma unroll
            for (int b = 0; b < TB; b++) acc[a * TB + b] = fma(w, ub[b], acc[a * TB + b]);
          }
        }
      }
    }
    __syncthreads();
    rows += tile_rows;
    if (sizeof(T) == 4 && rows + tile_rows > kCvRows && t0 + TP < c1) {
      if (G > 1) {
        // the sums pass through the tiles' shared memory: stage the next tile again
        flush(true);
        if (d < dp)
          for (int e = tid; e < 2 * TP * (dp - d); e += kCvThreads) {
            const int row = e / (dp - d), q = d + e - row * (dp - d);
            float *sz = reinterpret_cast<float *>(cv_smem + (row >= TP ? buf_bytes : 0));
            sz[(row >= TP ? row - TP : row) * xpitch + cv_pos<TB>(q, nb)] = 0.f;
          }
        stage(buf ^ 1, t0 + TP);
      } else {
        flush(true);
      }
      rows = 0;
    }
  }
  flush(false);
}

// Covs_j = CovSum_j / PosteriorSum_j, upper mirrored to lower (EM2/MatrixEM.cpp:370-373).
// 32 consecutive elements per CTA, the chunks split over 8 threads each and
// combined in a fixed order: one thread per element left the sums of small
// fits to a chain of L2 loads (d = 24, K = 21: 248 -> 9 us).
__global__ void __launch_bounds__(256)
k_final_cov(const double *__restrict__ part, int chunks, int K, int d, int nb, int nblk, int TB, int tri,
            const double *__restrict__ psum, double *__restrict__ sigma) {
  __shared__ double red[8][32];
  const int units = K * nblk, ne = tri ? TB * (TB + 1) / 2 : TB * TB;
  const int64_t per = (int64_t)units * ne;
  const int lane = threadIdx.x & 31, sl = threadIdx.x >> 5;
  const int64_t i = (int64_t)blockIdx.x * 32 + lane;
  double s = 0.0;
  if (i < per)
    for (int c = sl; c < chunks; c += 8) s += part[(size_t)c * per + i];
  red[sl][lane] = s;
  __syncthreads();
  if (sl || i >= per) return;
#pragma unroll
  for (int q = 1; q < 8; q++) s += red[q][lane];
  int e = (int)(i / units);
  const int unit = (int)(i - (int64_t)e * units), j = unit / nblk;
  int b = unit - j * nblk, bi = 0, ra = 0, rb;
  while (b >= nb - bi) {
    b -= nb - bi;
    bi++;
  }
  if (tri) {
    while (e >= TB - ra) {
      e -= TB - ra;
      ra++;
    }
    rb = ra + e;
  } else {
    ra = e / TB;
    rb = e - ra * TB;
  }
  const int a = bi * TB + ra, c = (bi + b) * TB + rb;
  if (a > c || c >= d) return;     // lower half of a diagonal block, padding
  const double v = s / psum[j];
  double *S = sigma + (size_t)j * d * d;
  S[(size_t)a * d + c] = v;
  S[(size_t)c * d + a] = v;
}

}  // namespace

// Schedule of the covariance sums for one handle (fixed by its shape).
//
//  TB, tri   8 x 8 blocks; one triangular block when d <= 8 (4 x 4 when d <= 4)
//  gx, upc   CTAs the units are spread over and units per CTA: the split of
//            at most 8 more CTAs than needed that leaves the fewest of the
//            256 threads without a unit (600 units on 3 x 200 threads would
//            idle 22 %; 5 x 120 with two point groups idle 6 %)
//  chunks    row chunks: the count whose waves over the SMs finish first,
//            counting two tiles' time for a CTA's start and flush
CovPlan cov_plan(int d, int64_t n, int k, bool fp64, bool hilo) {
  CovPlan p{};
  p.TB = d <= 4 ? 4 : 8;
  p.nb = (d + p.TB - 1) / p.TB;
  p.tri = p.nb == 1;
  p.nblk = p.nb * (p.nb + 1) / 2;
  const int ne = p.tri ? p.TB * (p.TB + 1) / 2 : p.TB * p.TB;
  const int units = k * p.nblk, g0 = (units + kCvThreads - 1) / kCvThreads;
  double best = -1.0;
  for (int gx = g0; gx <= std::min(units, g0 + 8); gx++) {
    const int upc = (units + gx - 1) / gx, ctas = (units + upc - 1) / upc;
    const int G = std::min(kCvMaxGroups, kCvThreads / upc);
    const double eff = (double)units * G / ((double)ctas * kCvThreads) * (1.0 - 0.01 * (gx - g0));
    if (eff > best) best = eff, p.gx = ctas, p.upc = upc, p.G = G;
  }
  const int m = std::max(8, (32 / p.G + 7) / 8 * 8);   // points per thread and tile
  p.TP = p.G * m;
  p.xpitch = p.TB == 4 ? 4 : 8 * p.nb + 4;             // odd multiple of 16 bytes: point groups in different banks
  p.cj = std::min(k, (p.upc + p.nblk - 2) / p.nblk + 1);
  p.rpitch = hilo ? p.TP + 8 : p.TP + (fp64 ? 2 : 4);
  const size_t rb = ((size_t)p.cj * p.rpitch * (fp64 ? 8 : 4) + 15) & ~(size_t)15;
  p.smem = 2 * ((size_t)p.TP * p.xpitch * sizeof(float) + rb);
  if (p.G > 1) p.smem = std::max(p.smem, (size_t)ne * kCvThreads * (fp64 ? 8 : 4));
  const int slots = (fp64 ? 1 : 2) * sm_count();
  const int64_t tiles = (n + p.TP - 1) / p.TP;
  double bt = 1e300;
  for (int64_t c = 1; c <= std::min<int64_t>(tiles, (int64_t)3 * slots / p.gx + 1); c++) {
    const int64_t tpc = (tiles + c - 1) / c, ch = (tiles + tpc - 1) / tpc;
    const double waves = std::ceil((double)p.gx * ch / slots), t = waves * (tpc + 2.0);
    if (t < bt) bt = t, p.chunks = (int)ch, p.rows = tpc * p.TP;
  }
  p.part = (size_t)p.chunks * units * ne;
  return p;
}

// partials + FP64 finalisation for one posterior source
template <typename T, class Src>
static int cov_pass(fem_em *h, Src src, const T *mu, int mu_ld) {
  const CovPlan &p = h->cov;
  const int d = h->d, K = h->k;
  if (p.smem > kCvMaxSmem) {
    set_error("covariance tiles of d = %d need %zu bytes of shared memory", d, p.smem);
    return FEM_ERR_UNSUPPORTED;
  }
  const dim3 grid(p.gx, p.chunks);
#define FEM_CV(TB, TRI)                                                                                        \
  do {                                                                                                         \
    FEM_CUDA(allow_dyn_smem(k_cov_units<T, TB, TRI, Src>, p.smem));                                            \
    k_cov_units<T, TB, TRI, Src><<<grid, kCvThreads, p.smem, h->stream>>>(                                     \
        h->X, h->n, d, K, src, mu, mu_ld, h->cpart, p.nb, p.nblk, p.rows, p.upc, p.G, p.TP, p.xpitch, p.rpitch, \
        p.cj);                                                                                                 \
  } while (0)
  if (p.TB == 4)
    FEM_CV(4, true);
  else if (p.tri)
    FEM_CV(8, true);
  else
    FEM_CV(8, false);
#undef FEM_CV
  FEM_CUDA(cudaGetLastError());
  const int64_t per = (int64_t)K * p.nblk * (p.tri ? p.TB * (p.TB + 1) / 2 : p.TB * p.TB);
  k_final_cov<<<(unsigned)((per + 31) / 32), 256, 0, h->stream>>>(h->cpart, p.chunks, K, d, p.nb, p.nblk, p.TB, p.tri,
                                                                  h->psum, h->sigma);
  FEM_CUDA(cudaGetLastError());
  return FEM_OK;
}

int em_cov_hilo(fem_em *h, const __half *Rh, const __half *Rl, int64_t pitch, const float *muf, int mu_ld) {
  FEM_TRY((cov_pass<float, PostHiLo>(h, PostHiLo{Rh, Rl, pitch}, muf, mu_ld)));
  h->launches += 2;
  return FEM_OK;
}

int em_cov_plain(fem_em *h) {
  if (h->cfg.precision == FEM_PREC_FP64)
    return cov_pass<double, PostTyped<double>>(h, PostTyped<double>{(const double *)h->R, h->n},
                                               (const double *)h->muT, h->d);
  return cov_pass<float, PostTyped<float>>(h, PostTyped<float>{(const float *)h->R, h->n}, (const float *)h->muT,
                                           h->d);
}

}  // namespace fem
