// em_cov.cu -- the CUDA-core M-step sums of the EM sweep: covariances (FP32,
// FP64, and FP32 from the mixed path's FP16 hi/lo posteriors) and means (FP32,
// FP64).
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
// rate, by the 128-bit shared-memory loads; in FP64 (d <= 8; k_cov_staged above) by
// the FP64 pipe (2 per clock and SM).  FP32 8 x 8 blocks multiply two columns per instruction
// (N = 250007, d = 16, K = 200: 0.89 -> 0.68 ms; copies without a division per
// element 0.65).  On the GB300, against a kernel that wrote sqrt(r) (x - mu)
// of every component to shared memory and used one thread per block:
//   N = 2^20, d = 64, K = 128, FP32 from FP16 hi/lo   82.9 -> 20.7 ms
//   N = 250007, d = 16, K = 200, FP32                  8.20 -> 0.58 ms
//   N = 200003, d = 24, K = 21, FP32 from FP16 hi/lo   0.75 -> 0.115 ms
//   N = 100000, d = 8, K = 10, FP64                    1.52 -> 0.14 ms
#include <algorithm>
#include <cmath>

#include "em_kernels.cuh"
#include "em_tri.cuh"
#include "fem_internal.cuh"

namespace fem {

namespace {

constexpr int kCvThreads = 256;
constexpr int kCvRows = 2048;              // rows an FP32 sum may span before it is added into FP64
constexpr int kCvMaxGroups = 64;
constexpr size_t kCvMaxSmem = 232448;
constexpr int kCvTile = 128;               // points per tile

__device__ __forceinline__ void cv_copy4(void *dst, const void *src, bool valid) {
  const uint32_t da = static_cast<uint32_t>(__cvta_generic_to_shared(dst));
  asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;\n" ::"r"(da), "l"(src), "r"(valid ? 4 : 0) : "memory");
}
// the first `bytes` of 16, zeros behind them
__device__ __forceinline__ void cv_copy16z(void *dst, const void *src, int bytes) {
  const uint32_t da = static_cast<uint32_t>(__cvta_generic_to_shared(dst));
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;\n" ::"r"(da), "l"(src), "r"(bytes) : "memory");
}
__device__ __forceinline__ void cv_copy16(void *dst, const void *src, bool valid) {
  const uint32_t da = static_cast<uint32_t>(__cvta_generic_to_shared(dst));
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;\n" ::"r"(da), "l"(src), "r"(valid ? 16 : 0) : "memory");
}

// ------------------------------------------------------- posterior sources
// A source stages rows t0 .. t0 + TP - 1 of cj components into shared memory
// (rows past `end` as zero) and reads one of them back.  `pitch` is the
// number of elements between two components there.

// thread t's elements t, t + 256, ... of a row-major array of `width` columns,
// without a division per element
struct CvWalk {
  int row, col, width, drow, dcol;
  __device__ __forceinline__ explicit CvWalk(int w)
      : row(threadIdx.x / w), col(threadIdx.x % w), width(w), drow(kCvThreads / w), dcol(kCvThreads % w) {}
  __device__ __forceinline__ void next() {
    row += drow, col += dcol;
    if (col >= width) col -= width, row++;
  }
};

// component-major array of T, rows post_ld(n) apart: 16 bytes at a time (TP and
// t0 are multiples of 4; element by element over unpadded rows 250007 x 16 x 200
// took 605 us here and 125 in k_means_units, now 578 and 91)
template <typename T>
struct PostTyped {
  const T *R;
  int64_t ld;
  static constexpr size_t kBytes = sizeof(T);
  __device__ void stage(unsigned char *buf, int pitch, int j0, int cj, int64_t t0, int TP, int64_t end) const {
    constexpr int V = 16 / sizeof(T);
    T *s = reinterpret_cast<T *>(buf);
    for (CvWalk w(TP / V); w.row < cj; w.next()) {
      const int p = V * w.col, m = (int)max((int64_t)0, min((int64_t)V, end - t0 - p));
      cv_copy16z(s + w.row * pitch + p, R + (size_t)(j0 + w.row) * ld + (m ? t0 + p : 0), m * (int)sizeof(T));
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

// a block's eight columns as pairs, its 16-byte halves `half` floats apart
__device__ __forceinline__ void cv_load2(const float *x, int half, uint64_t (&v)[4]) {
  const ulonglong2 a = *reinterpret_cast<const ulonglong2 *>(x);
  const ulonglong2 c = *reinterpret_cast<const ulonglong2 *>(x + half);
  v[0] = a.x, v[1] = a.y, v[2] = c.x, v[3] = c.y;
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
            int rpitch, int cjmax, const int *__restrict__ gate) {
  if (gate && !(gate[0] | gate[1])) return;
  constexpr int NE = cv_ne(TB, TRI);
  // FP32 blocks of 8 x 8: two columns per instruction
  constexpr bool PK = sizeof(T) == 4 && TB == 8 && !TRI;
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
  uint64_t ma2[4], mb2[4], acc2[PK ? NE / 2 : 1];
#pragma unroll
  for (int e = 0; e < NE; e++) acc[e] = T(0);
#pragma unroll
  for (int e = 0; e < (PK ? NE / 2 : 1); e++) acc2[e] = 0;
  if constexpr (PK) {
#pragma unroll
    for (int a = 0; a < 4; a++)
      ma2[a] = f2_pack(ma[2 * a], ma[2 * a + 1]), mb2[a] = f2_pack(mb[2 * a], mb[2 * a + 1]);
  }

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
      for (CvWalk w(d4); w.row < TP; w.next()) {
        const int p = w.row, q = 4 * w.col;
        const bool v = t0 + p < c1;
        cv_copy16(sx + p * xpitch + cv_pos<TB>(q, nb), X + (v ? (t0 + p) * d + q : 0), v);
      }
    } else {
      for (CvWalk w(d); w.row < TP; w.next()) {
        const int p = w.row, q = w.col;
        const bool v = t0 + p < c1;
        cv_copy4(sx + p * xpitch + cv_pos<TB>(q, nb), X + (v ? (t0 + p) * d + q : 0), v);
      }
    }
    R.stage(cv_smem + buf * buf_bytes + xbytes, rpitch, j_lo, cj, t0, TP, c1);
    asm volatile("cp.async.commit_group;\n" ::: "memory");
  };

  bool first = true;
  // adds the FP32 sums into this CTA's FP64 partials (or stores them), the groups'
  // sums of a unit in group order: in T as long as they span kCvRows rows together,
  // else without FP32 rounding (group_sum, two more FP64 conversions and additions a
  // sum: N = 200003, d = 24, K = 21, 658 rows a CTA, 5 us a sweep)
  int rows = 0;                                     // of each group since the last flush
  auto flush = [&](bool more) {
    if constexpr (PK) {
#pragma unroll
      for (int e = 0; e < NE / 2; e++) f2_unpack(acc2[e], acc[2 * e], acc[2 * e + 1]);
    }
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
        const T *v = red + e * kCvThreads + u;
        double s;
        if (rows * G <= kCvRows) {
          T t = v[0];
          for (int q = 1; q < G; q++) t += v[q * upc];
          s = (double)t;
        } else {
          s = group_sum(v, G, upc);
        }
        double *p = o + (size_t)e * units + u;
        *p = first ? s : *p + s;
      }
      __syncthreads();
    }
    first = false;
    if (more) {
#pragma unroll
      for (int e = 0; e < NE; e++) acc[e] = T(0);
#pragma unroll
      for (int e = 0; e < (PK ? NE / 2 : 1); e++) acc2[e] = 0;
    }
  };

  stage(0, c0);
  int buf = 0;
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
      if constexpr (PK) {
        const float *xa = sx + g * xpitch + 4 * bi, *xb = sx + g * xpitch + 4 * bj;
        const int xs = G * xpitch, half = 4 * nb;
        int o = roff + g;
#pragma unroll 1
        for (int p = g; p < live; p += G, xa += xs, xb += xs, o += G) {
          const float r = R.get(sr, o, rlo);
          uint64_t ua[4], ub[4];
          cv_load2(xa, half, ua);
          cv_load2(xb, half, ub);
#pragma unroll
          for (int a = 0; a < 4; a++) ua[a] = f2_sub(ua[a], ma2[a]), ub[a] = f2_sub(ub[a], mb2[a]);
#pragma unroll
          for (int a = 0; a < 8; a++) {
            float u0, u1;
            f2_unpack(ua[a / 2], u0, u1);
            const float w = r * (a & 1 ? u1 : u0);
            const uint64_t ww = f2_pack(w, w);
#pragma unroll
            for (int b = 0; b < 4; b++) acc2[4 * a + b] = f2_fma(ww, ub[b], acc2[4 * a + b]);
          }
        }
      } else {
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

// FP64 with more than one block per dimension.  The FP64 pipe is all that counts, and
// k_cov_units would spend 104 of its operations per point and 8 x 8 unit on 64
// products (conversions, differences and weights formed by every unit).  Here a CTA's
// rows are turned into u = x - mu_j and w = r_ij u for its cj components once per
// tile, in shared memory, and a unit only multiplies.  Partials as k_cov_units leaves
// them.  M-steps on the GB300, N = 60000, by the kernel that staged sqrt(r) (x - mu)
// and used one thread per block, by k_cov_units, and here: d = 9, K = 200 3.80, 7.33,
// 3.30 ms; d = 20, K = 60 3.67, 4.58, 2.35; d = 32, K = 20 3.66, 2.33, 1.66; d = 64, K =
// 60 17.9, 26.8, 15.7; d = 256, K = 9 37.9, 52.0, 34.7; N = 5000, d = 32, K = 9 0.48,
// 0.15, 0.12.
template <int TB>
__global__ void __launch_bounds__(kCvThreads, TB == 8 ? 1 : 2)
k_cov_staged(const float *__restrict__ X, int64_t n, int d, int K, PostTyped<double> R, const double *__restrict__ mu,
             double *__restrict__ part, int nb, int nblk, int64_t rows_per_chunk, int upc, int G, int TP, int xpitch,
             int rpitch, int cjmax) {
  constexpr int NE = TB * TB;
  extern __shared__ __align__(16) unsigned char cv_smem[];
  const int tid = threadIdx.x, units = K * nblk, u0 = blockIdx.x * upc;
  const int j_lo = u0 / nblk, cj = min(K - 1, (u0 + upc - 1) / nblk) - j_lo + 1;
  const int g = tid / upc, ul = tid - g * upc, unit = u0 + ul;
  const bool act = g < G && unit < units;
  const size_t xbytes = (size_t)TP * xpitch * sizeof(float), buf_bytes = xbytes + (size_t)cjmax * rpitch * sizeof(double);
  const int dp = nb * TB, zp = dp + 2;              // row pitch of u and w
  double *su = reinterpret_cast<double *>(cv_smem + 2 * buf_bytes), *sw = su + (size_t)cjmax * TP * zp;
  int j = j_lo, bi = 0, bj = 0;
  if (act) {
    j = unit / nblk;
    int b = unit - j * nblk;
    while (b >= nb - bi) {
      b -= nb - bi;
      bi++;
    }
    bj = bi + b;
  }
  double acc[NE];
#pragma unroll
  for (int e = 0; e < NE; e++) acc[e] = 0.0;
  const int64_t c0 = (int64_t)blockIdx.y * rows_per_chunk, c1 = min(n, c0 + rows_per_chunk);
  auto stage = [&](int buf, int64_t t0) {
    float *sx = reinterpret_cast<float *>(cv_smem + buf * buf_bytes);
    if ((d & 3) == 0) {
      for (CvWalk w(d >> 2); w.row < TP; w.next()) {
        const bool v = t0 + w.row < c1;
        cv_copy16(sx + w.row * xpitch + 4 * w.col, X + (v ? (t0 + w.row) * d + 4 * w.col : 0), v);
      }
    } else {
      for (CvWalk w(d); w.row < TP; w.next()) {
        const bool v = t0 + w.row < c1;
        cv_copy4(sx + w.row * xpitch + w.col, X + (v ? (t0 + w.row) * d + w.col : 0), v);
      }
    }
    R.stage(cv_smem + buf * buf_bytes + xbytes, rpitch, j_lo, cj, t0, TP, c1);
    asm volatile("cp.async.commit_group;\n" ::: "memory");
  };
  stage(0, c0);
  int buf = 0;
  for (int64_t t0 = c0; t0 < c1; t0 += TP, buf ^= 1) {
    if (t0 + TP < c1)
      stage(buf ^ 1, t0 + TP);
    else
      asm volatile("cp.async.commit_group;\n" ::: "memory");   // keeps the wait count uniform
    asm volatile("cp.async.wait_group 1;\n" ::: "memory");
    __syncthreads();
    const float *sx = reinterpret_cast<const float *>(cv_smem + buf * buf_bytes);
    const double *sr = reinterpret_cast<const double *>(cv_smem + buf * buf_bytes + xbytes);
    const int live = (int)min((int64_t)TP, c1 - t0);
    for (CvWalk w(dp); w.row < cj * TP; w.next()) {
      const int jj = w.row / TP, p = w.row - jj * TP, q = w.col;
      if (p >= live) continue;
      const double u = q < d ? (double)sx[p * xpitch + q] - __ldg(mu + (size_t)(j_lo + jj) * d + q) : 0.0;
      su[(size_t)w.row * zp + q] = u;
      sw[(size_t)w.row * zp + q] = sr[jj * rpitch + p] * u;
    }
    __syncthreads();
    if (act) {
      const double *wa = sw + (size_t)(j - j_lo) * TP * zp + bi * TB, *ub = su + (size_t)(j - j_lo) * TP * zp + bj * TB;
#pragma unroll 1
      for (int p = g; p < live; p += G) {
        double a[TB], b[TB];
#pragma unroll
        for (int q = 0; q < TB; q += 2) {
          const double2 va = *reinterpret_cast<const double2 *>(wa + p * zp + q);
          const double2 vb = *reinterpret_cast<const double2 *>(ub + p * zp + q);
          a[q] = va.x, a[q + 1] = va.y, b[q] = vb.x, b[q + 1] = vb.y;
        }
#pragma unroll
        for (int e = 0; e < NE; e++) acc[e] = fma(a[e / TB], b[e % TB], acc[e]);
      }
    }
    __syncthreads();
  }
  double *o = part + (size_t)blockIdx.y * NE * units + u0;
  if (G == 1) {
    if (act)
#pragma unroll
      for (int e = 0; e < NE; e++) o[(size_t)e * units + ul] = acc[e];
    return;
  }
  double *red = reinterpret_cast<double *>(cv_smem);   // NE x 256, over the tiles
  asm volatile("cp.async.wait_group 0;\n" ::: "memory");
  __syncthreads();
#pragma unroll
  for (int e = 0; e < NE; e++) red[e * kCvThreads + tid] = acc[e];
  __syncthreads();
  const int live = min(upc, units - u0);
  for (int i = tid; i < live * NE; i += kCvThreads) {
    const int e = i / live, u = i - e * live;
    o[(size_t)e * units + u] = group_sum(red + e * kCvThreads + u, G, upc);
  }
}

// Covs_j = CovSum_j / PosteriorSum_j, upper mirrored to lower (EM2/MatrixEM.cpp:370-373).
// 32 consecutive elements per CTA, the chunks split over 8 threads each and
// combined in a fixed order: one thread per element left the sums of small
// fits to a chain of L2 loads (d = 24, K = 21: 248 -> 9 us).
__global__ void __launch_bounds__(256)
k_final_cov(const double *__restrict__ part, int chunks, int K, int d, int nb, int nblk, int TB, int tri,
            const double *__restrict__ psum, double *__restrict__ sigma, const int *__restrict__ gate) {
  if (gate && !(gate[0] | gate[1])) return;
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

// ============================================================== means
// SimpleMatrixEM::doMStep means part (EM2/MatrixEM.cpp:319-343):
// PosteriorSum_j = sum_i r_ij and MeanSums_j = sum_i r_ij x_i as the product
// R^T [X | 1] (column d of a staged row is 1).  A thread owns 4 components x 4
// columns for every G-th group of 4 points; units, point groups and chunks as
// in k_cov_units.  FP32 sums span at most kMnRows rows, then go into the
// thread's FP64 sums; the point groups are combined in FP64, in order.
// part[chunk][component][0: sum r, 1 + q: sum r x_q].  Per 4 points 8 128-bit
// shared-memory loads feed 64 products, which is what bounds the FP32 form.
// Against one component x 8 or 16 columns per thread (GB300): N = 250007,
// d = 16, K = 200, FP32 239 -> 138 us; N = 100000, d = 8, K = 10, FP64 128 -> 54 us.
constexpr int kMnRows = 512;

template <typename T>
__device__ __forceinline__ void mn_load(const T *p, T (&v)[4]);
template <>
__device__ __forceinline__ void mn_load(const float *p, float (&v)[4]) {
  const float4 a = *reinterpret_cast<const float4 *>(p);
  v[0] = a.x, v[1] = a.y, v[2] = a.z, v[3] = a.w;
}
template <>
__device__ __forceinline__ void mn_load(const double *p, double (&v)[4]) {
  const double2 a = reinterpret_cast<const double2 *>(p)[0], b = reinterpret_cast<const double2 *>(p)[1];
  v[0] = a.x, v[1] = a.y, v[2] = b.x, v[3] = b.y;
}

template <typename T>
__global__ void __launch_bounds__(kCvThreads, 2)
k_means_units(const float *__restrict__ X, int64_t n, int d, int K, PostTyped<T> R, double *__restrict__ part, int nc,
              int64_t rows_per_chunk, int upc, int G, int TP, int xpitch, int rpitch, int cjmax) {
  extern __shared__ __align__(16) unsigned char cv_smem[];
  const int tid = threadIdx.x;
  const int units = (K + 3) / 4 * nc, u0 = blockIdx.x * upc;
  const int b_lo = u0 / nc, b_hi = min(units - 1, u0 + upc - 1) / nc;
  const int j_lo = 4 * b_lo, cj = min(K, 4 * b_hi + 4) - j_lo;
  const int g = tid / upc, ul = tid - g * upc, unit = u0 + ul;
  const bool act = g < G && unit < units;
  const int jb = act ? unit / nc : b_lo, cb = act ? unit - jb * nc : 0;
  const size_t xbytes = (size_t)TP * xpitch * sizeof(float);
  const size_t buf_bytes = xbytes + (size_t)cjmax * rpitch * sizeof(T);
  const int64_t c0 = (int64_t)blockIdx.y * rows_per_chunk, c1 = min(n, c0 + rows_per_chunk);
  // what the copies leave alone: columns d (ones) .. 4 nc - 1 (zero) of the
  // rows, and posteriors of components past K
  for (int e = tid; e < 2 * TP * (4 * nc - d); e += kCvThreads) {
    const int row = e / (4 * nc - d), q = d + e - row * (4 * nc - d);
    float *sx = reinterpret_cast<float *>(cv_smem + (row >= TP ? buf_bytes : 0));
    sx[(row >= TP ? row - TP : row) * xpitch + q] = q == d ? 1.f : 0.f;
  }
  for (int e = tid; e < 2 * (cjmax - cj) * rpitch; e += kCvThreads) {
    const int b = e / ((cjmax - cj) * rpitch), o = e - b * (cjmax - cj) * rpitch;
    reinterpret_cast<T *>(cv_smem + b * buf_bytes + xbytes)[cj * rpitch + o] = T(0);
  }
  auto stage = [&](int buf, int64_t t0) {
    float *sx = reinterpret_cast<float *>(cv_smem + buf * buf_bytes);
    if ((d & 3) == 0) {
      const int d4 = d >> 2;
      for (CvWalk w(d4); w.row < TP; w.next()) {
        const int p = w.row, q = 4 * w.col;
        const bool v = t0 + p < c1;
        cv_copy16(sx + p * xpitch + q, X + (v ? (t0 + p) * d + q : 0), v);
      }
    } else {
      for (CvWalk w(d); w.row < TP; w.next()) {
        const int p = w.row, q = w.col;
        const bool v = t0 + p < c1;
        cv_copy4(sx + p * xpitch + q, X + (v ? (t0 + p) * d + q : 0), v);
      }
    }
    R.stage(cv_smem + buf * buf_bytes + xbytes, rpitch, j_lo, cj, t0, TP, c1);
    asm volatile("cp.async.commit_group;\n" ::: "memory");
  };
  T acc[4][4];
  double dacc[4][4];
#pragma unroll
  for (int q = 0; q < 4; q++)
#pragma unroll
    for (int c = 0; c < 4; c++) acc[q][c] = T(0), dacc[q][c] = 0.0;
  auto fold = [&]() {
#pragma unroll
    for (int q = 0; q < 4; q++)
#pragma unroll
      for (int c = 0; c < 4; c++) dacc[q][c] += (double)acc[q][c], acc[q][c] = T(0);
  };
  stage(0, c0);
  int buf = 0, rows = 0;
  const int tile_rows = TP / G;
  for (int64_t t0 = c0; t0 < c1; t0 += TP, buf ^= 1) {
    if (t0 + TP < c1)
      stage(buf ^ 1, t0 + TP);
    else
      asm volatile("cp.async.commit_group;\n" ::: "memory");   // keeps the wait count uniform
    asm volatile("cp.async.wait_group 1;\n" ::: "memory");
    __syncthreads();
    if (act) {
      const float *sx = reinterpret_cast<const float *>(cv_smem + buf * buf_bytes) + 4 * cb;
      const T *sr = reinterpret_cast<const T *>(cv_smem + buf * buf_bytes + xbytes) + 4 * (jb - b_lo) * rpitch;
      for (int p = 4 * g; p < TP; p += 4 * G) {
        T r[4][4];
#pragma unroll
        for (int q = 0; q < 4; q++) mn_load(sr + q * rpitch + p, r[q]);
#pragma unroll
        for (int i = 0; i < 4; i++) {
          float x[4];
          mn_load(sx + (p + i) * xpitch, x);
#pragma unroll
          for (int c = 0; c < 4; c++) {
            const T xc = (T)x[c];
#pragma unroll
            for (int q = 0; q < 4; q++) acc[q][c] = fma(r[q][i], xc, acc[q][c]);
          }
        }
      }
    }
    __syncthreads();
    rows += tile_rows;
    if (sizeof(T) == 4 && rows + tile_rows > kMnRows) fold(), rows = 0;
  }
  fold();
  double *o = part + (size_t)blockIdx.y * K * (d + 1);
  auto put = [&](int u, int e, double v) {     // element e of unit u
    const int b = u / nc, c = 4 * (u - b * nc) + (e & 3), j = 4 * b + (e >> 2);
    if (j < K && c <= d) o[(size_t)j * (d + 1) + (c == d ? 0 : 1 + c)] = v;
  };
  if (G == 1) {
    if (act)
#pragma unroll
      for (int e = 0; e < 16; e++) put(unit, e, dacc[e >> 2][e & 3]);
    return;
  }
  double *red = reinterpret_cast<double *>(cv_smem);   // 16 x 256, over the tiles
  asm volatile("cp.async.wait_group 0;\n" ::: "memory");
  __syncthreads();
#pragma unroll
  for (int e = 0; e < 16; e++) red[e * kCvThreads + tid] = dacc[e >> 2][e & 3];
  __syncthreads();
  const int live = min(upc, units - u0);
  for (int i = tid; i < live * 16; i += kCvThreads) {
    const int e = i / live, u = i - e * live;
    double v = red[e * kCvThreads + u];
    for (int q = 1; q < G; q++) v += red[e * kCvThreads + q * upc + u];
    put(u0 + u, e, v);
  }
}

}  // namespace

// gx CTAs of upc units with G point groups each: the split of at most 8 more
// CTAs than needed that leaves the fewest of the threads without a unit (600
// units on 3 x 200 threads would idle 22 %; 5 x 120 with two groups idle 6 %)
void split_units(int units, int *gx, int *upc, int *G) {
  const int g0 = (units + kCvThreads - 1) / kCvThreads;
  double best = -1.0;
  for (int c = g0; c <= std::min(units, g0 + 8); c++) {
    const int u = (units + c - 1) / c, ctas = (units + u - 1) / u;
    const int g = std::min(kCvMaxGroups, kCvThreads / u);
    const double eff = (double)units * g / ((double)ctas * kCvThreads) * (1.0 - 0.01 * (c - g0));
    if (eff > best) best = eff, *gx = ctas, *upc = u, *G = g;
  }
}

// row chunks: the count whose waves over `slots` resident CTAs finish first,
// counting `extra` tiles' time for a CTA's start and end
void split_rows(int64_t n, int TP, int gx, int slots, double extra, int *chunks, int64_t *rows) {
  const int64_t tiles = (n + TP - 1) / TP;
  double bt = 1e300;
  for (int64_t c = 1; c <= std::min<int64_t>(tiles, (int64_t)3 * slots / gx + 1); c++) {
    const int64_t tpc = (tiles + c - 1) / c, ch = (tiles + tpc - 1) / tpc;
    const double t = std::ceil((double)gx * ch / slots) * (tpc + extra);
    if (t < bt) bt = t, *chunks = (int)ch, *rows = tpc * TP;
  }
}

// Schedule of k_cov_staged with TB x TB blocks; returns its FP64 operations per row, 0
// where no tile fits (every d and k of the FP64 form has one that does)
static double staged_plan(int d, int64_t n, int k, int TB, CovPlan *out) {
  CovPlan p{};
  p.TB = TB;
  p.nb = (d + TB - 1) / TB;
  p.nblk = p.nb * (p.nb + 1) / 2;
  split_units(k * p.nblk, &p.gx, &p.upc, &p.G);
  p.cj = std::min(k, (p.upc + p.nblk - 2) / p.nblk + 1);
  p.xpitch = (d + 3) & ~3;
  const size_t red = p.G > 1 ? (size_t)TB * TB * kCvThreads * sizeof(double) : 0;
  const size_t most = kCvMaxSmem / (TB == 8 ? 1 : 2) - 1024;
  for (int tile = 64;; tile /= 2) {
    if (tile < 8) return 0.0;
    p.TP = (p.G * std::max(1, tile / p.G) + 1) & ~1;
    p.rpitch = p.TP + 2;
    p.smem = std::max(red, 2 * ((size_t)p.TP * p.xpitch * sizeof(float) + (size_t)p.cj * p.rpitch * sizeof(double)) +
                               2 * (size_t)p.cj * p.TP * (p.nb * TB + 2) * sizeof(double));
    if (p.smem <= most) break;
  }
  split_rows(n, p.TP, p.gx, (TB == 8 ? 1 : 2) * sm_count(), 2.0, &p.chunks, &p.rows);
  p.part = (size_t)p.chunks * k * p.nblk * TB * TB;
  *out = p;
  return p.gx * ((double)p.upc * TB * TB + 3.0 * p.cj * p.nb * TB);
}

// Schedule of the covariance sums for one handle (fixed by its shape).
//
//  TB, tri   8 x 8 blocks; one triangular block when d <= 8 (4 x 4 when d <= 4).  FP64
//            with d > 8: k_cov_staged by 4 x 4 or 8 x 8 blocks, whichever takes fewer
//            operations (4 x 4 pads and doubles less, 8 x 8 stages a component's rows
//            for more products: d = 9, K = 200 3.3 against 5.7 ms, d = 64, K = 60 15.7
//            against 16.9, d = 256, K = 9 45.6 against 34.7, N = 60000)
//  units     split as split_units says, rows as split_rows says
CovPlan cov_plan(int d, int64_t n, int k, bool fp64, bool hilo) {
  if (fp64 && d > 8) {
    CovPlan q[2];
    const double c4 = staged_plan(d, n, k, 4, &q[0]), c8 = staged_plan(d, n, k, 8, &q[1]);
    return q[c4 > 0.0 && (c8 == 0.0 || c4 <= c8) ? 0 : 1];
  }
  CovPlan p{};
  p.TB = d <= 4 ? 4 : 8;
  p.nb = (d + p.TB - 1) / p.TB;
  p.tri = p.nb == 1;
  p.nblk = p.nb * (p.nb + 1) / 2;
  const int ne = p.tri ? p.TB * (p.TB + 1) / 2 : p.TB * p.TB;
  const int units = k * p.nblk;
  split_units(units, &p.gx, &p.upc, &p.G);
  p.xpitch = p.TB == 4 ? 4 : 8 * p.nb + 4;             // odd multiple of 16 bytes: point groups in different banks
  p.cj = std::min(k, (p.upc + p.nblk - 2) / p.nblk + 1);
  // kCvTile points a tile (250007 x 16 x 200: 32, 64, 128, 256 points 653, 625,
  // 605, 605 us), fewer where two CTAs would no longer share an SM
  for (int tile = kCvTile; tile >= 32; tile /= 2) {
    p.TP = p.G * std::max(8, (tile / p.G + 7) / 8 * 8);
    p.rpitch = hilo ? p.TP + 8 : p.TP + (fp64 ? 2 : 4);
    const size_t rb = ((size_t)p.cj * p.rpitch * (fp64 ? 8 : 4) + 15) & ~(size_t)15;
    p.smem = 2 * ((size_t)p.TP * p.xpitch * sizeof(float) + rb);
    if (p.smem <= kCvMaxSmem / 2 - 1024) break;
  }
  if (p.G > 1) p.smem = std::max(p.smem, (size_t)ne * kCvThreads * (fp64 ? 8 : 4));
  split_rows(n, p.TP, p.gx, (fp64 ? 1 : 2) * sm_count(), 2.0, &p.chunks, &p.rows);
  p.part = (size_t)p.chunks * units * ne;
  return p;
}

// Schedule of the means sums (TB = 4: 4 components x 4 columns per unit; nb =
// column groups of a row and its 1)
CovPlan means_plan(int d, int64_t n, int k, bool fp64) {
  CovPlan p{};
  p.TB = 4;
  p.nb = (d + 4) / 4;
  const int units = (k + 3) / 4 * p.nb;
  split_units(units, &p.gx, &p.upc, &p.G);
  p.xpitch = 4 * p.nb;
  p.cj = 4 * std::min((k + 3) / 4, (p.upc + p.nb - 2) / p.nb + 1);
  const size_t ts = fp64 ? 8 : 4;
  for (int m = std::max(2, 8 / p.G); m >= 1; m /= 2) {   // groups of 4 points per thread and tile
    p.TP = 4 * p.G * m;
    p.rpitch = p.TP + 16 / (int)ts;
    p.smem = 2 * ((size_t)p.TP * p.xpitch * sizeof(float) + (size_t)p.cj * p.rpitch * ts);
    if (p.smem <= kCvMaxSmem / 2) break;
  }
  if (p.G > 1) p.smem = std::max(p.smem, (size_t)16 * kCvThreads * sizeof(double));
  split_rows(n, p.TP, p.gx, 2 * sm_count(), 2.0, &p.chunks, &p.rows);
  p.part = (size_t)p.chunks * k * (d + 1);
  return p;
}

template <typename T>
static int means_pass(fem_em *h) {
  const CovPlan &p = h->means;
  FEM_CUDA(allow_dyn_smem(k_means_units<T>, p.smem));
  k_means_units<T><<<dim3(p.gx, p.chunks), kCvThreads, p.smem, h->stream>>>(
      h->X, h->n, h->d, h->k, PostTyped<T>{(const T *)h->R, post_ld(h->n)}, h->mpart, p.nb, p.rows, p.upc, p.G, p.TP, p.xpitch,
      p.rpitch, p.cj);
  FEM_CUDA(cudaGetLastError());
  return FEM_OK;
}

int em_means_plain(fem_em *h) {
  return h->cfg.precision == FEM_PREC_FP64 ? means_pass<double>(h) : means_pass<float>(h);
}

// partials + FP64 finalisation for one posterior source
template <typename T, class Src>
static int cov_pass(fem_em *h, Src src, const T *mu, int mu_ld, const int *gate = nullptr) {
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
        p.cj, gate);                                                                                           \
  } while (0)
  if (p.TB == 4 && p.tri) {
    FEM_CV(4, true);
  } else if (p.tri) {
    FEM_CV(8, true);
  } else if constexpr (sizeof(T) == 4) {
    FEM_CV(8, false);
  } else {
    auto launch = [&](auto kern) -> int {
      FEM_CUDA(allow_dyn_smem(kern, p.smem));
      kern<<<grid, kCvThreads, p.smem, h->stream>>>(h->X, h->n, d, K, src, mu, h->cpart, p.nb, p.nblk, p.rows, p.upc, p.G,
                                                    p.TP, p.xpitch, p.rpitch, p.cj);
      return FEM_OK;
    };
    FEM_TRY(p.TB == 8 ? launch(k_cov_staged<8>) : launch(k_cov_staged<4>));
  }
#undef FEM_CV
  FEM_CUDA(cudaGetLastError());
  const int64_t per = (int64_t)K * p.nblk * (p.tri ? p.TB * (p.TB + 1) / 2 : p.TB * p.TB);
  k_final_cov<<<(unsigned)((per + 31) / 32), 256, 0, h->stream>>>(h->cpart, p.chunks, K, d, p.nb, p.nblk, p.TB, p.tri,
                                                                  h->psum, h->sigma, gate);
  FEM_CUDA(cudaGetLastError());
  return FEM_OK;
}

int em_cov_hilo(fem_em *h, const __half *Rh, const __half *Rl, int64_t pitch, const float *muf, int mu_ld,
                const int *gate) {
  FEM_TRY((cov_pass<float, PostHiLo>(h, PostHiLo{Rh, Rl, pitch}, muf, mu_ld, gate)));
  h->launches += 2;
  return FEM_OK;
}

int em_cov_plain(fem_em *h) {
  if (h->cfg.precision == FEM_PREC_FP64)
    return cov_pass<double, PostTyped<double>>(h, PostTyped<double>{(const double *)h->R, post_ld(h->n)},
                                               (const double *)h->muT, h->d);
  return cov_pass<float, PostTyped<float>>(h, PostTyped<float>{(const float *)h->R, post_ld(h->n)}, (const float *)h->muT,
                                           h->d);
}

}  // namespace fem
