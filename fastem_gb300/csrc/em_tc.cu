// em_tc.cu -- tcgen05 mixed-precision EM sweep for sm_103a (d = 64).
//
// One sweep = SimpleMatrixEM::PrecomputeDensityMatrix + MStep
// (EM2/MatrixEM.cpp:275-378) as three tensor-core kernels and two FP64
// finalisers:
//
//  1. E-step (MatrixEMBase::BlockDensities + PostProcessDensityMatrix,
//     EM2/MatrixEM.cpp:39-51,69-81): ONE GEMM of the points against the
//     stacked inverse Cholesky factors of all components,
//       Y = X W^T,  W = [L_1^-1; ...; L_K^-1],  y_jk = (L_j^-1 x)_k,
//     in FP16 x 3 (x = xh + xl, W = Wh + Wl: Xh Wh^T + Xh Wl^T + Xl Wh^T)
//     with FP32 accumulation in TMEM.  A CTA works on a pair of 128-point
//     tiles so every W group fetched from L2 feeds two M=128 MMAs.  The
//     epilogue subtracts b_j = L_j^-1 mu_j (kept in shared memory), squares
//     and sums each component's 64 columns, adds the log coefficient (float
//     hi + lo) and keeps an online log-sum-exp per point; the posteriors
//     r_ij = exp(l_ij - LSE_i) of the previous pair are finished while the
//     current pair's groups drain, and stored as FP16 hi/lo pairs
//     (component-major).  The per-point log-likelihood is summed in FP64 with
//     the FP64 log coefficient of the winning component.
//     Within a group of 2 components the 128 accumulator columns are ordered
//     by 16-wide k-block, highest first, so K-step kb only needs the first
//     128-32kb columns (L^-1 is lower triangular): 37.5% of the MMA work is
//     skipped.
//  2. Means (doMStep means part, EM2/MatrixEM.cpp:319-343): S2 = R^T X and
//     S1 = R^T 1 as one GEMM per 64-point block, A = [Rh | Rl] (components
//     x points), B = [Xh^T; 1] / [Xl^T; 0] (80 rows x points); FP32 in TMEM,
//     flushed to FP64 every 4096 points.
//  3. Covariances (ComputeWeightedTempDataset + BlockCovariances,
//     EM2/MatrixEM.cpp:53-67,90-99) around the NEW means: producer warps
//     form z = sqrt(r) (x - mu_j) in FP32, store fp16(z) as the operand of
//     an M=128 (two components) x N=128 x K=16 MMA whose diagonal blocks are
//     Z_j^T Z_j, and accumulate the exact diagonal sum z^2 in FP32 -> FP64
//     (FP16 rounding would bias the diagonal upward by E[delta^2]).
//
// Every mbarrier wait is bounded; a timeout sets a status word, the roles
// leave their loops, in-flight copies and MMAs are drained and TMEM is
// released.
#include <cuda.h>
#include <cuda_fp16.h>

#include <algorithm>
#include <cfloat>
#include <climits>
#include <cmath>
#include <vector>

#include "em_kernels.cuh"
#include "fem_internal.cuh"
#include "tc_ptx.cuh"

namespace fem {

using namespace tc;

// ------------------------------------------------------------ constants
constexpr int kD = 64;                   // dimension handled by the tensor-core path
constexpr int kTileM = 128;              // E-step points per tile (two tiles per CTA step)
constexpr int kGroupN = 128;             // E-step accumulator columns per component group
constexpr int kCompPerGroup = kGroupN / kD;
constexpr int kWStages = 4;
constexpr uint32_t kXBytes = kTileM * kD * 2;    // one FP16 X tile (16 KB)
constexpr uint32_t kWBytes = kGroupN * kD * 2;   // one FP16 W group (16 KB)
constexpr int kEThreads = 320;  // warp 0 TMA, 1 MMA, 2..9 epilogue
constexpr int kBlk = 64;                 // M-step points per block (one 128-byte swizzle row)
constexpr int kFlushBlocks = 64;         // FP32 TMEM window: 64 blocks = 4096 points
constexpr int kMaxK = 128;               // components handled by one means M-tile
constexpr int kMStages = 3;              // means input ring
constexpr int kCIn = 6;                  // covariance input ring

struct __align__(1024) ESmem {
  __half xh[2][kTileM * kD];   // the two tiles of the current pair
  __half xl[2][kTileM * kD];
  __half wh[kWStages][kGroupN * kD];
  __half wl[kWStages][kGroupN * kD];
  float bias[kMaxK * kD];      // b = L^-1 mu, permuted like the accumulator columns
  float chi[kMaxK], clo[kMaxK];
  uint64_t x_full, x_empty;
  uint64_t w_full[kWStages], w_empty[kWStages];
  uint64_t acc_full[2][2], acc_empty[2][2];   // [TMEM buffer][tile of the pair]
  uint64_t mma_done;
  uint32_t tmem_base;
  double red[8];
};

// means kernel: A = Rh/Rl (128 comps x 64 points), B = [X^T; 1] (80 x 64)
constexpr int kMeanN = 80;
struct __align__(1024) MSmem {
  __half rh[kMStages][kMaxK * kBlk];
  __half rl[kMStages][kMaxK * kBlk];
  __half bh[kMStages][kMeanN * kBlk];   // rows 0..63 X_h^T, row 64 ones, rows 65..79 zero
  __half bl[kMStages][kMeanN * kBlk];   // rows 0..63 X_l^T, rows 64..79 zero
  uint64_t in_full[kMStages], in_empty[kMStages], acc_full[2], acc_empty[2], mma_done;
  uint32_t tmem_base;
};

// covariance kernel: 4 components per CTA (2 pairs), 64-point blocks
constexpr int kZStages = 3;              // operand (z) ring
constexpr int kCProd = 16;               // producer warps: 2 groups x 8 point chunks
struct __align__(1024) CSmem {
  __half z[kZStages][2][128 * kBlk];  // [stage][pair] 128 rows (comp q dims) x 64 points, SW128
  float xs[kCIn][kBlk * kD];     // X tile (points x dims)
  __half rh[kCIn][4 * kBlk];
  __half rl[kCIn][4 * kBlk];
  float sr[kCProd][4 * 8];       // per producer warp: sqrt(r) of its 8 points x 4 components
  double dred[8][4][kD];         // exact-diagonal partials of the 8 point chunks
  uint64_t in_full[kCIn], in_empty[kCIn], z_full[kZStages], z_empty[kZStages], acc_full[2], acc_empty[2],
      mma_done;
  uint32_t tmem_base;
};
constexpr int kCThreads = (2 + kCProd + 4) * 32;   // warp 0 TMA, 1 MMA, 2..17 producers, 18..21 flush
static_assert(sizeof(CSmem) + 1024 <= 232448, "covariance kernel shared memory");

// covariance kernel, z x^T form: 4 components per CTA (2 pairs), 64-point blocks
#ifndef FEM_COV_GROUPS
#define FEM_COV_GROUPS 4
#endif
#ifndef FEM_COV_SPLIT
#define FEM_COV_SPLIT 2
#endif
#ifndef FEM_COV_STAGGER
#define FEM_COV_STAGGER 0
#endif
constexpr int kZIn = 6;                  // input ring (blocks)
constexpr int kZA = 3;                   // TMEM A ring (blocks of 64 points, both pairs)
constexpr int kZSets = FEM_COV_GROUPS;   // producer groups of 4 warps (one per TMEM lane quarter)
constexpr int kZSplit = FEM_COV_SPLIT;   // groups sharing a block (each takes kBlk / 16 / kZSplit K steps)
constexpr int kZStagger = FEM_COV_STAGGER;
constexpr int kZN = 80;                  // accumulator columns per pair: 64 (x) + 16 (column 64 = sum z)
constexpr uint32_t kZDCol = kZN;         // accumulator column pitch (pairs, buffers)
constexpr uint32_t kZACol = 4 * kZN;     // first column of the A ring
constexpr uint32_t kZAStage = 2 * (kBlk / 2);   // A columns per block: 2 pairs x 32 (64 FP16 points)
constexpr int kZThreads = (2 + 4 * kZSets + 4) * 32;   // TMA, MMA, producers, flush
constexpr int kZCols = kD + 1;           // flushed columns per pair row: 64 sums z x_b, then sum z
struct __align__(1024) ZSmem {
  __half bh[kZIn][kZN * kBlk];   // rows 0..63 X_h^T (TMA), row 64 ones, rows 65..79 zero (SW128)
  __half bl[kZIn][kD * kBlk];    // X_l^T (TMA, SW128)
  __half rh[kZIn][4 * kBlk];     // posteriors (hi part) of the CTA's 4 components
  uint64_t in_full[kZIn], in_empty[kZIn], a_full[kZA], a_empty[kZA], acc_full[2], acc_empty[2], mma_done;
  uint32_t tmem_base;
};
static_assert(sizeof(ZSmem) + 1024 <= 232448, "covariance kernel shared memory");
static_assert(kZSets % kZSplit == 0 && (kBlk / 16) % kZSplit == 0, "covariance producer split");
static_assert(kZACol + kZA * kZAStage <= 512 && 3 * kZDCol + kZN <= kZACol, "covariance kernel TMEM columns");

// covariance kernel, split z x^T form: 4 components per CTA (2 pairs), 64-point blocks of four 16-point steps
constexpr int kSIn = 4;                  // input ring (blocks)
constexpr int kSSteps = kBlk / 16;
constexpr int kSA = 6;                   // TMEM A ring (steps)
constexpr int kSAccLong = 16, kSAccShort = 4;   // blocks a zh xg^T accumulator spans
constexpr int kSAccWeight = 24;          // the short span from 1 / 24 of all posterior weight in one component on
constexpr int kSWin = 64;                // blocks an FP32 register sum spans (4096 rows)
constexpr int kSCrossWin = 256;          // blocks the small products' accumulator spans
constexpr int kSRows = 2048;             // rows an FP32 diagonal sum spans
// TMEM columns: [pair] zh [xg; 1]^T, [pair] the small products, A ring (per pair 8 hi + 8 lo a step)
constexpr int kSN = kD + 16;             // accumulator columns per pair: 64 sums, sum z, 15 unused
constexpr uint32_t kSCross = 2 * kSN, kSACol = 4 * kSN, kSAStage = 32;
// warps 0 TMA, 1 MMA, 2 posteriors, 3 none; 4..19 producers (4 groups); 20..27 flush (a group of 4 per pair)
constexpr int kSThreads = 28 * 32;
constexpr int kSProd0 = 4, kSFlush0 = 20;
// registers per thread after the split: 128 threads x 56 + 512 x 64 + 256 x 96 =
// 64512 = the launch's 896 x 72 (with 24, 72, 96 the MMA warp spills in its loop: N =
// 2^20, d = 64, K = 128 5.93 ms against 5.32; 40, 64, 104: 5.36)
constexpr int kSRegLaunch = 72, kSRegCtl = 56, kSRegProd = 64, kSRegFlush = 96;
static_assert(128 * kSRegCtl + 512 * kSRegProd + 256 * kSRegFlush <= kSThreads * kSRegLaunch, "register split");
static_assert(kSACol + kSA * kSAStage <= 512, "split covariance TMEM columns");
struct __align__(1024) SSmem {
  __half bh[kSIn][kSN * kBlk];                       // rows 0..63 xg^T (TMA, SW128), row 64 ones, 65..79 zero
  __half bl[kSIn][kD * kBlk], bm[kSIn][kD * kBlk];   // xr^T, xm^T
  float x[kSIn][kBlk * kD];                          // FP32 rows (TMA)
  __half rh[kSIn][4 * kBlk], rl[kSIn][4 * kBlk];     // posteriors of the CTA's 4 components
  float rf[kSIn][4 * kBlk];                          // hi + lo
  float mu[4][kD];                                   // means of the CTA's components in column units
  float zs[4][kD], zm[4][kD];                        // 1 / zunit, -mu / zunit
  uint64_t in_full[kSIn], rf_full[kSIn], in_empty[kSIn], a_full[kSA], a_empty[kSA], acc_full, acc_empty, cross_full,
      cross_empty, mma_done;
  uint32_t tmem_base;
};
static_assert(sizeof(SSmem) + 1024 <= 232448, "split covariance shared memory");

struct TcEmPlan {
  CUtensorMap tm_xh, tm_xl, tm_wh, tm_wl;      // E-step
  CUtensorMap tm_rh, tm_rl, tm_xht, tm_xlt;    // means
  CUtensorMap tm_xgt, tm_xrt, tm_xmt;          // split covariance
  CUtensorMap tm_x32, tm_rh4, tm_rl4;          // covariances
  __half *Wh = nullptr, *Wl = nullptr;  // (K*d) x d, permuted rows
  float *bias = nullptr;                // K*d, permuted
  float *clo = nullptr;                 // log coefficient - float(log coefficient)
  __half *Rh = nullptr, *Rl = nullptr;  // K x np posteriors hi / lo
  __half *XhT = nullptr, *XlT = nullptr;  // d x np: fp16(x) and the rest
  // split covariance only, d x np: x in units of its dimension (x_unit): nearest integer, rest, what FP16 leaves of it
  __half *XgT = nullptr, *XrT = nullptr, *XmT = nullptr;
  int64_t np = 0;                       // padded row pitch (multiple of 64)
  float *lsc = nullptr;                 // E-step scratch: egrid x 2 x K x 256
  double *epart = nullptr;              // per-CTA log-likelihood
  double *mpart = nullptr;              // means partials: mgrid x 80 columns x 128 components
  double *cpart = nullptr;              // covariance partials: cgrid x 2 pairs x 64 columns x 128 rows
  double *dpart = nullptr;              // exact diagonals: cgrid x 4 x 64
  float *muf = nullptr;                 // new means (float) for the covariance producers
  float *chi = nullptr;                 // float(log coefficient); -inf for padding components
  float *X64 = nullptr;                 // n x 64 zero-padded FP32 rows when d < 64
  int *err = nullptr;                   // device status of the bounded waits
  float *amax = nullptr;                // upload: largest |x| of every dimension (split covariance), then of all (FP16 range check)
  float *zunit = nullptr;               // split covariance: unit of z per component and dimension
  int *coarse = nullptr;                // split covariance: grids too coarse, [0] before the sums and [1] by their result
  int *roles = nullptr;                 // bounded-wait expiry self-test: which waits gave up
  int egrid = 0, mgrid = 0, cgx = 0, cgy = 0;
  int64_t srows = 0;                    // split form: rows per chunk (0: not used)
  int kp = 0, d = 0;                    // components padded to a multiple of 4; true dimension
};

__device__ __forceinline__ void fence_proxy_async_smem() {
  asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
}

__device__ __forceinline__ void store_post(__half *Rh, __half *Rl, size_t o, float r) {
  const __half h = __float2half_rn(r);
  Rh[o] = h;
  Rl[o] = __float2half_rn(r - __half2float(h));
}

__device__ __forceinline__ float2 f2(float x) { return make_float2(x, x); }

// The split covariance's columns of X^T are in units of a power of two, h = 2^(E -
// 10) with 2^E <= max |x| < 2^(E + 1) over the column: x = h (xg + xr + xm), xg an
// integer of at most 2^11 (exact in FP16), |xr| <= 1/2 in FP16, xm what is left.
// Products of xg with a weight on a grid add up exactly in FP32 while they stay
// below 2^24 units, where the tensor core's truncation of a floating split would
// cut every addition.  (xg + xr alone are exact to 2^-24 of the column's maximum
// only, so the forms that read two parts take fp16(x) and its rest, 2^-22 of x.)
__device__ __forceinline__ int x_unit_exp(float cmax) { return cmax > 0.f ? max(ilogbf(cmax), -110) - 10 : 0; }
__device__ __forceinline__ float x_unit(float cmax) { return ldexpf(1.f, x_unit_exp(cmax)); }

// unit of z = r (x - mu) in the split covariance: 2^-9 of the standard
// deviation that the E-step used (var: its covariance's diagonal entry), so
// most rows are integers below 2^11, but no less than keeps |z| <= 2 max|x|
// below 2^15 units whatever var says, and no more than 2^-9 of max |x|
__device__ __forceinline__ float z_unit(double var, float cmax) {
  const int lo = x_unit_exp(cmax) - 3;
  int e = lo;
  if (var > 1e-60 && var < 1e60) e = max(lo, min(ilogb(sqrt(var)) - 9, lo + 4));
  return ldexpf(1.f, e);
}

// The split covariance's grids against the standard deviation sd of a component's
// dimension: z has 2^-13 of its unit left out, the tensor core cuts sums that an
// offset makes large, and the unit follows the column's maximum.  Up to max |x| = 32
// sd and a unit of 2^-8 sd the split form is as exact as FP32 sums on CUDA cores,
// beyond that those are formed (rms error of Sigma_ab / (sd_a sd_b) against 64-bit
// sums, N = 2^18, d = 64, K = 128, split and CUDA cores: 1.7e-9 and 2.0e-9 at 12 sd,
// 2.4e-9 and 1.9e-9 at 37, 5.6e-9 and 1.8e-9 at 100, 2.4e-8 and 1.8e-9 at 340).
constexpr float kSRange = 32.f, kSUnits = 256.f;
__device__ __forceinline__ bool split_too_coarse(double var, float cmax, float zunit) {
  const float sd = (float)sqrt(var);
  return cmax > 0.f && !(cmax <= kSRange * sd && kSUnits * zunit <= sd);
}

// ============================================================== E-step
// MB = ceil(d / 16): only the 16-wide blocks of dimensions that exist are
// multiplied and read back. A group's accumulator columns run from the last
// block of outputs to the first, and the zero blocks of d < 64 would take as
// much of the tensor core and of the epilogue as real ones (GB300, N = 200003,
// K = 24 padded: d = 24 76.7 -> 61.0 us; N = 3001,
// K = 4: d = 5 6.9 -> 5.9 us).
template <int MB>
__global__ void __launch_bounds__(kEThreads, 1)
k_estep_tc(const __grid_constant__ CUtensorMap tm_xh, const __grid_constant__ CUtensorMap tm_xl,
           const __grid_constant__ CUtensorMap tm_wh, const __grid_constant__ CUtensorMap tm_wl,
           const float *__restrict__ bias, const float *__restrict__ chi, const float *__restrict__ clo,
           const double *__restrict__ c64, float *__restrict__ lsc, __half *__restrict__ Rh,
           __half *__restrict__ Rl, int64_t np, double *__restrict__ part, int64_t n, int K, int *err) {
  extern __shared__ uint8_t smem_raw[];
  ESmem &S = smem_aligned<ESmem>(smem_raw);
  constexpr int kCol0 = 32 * (kD / 16 - MB);        // first accumulator column and B row in use
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int G = K / kCompPerGroup;
  const int64_t ntiles = (n + kTileM - 1) / kTileM;
  const int64_t npairs = (ntiles + 1) / 2;

  for (int e = threadIdx.x; e < K * kD; e += blockDim.x) S.bias[e] = bias[e];
  for (int j = threadIdx.x; j < K; j += blockDim.x) S.chi[j] = chi[j], S.clo[j] = clo[j];
  if (threadIdx.x == 0) {
    mbar_init(&S.x_full, 1), mbar_init(&S.x_empty, 1);
    for (int s = 0; s < kWStages; s++) mbar_init(&S.w_full[s], 1), mbar_init(&S.w_empty[s], 1);
    for (int s = 0; s < 2; s++)
      for (int t = 0; t < 2; t++) mbar_init(&S.acc_full[s][t], 1), mbar_init(&S.acc_empty[s][t], 4);
    mbar_init(&S.mma_done, 1);
    fence_mbar_init();
  }
  if (warp == 1) tmem_alloc(&S.tmem_base, 512);
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tbase = S.tmem_base;

  if (warp == 0) {
    // ------------------------------------------------ TMA producer
    if (elect_one()) {
      tma_prefetch_desc(&tm_xh);
      tma_prefetch_desc(&tm_xl);
      tma_prefetch_desc(&tm_wh);
      tma_prefetch_desc(&tm_wl);
      uint32_t xi = 0, wi = 0;
      bool ok = true;
      for (int64_t pr = blockIdx.x; pr < npairs && ok; pr += gridDim.x) {
        if (!(ok = mbar_wait_lazy(&S.x_empty, (xi & 1) ^ 1, err, 128))) break;
        const bool has1 = 2 * pr + 1 < ntiles;
        mbar_expect_tx(&S.x_full, (has1 ? 4 : 2) * kXBytes);
        tma_load_2d(S.xh[0], &tm_xh, &S.x_full, 0, (int)(2 * pr * kTileM));
        tma_load_2d(S.xl[0], &tm_xl, &S.x_full, 0, (int)(2 * pr * kTileM));
        if (has1) {
          tma_load_2d(S.xh[1], &tm_xh, &S.x_full, 0, (int)((2 * pr + 1) * kTileM));
          tma_load_2d(S.xl[1], &tm_xl, &S.x_full, 0, (int)((2 * pr + 1) * kTileM));
        }
        xi++;
        for (int g = 0; g < G; g++) {
          const int ws = wi % kWStages;
          if (!(ok = mbar_wait_lazy(&S.w_empty[ws], ((wi / kWStages) & 1) ^ 1, err, 128))) break;
          mbar_expect_tx(&S.w_full[ws], 2 * kWBytes);
          tma_load_2d(S.wh[ws], &tm_wh, &S.w_full[ws], 0, g * kGroupN);
          tma_load_2d(S.wl[ws], &tm_wl, &S.w_full[ws], 0, g * kGroupN);
          wi++;
        }
      }
      // drain: the last loads must land before the CTA may exit
      if (xi > 0) mbar_wait_drain(&S.x_full, (xi - 1) & 1);
      for (int s = 0; s < kWStages && wi > (uint32_t)s; s++) {
        const uint32_t u = wi - 1 - s;
        mbar_wait_drain(&S.w_full[u % kWStages], (u / kWStages) & 1);
      }
    }
  } else if (warp == 1) {
    // ------------------------------------------------ MMA issuer
    if (elect_one()) {
      uint32_t xi = 0, wi = 0, ai = 0;
      bool ok = true;
      for (int64_t pr = blockIdx.x; pr < npairs && ok; pr += gridDim.x) {
        if (!(ok = mbar_wait(&S.x_full, xi & 1, err))) break;
        tc_fence_after();
        const int nt = (2 * pr + 1 < ntiles) ? 2 : 1;
        uint64_t dxh[2], dxl[2];
        for (int t = 0; t < 2; t++) {
          dxh[t] = sdesc_sw128(smem_u32(S.xh[t]));
          dxl[t] = sdesc_sw128(smem_u32(S.xl[t]));
        }
        for (int g = 0; g < G; g++) {
          const int ws = wi % kWStages, ab = ai & 1;
          if (!(ok = mbar_wait(&S.w_full[ws], (wi / kWStages) & 1, err))) break;
          const uint64_t dwh = sdesc_sw128(smem_u32(S.wh[ws]));
          const uint64_t dwl = sdesc_sw128(smem_u32(S.wl[ws]));
          // each tile has its own accumulator barriers, so its epilogue warps
          // start as soon as its own products are done; a pair with one tile
          // still completes the second tile's phases (no products)
          for (int t = 0; t < 2; t++) {
            if (!(ok = mbar_wait(&S.acc_empty[ab][t], ((ai >> 1) & 1) ^ 1, err))) break;
            tc_fence_after();
            if (t < nt) {
              const uint32_t dt = tbase + (2 * ab + t) * kGroupN;
              // the small cross products Xh Wl and Xl Wh first, Xh Wh last: the
              // accumulator is rounded after every MMA, and it only grows to
              // |W x| during the final four steps
#pragma unroll
              for (int p = 0; p < 3; p++) {
                const uint64_t da = (p == 1) ? dxl[t] : dxh[t];
                const uint64_t db = (p == 0) ? dwl : dwh;
#pragma unroll
                for (int kb = 0; kb < MB; kb++) {
                  // +32 bytes per 16-element K step inside the 128-byte swizzle row
                  mma_f16(dt + kCol0, da + 2 * kb, db + kCol0 * 8 + 2 * kb, idesc_f16(kTileM, 32 * (MB - kb)),
                          (p | kb) != 0);
                }
              }
            }
            mma_commit(&S.acc_full[ab][t]);
          }
          if (!ok) break;
          mma_commit(&S.w_empty[ws]);
          wi++;
          ai++;
        }
        if (!ok) break;
        mma_commit(&S.x_empty);
        xi++;
      }
      // every MMA issued must complete before TMEM is released
      mma_commit(&S.mma_done);
      mbar_wait_drain(&S.mma_done, 0);
    }
  } else {
    // ------------------------------------------------ epilogue
    // 8 warps: warp w reads TMEM lanes 32 (w % 4) .. +31 of tile (w - 2) / 4
    const int quad = warp & 3;
    const int tile = (warp - 2) >> 2;
    const int row = quad * 32 + lane;
    const int prow = tile * kTileM + row;                 // point within the pair
    const uint32_t lane_addr = (uint32_t)(quad * 32) << 16;
    // l_ij scratch of this CTA: [pair parity][component][256 points of the pair]
    float *scr = lsc + (size_t)blockIdx.x * 2 * K * (2 * kTileM) + prow;
    double lsum = 0.0;
    bool ok = true;
    bool have_prev = false;
    int prev_par = 0;
    int64_t prev_i = -1;
    float prev_lse = 0.f;
    uint32_t ai = 0;
    int pc = 0;
    for (int64_t pr = blockIdx.x; pr < npairs && ok; pr += gridDim.x, pc++) {
      const int par = pc & 1;
      const bool live = tile < ((2 * pr + 1 < ntiles) ? 2 : 1);   // warp-uniform
      const int64_t pi = (live && (2 * pr + tile) * kTileM + row < n) ? (2 * pr + tile) * kTileM + row : -1;
      float mx = -INFINITY, se = 0.f, smax = 0.f;
      int jmax = 0;
      for (int g = 0; g < G; g++) {
        // posteriors of components 2g, 2g+1 of the previous pair: load early
        float lp[2] = {0.f, 0.f};
        if (have_prev && prev_i >= 0) {
#pragma unroll
          for (int q = 0; q < 2; q++) lp[q] = scr[(size_t)(prev_par * K + 2 * g + q) * (2 * kTileM)];
        }
        const int ab = ai & 1;
        if (!(ok = mbar_wait_warp(&S.acc_full[ab][tile], (ai >> 1) & 1, err))) break;
        tc_fence_after();
        float s[kCompPerGroup] = {0.f, 0.f};
        if (live) {
          const float *bg = S.bias + g * kGroupN;
          // 32-column block bp holds k-block (3 - bp) of both components:
          // column 32 bp + 16 q + t belongs to component q; 64-column loads
          // (32 first for an odd MB), column pairs in packed FP32 arithmetic
          float2 s2[kCompPerGroup] = {make_float2(0.f, 0.f), make_float2(0.f, 0.f)};
          auto add = [&](auto &v, int c0) {
            const float4 *b4 = reinterpret_cast<const float4 *>(bg + c0);
#pragma unroll
            for (int u = 0; u < (int)(sizeof(v) / 16); u++) {
              const float4 b = b4[u];
              const int q = (u >> 2) & 1;         // columns 4u .. 4u + 3
              const float2 y0 = __fadd2_rn(make_float2(__uint_as_float(v[4 * u]), __uint_as_float(v[4 * u + 1])),
                                           make_float2(-b.x, -b.y));
              const float2 y1 = __fadd2_rn(make_float2(__uint_as_float(v[4 * u + 2]), __uint_as_float(v[4 * u + 3])),
                                           make_float2(-b.z, -b.w));
              s2[q] = __ffma2_rn(y0, y0, s2[q]);
              s2[q] = __ffma2_rn(y1, y1, s2[q]);
            }
          };
          const uint32_t ta = tbase + lane_addr + (2 * ab + tile) * kGroupN;
          if constexpr (MB & 1) {
            uint32_t v[32];
            tmem_ld32(ta + kCol0, v);
            tmem_wait_ld();
            add(v, kCol0);
          }
#pragma unroll 1
          for (int c0 = kCol0 + 32 * (MB & 1); c0 < kGroupN; c0 += 64) {
            uint32_t v[64];
            tmem_ld64(ta + c0, v);
            tmem_wait_ld();
            add(v, c0);
          }
          s[0] = s2[0].x + s2[0].y;
          s[1] = s2[1].x + s2[1].y;
        }
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(&S.acc_empty[ab][tile]);
        ai++;
        if (have_prev && prev_i >= 0) {
#pragma unroll
          for (int q = 0; q < 2; q++) store_post(Rh, Rl, (size_t)(2 * g + q) * np + prev_i, expf(lp[q] - prev_lse));
        }
        if (live) {
#pragma unroll
          for (int q = 0; q < kCompPerGroup; q++) {
            const int j = g * kCompPerGroup + q;
            // c_j carried as float hi + lo: its rounding would shift every
            // posterior of component j by the same factor
            const float l = (S.chi[j] - 0.5f * s[q]) + S.clo[j];
            scr[(size_t)(par * K + j) * (2 * kTileM)] = l;
            if (l > mx) {
              se = se * __expf(mx - l) + 1.f;
              mx = l;
              jmax = j;
              smax = s[q];
            } else if (l > -INFINITY) {
              se += __expf(l - mx);
            }
          }
        }
      }
      if (!ok) break;
      prev_i = pi;
      prev_lse = mx + __logf(se);
      if (pi >= 0) lsum += c64[jmax] - 0.5 * (double)smax + (double)__logf(se);
      prev_par = par;
      have_prev = true;
    }
    // posteriors of the last pair
    if (ok && have_prev && prev_i >= 0) {
      for (int j0 = 0; j0 < K; j0 += 8) {
        float l8[8];
#pragma unroll
        for (int u = 0; u < 8; u++)
          l8[u] = (j0 + u < K) ? scr[(size_t)(prev_par * K + j0 + u) * (2 * kTileM)] : 0.f;
#pragma unroll
        for (int u = 0; u < 8; u++)
          if (j0 + u < K) store_post(Rh, Rl, (size_t)(j0 + u) * np + prev_i, expf(l8[u] - prev_lse));
      }
    }
    // deterministic reduction over the 256 epilogue threads
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) lsum += __shfl_down_sync(0xffffffffu, lsum, o);
    if (lane == 0) S.red[warp - 2] = lsum;
    asm volatile("bar.sync 1, 256;" ::: "memory");
    if (threadIdx.x == 64) {
      double t = 0.0;
      for (int w = 0; w < 8; w++) t += S.red[w];
      part[blockIdx.x] = t;
    }
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  if (warp == 1) tmem_dealloc(tbase, 512);
}

// =============================================================== means
// Per 64-point block: D[128 comps x 80] += Rh Bh^T + Rh Bl^T + Rl Bh^T with
// B rows 0..63 = X^T (hi / lo) and row 64 of Bh = 1 (gives sum_i r_ij).
// Four epilogue warps flush the FP32 accumulator to FP64 partials every
// kFlushBlocks blocks (double-buffered TMEM, 2 x 128 columns).
__global__ void __launch_bounds__(192, 1)
k_means_tc(const __grid_constant__ CUtensorMap tm_rh, const __grid_constant__ CUtensorMap tm_rl,
           const __grid_constant__ CUtensorMap tm_xht, const __grid_constant__ CUtensorMap tm_xlt,
           int64_t n, double *__restrict__ part, int *coarse, int *err) {
  extern __shared__ uint8_t smem_raw[];
  if (blockIdx.x == 0 && threadIdx.x < 2) coarse[threadIdx.x] = 0;   // this M-step's
  MSmem &S = smem_aligned<MSmem>(smem_raw);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int64_t nblocks = (n + kBlk - 1) / kBlk;
  // blocks of this CTA: b = blockIdx.x + t * gridDim.x, t < mine
  const int64_t mine = nblocks > blockIdx.x ? (nblocks - 1 - blockIdx.x) / gridDim.x + 1 : 0;
  const int64_t nwin = (mine + kFlushBlocks - 1) / kFlushBlocks;

  // constant rows 64..79 of the B tiles (row 64 of Bh = ones; the rest zero);
  // rows of 128 bytes, 16-byte chunk c of row r stored at c ^ (r & 7)
  for (int e = threadIdx.x; e < kMStages * 16 * kBlk; e += blockDim.x) {
    const int s = e / (16 * kBlk), rem = e - s * 16 * kBlk;
    const int r = 64 + rem / kBlk, col = rem % kBlk;   // logical (row, point)
    const int phys = r * kBlk + (((col >> 3) ^ (r & 7)) << 3) + (col & 7);
    S.bh[s][phys] = __float2half(r == 64 ? 1.f : 0.f);
    S.bl[s][phys] = __float2half(0.f);
  }
  fence_proxy_async_smem();
  if (threadIdx.x == 0) {
    for (int s = 0; s < kMStages; s++) mbar_init(&S.in_full[s], 1), mbar_init(&S.in_empty[s], 1);
    for (int s = 0; s < 2; s++) mbar_init(&S.acc_full[s], 1), mbar_init(&S.acc_empty[s], 4);
    mbar_init(&S.mma_done, 1);
    fence_mbar_init();
  }
  if (warp == 1) tmem_alloc(&S.tmem_base, 256);
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tbase = S.tmem_base;
  constexpr uint32_t kInBytes = 2 * kMaxK * kBlk * 2 + 2 * kD * kBlk * 2;

  if (warp == 0) {
    if (elect_one()) {
      bool ok = true;
      for (int64_t t = 0; t < mine && ok; t++) {
        const int s = (int)(t % kMStages);
        if (!(ok = mbar_wait_lazy(&S.in_empty[s], ((t / kMStages) & 1) ^ 1, err, 128))) break;
        const int p0 = (int)((blockIdx.x + t * gridDim.x) * kBlk);
        mbar_expect_tx(&S.in_full[s], kInBytes);
        tma_load_2d(S.rh[s], &tm_rh, &S.in_full[s], p0, 0);
        tma_load_2d(S.rl[s], &tm_rl, &S.in_full[s], p0, 0);
        tma_load_2d(S.bh[s], &tm_xht, &S.in_full[s], p0, 0);
        tma_load_2d(S.bl[s], &tm_xlt, &S.in_full[s], p0, 0);
      }
      for (int64_t u = mine - 1; u >= 0 && u >= mine - kMStages; u--)
        mbar_wait_drain(&S.in_full[u % kMStages], (u / kMStages) & 1);
    }
  } else if (warp == 1) {
    if (elect_one()) {
      bool ok = true;
      for (int64_t w = 0; w < nwin && ok; w++) {
        const int ab = w & 1;
        if (!(ok = mbar_wait(&S.acc_empty[ab], ((w >> 1) & 1) ^ 1, err))) break;
        const int64_t t1 = std::min<int64_t>(mine, (w + 1) * kFlushBlocks);
        for (int64_t t = w * kFlushBlocks; t < t1; t++) {
          const int s = (int)(t % kMStages);
          if (!(ok = mbar_wait(&S.in_full[s], (t / kMStages) & 1, err))) break;
          tc_fence_after();
          const uint64_t drh = sdesc_sw128(smem_u32(S.rh[s])), drl = sdesc_sw128(smem_u32(S.rl[s]));
          const uint64_t dbh = sdesc_sw128(smem_u32(S.bh[s])), dbl = sdesc_sw128(smem_u32(S.bl[s]));
#pragma unroll
          for (int p = 0; p < 3; p++) {
            const uint64_t da = (p == 2) ? drl : drh;
            const uint64_t db = (p == 1) ? dbl : dbh;
#pragma unroll
            for (int kb = 0; kb < kBlk / 16; kb++)
              mma_f16(tbase + ab * 128, da + 2 * kb, db + 2 * kb, idesc_f16(128, kMeanN),
                      (t != w * kFlushBlocks) || p || kb);
          }
          mma_commit(&S.in_empty[s]);
        }
        if (!ok) break;
        mma_commit(&S.acc_full[ab]);
      }
      mma_commit(&S.mma_done);
      mbar_wait_drain(&S.mma_done, 0);
    }
  } else {
    // flush: lane row = component; 80 columns -> this CTA's FP64 partial,
    // column-major (column c of component comp at o[c * kMaxK]) so a warp's
    // 32 components are 256 contiguous bytes
    const int quad = warp & 3;
    const int comp = quad * 32 + lane;
    double *o = part + (size_t)blockIdx.x * kMaxK * kMeanN + comp;
    for (int c = 0; c < kMeanN; c++) o[(size_t)c * kMaxK] = 0.0;
    bool ok = true;
    for (int64_t w = 0; w < nwin && ok; w++) {
      const int ab = w & 1;
      if (!(ok = mbar_wait_lazy_warp(&S.acc_full[ab], (w >> 1) & 1, err, 1000))) break;
      tc_fence_after();
      const uint32_t ta = tbase + ((uint32_t)(quad * 32) << 16) + ab * 128;
#pragma unroll 1
      for (int c0 = 0; c0 < 96; c0 += 32) {   // columns 80..95 are not used
        uint32_t v[32];
        tmem_ld32(ta + c0, v);
        tmem_wait_ld();
#pragma unroll
        for (int c = 0; c < 32; c++)
          if (c0 + c < kMeanN) o[(size_t)(c0 + c) * kMaxK] += (double)__uint_as_float(v[c]);
      }
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(&S.acc_empty[ab]);
    }
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  if (warp == 1) tmem_dealloc(tbase, 256);
}

// S1 = sum r, mu = S2 / S1, pi = S1 / N (FP64), and the units of the split
// covariance from the E-step's covariances.  One CTA per component; the
// CTAs' partials are split over its 4 thread sets (65 threads each: column 64
// holds S1) and combined in order
constexpr int kFMSplit = 4, kFMCols = kD + 1;
__global__ void __launch_bounds__(kFMSplit * kFMCols)
k_final_means_tc(const double *__restrict__ part, int G, int K, int d, int64_t n, double *__restrict__ mu,
                 double *__restrict__ pi, double *__restrict__ psum, float *__restrict__ muf,
                 const float *__restrict__ cmax, const double *__restrict__ sigma, float *__restrict__ zunit,
                 int *__restrict__ coarse) {
  const int j = blockIdx.x, q = threadIdx.x % kFMCols, w = threadIdx.x / kFMCols;
  __shared__ double red[kFMSplit][kFMCols];
  double s = 0.0;
#pragma unroll 8
  for (int g = w; g < G; g += kFMSplit) s += part[((size_t)g * kMeanN + q) * kMaxK + j];
  red[w][q] = s;
  __syncthreads();
  if (w) return;
  double s1 = 0.0;
#pragma unroll
  for (int u = 0; u < kFMSplit; u++) s1 += red[u][kD];
  if (q == kD) {
    psum[j] = s1;
    pi[j] = s1 / (double)n;
    return;
  }
#pragma unroll
  for (int u = 1; u < kFMSplit; u++) s += red[u][q];
  const double m = s / s1;
  if (q < d) mu[(size_t)j * d + q] = m;
  muf[(size_t)j * kD + q] = q < d ? (float)m : 0.f;
  const double var = q < d ? sigma[((size_t)j * d + q) * d + q] : 1.0;
  const float zu = q < d ? z_unit(var, cmax[q]) : 1.f;
  zunit[(size_t)j * kD + q] = zu;
  if (q < d && split_too_coarse(var, cmax[q], zu)) coarse[0] = 1;
}

// ========================================================= covariances
// CTA (blockIdx.x = group of 4 components, blockIdx.y = chunk of points).
// Producers (warps 2..17) form two groups of eight that take alternate
// blocks.  Warp c8 of a group owns the block's points 8 c8 .. 8 c8 + 7; lane a
// owns dimensions a and a + 32 (32 apart, so the eight rows a phase of a
// 16-byte store touches fall in eight different swizzle chunks).  For each of
// the 4 components q a thread writes z = sqrt(r) (x - mu) of its 8 points as
// one 16-byte store into rows (q % 2) * 64 + a (+ 32) of pair q / 2's operand
// tile and sums z^2 in FP32 / FP64 for the exact diagonal.
__global__ void __launch_bounds__(kCThreads, 1)
k_cov_tc(const __grid_constant__ CUtensorMap tm_x32, const __grid_constant__ CUtensorMap tm_rh4,
         const __grid_constant__ CUtensorMap tm_rl4, const float *__restrict__ muf, int64_t n,
         int64_t blocks_per_chunk, double *__restrict__ cpart, double *__restrict__ dpart, int *err) {
  extern __shared__ uint8_t smem_raw[];
  CSmem &S = smem_aligned<CSmem>(smem_raw);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int cg = blockIdx.x;                  // component group (4 components)
  const int64_t nblocks = (n + kBlk - 1) / kBlk;
  const int64_t b0 = (int64_t)blockIdx.y * blocks_per_chunk;
  const int64_t mine = std::max<int64_t>(0, std::min<int64_t>(nblocks, b0 + blocks_per_chunk) - b0);
  const int64_t nwin = (mine + kFlushBlocks - 1) / kFlushBlocks;
  const size_t cta = (size_t)blockIdx.y * gridDim.x + blockIdx.x;

  if (threadIdx.x == 0) {
    // each block is produced by one group of kCProd / 2 warps
    for (int s = 0; s < kCIn; s++) mbar_init(&S.in_full[s], 1), mbar_init(&S.in_empty[s], kCProd / 2);
    for (int s = 0; s < kZStages; s++) mbar_init(&S.z_full[s], kCProd / 2), mbar_init(&S.z_empty[s], 1);
    for (int s = 0; s < 2; s++) mbar_init(&S.acc_full[s], 1), mbar_init(&S.acc_empty[s], 4);
    mbar_init(&S.mma_done, 1);
    fence_mbar_init();
  }
  if (warp == 1) tmem_alloc(&S.tmem_base, 512);
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tbase = S.tmem_base;
  constexpr uint32_t kInBytes = kBlk * kD * 4 + 2 * 4 * kBlk * 2;

  if (warp == 0) {
    if (elect_one()) {
      bool ok = true;
      for (int64_t t = 0; t < mine && ok; t++) {
        const int s = (int)(t % kCIn);
        if (!(ok = mbar_wait_lazy(&S.in_empty[s], ((t / kCIn) & 1) ^ 1, err, 128))) break;
        const int p0 = (int)((b0 + t) * kBlk);
        mbar_expect_tx(&S.in_full[s], kInBytes);
        tma_load_2d(S.xs[s], &tm_x32, &S.in_full[s], 0, p0);
        tma_load_2d(S.rh[s], &tm_rh4, &S.in_full[s], p0, cg * 4);
        tma_load_2d(S.rl[s], &tm_rl4, &S.in_full[s], p0, cg * 4);
      }
      for (int64_t u = mine - 1; u >= 0 && u >= mine - kCIn; u--)
        mbar_wait_drain(&S.in_full[u % kCIn], (u / kCIn) & 1);
    }
  } else if (warp == 1) {
    if (elect_one()) {
      bool ok = true;
      constexpr uint32_t idesc = idesc_f16(128, 128);
      for (int64_t w = 0; w < nwin && ok; w++) {
        const int ab = w & 1;
        if (!(ok = mbar_wait(&S.acc_empty[ab], ((w >> 1) & 1) ^ 1, err))) break;
        const int64_t t1 = std::min<int64_t>(mine, (w + 1) * kFlushBlocks);
        for (int64_t t = w * kFlushBlocks; t < t1; t++) {
          const int s = (int)(t % kZStages);
          if (!(ok = mbar_wait(&S.z_full[s], (t / kZStages) & 1, err))) break;
          tc_fence_after();
#pragma unroll
          for (int pr = 0; pr < 2; pr++) {
            const uint64_t dz = sdesc_sw128(smem_u32(S.z[s][pr]));
#pragma unroll
            for (int kb = 0; kb < kBlk / 16; kb++)
              mma_f16(tbase + ab * 256 + pr * 128, dz + 2 * kb, dz + 2 * kb, idesc,
                      (t != w * kFlushBlocks) || kb);
          }
          mma_commit(&S.z_empty[s]);
        }
        if (!ok) break;
        mma_commit(&S.acc_full[ab]);
      }
      mma_commit(&S.mma_done);
      mbar_wait_drain(&S.mma_done, 0);
    }
  } else if (warp < 2 + kCProd) {
    // ------------------------------------------------ producers
    const int pw = warp - 2, grp = pw >> 3, c8 = pw & 7;
    const int a = lane;                          // dimensions a and a + 32
    float *srw = S.sr[pw];
    float2 nmu[4][2];
#pragma unroll
    for (int q = 0; q < 4; q++)
#pragma unroll
      for (int h = 0; h < 2; h++) {
        const float m = muf[(size_t)(cg * 4 + q) * kD + a + 32 * h];
        nmu[q][h] = make_float2(-m, -m);
      }
    double diag[4][2];
    float2 dwin[4][2];
#pragma unroll
    for (int q = 0; q < 4; q++)
#pragma unroll
      for (int h = 0; h < 2; h++) diag[q][h] = 0.0, dwin[q][h] = make_float2(0.f, 0.f);
    bool ok = true;
    int li = 0;                                  // blocks this group has produced
    for (int64_t tb = grp; tb < mine && ok; tb += 2, li++) {
      const int si = (int)(tb % kCIn), sz = (int)(tb % kZStages);
      if (!(ok = mbar_wait_warp(&S.in_full[si], (tb / kCIn) & 1, err))) break;
      {
        // lane -> component lane / 8, point c8 * 8 + lane % 8; rows past N
        // read zero-filled r and x, and get s = 0 besides
        const int q = lane >> 3, p = c8 * 8 + (lane & 7);
        const float r = __half2float(S.rh[si][q * kBlk + p]) + __half2float(S.rl[si][q * kBlk + p]);
        const float sv = ((b0 + tb) * kBlk + p < n) ? sqrtf(r) : 0.f;
        __syncwarp();                           // the previous block's reads of the slot are done
        srw[lane] = sv;
        __syncwarp();
      }
      const float *xr = S.xs[si] + (c8 * 8) * kD + a;
      float2 xv[2][4];                           // [dimension a / a + 32][point pair]
#pragma unroll
      for (int h = 0; h < 2; h++)
#pragma unroll
        for (int u = 0; u < 4; u++) xv[h][u] = make_float2(xr[(2 * u) * kD + 32 * h], xr[(2 * u + 1) * kD + 32 * h]);
      if (!(ok = mbar_wait_warp(&S.z_empty[sz], ((tb / kZStages) & 1) ^ 1, err))) break;
#pragma unroll
      for (int q = 0; q < 4; q++) {
        const float4 s0 = *reinterpret_cast<const float4 *>(srw + q * 8);
        const float4 s1 = *reinterpret_cast<const float4 *>(srw + q * 8 + 4);
        const float2 s2[4] = {make_float2(s0.x, s0.y), make_float2(s0.z, s0.w), make_float2(s1.x, s1.y),
                              make_float2(s1.z, s1.w)};
#pragma unroll
        for (int h = 0; h < 2; h++) {
          uint32_t w4[4];
#pragma unroll
          for (int u = 0; u < 4; u++) {
            const float2 z = __fmul2_rn(__fadd2_rn(xv[h][u], nmu[q][h]), s2[u]);
            dwin[q][h] = __ffma2_rn(z, z, dwin[q][h]);
            const __half2 hz = __floats2half2_rn(z.x, z.y);
            w4[u] = *reinterpret_cast<const uint32_t *>(&hz);
          }
          const int row = ((q & 1) << 6) + a + 32 * h;
          uint8_t *zrow = reinterpret_cast<uint8_t *>(S.z[sz][q >> 1]) + row * 128;
          *reinterpret_cast<uint4 *>(zrow + ((c8 ^ (row & 7)) << 4)) = make_uint4(w4[0], w4[1], w4[2], w4[3]);
        }
      }
      fence_proxy_async_smem();
      __syncwarp();
      if (lane == 0) {
        mbar_arrive(&S.z_full[sz]);
        mbar_arrive(&S.in_empty[si]);
      }
      if ((li + 1) % (kFlushBlocks / 2) == 0) {
#pragma unroll
        for (int q = 0; q < 4; q++)
#pragma unroll
          for (int h = 0; h < 2; h++)
            diag[q][h] += (double)dwin[q][h].x + (double)dwin[q][h].y, dwin[q][h] = make_float2(0.f, 0.f);
      }
    }
#pragma unroll
    for (int q = 0; q < 4; q++)
#pragma unroll
      for (int h = 0; h < 2; h++) diag[q][h] += (double)dwin[q][h].x + (double)dwin[q][h].y;
    // exact diagonal: group 0, then group 1 added, then the 8 point chunks in order
    if (grp == 0)
#pragma unroll
      for (int q = 0; q < 4; q++)
#pragma unroll
        for (int h = 0; h < 2; h++) S.dred[c8][q][a + 32 * h] = diag[q][h];
    asm volatile("bar.sync 2, %0;" ::"n"(kCProd * 32) : "memory");
    if (grp == 1)
#pragma unroll
      for (int q = 0; q < 4; q++)
#pragma unroll
        for (int h = 0; h < 2; h++) S.dred[c8][q][a + 32 * h] += diag[q][h];
    asm volatile("bar.sync 2, %0;" ::"n"(kCProd * 32) : "memory");
    if (grp == 0 && c8 == 0)
#pragma unroll
      for (int q = 0; q < 4; q++)
#pragma unroll
        for (int h = 0; h < 2; h++) {
          double v = S.dred[0][q][a + 32 * h];
          for (int c = 1; c < 8; c++) v += S.dred[c][q][a + 32 * h];
          dpart[(cta * 4 + q) * kD + a + 32 * h] = v;
        }
  } else {
    // ------------------------------------------------ flush warps 18..21
    const int quad = warp & 3;
    const int lrow = quad * 32 + lane;          // TMEM lane = row of the pair tile
    const int half = lrow >> 6;                 // 0: first component of the pair, 1: second
    // this CTA's FP64 partials, column-major per pair: column c of pair pr at
    // o[pr][c * 128] (row lrow), so a warp's 32 rows are 256 contiguous bytes
    double *o[2];
#pragma unroll
    for (int pr = 0; pr < 2; pr++) {
      o[pr] = cpart + (cta * 2 + pr) * (size_t)(kD * 128) + lrow;
      for (int c = 0; c < kD; c++) o[pr][(size_t)c * 128] = 0.0;
    }
    bool ok = true;
    for (int64_t w = 0; w < nwin && ok; w++) {
      const int ab = w & 1;
      if (!(ok = mbar_wait_lazy_warp(&S.acc_full[ab], (w >> 1) & 1, err, 1000))) break;
      tc_fence_after();
#pragma unroll
      for (int pr = 0; pr < 2; pr++) {
#pragma unroll 1
        for (int c0 = 0; c0 < kD; c0 += 32) {   // 32-column chunks
          uint32_t v[32];
          tmem_ld32(tbase + ((uint32_t)(quad * 32) << 16) + ab * 256 + pr * 128 + half * 64 + c0, v);
          tmem_wait_ld();
#pragma unroll
          for (int c = 0; c < 32; c++) o[pr][(size_t)(c0 + c) * 128] += (double)__uint_as_float(v[c]);
        }
      }
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(&S.acc_empty[ab]);
    }
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  if (warp == 1) tmem_dealloc(tbase, 512);
}

// Covs_j = sym(S3_j) / S1_j with the exact diagonal (FP64, chunks in order)
__global__ void k_final_cov_tc(const double *__restrict__ cpart, const double *__restrict__ dpart, int gx,
                               int gy, int d, const double *__restrict__ psum, double *__restrict__ sigma) {
  const int j = blockIdx.x, grp = j / 4, q = j % 4;
  const double inv = 1.0 / psum[j];
  double *Sg = sigma + (size_t)j * d * d;
  for (int e = threadIdx.x; e < d * d; e += blockDim.x) {
    const int a = e / d, b = e - a * d;
    if (b < a) continue;
    double s = 0.0;
    if (a == b) {
      for (int c = 0; c < gy; c++) s += dpart[(((size_t)c * gx + grp) * 4 + q) * kD + a];
    } else {
      // partials of CTA (chunk c, group grp): pair q / 2, rows (q % 2) * 64 + row, column-major
      for (int c = 0; c < gy; c++) {
        const double *P = cpart + (((size_t)c * gx + grp) * 2 + (q >> 1)) * (kD * 128) + (q & 1) * 64;
        s += 0.5 * (P[(size_t)b * 128 + a] + P[(size_t)a * 128 + b]);
      }
    }
    s *= inv;
    Sg[a * d + b] = s;
    Sg[b * d + a] = s;
  }
}

// ====================================================== covariances (z x^T)
// Sigma_j N_j = sum_i r_ij (x_i - mu_j)(x_i - mu_j)^T  (ComputeWeightedTempDataset
// + BlockCovariances, EM2/MatrixEM.cpp:53-67,90-99), around the NEW means, as
//   sum_i z_i x_i^T - (sum_i z_i) mu_j^T,   z_i = r_ij (x_i - mu_j),
// with x = xh + xl (the FP16 split of X) on the B side, shared by every
// component: the per-component operand z is formed once per (point,
// component) by CUDA cores and written straight into tensor memory as the A
// operand of an M = 128 (two components x 64 dimensions) MMA; B = [Xh^T; 1]
// (N = 80, the ones row gives sum z in column 64) and Xl^T (N = 64) come from
// global memory by TMA.  Every output element of an MMA is wanted (no
// cross-component blocks), and the subtraction of (sum z) mu^T uses the sums
// of the ROUNDED z, so FP16 rounding of z enters only as sum delta_i (x_i -
// mu)^T: unbiased, centred, no diagonal correction needed.
//
// CTA (blockIdx.x = group of 4 components = 2 pairs, blockIdx.y = chunk of
// 64-point blocks).  Warp 0: TMA; warp 1: MMA; warps 2..2+4 kZSets-1:
// producers in groups of 4 (group = (warp - 2) / 4; kZSplit groups share a
// block, each forming its own K steps, and the kZSets / kZSplit teams take
// alternate blocks, so a block's operand is ready after a fraction of one
// warp's work); a warp writes the TMEM lanes 32 (warp % 4) .. +31: dimension
// 32 (warp & 1) + lane of the component in slot (warp & 3) / 2 of both pairs.
// The last 4 warps flush the FP32 accumulators to FP64 partials every
// kFlushBlocks blocks (double buffered in TMEM).
__global__ void __launch_bounds__(kZThreads, 1)
k_cov_zx(const __grid_constant__ CUtensorMap tm_xht, const __grid_constant__ CUtensorMap tm_xlt,
         const __grid_constant__ CUtensorMap tm_rh4, const float *__restrict__ muf, int64_t n,
         int64_t blocks_per_chunk, double *__restrict__ cpart, int *err) {
  extern __shared__ uint8_t smem_raw[];
  ZSmem &S = smem_aligned<ZSmem>(smem_raw);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int cg = blockIdx.x;
  const int64_t nblocks = (n + kBlk - 1) / kBlk;
  const int64_t b0 = (int64_t)blockIdx.y * blocks_per_chunk;
  const int64_t mine = std::max<int64_t>(0, std::min<int64_t>(nblocks, b0 + blocks_per_chunk) - b0);
  const int64_t nwin = (mine + kFlushBlocks - 1) / kFlushBlocks;
  const size_t cta = (size_t)blockIdx.y * gridDim.x + blockIdx.x;

  // constant rows 64..79 of the Bh stages (row 64 ones, the rest zero);
  // 16-byte chunk c of row r stored at c ^ (r & 7)
  for (int e = threadIdx.x; e < kZIn * 16 * kBlk; e += blockDim.x) {
    const int st = e / (16 * kBlk), rem = e - st * 16 * kBlk;
    const int r = 64 + rem / kBlk, col = rem % kBlk;
    S.bh[st][r * kBlk + (((col >> 3) ^ (r & 7)) << 3) + (col & 7)] = __float2half(r == 64 ? 1.f : 0.f);
  }
  fence_proxy_async_smem();
  if (threadIdx.x == 0) {
    // a block is read by the MMA and by the kZSplit * 4 producer warps that form its operand
    for (int st = 0; st < kZIn; st++) mbar_init(&S.in_full[st], 1), mbar_init(&S.in_empty[st], 4 * kZSplit + 1);
    for (int st = 0; st < kZA; st++) mbar_init(&S.a_full[st], 4 * kZSplit), mbar_init(&S.a_empty[st], 1);
    for (int b = 0; b < 2; b++) mbar_init(&S.acc_full[b], 1), mbar_init(&S.acc_empty[b], 4);
    mbar_init(&S.mma_done, 1);
    fence_mbar_init();
  }
  if (warp == 1) tmem_alloc(&S.tmem_base, 512);
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tbase = S.tmem_base;
  constexpr uint32_t kInBytes = 2 * kD * kBlk * 2 + 4 * kBlk * 2;

  if (warp == 0) {
    // ------------------------------------------------ TMA
    if (elect_one()) {
      bool ok = true;
      for (int64_t t = 0; t < mine && ok; t++) {
        const int st = (int)(t % kZIn);
        if (!(ok = mbar_wait_lazy(&S.in_empty[st], ((t / kZIn) & 1) ^ 1, err, 128))) break;
        // CTAs of the same point chunk (one per component group) start kZStagger
        // blocks apart, so they do not all request the same tile at once
        const int64_t tb = (t + (int64_t)cg * kZStagger) % mine;
        const int p0 = (int)((b0 + tb) * kBlk);
        mbar_expect_tx(&S.in_full[st], kInBytes);
        tma_load_2d(S.bh[st], &tm_xht, &S.in_full[st], p0, 0);
        tma_load_2d(S.bl[st], &tm_xlt, &S.in_full[st], p0, 0);
        tma_load_2d(S.rh[st], &tm_rh4, &S.in_full[st], p0, cg * 4);
      }
      for (int64_t u = mine - 1; u >= 0 && u >= mine - kZIn; u--)
        mbar_wait_drain(&S.in_full[u % kZIn], (u / kZIn) & 1);
    }
  } else if (warp == 1) {
    // ------------------------------------------------ MMA
    if (elect_one()) {
      bool ok = true;
      constexpr uint32_t idh = idesc_f16(128, kZN), idl = idesc_f16(128, kD);
      for (int64_t w = 0; w < nwin && ok; w++) {
        const int ab = w & 1;
        if (!(ok = mbar_wait(&S.acc_empty[ab], ((w >> 1) & 1) ^ 1, err))) break;
        const int64_t t1 = std::min<int64_t>(mine, (w + 1) * kFlushBlocks);
        for (int64_t t = w * kFlushBlocks; t < t1 && ok; t++) {
          const int st = (int)(t % kZIn), sa = (int)(t % kZA);
          if (!(ok = mbar_wait(&S.in_full[st], (t / kZIn) & 1, err))) break;
          if (!(ok = mbar_wait(&S.a_full[sa], (t / kZA) & 1, err))) break;
          tc_fence_after();
          const uint64_t dbh = sdesc_sw128(smem_u32(S.bh[st])), dbl = sdesc_sw128(smem_u32(S.bl[st]));
#pragma unroll
          for (int kb = 0; kb < kBlk / 16; kb++) {
#pragma unroll
            for (int pr = 0; pr < 2; pr++) {
              const uint32_t dt = tbase + ab * 2 * kZDCol + pr * kZDCol;
              const uint32_t at = tbase + kZACol + sa * kZAStage + pr * (kBlk / 2) + kb * 8;
              // +32 bytes per 16-point K step inside the 128-byte swizzle row
              mma_f16_ta(dt, at, dbh + 2 * kb, idh, (t != w * kFlushBlocks) || kb);
              mma_f16_ta(dt, at, dbl + 2 * kb, idl, 1);
            }
          }
          mma_commit(&S.a_empty[sa]);
          mma_commit(&S.in_empty[st]);
        }
        if (!ok) break;
        mma_commit(&S.acc_full[ab]);
      }
      mma_commit(&S.mma_done);
      mbar_wait_drain(&S.mma_done, 0);
    }
  } else if (warp < 2 + 4 * kZSets) {
    // ------------------------------------------------ producers
    const int pw = warp - 2, grp = pw >> 2, quad = warp & 3;
    const int team = grp / kZSplit, part = grp % kZSplit;   // team: blocks; part: K steps within a block
    constexpr int kTeams = kZSets / kZSplit, kSteps = kBlk / 16 / kZSplit;
    const int slot = quad >> 1;                  // component slot within each pair
    const int a = 32 * (quad & 1) + lane;        // dimension = TMEM lane within the slot
    const uint32_t lane_addr = (uint32_t)(quad * 32) << 16;
    float mu[2];
#pragma unroll
    for (int pr = 0; pr < 2; pr++) mu[pr] = muf[(size_t)(cg * 4 + 2 * pr + slot) * kD + a];
    bool ok = true;
    for (int64_t t = team; t < mine && ok; t += kTeams) {
      const int st = (int)(t % kZIn), sa = (int)(t % kZA);
      if (!(ok = mbar_wait_warp(&S.in_full[st], (t / kZIn) & 1, err))) break;
      if (!(ok = mbar_wait_warp(&S.a_empty[sa], ((t / kZA) & 1) ^ 1, err))) break;
      tc_fence_after();
      const uint8_t *rowh = reinterpret_cast<const uint8_t *>(S.bh[st]) + a * 128;
      const uint8_t *rowl = reinterpret_cast<const uint8_t *>(S.bl[st]) + a * 128;
#pragma unroll 1
      for (int kb = part * kSteps; kb < (part + 1) * kSteps; kb++) {
        // x = xh + xl (exact in FP32) of the 16 points of this K step, dimension a
        float2 x[8];
#pragma unroll
        for (int hc = 0; hc < 2; hc++) {
          const int c = 2 * kb + hc, pc = (c ^ (a & 7)) << 4;
          const uint4 vh = *reinterpret_cast<const uint4 *>(rowh + pc);
          const uint4 vl = *reinterpret_cast<const uint4 *>(rowl + pc);
          const uint32_t wh[4] = {vh.x, vh.y, vh.z, vh.w}, wl[4] = {vl.x, vl.y, vl.z, vl.w};
#pragma unroll
          for (int q = 0; q < 4; q++)
            x[4 * hc + q] = __fadd2_rn(__half22float2(*reinterpret_cast<const __half2 *>(&wh[q])),
                                       __half22float2(*reinterpret_cast<const __half2 *>(&wl[q])));
        }
#pragma unroll
        for (int pr = 0; pr < 2; pr++) {
          // z = fp16(x - mu) * r_hi, two points per half2 (the posteriors' hi
          // part: an 11-bit weight, its rounding as random as z's own)
          const uint4 *r4 = reinterpret_cast<const uint4 *>(S.rh[st] + (2 * pr + slot) * kBlk + 16 * kb);
          const uint4 ra = r4[0], rb = r4[1];
          const uint32_t rw[8] = {ra.x, ra.y, ra.z, ra.w, rb.x, rb.y, rb.z, rb.w};
          const float2 nm = make_float2(-mu[pr], -mu[pr]);
          uint32_t packed[8];
#pragma unroll
          for (int q = 0; q < 8; q++) {
            const float2 dz = __fadd2_rn(x[q], nm);
            const __half2 z = __hmul2(__floats2half2_rn(dz.x, dz.y), *reinterpret_cast<const __half2 *>(&rw[q]));
            packed[q] = *reinterpret_cast<const uint32_t *>(&z);
          }
          tmem_st8(tbase + lane_addr + kZACol + sa * kZAStage + pr * (kBlk / 2) + kb * 8, packed);
        }
      }
      tmem_wait_st();
      tc_fence_before();
      __syncwarp();
      if (lane == 0) {
        mbar_arrive(&S.a_full[sa]);
        mbar_arrive(&S.in_empty[st]);
      }
    }
  } else {
    // ------------------------------------------------ flush warps
    const int quad = warp & 3;
    const int lrow = quad * 32 + lane;          // TMEM lane = row of the pair tile
    // this CTA's FP64 partials, column-major per pair: column c of pair pr
    // at o[pr][c * 128] (row lrow), so a warp's 32 rows are 256 contiguous bytes
    double *o[2];
#pragma unroll
    for (int pr = 0; pr < 2; pr++) {
      o[pr] = cpart + (cta * 2 + pr) * (size_t)(kZCols * 128) + lrow;
      for (int c = 0; c < kZCols; c++) o[pr][(size_t)c * 128] = 0.0;
    }
    bool ok = true;
    for (int64_t w = 0; w < nwin && ok; w++) {
      const int ab = w & 1;
      if (!(ok = mbar_wait_lazy_warp(&S.acc_full[ab], (w >> 1) & 1, err, 1000))) break;
      tc_fence_after();
#pragma unroll
      for (int pr = 0; pr < 2; pr++) {
        const uint32_t ta = tbase + ((uint32_t)(quad * 32) << 16) + ab * 2 * kZDCol + pr * kZDCol;
#pragma unroll 1
        for (int c0 = 0; c0 < kD; c0 += 16) {   // 16-column loads (the pair pitch is 80 columns)
          uint32_t v[16];
          tmem_ld16(ta + c0, v);
          tmem_wait_ld();
#pragma unroll
          for (int c = 0; c < 16; c++) o[pr][(size_t)(c0 + c) * 128] += (double)__uint_as_float(v[c]);
        }
        uint32_t v16[16];
        tmem_ld16(ta + kD, v16);
        tmem_wait_ld();
        o[pr][(size_t)kD * 128] += (double)__uint_as_float(v16[0]);
      }
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(&S.acc_empty[ab]);
    }
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  if (warp == 1) tmem_dealloc(tbase, 512);
}

// Sigma_j = sym(sum z x^T - (sum z) muf^T) / N_j - (mu - muf)(mu - muf)^T:
// the scatter around the FP32 means the producers used, moved to the FP64
// means; chunks summed in order (FP64)
// (a CTA owns rows 8 blockIdx.y .. + 7 of component blockIdx.x; a thread's sum
// over the chunks, up to 304 of them, is a chain of L2 loads, so the time is the
// number of sums per thread: only rows and columns below d, and 8 rows a CTA
// instead of 16: N = 600000, K = 6, d = 8 251 -> 57 us, K = 10, d = 60 171 -> 78)
constexpr int kFCRows = 8;
__global__ void __launch_bounds__(512)
k_final_cov_zx(const double *__restrict__ cpart, int gx, int gy, int d, const double *__restrict__ psum,
               const double *__restrict__ mu, const float *__restrict__ muf, double *__restrict__ sigma) {
  const int j = blockIdx.x, grp = j / 4, c = j % 4, pr = c >> 1, slot = c & 1;
  const int a0 = blockIdx.y * kFCRows;
  // S[a][b] = sum z_a x_b for the block's rows a, and S[b][a] for its columns
  __shared__ double sr[kFCRows][kD + 1], sc[kD][kFCRows + 1];
  __shared__ double sz[kD];                    // sum z of component j, per dimension
  const double *P0 = cpart + ((size_t)grp * 2 + pr) * (kZCols * 128) + slot * 64;
  const size_t step = (size_t)gx * 2 * (kZCols * 128);
  const int ri = min(kFCRows, d - a0);         // rows that exist; columns from d on are not summed
  for (int e = threadIdx.x; e < 2 * ri * d + d; e += blockDim.x) {
    // rows: (b, a0 + i) at P[b * 128 + a0 + i]; columns: (a0 + i, b) at P[(a0 + i) * 128 + b]; sum z: P[64 * 128 + a]
    size_t o;
    double *dst;
    if (e < ri * d) {
      const int i = e % ri, b = e / ri;
      o = (size_t)b * 128 + a0 + i, dst = &sr[i][b];
    } else if (e < 2 * ri * d) {
      const int r = e - ri * d, b = r % d, i = r / d;
      o = (size_t)(a0 + i) * 128 + b, dst = &sc[b][i];
    } else {
      const int a = e - 2 * ri * d;
      o = (size_t)kD * 128 + a, dst = &sz[a];
    }
    double v = 0.0;
#pragma unroll 8
    for (int ch = 0; ch < gy; ch++) v += P0[ch * step + o];
    *dst = v;
  }
  __syncthreads();
  const double inv = 1.0 / psum[j];
  double *Sg = sigma + (size_t)j * d * d;
  for (int e = threadIdx.x; e < kFCRows * kD; e += blockDim.x) {
    const int i = e / kD, a = a0 + i, b = e - i * kD;
    if (a >= d || b >= d || b < a) continue;
    const double ma = muf[(size_t)j * kD + a], mb = muf[(size_t)j * kD + b];
    const double ca = sr[i][b] - sz[a] * mb, cb = sc[b][i] - sz[b] * ma;
    const double v = 0.5 * (ca + cb) * inv - (mu[(size_t)j * d + a] - ma) * (mu[(size_t)j * d + b] - mb);
    Sg[a * d + b] = v;
    Sg[b * d + a] = v;
  }
}

// ================================================ covariances (split z x^T)
// The z x^T form above with z = r (x - mu) split into FP16 hi + lo as well,
// for fits whose components hold too few points for z's single rounding to
// average out, and x = xg + xr + xm in units of its dimension:
//   sum z x^T = sum zh xg^T + (sum zh (xr + xm)^T + sum zl (xg + xr)^T).
// To reach the accuracy of FP32 sums on CUDA cores:
//  * the tensor core truncates its FP32 accumulator, so z is put on a grid as x
//    is (z_unit: zh an integer, |zl| <= 1/2): zh xg^T then adds up exactly below
//    2^24 units.  Sums pass that more often the more rows a component has among
//    them, so the accumulator spans 16 blocks where none of the CTA's components
//    has a 24th of all weight and 4 elsewhere (rms error of Sigma_ab / (sd_a sd_b)
//    with 16 throughout: K = 12 3.2e-9, half the weight in one of 128 1.3e-8; now
//    1.2e-9 and 2.5e-9; CUDA cores 1.5e-9 and 4.2e-9).  With a floating split every
//    addition truncates: 4e-8 to 7e-8 off where CUDA cores are at 1e-8;
//  * the small products have an accumulator of their own (over a whole chunk its
//    truncation shows: N = 2^20, K = 128 1.4e-9, every kSCrossWin blocks 9e-10, CUDA
//    cores 1.1e-9); z comes from the FP32 rows, and x on the B side has a third
//    part xm;
//  * x on the B side is shared by all components and so not centred: a sum
//    holds (sum z) mu^T, random and |mu| / sigma times larger than what is
//    wanted.  A row of ones in B gives sum zh (exact) and sum zl beside the
//    sums, and flush warps take the product off before they add to FP32
//    registers (round to nearest); those go to FP64 every kSWin blocks;
//  * the diagonal is summed by the producers from the unrounded z (FP32 over
//    at most kSRows rows, then FP64);
//  * where a grid is too coarse for a component (split_too_coarse, by the E-step's
//    covariances before and by the result behind) the sums are formed on CUDA cores
//    instead: this kernel or that one returns at once.
// Sums are in units of z (rows) and x (columns), whatever the data's scale.
// Warp roles: 0 TMA, 1 MMA, 2 turns the posteriors into FP32 once per block;
// four producer groups of 4 warps, group g forming step g of every block (a
// warp's lanes and dimensions as in k_cov_zx); a flush group of 4 warps per pair, 64
// sums per thread (which is why the registers are split unevenly).
// What bounds it: shared memory, read by producers (x, posteriors) and by the
// 40 MMAs of a block (B), written by TMA, ~1800 of the ~3000 cycles a block
// takes; without 24 of the MMAs it is 13 % faster, with waits that sleep
// instead of polling no different.  GB300, with its finalisation, against the
// FP32 CUDA-core form: N = 2^20, d = 64, K = 128 20.7 -> 5.3 ms, N = 250000,
// d = 64, K = 24 0.98 -> 0.35 ms; error of Sigma (Frobenius) against 64-bit
// sums over the same posteriors 9.5e-9 and 1.0e-8 (CUDA cores 1.0e-8 and 1.7e-8).
__global__ void __launch_bounds__(kSThreads, 1)
k_cov_split(const __grid_constant__ CUtensorMap tm_xgt, const __grid_constant__ CUtensorMap tm_xrt,
            const __grid_constant__ CUtensorMap tm_xmt, const __grid_constant__ CUtensorMap tm_x32,
            const __grid_constant__ CUtensorMap tm_rh4, const __grid_constant__ CUtensorMap tm_rl4,
            const float *__restrict__ muf, const float *__restrict__ cmax, const float *__restrict__ zunit, int64_t n,
            int64_t rows_per_chunk, const double *__restrict__ psum, int K, double *__restrict__ cpart,
            double *__restrict__ dpart, const int *__restrict__ coarse, int *err) {
  if (coarse[0]) return;
  extern __shared__ uint8_t smem_raw[];
  SSmem &S = smem_aligned<SSmem>(smem_raw);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int cg = blockIdx.x;
  const int64_t r0 = (int64_t)blockIdx.y * rows_per_chunk, r1 = std::min<int64_t>(n, r0 + rows_per_chunk);
  const int mine = (int)((r1 - r0 + kBlk - 1) / kBlk);     // blocks of this chunk
  const size_t cta = (size_t)blockIdx.y * gridDim.x + blockIdx.x;

  if (threadIdx.x == 0) {
    // a block is read by the MMA and by the 16 producer warps
    for (int st = 0; st < kSIn; st++)
      mbar_init(&S.in_full[st], 1), mbar_init(&S.rf_full[st], 1), mbar_init(&S.in_empty[st], 17);
    for (int sl = 0; sl < kSA; sl++) mbar_init(&S.a_full[sl], 4), mbar_init(&S.a_empty[sl], 1);
    mbar_init(&S.acc_full, 1);
    mbar_init(&S.acc_empty, 8);
    mbar_init(&S.cross_full, 1);
    mbar_init(&S.cross_empty, 8);
    mbar_init(&S.mma_done, 1);
    fence_mbar_init();
  }
  double wmax = 0.0;
  for (int q = 0; q < 4 && 4 * cg + q < K; q++) wmax = fmax(wmax, psum[4 * cg + q]);
  const int am = (kSAccWeight * wmax <= (double)n ? kSAccLong : kSAccShort) - 1;   // span - 1
  // 16-byte chunk c of row r stored at c ^ (r & 7)
  for (int e = threadIdx.x; e < kSIn * 16 * kBlk; e += blockDim.x) {
    const int st = e / (16 * kBlk), rem = e - st * 16 * kBlk;
    const int r = kD + rem / kBlk, col = rem % kBlk;
    S.bh[st][r * kBlk + (((col >> 3) ^ (r & 7)) << 3) + (col & 7)] = __float2half(r == kD ? 1.f : 0.f);
  }
  fence_proxy_async_smem();
  for (int e = threadIdx.x; e < 4 * kD; e += blockDim.x) {
    const float m = muf[(size_t)cg * 4 * kD + e];
    const int ez = ilogbf(zunit[(size_t)cg * 4 * kD + e]);
    S.mu[e / kD][e % kD] = ldexpf(m, -x_unit_exp(cmax[e % kD]));
    S.zs[e / kD][e % kD] = ldexpf(1.f, -ez);
    S.zm[e / kD][e % kD] = ldexpf(-m, -ez);
  }
  if (warp == 1) tmem_alloc(&S.tmem_base, 512);
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tbase = S.tmem_base;
  constexpr uint32_t kInBytes = 3 * kD * kBlk * 2 + kBlk * kD * 4 + 2 * 4 * kBlk * 2;

  // no function calls behind this point: a call may use registers that the
  // split has taken away
  if (warp < kSProd0) {
    reg_dec<kSRegCtl>();
    if (warp == 0) {
      // ---------------------------------------------- TMA
      if (elect_one()) {
        bool ok = true;
        for (int t = 0; t < mine && ok; t++) {
          const int st = t % kSIn;
          if (!(ok = mbar_wait_lazy(&S.in_empty[st], ((t / kSIn) & 1) ^ 1, err, 128))) break;
          const int p0 = (int)(r0 + (int64_t)t * kBlk);
          mbar_expect_tx(&S.in_full[st], kInBytes);
          tma_load_2d(S.bh[st], &tm_xgt, &S.in_full[st], p0, 0);
          tma_load_2d(S.bl[st], &tm_xrt, &S.in_full[st], p0, 0);
          tma_load_2d(S.bm[st], &tm_xmt, &S.in_full[st], p0, 0);
          tma_load_2d(S.x[st], &tm_x32, &S.in_full[st], 0, p0);
          tma_load_2d(S.rh[st], &tm_rh4, &S.in_full[st], p0, cg * 4);
          tma_load_2d(S.rl[st], &tm_rl4, &S.in_full[st], p0, cg * 4);
        }
        for (int u = mine - 1; u >= 0 && u >= mine - kSIn; u--)
          mbar_wait_drain(&S.in_full[u % kSIn], (u / kSIn) & 1);
      }
    } else if (warp == 1) {
      // ---------------------------------------------- MMA
      if (elect_one()) {
        bool ok = true;
        constexpr uint32_t id = idesc_f16(128, kD), idn = idesc_f16(128, kSN);
        uint32_t sl = 0, sp = 0, ap = 0;           // operand slot and its phase; accumulator phase
        for (int t = 0; t < mine && ok; t++) {
          const int st = t % kSIn;
          if (!(ok = mbar_wait(&S.in_full[st], (t / kSIn) & 1, err))) break;
          const uint64_t dbh = sdesc_sw128(smem_u32(S.bh[st])), dbl = sdesc_sw128(smem_u32(S.bl[st]));
          const uint64_t dbm = sdesc_sw128(smem_u32(S.bm[st]));
#pragma unroll 1
          for (int kb = 0; kb < kSSteps; kb++) {
            if (!(ok = mbar_wait(&S.a_full[sl], sp, err))) break;
            tc_fence_after();
            const uint32_t at = tbase + kSACol + sl * kSAStage;
            if (t % kSCrossWin == 0 && kb == 0) {
              if (!(ok = mbar_wait(&S.cross_empty, ((t / kSCrossWin) & 1) ^ 1, err))) break;
              tc_fence_after();
            }
#pragma unroll
            for (int pr = 0; pr < 2; pr++) {
              // +32 bytes per 16-point step inside the 128-byte swizzle row
              const uint32_t dc = tbase + kSCross + pr * kSN, ah = at + 16 * pr, al = ah + 8;
              mma_f16_ta(dc, al, dbh + 2 * kb, idn, (t % kSCrossWin | kb) != 0);
              mma_f16_ta(dc, al, dbl + 2 * kb, id, 1);
              mma_f16_ta(dc, ah, dbl + 2 * kb, id, 1);
              mma_f16_ta(dc, ah, dbm + 2 * kb, id, 1);
            }
            if ((t & am) == 0 && kb == 0) {
              if (!(ok = mbar_wait(&S.acc_empty, ap ^ 1, err))) break;
              tc_fence_after();
            }
#pragma unroll
            for (int pr = 0; pr < 2; pr++)
              mma_f16_ta(tbase + pr * kSN, at + 16 * pr, dbh + 2 * kb, idn, (t & am) || kb);
            mma_commit(&S.a_empty[sl]);
            if (++sl == kSA) sl = 0, sp ^= 1;
          }
          if (!ok) break;
          mma_commit(&S.in_empty[st]);
          if ((t & am) == am || t + 1 == mine) mma_commit(&S.acc_full), ap ^= 1;
          if (t % kSCrossWin == kSCrossWin - 1 || t + 1 == mine) mma_commit(&S.cross_full);
        }
        mma_commit(&S.mma_done);
        mbar_wait_drain(&S.mma_done, 0);
      }
    } else if (warp == 2) {
      // ---------------------------------------------- posteriors: lane = 8 points of component lane / 8
      bool ok = true;
      for (int t = 0; t < mine && ok; t++) {
        const int st = t % kSIn;
        if (!(ok = mbar_wait_lazy_warp(&S.in_full[st], (t / kSIn) & 1, err, 64))) break;
        const uint4 vh = reinterpret_cast<const uint4 *>(S.rh[st])[lane];
        const uint4 vl = reinterpret_cast<const uint4 *>(S.rl[st])[lane];
        const uint32_t wh[4] = {vh.x, vh.y, vh.z, vh.w}, wl[4] = {vl.x, vl.y, vl.z, vl.w};
        float2 r[4];
#pragma unroll
        for (int q = 0; q < 4; q++)
          r[q] = __fadd2_rn(__half22float2(*reinterpret_cast<const __half2 *>(&wh[q])),
                            __half22float2(*reinterpret_cast<const __half2 *>(&wl[q])));
        float4 *o = reinterpret_cast<float4 *>(S.rf[st]) + 2 * lane;
        o[0] = make_float4(r[0].x, r[0].y, r[1].x, r[1].y);
        o[1] = make_float4(r[2].x, r[2].y, r[3].x, r[3].y);
        __syncwarp();
        if (lane == 0) mbar_arrive(&S.rf_full[st]);
      }
    }
  } else if (warp < kSFlush0) {
    reg_dec<kSRegProd>();
    // ------------------------------------------------ producers
    const int grp = (warp - kSProd0) >> 2, quad = warp & 3;   // group = the step it forms of every block
    const int slot = quad >> 1;                  // component slot within each pair
    const int a = 32 * (quad & 1) + lane;        // dimension = TMEM lane within the slot
    const uint32_t lane_addr = (uint32_t)(quad * 32) << 16;
    // (x - mu) / zunit = x xs + nm, one rounding: the unit is a power of two
    float2 xs[2], nm[2], dg[2];
    double ddg[2] = {0.0, 0.0};
#pragma unroll
    for (int pr = 0; pr < 2; pr++) {
      xs[pr] = f2(S.zs[2 * pr + slot][a]);
      nm[pr] = f2(S.zm[2 * pr + slot][a]);
      dg[pr] = make_float2(0.f, 0.f);
    }
    // w + c0 - c0 is w rounded to an integer (c0 = 1.5 2^23)
    const float2 c0 = f2(12582912.f), n0 = f2(-12582912.f);
    bool ok = true;
    int rows = 0;
    int sl = grp, sp = 0;                          // operand slot of step 4 t + grp (mod kSA) and its phase
    for (int t = 0; t < mine && ok; t++) {
      const int st = t % kSIn;
      if (!(ok = mbar_wait_warp(&S.in_full[st], (t / kSIn) & 1, err))) break;
      float2 x[8];                                 // the step's 16 points, dimension a
      const float *xr = S.x[st] + 16 * grp * kD + a;
#pragma unroll
      for (int q = 0; q < 8; q++) x[q] = make_float2(xr[2 * q * kD], xr[(2 * q + 1) * kD]);
      if (!(ok = mbar_wait_warp(&S.rf_full[st], (t / kSIn) & 1, err))) break;
      if (!(ok = mbar_wait_warp(&S.a_empty[sl], sp ^ 1, err))) break;
      tc_fence_after();
#pragma unroll
      for (int pr = 0; pr < 2; pr++) {
        const float4 *r4 = reinterpret_cast<const float4 *>(S.rf[st] + (2 * pr + slot) * kBlk + 16 * grp);
        uint32_t hi[8], lo[8];
#pragma unroll
        for (int q = 0; q < 4; q++) {
          const float4 r = r4[q];
#pragma unroll
          for (int u = 0; u < 2; u++) {
            const float2 dz = __ffma2_rn(x[2 * q + u], xs[pr], nm[pr]);
            const float2 rr = u ? make_float2(r.z, r.w) : make_float2(r.x, r.y);
            const float2 w = __fmul2_rn(dz, rr);
            dg[pr] = __ffma2_rn(w, dz, dg[pr]);
            const float2 wi = __fadd2_rn(__ffma2_rn(dz, rr, c0), n0);
            const __half2 h = __floats2half2_rn(wi.x, wi.y);
            const float2 hf = __half22float2(h);
            const float2 wl = __fadd2_rn(w, make_float2(-hf.x, -hf.y));
            const __half2 l = __floats2half2_rn(wl.x, wl.y);
            hi[2 * q + u] = *reinterpret_cast<const uint32_t *>(&h);
            lo[2 * q + u] = *reinterpret_cast<const uint32_t *>(&l);
          }
        }
        const uint32_t at = tbase + lane_addr + kSACol + sl * kSAStage + 16 * pr;
        tmem_st8(at, hi);
        tmem_st8(at + 8, lo);
      }
      tmem_wait_st();
      tc_fence_before();
      __syncwarp();
      if (lane == 0) {
        mbar_arrive(&S.a_full[sl]);
        mbar_arrive(&S.in_empty[st]);
      }
      sl += kSSteps;
      if (sl >= kSA) sl -= kSA, sp ^= 1;
      rows += 16;
      if (rows == kSRows) {
        rows = 0;
#pragma unroll
        for (int pr = 0; pr < 2; pr++) {
          ddg[pr] += (double)(dg[pr].x + dg[pr].y);
          dg[pr] = make_float2(0.f, 0.f);
        }
      }
    }
#pragma unroll
    for (int pr = 0; pr < 2; pr++)   // [cta][producer group][component][dimension]
      dpart[((cta * 4 + grp) * 4 + 2 * pr + slot) * kD + a] = ddg[pr] + (double)(dg[pr].x + dg[pr].y);
  } else {
    reg_inc<kSRegFlush>();
    // ------------------------------------------------ flush warps: TMEM lane = row of the pair tile
    const int pr = (warp - kSFlush0) >> 2, quad = warp & 3, lrow = quad * 32 + lane;
    // this CTA's FP64 partials, column-major per pair: column c of pair pr at
    // cpart[..][(pr * 64 + c) * 128], so a warp's 32 rows are 256 contiguous bytes
    double *o = cpart + cta * (size_t)(2 * kD * 128) + (size_t)pr * (kD * 128) + lrow;
    const float *mu = S.mu[2 * pr + (quad >> 1)];
    float acc[kD];
#pragma unroll
    for (int c = 0; c < kD; c++) acc[c] = 0.f;
    const uint32_t ta = tbase + ((uint32_t)(quad * 32) << 16) + pr * kSN;
    auto take = [&](uint32_t from) {
      uint32_t v[16];
      tmem_ld16(from + kD, v);
      tmem_wait_ld();
      const float sz = __uint_as_float(v[0]);
#pragma unroll
      for (int c0 = 0; c0 < kD; c0 += 16) {
        tmem_ld16(from + c0, v);
        tmem_wait_ld();
#pragma unroll
        for (int c = 0; c < 16; c += 4) {
          const float4 m = *reinterpret_cast<const float4 *>(mu + c0 + c);
          acc[c0 + c] += fmaf(-sz, m.x, __uint_as_float(v[c]));
          acc[c0 + c + 1] += fmaf(-sz, m.y, __uint_as_float(v[c + 1]));
          acc[c0 + c + 2] += fmaf(-sz, m.z, __uint_as_float(v[c + 2]));
          acc[c0 + c + 3] += fmaf(-sz, m.w, __uint_as_float(v[c + 3]));
        }
      }
    };
    bool ok = true, first = true;
    uint32_t ap = 0;
    for (int t0 = 0; t0 < mine && ok; t0 += am + 1, ap ^= 1) {
      const int t1 = std::min(mine, t0 + am + 1);
      if (!(ok = mbar_wait_lazy_warp(&S.acc_full, ap, err, 500))) break;
      tc_fence_after();
      take(ta);
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(&S.acc_empty);
      if (t1 == mine || t1 % kSCrossWin == 0) {
        if (!(ok = mbar_wait_warp(&S.cross_full, ((t1 - 1) / kSCrossWin) & 1, err))) break;
        tc_fence_after();
        take(ta + kSCross);
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(&S.cross_empty);
      }
      if (t1 == mine || t1 % kSWin == 0) {
#pragma unroll
        for (int c = 0; c < kD; c++) {
          double *q = o + (size_t)c * 128;
          *q = first ? (double)acc[c] : *q + (double)acc[c];
          acc[c] = 0.f;
        }
        first = false;
      }
    }
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  if (warp == 1) tmem_dealloc(tbase, 512);
}

// Sigma_j = sym(sum z (x - muf)^T) / N_j - (mu - muf)(mu - muf)^T, the
// producers' sums on the diagonal; chunks summed in order (FP64).
// A CTA owns rows 8 blockIdx.y .. + 7 of component blockIdx.x.
__global__ void __launch_bounds__(512)
k_final_cov_split(const double *__restrict__ cpart, const double *__restrict__ dpart, int gx, int gy, int d,
                  const double *__restrict__ psum, const double *__restrict__ mu, const float *__restrict__ muf,
                  const float *__restrict__ cmax, const float *__restrict__ zunit, double *__restrict__ sigma,
                  int *coarse) {
  if (coarse[0]) return;
  const int j = blockIdx.x, grp = j / 4, c = j % 4, pr = c >> 1, slot = c & 1;
  const int a0 = blockIdx.y * kFCRows;
  __shared__ double sr[kFCRows][kD + 1], sc[kD][kFCRows + 1], sd[kFCRows];
  const double *P0 = cpart + ((size_t)grp * 2 + pr) * (kD * 128) + slot * 64;
  const size_t step = (size_t)gx * 2 * (kD * 128);
  for (int e = threadIdx.x; e < 2 * kFCRows * kD + kFCRows; e += blockDim.x) {
    double v = 0.0;
    if (e < 2 * kFCRows * kD) {
      // rows: (b, a0 + i) at P[b * 128 + a0 + i]; columns: (a0 + i, b) at P[(a0 + i) * 128 + b]
      const int r = e % (kFCRows * kD);
      const bool rowpart = e < kFCRows * kD;
      const int i = rowpart ? r % kFCRows : r / kD, b = rowpart ? r / kFCRows : r % kD;
      const size_t o = rowpart ? (size_t)b * 128 + a0 + i : (size_t)(a0 + i) * 128 + b;
#pragma unroll 8
      for (int ch = 0; ch < gy; ch++) v += P0[ch * step + o];
      (rowpart ? sr[i][b] : sc[b][i]) = v;
    } else {
      const int i = e - 2 * kFCRows * kD;
      for (int ch = 0; ch < gy; ch++)
#pragma unroll
        for (int g = 0; g < 4; g++) v += dpart[((((size_t)ch * gx + grp) * 4 + g) * 4 + c) * kD + a0 + i];
      sd[i] = v;
    }
  }
  __syncthreads();
  const double inv = 1.0 / psum[j];
  double *Sg = sigma + (size_t)j * d * d;
  for (int e = threadIdx.x; e < kFCRows * kD; e += blockDim.x) {
    const int i = e / kD, a = a0 + i, b = e - i * kD;
    if (a >= d || b >= d || b < a) continue;
    const double da = mu[(size_t)j * d + a] - (double)muf[(size_t)j * kD + a];
    const double db = mu[(size_t)j * d + b] - (double)muf[(size_t)j * kD + b];
    const double ga = zunit[(size_t)j * kD + a], gb = zunit[(size_t)j * kD + b];
    const double t = a == b ? sd[i] * ga * ga
                            : 0.5 * (sr[i][b] * (ga * x_unit(cmax[b])) + sc[b][i] * (gb * x_unit(cmax[a])));
    const double v = t * inv - da * db;
    if (a == b && split_too_coarse(v, cmax[a], zunit[(size_t)j * kD + a])) coarse[1] = 1;
    Sg[a * d + b] = v;
    Sg[b * d + a] = v;
  }
}

// ================================================= bounded-wait expiry
// The exit path every warp-specialised kernel here relies on, run on purpose:
// one CTA with the roles of those kernels, whose producer never delivers.
// Warp 1 allocates all 512 TMEM columns (as the E-step and covariance kernels
// do) and waits for a barrier nothing arrives on, with `budget` cycles: the
// wait runs out, sets the status word and returns false; its drain wait
// (which ignores the status word, as the drains before TMEM release do) runs
// out too.  Warps 2 and 3 wait, off the critical path, for a barrier warp 1
// would have completed; they leave because the status word is set, not by
// their own (long) budget.  Every warp then reaches the final barrier and
// warp 1 releases TMEM.  roles[0..3] record which waits gave up.
__global__ void __launch_bounds__(128, 1) k_wait_expiry(long long budget, int *err, int *roles) {
  __shared__ uint64_t full, done;
  __shared__ uint32_t tslot;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  if (threadIdx.x == 0) {
    mbar_init(&full, 1);
    mbar_init(&done, 1);
    fence_mbar_init();
  }
  if (warp == 1) tmem_alloc(&tslot, 512);
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  if (warp == 1) {
    if (mbar_wait_warp(&full, 0, err, budget)) {
      if (lane == 0) mbar_arrive(&done);
    } else if (lane == 0) {
      roles[0] = 1;
    }
    if (lane == 0 && !mbar_wait_drain(&full, 0, budget)) roles[1] = 1;
  } else if (warp >= 2) {
    if (!mbar_wait_lazy_warp(&done, 0, err, 200) && lane == 0) roles[warp] = 1;
  }
  // warp 0, the producer, delivers nothing
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  if (warp == 1) tmem_dealloc(tslot, 512);
}

// ================================================ operand preparation
// W = L^-1 (FP64) -> FP16 hi/lo in the permuted row order; b = L^-1 mu;
// row of (component j, output k) = group j/2, k-block position 3 - k/16,
// component j%2, k%16
__device__ __forceinline__ int w_row(int j, int k) {
  return (j / kCompPerGroup) * kGroupN + (kD / 16 - 1 - k / 16) * (16 * kCompPerGroup) +
         (j % kCompPerGroup) * 16 + (k & 15);
}

// Dimensions d..63 of a component with d < 64 get zero rows and columns
// (x and mu are zero there, so y = 0), components K..Kp-1 (padding to a
// multiple of 4) get W = 0 and a log coefficient of -inf (posterior 0).
__global__ void k_prep_w(const double *__restrict__ linv, const double *__restrict__ mu, int K, int d,
                         __half *__restrict__ Wh, __half *__restrict__ Wl, float *__restrict__ bias,
                         const double *__restrict__ logc, float *__restrict__ chi, float *__restrict__ clo) {
  const int j = blockIdx.x;
  const bool live = j < K;
  if (threadIdx.x == 0) {
    chi[j] = live ? (float)logc[j] : -INFINITY;
    clo[j] = live ? (float)(logc[j] - (double)(float)logc[j]) : 0.f;
  }
  for (int e = threadIdx.x; e < kD * kD; e += blockDim.x) {
    const int k = e / kD, m = e - k * kD;
    const int row = w_row(j, k);
    const double w = (live && k < d && m < d) ? linv[((size_t)j * d + k) * d + m] : 0.0;
    const __half h = __double2half(w);
    Wh[(size_t)row * kD + m] = h;
    Wl[(size_t)row * kD + m] = __double2half(w - (double)__half2float(h));
  }
  for (int k = threadIdx.x; k < kD; k += blockDim.x) {
    double b = 0.0;
    if (live && k < d)
      for (int m = 0; m <= k; m++) b += linv[((size_t)j * d + k) * d + m] * mu[(size_t)j * d + m];
    bias[w_row(j, k)] = (float)b;
  }
}

// largest |x| of every dimension (cmax[0..d - 1], zero at the start): the units of
// the split covariance
__global__ void __launch_bounds__(256)
k_col_max(const float *__restrict__ X, int64_t n, int d, float *__restrict__ cmax) {
  __shared__ int sm[kD];
  if (threadIdx.x < kD) sm[threadIdx.x] = 0;
  __syncthreads();
  // a thread stays in one column: blocks and strides are whole rows
  const int rows = 256 / d, c = threadIdx.x % d, r = threadIdx.x / d;
  float m = 0.f;
  if (r < rows) {
#pragma unroll 4
    for (int64_t i = (int64_t)blockIdx.x * rows + r; i < n; i += (int64_t)gridDim.x * rows)
      m = fmaxf(m, fabsf(X[i * d + c]));
    atomicMax(&sm[c], __float_as_int(m));
  }
  __syncthreads();
  // non-negative floats order like their bits
  if (threadIdx.x < d) atomicMax(reinterpret_cast<int *>(cmax) + threadIdx.x, sm[threadIdx.x]);
}

// x -> xh = fp16(x), xl = fp16(x - xh), row-major and transposed (d x np) (rows of
// d < 64 values are zero-padded to 64; X64 receives the padded FP32 rows when it is
// not null), and the largest |x|.  UNITS: the split covariance's three parts as well.
template <bool UNITS>
__global__ void k_split_x(const float *__restrict__ X, int64_t n, int d, __half *__restrict__ Xh,
                          __half *__restrict__ Xl, __half *__restrict__ XhT, __half *__restrict__ XlT,
                          __half *__restrict__ XgT, __half *__restrict__ XrT, __half *__restrict__ XmT, int64_t np,
                          float *__restrict__ X64, const float *__restrict__ cmax, float *__restrict__ amax) {
  constexpr int kParts = UNITS ? 5 : 2;
  __shared__ __half t[kParts][kD][65];
  __shared__ float sinv[kD];
  if (UNITS && threadIdx.x < kD) sinv[threadIdx.x] = ldexpf(1.f, -x_unit_exp(cmax[threadIdx.x]));
  __syncthreads();
  __half *const out[5] = {XhT, XlT, XgT, XrT, XmT};
  float m = 0.f;
  const int64_t nt = (n + 63) / 64;
  for (int64_t tile = blockIdx.x; tile < nt; tile += gridDim.x) {
    const int64_t r0 = tile * 64;
    for (int e = threadIdx.x; e < 64 * kD; e += blockDim.x) {
      const int r = e / kD, c = e - r * kD;
      if (r0 + r < n) {
        const float x = c < d ? X[(r0 + r) * d + c] : 0.f;
        if (X64) X64[(r0 + r) * kD + c] = x;
        const __half h = __float2half_rn(x);
        const __half l = __float2half_rn(x - __half2float(h));
        Xh[(r0 + r) * kD + c] = t[0][c][r] = h;
        Xl[(r0 + r) * kD + c] = t[1][c][r] = l;
        m = fmaxf(m, fabsf(x));
        if constexpr (UNITS) {
          const float u = x * sinv[c], ui = rintf(u);
          const __half ur = __float2half_rn(u - ui);
          t[2][c][r] = __float2half_rn(ui);
          t[3][c][r] = ur;
          t[4][c][r] = __float2half_rn((u - ui) - __half2float(ur));
        }
      }
    }
    __syncthreads();
    for (int e = threadIdx.x; e < 64 * kD; e += blockDim.x) {
      const int c = e / 64, r = e - c * 64;
      if (r0 + r < n)
#pragma unroll
        for (int p = 0; p < kParts; p++) out[p][(size_t)c * np + r0 + r] = t[p][c][r];
    }
    __syncthreads();
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) m = fmaxf(m, __shfl_down_sync(0xffffffffu, m, o));
  // non-negative floats order like their bits
  if ((threadIdx.x & 31) == 0) atomicMax(reinterpret_cast<int *>(amax), __float_as_int(m));
}

// one warp, a lane's terms first, then a fixed tree
__global__ void k_reduce_parts(const double *__restrict__ part, int np, DevStatus *st,
                               const int *__restrict__ err) {
  double s = 0.0;
#pragma unroll 8
  for (int b = threadIdx.x; b < np; b += 32) s += part[b];
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
  if (threadIdx.x == 0) {
    st->logl = s;
    if (*err) st->timeout = 1;
  }
}

__global__ void k_flag_timeout(DevStatus *st, const int *__restrict__ err) {
  if (threadIdx.x == 0 && *err) st->timeout = 1;
}

// posteriors (hi + lo) -> n x K double rows
__global__ void k_post_rows_tc(const __half *__restrict__ Rh, const __half *__restrict__ Rl, int64_t np,
                               int K, int64_t r0, int64_t rows, double *__restrict__ out) {
  const int64_t e = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (e >= rows * K) return;
  const int64_t i = e / K;
  const int j = (int)(e - i * K);
  const size_t o = (size_t)j * np + r0 + i;
  out[e] = (double)__half2float(Rh[o]) + (double)__half2float(Rl[o]);
}

__global__ void k_classes_tc(const __half *__restrict__ Rh, const __half *__restrict__ Rl, int64_t np,
                             int64_t n, int K, int32_t *__restrict__ cls) {
  const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  float best = -1.f;
  int bj = -1;
  for (int j = 0; j < K; j++) {
    const float v = __half2float(Rh[(size_t)j * np + i]) + __half2float(Rl[(size_t)j * np + i]);
    if (v > best) {
      best = v;
      bj = j;
    }
  }
  cls[i] = bj;
}

// ============================================================== host side
static size_t esmem_bytes() { return sizeof(ESmem) + 1024; }
static size_t msmem_bytes() { return sizeof(MSmem) + 1024; }
static size_t csmem_bytes() { return sizeof(CSmem) + 1024; }
static size_t zsmem_bytes() { return sizeof(ZSmem) + 1024; }
static size_t ssmem_bytes() { return sizeof(SSmem) + 1024; }

static int fp16_map(CUtensorMap *m, const void *base, uint64_t cols, uint64_t rows, uint64_t pitch_elems,
                    uint32_t box_cols, uint32_t box_rows, CUtensorMapSwizzle swz) {
  return encode_tmap_2d(m, CU_TENSOR_MAP_DATA_TYPE_FLOAT16, 2, base, cols, rows, box_cols, box_rows, swz,
                        pitch_elems * 2);
}

// the covariance kernel works on groups of 4 components
// d <= 64 (zero-padded to 64) and K <= 128 (padded to a multiple of 4)
bool em_tc_supported(int d, int k) {
  return (d >= 1 && d <= kD && k >= 1 && k <= kMaxK) || em_wide_supported(d, k);
}

// The tensor-core covariance rounds z to FP16 once; that error averages out
// over the points of a component (relative ~2^-12 / sqrt(N_j)).  With fewer
// than 16384 points per component on average it would not, so such fits take
// the FP32 CUDA-core covariance (its cost is small at that size).
static bool em_tc_small_components(int64_t n, int k, int d) { return d <= kD && n < (int64_t)16384 * k; }

// covariance kernel selection while both forms are compared (FEM_COV_KERNEL=zz
// selects the z z^T form)
static bool cov_zx_enabled() {
  static const bool zx = [] {
    const char *v = getenv("FEM_COV_KERNEL");
    return !(v && v[0] == 'z' && v[1] == 'z');
  }();
  return zx;
}

// Small components: the split tensor-core form or the CUDA-core one.  The
// split form pads to 64 dimensions and 4 components, the CUDA-core form costs
// 8 x 8 blocks of the triangle, so it is ahead up to d = 32 (N = 10^5, K = 12,
// d = 32: 86 against 130 us; N = 200003, K = 21, d = 24: 147 against 240) and
// the split form above (N = 500000, K = 64, d = 48: 1.3 against 3.5 ms; N =
// 2^20, K = 128, d = 64: 5.3 against 20.7 ms), once every SM has 16 or more of
// its (64-point block, 4-component group) units to pay for a CTA's start and
// end (K = 8, d = 64: N = 20000, 4 a SM, 57 against 102 us; N = 100000, 20 a
// SM, 227 against 143 us).
static bool cov_split_wins(int64_t n, int d, int kp) {
  cudaFuncAttributes a;
  // its register split presumes the launch's share
  if (cudaFuncGetAttributes(&a, k_cov_split) != cudaSuccess || a.numRegs < kSRegLaunch) return false;
  return d > 32 && (n + kBlk - 1) / kBlk * (kp / 4) >= (int64_t)16 * sm_count();
}

static decltype(&k_estep_tc<4>) estep_tc_kernel(int d) {
  return d <= 16 ? k_estep_tc<1> : d <= 32 ? k_estep_tc<2> : d <= 48 ? k_estep_tc<3> : k_estep_tc<4>;
}

int em_tc_create(fem_em *h) {
  if (h->d > kD) return em_wide_create(h);
  TcEmPlan *p = new TcEmPlan();
  h->tc = p;
  const int K = (h->k + 3) / 4 * 4;     // kernels see K padded to a multiple of 4
  const int64_t n = h->n;
  p->kp = K;
  p->d = h->d;
  p->np = (n + 63) / 64 * 64;
  const int sms = sm_count();
  FEM_TRY(dalloc(&h->Xhi, (size_t)n * kD));
  FEM_TRY(dalloc(&h->Xlo, (size_t)n * kD));
  FEM_TRY(dalloc(&p->XhT, (size_t)kD * p->np));
  FEM_TRY(dalloc(&p->XlT, (size_t)kD * p->np));
  FEM_TRY(dalloc(&p->Rh, (size_t)K * p->np));
  FEM_TRY(dalloc(&p->Rl, (size_t)K * p->np));
  FEM_TRY(dalloc(&p->Wh, (size_t)K * kD * kD));
  FEM_TRY(dalloc(&p->Wl, (size_t)K * kD * kD));
  FEM_TRY(dalloc(&p->bias, (size_t)K * kD));
  FEM_TRY(dalloc(&p->clo, K));
  FEM_TRY(dalloc(&p->muf, (size_t)K * kD));
  FEM_TRY(dalloc(&p->chi, K));
  FEM_CUDA(cudaMemset(p->muf, 0, (size_t)K * kD * sizeof(float)));
  if (h->d < kD) FEM_TRY(dalloc(&p->X64, (size_t)n * kD));
  FEM_TRY(dalloc(&p->err, 1));
  FEM_CUDA(cudaMemset(p->err, 0, sizeof(int)));
  FEM_TRY(dalloc(&p->amax, kD + 1));
  FEM_CUDA(cudaMemset(p->amax, 0, (kD + 1) * sizeof(float)));
  FEM_TRY(dalloc(&p->zunit, (size_t)K * kD));
  FEM_TRY(dalloc(&p->coarse, 2));
  FEM_TRY(dalloc(&p->roles, 4));
  const int64_t npairs = ((n + kTileM - 1) / kTileM + 1) / 2;
  p->egrid = (int)std::min<int64_t>(sms, npairs);
  FEM_TRY(dalloc(&p->epart, p->egrid));
  FEM_TRY(dalloc(&p->lsc, (size_t)p->egrid * 2 * K * 2 * kTileM));
  const int64_t nblocks = (n + kBlk - 1) / kBlk;
  p->mgrid = (int)std::min<int64_t>(sms, nblocks);
  FEM_TRY(dalloc(&p->mpart, (size_t)p->mgrid * kMaxK * kMeanN));
  p->cgx = K / 4;
  if (em_tc_small_components(n, h->k, h->d)) {
    if (cov_split_wins(n, h->d, K)) {
      // a CTA's start and end (TMEM, pipeline fill, FP64 stores) cost about 12 blocks
      split_rows(n, kBlk, p->cgx, sms, 12.0, &p->cgy, &p->srows);
      FEM_TRY(dalloc(&p->cpart, (size_t)p->cgx * p->cgy * 2 * kD * 128));
      FEM_TRY(dalloc(&p->dpart, (size_t)p->cgx * p->cgy * 4 * 4 * kD));
      __half **parts[3] = {&p->XgT, &p->XrT, &p->XmT};
      CUtensorMap *maps[3] = {&p->tm_xgt, &p->tm_xrt, &p->tm_xmt};
      for (int q = 0; q < 3; q++) {
        FEM_TRY(dalloc(parts[q], (size_t)kD * p->np));
        FEM_TRY(encode_tmap_2d(maps[q], CU_TENSOR_MAP_DATA_TYPE_FLOAT16, 2, *parts[q], (uint64_t)n, kD, kBlk, kD,
                               CU_TENSOR_MAP_SWIZZLE_128B, (uint64_t)p->np * 2));
      }
    }
  } else {
    p->cgy = (int)std::max<int64_t>(1, std::min<int64_t>(nblocks, (4 * sms + p->cgx - 1) / p->cgx));
    FEM_TRY(dalloc(&p->cpart, (size_t)p->cgx * p->cgy * std::max(4 * kD * kD, 2 * kZCols * 128)));
    FEM_TRY(dalloc(&p->dpart, (size_t)p->cgx * p->cgy * 4 * kD));
  }
  // E-step operands
  FEM_TRY(fp16_map(&p->tm_xh, h->Xhi, kD, n, kD, kD, kTileM, CU_TENSOR_MAP_SWIZZLE_128B));
  FEM_TRY(fp16_map(&p->tm_xl, h->Xlo, kD, n, kD, kD, kTileM, CU_TENSOR_MAP_SWIZZLE_128B));
  FEM_TRY(fp16_map(&p->tm_wh, p->Wh, kD, (uint64_t)K * kD, kD, kD, kGroupN, CU_TENSOR_MAP_SWIZZLE_128B));
  FEM_TRY(fp16_map(&p->tm_wl, p->Wl, kD, (uint64_t)K * kD, kD, kD, kGroupN, CU_TENSOR_MAP_SWIZZLE_128B));
  // means operands: rows of np-pitched component-major / transposed arrays
  FEM_TRY(encode_tmap_2d(&p->tm_rh, CU_TENSOR_MAP_DATA_TYPE_FLOAT16, 2, p->Rh, (uint64_t)n, (uint64_t)K, kBlk,
                         kMaxK, CU_TENSOR_MAP_SWIZZLE_128B, (uint64_t)p->np * 2));
  FEM_TRY(encode_tmap_2d(&p->tm_rl, CU_TENSOR_MAP_DATA_TYPE_FLOAT16, 2, p->Rl, (uint64_t)n, (uint64_t)K, kBlk,
                         kMaxK, CU_TENSOR_MAP_SWIZZLE_128B, (uint64_t)p->np * 2));
  FEM_TRY(encode_tmap_2d(&p->tm_xht, CU_TENSOR_MAP_DATA_TYPE_FLOAT16, 2, p->XhT, (uint64_t)n, kD, kBlk, kD,
                         CU_TENSOR_MAP_SWIZZLE_128B, (uint64_t)p->np * 2));
  FEM_TRY(encode_tmap_2d(&p->tm_xlt, CU_TENSOR_MAP_DATA_TYPE_FLOAT16, 2, p->XlT, (uint64_t)n, kD, kBlk, kD,
                         CU_TENSOR_MAP_SWIZZLE_128B, (uint64_t)p->np * 2));
  // covariance operands (no swizzle: read by CUDA cores)
  FEM_TRY(encode_tmap_2d(&p->tm_x32, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 4, p->X64 ? p->X64 : h->X, kD, (uint64_t)n, kD,
                         kBlk,
                         CU_TENSOR_MAP_SWIZZLE_NONE, 0));
  FEM_TRY(encode_tmap_2d(&p->tm_rh4, CU_TENSOR_MAP_DATA_TYPE_FLOAT16, 2, p->Rh, (uint64_t)n, (uint64_t)K, kBlk, 4,
                         CU_TENSOR_MAP_SWIZZLE_NONE, (uint64_t)p->np * 2));
  FEM_TRY(encode_tmap_2d(&p->tm_rl4, CU_TENSOR_MAP_DATA_TYPE_FLOAT16, 2, p->Rl, (uint64_t)n, (uint64_t)K, kBlk, 4,
                         CU_TENSOR_MAP_SWIZZLE_NONE, (uint64_t)p->np * 2));
  FEM_CUDA(cudaFuncSetAttribute(estep_tc_kernel(h->d), cudaFuncAttributeMaxDynamicSharedMemorySize, (int)esmem_bytes()));
  FEM_CUDA(cudaFuncSetAttribute(k_means_tc, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)msmem_bytes()));
  FEM_CUDA(cudaFuncSetAttribute(k_cov_tc, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)csmem_bytes()));
  FEM_CUDA(cudaFuncSetAttribute(k_cov_zx, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)zsmem_bytes()));
  FEM_CUDA(cudaFuncSetAttribute(k_cov_split, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)ssmem_bytes()));
  return FEM_OK;
}

bool em_tc_cuda_core_cov(const fem_em *h) { return h->tc && em_tc_small_components(h->n, h->k, h->d); }

void em_tc_destroy(fem_em *h) {
  em_wide_destroy(h);
  TcEmPlan *p = h->tc;
  if (!p) return;
  dfree(p->Wh);
  dfree(p->Wl);
  dfree(p->bias);
  dfree(p->clo);
  dfree(p->Rh);
  dfree(p->Rl);
  dfree(p->XhT);
  dfree(p->XlT);
  dfree(p->XgT);
  dfree(p->XrT);
  dfree(p->XmT);
  dfree(p->lsc);
  dfree(p->epart);
  dfree(p->mpart);
  dfree(p->cpart);
  dfree(p->dpart);
  dfree(p->muf);
  dfree(p->chi);
  dfree(p->X64);
  dfree(p->err);
  dfree(p->amax);
  dfree(p->zunit);
  dfree(p->coarse);
  dfree(p->roles);
  delete p;
  h->tc = nullptr;
}

int em_tc_upload(fem_em *h) {
  if (h->wide) return em_wide_upload(h);
  TcEmPlan *p = h->tc;
  float *amax = p->amax;
  FEM_CUDA(cudaMemsetAsync(amax, 0, (kD + 1) * sizeof(float), h->stream));
  const int blocks = (int)std::min<int64_t>(4 * sm_count(), (h->n + 63) / 64);
  if (p->srows) k_col_max<<<blocks, 256, 0, h->stream>>>(h->X, h->n, h->d, amax);
  (p->srows ? k_split_x<true> : k_split_x<false>)<<<blocks, 256, 0, h->stream>>>(
      h->X, h->n, h->d, h->Xhi, h->Xlo, p->XhT, p->XlT, p->XgT, p->XrT, p->XmT, p->np, p->X64, amax, amax + kD);
  float m = 0.f;
  cudaMemcpyAsync(&m, amax + kD, sizeof(float), cudaMemcpyDeviceToHost, h->stream);
  cudaError_t e = cudaStreamSynchronize(h->stream);
  if (e != cudaSuccess) {
    set_error("dataset split failed: %s", cudaGetErrorString(e));
    return FEM_ERR_CUDA;
  }
  if (!(m < 32768.f)) {
    set_error("mixed precision needs |x| < 32768 (FP16 operands); max |x| = %g", m);
    return FEM_ERR_UNSUPPORTED;
  }
  return FEM_OK;
}

int em_tc_prepare(fem_em *h) {
  if (h->wide) return em_wide_prepare(h);
  TcEmPlan *p = h->tc;
  k_prep_w<<<p->kp, 256, 0, h->stream>>>(h->linv, h->mu, h->k, h->d, p->Wh, p->Wl, p->bias, h->logc, p->chi,
                                         p->clo);
  FEM_CUDA(cudaGetLastError());
  h->launches += 1;
  return FEM_OK;
}

int em_tc_estep(fem_em *h) {
  if (h->wide) return em_wide_estep(h);
  TcEmPlan *p = h->tc;
  estep_tc_kernel(h->d)<<<p->egrid, kEThreads, esmem_bytes(), h->stream>>>(
      p->tm_xh, p->tm_xl, p->tm_wh, p->tm_wl, p->bias, p->chi, p->clo, h->logc, p->lsc, p->Rh, p->Rl, p->np,
      p->epart, h->n, p->kp, p->err);
  FEM_CUDA(cudaGetLastError());
  k_reduce_parts<<<1, 32, 0, h->stream>>>(p->epart, p->egrid, h->dstat, p->err);
  FEM_CUDA(cudaGetLastError());
  h->launches += 2;
  return FEM_OK;
}

int em_tc_mstep(fem_em *h) {
  if (h->wide) return em_wide_mstep(h);
  TcEmPlan *p = h->tc;
  const int K = h->k;
  k_means_tc<<<p->mgrid, 192, msmem_bytes(), h->stream>>>(p->tm_rh, p->tm_rl, p->tm_xht, p->tm_xlt, h->n,
                                                           p->mpart, p->coarse, p->err);
  FEM_CUDA(cudaGetLastError());
  k_final_means_tc<<<K, kFMSplit * kFMCols, 0, h->stream>>>(p->mpart, p->mgrid, K, h->d, h->n, h->mu, h->pi, h->psum,
                                                               p->muf, p->amax, h->sigma, p->zunit, p->coarse);
  FEM_CUDA(cudaGetLastError());
  if (em_tc_small_components(h->n, h->k, h->d)) {
    timing_begin(h, 8);
    if (p->srows) {
      k_cov_split<<<dim3(p->cgx, p->cgy), kSThreads, ssmem_bytes(), h->stream>>>(
          p->tm_xgt, p->tm_xrt, p->tm_xmt, p->tm_x32, p->tm_rh4, p->tm_rl4, p->muf, p->amax, p->zunit, h->n, p->srows, h->psum,
          K, p->cpart, p->dpart, p->coarse, p->err);
      FEM_CUDA(cudaGetLastError());
      k_final_cov_split<<<dim3(K, (h->d + kFCRows - 1) / kFCRows), 512, 0, h->stream>>>(
          p->cpart, p->dpart, p->cgx, p->cgy, h->d, h->psum, h->mu, p->muf, p->amax, p->zunit, h->sigma, p->coarse);
      FEM_CUDA(cudaGetLastError());
      h->launches += 2;
    }
    // the only form, or where the split one's grids are too coarse
    FEM_TRY(em_cov_hilo(h, p->Rh, p->Rl, p->np, p->muf, kD, p->srows ? p->coarse : nullptr));
    timing_begin(h, 9);
    k_flag_timeout<<<1, 32, 0, h->stream>>>(h->dstat, p->err);
    h->launches += 3;
    return FEM_OK;
  }
  const int64_t nblocks = (h->n + kBlk - 1) / kBlk;
  const int64_t bpc = (nblocks + p->cgy - 1) / p->cgy;
  timing_begin(h, 8);
  if (cov_zx_enabled()) {
    k_cov_zx<<<dim3(p->cgx, p->cgy), kZThreads, zsmem_bytes(), h->stream>>>(
        p->tm_xht, p->tm_xlt, p->tm_rh4, p->muf, h->n, bpc, p->cpart, p->err);
    FEM_CUDA(cudaGetLastError());
    timing_begin(h, 9);
    k_final_cov_zx<<<dim3(K, (h->d + kFCRows - 1) / kFCRows), 512, 0, h->stream>>>(p->cpart, p->cgx, p->cgy, h->d, h->psum,
                                                                          h->mu, p->muf, h->sigma);
  } else {
    k_cov_tc<<<dim3(p->cgx, p->cgy), kCThreads, csmem_bytes(), h->stream>>>(p->tm_x32, p->tm_rh4, p->tm_rl4, p->muf,
                                                                           h->n, bpc, p->cpart, p->dpart, p->err);
    FEM_CUDA(cudaGetLastError());
    timing_begin(h, 9);
    k_final_cov_tc<<<K, 256, 0, h->stream>>>(p->cpart, p->dpart, p->cgx, p->cgy, h->d, h->psum, h->sigma);
  }
  FEM_CUDA(cudaGetLastError());
  k_flag_timeout<<<1, 32, 0, h->stream>>>(h->dstat, p->err);
  h->launches += 5;
  return FEM_OK;
}

// a wait that ran out in an earlier call leaves the status word set; each new
// call starts from zero (the context itself stays usable: nothing faulted)
int em_tc_reset_err(fem_em *h) {
  if (h->wide) return em_wide_reset_err(h);
  FEM_CUDA(cudaMemsetAsync(h->tc->err, 0, sizeof(int), h->stream));
  return FEM_OK;
}

int em_tc_wait_selftest(fem_em *h, long long budget, int *roles) {
  TcEmPlan *p = h->tc;
  FEM_CUDA(cudaMemsetAsync(p->roles, 0, 4 * sizeof(int), h->stream));
  k_wait_expiry<<<1, 128, 0, h->stream>>>(budget, p->err, p->roles);
  FEM_CUDA(cudaGetLastError());
  k_flag_timeout<<<1, 32, 0, h->stream>>>(h->dstat, p->err);
  FEM_CUDA(cudaGetLastError());
  int r[4] = {0, 0, 0, 0};
  FEM_CUDA(cudaMemcpyAsync(r, p->roles, sizeof r, cudaMemcpyDeviceToHost, h->stream));
  FEM_CUDA(cudaStreamSynchronize(h->stream));
  *roles = (r[0] ? 1 : 0) | (r[1] ? 2 : 0) | (r[2] ? 4 : 0) | (r[3] ? 8 : 0);
  h->launches += 2;
  return FEM_OK;
}

int em_tc_post_rows(fem_em *h, int64_t r0, int64_t rows, double *dout) {
  if (h->wide) return em_wide_post_rows(h, r0, rows, dout);
  TcEmPlan *p = h->tc;
  const int64_t tot = rows * h->k;
  k_post_rows_tc<<<(unsigned)((tot + 255) / 256), 256, 0, h->stream>>>(p->Rh, p->Rl, p->np, h->k, r0, rows, dout);
  FEM_CUDA(cudaGetLastError());
  return FEM_OK;
}

void em_tc_posteriors(fem_em *h, const __half **rh, const __half **rl, int64_t *pitch) {
  if (h->wide) return em_wide_posteriors(h, rh, rl, pitch);
  *rh = h->tc->Rh;
  *rl = h->tc->Rl;
  *pitch = h->tc->np;
}

int em_tc_classes(fem_em *h, int32_t *dcls) {
  if (h->wide) return em_wide_classes(h, dcls);
  TcEmPlan *p = h->tc;
  k_classes_tc<<<(unsigned)((h->n + 255) / 256), 256, 0, h->stream>>>(p->Rh, p->Rl, p->np, h->n, h->k, dcls);
  FEM_CUDA(cudaGetLastError());
  return FEM_OK;
}

}  // namespace fem
