// km_tc.cu -- Lloyd k-means assignment as a tcgen05 GEMM plus argmin
// (NaiveKMA::ComputeMSEAndCorrect, Clust/KMAlgorithm.cpp:205-255, for d = 32).
//
// Distances are translation invariant, so both sides are first centred on a point g
// amid the data and scaled by a power of two that brings the rows' typical largest
// distance from it to 1/2..1: x' = t (x - g), c' = t (c - g).  (Scaled by max |x|,
// an offset or one row far out pushes all others below FP16's normal range and
// leaves them open.)  For a tile of 128 points the tensor cores form
//   D_j = x'.c'_j - ||c'_j||^2 / 2,   ||x' - c'_j||^2 = ||x'||^2 - 2 D_j,
// for all K <= 256 centroids in FP32 (TMEM), from FP16 splits:
//   A row  = [xh | xl]            (64 halves, one 128-byte swizzled row)
//   B1 row = [ch | ch], B2 row = [cl | n | 0],  n = -||c'||^2 / 256 in three parts
//   A.B2 + A.B1 = xh.cl + (xh + xl).ch,  and a constant A (128, 128, 128, 0 ...) times n
// (issued small products first).  The epilogue reads the tile's accumulator
// twice: for the largest D_j, then for one bit per centroid within a rigorous
// bound on its error (split residuals, tensor-core accumulation) of it.  A row
// with one candidate is decided; the others are decided among theirs, in the
// FP32 difference form and, where its bound leaves several, in FP64 difference
// form, index order, strict < -- the reference's rule, bit for bit.  Rows are
// then added to exact fixed-point centroid sums in shared memory, so the update
// is order independent.
//
// Warp roles (448 threads): 0 TMA, 1 MMA (TMEM owner), 2..5 operand
// producers (FP32 row -> [xh | xl], ||x||), 6..13 epilogue in two groups of
// four, one group per TMEM accumulator buffer (alternate tiles).
//
// Bound by the epilogue: instruction issue, and shared memory for the sums (64
// atomics a row) and the MMA operands.  N = 2^24, K = 256 on the GB300, ms an
// iteration: 3.51 with ||c'||^2 added per value, the three smallest kept in one
// pass and 64-bit atomics; 3.06 with two 32-bit atomics a value; 2.79 with the
// two passes; 2.47 with the rows taken from the stage before the scan (its
// three stages then no longer wait for the sums); 1.74 with ||c'||^2 / 2 from
// the tensor cores (128 16-byte loads a row less).  HBM would take 0.33.
#include <algorithm>
#include <cfloat>
#include <climits>
#include <cmath>

#include "km_kernels.cuh"
#include "tc_ptx.cuh"

namespace fem {

using namespace tc;

namespace {

constexpr int kKmD = 32;                 // dimension handled here
constexpr int kKmTile = 128;             // points per tile (MMA M)
constexpr int kKmMaxK = 256;             // centroids (MMA N)
constexpr int kKmXStages = 3;
constexpr int kKmAStages = 2;
constexpr int kKmAccPitch = kKmD + 1;    // padded rows of the fixed-point sums
constexpr int kKmThreads = 14 * 32;
constexpr uint32_t kKmXBytes = kKmTile * kKmD * 4;       // 16 KB FP32 tile
// constants of the bound (see k_km_tc_prep)
constexpr float kKmRel = 1.52587890625e-5f;               // 2^-16
constexpr float kKmRelN = 3.814697265625e-6f;             // 2^-18
constexpr float kKmAbs = 3.814697265625e-6f;              // 2^-18
constexpr int kKmMany = 16;                               // candidates that a row's dimensions are spread over lanes for
constexpr float kKmFar = 3600.f;                          // ||c'||^2 / 256 within FP16 up to 4095
constexpr int kKmInf = 0x7f800000;                        // bits of infinity
constexpr uint32_t kKmOnes = 4096;                        // constant A operand: 128 rows x 32 bytes

struct __align__(1024) KmSmem {
  __half b1[kKmMaxK * 64];                 // [ch | ch]  (SW128)
  __half b2[kKmMaxK * 64];                 // [cl | n | 0]  (SW128)
  __half a[kKmAStages][kKmTile * 64];      // [xh | xl]  (SW128)
  float x[kKmXStages][kKmTile * kKmD];     // FP32 rows  (SW128, TMA)
  long long acc[kKmMaxK * kKmAccPitch];    // fixed-point sums
  __half ones[kKmOnes / 2];                // every 16 bytes: 128 128 128 0 0 0 0 0
  float lo, hi;                            // smallest ||c'||, largest that is used
  alignas(16) float g[kKmD];               // -t g
  float slack[kKmXStages][kKmTile];        // per row of each X stage twice the bound on any D, inf: every centroid
  int cnt[kKmMaxK];
  unsigned cand[8][kKmMaxK / 32][32];      // per epilogue warp: a row's candidate centroids, 32 a word, first = top bit
  uint64_t b_full, x_full[kKmXStages], x_empty[kKmXStages], a_full[kKmAStages], a_empty[kKmAStages],
      acc_full[2], acc_empty[2], mma_done;
  uint32_t tmem_base;
};
static_assert(sizeof(KmSmem) + 1024 <= 232448, "k-means kernel shared memory");

struct KmTcPlanImpl {
  CUtensorMap tm_x, tm_b1, tm_b2;
  __half *b1 = nullptr, *b2 = nullptr;   // Kp x 64
  int *err = nullptr;
  int kp = 0;
};

__device__ __forceinline__ void fence_proxy_async_smem_km() {
  asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
}

// Centroid operands (FP64 centroids in), a warp per centroid, lane = dimension, and
// their range of norms (one CTA for all of them took 70 us at K = 256, an iteration
// over 20000 rows 167 instead of 99 us).  With N = ||c'_j||,
//   |D_j - (x'.c'_j - ||c'_j||^2 / 2)| <= B(N) = ||x'|| (2^-16 N + 2^-18) +
//                                         2^-18 N^2 / 2 + 2^-18 N + 2^-18:
// the tensor core cuts each of the 16 terms of a product and the accumulator to
// 2^-23 of the largest (7 products: 7 x 17 x 2^-23 of ||x'|| ||c'||, 17 x 2^-23
// of ||c'||^2 / 2 for the last), the splits leave 2^-22 of each side, x - g
// rounds to 2^-24, and halves below FP16's normal range are off by 2^-25: 2^-18
// of ||x'|| and N cover that of the operands, and the norm's three parts leave up
// to 2^-25 times the constant 128 however small row and centroid are.
//
// A row's nearest centroid is no farther from g than L = l + 2 ||x'||, l the
// smallest ||c'||: the centroid at l is at most l + ||x'|| away.  The rows screen
// with B(min(h, 1.01 L + 1/8)), h the largest norm used.  A centroid beyond that,
// at N, has D_j at least (0.01 N + 1/8) / 1.01 N / 2 below the one at l, more
// than B(N) and the row's bound together (||x'|| <= N / 2), so it is neither the
// largest nor the one left out, and one centroid far out does not open every row.
// Beyond kKmFar a centroid gets n of the padding, and rows that could be its
// (1.01 L + 1/8 > kKmFar: rows far out, or all centroids far outside the data) take
// every centroid as a candidate.
__global__ void __launch_bounds__(128)
k_km_tc_prep(const double *__restrict__ cent, const float *__restrict__ g, const float *__restrict__ xscale, int K, int Kp,
             __half *__restrict__ b1, __half *__restrict__ b2, int *__restrict__ range) {
  const int j = blockIdx.x * 4 + (threadIdx.x >> 5), lane = threadIdx.x & 31;
  if (j >= Kp) return;
  double c = j < K ? (double)*xscale * (cent[(size_t)j * kKmD + lane] - (double)g[lane]) : 0.0, n = c * c;
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) n += __shfl_xor_sync(0xffffffffu, n, o);
  const float nrm = (float)sqrt(n);
  const bool used = j < K && nrm <= kKmFar;
  if (!used) c = 0.0;
  const __half ch = __double2half(c);
  b1[(size_t)j * 64 + lane] = b1[(size_t)j * 64 + 32 + lane] = ch;              // [ch | ch]
  b2[(size_t)j * 64 + lane] = __double2half(c - (double)__half2float(ch));      // [cl | n | 0]
  n = used ? -n / 256.0 : -65504.0;
  __half part = __float2half(0.f);
  for (int u = 0; u < 3; u++) {
    const __half h = __double2half(n);
    if (lane == u) part = h;
    n = used ? n - (double)__half2float(h) : 0.0;
  }
  b2[(size_t)j * 64 + 32 + lane] = part;
  // non-negative floats order like their bits; both start at zero
  if (lane == 0 && j < K && nrm >= 0.f) {
    atomicMax(range, kKmInf - __float_as_int(nrm));
    if (used) atomicMax(range + 1, __float_as_int(nrm));
  }
}

// bound on the distance of an FP32 difference-form sum (any order) from the exact value
__device__ __forceinline__ float km_bound32(float s, float cn) {
  const float u = 5.9604645e-8f;  // 2^-24
  return 2.f * ((float)(kKmD + 4) * u * s + 2.01f * u * sqrtf(fmaxf(s, 0.f)) * cn + u * u * cn * cn) + 1e-30f;
}

template <bool W32>
__global__ void __launch_bounds__(kKmThreads, 1)
k_km_assign_tc(const __grid_constant__ CUtensorMap tm_x, const __grid_constant__ CUtensorMap tm_b1,
               const __grid_constant__ CUtensorMap tm_b2, const int *__restrict__ range,
               const double *__restrict__ cent, const float *__restrict__ centf,
               const float *__restrict__ cnorm, const float *__restrict__ X, const float *__restrict__ gs, int64_t n,
               int K, int Kp, const float *__restrict__ xscale_at, int32_t *__restrict__ labels,
               long long *__restrict__ accg, int *__restrict__ cntg, float scale, float scale_hi, int lo_bits,
               int64_t epoch, DevStatus *st, int *err) {
  extern __shared__ uint8_t smem_raw[];
  KmSmem &S = smem_aligned<KmSmem>(smem_raw);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const float xscale = *xscale_at;
  const int64_t ntiles = (n + kKmTile - 1) / kKmTile;
  const int64_t mine = ntiles > blockIdx.x ? (ntiles - 1 - blockIdx.x) / gridDim.x + 1 : 0;

  for (int e = threadIdx.x; e < kKmMaxK * kKmAccPitch; e += blockDim.x) S.acc[e] = 0;
  for (int j = threadIdx.x; j < kKmMaxK; j += blockDim.x) S.cnt[j] = 0;
  for (uint32_t e = threadIdx.x; e < kKmOnes / 2; e += blockDim.x) S.ones[e] = __float2half((e & 7) < 3 ? 128.f : 0.f);
  fence_proxy_async_smem_km();
  if (threadIdx.x < kKmD) S.g[threadIdx.x] = -xscale * gs[threadIdx.x];
  if (threadIdx.x == 0) {
    S.lo = __int_as_float(kKmInf - range[0]);
    S.hi = __int_as_float(range[1]);
    mbar_init(&S.b_full, 1);
    for (int s = 0; s < kKmXStages; s++) mbar_init(&S.x_full[s], 1), mbar_init(&S.x_empty[s], 4);
    for (int s = 0; s < kKmAStages; s++) mbar_init(&S.a_full[s], 4), mbar_init(&S.a_empty[s], 1);
    for (int s = 0; s < 2; s++) mbar_init(&S.acc_full[s], 1), mbar_init(&S.acc_empty[s], 4);
    mbar_init(&S.mma_done, 1);
    fence_mbar_init();
  }
  if (warp == 1) tmem_alloc(&S.tmem_base, 512);
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tbase = S.tmem_base;

  if (warp == 0) {
    // ------------------------------------------------ TMA
    if (elect_one()) {
      tma_prefetch_desc(&tm_x);
      mbar_expect_tx(&S.b_full, 2u * Kp * 128u);
      tma_load_2d(S.b1, &tm_b1, &S.b_full, 0, 0);
      tma_load_2d(S.b2, &tm_b2, &S.b_full, 0, 0);
      bool ok = true;
      for (int64_t i = 0; i < mine && ok; i++) {
        const int s = (int)(i % kKmXStages);
        if (!(ok = mbar_wait_lazy(&S.x_empty[s], ((i / kKmXStages) & 1) ^ 1, err, 64))) break;
        mbar_expect_tx(&S.x_full[s], kKmXBytes);
        tma_load_2d(S.x[s], &tm_x, &S.x_full[s], 0, (int)((blockIdx.x + i * gridDim.x) * kKmTile));
      }
      mbar_wait_drain(&S.b_full, 0);
      for (int64_t u = mine - 1; u >= 0 && u >= mine - kKmXStages; u--)
        mbar_wait_drain(&S.x_full[u % kKmXStages], (u / kKmXStages) & 1);
    }
  } else if (warp == 1) {
    // ------------------------------------------------ MMA issuer
    if (elect_one()) {
      bool ok = mbar_wait(&S.b_full, 0, err);
      tc_fence_after();
      const uint64_t db1 = sdesc_sw128(smem_u32(S.b1)), db2 = sdesc_sw128(smem_u32(S.b2));
      const uint32_t idesc = idesc_f16(kKmTile, Kp);
      // the constant operand has no swizzle: 8-row x 16-byte core matrices, 128
      // bytes apart along K, 256 along the rows
      const uint64_t dones = ((uint64_t)(smem_u32(S.ones) & 0x3FFFF) >> 4) | (uint64_t)(128 >> 4) << 16 |
                             (uint64_t)(256 >> 4) << 32 | (uint64_t)1 << 46;
      for (int64_t i = 0; i < mine && ok; i++) {
        const int as = (int)(i % kKmAStages), ab = (int)(i & 1);
        if (!(ok = mbar_wait(&S.acc_empty[ab], ((i >> 1) & 1) ^ 1, err))) break;
        if (!(ok = mbar_wait(&S.a_full[as], (i / kKmAStages) & 1, err))) break;
        tc_fence_after();
        const uint64_t da = sdesc_sw128(smem_u32(S.a[as]));
        const uint32_t d = tbase + ab * kKmMaxK;
        // xh.cl (k-blocks 0, 1 of B2), xl.ch (k-blocks 2, 3 of B1), xh.ch (0, 1 of B1)
        mma_f16(d, da + 0, db2 + 0, idesc, 0);
        mma_f16(d, da + 2, db2 + 2, idesc, 1);
        mma_f16(d, da + 4, db1 + 4, idesc, 1);
        mma_f16(d, da + 6, db1 + 6, idesc, 1);
        mma_f16(d, da + 0, db1 + 0, idesc, 1);
        mma_f16(d, da + 2, db1 + 2, idesc, 1);
        mma_f16(d, dones, db2 + 4, idesc, 1);      // n (k-block 2 of B2)
        mma_commit(&S.a_empty[as]);
        mma_commit(&S.acc_full[ab]);
      }
      mma_commit(&S.mma_done);
      mbar_wait_drain(&S.mma_done, 0);
    }
  } else if (warp < 6) {
    // ------------------------------------------------ producers: row r
    const int r = (warp - 2) * 32 + lane;
    bool ok = true;
    for (int64_t i = 0; i < mine && ok; i++) {
      const int s = (int)(i % kKmXStages), as = (int)(i % kKmAStages);
      // (sleeping: they have slack, and polling takes issue slots from the epilogue)
      if (!(ok = mbar_wait_lazy_warp(&S.x_full[s], (i / kKmXStages) & 1, err, 64))) break;
      if (!(ok = mbar_wait_lazy_warp(&S.a_empty[as], ((i / kKmAStages) & 1) ^ 1, err, 64))) break;
      const float4 *xr = reinterpret_cast<const float4 *>(S.x[s] + r * kKmD);
      uint4 *ar = reinterpret_cast<uint4 *>(S.a[as] + r * 64);
      float ss = 0.f;
#pragma unroll
      for (int c2 = 0; c2 < 4; c2++) {          // 8 floats -> one 16-byte chunk of xh and of xl
        const float4 u = xr[(2 * c2) ^ (r & 7)];
        const float4 w = xr[(2 * c2 + 1) ^ (r & 7)];
        const float4 g0 = *reinterpret_cast<const float4 *>(S.g + 8 * c2), g1 = *reinterpret_cast<const float4 *>(S.g + 8 * c2 + 4);
        // t (x - g): one rounding, t is a power of two
        const float v[8] = {fmaf(u.x, xscale, g0.x), fmaf(u.y, xscale, g0.y), fmaf(u.z, xscale, g0.z),
                            fmaf(u.w, xscale, g0.w), fmaf(w.x, xscale, g1.x), fmaf(w.y, xscale, g1.y),
                            fmaf(w.z, xscale, g1.z), fmaf(w.w, xscale, g1.w)};
        uint32_t hh[4], ll[4];
#pragma unroll
        for (int e = 0; e < 4; e++) {
          const __half2 h = __floats2half2_rn(v[2 * e], v[2 * e + 1]);
          const float2 hf = __half22float2(h);
          const __half2 l = __floats2half2_rn(v[2 * e] - hf.x, v[2 * e + 1] - hf.y);
          hh[e] = *reinterpret_cast<const uint32_t *>(&h);
          ll[e] = *reinterpret_cast<const uint32_t *>(&l);
          ss = fmaf(v[2 * e], v[2 * e], ss);
          ss = fmaf(v[2 * e + 1], v[2 * e + 1], ss);
        }
        ar[c2 ^ (r & 7)] = make_uint4(hh[0], hh[1], hh[2], hh[3]);
        ar[(4 + c2) ^ (r & 7)] = make_uint4(ll[0], ll[1], ll[2], ll[3]);
      }
      // the row's bound on D (see k_km_tc_prep), ||x'|| rounded up a little; here,
      // since the epilogue has no issue slots to spare
      const float xn = sqrtf(ss) * 1.00001f, reach = fmaf(1.01f, fmaf(2.f, xn, S.lo), 0.125f), cn = fminf(S.hi, reach);
      const float bound = fmaf(xn, fmaf(kKmRel, cn, kKmAbs), fmaf(fmaf(0.5f * kKmRelN, cn, kKmAbs), cn, kKmAbs));
      S.slack[s][r] = reach <= kKmFar ? 2.01f * bound : INFINITY;      // (a row with NaN: every centroid)
      fence_proxy_async_smem_km();
      __syncwarp();
      if (lane == 0) mbar_arrive(&S.a_full[as]);
    }
  } else {
    // ------------------------------------------------ epilogue: group g, TMEM lanes of warp % 4
    const int g = (warp - 6) >> 2, quad = warp & 3;
    const int r = quad * 32 + lane;
    const uint32_t lane_addr = (uint32_t)(quad * 32) << 16;
    int64_t rechecks = 0;
    bool ok = true;
    const bool track = st->track_changes;
    int *acch = reinterpret_cast<int *>(S.acc), *accl = acch + kKmMaxK * kKmAccPitch;
    const float scale_lo = __int_as_float((lo_bits + 127) << 23);   // 2^lo_bits
    constexpr float kMagic = 12582912.f;                            // 1.5 2^23
    for (int64_t e0 = 0; e0 < mine; e0 += epoch) {
    const int64_t e1 = min(mine, e0 + epoch);
    for (int64_t i = e0 + g; i < e1 && ok; i += 2) {
      const int s = (int)(i % kKmXStages);
      if (!(ok = mbar_wait_warp(&S.acc_full[g], (i >> 1) & 1, err))) break;
      tc_fence_after();
      // the warp's 32 rows, lane = dimension, for the sums: taken now, so that the
      // stage is free for the next copy while this tile is scanned
      const float slack = S.slack[s][r];
      float xr[32];
#pragma unroll
      for (int rr = 0; rr < 32; rr++) {
        const int rq = quad * 32 + rr;
        xr[rr] = S.x[s][rq * kKmD + ((((lane >> 2) ^ (rq & 7)) << 2) + (lane & 3))];
      }
      __syncwarp();
      if (lane == 0) mbar_arrive(&S.x_empty[s]);
      // first the largest D_j, then a bit for every centroid within the bounds
      // of it: a sign per value, shifted into the word
      const uint32_t dcol = tbase + lane_addr + g * kKmMaxK;
      float m[4] = {-INFINITY, -INFINITY, -INFINITY, -INFINITY};
#pragma unroll 1
      for (int c0 = 0; c0 < Kp; c0 += 64) {
        uint32_t dv[64];
        tmem_ld64(dcol + c0, dv);
        tmem_wait_ld();
        const int cols = Kp - c0;                   // a multiple of 16
#pragma unroll
        for (int t = 0; t < 64; t += 16) {
          if (t >= cols) break;
#pragma unroll
          for (int e = 0; e < 16; e++) m[e & 3] = fmaxf(m[e & 3], __uint_as_float(dv[t + e]));
        }
      }
      const float mv = fmaxf(fmaxf(m[0], m[1]), fmaxf(m[2], m[3]));
      const int64_t row = (blockIdx.x + i * gridDim.x) * kKmTile + r;
      // the winner's exact value is at least mv - bound, so the reference's
      // choice has D > thr
      const float thr = mv - slack;
      const bool all = !(slack < INFINITY);
      const float2 thr2 = make_float2(thr, thr), neg = make_float2(-1.f, -1.f);
      unsigned (*cw)[32] = S.cand[warp - 6];
      int cnt = 0, lab = -1;
#pragma unroll 1
      for (int c0 = 0; c0 < Kp; c0 += 64) {
        uint32_t dv[64];
        tmem_ld64(dcol + c0, dv);
        tmem_wait_ld();
#pragma unroll
        for (int hw = 0; hw < 2; hw++) {
          unsigned b8[4] = {0, 0, 0, 0};           // four chains of eight bits
#pragma unroll
          for (int u = 0; u < 4; u++)
#pragma unroll
            for (int t = 32 * hw + 8 * u; t < 32 * hw + 8 * u + 8; t += 2) {
              const float2 v = __ffma2_rn(make_float2(__uint_as_float(dv[t]), __uint_as_float(dv[t + 1])), neg, thr2);
              b8[u] = __funnelshift_l(__float_as_uint(v.x), b8[u], 1);
              b8[u] = __funnelshift_l(__float_as_uint(v.y), b8[u], 1);
            }
          unsigned word = (b8[0] << 24) | (b8[1] << 16) | (b8[2] << 8) | b8[3];
          // columns past K (padding, and what an unused column last held)
          const int left = K - c0 - 32 * hw;
          if (all) word = 0xffffffffu;
          word &= left >= 32 ? 0xffffffffu : ~(0xffffffffu >> max(left, 0));
          cw[(c0 >> 5) + hw][lane] = word;
          cnt += __popc(word);
          if (word) lab = c0 + 32 * hw + __clz(word);
        }
      }
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(&S.acc_empty[g]);

      // rows with several candidates, by the whole warp (lane = dimension):
      // FP32 difference form with its bound, then the reference's FP64 sums
      // among what that leaves (index order, strict <)
      for (unsigned open = __ballot_sync(0xffffffffu, row < n && cnt > 1); open; open &= open - 1) {
        const int b = __ffs(open) - 1;
        const float xv = __ldg(X + (row - lane + b) * kKmD + lane);
        if (__shfl_sync(0xffffffffu, cnt, b) > kKmMany) {
          // the same over all centroids, lane = centroid: a row far outside the data
          // has every one as its candidate, a chain of K reductions the other way
          auto dist32 = [&](int j) {
            float s = 0.f;
#pragma unroll 8
            for (int q = 0; q < kKmD; q++) {
              const float t = __shfl_sync(0xffffffffu, xv, q) - centf[(size_t)min(j, K - 1) * kKmD + q];
              s = fmaf(t, t, s);
            }
            return s;
          };
          float U = INFINITY;
          for (int j0 = 0; j0 < K; j0 += 32) {
            const float s = dist32(j0 + lane);
            if (j0 + lane < K) U = fminf(U, s + km_bound32(s, cnorm[j0 + lane]));
          }
#pragma unroll
          for (int o = 16; o > 0; o >>= 1) U = fminf(U, __shfl_xor_sync(0xffffffffu, U, o));
          double best = DBL_MAX;
          int l = INT_MAX;
          for (int j0 = 0; j0 < K; j0 += 32) {
            const int j = j0 + lane;
            const float s = dist32(j);
            const bool in = j < K && s - km_bound32(s, cnorm[min(j, K - 1)]) <= U;
            if (!__any_sync(0xffffffffu, in)) continue;
            double d64 = 0.0;
#pragma unroll 4
            for (int q = 0; q < kKmD; q++) {
              const double t = __dsub_rn(cent[(size_t)min(j, K - 1) * kKmD + q], (double)__shfl_sync(0xffffffffu, xv, q));
              d64 = __dadd_rn(d64, __dmul_rn(t, t));
            }
            if (in && d64 < best) best = d64, l = j;     // a lane's centroids come in index order
          }
#pragma unroll
          for (int o = 16; o > 0; o >>= 1) {
            const double ob = __shfl_xor_sync(0xffffffffu, best, o);
            const int ol = __shfl_xor_sync(0xffffffffu, l, o);
            if (ob < best || (ob == best && ol < l)) best = ob, l = ol;
          }
          if (lane == b) lab = l == INT_MAX ? -1 : l;
          continue;
        }
        auto dist = [&](int j) {
          const float t = xv - centf[(size_t)j * kKmD + lane];
          float sj = t * t;
#pragma unroll
          for (int o = 16; o > 0; o >>= 1) sj += __shfl_xor_sync(0xffffffffu, sj, o);
          return sj;
        };
        float U = INFINITY, l1 = INFINITY, l2 = INFINITY;
        int l = -1;
        for (int w = 0; 32 * w < Kp; w++)
          for (unsigned bits = cw[w][b]; bits;) {
            const int z = __clz(bits), j = 32 * w + z;
            bits &= ~(0x80000000u >> z);
            const float sj = dist(j), e = km_bound32(sj, cnorm[j]), lb = sj - e;
            U = fminf(U, sj + e);
            if (lb < l1)
              l2 = l1, l1 = lb, l = j;
            else
              l2 = fminf(l2, lb);
          }
        if (!(l2 > U)) {
          double best = DBL_MAX;
          for (int w = 0; 32 * w < Kp; w++)
            for (unsigned bits = cw[w][b]; bits;) {
              const int z = __clz(bits), j = 32 * w + z;
              bits &= ~(0x80000000u >> z);
              const float sj = dist(j);
              if (!(sj - km_bound32(sj, cnorm[j]) <= U)) continue;
              double d64 = 0.0;
              for (int q = 0; q < kKmD; q++) {
                const double t = __dsub_rn(cent[(size_t)j * kKmD + q], (double)__shfl_sync(0xffffffffu, xv, q));
                d64 = __dadd_rn(d64, __dmul_rn(t, t));
              }
              if (d64 < best) best = d64, l = j;
            }
        }
        if (lane == b) lab = l;
      }
      if (row < n) {
        if (cnt != 1) rechecks++;
        if (track && labels[row] != lab) st->changed = 1;
        labels[row] = lab;
        if (lab >= 0) atomicAdd(&S.cnt[lab], 1);      // -1: a row with NaN
      }
      // exact fixed-point sums, one row of the warp at a time: lane q adds
      // dimension q, so each atomic instruction updates 32 consecutive words of
      // one centroid row (conflict-free) instead of 32 scattered rows.  W32: the
      // integer x 2^shift = hi 2^lo_bits + lo goes into two 32-bit sums (native
      // atomics; hi = x scale_hi rounded, lo the rest, both exact), which are
      // moved to the 64-bit sums in global memory every `epoch` tiles, before
      // either can overflow
      {
        const int mylab = row < n ? lab : -1;
        if constexpr (W32) {
          // without branches, so that the rows' loads and sums overlap: a row
          // that counts nowhere adds zeros to centroid 0
#pragma unroll
          for (int rr = 0; rr < 32; rr++) {
            const int l = __shfl_sync(0xffffffffu, mylab, rr);
            const float xv = l >= 0 ? xr[rr] : 0.f;
            const float hm = fmaf(xv, scale_hi, kMagic), hf = hm - kMagic;
            const float lm = fmaf(fmaf(xv, scale_hi, -hf), scale_lo, kMagic);
            int *o = acch + max(l, 0) * kKmAccPitch + lane;
            atomicAdd(o, __float_as_int(hm) - __float_as_int(kMagic));
            atomicAdd(o + kKmMaxK * kKmAccPitch, __float_as_int(lm) - __float_as_int(kMagic));
          }
        } else {
#pragma unroll
          for (int rr = 0; rr < 32; rr++) {
            const int l = __shfl_sync(0xffffffffu, mylab, rr);
            if (l >= 0)
              atomicAdd(reinterpret_cast<unsigned long long *>(S.acc + l * kKmAccPitch + lane),
                        (unsigned long long)__float2ll_rn(xr[rr] * scale));
          }
        }
      }
    }
    if constexpr (W32) {
      // all eight warps come here once per epoch, also when a wait gave up
      ok = bar_and(1, 256, ok);
      long long *o = accg + (size_t)blockIdx.x * K * kKmD;
#pragma unroll 4
      for (int e = threadIdx.x - 6 * 32; e < K * kKmD; e += 256) {
        const int w = (e / kKmD) * kKmAccPitch + e % kKmD;
        const long long v = ((long long)acch[w] << lo_bits) + accl[w];
        acch[w] = 0, accl[w] = 0;
        o[e] = e0 == 0 ? v : o[e] + v;
      }
      ok = bar_and(1, 256, ok);
    }
    if (!ok) break;
    }
    if (rechecks) atomicAdd((unsigned long long *)&st->rechecked, (unsigned long long)rechecks);
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  if (warp == 1) tmem_dealloc(tbase, 512);
  // per-CTA partials in the layout k_km_final reads: [cta][j][q], [cta][j]
  if (!W32 || mine == 0)
    for (int e = threadIdx.x; e < K * kKmD; e += blockDim.x) {
      const int j = e / kKmD, q = e - j * kKmD;
      accg[(size_t)blockIdx.x * K * kKmD + e] = W32 ? 0 : S.acc[j * kKmAccPitch + q];
    }
  for (int j = threadIdx.x; j < K; j += blockDim.x) cntg[(size_t)blockIdx.x * K + j] = S.cnt[j];
}

__global__ void k_km_tc_flag(DevStatus *st, const int *__restrict__ err) {
  if (*err) st->timeout = 1;
}

}  // namespace

bool km_tc_supported(int d, int k) { return d == kKmD && k >= 1 && k <= kKmMaxK; }

int km_tc_create(fem_km *h) {
  KmTcPlanImpl *p = new (std::nothrow) KmTcPlanImpl();
  if (!p) return FEM_ERR_BAD_ARG;
  h->tc = p;
  p->kp = (h->k + 15) / 16 * 16;
  FEM_TRY(dalloc(&p->b1, (size_t)p->kp * 64));
  FEM_TRY(dalloc(&p->b2, (size_t)p->kp * 64));
  FEM_TRY(dalloc(&p->err, 1));
  FEM_CUDA(cudaMemset(p->err, 0, sizeof(int)));
  FEM_TRY(encode_tmap_2d(&p->tm_x, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 4, h->X, kKmD, (uint64_t)h->n, kKmD,
                         kKmTile, CU_TENSOR_MAP_SWIZZLE_128B));
  FEM_TRY(encode_tmap_2d(&p->tm_b1, CU_TENSOR_MAP_DATA_TYPE_FLOAT16, 2, p->b1, 64, (uint64_t)p->kp, 64, p->kp,
                         CU_TENSOR_MAP_SWIZZLE_128B));
  FEM_TRY(encode_tmap_2d(&p->tm_b2, CU_TENSOR_MAP_DATA_TYPE_FLOAT16, 2, p->b2, 64, (uint64_t)p->kp, 64, p->kp,
                         CU_TENSOR_MAP_SWIZZLE_128B));
  FEM_CUDA(cudaFuncSetAttribute(k_km_assign_tc<false>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                (int)(sizeof(KmSmem) + 1024)));
  FEM_CUDA(cudaFuncSetAttribute(k_km_assign_tc<true>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                (int)(sizeof(KmSmem) + 1024)));
  return FEM_OK;
}

void km_tc_destroy(fem_km *h) {
  KmTcPlanImpl *p = static_cast<KmTcPlanImpl *>(h->tc);
  if (!p) return;
  dfree(p->b1);
  dfree(p->b2);
  dfree(p->err);
  delete p;
  h->tc = nullptr;
}

int km_tc_assign(fem_km *h) {
  KmTcPlanImpl *p = static_cast<KmTcPlanImpl *>(h->tc);
  int xe = 0;
  std::frexp((double)std::max(h->xmax, 1e-25f), &xe);      // |x| <= xmax < 2^xe
  k_km_tc_prep<<<p->kp / 4, 128, 0, h->stream>>>(h->cent, h->gs, h->xscale, h->k, p->kp, p->b1, p->b2, h->range);
  FEM_CUDA(cudaGetLastError());
  // |x| 2^shift < 2^bits: hi takes bits / 2 of them, lo the lo_bits below; both
  // sums stay within 32 bits for `rows` rows of one centroid.  From 1024 rows on
  // (datasets above about 250,000 rows; the shift is capped below) the 32-bit
  // sums are ahead: N = 2^24, K = 256, 3.5 -> 3.06 ms with nothing else changed.
  const int bits = xe + h->shift, hi_bits = bits / 2, lo_bits = bits - hi_bits;
  const int64_t rows = bits >= 4 ? (int64_t)1 << std::min(31 - hi_bits, 32 - lo_bits) : 0;
  const bool w32 = rows >= 1024 && hi_bits - xe < 100 && hi_bits - xe > -100;
  const int64_t epoch = w32 ? rows / kKmTile / 2 * 2 - 2 : h->n;   // even: the two groups alternate
#define FEM_KT(W)                                                                                                \
  k_km_assign_tc<W><<<h->grid, kKmThreads, sizeof(KmSmem) + 1024, h->stream>>>(                                  \
      p->tm_x, p->tm_b1, p->tm_b2, h->range, h->cent, h->centf, h->cnorm, h->X, h->gs, h->n, h->k, p->kp,        \
      h->xscale, h->labels, h->acc, h->cnt, ldexpf(1.f, h->shift), ldexpf(1.f, hi_bits - xe), lo_bits, epoch, h->dstat, p->err)
  if (w32)
    FEM_KT(true);
  else
    FEM_KT(false);
#undef FEM_KT
  FEM_CUDA(cudaGetLastError());
  k_km_tc_flag<<<1, 1, 0, h->stream>>>(h->dstat, p->err);
  FEM_CUDA(cudaGetLastError());
  return FEM_OK;
}

}  // namespace fem
