// Complex128 GEMM on the 5th-generation tensor cores: C = +-A B (+ C) with FP64
// accuracy from FP16 digits (the error-free splitting of Ozaki, Ogita, Oishi and
// Rump, "Error-free transformations of matrix multiplication by using fast
// routines", Numer. Algorithms 59, 2012, in the fixed-point form with one
// exponent per row of A and column of B).
//
// A complex product is one real product of the interleaved rows of A (2K reals)
// with the expanded columns B' (two real columns per complex one, as in
// tc_gemm.cu).  Every row of A and column of B is scaled by a power of two so
// that its entries are 63-bit integers X (largest below 2^62, rounded to nearest:
// 2^-62 of the largest entry at most), and cut into eight signed base-256 digits,
// X = sum_i q_i 256^(7-i), |q_i| <= 128, exact in FP16.  The products of digit
// slices i and j with i + j = l <= 8 are accumulated in FP32 in one tensor-memory
// accumulator per level l: sums of at most 8 * 128 products of at most 2^14,
// integers up to 2^24, so every sum is exact.  The epilogue adds the nine levels
// as integers, sum_l a_l 256^(7-l), rounds once to a double, applies the two
// exponents and adds C with one FP64 addition per value.
//
// Accuracy.  In units of 2^ea 2^eb (the row of A below 2^ea, the column of B below
// 2^eb) the rounding of the operands is at most 2^-63 (Sa + Sb), Sa and Sb the sums
// of their moduli (up to 2K each), and the dropped levels (l >= 9) at most
// 2^-60.4 K / 64: of the size of the operands' largest entries, not of the terms of
// this result.  An FP64 sum is bounded term by term, by 2K 2^-53 sum_k |a_k| |b_k|.
// So an entry is kept only where the first bound is within the second, |c| or one
// of two terms of the sum standing for it from below; every other entry (rows or
// columns whose entries differ by many powers of two where the other operand's
// large entries meet small ones) is computed again in FP64 by the epilogue, from A
// and B themselves.  On the matrices of uniform meshes that is 0.01 % of the entries of
// the rank updates and 2 % of those of the panels of Sigma; where two particles' sizes
// differ by 30 (areas by 1000) 2 to 14 % and 20 %.
//
// Why: FP64 runs at two multiply-adds per clock and SM here (1.25 TFLOP/s), the FP16
// tensor cores 1500 times as fast; the 43 exact slice products, and an epilogue that
// needs one FP64 operation per value and 64-deep product instead of 128, are still far
// less.  Alone on the GPU 27 us instead of 277 us at 508 x 508 x 64, 70 to 75 instead of
// 1070 at 1350 x 1350, 418 to 448 instead of 7180 at 4000 x 4000 (36 products of slice
// pairs with one instruction each, on 64-column tiles, took 35, 86 and 496).  Where every
// entry is computed again: 226, 1440 and 11 400 us.
//
// Tile: 128 rows x 32 real columns, nine accumulators of 32 columns side by side in
// tensor memory, K chunks of 32 halves (64-byte swizzle rows) of all sixteen slices
// (80 KB), two of them in flight.  The slices of B lie one after the other in shared
// memory, so one instruction multiplies slice i of A with slices 0 .. 8 - i of B into
// levels i .. 8: eight instructions per 16 halves instead of 43.  Roles as in
// tc_gemm.cu: TMA producer, MMA issuer, eight epilogue warps (two per scheduler, so
// that one converts while the other waits for FP64); persistent with a tile counter.
#include <cuda.h>
#include <cuda_fp16.h>
#include <cudaTypedefs.h>

#include <algorithm>

#include "profile.cuh"
#include "tc_gemm.cuh"
#include "tc_prims.cuh"

namespace mnpbem {

constexpr int Z_S = 8;                                  // digit slices
constexpr int Z_L = Z_S + 1;                            // levels kept
constexpr int Z_KR = 2 * TC64_K;                        // reals per row of A
constexpr int Z_BM = 128, Z_BN = 32, Z_BK = 32, Z_KT = Z_KR / Z_BK;
constexpr int Z_A_BYTES = Z_BM * Z_BK * 2, Z_B_BYTES = Z_BN * Z_BK * 2;
constexpr int Z_STAGE = Z_S * (Z_A_BYTES + Z_B_BYTES);  // 80 KB
constexpr int Z_ST = 2;
constexpr int Z_EPI = 8;                                // epilogue warps: two per 32 rows, half of the columns each
constexpr int Z_CH = 8;                                 // columns per epilogue step
static_assert(Z_CH == 8 && Z_S == 8, "tmem_ld_levels");
static_assert(Z_L * Z_BN <= 512 && Z_BN * Z_S <= 256, "accumulators, columns of one instruction");
constexpr int Z_THREADS = 32 * (2 + Z_EPI);
constexpr int Z_SMEM = Z_ST * Z_STAGE + Z_EPI * 32 * Z_CH * 8 + 1024;
__device__ __forceinline__ constexpr uint32_t z_idesc(int n) {
  return (1u << 4) | ((uint32_t)(n >> 3) << 17) | ((uint32_t)(Z_BM >> 4) << 24);
}
constexpr int Z_NAN = 1 << 28;                          // exponent of a row / column with a non-finite entry

// ------------------------------------------------------------ digit slices
// |x| as an integer key: larger magnitude, larger key
__device__ __forceinline__ unsigned long long mag_bits(double x) {
  return (unsigned long long)__double_as_longlong(x) & 0x7fffffffffffffffull;
}
// exponent e with max < 2^e from the bits of the largest magnitude (0 for a zero row)
__device__ __forceinline__ int row_exp(unsigned long long mx) {
  const int be = (int)(mx >> 52);
  if (mx == 0) return 0;
  if (be == 0x7ff) return Z_NAN;
  if (be == 0) return -1074 + 64 - __clzll((long long)mx);      // subnormal: the position of its top bit
  return be - 1022;
}
// x 2^(62 - e) rounded to nearest, as an integer (|x| < 2^e)
__device__ __forceinline__ long long fixed62(double x, int e) {
  const unsigned long long b = mag_bits(x);
  const int be = (int)(b >> 52);
  const unsigned long long m = be ? ((b & 0xfffffffffffffull) | 0x10000000000000ull) : b;
  const int sh = (be ? be : 1) - 1075 + 62 - e;                 // x = m 2^(be - 1075); sh <= 9
  unsigned long long r;
  if (sh >= 0) r = m << sh;
  else if (sh >= -53) r = (m + (1ull << (-sh - 1))) >> -sh;
  else r = 0;
  return __double_as_longlong(x) < 0 ? -(long long)r : (long long)r;
}
// signed base-256 digits, q[0] the most significant
__device__ __forceinline__ void digits(long long v, int (&q)[Z_S]) {
#pragma unroll
  for (int s = Z_S - 1; s > 0; --s) {
    const int d = (int)(signed char)(v & 0xff);
    q[s] = d;
    v = (v - d) >> 8;
  }
  q[0] = (int)v;                                                // |v| <= 2^62 / 256^7 + 1
}

// what the epilogue needs of a row of A or a column of B: its exponent, the sum of
// its moduli over 2^e (real and imaginary parts apart; 0 for a zero or non-finite one)
// and the position of its largest entry
struct SliceInfo {
  int e;
  float sum;
  int k, pad;
};
// all lanes of a warp: v[u] the entry at lane + 32 u.  Digits of both parts.
__device__ __forceinline__ SliceInfo slice_entries(const double2 (&v)[2], int lane, int (&qr)[2][Z_S],
                                                   int (&qi)[2][Z_S]) {
  unsigned long long m[2];
#pragma unroll
  for (int u = 0; u < 2; ++u) m[u] = max(mag_bits(v[u].x), mag_bits(v[u].y));
  unsigned long long mx = max(m[0], m[1]);
#pragma unroll
  for (int o = 16; o; o >>= 1) mx = max(mx, __shfl_xor_sync(0xffffffffu, mx, o));
  const unsigned b0 = __ballot_sync(0xffffffffu, m[0] == mx), b1 = __ballot_sync(0xffffffffu, m[1] == mx);
  SliceInfo s;
  s.e = row_exp(mx);
  s.k = b0 ? __ffs(b0) - 1 : 31 + __ffs(b1);
  s.pad = 0;
  const bool fin = s.e != Z_NAN;
  float sum = 0.f;
#pragma unroll
  for (int u = 0; u < 2; ++u) {
    const long long xr = fin ? fixed62(v[u].x, s.e) : 0, xi = fin ? fixed62(v[u].y, s.e) : 0;
    sum += (fabsf(__ll2float_rn(xr)) + fabsf(__ll2float_rn(xi))) * 0x1p-62f;
    digits(xr, qr[u]);
    digits(xi, qi[u]);
  }
#pragma unroll
  for (int o = 16; o; o >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, o);
  s.sum = sum;
  return s;
}

// A [M][K] -> a8 [S][M][Z_KR] (slice s of row i: digit s of its 2K reals, zero
// beyond), ea [M].  One warp per row.
__global__ void __launch_bounds__(256) k_slice_a(const double2* __restrict__ A, int64_t lda, int M, int K,
                                                 __half* __restrict__ a8, SliceInfo* __restrict__ ea, int* tile_ctr) {
  if (blockIdx.x == 0 && threadIdx.x == 0) *tile_ctr = 0;   // of the product that follows
  const int row = blockIdx.x * 8 + (threadIdx.x >> 5), lane = threadIdx.x & 31;
  if (row >= M) return;
  double2 v[2];
#pragma unroll
  for (int u = 0; u < 2; ++u) {
    const int k = lane + 32 * u;
    v[u] = k < K ? A[(int64_t)row * lda + k] : make_double2(0, 0);
  }
  int qr[2][Z_S], qi[2][Z_S];
  const SliceInfo si = slice_entries(v, lane, qr, qi);
  if (lane == 0) ea[row] = si;
#pragma unroll
  for (int u = 0; u < 2; ++u)
#pragma unroll
    for (int s = 0; s < Z_S; ++s)
      reinterpret_cast<__half2*>(a8 + ((int64_t)s * M + row) * Z_KR)[lane + 32 * u] =
          __halves2half2(__int2half_rn(qr[u][s]), __int2half_rn(qi[u][s]));
}

// B [K][N] -> b8 [S][2N][Z_KR]: row 2j holds (Re b, -Im b) of column j, row 2j + 1
// (Im b, Re b); eb [N]; and a copy bc [K][N], from which the epilogue computes entries
// again (C may overlap B).  CTA of 256 threads = 16 columns: the block of B through
// shared memory, then one warp per column at a time, lanes along k.
constexpr int ZB_COLS = 16;
__global__ void __launch_bounds__(256) k_slice_b(const double2* __restrict__ B, int64_t ldb, int K, int N,
                                                 __half* __restrict__ b8, SliceInfo* __restrict__ eb,
                                                 double2* __restrict__ bc) {
  __shared__ double2 t[TC64_K][ZB_COLS + 1];
  const int j0 = blockIdx.x * ZB_COLS;
  for (int e = threadIdx.x; e < TC64_K * ZB_COLS; e += 256) {
    const int k = e / ZB_COLS, c = e % ZB_COLS;
    const bool in = k < K && j0 + c < N;
    t[k][c] = in ? B[(int64_t)k * ldb + j0 + c] : make_double2(0, 0);
    if (in) bc[(int64_t)k * N + j0 + c] = t[k][c];
  }
  __syncthreads();
  const int lane = threadIdx.x & 31;
  for (int c = threadIdx.x >> 5; c < ZB_COLS; c += 8) {
    const int j = j0 + c;
    if (j >= N) break;
    double2 v[2];
#pragma unroll
    for (int u = 0; u < 2; ++u) v[u] = t[lane + 32 * u][c];
    int qr[2][Z_S], qi[2][Z_S];
    const SliceInfo si = slice_entries(v, lane, qr, qi);
    if (lane == 0) eb[j] = si;
#pragma unroll
    for (int u = 0; u < 2; ++u)
#pragma unroll
      for (int s = 0; s < Z_S; ++s) {
        const __half re = __int2half_rn(qr[u][s]), im = __int2half_rn(qi[u][s]);
        __half2* r0 = reinterpret_cast<__half2*>(b8 + ((int64_t)s * 2 * N + 2 * j) * Z_KR);
        r0[lane + 32 * u] = __halves2half2(re, __hneg(im));
        r0[Z_KR / 2 + lane + 32 * u] = __halves2half2(im, re);
      }
  }
}

// ----------------------------------------------------------------- epilogue
// hi + lo 2^-40 (0 <= lo < 2^40) as a double, rounded once to nearest even; |hi| <
// 2^50.  Two FP64 operations: hi enters through the bits of 1.5 2^52 + hi, lo through
// those of 2^52 + lo, and the constants cancel in exact steps.
__device__ __forceinline__ double fixed_to_double(long long hi, long long lo) {
  const double xh = __longlong_as_double(hi + 0x4338000000000000ll) - (6755399441055744.0 + 4096.0);   // hi - 2^12
  const double xl = __longlong_as_double(0x4330000000000000ll | lo);                                   // 2^52 + lo
  return fma(xl, 0x1p-40, xh);
}
// v 2^ex for v = 0 or 2^-40 <= |v| < 2^51 and |ex| <= Z_EXMAX: the exponent field stays
// in range, no branch and no FP64 operation (a branch per value serialised the FP64
// latencies: 8400 cycles per 16 columns instead of 4800)
constexpr int Z_EXMAX = 960;
__device__ __forceinline__ double shift_exp(double v, int ex) {
  const long long b = __double_as_longlong(v);
  return __longlong_as_double((b << 1) == 0 ? b : b + ((long long)ex << 52));
}

// eight columns of four consecutive levels (one asm statement: nothing may touch
// the registers between the loads and the wait)
__device__ __forceinline__ void tmem_ld_levels(uint32_t taddr, uint32_t (&a)[4][8]) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%32];\n"
      " tcgen05.ld.sync.aligned.32x32b.x8.b32 {%8, %9, %10, %11, %12, %13, %14, %15}, [%33];\n"
      " tcgen05.ld.sync.aligned.32x32b.x8.b32 {%16, %17, %18, %19, %20, %21, %22, %23}, [%34];\n"
      " tcgen05.ld.sync.aligned.32x32b.x8.b32 {%24, %25, %26, %27, %28, %29, %30, %31}, [%35];\n"
      " tcgen05.wait::ld.sync.aligned;"
      : "=r"(a[0][0]), "=r"(a[0][1]), "=r"(a[0][2]), "=r"(a[0][3]), "=r"(a[0][4]), "=r"(a[0][5]), "=r"(a[0][6]), "=r"(a[0][7]),
        "=r"(a[1][0]), "=r"(a[1][1]), "=r"(a[1][2]), "=r"(a[1][3]), "=r"(a[1][4]), "=r"(a[1][5]), "=r"(a[1][6]), "=r"(a[1][7]),
        "=r"(a[2][0]), "=r"(a[2][1]), "=r"(a[2][2]), "=r"(a[2][3]), "=r"(a[2][4]), "=r"(a[2][5]), "=r"(a[2][6]), "=r"(a[2][7]),
        "=r"(a[3][0]), "=r"(a[3][1]), "=r"(a[3][2]), "=r"(a[3][3]), "=r"(a[3][4]), "=r"(a[3][5]), "=r"(a[3][6]), "=r"(a[3][7])
      : "r"(taddr), "r"(taddr + Z_BN), "r"(taddr + 2 * Z_BN), "r"(taddr + 3 * Z_BN)
      : "memory");
}
// and of one level
__device__ __forceinline__ void tmem_ld_level(uint32_t taddr, uint32_t (&a)[8]) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];\n"
      " tcgen05.wait::ld.sync.aligned;"
      : "=r"(a[0]), "=r"(a[1]), "=r"(a[2]), "=r"(a[3]), "=r"(a[4]), "=r"(a[5]), "=r"(a[6]), "=r"(a[7])
      : "r"(taddr)
      : "memory");
}

// High word of a positive double from a positive normal float, for comparisons
__device__ __forceinline__ int hi_word(float t) { return (__float_as_int(t) >> 3) + (896 << 20); }
__device__ __forceinline__ int hi_mag(double x) { return __double2hiint(x) & 0x7fffffff; }
__device__ __forceinline__ int hi_mag(double2 x) { return max(hi_mag(x.x), hi_mag(x.y)); }
// |x| 2^ex >= the double of high word t (x normal; ex 2^20 added to the exponent field)
__device__ __forceinline__ bool mag_at_least(double2 x, int ex, int t) {
  const int h = hi_mag(x);
  return (h >> 20) != 0 && (long long)h + ((long long)ex << 20) >= (long long)t;
}

// Entries (rows of the bits of m, one column) of A B in FP64 by a warp, lane = k and
// k + 32: four rows at a time, the eight sums over the lanes by halves (eleven FP64
// additions per lane instead of forty).  The lane of a row gets its entry in re, im.
__device__ __forceinline__ void entries_fp64(const double2* __restrict__ Arow0, long long lda,
                                             const double2* __restrict__ Bcol, long long ldb, int K, unsigned m, int lane,
                                             double& re, double& im) {
  const double2 z = make_double2(0, 0);
  const double2 b0 = lane < K ? __ldg(Bcol + lane * ldb) : z, b1 = lane + 32 < K ? __ldg(Bcol + (lane + 32) * ldb) : z;
  while (m) {
    int r[4];
    double v[8];
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      r[u] = m ? __ffs(m) - 1 : -1;
      m &= m - 1;
      double2 a0 = z, a1 = z;
      if (r[u] >= 0) {
        if (lane < K) a0 = __ldg(Arow0 + r[u] * lda + lane);
        if (lane + 32 < K) a1 = __ldg(Arow0 + r[u] * lda + lane + 32);
      }
      v[2 * u] = fma(-a1.y, b1.y, fma(a1.x, b1.x, fma(-a0.y, b0.y, a0.x * b0.x)));
      v[2 * u + 1] = fma(a1.y, b1.x, fma(a1.x, b1.y, fma(a0.y, b0.x, a0.x * b0.y)));
    }
    const bool up = lane & 16, up2 = lane & 8;
    double w[4], s[2];
#pragma unroll
    for (int q = 0; q < 4; ++q)
      w[q] = (up ? v[4 + q] : v[q]) + __shfl_xor_sync(0xffffffffu, up ? v[q] : v[4 + q], 16);
#pragma unroll
    for (int q = 0; q < 2; ++q) {
      s[q] = (up2 ? w[2 + q] : w[q]) + __shfl_xor_sync(0xffffffffu, up2 ? w[q] : w[2 + q], 8);
#pragma unroll
      for (int o = 4; o; o >>= 1) s[q] += __shfl_xor_sync(0xffffffffu, s[q], o);
    }
#pragma unroll
    for (int u = 0; u < 4; ++u) {      // entry u: lanes 8 u .. 8 u + 7
      const double x = __shfl_sync(0xffffffffu, s[0], 8 * u), y = __shfl_sync(0xffffffffu, s[1], 8 * u);
      if (lane == r[u]) {
        re = x;
        im = y;
      }
    }
  }
}

// shared-memory matrix descriptor: K-major, 64-byte swizzle, 8-row groups 512 B apart
__device__ __forceinline__ uint64_t desc_sw64(uint32_t addr) {
  uint64_t d = 0;
  d |= (uint64_t)((addr & 0x3FFFFu) >> 4);
  d |= (uint64_t)1 << 16;
  d |= (uint64_t)(512u >> 4) << 32;
  d |= (uint64_t)1 << 46;
  d |= (uint64_t)4 << 61;
  return d;
}

__device__ __forceinline__ SliceInfo load_info(const SliceInfo* p) {
  const int4 v = __ldg(reinterpret_cast<const int4*>(p));
  return {v.x, __int_as_float(v.y), v.z, 0};
}

__global__ void __launch_bounds__(Z_THREADS, 1)
    k_tc_gemm64(const __grid_constant__ CUtensorMap mapA, const __grid_constant__ CUtensorMap mapB,
                double2* __restrict__ C, long long ldc, int M, int N, int K, int negate, int accumulate,
                const double2* __restrict__ A, long long lda, const double2* __restrict__ B, long long ldb,
                const SliceInfo* __restrict__ ea, const SliceInfo* __restrict__ eb, int* tile_ctr, int* err) {
  extern __shared__ unsigned char smem_raw[];
  __shared__ __align__(8) unsigned long long bars[2 * Z_ST + 2 + 4];
  __shared__ int tq[2];
  __shared__ uint32_t tmem_slot;
  const uint32_t base = (smem_u32(smem_raw) + 1023u) & ~1023u;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int N2 = 2 * N;
  const int MT = (M + Z_BM - 1) / Z_BM, NT = (N2 + Z_BN - 1) / Z_BN;
  const int ntiles = MT * NT;
  const uint32_t full0 = smem_u32(&bars[0]), empty0 = smem_u32(&bars[Z_ST]);
  const uint32_t accf = smem_u32(&bars[2 * Z_ST]), acce = smem_u32(&bars[2 * Z_ST + 1]);
  const uint32_t tqf0 = smem_u32(&bars[2 * Z_ST + 2]), tqe0 = smem_u32(&bars[2 * Z_ST + 4]);
  if (threadIdx.x == 0) {
    for (int s = 0; s < Z_ST; ++s) {
      mbar_init(full0 + 8 * s, 1);
      mbar_init(empty0 + 8 * s, 1);
    }
    mbar_init(accf, 1);
    mbar_init(acce, Z_EPI);
    for (int q = 0; q < 2; ++q) {
      mbar_init(tqf0 + 8 * q, 1);
      mbar_init(tqe0 + 8 * q, 1 + Z_EPI);
    }
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  __syncwarp();
  if (warp == 0) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&tmem_slot)),
                 "r"(512u)
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = tmem_slot;
  const float thr_sum = 0x1p25f / (float)K;

  int issued = 0;
  if (warp == 0) {
    if (lane == 0) {
      // ---------------- tile scheduler + TMA producer
      int it = 0;
      for (int j = 0;; ++j) {
        const int q = j & 1;
        if (j >= 2 && !mbar_wait(tqe0 + 8 * q, ((j >> 1) - 1) & 1, err, 16)) break;
        int t = *(volatile int*)err ? -1 : atomicAdd(tile_ctr, 1);
        if (t >= ntiles) t = -1;
        tq[q] = t;
        mbar_arrive(tqf0 + 8 * q);
        if (t < 0) break;
        int mt, nt;
        tile_coords(t, MT, NT, mt, nt);
        bool ok = true;
        for (int kt = 0; kt < Z_KT; ++kt, ++it) {
          const int s = it % Z_ST;
          if (it >= Z_ST && !mbar_wait(empty0 + 8 * s, ((it / Z_ST) - 1) & 1, err, 1)) { ok = false; break; }
          const uint32_t sa = base + s * Z_STAGE, sb = sa + Z_S * Z_A_BYTES;
          mbar_expect_tx(full0 + 8 * s, Z_STAGE);
#pragma unroll
          for (int d = 0; d < Z_S; ++d) {
            tma_load_2d(sa + d * Z_A_BYTES, &mapA, full0 + 8 * s, kt * Z_BK, d * M + mt * Z_BM);
            tma_load_2d(sb + d * Z_B_BYTES, &mapB, full0 + 8 * s, kt * Z_BK, d * N2 + nt * Z_BN);
          }
          issued = it + 1;
        }
        if (!ok) {
          const int q2 = (j + 1) & 1;
          if (j + 1 < 2 || mbar_wait(tqe0 + 8 * q2, (((j + 1) >> 1) - 1) & 1, err, 16)) {
            tq[q2] = -1;
            mbar_arrive(tqf0 + 8 * q2);
          }
          break;
        }
      }
    }
  } else if (warp == 1) {
    if (lane == 0) {
      // ---------------- MMA issuer: slice i of A times slices 0 .. 8 - i of B into levels i .. 8
      int it = 0;
      for (int j = 0;; ++j) {
        const int q = j & 1;
        if (!mbar_wait(tqf0 + 8 * q, (j >> 1) & 1, err, 32)) break;
        const int t = *(volatile int*)&tq[q];
        mbar_arrive(tqe0 + 8 * q);
        if (t < 0) break;
        if (j >= 1 && !mbar_wait(acce, (j - 1) & 1, err, 64)) break;
        tc_fence_after();
        bool ok = true;
        for (int kt = 0; kt < Z_KT; ++kt, ++it) {
          const int s = it % Z_ST;
          if (!mbar_wait(full0 + 8 * s, (it / Z_ST) & 1, err, 2)) { ok = false; break; }
          tc_fence_after();
          const uint32_t sa = base + s * Z_STAGE, sb = sa + Z_S * Z_A_BYTES;
#pragma unroll
          for (int kk = 0; kk < Z_BK / 16; ++kk) {        // 16 halves = 32 bytes along K inside the swizzle row
            const uint64_t db = desc_sw64(sb) + 2 * kk;
            const bool first = kt == 0 && kk == 0;
#pragma unroll
            for (int i = 0; i < Z_S; ++i) {
              const uint64_t da = desc_sw64(sa + i * Z_A_BYTES) + 2 * kk;
              int nb = i == 0 ? Z_S : Z_L - i;            // slices of B
              if (i == 1 && first) {
                // level 8 starts here: its slice of B apart, without the accumulator
                --nb;
                mma_f16(tmem + (uint32_t)((Z_L - 1) * Z_BN), da, desc_sw64(sb + (Z_S - 1) * Z_B_BYTES) + 2 * kk,
                        z_idesc(Z_BN), 0u);
              }
              mma_f16(tmem + (uint32_t)(i * Z_BN), da, db, z_idesc(nb * Z_BN), (first && i == 0) ? 0u : 1u);
            }
          }
          mma_commit(empty0 + 8 * s);
        }
        if (!ok) break;
        mma_commit(accf);
      }
    }
  } else {
    // ---------------- epilogue warps: TMEM lane quarter (warp % 4) = 32 rows of the
    // tile, columns 16 half .. 16 half + 15
    const int quarter = warp & 3, half = (warp - 2) >> 2;
    double* stage = reinterpret_cast<double*>(smem_raw + (base - smem_u32(smem_raw)) + Z_ST * Z_STAGE) +
                    (warp - 2) * 32 * Z_CH;
    for (int j = 0;; ++j) {
      const int q = j & 1;
      int t = -1;
      const bool okq = __all_sync(0xffffffffu, mbar_wait(tqf0 + 8 * q, (j >> 1) & 1, err, 128) ? 1 : 0) != 0;
      if (okq) t = *(volatile int*)&tq[q];
      __syncwarp();
      if (lane == 0 && okq) mbar_arrive(tqe0 + 8 * q);
      if (!okq || t < 0) break;
      const bool ok = __all_sync(0xffffffffu, mbar_wait(accf, j & 1, err, 4) ? 1 : 0) != 0;
      if (!ok) break;
      tc_fence_after();
      int mt, nt;
      tile_coords(t, MT, NT, mt, nt);
      const int row0 = mt * Z_BM + quarter * 32, c0 = nt * (Z_BN / 2);     // c0: complex column
      const SliceInfo none = {0, 0.f, 0, 0};
      const SliceInfo ra = row0 + lane < M ? load_info(ea + row0 + lane) : none;
      constexpr int NCH = Z_BN / 2 / Z_CH;
      for (int ch = half * NCH; ch < (half + 1) * NCH; ++ch) {
        const int cc0 = c0 + ch * (Z_CH / 2);
        // this lane's part of C for the coalesced pass below: four lanes per row
        double2 old[Z_CH / 2];
        if (accumulate) {
#pragma unroll
          for (int i = 0; i < Z_CH / 2; ++i) {
            const int row = row0 + 8 * i + (lane >> 2), cc = cc0 + (lane & 3);
            old[i] = (row < M && cc < N) ? C[(long long)row * ldc + cc] : make_double2(0, 0);
          }
        }
        uint32_t ah[4][Z_CH], aw[4][Z_CH], al[Z_CH];    // levels 0 .. 3, 4 .. 7 and 8
        const uint32_t ta = tmem + ((uint32_t)(quarter * 32) << 16) + (uint32_t)(ch * Z_CH);
        tmem_ld_levels(ta, ah);
        tmem_ld_levels(ta + 4 * Z_BN, aw);
        tmem_ld_level(ta + 8 * Z_BN, al);
        if (ch == (half + 1) * NCH - 1) {
          // the accumulators have been read: the MMA warp may overwrite them
          tc_fence_before();
          __syncwarp();
          if (lane == 0) mbar_arrive(acce);
        }
        if (row0 < M && cc0 < N) {
          int ex[Z_CH / 2], thr[Z_CH / 2], kb[Z_CH / 2];  // of (row = lane, complex column)
          bool far = false;
#pragma unroll
          for (int c = 0; c < Z_CH / 2; ++c) {
            const SliceInfo cb = cc0 + c < N ? load_info(eb + cc0 + c) : none;
            ex[c] = ra.e + cb.e - 36;
            far = far || ex[c] > Z_EXMAX || ex[c] < -Z_EXMAX;
            // the smallest |c| that the bound on the operands' rounding and the dropped
            // levels allows, (Sa + Sb) 2^-11 / K + 2^-14, in units of val (2^-36)
            thr[c] = ra.sum > 0.f && cb.sum > 0.f ? hi_word((ra.sum + cb.sum) * thr_sum + 0x1p22f) : 0;
            kb[c] = cb.k;
          }
          double val[Z_CH];
#pragma unroll
          for (int c = 0; c < Z_CH; ++c) {
            long long h = 0, w = 0;
#pragma unroll
            for (int l = 0; l < 4; ++l) {
              h = (h << 8) + (long long)__float2int_rn(__uint_as_float(ah[l][c]));
              w = (w << 8) + (long long)__float2int_rn(__uint_as_float(aw[l][c]));
            }
            w = (w << 8) + (long long)__float2int_rn(__uint_as_float(al[c]));
            // sum of the levels = (h 2^40 + w) 2^48 units of 2^-124
            val[c] = fixed_to_double(h + (w >> 40), w & ((1ll << 40) - 1));
          }
          // entries that the digits may hold less accurately than an FP64 sum: |c| below
          // the threshold, and so are the terms of the column's and of the row's largest
          // entry (an entry of at least half 2^e on the other side)
          bool again[Z_CH / 2];
#pragma unroll
          for (int c = 0; c < Z_CH / 2; ++c) {
            again[c] = hi_mag(make_double2(val[2 * c], val[2 * c + 1])) < thr[c];
            if (again[c]) {
              const double2 a1 = __ldg(A + (long long)(row0 + lane) * lda + kb[c]);
              const double2 b1 = __ldg(B + (long long)ra.k * ldb + cc0 + c);
              const int eb_c = ex[c] + 36 - ra.e;
              again[c] = !mag_at_least(a1, 35 - ra.e, thr[c]) && !mag_at_least(b1, 35 - eb_c, thr[c]);
            }
          }
          if (!__any_sync(0xffffffffu, far)) {
#pragma unroll
            for (int c = 0; c < Z_CH; ++c) val[c] = shift_exp(val[c], ex[c >> 1]);
          } else {                                       // results near the ends of the range, or non-finite operands
#pragma unroll
            for (int c = 0; c < Z_CH; ++c) {
              const int e = ex[c >> 1], e1 = max(min(e / 2, Z_EXMAX), -Z_EXMAX), e2 = max(min(e - e1, Z_EXMAX), -Z_EXMAX);
              const double f1 = __longlong_as_double(e > Z_NAN / 2 ? 0x7ff8000000000000ll : (long long)(1023 + e1) << 52);
              val[c] = val[c] * f1 * __longlong_as_double((long long)(1023 + e2) << 52);
            }
          }
#pragma unroll
          for (int c = 0; c < Z_CH / 2; ++c) {
            const unsigned m = __ballot_sync(0xffffffffu, again[c]);
            if (m) entries_fp64(A + (long long)row0 * lda, lda, B + cc0 + c, ldb, K, m, lane, val[2 * c], val[2 * c + 1]);
          }
          // row = lane; 16-byte units (re, im) spread over the banks by the row
          double2* st2 = reinterpret_cast<double2*>(stage);
#pragma unroll
          for (int c = 0; c < Z_CH / 2; ++c)
            st2[lane * (Z_CH / 2) + (c ^ ((lane >> 1) & 3))] =
                negate ? make_double2(-val[2 * c], -val[2 * c + 1]) : make_double2(val[2 * c], val[2 * c + 1]);
          __syncwarp();
#pragma unroll
          for (int i = 0; i < Z_CH / 2; ++i) {
            const int rr = 8 * i + (lane >> 2), row = row0 + rr, cc = cc0 + (lane & 3);
            double2 v = st2[rr * (Z_CH / 2) + ((lane & 3) ^ ((rr >> 1) & 3))];
            if (accumulate) v = cadd(v, old[i]);
            if (row < M && cc < N) C[(long long)row * ldc + cc] = v;
          }
          __syncwarp();
        }
      }
    }
  }
  // ---------------- drain loads still in flight after an error, free TMEM
  if (warp == 0 && lane == 0 && *(volatile int*)err) {
    for (int i = issued - Z_ST > 0 ? issued - Z_ST : 0; i < issued; ++i)
      mbar_wait(full0 + 8 * (i % Z_ST), (i / Z_ST) & 1, err, 8);
  }
  tc_fence_before();
  __syncthreads();
  if (warp == 0) {
    tc_fence_after();
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(512u) : "memory");
  }
}

// --------------------------------------------------------------------- host
bool tc_gemm64_prepare() {
  return cudaFuncSetAttribute(k_tc_gemm64, cudaFuncAttributeMaxDynamicSharedMemorySize, Z_SMEM) == cudaSuccess;
}

bool tc_gemm64_eligible(TcGemmCtx& c, int64_t M, int64_t N, int64_t K, double2 alpha, double2 beta) {
  if (!tc_device_ready(c)) return false;
  if (alpha.y != 0.0 || (alpha.x != 1.0 && alpha.x != -1.0) || beta.y != 0.0 || (beta.x != 0.0 && beta.x != 1.0))
    return false;
  return K >= 16 && K <= TC64_K && M >= 16 && N >= 16 && Z_S * M < (1ll << 30) && Z_S * 2 * N < (1ll << 30);
}

mnpbem_status tc_gemm_c128(TcGemmCtx& c, int64_t M, int64_t N, int64_t K, double alpha, const double2* A, int64_t lda,
                           const double2* B, int64_t ldb, bool accumulate, double2* C, int64_t ldc, cudaStream_t st) {
  MNP_TRY(c.a8.ensure(sizeof(__half) * Z_S * M * Z_KR));
  MNP_TRY(c.b8.ensure(sizeof(__half) * Z_S * 2 * N * Z_KR + sizeof(double2) * K * N));
  MNP_TRY(c.exps.ensure(sizeof(SliceInfo) * (M + N)));
  MNP_TRY(tc_error_word(c, st));
  MNP_TRY(c.ctr.ensure(sizeof(int)));
  __half *a8 = c.a8.as<__half>(), *b8 = c.b8.as<__half>();
  double2* bc = reinterpret_cast<double2*>(b8 + (int64_t)Z_S * 2 * N * Z_KR);
  SliceInfo *ea = c.exps.as<SliceInfo>(), *eb = ea + M;
  {
    ProfScope ps(PH_ELEMWISE, st, 0.0, 16.0 * K * (M + 2.0 * N) + 2.0 * Z_S * Z_KR * (M + 2.0 * N));
    k_slice_a<<<(unsigned)cdiv_up(M, (int64_t)8), 256, 0, st>>>(A, lda, (int)M, (int)K, a8, ea, c.ctr.as<int>());
    k_slice_b<<<(unsigned)cdiv_up(N, (int64_t)ZB_COLS), 256, 0, st>>>(B, ldb, (int)K, (int)N, b8, eb, bc);
    MNP_CHECK_LAUNCH();
  }
  CUtensorMap ma, mb;
  if (!tc_f16_map(c, &ma, a8, Z_KR, (uint64_t)Z_S * M, Z_BK, Z_BM) ||
      !tc_f16_map(c, &mb, b8, Z_KR, (uint64_t)Z_S * 2 * N, Z_BK, Z_BN)) {
    set_error("cuTensorMapEncodeTiled failed");
    return MNPBEM_ERR_CUDA;
  }
  const int64_t tiles = cdiv_up(M, (int64_t)Z_BM) * cdiv_up(2 * N, (int64_t)Z_BN);
  if (tiles >= (1ll << 31)) { set_error("tc_gemm_c128: too many tiles"); return MNPBEM_ERR_INVALID_ARG; }
  ProfScope ps(M >= 128 && N >= 128 ? PH_GEMM_BIG : PH_GEMM_SMALL, st, 8.0 * M * N * K,
               16.0 * ((double)M * K + (double)K * N + 2.0 * M * N));
  const int ctas = c.num_sms > 0 ? c.num_sms : 148;
  k_tc_gemm64<<<(unsigned)std::min<int64_t>(tiles, ctas), Z_THREADS, Z_SMEM, st>>>(
      ma, mb, C, (long long)ldc, (int)M, (int)N, (int)K, alpha < 0 ? 1 : 0, accumulate ? 1 : 0, A, (long long)lda, bc,
      (long long)N, ea, eb, c.ctr.as<int>(), c.err.as<int>());
  MNP_CHECK_LAUNCH();
  return MNPBEM_OK;
}

}  // namespace mnpbem
