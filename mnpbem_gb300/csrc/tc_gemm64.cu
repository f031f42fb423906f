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
// 2^-63 of the largest entry), and cut into eight signed base-256 digits,
// X = sum_i q_i 256^(7-i), |q_i| <= 128, exact in FP16.  The products of digit
// slices i and j with i + j = l <= 7 are accumulated in FP32 in one tensor-memory
// accumulator per level l: sums of at most 8 * 128 products of at most 2^14,
// integers up to 2^24, so every sum is exact.  The epilogue adds the eight levels
// as integers, sum_l a_l 256^(7-l), rounds once to a double, applies the two
// exponents and adds C with one FP64 addition per value.  The dropped levels
// (l >= 8) are below 2^-58 of (largest of the row) x (largest of the column) for K =
// 64, the rounding of an FP64 sum of 128 products about 2^-51.5 of it.
//
// Why: FP64 runs at two multiply-adds per clock and SM here (1.25 TFLOP/s), the
// FP16 tensor cores 1500 times as fast; 36 exact slice products, and an epilogue
// that needs one FP64 operation per value and 64-deep product instead of 128,
// leave 37 us instead of 272 us per product of the FP64 solve at 508 faces and 54 us
// instead of 473 us at 1350 faces (two wavelengths in flight).
//
// Tile: 128 rows x 64 real columns, eight accumulators of 64 columns (all 512
// tensor-memory columns), K chunks of 32 halves (64-byte swizzle rows) of all
// sixteen slices (96 KB), two of them in flight.  Roles as in tc_gemm.cu: TMA
// producer, MMA issuer, eight epilogue warps (two per scheduler, so that one
// converts while the other waits for FP64); persistent with a tile counter.
#include <cuda.h>
#include <cuda_fp16.h>
#include <cudaTypedefs.h>

#include <algorithm>

#include "profile.cuh"
#include "tc_gemm.cuh"
#include "tc_prims.cuh"

namespace mnpbem {

constexpr int Z_S = 8;                                  // digit slices
constexpr int Z_KR = 2 * TC64_K;                        // reals per row of A
constexpr int Z_BM = 128, Z_BN = 64, Z_BK = 32, Z_KT = Z_KR / Z_BK;
constexpr int Z_A_BYTES = Z_BM * Z_BK * 2, Z_B_BYTES = Z_BN * Z_BK * 2;
constexpr int Z_STAGE = Z_S * (Z_A_BYTES + Z_B_BYTES);  // 96 KB
constexpr int Z_ST = 2;
constexpr int Z_EPI = 8;                                // epilogue warps: two per 32 rows, half of the columns each
constexpr int Z_CH = 8;                                 // columns per epilogue step
static_assert(Z_CH == 8 && Z_S == 8, "tmem_ld_levels");
constexpr int Z_THREADS = 32 * (2 + Z_EPI);
constexpr int Z_SMEM = Z_ST * Z_STAGE + Z_EPI * 32 * Z_CH * 8 + 1024;
constexpr uint32_t Z_IDESC = (1u << 4) | ((uint32_t)(Z_BN >> 3) << 17) | ((uint32_t)(Z_BM >> 4) << 24);
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

// A [M][K] -> a8 [S][M][Z_KR] (slice s of row i: digit s of its 2K reals, zero
// beyond), ea [M].  One warp per row.
__global__ void __launch_bounds__(256) k_slice_a(const double2* __restrict__ A, int64_t lda, int M, int K,
                                                 __half* __restrict__ a8, int* __restrict__ ea, int* tile_ctr) {
  if (blockIdx.x == 0 && threadIdx.x == 0) *tile_ctr = 0;   // of the product that follows
  const int row = blockIdx.x * 8 + (threadIdx.x >> 5), lane = threadIdx.x & 31;
  if (row >= M) return;
  double2 v[2];
  unsigned long long mx = 0;
#pragma unroll
  for (int u = 0; u < 2; ++u) {
    const int k = lane + 32 * u;
    v[u] = k < K ? A[(int64_t)row * lda + k] : make_double2(0, 0);
    mx = max(mx, max(mag_bits(v[u].x), mag_bits(v[u].y)));
  }
#pragma unroll
  for (int o = 16; o; o >>= 1) mx = max(mx, __shfl_xor_sync(0xffffffffu, mx, o));
  const int e = row_exp(mx);
  if (lane == 0) ea[row] = e;
  const bool fin = e != Z_NAN;
#pragma unroll
  for (int u = 0; u < 2; ++u) {
    int qr[Z_S], qi[Z_S];
    digits(fin ? fixed62(v[u].x, e) : 0, qr);
    digits(fin ? fixed62(v[u].y, e) : 0, qi);
#pragma unroll
    for (int s = 0; s < Z_S; ++s)
      reinterpret_cast<__half2*>(a8 + ((int64_t)s * M + row) * Z_KR)[lane + 32 * u] =
          __halves2half2(__int2half_rn(qr[s]), __int2half_rn(qi[s]));
  }
}

// B [K][N] -> b8 [S][2N][Z_KR]: row 2j holds (Re b, -Im b) of column j, row 2j + 1
// (Im b, Re b); eb [N].  CTA of 256 threads = 16 columns: the block of B through
// shared memory, then one warp per column at a time, lanes along k.
constexpr int ZB_COLS = 16;
__global__ void __launch_bounds__(256) k_slice_b(const double2* __restrict__ B, int64_t ldb, int K, int N,
                                                 __half* __restrict__ b8, int* __restrict__ eb) {
  __shared__ double2 t[TC64_K][ZB_COLS + 1];
  const int j0 = blockIdx.x * ZB_COLS;
  for (int e = threadIdx.x; e < TC64_K * ZB_COLS; e += 256) {
    const int k = e / ZB_COLS, c = e % ZB_COLS;
    t[k][c] = (k < K && j0 + c < N) ? B[(int64_t)k * ldb + j0 + c] : make_double2(0, 0);
  }
  __syncthreads();
  const int lane = threadIdx.x & 31;
  for (int c = threadIdx.x >> 5; c < ZB_COLS; c += 8) {
    const int j = j0 + c;
    if (j >= N) break;
    double2 v[2];
    unsigned long long mx = 0;
#pragma unroll
    for (int u = 0; u < 2; ++u) {
      v[u] = t[lane + 32 * u][c];
      mx = max(mx, max(mag_bits(v[u].x), mag_bits(v[u].y)));
    }
#pragma unroll
    for (int o = 16; o; o >>= 1) mx = max(mx, __shfl_xor_sync(0xffffffffu, mx, o));
    const int e = row_exp(mx);
    if (lane == 0) eb[j] = e;
    const bool fin = e != Z_NAN;
#pragma unroll
    for (int u = 0; u < 2; ++u) {
      int qr[Z_S], qi[Z_S];
      digits(fin ? fixed62(v[u].x, e) : 0, qr);
      digits(fin ? fixed62(v[u].y, e) : 0, qi);
#pragma unroll
      for (int s = 0; s < Z_S; ++s) {
        const __half re = __int2half_rn(qr[s]), im = __int2half_rn(qi[s]);
        __half2* r0 = reinterpret_cast<__half2*>(b8 + ((int64_t)s * 2 * N + 2 * j) * Z_KR);
        r0[lane + 32 * u] = __halves2half2(re, __hneg(im));
        r0[Z_KR / 2 + lane + 32 * u] = __halves2half2(im, re);
      }
    }
  }
}

// ----------------------------------------------------------------- epilogue
// hi + lo 2^-32 as a double, rounded once to nearest even; |hi| < 2^50.  Two FP64
// operations: hi enters through the bits of 1.5 2^52 + hi, lo through those of
// 2^52 + lo, and the constants cancel in exact steps.
__device__ __forceinline__ double fixed_to_double(long long hi, unsigned lo) {
  const double xh = __longlong_as_double(hi + 0x4338000000000000ll) - (6755399441055744.0 + 1048576.0);   // hi - 2^20
  const double xl = __longlong_as_double(0x4330000000000000ll | (long long)lo);                           // 2^52 + lo
  return fma(xl, 0x1p-32, xh);
}
// v 2^ex for v = 0 or 2^-32 <= |v| < 2^51 and |ex| <= Z_EXMAX: the exponent field stays
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

__global__ void __launch_bounds__(Z_THREADS, 1)
    k_tc_gemm64(const __grid_constant__ CUtensorMap mapA, const __grid_constant__ CUtensorMap mapB,
                double2* __restrict__ C, long long ldc, int M, int N, int negate, int accumulate,
                const int* __restrict__ ea, const int* __restrict__ eb, int* tile_ctr, int* err) {
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
      // ---------------- MMA issuer: level l = i + j into accumulator l
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
          for (int l = 0; l < Z_S; ++l)
            for (int i = 0; i <= l; ++i) {
              const uint64_t da = desc_sw64(sa + i * Z_A_BYTES), db = desc_sw64(sb + (l - i) * Z_B_BYTES);
#pragma unroll
              for (int kk = 0; kk < Z_BK / 16; ++kk)    // 16 halves = 32 bytes along K inside the swizzle row
                mma_f16(tmem + (uint32_t)(l * Z_BN), da + 2 * kk, db + 2 * kk, Z_IDESC,
                        (kt > 0 || i > 0 || kk > 0) ? 1u : 0u);
            }
          mma_commit(empty0 + 8 * s);
        }
        if (!ok) break;
        mma_commit(accf);
      }
    }
  } else {
    // ---------------- epilogue warps: TMEM lane quarter (warp % 4) = 32 rows of the
    // tile, columns 32 half .. 32 half + 31
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
      const int er = row0 + lane < M ? __ldg(ea + row0 + lane) : 0;
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
        uint32_t ah[4][Z_CH], aw[4][Z_CH];              // levels 0 .. 3 and 4 .. 7
        const uint32_t ta = tmem + ((uint32_t)(quarter * 32) << 16) + (uint32_t)(ch * Z_CH);
        tmem_ld_levels(ta, ah);
        tmem_ld_levels(ta + 4 * Z_BN, aw);
        if (ch == (half + 1) * NCH - 1) {
          // the accumulators have been read: the MMA warp may overwrite them
          tc_fence_before();
          __syncwarp();
          if (lane == 0) mbar_arrive(acce);
        }
        if (row0 < M && cc0 < N) {
          int ex[Z_CH / 2];                              // exponents of (row = lane, complex column)
          bool far = false;
#pragma unroll
          for (int c = 0; c < Z_CH / 2; ++c) {
            ex[c] = er + (cc0 + c < N ? __ldg(eb + cc0 + c) : 0) - 36;
            far = far || ex[c] > Z_EXMAX || ex[c] < -Z_EXMAX;
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
            // sum of the levels = (h 2^32 + w) 2^56 units of 2^-124
            val[c] = fixed_to_double(h + (w >> 32), (unsigned)w);
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
bool tc_gemm64_eligible(TcGemmCtx& c, int64_t M, int64_t N, int64_t K, double2 alpha, double2 beta) {
  if (!tc_device_ready(c)) return false;
  if (alpha.y != 0.0 || (alpha.x != 1.0 && alpha.x != -1.0) || beta.y != 0.0 || (beta.x != 0.0 && beta.x != 1.0))
    return false;
  return K >= 16 && K <= TC64_K && M >= 16 && N >= 16 && Z_S * M < (1ll << 30) && Z_S * 2 * N < (1ll << 30);
}

mnpbem_status tc_gemm_c128(TcGemmCtx& c, int64_t M, int64_t N, int64_t K, double alpha, const double2* A, int64_t lda,
                           const double2* B, int64_t ldb, bool accumulate, double2* C, int64_t ldc, cudaStream_t st) {
  MNP_TRY(c.a8.ensure(sizeof(__half) * Z_S * M * Z_KR));
  MNP_TRY(c.b8.ensure(sizeof(__half) * Z_S * 2 * N * Z_KR));
  MNP_TRY(c.exps.ensure(sizeof(int) * (M + N)));
  MNP_TRY(c.err.ensure(sizeof(int)));
  MNP_TRY(c.ctr.ensure(sizeof(int)));
  static bool attr = false;
  if (!attr) {
    MNP_CUDA(cudaFuncSetAttribute(k_tc_gemm64, cudaFuncAttributeMaxDynamicSharedMemorySize, Z_SMEM));
    attr = true;
  }
  __half *a8 = c.a8.as<__half>(), *b8 = c.b8.as<__half>();
  int *ea = c.exps.as<int>(), *eb = ea + M;
  if (!c.err_cleared) {
    MNP_CUDA(cudaMemsetAsync(c.err.ptr, 0, sizeof(int), st));
    c.err_cleared = true;
  }
  {
    ProfScope ps(PH_ELEMWISE, st, 0.0, 16.0 * K * (M + N) + 2.0 * Z_S * Z_KR * (M + 2.0 * N));
    k_slice_a<<<(unsigned)cdiv_up(M, (int64_t)8), 256, 0, st>>>(A, lda, (int)M, (int)K, a8, ea, c.ctr.as<int>());
    k_slice_b<<<(unsigned)cdiv_up(N, (int64_t)ZB_COLS), 256, 0, st>>>(B, ldb, (int)K, (int)N, b8, eb);
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
      ma, mb, C, (long long)ldc, (int)M, (int)N, alpha < 0 ? 1 : 0, accumulate ? 1 : 0, ea, eb, c.ctr.as<int>(),
      c.err.as<int>());
  MNP_CHECK_LAUNCH();
  return MNPBEM_OK;
}

}  // namespace mnpbem
