// Dense complex kernels: SIMT products (general, few tiles, few columns), block
// inverses, and the block LDU factors, their triangular sweeps and the blocked
// Gauss-Jordan inversion that replace MATLAB's inv() in
// BEM/@bemret/private/initmat.m:27-28,50,72.
//
// Gauss-Jordan without row interchanges: the matrices inverted by bemret
// (G1, G2, Sigma1 - Sigma2, Sigma) are strongly diagonally dominant (the
// diagonal is the column maximum in practice), which is the same property the
// reference's own native dense LU relies on (mex/hlib/lu.cpp:79-105 factorises
// without pivoting).  Each block step costs one rank-nb update of the whole
// matrix, so all O(n^3) work is a GEMM.  A pivot guard reports singular blocks.
#include <cooperative_groups.h>

#include <atomic>

#include "dense.cuh"
#include "ds_math.cuh"
#include "mbarrier.cuh"
#include "profile.cuh"
#include "tc_gemm.cuh"

namespace mnpbem {

// ----------------------------------------------------------------- SIMT GEMM
template <typename R, int BK>
__global__ void __launch_bounds__(256) k_gemm_nn(int64_t M, int64_t N, int64_t K, cplx<R> alpha,
                                                 const cplx<R>* __restrict__ A, int64_t lda,
                                                 const cplx<R>* __restrict__ B, int64_t ldb,
                                                 cplx<R> beta, cplx<R>* __restrict__ C,
                                                 int64_t ldc) {
  using Cx = cplx<R>;
  __shared__ Cx As[BK][64 + 1];
  __shared__ Cx Bs[BK][64];
  const int t = threadIdx.x, tx = t & 15, ty = t >> 4;
  const int64_t m0 = (int64_t)blockIdx.y * 64, n0 = (int64_t)blockIdx.x * 64;
  Cx acc[4][4];
#pragma unroll
  for (int r = 0; r < 4; ++r)
#pragma unroll
    for (int c = 0; c < 4; ++c) acc[r][c] = mk<R>(0, 0);
  for (int64_t k0 = 0; k0 < K; k0 += BK) {
    for (int l = t; l < 64 * BK; l += 256) {
      int r = l / BK, c = l % BK;
      int64_t gr = m0 + r, gc = k0 + c;
      As[c][r] = (gr < M && gc < K) ? A[gr * lda + gc] : mk<R>(0, 0);
    }
    for (int l = t; l < BK * 64; l += 256) {
      int r = l / 64, c = l % 64;
      int64_t gr = k0 + r, gc = n0 + c;
      Bs[r][c] = (gr < K && gc < N) ? B[gr * ldb + gc] : mk<R>(0, 0);
    }
    __syncthreads();
#pragma unroll
    for (int kk = 0; kk < BK; ++kk) {
      Cx a[4], b[4];
#pragma unroll
      for (int r = 0; r < 4; ++r) a[r] = As[kk][ty + 16 * r];
#pragma unroll
      for (int c = 0; c < 4; ++c) b[c] = Bs[kk][tx + 16 * c];
#pragma unroll
      for (int r = 0; r < 4; ++r)
#pragma unroll
        for (int c = 0; c < 4; ++c) cfma(acc[r][c], a[r], b[c]);
    }
    __syncthreads();
  }
  const bool zero_beta = (beta.x == 0 && beta.y == 0);
#pragma unroll
  for (int r = 0; r < 4; ++r) {
    int64_t gr = m0 + ty + 16 * r;
    if (gr >= M) continue;
#pragma unroll
    for (int c = 0; c < 4; ++c) {
      int64_t gc = n0 + tx + 16 * c;
      if (gc >= N) continue;
      Cx v = cmul(alpha, acc[r][c]);
      if (!zero_beta) v = cadd(v, cmul(beta, C[gr * ldc + gc]));
      C[gr * ldc + gc] = v;
    }
  }
}

// The same product for a few tiles (panel products of a last, narrow block): 16 x
// 32 tiles and the k range of a step shared by four groups of 64 threads, whose
// sums are added in a fixed order at the end.  Bound by latency: with 64 x 64
// tiles such a product ran on one to eight SMs and K = 256 took 46 us whatever the
// size, now 8 (64 x 64 x 64: 16 and 4; 512 x 512 x 64, 64 old tiles: 16 and 9).
constexpr int SG_M = 16, SG_N = 32, SG_K = 64;
__global__ void __launch_bounds__(256) k_gemm_small(int64_t M, int64_t N, int64_t K, float2 alpha,
                                                    const float2* __restrict__ A, int64_t lda,
                                                    const float2* __restrict__ B, int64_t ldb, float2 beta,
                                                    float2* __restrict__ C, int64_t ldc) {
  __shared__ float2 As[SG_K][SG_M + 1], Bs[SG_K][SG_N], red[4][SG_M * SG_N];
  const int t = threadIdx.x, g = t >> 6, u = t & 63, tx = u & 15, ty = u >> 4;
  const int64_t m0 = (int64_t)blockIdx.y * SG_M, n0 = (int64_t)blockIdx.x * SG_N;
  float2 acc[4][2];
#pragma unroll
  for (int r = 0; r < 4; ++r) acc[r][0] = acc[r][1] = make_float2(0.f, 0.f);
  float2 pa[4], pb[8];
  const auto fetch = [&](int64_t k0) {
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      const int e = t + 256 * q;
      const int64_t r = m0 + (e >> 6), k = k0 + (e & 63);
      pa[q] = (r < M && k < K) ? A[r * lda + k] : make_float2(0.f, 0.f);
    }
#pragma unroll
    for (int q = 0; q < 8; ++q) {
      const int e = t + 256 * q;
      const int64_t k = k0 + (e >> 5), c = n0 + (e & 31);
      pb[q] = (k < K && c < N) ? B[k * ldb + c] : make_float2(0.f, 0.f);
    }
  };
  fetch(0);
  for (int64_t k0 = 0; k0 < K; k0 += SG_K) {
    __syncthreads();
#pragma unroll
    for (int q = 0; q < 4; ++q) As[(t + 256 * q) & 63][(t + 256 * q) >> 6] = pa[q];
#pragma unroll
    for (int q = 0; q < 8; ++q) Bs[(t + 256 * q) >> 5][(t + 256 * q) & 31] = pb[q];
    __syncthreads();
    if (k0 + SG_K < K) fetch(k0 + SG_K);
#pragma unroll
    for (int q = 0; q < SG_K / 4; ++q) {
      const int kk = g * (SG_K / 4) + q;
      const float2 b0 = Bs[kk][tx], b1 = Bs[kk][tx + 16];
#pragma unroll
      for (int r = 0; r < 4; ++r) {
        const float2 a = As[kk][ty + 4 * r];
        cfma(acc[r][0], a, b0);
        cfma(acc[r][1], a, b1);
      }
    }
  }
#pragma unroll
  for (int r = 0; r < 4; ++r) {
    red[g][(ty + 4 * r) * SG_N + tx] = acc[r][0];
    red[g][(ty + 4 * r) * SG_N + tx + 16] = acc[r][1];
  }
  __syncthreads();
  const bool zero_beta = (beta.x == 0 && beta.y == 0);
  for (int e = t; e < SG_M * SG_N; e += 256) {
    const int64_t r = m0 + e / SG_N, c = n0 + e % SG_N;
    if (r >= M || c >= N) continue;
    const float2 v = cadd(cadd(red[0][e], red[1][e]), cadd(red[2][e], red[3][e]));
    float2 out = cmul(alpha, v);
    if (!zero_beta) out = cadd(out, cmul(beta, C[r * ldc + c]));
    C[r * ldc + c] = out;
  }
}

// ------------------------------------------------------- thin GEMM (N <= 16)
// Matrix times a few vectors, memory-bound on A.  A block of 8 warps owns
// TR rows; warp w streams its own slice of K (no barriers in the main loop),
// lanes stride by 32 over consecutive k (coalesced rows of A), each B row is
// read once per lane through L1 and reused for the TR rows.  The 8 partial
// sums per entry are combined in shared memory at the end.
constexpr int THIN_NMAX = 16, THIN_WARPS = 8;

template <typename R, int N, int TR>
__global__ void __launch_bounds__(32 * THIN_WARPS) k_gemm_thin(int64_t M, int64_t K, cplx<R> alpha,
                                                             const cplx<R>* __restrict__ A, int64_t lda,
                                                             const cplx<R>* __restrict__ B, int64_t ldb,
                                                             cplx<R> beta, cplx<R>* __restrict__ C,
                                                             int64_t ldc) {
  using Cx = cplx<R>;
  __shared__ Cx red[THIN_WARPS][TR][N];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int64_t row0 = (int64_t)blockIdx.x * TR;
  const int64_t kw = (K + THIN_WARPS - 1) / THIN_WARPS;
  const int64_t kbeg = warp * kw, kend = min(K, kbeg + kw);
  const Cx* arow[TR];
#pragma unroll
  for (int r = 0; r < TR; ++r) arow[r] = A + min(row0 + r, M - 1) * lda;
  Cx acc[TR][N];
#pragma unroll
  for (int r = 0; r < TR; ++r)
#pragma unroll
    for (int c = 0; c < N; ++c) acc[r][c] = mk<R>(0, 0);
#pragma unroll 2
  for (int64_t k = kbeg + lane; k < kend; k += 32) {
    Cx bv[N];
#pragma unroll
    for (int c = 0; c < N; ++c) bv[c] = __ldg(B + k * ldb + c);
#pragma unroll
    for (int r = 0; r < TR; ++r) {
      const Cx av = __ldg(arow[r] + k);
#pragma unroll
      for (int c = 0; c < N; ++c) cfma(acc[r][c], av, bv[c]);
    }
  }
#pragma unroll
  for (int r = 0; r < TR; ++r)
#pragma unroll
    for (int c = 0; c < N; ++c) {
      Cx v = acc[r][c];
      for (int o = 16; o; o >>= 1) {
        v.x += __shfl_xor_sync(0xffffffffu, v.x, o);
        v.y += __shfl_xor_sync(0xffffffffu, v.y, o);
      }
      if (lane == 0) red[warp][r][c] = v;
    }
  __syncthreads();
  const bool zero_beta = (beta.x == 0 && beta.y == 0);
  for (int t = threadIdx.x; t < TR * N; t += blockDim.x) {
    const int r = t / N, c = t % N;
    const int64_t row = row0 + r;
    if (row >= M) continue;
    Cx v = mk<R>(0, 0);
#pragma unroll
    for (int w = 0; w < THIN_WARPS; ++w) v = cadd(v, red[w][r][c]);
    Cx out = cmul(alpha, v);
    if (!zero_beta) out = cadd(out, cmul(beta, C[row * ldc + c]));
    C[row * ldc + c] = out;
  }
}

// complex64 products with few columns: C (complex64) = alpha A B + beta C (MODE 0, N
// <= 16), or C (complex128) = A B (MODE 1, N <= 8).  Bound by HBM on A (at 4000 rows and
// more far larger than what the caches keep between products).  A CTA of eight
// warps owns 8 RW rows over all of K; B comes in chunks of 512 to 128 rows through
// shared memory (transposed, so that a lane reads its two neighbouring k as one
// 16-byte word per column), the next chunk's entries being loaded while this one
// is used; a lane keeps 4 x RW 16-byte loads of A in flight (two beyond eight
// columns), two CTAs per SM.  The order of every sum is fixed, and a lane adds up each
// chunk by itself first, so that no long chain of FP32 additions builds up (one chain
// per lane costs 1 to 10 % less time but its rounding error is 2.5 times that of a K
// range split over the warps).  Needs an even lda and a 16-byte aligned A; an odd K
// leaves one k to lane 0.  The kernels it replaces read B through L1 per element
// (register tiles: 1.85 TB/s at 12 000 rows) or waited on it per chunk (rows
// streamed by bulk copies: 3.2 TB/s at 24 000); this one reaches 6.0 to
// 6.5 TB/s at 24 000 rows, 5.2 at 12 000 and 3.3 at 4000 up to four columns.  Beyond
// six columns the reads of B from shared memory bound it (12 000 rows: N = 8 452 us,
// 12 700, 16 1081; the register tiles took 1126 and 3859 for the last two).
constexpr int TV_WARPS = 8;
template <int N, int RW, int MODE>
__global__ void __launch_bounds__(32 * TV_WARPS, 2) k_gemm_thin_c64(int64_t M, int64_t K, float2 alpha,
                                                                  const float2* __restrict__ A, int64_t lda,
                                                                  const float2* __restrict__ B, int64_t ldb,
                                                                  float2 beta, void* __restrict__ Cv, int64_t ldc) {
  constexpr int TV_KC = N <= 4 ? 512 : N <= 8 ? 256 : 128;   // k per chunk
  constexpr int U = TV_KC >= 256 ? 4 : 2;              // loads per row in flight
  __shared__ __align__(16) float2 xs[N][TV_KC + 4];
  constexpr int NE = (TV_KC * N + 32 * TV_WARPS - 1) / (32 * TV_WARPS);   // entries of a chunk of B per thread
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int64_t row0 = ((int64_t)blockIdx.x * TV_WARPS + warp) * RW;
  const float2* arow[RW];
#pragma unroll
  for (int r = 0; r < RW; ++r) arow[r] = A + min(row0 + r, M - 1) * lda;
  float2 acc[RW][N];
#pragma unroll
  for (int r = 0; r < RW; ++r)
#pragma unroll
    for (int c = 0; c < N; ++c) acc[r][c] = make_float2(0.f, 0.f);
  const int64_t Ke = K & ~(int64_t)1;                  // even part
  float2 nb[NE];
  const auto fetch = [&](int64_t k0) {
#pragma unroll
    for (int q = 0; q < NE; ++q) {
      const int e = threadIdx.x + 32 * TV_WARPS * q;
      const int64_t k = k0 + e / N;
      nb[q] = k < Ke && e < TV_KC * N ? __ldg(B + k * ldb + e % N) : make_float2(0.f, 0.f);
    }
  };
  fetch(0);
  for (int64_t k0 = 0; k0 < Ke; k0 += TV_KC) {
    __syncthreads();
#pragma unroll
    for (int q = 0; q < NE; ++q) {
      const int e = threadIdx.x + 32 * TV_WARPS * q;
      if (e < TV_KC * N) xs[e % N][e / N] = nb[q];
    }
    __syncthreads();
    if (k0 + TV_KC < Ke) fetch(k0 + TV_KC);
    float2 part[RW][N];
#pragma unroll
    for (int r = 0; r < RW; ++r)
#pragma unroll
      for (int c = 0; c < N; ++c) part[r][c] = make_float2(0.f, 0.f);
#pragma unroll
    for (int h = 0; h < TV_KC / (64 * U); ++h) {       // 64 U k at a time: U 16-byte loads per row
      float4 a[U][RW];
#pragma unroll
      for (int u = 0; u < U; ++u) {
        const int64_t k = k0 + 64 * U * h + 64 * u + 2 * lane;
#pragma unroll
        for (int r = 0; r < RW; ++r)
          a[u][r] = k < Ke ? __ldg(reinterpret_cast<const float4*>(arow[r] + k)) : make_float4(0.f, 0.f, 0.f, 0.f);
      }
#pragma unroll
      for (int u = 0; u < U; ++u) {
        const int kk = 64 * U * h + 64 * u + 2 * lane;
#pragma unroll
        for (int c = 0; c < N; ++c) {
          const float4 b = *reinterpret_cast<const float4*>(&xs[c][kk]);
#pragma unroll
          for (int r = 0; r < RW; ++r) {
            cfma(part[r][c], make_float2(a[u][r].x, a[u][r].y), make_float2(b.x, b.y));
            cfma(part[r][c], make_float2(a[u][r].z, a[u][r].w), make_float2(b.z, b.w));
          }
        }
      }
    }
#pragma unroll
    for (int r = 0; r < RW; ++r)
#pragma unroll
      for (int c = 0; c < N; ++c) acc[r][c] = cadd(acc[r][c], part[r][c]);
  }
  if ((K & 1) && lane == 0) {
#pragma unroll
    for (int r = 0; r < RW; ++r)
#pragma unroll
      for (int c = 0; c < N; ++c) cfma(acc[r][c], arow[r][K - 1], B[(K - 1) * ldb + c]);
  }
  const bool zero_beta = (beta.x == 0 && beta.y == 0);
#pragma unroll
  for (int r = 0; r < RW; ++r)
#pragma unroll
    for (int c = 0; c < N; ++c) {
      float2 v = acc[r][c];
#pragma unroll
      for (int o = 16; o; o >>= 1) {
        v.x += __shfl_xor_sync(0xffffffffu, v.x, o);
        v.y += __shfl_xor_sync(0xffffffffu, v.y, o);
      }
      const int64_t row = row0 + r;
      if (lane == (r * N + c) % 32 && row < M) {
        if (MODE == 0) {
          float2* C = reinterpret_cast<float2*>(Cv);
          float2 out = cmul(alpha, v);
          if (!zero_beta) out = cadd(out, cmul(beta, C[row * ldc + c]));
          C[row * ldc + c] = out;
        } else {
          reinterpret_cast<double2*>(Cv)[row * ldc + c] = make_double2(v.x, v.y);
        }
      }
    }
}

template <int MODE>
static mnpbem_status launch_thin_c64(int64_t M, int64_t N, int64_t K, const float2* A, int64_t lda, const float2* B,
                                     int64_t ldb, float2 alpha, float2 beta, void* C, int64_t ldc, cudaStream_t st) {
  // rows per warp: four with up to two columns, two up to six, one beyond (the sums
  // and the loads in flight fill the registers: at 24 000 rows N = 3 takes 707 us
  // with two and 873 with four, N = 4 763 and 951; 2904 rows, N = 8: 50 us with
  // one, 56 with two); fewer where the rows would not give every SM a CTA
#define TV_CASE(NN, RW)                                                                                              \
  k_gemm_thin_c64<NN, RW, MODE><<<(unsigned)cdiv_up(M, (int64_t)(TV_WARPS * RW)), 32 * TV_WARPS, 0, st>>>(           \
      M, K, alpha, A, lda, B, ldb, beta, C, ldc)
#define TV_N(NN, RW)                                     \
  case NN:                                               \
    if (M >= 2 * 152 * TV_WARPS * RW) TV_CASE(NN, RW);   \
    else if (M >= 152 * TV_WARPS * 2) TV_CASE(NN, 2);    \
    else TV_CASE(NN, 1);                                 \
    break;
#define TV_1(NN) case NN: TV_CASE(NN, 1); break;
  switch (N) {
    TV_N(1, 4) TV_N(2, 4) TV_N(3, 2) TV_N(4, 2) TV_N(5, 2) TV_N(6, 2) TV_N(7, 1) TV_N(8, 1)
    default:
      if constexpr (MODE == 0) {
        switch (N) {
          TV_1(9) TV_1(10) TV_1(11) TV_1(12) TV_1(13) TV_1(14) TV_1(15) TV_1(16)
          default: break;
        }
      }
      if (MODE != 0 || N < 1 || N > THIN_NMAX) {
        set_error("thin product: unsupported number of columns");
        return MNPBEM_ERR_INVALID_ARG;
      }
  }
#undef TV_1
#undef TV_N
#undef TV_CASE
  MNP_CHECK_LAUNCH();
  return MNPBEM_OK;
}

// ------------------------------------------- double-single thin GEMM (N <= 16)
constexpr int DS_WARPS = 8, DS_TR = 4;

// B (complex128) -> hi / lo complex64 planes
__global__ void k_split_hi_lo(const double2* __restrict__ B, int64_t count, float2* hi, float2* lo) {
  const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= count) return;
  const double2 b = B[i];
  const float2 h = make_float2((float)b.x, (float)b.y);
  hi[i] = h;
  lo[i] = make_float2((float)(b.x - (double)h.x), (float)(b.y - (double)h.y));
}

template <int N, int TR, int UNR>
__global__ void __launch_bounds__(32 * DS_WARPS) k_gemm_thin_ds(int64_t M, int64_t K, const float2* __restrict__ Ahi,
                                                              const float2* __restrict__ Alo, int64_t lda,
                                                              const float2* __restrict__ Bh,
                                                              const float2* __restrict__ Bl, int64_t ldb,
                                                              double2* __restrict__ C, int64_t ldc) {
  __shared__ DS red[DS_WARPS][TR][N][2];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int64_t row0 = (int64_t)blockIdx.x * TR;
  const int64_t kw = (K + DS_WARPS - 1) / DS_WARPS;
  const int64_t kbeg = warp * kw, kend = min(K, kbeg + kw);
  int64_t roff[TR];
#pragma unroll
  for (int r = 0; r < TR; ++r) roff[r] = min(row0 + r, M - 1) * lda;
  DS re[TR][N], im[TR][N];
#pragma unroll
  for (int r = 0; r < TR; ++r)
#pragma unroll
    for (int c = 0; c < N; ++c) re[r][c] = im[r][c] = DS{0.f, 0.f};
#pragma unroll UNR
  for (int64_t k = kbeg + lane; k < kend; k += 32) {
    float2 xh[N], xl[N];
#pragma unroll
    for (int c = 0; c < N; ++c) {
      xh[c] = __ldg(Bh + k * ldb + c);
      xl[c] = __ldg(Bl + k * ldb + c);
    }
#pragma unroll
    for (int r = 0; r < TR; ++r) {
      const float2 ah = __ldg(Ahi + roff[r] + k), al = __ldg(Alo + roff[r] + k);
#pragma unroll
      for (int c = 0; c < N; ++c) {
        ds_cfma(re[r][c], im[r][c], ah, al, xh[c], xl[c]);
      }
    }
  }
#pragma unroll
  for (int r = 0; r < TR; ++r)
#pragma unroll
    for (int c = 0; c < N; ++c) {
      DS a = re[r][c], b = im[r][c];
      for (int o = 16; o; o >>= 1) {
        DS oa{__shfl_xor_sync(0xffffffffu, a.hi, o), __shfl_xor_sync(0xffffffffu, a.lo, o)};
        DS ob{__shfl_xor_sync(0xffffffffu, b.hi, o), __shfl_xor_sync(0xffffffffu, b.lo, o)};
        a = ds_add(a, oa);
        b = ds_add(b, ob);
      }
      if (lane == 0) { red[warp][r][c][0] = a; red[warp][r][c][1] = b; }
    }
  __syncthreads();
  for (int t = threadIdx.x; t < TR * N; t += blockDim.x) {
    const int r = t / N, c = t % N;
    const int64_t row = row0 + r;
    if (row >= M) continue;
    DS a{0.f, 0.f}, b{0.f, 0.f};
#pragma unroll
    for (int w = 0; w < DS_WARPS; ++w) {
      a = ds_add(a, red[w][r][c][0]);
      b = ds_add(b, red[w][r][c][1]);
    }
    C[row * ldc + c] = make_double2((double)a.hi + (double)a.lo, (double)b.hi + (double)b.lo);
  }
}

// FP32 variant of the same product from the hi planes only (plain FMA
// accumulation): for refinement steps whose residual is still large.
template <int N>
__global__ void __launch_bounds__(32 * DS_WARPS) k_gemm_thin_hi(int64_t M, int64_t K, const float2* __restrict__ Ahi,
                                                              int64_t lda, const float2* __restrict__ Bh, int64_t ldb,
                                                              double2* __restrict__ C, int64_t ldc) {
  __shared__ float2 red[DS_WARPS][DS_TR][N];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int64_t row0 = (int64_t)blockIdx.x * DS_TR;
  const int64_t kw = (K + DS_WARPS - 1) / DS_WARPS;
  const int64_t kbeg = warp * kw, kend = min(K, kbeg + kw);
  int64_t roff[DS_TR];
#pragma unroll
  for (int r = 0; r < DS_TR; ++r) roff[r] = min(row0 + r, M - 1) * lda;
  float2 acc[DS_TR][N];
#pragma unroll
  for (int r = 0; r < DS_TR; ++r)
#pragma unroll
    for (int c = 0; c < N; ++c) acc[r][c] = make_float2(0.f, 0.f);
#pragma unroll 2
  for (int64_t k = kbeg + lane; k < kend; k += 32) {
    float2 xh[N];
#pragma unroll
    for (int c = 0; c < N; ++c) xh[c] = __ldg(Bh + k * ldb + c);
#pragma unroll
    for (int r = 0; r < DS_TR; ++r) {
      const float2 ah = __ldg(Ahi + roff[r] + k);
#pragma unroll
      for (int c = 0; c < N; ++c) cfma(acc[r][c], ah, xh[c]);
    }
  }
#pragma unroll
  for (int r = 0; r < DS_TR; ++r)
#pragma unroll
    for (int c = 0; c < N; ++c) {
      float2 v = acc[r][c];
      for (int o = 16; o; o >>= 1) {
        v.x += __shfl_xor_sync(0xffffffffu, v.x, o);
        v.y += __shfl_xor_sync(0xffffffffu, v.y, o);
      }
      if (lane == 0) red[warp][r][c] = v;
    }
  __syncthreads();
  for (int t = threadIdx.x; t < DS_TR * N; t += blockDim.x) {
    const int r = t / N, c = t % N;
    const int64_t row = row0 + r;
    if (row >= M) continue;
    float2 v = make_float2(0.f, 0.f);
#pragma unroll
    for (int w = 0; w < DS_WARPS; ++w) v = cadd(v, red[w][r][c]);
    C[row * ldc + c] = make_double2(v.x, v.y);
  }
}

__device__ int g_sweep_err;   // a bounded wait of the triangular sweeps expired

// the current device's number, as an index into per-device tables (the last entry is
// shared by all devices beyond it and never kept)
constexpr int MAX_DEVICES = 64;
static int device_index() {
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess) cudaGetLastError();
  return dev >= 0 && dev < MAX_DEVICES ? dev : MAX_DEVICES;
}
static int num_sms() {
  static std::atomic<int> kept[MAX_DEVICES];
  const int d = device_index();
  int sms = d < MAX_DEVICES ? kept[d].load() : 0;
  if (!sms) {
    int dev = 0;
    cudaGetDevice(&dev);
    if (cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess || sms <= 0) {
      cudaGetLastError();
      sms = 148;
    }
    if (d < MAX_DEVICES) kept[d] = sms;
  }
  return sms;
}

mnpbem_status sweep_check(cudaStream_t st) {
  int* p = nullptr;
  MNP_CUDA(cudaGetSymbolAddress(reinterpret_cast<void**>(&p), g_sweep_err));
  int h = 0;
  MNP_CUDA(cudaMemcpyAsync(&h, p, sizeof(int), cudaMemcpyDeviceToHost, st));
  MNP_CUDA(cudaStreamSynchronize(st));
  if (h) {
    MNP_CUDA(cudaMemsetAsync(p, 0, sizeof(int), st));
    set_error("triangular sweep: a bounded wait expired (code %d)", h);
    return MNPBEM_ERR_TIMEOUT;
  }
  return MNPBEM_OK;
}

// B[:, 0:N] (row stride ldb) -> packed hi / lo planes [K][N]
__global__ void k_split_hi_lo_cols(const double2* __restrict__ B, int64_t ldb, int64_t K, int N, float2* hi,
                                   float2* lo) {
  const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= K * N) return;
  const int64_t k = i / N;
  const double2 b = B[k * ldb + (i - k * N)];
  const float2 h = make_float2((float)b.x, (float)b.y);
  hi[i] = h;
  lo[i] = make_float2((float)(b.x - (double)h.x), (float)(b.y - (double)h.y));
}

static mnpbem_status gemm_thin_ds_block(int64_t M, int64_t N, int64_t K, const float2* Ahi, const float2* Alo,
                                        int64_t lda, const double2* B, int64_t ldb, double2* C, int64_t ldc,
                                        float2* bsplit, cudaStream_t st) {
  float2* Bh = bsplit;
  float2* Bl = bsplit + K * N;
  {
    ProfScope ps(PH_ELEMWISE, st, 0.0, 0.0, 1);
    if (ldb == N)
      k_split_hi_lo<<<(unsigned)cdiv_up(K * N, 256), 256, 0, st>>>(B, K * N, Bh, Bl);
    else
      k_split_hi_lo_cols<<<(unsigned)cdiv_up(K * N, 256), 256, 0, st>>>(B, ldb, K, (int)N, Bh, Bl);
    MNP_CHECK_LAUNCH();
  }
  const unsigned nblk = (unsigned)cdiv_up(M, (int64_t)DS_TR);
  if (!Alo) {
    ProfScope ps(PH_GEMM_SMALL, st, 8.0 * M * N * K, 8.0 * M * K + 8.0 * K * N + 16.0 * M * N);
    if (!(lda & 1) && !(reinterpret_cast<uintptr_t>(Ahi) & 15))
      return launch_thin_c64<1>(M, N, K, Ahi, lda, Bh, N, make_float2(1.f, 0.f), make_float2(0.f, 0.f), C, ldc, st);
#define HI_CASE(NN)                                                                                \
  case NN:                                                                                         \
    k_gemm_thin_hi<NN><<<nblk, 32 * DS_WARPS, 0, st>>>(M, K, Ahi, lda, Bh, N, C, ldc);        \
    break;
    switch (N) {
      HI_CASE(1) HI_CASE(2) HI_CASE(3) HI_CASE(4) HI_CASE(5) HI_CASE(6) HI_CASE(7) HI_CASE(8)
    }
#undef HI_CASE
    MNP_CHECK_LAUNCH();
    return MNPBEM_OK;
  }
  ProfScope ps(PH_GEMM_SMALL, st, 8.0 * M * N * K, 16.0 * M * K + 16.0 * K * N + 16.0 * M * N);
  // two rows per block (80 registers, 3 blocks per SM) measured faster than
  // four rows (128 registers) or an unrolled k loop
  constexpr int TR = 2;
  const unsigned nb2 = (unsigned)cdiv_up(M, (int64_t)TR);
#define DS_CASE(NN)                                                                                        \
  case NN:                                                                                                 \
    k_gemm_thin_ds<NN, TR, 1><<<nb2, 32 * DS_WARPS, 0, st>>>(M, K, Ahi, Alo, lda, Bh, Bl, N, C, ldc);       \
    break;
  switch (N) {
    DS_CASE(1) DS_CASE(2) DS_CASE(3) DS_CASE(4) DS_CASE(5) DS_CASE(6) DS_CASE(7) DS_CASE(8)
  }
#undef DS_CASE
  MNP_CHECK_LAUNCH();
  return MNPBEM_OK;
}

// columns in blocks of at most 8 (the kernels' register-tiled widths)
mnpbem_status gemm_thin_ds(int64_t M, int64_t N, int64_t K, const float2* Ahi, const float2* Alo,
                           int64_t lda, const double2* B, int64_t ldb, double2* C, int64_t ldc,
                           float2* bsplit, cudaStream_t st) {
  if (M <= 0 || N <= 0) return MNPBEM_OK;
  if (K <= 0 || ldb < N) { set_error("gemm_thin_ds: invalid sizes"); return MNPBEM_ERR_INVALID_ARG; }
  for (int64_t c0 = 0; c0 < N; c0 += 8) {
    const int64_t w = std::min<int64_t>(8, N - c0);
    MNP_TRY(gemm_thin_ds_block(M, w, K, Ahi, Alo, lda, B + c0, ldb, C + c0, ldc, bsplit, st));
  }
  return MNPBEM_OK;
}

template <typename R>
mnpbem_status gemm_simt(int64_t M, int64_t N, int64_t K, cplx<R> alpha, const cplx<R>* A,
                        int64_t lda, const cplx<R>* B, int64_t ldb, cplx<R> beta, cplx<R>* C,
                        int64_t ldc, cudaStream_t st) {
  if (M <= 0 || N <= 0) return MNPBEM_OK;
  if (sizeof(R) == 4 && N <= THIN_NMAX && K > 1 && !(lda & 1) && !(reinterpret_cast<uintptr_t>(A) & 15)) {
    ProfScope ps(PH_GEMM_SMALL, st, 8.0 * M * N * K,
                 (double)sizeof(cplx<R>) * ((double)M * K + (double)K * N + 2.0 * M * N));
    const float2* Af = reinterpret_cast<const float2*>(A);
    const float2* Bf = reinterpret_cast<const float2*>(B);
    float2* Cf = reinterpret_cast<float2*>(C);
    const float2 al = make_float2((float)alpha.x, (float)alpha.y), be = make_float2((float)beta.x, (float)beta.y);
    return launch_thin_c64<0>(M, N, K, Af, lda, Bf, ldb, al, be, Cf, ldc, st);
  }
  if (N <= THIN_NMAX && K > 0) {
    ProfScope ps(PH_GEMM_SMALL, st, 8.0 * M * N * K,
                 (double)sizeof(cplx<R>) * ((double)M * K + (double)K * N + 2.0 * M * N));
    // rows per block: fewer for wide B so that the accumulators stay in registers
#define THIN_CASE(NN)                                                                              \
  case NN: {                                                                                       \
    constexpr int TR = NN <= 8 ? 4 : (sizeof(R) == 8 ? 1 : 2);                                     \
    k_gemm_thin<R, NN, TR><<<(unsigned)cdiv_up(M, TR), 32 * THIN_WARPS, 0, st>>>(M, K, alpha, A, lda, B, ldb, beta, C, ldc); \
    break;                                                                                         \
  }
    switch (N) {
      THIN_CASE(1) THIN_CASE(2) THIN_CASE(3) THIN_CASE(4) THIN_CASE(5) THIN_CASE(6) THIN_CASE(7)
      THIN_CASE(8) THIN_CASE(9) THIN_CASE(10) THIN_CASE(11) THIN_CASE(12) THIN_CASE(13) THIN_CASE(14)
      THIN_CASE(15) THIN_CASE(16)
    }
#undef THIN_CASE
    MNP_CHECK_LAUNCH();
    return MNPBEM_OK;
  }
  dim3 grid((unsigned)cdiv_up(N, 64), (unsigned)cdiv_up(M, 64));
  if (grid.y > 65535) { set_error("gemm_simt: M too large"); return MNPBEM_ERR_INVALID_ARG; }
  constexpr int BK = sizeof(R) == 4 ? 16 : 8;
  const bool big = M >= 128 && N >= 128;
  // complex64 products that would leave half of the SMs without a 64 x 64 tile
  // (76 tiles and fewer: 512 x 512 x 64, 64 tiles, 9 us and 16 with the large tile);
  // C may not overlap A or B in either
  if constexpr (sizeof(R) == 4) {
    if (K >= 16 && (int64_t)grid.x * grid.y <= 76) {
      ProfScope ps(PH_GEMM_SMALL, st, 8.0 * M * N * K, 8.0 * ((double)M * K + (double)K * N + 2.0 * M * N));
      k_gemm_small<<<dim3((unsigned)cdiv_up(N, (int64_t)SG_N), (unsigned)cdiv_up(M, (int64_t)SG_M)), 256, 0, st>>>(
          M, N, K, alpha, A, lda, B, ldb, beta, C, ldc);
      MNP_CHECK_LAUNCH();
      return MNPBEM_OK;
    }
  }
  ProfScope ps(big ? PH_GEMM_BIG : PH_GEMM_SMALL, st, 8.0 * M * N * K,
               (double)sizeof(cplx<R>) * ((double)M * K + (double)K * N + 2.0 * M * N));
  k_gemm_nn<R, BK><<<grid, 256, 0, st>>>(M, N, K, alpha, A, lda, B, ldb, beta, C, ldc);
  MNP_CHECK_LAUNCH();
  return MNPBEM_OK;
}
template mnpbem_status gemm_simt<float>(int64_t, int64_t, int64_t, float2, const float2*, int64_t,
                                        const float2*, int64_t, float2, float2*, int64_t, cudaStream_t);
template mnpbem_status gemm_simt<double>(int64_t, int64_t, int64_t, double2, const double2*, int64_t,
                                         const double2*, int64_t, double2, double2*, int64_t,
                                         cudaStream_t);

// --------------------------------------------------- block inversion
// Largest per-block condition proxy max|A_kk| * max|inv(A_kk)|, kept as the
// bits of a non-negative float in status[1] (integer order = float order).
__device__ __forceinline__ void record_cond(int* status, double amax, double xmax) {
  double c = amax * xmax;
  if (!(c == c) || c > 3.0e38) c = 3.0e38;
  atomicMax(status + 1, __float_as_int((float)c));
}

// 1 / x in FP32: the hardware's approximate reciprocal and one Newton step
// (x in 1e-30 .. 1e30; within 1 ulp of the rounded quotient, and without the
// division's range handling on the serial chain of the pivot steps)
__device__ __forceinline__ float rcp_newton(float x) {
  float r;
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
  return fmaf(r, fmaf(-x, r, 1.f), r);
}

// Row of the largest key among 64 candidates, keys of rows lane and lane + 32 in
// k0 and k1 (0 = not a candidate); the lowest row on ties.  Every lane gets it.
__device__ __forceinline__ int argmax64(unsigned k0, unsigned k1) {
  const unsigned mx = __reduce_max_sync(0xffffffffu, max(k0, k1));
  const unsigned b0 = __ballot_sync(0xffffffffu, k0 == mx), b1 = __ballot_sync(0xffffffffu, k1 == mx);
  return b0 ? __ffs(b0) - 1 : 31 + __ffs(b1);
}

// In-place Gauss-Jordan of one w x w complex64 block (w <= 64) with partial
// pivoting inside the block.  256 threads as a 16 x 16 grid; thread (ty, tx)
// keeps the 16 entries (ty + 16 i, tx + 16 j) in registers.  Pivoting is
// implicit: step p takes as pivot row r_p the row, among those not yet used,
// with the largest |a_rp| in column p, and eliminates with (r_p, p) in place of
// (p, p).  The matrix M this leaves satisfies inv(A)[q][r_k] = M[r_q][k], so the
// block is written out through the permutation, to X and, when X2 is given, to
// X2 as well (X2 may be the input: it is read before the first barrier).  Two
// __syncthreads per step: after the pivot column is published, and after the
// pivot row is.
// Bound by the latency of the chain of 64 steps (one CTA).  Each warp finds the
// pivot with one integer reduction over the 64 candidates' moduli; a scan of
// the column by every thread took most of a step (160 us per block of 64 in a
// sweep, 41 us now).
__global__ void __launch_bounds__(256) k_block_inv(const float2* A, int64_t lda, int w, float2* X, int64_t ldx,
                                                   float2* X2, int64_t ldx2, int* status) {
  __shared__ float2 prow[2][64], pcol[2][64];
  __shared__ int prow_of[64], pos_of[64];
  __shared__ float red[2][8];
  const int t = threadIdx.x, tx = t & 15, ty = t >> 4, lane = t & 31;
  float2 a[4][4];
  float amax = 0.f;
#pragma unroll
  for (int i = 0; i < 4; ++i)
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const int r = ty + 16 * i, c = tx + 16 * j;
      a[i][j] = (r < w && c < w) ? A[r * lda + c] : make_float2(r == c ? 1.f : 0.f, 0.f);
      if (r < w && c < w) amax = fmaxf(amax, sqrtf(a[i][j].x * a[i][j].x + a[i][j].y * a[i][j].y));
    }
  // rows still free, lane and lane + 32 (the same in every warp)
  bool free0 = lane < w, free1 = lane + 32 < w;
  for (int p = 0; p < w; ++p) {
    const int buf = p & 1;
    // 1. publish column p
#pragma unroll
    for (int j = 0; j < 4; ++j)
      if (tx + 16 * j == p) {
#pragma unroll
        for (int i = 0; i < 4; ++i) pcol[buf][ty + 16 * i] = a[i][j];
      }
    __syncthreads();
    // 2. pivot row: largest modulus among the free rows (first one on ties);
    //    the bits of a non-negative float order as integers, + 1 keeps a free
    //    row with a zero entry above the used ones
    const float2 v0 = pcol[buf][lane], v1 = pcol[buf][lane + 32];
    const unsigned k0 = free0 ? __float_as_uint(v0.x * v0.x + v0.y * v0.y) + 1u : 0u;
    const unsigned k1 = free1 ? __float_as_uint(v1.x * v1.x + v1.y * v1.y) + 1u : 0u;
    const int rp = argmax64(k0, k1);
    free0 = free0 && rp != lane;
    free1 = free1 && rp != lane + 32;
    // 3. publish the pivot row
#pragma unroll
    for (int i = 0; i < 4; ++i)
      if (ty + 16 * i == rp) {
#pragma unroll
        for (int j = 0; j < 4; ++j) prow[buf][tx + 16 * j] = a[i][j];
      }
    const float2 piv = pcol[buf][rp];
    const float n2 = piv.x * piv.x + piv.y * piv.y;
    const float rn2 = rcp_newton(n2);
    const float2 inv = make_float2(piv.x * rn2, -piv.y * rn2);
    if (t == 0) {
      if (!(n2 > 1e-30f && n2 < 1e30f)) atomicOr(status, 1);
      prow_of[p] = rp;
      pos_of[rp] = p;
    }
    // a_rc <- a_rc - m_r row_c with m_r = a_rp / a_pp; the pivot row keeps
    // row_c / a_pp (from 0 with m = -1 / a_pp), the pivot column -m_r (from 0
    // with row_p = 1)
    float2 m[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      m[i] = cmul(pcol[buf][ty + 16 * i], inv);
      if (ty + 16 * i == rp) {
        m[i] = make_float2(-inv.x, -inv.y);
#pragma unroll
        for (int j = 0; j < 4; ++j) a[i][j] = make_float2(0.f, 0.f);
      }
    }
    __syncthreads();
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      float2 row = prow[buf][tx + 16 * j];
      if (tx + 16 * j == p) {
        row = make_float2(1.f, 0.f);
#pragma unroll
        for (int i = 0; i < 4; ++i) a[i][j] = make_float2(0.f, 0.f);
      }
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        a[i][j].x = fmaf(-m[i].x, row.x, a[i][j].x);
        a[i][j].y = fmaf(-m[i].x, row.y, a[i][j].y);
        a[i][j].x = fmaf(m[i].y, row.y, a[i][j].x);
        a[i][j].y = fmaf(-m[i].y, row.x, a[i][j].y);
      }
    }
  }
  __syncthreads();
  float xmax = 0.f;
#pragma unroll
  for (int i = 0; i < 4; ++i)
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const int r = ty + 16 * i, c = tx + 16 * j;
      if (r < w && c < w) {
        X[(int64_t)pos_of[r] * ldx + prow_of[c]] = a[i][j];
        if (X2) X2[(int64_t)pos_of[r] * ldx2 + prow_of[c]] = a[i][j];
        xmax = fmaxf(xmax, sqrtf(a[i][j].x * a[i][j].x + a[i][j].y * a[i][j].y));
      }
    }
  // block maxima of |A| and |X| for the condition proxy
  for (int o = 16; o; o >>= 1) {
    amax = fmaxf(amax, __shfl_xor_sync(0xffffffffu, amax, o));
    xmax = fmaxf(xmax, __shfl_xor_sync(0xffffffffu, xmax, o));
  }
  if (lane == 0) { red[0][t >> 5] = amax; red[1][t >> 5] = xmax; }
  __syncthreads();
  if (t == 0) {
    float am = 0.f, xm = 0.f;
    for (int k = 0; k < 8; ++k) { am = fmaxf(am, red[0][k]); xm = fmaxf(xm, red[1][k]); }
    record_cond(status, am, xm);
  }
}

// The same elimination for a complex128 block (w <= 64) on a cluster of eight
// CTAs: CTA q keeps columns 8 q .. 8 q + 7 (thread = row, two columns each), so
// that the FP64 pipes of eight SMs share the rank-1 updates (FP64 runs at two
// FMA per clock per SM: 64^3 complex multiply-adds are 270 us on one SM).
// Step p: every warp picks the pivot row from integer keys of |re| + |im| (the
// pivot measure of LAPACK's izamax); the row's eight local columns go to shared
// memory, and each thread updates its two entries.  The owner of column p + 1
// updates it first and writes it, with its keys, into every CTA's shared memory
// before it arrives at the cluster barrier of step p + 1, so that the exchange
// overlaps the other updates.  The buffers alternate: a CTA that writes column
// p + 2 has passed barrier p + 1, at which every CTA arrives after reading
// column p, and one that writes its pivot row p + 2 has passed barrier p + 2,
// at which its threads arrive after update p.
// One CTA with the pivot scan in every thread took 1059 us per block of 64;
// this takes 105 us.
constexpr int BD_CL = 8, BD_THREADS = 256;
__global__ void __cluster_dims__(BD_CL, 1, 1) __launch_bounds__(BD_THREADS)
    k_block_inv_c128(const double2* A, int64_t lda, int w, double2* X, int64_t ldx, double2* X2, int64_t ldx2,
                     int* status) {
  namespace cg = cooperative_groups;
  cg::cluster_group cluster = cg::this_cluster();
  __shared__ double2 pcol[2][64], prow[2][8];
  __shared__ unsigned pkey[2][64];
  __shared__ int prow_of[64], pos_of[64];
  __shared__ double red[2][BD_THREADS / 32], cond_loc[2];
  const int rank = (int)cluster.block_rank();
  const int t = threadIdx.x, lane = t & 31, r = t & 63, cg2 = t >> 6;
  double2 a[2];
  double amax = 0.0, xmax = 0.0;
#pragma unroll
  for (int j = 0; j < 2; ++j) {
    const int c = 8 * rank + 2 * cg2 + j;
    a[j] = (r < w && c < w) ? A[(int64_t)r * lda + c] : make_double2(r == c ? 1.0 : 0.0, 0.0);
    if (r < w && c < w) amax = fmax(amax, sqrt(cabs2(a[j])));
  }
  bool free0 = lane < w, free1 = lane + 32 < w;
  // column p (value v of this thread's row) and its keys into every CTA
  const auto publish = [&](int p, double2 v) {
    const unsigned key = (unsigned)__double2hiint(fabs(v.x) + fabs(v.y)) + 1u;
#pragma unroll
    for (int q = 0; q < BD_CL; ++q) {
      cluster.map_shared_rank(&pcol[p & 1][0], q)[r] = v;
      cluster.map_shared_rank(&pkey[p & 1][0], q)[r] = key;
    }
  };
  cluster.sync();   // every CTA runs before its shared memory is written
  if (rank == 0 && cg2 == 0) publish(0, a[0]);
  cluster.barrier_arrive();
  for (int p = 0; p < w; ++p) {
    const int buf = p & 1, lc = p - 8 * rank;      // local column of the pivot, if 0 <= lc < 8
    cluster.barrier_wait();
    const unsigned k0 = free0 ? pkey[buf][lane] : 0u, k1 = free1 ? pkey[buf][lane + 32] : 0u;
    const int rp = argmax64(k0, k1);
    free0 = free0 && rp != lane;
    free1 = free1 && rp != lane + 32;
    const bool isrow = r == rp;
    // the pivot row's local entries, scaled by the reciprocal pivot in one warp
    // (1 in the pivot column): a_rc <- a_rc - m_r row_c with m_r = a_rp, the
    // pivot row (m = -1) and the pivot column starting from 0
    if (isrow) {
      prow[buf][2 * cg2] = lc == 2 * cg2 ? make_double2(1.0, 0.0) : a[0];
      prow[buf][2 * cg2 + 1] = lc == 2 * cg2 + 1 ? make_double2(1.0, 0.0) : a[1];
      a[0] = a[1] = make_double2(0.0, 0.0);
    }
    double2 inv = make_double2(0.0, 0.0);
    if (t < 32) {
      const double2 piv = pcol[buf][rp];
      const double n2 = piv.x * piv.x + piv.y * piv.y, rn2 = 1.0 / n2;
      inv = make_double2(piv.x * rn2, -piv.y * rn2);
      if (t == 0) {
        if (rank == 0 && !(n2 > 1e-30 && n2 < 1e30)) atomicOr(status, 1);
        prow_of[p] = rp;
        pos_of[rp] = p;
      }
    }
    const double2 m = isrow ? make_double2(-1.0, 0.0) : pcol[buf][r];
    __syncthreads();
    if (t < 8) prow[buf][t] = cmul(prow[buf][t], inv);
    __syncthreads();
    const auto update = [&](int j) {
      const double2 row = prow[buf][2 * cg2 + j];
      const double2 base = lc == 2 * cg2 + j ? make_double2(0.0, 0.0) : a[j];
      a[j].x = fma(m.y, row.y, fma(-m.x, row.x, base.x));
      a[j].y = fma(-m.y, row.x, fma(-m.x, row.y, base.y));
    };
    // the next pivot column first: its exchange overlaps the other updates
    const int nx = lc + 1 - 2 * cg2;               // local index of column p + 1 in this thread, if 0 or 1
    const bool next = p + 1 < w && lc + 1 >= 0 && lc + 1 < 8 && (nx == 0 || nx == 1);
    if (next) {
      if (nx == 0) { update(0); publish(p + 1, a[0]); }
      else { update(1); publish(p + 1, a[1]); }
    }
    cluster.barrier_arrive();
    if (!next || nx != 0) update(0);
    if (!next || nx != 1) update(1);
  }
  cluster.barrier_wait();
#pragma unroll
  for (int j = 0; j < 2; ++j) {
    const int c = 8 * rank + 2 * cg2 + j;
    if (r < w && c < w) {
      X[(int64_t)pos_of[r] * ldx + prow_of[c]] = a[j];
      if (X2) X2[(int64_t)pos_of[r] * ldx2 + prow_of[c]] = a[j];
      xmax = fmax(xmax, sqrt(cabs2(a[j])));
    }
  }
  for (int o = 16; o; o >>= 1) {
    amax = fmax(amax, __shfl_xor_sync(0xffffffffu, amax, o));
    xmax = fmax(xmax, __shfl_xor_sync(0xffffffffu, xmax, o));
  }
  if (lane == 0) { red[0][t >> 5] = amax; red[1][t >> 5] = xmax; }
  __syncthreads();
  if (t < 2) {
    double mx = 0.0;
    for (int k = 0; k < BD_THREADS / 32; ++k) mx = fmax(mx, red[t][k]);
    cond_loc[t] = mx;
  }
  cluster.sync();
  if (rank == 0 && t == 0) {
    double am = 0.0, xm = 0.0;
    for (int q = 0; q < BD_CL; ++q) {
      const double* cl = cluster.map_shared_rank(cond_loc, q);
      am = fmax(am, cl[0]);
      xm = fmax(xm, cl[1]);
    }
    record_cond(status, am, xm);
  }
  cluster.sync();   // no CTA may exit while another can still read its shared memory
}

static mnpbem_status launch_block_inv(const float2* A, int64_t lda, int w, float2* X, int64_t ldx, float2* X2,
                                      int64_t ldx2, int* status, cudaStream_t st) {
  ProfScope ps(PH_BLOCKINV, st, 8.0 * w * w * w, 0.0);
  k_block_inv<<<1, 256, 0, st>>>(A, lda, w, X, ldx, X2, ldx2, status);
  MNP_CHECK_LAUNCH();
  return MNPBEM_OK;
}
static mnpbem_status launch_block_inv(const double2* A, int64_t lda, int w, double2* X, int64_t ldx, double2* X2,
                                      int64_t ldx2, int* status, cudaStream_t st) {
  ProfScope ps(PH_BLOCKINV, st, 8.0 * w * w * w, 0.0);
  k_block_inv_c128<<<BD_CL, BD_THREADS, 0, st>>>(A, lda, w, X, ldx, X2, ldx2, status);
  MNP_CHECK_LAUNCH();
  return MNPBEM_OK;
}

// ------------------------------------- 256-wide pivot block on a CTA cluster
// In-place Gauss-Jordan of one w x w complex64 block (w <= 256) by a cluster
// of PB_CL CTAs.  CTA r keeps rows [r*PB_RPC, (r+1)*PB_RPC) in registers: thread
// (ty, tx) the 4 x 4 entries of rows 4 ty + i and columns tx + 64 j.  The pivots
// are taken in panels of 16:
//   1. the CTA that owns the panel rows has written them (P, 16 x 256, raw) and
//      the inverse X of their pivot block to a scratch in global memory; every
//      CTA stages its own 16 panel-column entries C; cluster barrier;
//   2. every CTA reads X and P back (L2); four warps form D = C X for the CTA's
//      rows (for the panel rows themselves D = -X) while the others stage P in
//      shared memory, with the panel's own columns replaced by the identity;
//   3. a_ij <- [i, j not pivots] a_ij - sum_k D_ik P_kj.  Meanwhile four more
//      warps of the CTA that owns the next panel apply the same update to the
//      next 16 x 16 pivot block and invert it (one warp alone, competing with
//      the update for its scheduler, took longer than the update).
// The panel goes through L2 because a broadcast out of one SM's shared memory
// (distributed shared memory, 7 x 32 KB from one source per panel) is limited
// by that SM's port, and D = C X (32 x 16 x 16 per CTA) replaces R = X P on one
// CTA.  One cluster barrier per panel, 16 panels for w = 256: the scratch and
// the next pivot block alternate between two buffers, and a CTA that writes
// panel p + 2 has passed barrier p + 1, which every CTA reaches after reading
// panel p.
// The rank-16 updates are 34 us of FP32 FMA on eight SMs; 95 us measured
// for w = 256 (248 us with the pivot block and R on the owner and R read from
// its shared memory).
// Rows and columns beyond w are identity and stay identity.
constexpr int PB_W = 256, PB_CL = 8, PB_RPC = PB_W / PB_CL, PB_THREADS = 512, PB_PAN = 16;
constexpr int PB_LD = PB_RPC + 2;      // row stride of C and D: 16-byte aligned, spread over the banks
constexpr int PB_BUF = PB_PAN * (PB_W + PB_PAN);   // one panel and the inverse of its pivot block
constexpr int PB_SCRATCH = 2 * PB_BUF * (int)sizeof(float2);
constexpr int PB_ALL = PB_THREADS + 128;           // and the pivot warps
static_assert(PB_RPC % PB_PAN == 0, "a panel lies inside one CTA");
static_assert(PB_THREADS == 64 * (PB_RPC / 4), "4 x 4 entries per thread");

__device__ __forceinline__ void named_sync(int id, int threads) {
  asm volatile("bar.sync %0, %1;" ::"r"(id), "r"(threads) : "memory");
}

// (c.x, c.y) += a (b.x, b.y), lane by lane: two FP32 multiply-adds in one instruction
__device__ __forceinline__ void fma2(float2& c, float2 a, float2 b) {
  unsigned long long cc, aa, bb;
  asm("mov.b64 %0, {%1, %2};" : "=l"(cc) : "f"(c.x), "f"(c.y));
  asm("mov.b64 %0, {%1, %2};" : "=l"(aa) : "f"(a.x), "f"(a.y));
  asm("mov.b64 %0, {%1, %2};" : "=l"(bb) : "f"(b.x), "f"(b.y));
  asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(cc) : "l"(aa), "l"(bb));
  asm("mov.b64 {%0, %1}, %2;" : "=f"(c.x), "=f"(c.y) : "l"(cc));
}

// 16 x 16 Gauss-Jordan by four warps (threads u = 0 .. 127): warp q holds
// columns 4 q .. 4 q + 3, lane (r, h) row r and columns 4 q + 2 h, + 1 in v.
// The pivot column passes through shared memory (one named barrier per step),
// the pivot row through shuffles.  col: [2][16].
__device__ __forceinline__ bool quad_inv16(float2 (&v)[2], int u, float2 (*col)[PB_PAN]) {
  const int r = u & 15, h = (u >> 4) & 1, q = u >> 5;
  bool ok = true;
#pragma unroll
  for (int k = 0; k < PB_PAN; ++k) {
    const int kq = k >> 2, kh = (k >> 1) & 1, kr = k & 1;
    if (q == kq && h == kh) {
      col[k & 1][r] = v[kr];
      v[kr] = make_float2(r == k ? 1.f : 0.f, 0.f);    // the pivot column starts from the identity
    }
    float2 row[2];
#pragma unroll
    for (int c = 0; c < 2; ++c)
      row[c] = make_float2(__shfl_sync(0xffffffffu, v[c].x, k + 16 * h), __shfl_sync(0xffffffffu, v[c].y, k + 16 * h));
    named_sync(2, 128);
    const float2 piv = col[k & 1][k], ck = col[k & 1][r];
    const float n2 = piv.x * piv.x + piv.y * piv.y;
    ok = ok && n2 > 1e-30f && n2 < 1e30f;
    const float rn = rcp_newton(n2);
    const float2 inv = make_float2(piv.x * rn, -piv.y * rn);
    // a_rc - (a_rk / a_kk) row_c; row k itself: 0 + row_c / a_kk
    const bool isrow = r == k;
    const float2 m = isrow ? make_float2(-inv.x, -inv.y) : cmul(ck, inv);
#pragma unroll
    for (int c = 0; c < 2; ++c) {
      const float2 b = isrow ? make_float2(0.f, 0.f) : v[c];
      v[c].x = fmaf(m.y, row[c].y, fmaf(-m.x, row[c].x, b.x));
      v[c].y = fmaf(-m.y, row[c].x, fmaf(-m.x, row[c].y, b.y));
    }
  }
  return ok;
}

__global__ void __cluster_dims__(PB_CL, 1, 1) __launch_bounds__(PB_ALL, 1)
    k_block_inv_cluster(const float2* A, int64_t lda, int w, float2* X, int64_t ldx, int* status,
                        float2* __restrict__ Xr, float2* Pg) {
  namespace cg = cooperative_groups;
  cg::cluster_group cluster = cg::this_cluster();
  __shared__ __align__(16) float2 Ps[PB_PAN][PB_W];    // panel rows, panel columns = identity
  __shared__ __align__(16) float2 Cs[PB_PAN][PB_LD];   // own panel-column entries, [k][row]
  __shared__ __align__(16) float4 Ds[PB_PAN][PB_RPC];  // D = C X as (-re, -re, im, -im), [k][row]
  __shared__ float2 colb[2][PB_PAN];
  __shared__ __align__(16) float2 Xs[PB_PAN][PB_PAN];
  __shared__ __align__(16) float2 Nb[2][PB_PAN][PB_PAN + 1];   // next pivot block before this panel's update
  __shared__ float cond_red[PB_THREADS / 32], cond_loc[2];
  const int rank = (int)cluster.block_rank();
  const int t = threadIdx.x, tx = t & 63, ty = t >> 6, warp = t >> 5, lane = t & 31;
  const bool main = t < PB_THREADS;                    // the last four warps invert pivot blocks
  const int row0 = rank * PB_RPC + 4 * ty;             // first of this thread's rows
  const int pr = lane & 15, pc = 4 * ((t >> 5) & 3) + 2 * (lane >> 4);   // pivot warps: row and first column
  const int npan = (w + PB_PAN - 1) / PB_PAN;
  float2 a[4][4];
  float amax = 0.f;
  if (main) {
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const int gr = row0 + i, c = tx + 64 * j;
        a[i][j] = (gr < w && c < w) ? A[(int64_t)gr * lda + c] : make_float2(gr == c ? 1.f : 0.f, 0.f);
        if (gr < w && c < w) amax = fmaxf(amax, sqrtf(a[i][j].x * a[i][j].x + a[i][j].y * a[i][j].y));
      }
  }
  // CTA maximum of a per-thread value into cond_loc[slot]
  const auto cta_max = [&](float v, int slot) {
    for (int o = 16; o; o >>= 1) v = fmaxf(v, __shfl_xor_sync(0xffffffffu, v, o));
    if (main && lane == 0) cond_red[warp] = v;
    __syncthreads();
    if (t == 0) {
      float mx = 0.f;
      for (int k = 0; k < PB_THREADS / 32; ++k) mx = fmaxf(mx, cond_red[k]);
      cond_loc[slot] = mx;
    }
    __syncthreads();
  };
  cta_max(amax, 0);
  // panel pp (raw rows, pivot block inverted) into its scratch buffer, by the owner
  const auto put_panel = [&](int pp) {
    const int lp0 = pp * PB_PAN % PB_RPC;
    if (rank == pp * PB_PAN / PB_RPC && 4 * ty >= lp0 && 4 * ty < lp0 + PB_PAN) {
      float2* Pb = Pg + (pp & 1) * PB_BUF;
#pragma unroll
      for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) Pb[(4 * ty + i - lp0) * PB_W + tx + 64 * j] = a[i][j];
    }
  };
  const auto put_inverse = [&](int pp, float2 (&v)[2]) {
    const bool ok = quad_inv16(v, t - PB_THREADS, colb);
    if (!ok && lane == 0) atomicOr(status, 1);
    *reinterpret_cast<float4*>(Pg + (pp & 1) * PB_BUF + PB_PAN * PB_W + pr * PB_PAN + pc) =
        make_float4(v[0].x, v[0].y, v[1].x, v[1].y);
  };
  if (main) {
    put_panel(0);
  } else if (rank == 0) {
    float2 v[2];
#pragma unroll
    for (int c = 0; c < 2; ++c)
      v[c] = (pr < w && pc + c < w) ? A[(int64_t)pr * lda + pc + c] : make_float2(pr == pc + c ? 1.f : 0.f, 0.f);
    put_inverse(0, v);
  }
  for (int pp = 0; pp < npan; ++pp) {
    const int p0 = pp * PB_PAN, owner = p0 / PB_RPC, lp0 = p0 % PB_RPC;
    const int p1 = p0 + PB_PAN, lp1 = p1 % PB_RPC;             // the next panel
    const bool nown = pp + 1 < npan && rank == p1 / PB_RPC;
    const float2* Pb = Pg + (pp & 1) * PB_BUF;
    const int jp = p0 >> 6, cp = tx - (p0 & 63);       // this thread's panel column, if 0 <= cp < 16
    const bool inpan = cp >= 0 && cp < PB_PAN;
    const bool prow = rank == owner && 4 * ty >= lp0 && 4 * ty < lp0 + PB_PAN;
    if (main) {
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        if (inpan && j == jp) {
#pragma unroll
          for (int i = 0; i < 4; ++i) Cs[cp][4 * ty + i] = a[i][j];
        }
        const int cn = tx + 64 * j - p1;
        if (nown && 4 * ty >= lp1 && 4 * ty < lp1 + PB_PAN && cn >= 0 && cn < PB_PAN) {
#pragma unroll
          for (int i = 0; i < 4; ++i) Nb[pp & 1][4 * ty + i - lp1][cn] = a[i][j];
        }
      }
    }
    cluster.sync();
    if (warp < 4) {
      // D = C X: X through shared memory, warp = four pivots, lane = row
      const float4 q = __ldcg(reinterpret_cast<const float4*>(Pb + PB_PAN * PB_W) + t);
      reinterpret_cast<float4*>(&Xs[0][0])[t] = q;
      named_sync(1, 128);
      const int k0 = 4 * warp;
      float2 d[4];
#pragma unroll
      for (int q2 = 0; q2 < 4; ++q2) d[q2] = make_float2(0.f, 0.f);
      if (rank == owner && lane >= lp0 && lane < lp0 + PB_PAN) {
#pragma unroll
        for (int q2 = 0; q2 < 4; ++q2) d[q2] = make_float2(-Xs[lane - lp0][k0 + q2].x, -Xs[lane - lp0][k0 + q2].y);
      } else {
#pragma unroll
        for (int l = 0; l < PB_PAN; ++l) {
          const float2 cv = Cs[l][lane];
          const float4 x01 = *reinterpret_cast<const float4*>(&Xs[l][k0]);
          const float4 x23 = *reinterpret_cast<const float4*>(&Xs[l][k0 + 2]);
          cfma(d[0], cv, make_float2(x01.x, x01.y));
          cfma(d[1], cv, make_float2(x01.z, x01.w));
          cfma(d[2], cv, make_float2(x23.x, x23.y));
          cfma(d[3], cv, make_float2(x23.z, x23.w));
        }
      }
#pragma unroll
      for (int q2 = 0; q2 < 4; ++q2) Ds[k0 + q2][lane] = make_float4(-d[q2].x, -d[q2].x, d[q2].y, -d[q2].y);
    } else if (main) {
      constexpr int NL = PB_PAN * PB_W / 2, NT = PB_THREADS - 128, NQ = (NL + NT - 1) / NT;
      float4 q[NQ];
#pragma unroll
      for (int u = 0; u < NQ; ++u) {
        const int e = t - 128 + u * NT;
        if (e < NL) q[u] = __ldcg(reinterpret_cast<const float4*>(Pb) + e);
      }
#pragma unroll
      for (int u = 0; u < NQ; ++u) {
        const int e = t - 128 + u * NT, k = e / (PB_W / 2), c = 2 * (e % (PB_W / 2));
        if (c >= p0 && c < p1)
          q[u] = make_float4(c - p0 == k ? 1.f : 0.f, 0.f, c + 1 - p0 == k ? 1.f : 0.f, 0.f);
        if (e < NL) *reinterpret_cast<float4*>(&Ps[k][c]) = q[u];
      }
    }
    __syncthreads();
    if (main) {
      if (prow) {
#pragma unroll
        for (int i = 0; i < 4; ++i)
#pragma unroll
          for (int j = 0; j < 4; ++j) a[i][j] = make_float2(0.f, 0.f);
      }
      if (inpan) {
#pragma unroll
        for (int j = 0; j < 4; ++j)
          if (j == jp) {
#pragma unroll
            for (int i = 0; i < 4; ++i) a[i][j] = make_float2(0.f, 0.f);
          }
      }
#pragma unroll 4
      for (int k = 0; k < PB_PAN; ++k) {
        float4 d[4];
#pragma unroll
        for (int i = 0; i < 4; ++i) d[i] = Ds[k][4 * ty + i];
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          const float2 rv = Ps[k][tx + 64 * j], rs = make_float2(rv.y, rv.x);
#pragma unroll
          for (int i = 0; i < 4; ++i) {
            fma2(a[i][j], make_float2(d[i].x, d[i].y), rv);
            fma2(a[i][j], make_float2(d[i].z, d[i].w), rs);
          }
        }
      }
      if (nown) put_panel(pp + 1);
    } else if (nown) {
      float2 v[2] = {Nb[pp & 1][pr][pc], Nb[pp & 1][pr][pc + 1]};
#pragma unroll 4
      for (int k = 0; k < PB_PAN; ++k) {
        const float4 d = Ds[k][lp1 + pr];
        const float4 q = *reinterpret_cast<const float4*>(&Ps[k][p1 + pc]);
        const float2 d0 = make_float2(d.x, d.y), d1 = make_float2(d.z, d.w);
        fma2(v[0], d0, make_float2(q.x, q.y));
        fma2(v[0], d1, make_float2(q.y, q.x));
        fma2(v[1], d0, make_float2(q.z, q.w));
        fma2(v[1], d1, make_float2(q.w, q.z));
      }
      put_inverse(pp + 1, v);
    }
  }
  float xmax = 0.f;
  if (main) {
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
      for (int j = 0; j < 4; ++j)
        if (row0 + i < w && tx + 64 * j < w)
          xmax = fmaxf(xmax, sqrtf(a[i][j].x * a[i][j].x + a[i][j].y * a[i][j].y));
  }
  cta_max(xmax, 1);
  cluster.sync();
  if (rank == 0 && t == 0) {
    float am = 0.f, xm = 0.f;
    for (int r = 0; r < PB_CL; ++r) {
      const float* cl = cluster.map_shared_rank(cond_loc, r);
      am = fmaxf(am, cl[0]);
      xm = fmaxf(xm, cl[1]);
    }
    record_cond(status, am, xm);
  }
  if (main) {
  // X may be the input block itself: every CTA read its rows at the start
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const int gr = row0 + i;
    if (gr >= w) continue;
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const int c = tx + 64 * j;
      if (c < w) {
        X[(int64_t)gr * ldx + c] = a[i][j];
        if (Xr) {   // copy rounded to TF32 (nearest): the A operand of tensor-core products
          uint32_t x, y;
          asm("cvt.rna.tf32.f32 %0, %1;" : "=r"(x) : "f"(a[i][j].x));
          asm("cvt.rna.tf32.f32 %0, %1;" : "=r"(y) : "f"(a[i][j].y));
          Xr[(int64_t)gr * w + c] = make_float2(__uint_as_float(x), __uint_as_float(y));
        }
      }
    }
  }
  }
  cluster.sync();   // no CTA may exit while another can still read its shared memory
}

static mnpbem_status launch_block_inv_cluster(const float2* A, int64_t lda, int w, float2* X, int64_t ldx,
                                              int* status, DevBuf& pan, cudaStream_t st, float2* Xr = nullptr) {
  MNP_TRY(pan.ensure(PB_SCRATCH));
  ProfScope ps(PH_BLOCKINV, st, 8.0 * w * w * w, 0.0);
  k_block_inv_cluster<<<PB_CL, PB_ALL, 0, st>>>(A, lda, w, X, ldx, status, Xr, pan.as<float2>());
  MNP_CHECK_LAUNCH();
  return MNPBEM_OK;
}

// ------------------------------------------------ TF32 rounding in place
// The tensor cores read an FP32 operand as TF32 by dropping its 13 low
// mantissa bits (truncation, biased towards zero); operands rounded to nearest
// beforehand (cvt.rna.tf32) carry half the error and no bias.  The B operand
// is rounded when it is expanded; this rounds an A operand.
__global__ void k_round_tf32(float* x, int64_t count) {
  const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= count) return;
  uint32_t r;
  asm("cvt.rna.tf32.f32 %0, %1;" : "=r"(r) : "f"(x[i]));
  x[i] = __uint_as_float(r);
}

void round_tf32(float* x, int64_t count, cudaStream_t st) {
  if (count <= 0) return;
  ProfScope ps(PH_ELEMWISE, st, 0.0, 8.0 * count, 1);
  k_round_tf32<<<(unsigned)cdiv_up(count, 256), 256, 0, st>>>(x, count);
}

__device__ __forceinline__ float rna_tf32(float x) {
  uint32_t r;
  asm("cvt.rna.tf32.f32 %0, %1;" : "=r"(r) : "f"(x));
  return __uint_as_float(r);
}
// dst[rows][cols] (row stride ldd) <- src[rows][cols] (row stride lds),
// rounded to TF32 (nearest) when rna: the A operand of a tensor-core product;
// rows z0 .. z1 - 1 become zero
template <typename R>
__global__ void k_copy_panel(const cplx<R>* __restrict__ src, int64_t lds, int64_t rows, int cols,
                             cplx<R>* __restrict__ dst, int64_t ldd, int rna, int64_t z0, int64_t z1) {
  const int64_t idx = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (idx >= rows * cols) return;
  const int64_t i = idx / cols;
  const int c = (int)(idx - i * cols);
  cplx<R> v = (i >= z0 && i < z1) ? mk<R>(0, 0) : src[i * lds + c];
  if constexpr (sizeof(R) == 4)
    if (rna) v = mk<R>(rna_tf32(v.x), rna_tf32(v.y));
  dst[i * ldd + c] = v;
}
// The same for complex64 in 16-byte pieces (even strides and columns, aligned
// bases): four loads in flight per thread.  Bound by HBM at 24 000 rows and by its
// share of the SMs beside other wavelengths' kernels at 4000: the panels of a
// 24 000-face solve 12.8 ms in single entries, 11.7 now; sweep of 4000 faces, eight
// wavelengths in flight, 121 and 117 ms.
__global__ void __launch_bounds__(256) k_copy_panel4(const float2* __restrict__ src, int64_t lds, unsigned total,
                                                   unsigned cols2, float2* __restrict__ dst, int64_t ldd, int rna,
                                                   int64_t z0, int64_t z1) {
  float4 v[4];
  unsigned row[4], col[4];
#pragma unroll
  for (int u = 0; u < 4; ++u) {
    const unsigned idx = blockIdx.x * 1024u + 256u * u + threadIdx.x;
    row[u] = idx / cols2;
    col[u] = 2 * (idx - row[u] * cols2);
    v[u] = make_float4(0.f, 0.f, 0.f, 0.f);
    if (idx < total && (row[u] < z0 || row[u] >= z1))
      v[u] = *reinterpret_cast<const float4*>(src + (int64_t)row[u] * lds + col[u]);
  }
#pragma unroll
  for (int u = 0; u < 4; ++u) {
    if (blockIdx.x * 1024u + 256u * u + threadIdx.x >= total) break;
    if (rna) v[u] = make_float4(rna_tf32(v[u].x), rna_tf32(v[u].y), rna_tf32(v[u].z), rna_tf32(v[u].w));
    *reinterpret_cast<float4*>(dst + (int64_t)row[u] * ldd + col[u]) = v[u];
  }
}

template <typename R>
static void copy_panel(const cplx<R>* src, int64_t lds, int64_t rows, int cols, cplx<R>* dst, int64_t ldd, bool rna,
                       cudaStream_t st, int64_t z0 = 0, int64_t z1 = 0) {
  if (rows <= 0 || cols <= 0) return;
  ProfScope ps(PH_ELEMWISE, st, 0.0, 2.0 * sizeof(cplx<R>) * rows * cols, 1);
  const int64_t cnt = rows * cols;
  if constexpr (sizeof(R) == 4) {
    const uintptr_t al = reinterpret_cast<uintptr_t>(src) | reinterpret_cast<uintptr_t>(dst);
    if (!((lds | ldd | cols) & 1) && !(al & 15) && cnt < (1ll << 32)) {
      k_copy_panel4<<<(unsigned)cdiv_up(cnt / 2, (int64_t)1024), 256, 0, st>>>(
          src, lds, (unsigned)(cnt / 2), (unsigned)(cols / 2), dst, ldd, rna ? 1 : 0, z0, z1);
      return;
    }
  }
  k_copy_panel<R><<<(unsigned)cdiv_up(cnt, (int64_t)256), 256, 0, st>>>(src, lds, rows, cols, dst, ldd, rna ? 1 : 0, z0,
                                                                        z1);
}

// --------------------------------------------------- blocked Gauss-Jordan
template <typename R>
mnpbem_status gj_status_copy(GJWork<R>& w, int* host2, cudaStream_t st) {
  host2[0] = host2[1] = 0;
  if (w.status.ptr) MNP_CUDA(cudaMemcpyAsync(host2, w.status.ptr, sizeof(int), cudaMemcpyDeviceToHost, st));
  if (w.inner && w.inner->status.ptr)
    MNP_CUDA(cudaMemcpyAsync(host2 + 1, w.inner->status.ptr, sizeof(int), cudaMemcpyDeviceToHost, st));
  return MNPBEM_OK;
}
template mnpbem_status gj_status_copy<float>(GJWork<float>&, int*, cudaStream_t);
template mnpbem_status gj_status_copy<double>(GJWork<double>&, int*, cudaStream_t);

template <typename R>
mnpbem_status gj_invert(cplx<R>* A, int64_t n, int64_t lda, GJWork<R>& w, GemmFn<R> big_gemm,
                        void* ctx, cudaStream_t st, bool read_status) {
  using Cx = cplx<R>;
  const int nb = w.nb;
  const size_t cs = sizeof(Cx);
  MNP_TRY(w.ccol.ensure(cs * n * nb));
  MNP_TRY(w.rrow.ensure(cs * n * nb));
  MNP_TRY(w.ncol.ensure(cs * n * nb));
  MNP_TRY(w.xblk.ensure(cs * nb * nb));
  MNP_TRY(w.status.ensure(2 * sizeof(int)));
  if (!w.nested) MNP_CUDA(cudaMemsetAsync(w.status.ptr, 0, 2 * sizeof(int), st));
  if (!w.nested && nb > 64 && (sizeof(R) == 8 || nb > PB_W)) {
    // pivot blocks wider than 64 are inverted by an inner Gauss-Jordan whose
    // pivot status this (outer) level clears now and reads at the end
    if (!w.inner) w.inner.reset(new GJWork<R>());
    // complex64 with pivot blocks wider than 256: 256-wide inner steps whose
    // own pivot blocks go to the cluster kernel; otherwise 64-wide steps
    w.inner->nb = (sizeof(R) == 4 && nb > PB_W) ? PB_W : 64;
    w.inner->nested = true;
    MNP_TRY(w.inner->status.ensure(2 * sizeof(int)));
    MNP_CUDA(cudaMemsetAsync(w.inner->status.ptr, 0, 2 * sizeof(int), st));
  }
  Cx* Ccol = w.ccol.template as<Cx>();   // [n][nb]
  Cx* Rrow = w.rrow.template as<Cx>();   // [nb][n]
  Cx* Ncol = w.ncol.template as<Cx>();   // [n][nb]
  Cx* X = w.xblk.template as<Cx>();      // [nb][nb]
  const Cx one = mk<R>(1, 0), zero = mk<R>(0, 0), mone = mk<R>(-1, 0);
  for (int64_t k0 = 0; k0 < n; k0 += nb) {
    const int bw = (int)std::min<int64_t>(nb, n - k0);
    if constexpr (sizeof(R) == 4) {
      // Fused step on the tensor-core path (all three products eligible):
      //   X <- inv(A_kk) read in place; Ccol <- TF32(A[:, k]) with rows k zeroed;
      //   A[k, :] <- X A[k, :] in place (the product copies its B operand before it
      //   runs); A[:, k] <- -Ccol X (rows k become 0); A <- A - Ccol A[k, :] with the
      //   k columns of the B operand read as zero (rows and columns k unchanged);
      //   A_kk <- X.  The same products as the general step below, without its
      //   panel copies and write-backs.
      TcGemmCtx* tc = reinterpret_cast<TcGemmCtx*>(ctx);
      const float2 b0 = make_float2(0.f, 0.f), b1 = make_float2(1.f, 0.f);
      float2* Af = reinterpret_cast<float2*>(A);
      float2* Cf = reinterpret_cast<float2*>(Ccol);
      float2* Xf = reinterpret_cast<float2*>(X);
      if (tc && w.fused && (bw <= PB_W || w.inner) && tc_gemm_eligible(*tc, bw, n, bw, Xf, bw, Af + k0 * lda, lda, b0) &&
          tc_gemm_eligible(*tc, n, bw, bw, Cf, bw, Af + k0, lda, b0) &&
          tc_gemm_eligible(*tc, n, n, bw, Cf, bw, Af, lda, b1)) {
        if (bw <= 64) {
          MNP_TRY(launch_block_inv(Af + k0 * lda + k0, lda, bw, Xf, bw, nullptr, 0, w.status.template as<int>(), st));
        } else if (bw <= PB_W) {
          MNP_TRY(launch_block_inv_cluster(Af + k0 * lda + k0, lda, bw, Xf, bw, w.status.template as<int>(), w.pan, st));
        } else {
          // wider pivot blocks: inner Gauss-Jordan (256-wide steps) on a copy
          MNP_CUDA(cudaMemcpy2DAsync(X, cs * bw, A + k0 * lda + k0, cs * lda, cs * bw, bw, cudaMemcpyDeviceToDevice,
                                     st));
          MNP_TRY(gj_invert<R>(X, bw, bw, *w.inner, big_gemm, ctx, st));
        }
        // the column panel without the pivot rows: the A operand of the column-panel
        // product and of the rank update
        copy_panel<float>(Af + k0, lda, n, bw, Cf, bw, w.round_a, st, k0, k0 + bw);
        MNP_CHECK_LAUNCH();
        MNP_TRY(tc_gemm_c64(*tc, bw, n, bw, b1, Xf, bw, Af + k0 * lda, lda, b0, Af + k0 * lda, lda, st));
        MNP_TRY(tc_gemm_c64(*tc, n, bw, bw, make_float2(-1.f, 0.f), Cf, bw, Xf, bw, b0, Af + k0, lda, st));
        MNP_TRY(tc_gemm_c64(*tc, n, n, bw, make_float2(-1.f, 0.f), Cf, bw, Af + k0 * lda, lda, b1, Af, lda, st,
                            k0, k0 + bw));
        MNP_CUDA(cudaMemcpy2DAsync(A + k0 * lda + k0, cs * lda, X, cs * bw, cs * bw, bw, cudaMemcpyDeviceToDevice, st));
        continue;
      }
    }
    // 1. Ccol <- A[:, k-block]
    MNP_CUDA(cudaMemcpy2DAsync(Ccol, cs * bw, A + k0, cs * lda, cs * bw, n, cudaMemcpyDeviceToDevice, st));
    // 2. X <- inv(A_kk): one shared-memory kernel for blocks up to 64, else
    //    an inner Gauss-Jordan with 64-wide steps on a copy of the block
    if (bw <= 64) {
      MNP_TRY(launch_block_inv(Ccol + k0 * bw, bw, bw, X, bw, nullptr, 0, w.status.template as<int>(), st));
    } else if (sizeof(R) == 4 && bw <= PB_W) {
      MNP_TRY(launch_block_inv_cluster(reinterpret_cast<const float2*>(Ccol + k0 * bw), bw, bw,
                                       reinterpret_cast<float2*>(X), bw, w.status.template as<int>(), w.pan, st));
    } else {
      MNP_CUDA(cudaMemcpyAsync(X, Ccol + k0 * bw, cs * bw * bw, cudaMemcpyDeviceToDevice, st));
      MNP_TRY(gj_invert<R>(X, bw, bw, *w.inner, big_gemm, ctx, st));
    }
    // 3. R <- X * A[k-block, :], then zero its k-block columns
    MNP_TRY(big_gemm(bw, n, bw, one, X, bw, A + k0 * lda, lda, zero, Rrow, n, st, ctx));
    MNP_CUDA(cudaMemset2DAsync(Rrow + k0, cs * n, 0, cs * bw, bw, st));
    // 4. new column block <- -Ccol * X, then zero Ccol's k-block rows
    //    (on the tensor-core path Ccol, the A operand of this product and of
    //    the rank update, is first rounded to TF32; the pivot block it holds
    //    has already been inverted in full FP32)
    if (sizeof(R) == 4 && ctx && w.round_a) round_tf32(reinterpret_cast<float*>(Ccol), 2 * n * bw, st);
    MNP_TRY(big_gemm(n, bw, bw, mone, Ccol, bw, X, bw, zero, Ncol, bw, st, ctx));
    MNP_CUDA(cudaMemsetAsync(Ccol + k0 * bw, 0, cs * bw * bw, st));
    // 5. A <- A - Ccol * R  (rank-bw update of the whole matrix)
    MNP_TRY(big_gemm(n, n, bw, mone, Ccol, bw, Rrow, n, one, A, lda, st, ctx));
    // 6. write back row block, column block and the inverted pivot block
    MNP_CUDA(cudaMemcpy2DAsync(A + k0 * lda, cs * lda, Rrow, cs * n, cs * n, bw, cudaMemcpyDeviceToDevice, st));
    MNP_CUDA(cudaMemcpy2DAsync(A + k0, cs * lda, Ncol, cs * bw, cs * bw, n, cudaMemcpyDeviceToDevice, st));
    MNP_CUDA(cudaMemcpy2DAsync(A + k0 * lda + k0, cs * lda, X, cs * bw, cs * bw, bw, cudaMemcpyDeviceToDevice, st));
  }
  if (w.nested || !read_status) return MNPBEM_OK;
  int hs = 0;
  MNP_CUDA(cudaMemcpyAsync(&hs, w.status.ptr, sizeof(int), cudaMemcpyDeviceToHost, st));
  MNP_CUDA(cudaStreamSynchronize(st));
  if (w.inner) {
    int hi = 0;
    MNP_CUDA(cudaMemcpyAsync(&hi, w.inner->status.ptr, sizeof(int), cudaMemcpyDeviceToHost, st));
    MNP_CUDA(cudaStreamSynchronize(st));
    hs |= hi;
  }
  if (hs) {
    set_error("block Gauss-Jordan inversion: zero or non-finite pivot");
    return MNPBEM_ERR_SINGULAR;
  }
  return MNPBEM_OK;
}

template mnpbem_status gj_invert<float>(float2*, int64_t, int64_t, GJWork<float>&, GemmFn<float>,
                                        void*, cudaStream_t, bool);
template mnpbem_status gj_invert<double>(double2*, int64_t, int64_t, GJWork<double>&,
                                         GemmFn<double>, void*, cudaStream_t, bool);

// ------------------------------------------------------ block LDU factors
// A_kk <- inv(A_kk) in place, with a copy in X (ld bw): 64-wide blocks with
// partial pivoting, 256-wide complex64 blocks on a CTA cluster, whose copy in X
// is rounded to TF32 (nearest) for the tensor-core products (the tensor cores
// would otherwise truncate it)
template <typename R>
mnpbem_status block_inverse(cplx<R>* Akk, int64_t lda, int bw, cplx<R>* X, int* status, DevBuf& pan,
                            cudaStream_t st) {
  if (bw <= 64) return launch_block_inv(Akk, lda, bw, X, bw, Akk, lda, status, st);
  if (sizeof(R) == 4 && bw <= PB_W)
    return launch_block_inv_cluster(reinterpret_cast<const float2*>(Akk), lda, bw, reinterpret_cast<float2*>(Akk), lda,
                                    status, pan, st, reinterpret_cast<float2*>(X));
  set_error("block LDU: diagonal blocks of %d rows are not supported in this precision", bw);
  return MNPBEM_ERR_UNSUPPORTED;
}

template mnpbem_status block_inverse<float>(float2*, int64_t, int, float2*, int*, DevBuf&, cudaStream_t);
template mnpbem_status block_inverse<double>(double2*, int64_t, int, double2*, int*, DevBuf&, cudaStream_t);

template <typename R>
mnpbem_status ldu_factor(cplx<R>* A, int64_t n, int64_t lda, LDUWork<R>& w, int* status, GemmFn<R> gemm,
                         void* ctx, cudaStream_t st) {
  using Cx = cplx<R>;
  const int b = w.b, B = w.b * std::max(1, w.m);
  if (n <= 0) return MNPBEM_OK;
  const size_t cs = sizeof(Cx);
  MNP_TRY(w.ccol.ensure(cs * n * B));
  MNP_TRY(w.xblk.ensure(cs * b * b));
  const bool tc = sizeof(R) == 4 && ctx != nullptr;
  MNP_TRY(w.rrow.ensure(cs * n * b));
  const bool rna = tc && w.round_a;
  Cx* Cc = w.ccol.template as<Cx>();     // [n][B]: row i holds row k0 + i of the outer step's column panel
  Cx* X = w.xblk.template as<Cx>();
  const Cx one = mk<R>(1, 0), zero = mk<R>(0, 0), mone = mk<R>(-1, 0);
  for (int64_t k0 = 0; k0 < n; k0 += B) {
    const int64_t Bw = std::min<int64_t>(B, n - k0), e = k0 + Bw;
    for (int64_t s = 0; s < Bw; s += b) {
      const int64_t ks = k0 + s;
      const int bs = (int)std::min<int64_t>(b, e - ks);
      const int64_t kb = ks + bs, below = n - kb;
      MNP_TRY(block_inverse<R>(A + ks * lda + ks, lda, bs, X, status, w.pan, st));
      if (below > 0) {
        Cx* Cs = Cc + (kb - k0) * B + s;
        // unscaled column panel (the A operand of every update of this step)
        copy_panel<R>(A + kb * lda + ks, lda, below, bs, Cs, B, rna, st);
        MNP_CHECK_LAUNCH();
        // L panel: A[kb:, ks:kb] = C X
        MNP_TRY(gemm(below, bs, bs, one, Cs, B, X, bs, zero, A + kb * lda + ks, lda, st, ctx));
        // U row: A[ks:kb, kb:] = X A[ks:kb, kb:] (the tensor-core products copy their
        // B operand before they run, so they may write in place; the CUDA-core
        // products may not)
        bool inplace = false;
        if (ctx) {
          TcGemmCtx& tcc = *reinterpret_cast<TcGemmCtx*>(ctx);
          if constexpr (sizeof(R) == 4)
            inplace = tc_gemm_eligible(tcc, bs, below, bs, X, bs, A + ks * lda + kb, lda, make_float2(0.f, 0.f));
          else
            inplace = tc_gemm64_eligible(tcc, bs, below, bs, one, zero);
        }
        if (inplace) {
          MNP_TRY(gemm(bs, below, bs, one, X, bs, A + ks * lda + kb, lda, zero, A + ks * lda + kb, lda, st, ctx));
        } else {
          Cx* Rr = w.rrow.template as<Cx>();
          MNP_CUDA(cudaMemcpy2DAsync(Rr, cs * below, A + ks * lda + kb, cs * lda, cs * below, bs,
                                     cudaMemcpyDeviceToDevice, st));
          MNP_TRY(gemm(bs, below, bs, one, X, bs, Rr, below, zero, A + ks * lda + kb, lda, st, ctx));
        }
        if (kb < e) {
          // the later column panels of this outer step (all rows below) ...
          MNP_TRY(gemm(below, e - kb, bs, mone, Cs, B, A + ks * lda + kb, lda, one, A + kb * lda + kb, lda, st, ctx));
          // ... and the later rows of this outer step over the trailing columns
          if (e < n)
            MNP_TRY(gemm(e - kb, n - e, bs, mone, Cs, B, A + ks * lda + e, lda, one, A + kb * lda + e, lda, st, ctx));
        }
      }
    }
    // trailing update of rank Bw
    if (e < n) MNP_TRY(gemm(n - e, n - e, Bw, mone, Cc + (e - k0) * B, B, A + k0 * lda + e, lda, one, A + e * lda + e,
                            lda, st, ctx));
  }
  return MNPBEM_OK;
}

template <typename R>
mnpbem_status ldu_rsolve(cplx<R>* H, int64_t n, int64_t ldh, const cplx<R>* F, int64_t ldf, LDUWork<R>& w,
                         GemmFn<R> gemm, void* ctx, cudaStream_t st) {
  using Cx = cplx<R>;
  const int b = w.b, B = w.b * std::max(1, w.m);
  if (n <= 0) return MNPBEM_OK;
  MNP_TRY(w.ccol.ensure(sizeof(Cx) * n * B));
  const bool rna = sizeof(R) == 4 && ctx != nullptr && w.round_a;
  Cx* Cc = w.ccol.template as<Cx>();     // [n][B]: columns of the outer step
  const Cx one = mk<R>(1, 0), zero = mk<R>(0, 0), mone = mk<R>(-1, 0);
  // 1. W U = H (U unit upper), columns in increasing order; then V = W D^-1
  //    (D^-1 = the stored X_k) on each outer step's columns once they are final
  for (int64_t k0 = 0; k0 < n; k0 += B) {
    const int64_t Bw = std::min<int64_t>(B, n - k0), e = k0 + Bw;
    for (int64_t s = 0; s < Bw; s += b) {
      const int64_t ks = k0 + s;
      const int bs = (int)std::min<int64_t>(b, e - ks);
      copy_panel<R>(H + ks, ldh, n, bs, Cc + s, B, rna, st);
      MNP_CHECK_LAUNCH();
      if (ks + bs < e)
        MNP_TRY(gemm(n, e - ks - bs, bs, mone, Cc + s, B, F + ks * ldf + ks + bs, ldf, one, H + ks + bs, ldh, st, ctx));
    }
    if (e < n) MNP_TRY(gemm(n, n - e, Bw, mone, Cc, B, F + k0 * ldf + e, ldf, one, H + e, ldh, st, ctx));
    for (int64_t s = 0; s < Bw; s += b) {
      const int64_t ks = k0 + s;
      const int bs = (int)std::min<int64_t>(b, e - ks);
      MNP_TRY(gemm(n, bs, bs, one, Cc + s, B, F + ks * ldf + ks, ldf, zero, H + ks, ldh, st, ctx));
    }
  }
  // 2. S L = V (L unit lower), columns in decreasing order
  const int64_t nout = cdiv_up(n, (int64_t)B);
  for (int64_t q = nout - 1; q >= 0; --q) {
    const int64_t k0 = q * B, Bw = std::min<int64_t>(B, n - k0), e = k0 + Bw;
    const int64_t nin = cdiv_up(Bw, (int64_t)b);
    for (int64_t t = nin - 1; t >= 0; --t) {
      const int64_t ks = k0 + t * b;
      const int bs = (int)std::min<int64_t>(b, e - ks);
      copy_panel<R>(H + ks, ldh, n, bs, Cc + t * b, B, rna, st);
      MNP_CHECK_LAUNCH();
      if (ks > k0) MNP_TRY(gemm(n, ks - k0, bs, mone, Cc + t * b, B, F + ks * ldf + k0, ldf, one, H + k0, ldh, st, ctx));
    }
    if (k0 > 0) MNP_TRY(gemm(n, k0, Bw, mone, Cc, B, F + k0 * ldf, ldf, one, H, ldh, st, ctx));
  }
  return MNPBEM_OK;
}

// ------------------------------------------------- triangular sweeps
// The solves L y = x and U x = D^-1 y of the LDU factors for a few right-hand
// sides, each sweep one launch over up to SWEEP_MAXPROB systems of one block
// size (the diagonal blocks of G1 and G2 are solved together).  A work item is
// a slice of RS = 8 RW rows of one block row; the CTAs take the items in the
// order of their block rows from a counter, keep the slice's sums in registers
// while they walk the block row, and wait for block k only when they need its
// solution.  An item waits for items with smaller numbers alone, and these have
// been taken by CTAs that run: no co-residency is needed, so the sweep neither
// waits for a whole free GPU nor keeps other streams' kernels out while it
// waits.  Forward: y_i = x_i - sum_{k<i} L_ik y_k into T.  Backward:
// x_i = X_i y_i - sum_{k>i} U_ik x_k (X_i the stored inverse of D_i) into X.
// Blocks complete in order, so one counter of finished slices per system says
// how many are ready.  A thread's entries of the next block are loaded as those
// of this one are used; they do not depend on the wait.
// The waits are bounded by wall clock: on expiry an error word is set, an abort
// word releases the other CTAs, and all return.
// Bound by the chain of block rows (about 3 us each) at a few thousand rows and by
// HBM at 24 000 (800 us for 2.3 GB).  Against the cooperative sweep before it (a
// grid barrier per block row), with eight wavelengths of 4000 faces in flight:
// 72 us against 131 to 150 us per sweep, 12 sweeps instead of 18 per direction and
// wavelength, and no separate product with D^-1 (90 us on one CTA per block).
constexpr int SWEEP_THREADS = 256;

template <typename R> struct SweepArgs {
  LduProblem<R> p[SWEEP_MAXPROB];
  int nprob, b, N, items;
  unsigned* ctl;            // [0], [1] item counters, [2] abort, [4 + 2 q + direction] finished slices
};

template <typename R, int NB, int RW, int CPL, bool LOWER>
__global__ void __launch_bounds__(SWEEP_THREADS, 2) k_ldu_sweep(const __grid_constant__ SweepArgs<R> a) {
  using Cx = cplx<R>;
  constexpr int RS = 8 * RW;
  extern __shared__ __align__(16) unsigned char sweep_smem[];
  Cx* xs = reinterpret_cast<Cx*>(sweep_smem);        // [2][NB][b + 4]
  __shared__ int item_s, known_s;
  const int b = a.b, N = a.N, xld = b + 4;
  const int S = (b + RS - 1) / RS;
  const int t = threadIdx.x, lane = t & 31, warp = t >> 5;
  volatile unsigned* abortw = a.ctl + 2;
  for (;;) {
    __syncthreads();
    if (t == 0) item_s = (int)atomicAdd(a.ctl + (LOWER ? 0 : 1), 1u);
    __syncthreads();
    const int item = item_s;
    if (item >= a.items) return;
    const int q = item % a.nprob, lv = item / a.nprob, i = lv / S, s = lv - i * S;
    const LduProblem<R>& p = a.p[q];
    const int nblk = (int)((p.n + b - 1) / b);
    if (i >= nblk) continue;
    const int blk = LOWER ? i : nblk - 1 - i;
    unsigned* arrived = a.ctl + 4 + 2 * q + (LOWER ? 0 : 1);
    const int64_t row0 = (int64_t)blk * b + s * RS + warp * RW;
    const int64_t rend = min(p.n, (int64_t)(blk + 1) * b);
    const Cx* frow[RW];
    bool act[RW];
#pragma unroll
    for (int r = 0; r < RW; ++r) {
      act[r] = row0 + r < rend;
      frow[r] = p.F + (act[r] ? row0 + r : (int64_t)blk * b) * p.ldf;
    }
    Cx acc[RW][NB], f[RW][CPL];
#pragma unroll
    for (int r = 0; r < RW; ++r)
#pragma unroll
      for (int c = 0; c < NB; ++c) acc[r][c] = mk<R>(0, 0);
    // step c of the walk: forward block c; backward the diagonal block, then nblk - c
    const int nstep = LOWER ? i : i + 1;
    const auto col_block = [&](int c) { return LOWER ? c : (c == 0 ? blk : nblk - c); };
    const auto load_f = [&](int c, int r, int u) {
      const int k = col_block(c), l = lane + 32 * u;
      const int64_t k0 = (int64_t)k * b;
      if (k0 + l < p.n && l < b) f[r][u] = __ldg(frow[r] + k0 + l);
      else f[r][u] = mk<R>(0, 0);
    };
    if (nstep > 0) {
#pragma unroll
      for (int r = 0; r < RW; ++r)
#pragma unroll
        for (int u = 0; u < CPL; ++u) load_f(0, r, u);
    }
    int known = 0;                                     // slices known to have finished
    for (int c = 0; c < nstep; ++c) {
      const int need = LOWER ? (c + 1) * S : c * S;
      if (need > known) {
        if (t == 0) {
          unsigned v;
          const unsigned long long t0 = gtimer();
          for (;;) {
            asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(arrived) : "memory");
            if (v >= (unsigned)need) break;
            if (*abortw) { v = 0; break; }
            if (gtimer() - t0 > MBAR_WAIT_NS) {
              atomicOr(&g_sweep_err, 64);
              *abortw = 1u;
              v = 0;
              break;
            }
          }
          known_s = (int)v;
        }
        __syncthreads();
        known = known_s;
        if (known < need) return;
      }
      const int64_t k0 = (int64_t)col_block(c) * b;
      const int bs = (int)min((int64_t)b, p.n - k0);
      const bool from_t = LOWER || c == 0;
      const Cx* src = from_t ? p.T + k0 * N : p.X + k0 * p.ldx;
      const int64_t lds = from_t ? N : p.ldx;
      Cx* xb = xs + (c & 1) * NB * xld;
      for (int e = t; e < b * NB; e += SWEEP_THREADS) {
        const int r = e / NB, cc = e % NB;
        xb[cc * xld + r] = (r < bs && cc < N) ? __ldcg(src + r * lds + cc) : mk<R>(0, 0);
      }
      __syncthreads();
      const bool more = c + 1 < nstep;
#pragma unroll
      for (int u = 0; u < CPL; ++u) {
        const int l = min(lane + 32 * u, b - 1);       // beyond b: f is zero
        Cx xv[NB];
#pragma unroll
        for (int cc = 0; cc < NB; ++cc) xv[cc] = xb[cc * xld + l];
#pragma unroll
        for (int r = 0; r < RW; ++r) {
#pragma unroll
          for (int cc = 0; cc < NB; ++cc) cfma(acc[r][cc], f[r][u], xv[cc]);
          if (more) load_f(c + 1, r, u);
        }
      }
      if (!LOWER && c == 0) {
#pragma unroll
        for (int r = 0; r < RW; ++r)
#pragma unroll
          for (int cc = 0; cc < NB; ++cc) acc[r][cc] = mk<R>(-acc[r][cc].x, -acc[r][cc].y);
      }
    }
#pragma unroll
    for (int r = 0; r < RW; ++r)
#pragma unroll
      for (int cc = 0; cc < NB; ++cc) {
        Cx v = acc[r][cc];
#pragma unroll
        for (int o = 16; o; o >>= 1) {
          v.x += __shfl_xor_sync(0xffffffffu, v.x, o);
          v.y += __shfl_xor_sync(0xffffffffu, v.y, o);
        }
        if (act[r] && lane == cc && cc < N) {
          Cx* xp = p.X + (row0 + r) * p.ldx + cc;
          if (LOWER) p.T[(row0 + r) * N + cc] = csub(*xp, v);
          else *xp = mk<R>(-v.x, -v.y);
        }
      }
    __syncthreads();
    if (t == 0) {
      __threadfence();
      atomicAdd(arrived, 1u);
    }
  }
}

template <typename R, int NB, int RW, bool LOWER>
static mnpbem_status launch_sweep(SweepArgs<R> a, int maxblk, cudaStream_t st) {
  constexpr int CPL = sizeof(R) == 4 ? 8 : 2;          // entries per lane and block row: b <= 32 CPL
  auto kern = k_ldu_sweep<R, NB, RW, CPL, LOWER>;
  const int smem = (int)sizeof(cplx<R>) * 2 * NB * (a.b + 4);
  constexpr int SMEM_MAX = (int)sizeof(cplx<R>) * 2 * NB * (32 * CPL + 4);
  // CTAs per SM, kept per device together with the kernel's shared-memory attribute
  static std::atomic<int> kept[MAX_DEVICES];
  const int d = device_index();
  int per_sm = d < MAX_DEVICES ? kept[d].load() : 0;
  if (!per_sm) {
    MNP_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, SMEM_MAX));
    MNP_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kern, SWEEP_THREADS, SMEM_MAX));
    per_sm = std::max(1, per_sm);
    if (d < MAX_DEVICES) kept[d] = per_sm;
  }
  const int S = (a.b + 8 * RW - 1) / (8 * RW);
  a.items = maxblk * S * a.nprob;
  double half = 0.0;
  for (int q = 0; q < a.nprob; ++q) half += 0.5 * (double)a.p[q].n * a.p[q].n;
  ProfScope ps(PH_GEMM_SMALL, st, 8.0 * half * a.N, (double)sizeof(cplx<R>) * half);
  kern<<<(unsigned)std::min(a.items, per_sm * num_sms()), SWEEP_THREADS, smem, st>>>(a);
  MNP_CHECK_LAUNCH();
  return MNPBEM_OK;
}

template <typename R>
mnpbem_status ldu_solve_few(const LduProblem<R>* probs, int nprob, int b, int64_t N, const LduSweepWs& ws,
                            cudaStream_t st) {
  if (nprob < 1 || nprob > SWEEP_MAXPROB || N < 1 || N > 16 || b < 1 || b > (sizeof(R) == 4 ? 256 : 64) || !ws.ctl) {
    set_error("ldu_solve_few: invalid arguments");
    return MNPBEM_ERR_INVALID_ARG;
  }
  SweepArgs<R> a;
  a.nprob = 0;
  a.b = b;
  a.N = (int)N;
  a.ctl = ws.ctl;
  int64_t rows = 0, maxn = 0;
  for (int q = 0; q < nprob; ++q) {
    if (probs[q].n <= 0) continue;
    a.p[a.nprob] = probs[q];
    a.p[a.nprob].T = reinterpret_cast<cplx<R>*>(ws.tmp) + rows * N;
    rows += probs[q].n;
    maxn = std::max(maxn, probs[q].n);
    ++a.nprob;
  }
  if (a.nprob == 0) return MNPBEM_OK;
  if (sizeof(cplx<R>) * rows * N > ws.tmp_bytes) { set_error("ldu_solve_few: workspace too small"); return MNPBEM_ERR_INVALID_ARG; }
  MNP_CUDA(cudaMemsetAsync(ws.ctl, 0, SWEEP_CTL * sizeof(unsigned), st));
  const int mb = (int)cdiv_up(maxn, (int64_t)b);
  // rows per warp: two, one where 16 sums per row fill the registers
  if (N <= 4) {
    MNP_TRY((launch_sweep<R, 4, 2, true>(a, mb, st)));
    return launch_sweep<R, 4, 2, false>(a, mb, st);
  }
  if (N <= 8) {
    MNP_TRY((launch_sweep<R, 8, 2, true>(a, mb, st)));
    return launch_sweep<R, 8, 2, false>(a, mb, st);
  }
  MNP_TRY((launch_sweep<R, 16, 1, true>(a, mb, st)));
  return launch_sweep<R, 16, 1, false>(a, mb, st);
}

template <typename R>
mnpbem_status ldu_solve(const cplx<R>* F, int64_t n, int64_t ldf, int b, cplx<R>* X, int64_t ldx, int64_t N,
                        cplx<R>* tmp, GemmFn<R> gemm, void* ctx, cudaStream_t st) {
  using Cx = cplx<R>;
  if (n <= 0 || N <= 0) return MNPBEM_OK;
  if (!tmp) { set_error("ldu_solve: workspace required"); return MNPBEM_ERR_INVALID_ARG; }
  const Cx one = mk<R>(1, 0), zero = mk<R>(0, 0), mone = mk<R>(-1, 0);
  const int64_t nblk = cdiv_up(n, (int64_t)b);
  // forward: L unit lower
  for (int64_t k = 0; k + 1 < nblk; ++k) {
    const int64_t k0 = k * b, kb = k0 + b;
    MNP_TRY(gemm(n - kb, N, b, mone, F + kb * ldf + k0, ldf, X + k0 * ldx, ldx, one, X + kb * ldx, ldx, st, ctx));
  }
  // block diagonal
  for (int64_t k = 0; k < nblk; ++k) {
    const int64_t k0 = k * b;
    const int bs = (int)std::min<int64_t>(b, n - k0);
    MNP_CUDA(cudaMemcpy2DAsync(tmp, sizeof(Cx) * N, X + k0 * ldx, sizeof(Cx) * ldx, sizeof(Cx) * N, bs,
                               cudaMemcpyDeviceToDevice, st));
    MNP_TRY(gemm(bs, N, bs, one, F + k0 * ldf + k0, ldf, tmp, N, zero, X + k0 * ldx, ldx, st, ctx));
  }
  // backward: U unit upper
  for (int64_t k = nblk - 1; k >= 1; --k) {
    const int64_t k0 = k * b;
    const int bs = (int)std::min<int64_t>(b, n - k0);
    MNP_TRY(gemm(k0, N, bs, mone, F + k0, ldf, X + k0 * ldx, ldx, one, X, ldx, st, ctx));
  }
  return MNPBEM_OK;
}

template mnpbem_status ldu_factor<float>(float2*, int64_t, int64_t, LDUWork<float>&, int*, GemmFn<float>, void*,
                                         cudaStream_t);
template mnpbem_status ldu_factor<double>(double2*, int64_t, int64_t, LDUWork<double>&, int*, GemmFn<double>, void*,
                                          cudaStream_t);
template mnpbem_status ldu_rsolve<float>(float2*, int64_t, int64_t, const float2*, int64_t, LDUWork<float>&,
                                         GemmFn<float>, void*, cudaStream_t);
template mnpbem_status ldu_rsolve<double>(double2*, int64_t, int64_t, const double2*, int64_t, LDUWork<double>&,
                                          GemmFn<double>, void*, cudaStream_t);
template mnpbem_status ldu_solve<float>(const float2*, int64_t, int64_t, int, float2*, int64_t, int64_t, float2*,
                                        GemmFn<float>, void*, cudaStream_t);
template mnpbem_status ldu_solve<double>(const double2*, int64_t, int64_t, int, double2*, int64_t, int64_t, double2*,
                                         GemmFn<double>, void*, cudaStream_t);
template mnpbem_status ldu_solve_few<float>(const LduProblem<float>*, int, int, int64_t, const LduSweepWs&,
                                            cudaStream_t);
template mnpbem_status ldu_solve_few<double>(const LduProblem<double>*, int, int, int64_t, const LduSweepWs&,
                                             cudaStream_t);

}  // namespace mnpbem
