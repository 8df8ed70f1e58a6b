// approx.cu -- SketchySVD::initial_approx + low_rank_approx
// (src/Skema_SketchySVD.cpp:338-664) on the device, in FP64.
//
//   P = orth(X^T)          (reference: dgeqrf+dorgqr, :355-357)
//   Q = orth(Y)            (:381-383; here Y is not overwritten)
//   [U1, T1] = qr(Phi~ Q)  (:409, :453)
//   [U2, T2] = qr(Psi~ P)  (:430, :476)
//   Z2 = U1^T Z U2         (:500, :515)
//   Z2 = T1 \ Z2           (dgels on the triangular T1, :532)
//   C  = (T2 \ Z2^T)^T     (:549-562)
//   [Uc, S, Vc] = svd(C)   (dgesvd, :609)
//   U = Q Uc(:, 1:r), V = P Vc(:, 1:r), S(1:r)   (:627, :645, :657-660)
//
// orth/qr use CholeskyQR2 (Gram on the device, Cholesky in one CTA, triangular
// solve of the rows), with the shifted CholeskyQR pre-pass of Fukaya,
// Kannan, Nakatsukasa, Yamamoto and Yanagisawa (SIAM J. Sci. Comput. 2020)
// when the Gram matrix is not numerically positive definite. The Q factor
// equals Householder's up to column signs, so S is unchanged and U, V match
// LAPACK's up to sign. The SVD of the k x k core is a one-sided (Hestenes)
// Jacobi SVD with round-robin pair ordering in one cluster of CTAs.
#include <cooperative_groups.h>
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <initializer_list>
#include <limits>
#include <memory>
#include <vector>

#include "internal.h"

namespace skema {

namespace {

// ---------------------------------------------------------------- DGEMM ----
// FP64 tensor cores: mma.sync m8n8k4 (D = A B + C, 8 x 4 by 4 x 8). Per lane:
// A holds element (lane / 4, lane % 4), B element (lane % 4, lane / 4), C / D
// elements (lane / 4, 2 (lane % 4) + i), i < 2.
__device__ __forceinline__ void dmma(double (&d)[2], double a, double b) {
  asm volatile("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0, %1}, {%2}, {%3}, {%0, %1};"
               : "+d"(d[0]), "+d"(d[1])
               : "d"(a), "d"(b));
}

// The sm_90 shape m16n8k16: A element (lane / 4 + 8 (i % 2), lane % 4 + 4 (i / 2)),
// i < 8; B (lane % 4 + 4 i, lane / 4), i < 4; D (lane / 4 + 8 (i / 2),
// 2 (lane % 4) + i % 2), i < 4.
__device__ __forceinline__ void dmma16(double (&d)[4], const double (&a)[8], const double (&b)[4]) {
  asm volatile(
      "mma.sync.aligned.m16n8k16.row.col.f64.f64.f64.f64 {%0, %1, %2, %3}, {%4, %5, %6, %7, %8, %9, %10, %11}, "
      "{%12, %13, %14, %15}, {%0, %1, %2, %3};"
      : "+d"(d[0]), "+d"(d[1]), "+d"(d[2]), "+d"(d[3])
      : "d"(a[0]), "d"(a[1]), "d"(a[2]), "d"(a[3]), "d"(a[4]), "d"(a[5]), "d"(a[6]), "d"(a[7]), "d"(b[0]), "d"(b[1]),
        "d"(b[2]), "d"(b[3]));
}

// C(i,j) = alpha * sum A(i,kk) B(kk,j) + beta*C(i,j); A, B may be float or
// double (widened when they are staged); FP64 accumulation. WM x WN warps of
// MB x NB blocks of 16 x 8 each; K steps of 16 through double-buffered shared memory
// whose rows are 4 (mod 16) doubles long, so that a fragment's 4 x 8 reads hit
// distinct banks. atomic: the K range is split over grid.z and the parts are
// added to C. Two shapes: 128 x 8 NB for a tall C (eight warps along M, so each
// A value is staged and widened once for all columns) and 32 x 32, four warps,
// for the k-sized products, which would fill a few SMs only with larger tiles.
// The residual pass on 50,000 x 10,000 at r = 50 (1e11 FP64 flop) takes 4.5 ms
// in these products (22 TFLOP/s; the tensor and the FMA pipe both peak at 66 FMA
// per cycle and SM, 37 TFLOP/s), the 64 x 64 SIMT form took 11.1.
template <typename TA, typename TB, int WM, int WN, int MB, int NB>
__global__ void __launch_bounds__(32 * WM * WN)
    dgemm_mma_kernel(int64_t M, int64_t N, int64_t K, double alpha, const TA* __restrict__ A, int64_t ars, int64_t acs,
                     const TB* __restrict__ B, int64_t brs, int64_t bcs, double beta, double* __restrict__ C,
                     int64_t crs, int64_t ccs, int64_t kchunk, int atomic) {
  constexpr int NT = 32 * WM * WN, BM = 16 * MB * WM, BN = 8 * NB * WN, KS = 16;
  constexpr int lda = (BM + 15) / 16 * 16 + 4, ldb = (BN + 15) / 16 * 16 + 4;
  constexpr int QA = BM * KS / NT, QB = (BN * KS + NT - 1) / NT;
  extern __shared__ __align__(16) double dg_smem[];
  double* As = dg_smem;                   // 2 x KS x lda
  double* Bs = dg_smem + 2 * KS * lda;    // 2 x KS x ldb
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, lr = lane & 3, lc = lane >> 2;
  const int64_t m0 = (int64_t)blockIdx.x * BM, n0 = (int64_t)blockIdx.y * BN;
  const int64_t kb = (int64_t)blockIdx.z * kchunk, ke = min(K, kb + kchunk);
  if (kb >= ke) return;
  const bool am = ars == 1, bn = bcs == 1;
  TA ra[QA];
  TB rb[QB];
  auto load = [&](int64_t k0) {
#pragma unroll
    for (int q = 0; q < QA; ++q) {
      const int e = tid + NT * q;
      const int m = am ? e % BM : e / KS, k = am ? e / BM : e % KS;
      ra[q] = (m0 + m < M && k0 + k < ke) ? A[(m0 + m) * ars + (k0 + k) * acs] : TA(0);
    }
#pragma unroll
    for (int q = 0; q < QB; ++q) {
      const int e = tid + NT * q;
      const int n = bn ? e % BN : e / KS, k = bn ? e / BN : e % KS;
      rb[q] = (e < BN * KS && n0 + n < N && k0 + k < ke) ? B[(k0 + k) * brs + (n0 + n) * bcs] : TB(0);
    }
  };
  auto store = [&](int buf) {
#pragma unroll
    for (int q = 0; q < QA; ++q) {
      const int e = tid + NT * q;
      As[(buf * KS + (am ? e / BM : e % KS)) * lda + (am ? e % BM : e / KS)] = (double)ra[q];
    }
#pragma unroll
    for (int q = 0; q < QB; ++q) {
      const int e = tid + NT * q;
      if (e < BN * KS) Bs[(buf * KS + (bn ? e / BN : e % KS)) * ldb + (bn ? e % BN : e / KS)] = (double)rb[q];
    }
  };
  const int wm = (warp % WM) * 16 * MB, wn = (warp / WM) * 8 * NB;
  double acc[MB][NB][4];
#pragma unroll
  for (int i = 0; i < MB; ++i)
#pragma unroll
    for (int j = 0; j < NB; ++j) acc[i][j][0] = acc[i][j][1] = acc[i][j][2] = acc[i][j][3] = 0.0;
  load(kb);
  store(0);
  __syncthreads();
  int buf = 0;
  for (int64_t k0 = kb; k0 < ke; k0 += KS, buf ^= 1) {
    const bool more = k0 + KS < ke;
    if (more) load(k0 + KS);
    const double* as = As + (buf * KS + lr) * lda + wm + lc;
    const double* bs = Bs + (buf * KS + lr) * ldb + wn + lc;
    double a[MB][8];
#pragma unroll
    for (int i = 0; i < MB; ++i)
#pragma unroll
      for (int h = 0; h < 8; ++h) a[i][h] = as[(h >> 1) * 4 * lda + 16 * i + 8 * (h & 1)];
#pragma unroll
    for (int j = 0; j < NB; ++j) {
      double b[4];
#pragma unroll
      for (int h = 0; h < 4; ++h) b[h] = bs[4 * h * ldb + 8 * j];
#pragma unroll
      for (int i = 0; i < MB; ++i) dmma16(acc[i][j], a[i], b);
    }
    if (more) store(buf ^ 1);  // read last one step ago, before the barrier
    __syncthreads();
  }
#pragma unroll
  for (int i = 0; i < MB; ++i)
#pragma unroll
    for (int j = 0; j < NB; ++j)
#pragma unroll
      for (int h = 0; h < 4; ++h) {
        const int64_t gm = m0 + wm + 16 * i + lc + 8 * (h >> 1), gn = n0 + wn + 8 * j + 2 * lr + (h & 1);
        if (gm >= M || gn >= N) continue;
        double* cp = C + gm * crs + gn * ccs;
        const double v = alpha * acc[i][j][h];
        if (atomic)
          atomicAdd(cp, v);
        else
          *cp = (beta == 0.0) ? v : fma(beta, *cp, v);
      }
}

__global__ void dscale_kernel(double* C, int64_t crs, int64_t ccs, int64_t M, int64_t N, double b) {
  for (int64_t q = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; q < M * N;
       q += (int64_t)gridDim.x * blockDim.x) {
    const int64_t i = q % M, j = q / M;
    double* p = C + i * crs + j * ccs;
    *p = (b == 0.0) ? 0.0 : b * *p;
  }
}

template <typename TA, typename TB, int WM, int WN, int MB, int NB>
void launch_dgemm(skema_ctx* c, int64_t M, int64_t N, int64_t K, double alpha, const TA* A, int64_t ars, int64_t acs,
                  const TB* B, int64_t brs, int64_t bcs, double beta, double* C, int64_t crs, int64_t ccs,
                  bool allow_split) {
  constexpr int64_t BM = 16 * MB * WM, BN = 8 * NB * WN;
  constexpr size_t smem = sizeof(double) * 2 * 16 * ((BM + 15) / 16 * 16 + 4 + (BN + 15) / 16 * 16 + 4);
  const int64_t gx = (M + BM - 1) / BM, gy = (N + BN - 1) / BN;
  if (gy > 65535) fail(SKEMA_EUNSUPPORTED, "dgemm: N too large");
  // K ranges of 256 or more, about four CTAs per SM in all; with tiles for
  // two to eight per SM, ranges of 1024 or more and sixteen per SM, so that
  // no SM is left with one tile more than the others
  int64_t split = 1;
  if (allow_split && gx * gy < 2 * c->sm_count && K >= 512)
    split = std::min<int64_t>((4 * c->sm_count + gx * gy - 1) / (gx * gy), K / 256);
  if (allow_split && gx * gy < 8 * c->sm_count)
    split = std::max(split, std::min<int64_t>((16 * c->sm_count + gx * gy - 1) / (gx * gy), K / 1024));
  if (split > 1) {
    dscale_kernel<<<(int)std::min<int64_t>((M * N + 255) / 256, 4096), 256, 0, c->stream>>>(C, crs, ccs, M, N, beta);
    SKEMA_LAUNCHED(c);
  }
  const int64_t kchunk = ((K + split - 1) / split + 15) / 16 * 16;
  const int64_t gz = std::max<int64_t>(1, (K + kchunk - 1) / kchunk);
  auto kern = dgemm_mma_kernel<TA, TB, WM, WN, MB, NB>;
  SKEMA_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
  kern<<<dim3((unsigned)gx, (unsigned)gy, (unsigned)gz), 32 * WM * WN, smem, c->stream>>>(
      M, N, K, alpha, A, ars, acs, B, brs, bcs, beta, C, crs, ccs, kchunk, split > 1 ? 1 : 0);
  SKEMA_LAUNCHED(c);
}

template <typename TA, typename TB>
void dgemm(skema_ctx* c, int64_t M, int64_t N, int64_t K, double alpha, const TA* A, int64_t ars,
           int64_t acs, const TB* B, int64_t brs, int64_t bcs, double beta, double* C, int64_t crs,
           int64_t ccs, bool allow_split = true) {
  if (M <= 0 || N <= 0) return;
  if (K <= 0) {
    dscale_kernel<<<(int)std::min<int64_t>((M * N + 255) / 256, 4096), 256, 0, c->stream>>>(C, crs, ccs, M, N, beta);
    SKEMA_LAUNCHED(c);
    return;
  }
  auto go = [&](auto launch) {
    launch(c, M, N, K, alpha, A, ars, acs, B, brs, bcs, beta, C, crs, ccs, allow_split);
  };
  if (M < 1024) {
    go(launch_dgemm<TA, TB, 2, 2, 1, 2>);
    return;
  }
  switch (std::min<int64_t>(8, (N + 7) / 8)) {
    case 1: go(launch_dgemm<TA, TB, 8, 1, 1, 1>); break;
    case 2: go(launch_dgemm<TA, TB, 8, 1, 1, 2>); break;
    case 3: go(launch_dgemm<TA, TB, 8, 1, 1, 3>); break;
    case 4: go(launch_dgemm<TA, TB, 8, 1, 1, 4>); break;
    case 5: go(launch_dgemm<TA, TB, 8, 1, 1, 5>); break;
    case 6: go(launch_dgemm<TA, TB, 8, 1, 1, 6>); break;
    case 7: go(launch_dgemm<TA, TB, 8, 1, 1, 7>); break;
    default: go(launch_dgemm<TA, TB, 8, 1, 1, 8>); break;
  }
}

// ----------------------------------------- tall-skinny FP64 products -------
// G += A^T A for a tall column-major A (rows x k, ld lda, k <= 256; T float
// or double, widened to FP64 exactly). A CTA stages 32 rows of all k columns in
// shared memory (128- or 256-byte runs of a column, widened once; a column's
// 32 rows are 36 doubles apart, so fragment reads hit distinct banks) and its
// warps form the 16 x 8 blocks on or above the diagonal with m16n8k16, up to
// NT each, in registers over all of the CTA's rows; blockIdx.y takes a group of
// blocks when they do not all fit. Up to three blocks a warp (k <= 96), two CTAs
// per SM run and each loads its next rows while it multiplies (502 and 490 us
// without). The parts go to G (column-major k x k, zeroed
// beforehand) with atomics, mirrored below the diagonal. Bound by the FP64
// pipe: 1e6 x 81 takes 358 us from FP32 and 386 from FP64 (793 and 734 with
// fragments read from global memory by every warp that needs them).
constexpr int kGramTiles = 6, kGramLd = 36;
template <typename T, int NT>
__global__ void __launch_bounds__(NT <= 3 ? 384 : 512, NT <= 3 ? 2 : 1)
    gram_mma_kernel(const T* __restrict__ A, int64_t lda, int k, int64_t rows, double* __restrict__ G,
                    int64_t rows_per_cta) {
  extern __shared__ __align__(16) double gr_smem[];  // (k up to 16) x kGramLd
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, nw = blockDim.x >> 5, lr = lane & 3, lc = lane >> 2;
  const int nm = (k + 15) >> 4, nn = (k + 7) >> 3;
  // this warp's blocks (mi, ni), ni >= 2 mi, m-major, consecutive
  int mi[NT], ni[NT], cnt = 0;
  {
    const int per = NT * nw;
    int total = 0;
    for (int m = 0; m < nm; ++m) total += nn - 2 * m;
    const int first = (int)blockIdx.y * per, last = min(total, first + per), n = last - first;
    int t = first + (int)((int64_t)n * warp / nw);
    const int te = first + (int)((int64_t)n * (warp + 1) / nw);
    int m = 0, base = 0;
    while (m < nm - 1 && t >= base + nn - 2 * m) base += nn - 2 * m, ++m;
#pragma unroll
    for (int q = 0; q < NT; ++q) {
      mi[q] = ni[q] = 0;
      if (t < te) {
        while (t >= base + nn - 2 * m) base += nn - 2 * m, ++m;
        mi[q] = m;
        ni[q] = 2 * m + t - base;
        ++cnt;
        ++t;
      }
    }
  }
  double acc[NT][4];
#pragma unroll
  for (int q = 0; q < NT; ++q) acc[q][0] = acc[q][1] = acc[q][2] = acc[q][3] = 0.0;
  const int64_t r0 = (int64_t)blockIdx.x * rows_per_cta, r1 = min(rows, r0 + rows_per_cta);
  const int kpad = nm * 16;
  // NT <= 3 (k up to 96, eight columns a warp): the next rows are loaded while
  // the current ones multiply
  constexpr int PF = NT <= 3 ? 8 : 0;
  T nx[PF > 0 ? PF : 1];
  auto prefetch = [&](int64_t r) {
#pragma unroll
    for (int u = 0; u < PF; ++u) {
      const int cc = warp + u * nw;
      nx[u] = (r + lane < r1 && cc < k) ? A[(int64_t)cc * lda + r + lane] : T(0);
    }
  };
  prefetch(r0);
  for (int64_t r = r0; r < r1; r += 32) {
    const bool rv = r + lane < r1;
#pragma unroll
    for (int u = 0; u < PF; ++u)
      if (warp + u * nw < kpad) gr_smem[(warp + u * nw) * kGramLd + lane] = (double)nx[u];
    for (int c = warp + PF * nw; c < kpad; c += 4 * nw) {
      T v[4];
#pragma unroll
      for (int u = 0; u < 4; ++u) {
        const int cc = c + u * nw;
        v[u] = (rv && cc < k) ? A[(int64_t)cc * lda + r + lane] : T(0);
      }
#pragma unroll
      for (int u = 0; u < 4; ++u)
        if (c + u * nw < kpad) gr_smem[(c + u * nw) * kGramLd + lane] = (double)v[u];
    }
    __syncthreads();
    prefetch(r + 32);
#pragma unroll
    for (int h = 0; h < 32; h += 16) {
      double a[8];
      int held = -1;
#pragma unroll
      for (int q = 0; q < NT; ++q) {
        if (q >= cnt) continue;
        if (mi[q] != held) {
          held = mi[q];
#pragma unroll
          for (int i = 0; i < 8; ++i)
            a[i] = gr_smem[(16 * held + lc + 8 * (i & 1)) * kGramLd + h + lr + 4 * (i >> 1)];
        }
        double b[4];
#pragma unroll
        for (int i = 0; i < 4; ++i) b[i] = gr_smem[(8 * ni[q] + lc) * kGramLd + h + lr + 4 * i];
        dmma16(acc[q], a, b);
      }
    }
    __syncthreads();
  }
#pragma unroll
  for (int q = 0; q < NT; ++q) {
    if (q >= cnt) continue;
#pragma unroll
    for (int h = 0; h < 4; ++h) {
      const int gi = 16 * mi[q] + lc + 8 * (h >> 1), gj = 8 * ni[q] + 2 * lr + (h & 1);
      if (gi >= k || gj >= k || gi > gj) continue;
      atomicAdd(G + gi + (int64_t)gj * k, acc[q][h]);
      if (gi != gj) atomicAdd(G + gj + (int64_t)gi * k, acc[q][h]);
    }
  }
}

// C += A^T B for two tall column-major matrices with the same rows (A rows x
// ka, B rows x kb, kb <= 256; T float or double; C column-major with ld ka,
// zeroed beforehand), which is how a dense map meets a tall basis (Phi~ Q =
// (Phi~^T)^T Q). The product is cut into 32 x 32 tiles, each formed by P warps
// of the CTA that split the CTA's rows four at a time; a warp holds its tile as
// 4 x 4 MMA blocks (m8n8k4). For a step of four rows the fragment of column
// block c is (r + lane % 4, c + lane / 4), for A and B alike. The partial tiles
// go to C with atomics.
template <typename TA, typename TB>
__global__ void __launch_bounds__(512) atb_mma_kernel(const TA* __restrict__ A, int64_t lda, int ka,
                                                      const TB* __restrict__ B, int64_t ldb, int kb, int64_t rows,
                                                      double* __restrict__ G, int64_t rows_per_cta, int P) {
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int nia = (ka + 31) >> 5, njb = (kb + 31) >> 5;
  const int ntiles = nia * njb;
  // blockIdx.y takes a group of tiles when they do not all fit one CTA
  const int per_cta = (int)(blockDim.x >> 5) / P;
  const int tile = (int)blockIdx.y * per_cta + warp / P, part = warp % P;
  if (tile >= ntiles) return;
  const int ti = tile / njb, tj = tile - (tile / njb) * njb;
  const int64_t r0 = (int64_t)blockIdx.x * rows_per_cta, r1 = min(rows, r0 + rows_per_cta);
  const int lr = lane & 3, lc = lane >> 2;
  const TA* ci[4];
  const TB* cj[4];
  bool vi[4], vj[4];
#pragma unroll
  for (int m = 0; m < 4; ++m) {
    const int coli = 32 * ti + 8 * m + lc, colj = 32 * tj + 8 * m + lc;
    vi[m] = coli < ka;
    vj[m] = colj < kb;
    ci[m] = A + (int64_t)(vi[m] ? coli : 0) * lda;
    cj[m] = B + (int64_t)(vj[m] ? colj : 0) * ldb;
  }
  double acc[4][4][2];
#pragma unroll
  for (int m = 0; m < 4; ++m)
#pragma unroll
    for (int n = 0; n < 4; ++n) acc[m][n][0] = acc[m][n][1] = 0.0;
  // two steps of four rows per iteration: their 16 loads are in flight
  // together before the 32 MMAs that use them
  for (int64_t r = r0 + 4 * part; r < r1; r += 8 * P) {
    double a[2][4], b[2][4];
#pragma unroll
    for (int u = 0; u < 2; ++u) {
      const int64_t row = r + 4 * P * u + lr;
      const bool rv = row < r1;
#pragma unroll
      for (int m = 0; m < 4; ++m) {
        a[u][m] = (rv && vi[m]) ? (double)ci[m][row] : 0.0;
        b[u][m] = (rv && vj[m]) ? (double)cj[m][row] : 0.0;
      }
    }
#pragma unroll
    for (int u = 0; u < 2; ++u)
#pragma unroll
      for (int m = 0; m < 4; ++m)
#pragma unroll
        for (int n = 0; n < 4; ++n) dmma(acc[m][n], a[u][m], b[u][n]);
  }
#pragma unroll
  for (int m = 0; m < 4; ++m)
#pragma unroll
    for (int n = 0; n < 4; ++n)
#pragma unroll
      for (int i = 0; i < 2; ++i) {
        const int gi = 32 * ti + 8 * m + lc, gj = 32 * tj + 8 * n + 2 * lr + i;
        if (gi >= ka || gj >= kb) continue;
        atomicAdd(G + gi + (int64_t)gj * ka, acc[m][n][i]);
      }
}

// C = A B for a tall column-major A (rows x k, ld lda; T float or double)
// and a small B (k x n2, column-major ld ldb, k, n2 <= 8 NB). B stays in
// shared memory for the CTA's life as 4-row slices laid out for its MMA
// fragments; each warp takes 16-row tiles of C with every column block in
// registers. K goes in batches of 32 whose A values are loaded one batch
// ahead; a column block then takes its eight B values and two m16n8k16 MMAs of
// the batch together. UPPER: B is upper triangular, so column block nb only
// needs the rows of B up to its last column and the batches past it are
// skipped (about half the work for Q R^{-1}); the test per batch, not per four
// rows, is what lets the B loads run ahead of the MMAs. C is column-major
// (ld ldc) and written, not accumulated. Bound by the FP64 pipe and by the
// 64-byte pieces of C: 1e6 x 81 by 81 x 81 takes 490 us (934 with m8n8k4 and a
// test per four rows).
template <typename T, int NB, bool UPPER>
__global__ void __launch_bounds__(256) tsm_mma_kernel(const T* __restrict__ A, int64_t lda, int64_t rows, int k,
                                                      const double* __restrict__ B, int64_t ldb, int n2,
                                                      double* __restrict__ C, int64_t ldc, int col0) {
  // B and C are the columns [col0, col0 + n2) of the whole product (col0
  // places them against the triangle for UPPER)
  extern __shared__ double tsm_smem[];
  // Bs[kk * ldbs + col], ldbs = 8 NB + 4 (mod 16) so a fragment's 4 x 8
  // reads hit 16 distinct bank pairs per half-warp
  constexpr int ldbs = (8 * NB + 15) / 16 * 16 + 4;
  const int kp = (k + 31) & ~31;  // whole batches; rows past k are zeros
  for (int q = threadIdx.x; q < kp * 8 * NB; q += blockDim.x) {
    const int kk = q / (8 * NB), col = q - kk * (8 * NB);
    tsm_smem[kk * ldbs + col] = (kk < k && col < n2) ? B[kk + (int64_t)col * ldb] : 0.0;
  }
  __syncthreads();
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, nwarp = blockDim.x >> 5;
  const int lr = lane & 3, lc = lane >> 2;
  for (int64_t r0 = ((int64_t)blockIdx.x * nwarp + warp) * 16; r0 < rows; r0 += (int64_t)gridDim.x * nwarp * 16) {
    double acc[NB][4];
#pragma unroll
    for (int n = 0; n < NB; ++n) acc[n][0] = acc[n][1] = acc[n][2] = acc[n][3] = 0.0;
    const int64_t ra = r0 + lc, rb = r0 + 8 + lc;
    const bool va = ra < rows, vb = rb < rows;
    T q0[8], q1[8];
    auto load = [&](int kb) {
#pragma unroll
      for (int j = 0; j < 8; ++j) {
        const int kk = kb + 4 * j + lr;
        const bool kv = kk < k;
        q0[j] = (va && kv) ? A[ra + (int64_t)kk * lda] : T(0);
        q1[j] = (vb && kv) ? A[rb + (int64_t)kk * lda] : T(0);
      }
    };
    load(0);
    for (int kb = 0; kb < kp; kb += 32) {
      double a[2][8];
#pragma unroll
      for (int j = 0; j < 8; ++j) {
        a[j >> 2][2 * (j & 3)] = (double)q0[j];
        a[j >> 2][2 * (j & 3) + 1] = (double)q1[j];
      }
      if (kb + 32 < kp) load(kb + 32);
      const double* bs = tsm_smem + (kb + lr) * ldbs + lc;
#pragma unroll
      for (int n = 0; n < NB; ++n) {
        if (UPPER && col0 + 8 * n + 7 < kb) continue;  // B(kb.., block n) is zero
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          double b[4];
#pragma unroll
          for (int i = 0; i < 4; ++i) b[i] = bs[(16 * h + 4 * i) * ldbs + 8 * n];
          dmma16(acc[n], a[h], b);
        }
      }
    }
#pragma unroll
    for (int m = 0; m < 2; ++m) {
      const int64_t row = r0 + 8 * m + lc;
      if (row >= rows) continue;
#pragma unroll
      for (int n = 0; n < NB; ++n)
#pragma unroll
        for (int i = 0; i < 2; ++i) {
          const int col = 8 * n + 2 * lr + i;
          if (col < n2) C[row + (int64_t)col * ldc] = acc[n][2 * m + i];
        }
    }
  }
}

// C (ka x kb, column-major, zeroed beforehand) += A^T B.
template <typename TA, typename TB>
void launch_atb_mma(skema_ctx* c, const TA* A, int64_t lda, int64_t ka, const TB* B, int64_t ldb, int64_t kb,
                    int64_t rows, double* G) {
  const int nia = (int)((ka + 31) / 32), njb = (int)((kb + 31) / 32);
  const int tiles = nia * njb;
  // up to 16 warps per CTA: P warps per tile when the tiles leave room,
  // else groups of 16 tiles over blockIdx.y
  const int P = std::max(1, 16 / tiles);
  const int per_cta = std::min(tiles, 16 / P);
  const int groups = (tiles + per_cta - 1) / per_cta;
  const int64_t ctas = std::max<int64_t>(1, std::min<int64_t>((rows + 1023) / 1024, (int64_t)c->sm_count));
  const int64_t per = ((rows + ctas - 1) / ctas + 3) / 4 * 4;
  const dim3 grid((unsigned)((rows + per - 1) / per), (unsigned)groups);
  atb_mma_kernel<TA, TB><<<grid, 32 * per_cta * P, 0, c->stream>>>(A, lda, (int)ka, B, ldb, (int)kb, rows, G, per, P);
  SKEMA_LAUNCHED(c);
}

// G (k x k, column-major, zeroed beforehand) += A^T A.
template <typename T>
void launch_gram(skema_ctx* c, const T* A, int64_t lda, int64_t k, int64_t rows, double* G) {
  int tiles = 0;
  for (int64_t m = 0; m < (k + 15) / 16; ++m) tiles += (int)((k + 7) / 8 - 2 * m);
  // up to 16 warps, as many as share the blocks evenly: the fewest blocks per
  // warp, then the fewest warps
  const int groups = (tiles + 16 * kGramTiles - 1) / (16 * kGramTiles);
  const int per_cta = (tiles + groups - 1) / groups;
  int depth = (per_cta + 15) / 16, warps = std::max(4, (per_cta + depth - 1) / depth);
  if (depth <= 3 && warps > 12) depth = (per_cta + 11) / 12, warps = (per_cta + depth - 1) / depth;
  const size_t smem = sizeof(double) * (size_t)((k + 15) / 16 * 16 * kGramLd);
  const bool few = depth <= 3;
  const int64_t ctas =
      std::max<int64_t>(1, std::min<int64_t>((rows + 63) / 64, (few ? 2 : 1) * (int64_t)c->sm_count / groups));
  const int64_t per = ((rows + ctas - 1) / ctas + 31) / 32 * 32;
  auto kern = few ? gram_mma_kernel<T, 3> : gram_mma_kernel<T, kGramTiles>;
  const int ny = (tiles + warps * (few ? 3 : kGramTiles) - 1) / (warps * (few ? 3 : kGramTiles));
  SKEMA_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
  kern<<<dim3((unsigned)((rows + per - 1) / per), (unsigned)ny), 32 * warps, smem, c->stream>>>(A, lda, (int)k, rows, G,
                                                                                               per);
  SKEMA_LAUNCHED(c);
}

template <typename T, int NB>
void launch_tsm_nb(skema_ctx* c, const T* A, int64_t lda, int64_t rows, int64_t k, const double* B, int64_t ldb,
                   int64_t n2, double* C, int64_t ldc, bool upper, int col0) {
  constexpr int ldbs = (8 * NB + 15) / 16 * 16 + 4;
  const size_t smem = sizeof(double) * (size_t)(((k + 31) & ~31) * ldbs);
  auto kern = upper ? tsm_mma_kernel<T, NB, true> : tsm_mma_kernel<T, NB, false>;
  SKEMA_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
  const int64_t tiles = (rows + 15) / 16;
  const int grid = (int)std::max<int64_t>(1, std::min<int64_t>((tiles + 7) / 8, 4 * (int64_t)c->sm_count));
  kern<<<grid, 256, smem, c->stream>>>(A, lda, rows, (int)k, B, ldb, (int)n2, C, ldc, col0);
  SKEMA_LAUNCHED(c);
}

// G (k x k, column-major) = A^T A for column-major A (rows x k, ld lda).
constexpr int64_t kTallMaxK = 256;  // the tall products take k up to this
constexpr int64_t kTallMinRows = 1024;  // and rows from this on
template <typename T>
void gram_t(skema_ctx* c, const T* A, int64_t lda, int64_t rows, int64_t k, double* G) {
  SKEMA_CUDA(cudaMemsetAsync(G, 0, sizeof(double) * (size_t)(k * k), c->stream));
  if (rows > 0) launch_gram<T>(c, A, lda, k, rows, G);
}
void gram(skema_ctx* c, const double* A, int64_t lda, int64_t rows, int64_t k, double* G) {
  if (rows <= 0) {  // an empty row block (a rank without rows) adds nothing
    SKEMA_CUDA(cudaMemsetAsync(G, 0, sizeof(double) * (size_t)(k * k), c->stream));
    return;
  }
  // the k-sized products of a larger k take the 32 x 32 tiles of dgemm, whose
  // grid does not shrink with the rows (403 x 201: 15 us against 77; 300 x 81 the
  // same within 2 us; 1,000 x 9 36 against 10)
  if (k > kTallMaxK || (rows < kTallMinRows && k > 40)) {
    dgemm<double, double>(c, k, k, rows, 1.0, A, lda, 1, A, 1, lda, 0.0, G, 1, k);
    return;
  }
  gram_t<double>(c, A, lda, rows, k, G);
}

// Column block width of the tall product: B's k x (8 NB) slice (padded)
// stays in shared memory, at most 220 KB.
int tsm_chunk_blocks(int64_t k) {
  const int64_t kp = (k + 31) & ~31;
  for (int nb = 16; nb > 1; --nb) {
    const int64_t ldbs = (8 * nb + 15) / 16 * 16 + 4;
    if (kp * ldbs * (int64_t)sizeof(double) <= 220 * 1024) return nb;
  }
  return 1;
}

// C (rows x n2) = A (rows x k) B (k x n2), all column-major; upper: B is
// upper triangular (its zeros below the diagonal are not read). Column
// blocks of B beyond what shared memory holds go in further launches.
template <typename T>
void tall_times_small_t(skema_ctx* c, const T* A, int64_t lda, int64_t rows, int64_t k, const double* B,
                        int64_t ldb, int64_t n2, double* C, int64_t ldc, bool upper) {
  const int64_t chunk = 8 * (int64_t)tsm_chunk_blocks(k);
  for (int64_t c0 = 0; c0 < n2; c0 += chunk) {
    const int64_t w = std::min(chunk, n2 - c0);
    const double* Bc = B + c0 * ldb;
    double* Cc = C + c0 * ldc;
    const int col0 = (int)c0;
    switch ((w + 7) / 8) {
      case 1: launch_tsm_nb<T, 1>(c, A, lda, rows, k, Bc, ldb, w, Cc, ldc, upper, col0); break;
      case 2: launch_tsm_nb<T, 2>(c, A, lda, rows, k, Bc, ldb, w, Cc, ldc, upper, col0); break;
      case 3: launch_tsm_nb<T, 3>(c, A, lda, rows, k, Bc, ldb, w, Cc, ldc, upper, col0); break;
      case 4: launch_tsm_nb<T, 4>(c, A, lda, rows, k, Bc, ldb, w, Cc, ldc, upper, col0); break;
      case 5: launch_tsm_nb<T, 5>(c, A, lda, rows, k, Bc, ldb, w, Cc, ldc, upper, col0); break;
      case 6: launch_tsm_nb<T, 6>(c, A, lda, rows, k, Bc, ldb, w, Cc, ldc, upper, col0); break;
      case 7: launch_tsm_nb<T, 7>(c, A, lda, rows, k, Bc, ldb, w, Cc, ldc, upper, col0); break;
      case 8: launch_tsm_nb<T, 8>(c, A, lda, rows, k, Bc, ldb, w, Cc, ldc, upper, col0); break;
      case 9: launch_tsm_nb<T, 9>(c, A, lda, rows, k, Bc, ldb, w, Cc, ldc, upper, col0); break;
      case 10: launch_tsm_nb<T, 10>(c, A, lda, rows, k, Bc, ldb, w, Cc, ldc, upper, col0); break;
      case 11: launch_tsm_nb<T, 11>(c, A, lda, rows, k, Bc, ldb, w, Cc, ldc, upper, col0); break;
      case 12: launch_tsm_nb<T, 12>(c, A, lda, rows, k, Bc, ldb, w, Cc, ldc, upper, col0); break;
      case 13: launch_tsm_nb<T, 13>(c, A, lda, rows, k, Bc, ldb, w, Cc, ldc, upper, col0); break;
      case 14: launch_tsm_nb<T, 14>(c, A, lda, rows, k, Bc, ldb, w, Cc, ldc, upper, col0); break;
      case 15: launch_tsm_nb<T, 15>(c, A, lda, rows, k, Bc, ldb, w, Cc, ldc, upper, col0); break;
      default: launch_tsm_nb<T, 16>(c, A, lda, rows, k, Bc, ldb, w, Cc, ldc, upper, col0); break;
    }
  }
}
void tall_times_small(skema_ctx* c, const double* A, int64_t lda, int64_t rows, int64_t k, const double* B,
                      int64_t ldb, int64_t n2, double* C, int64_t ldc, bool upper = false) {
  if (rows <= 0 || n2 <= 0) return;
  if (k > kTallMaxK || rows < kTallMinRows) {
    dgemm<double, double>(c, rows, n2, k, 1.0, A, 1, lda, B, 1, ldb, 0.0, C, 1, ldc, false);
    return;
  }
  tall_times_small_t<double>(c, A, lda, rows, k, B, ldb, n2, C, ldc, upper);
}

// ----------------------------------------------------- conversions ----------
__global__ void f2d_kernel(const float* __restrict__ S, int64_t srs, int64_t scs,
                           double* __restrict__ D, int64_t drs, int64_t dcs, int64_t M, int64_t N) {
  for (int64_t q = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; q < M * N;
       q += (int64_t)gridDim.x * blockDim.x) {
    int64_t i, j;
    if (drs == 1) { i = q % M; j = q / M; } else { i = q / N; j = q % N; }
    D[i * drs + j * dcs] = (double)S[i * srs + j * scs];
  }
}

// ----------------------------------------------------------- Cholesky -------
// In place on the lower triangle of the column-major k x k G (one CTA).
// status[0] = 0 ok, j+1 if the j-th pivot was not positive.
__global__ void cholesky_kernel(double* G, int64_t k, int* status) {
  __shared__ double piv;
  __shared__ int bad;
  if (threadIdx.x == 0) bad = 0;
  __syncthreads();
  for (int64_t j = 0; j < k; ++j) {
    if (threadIdx.x == 0) {
      const double d = G[j + j * k];
      if (!(d > 0.0) && !bad) bad = (int)(j + 1);
      piv = (d > 0.0) ? sqrt(d) : 1.0;
      G[j + j * k] = piv;
    }
    __syncthreads();
    if (bad) break;
    for (int64_t i = j + 1 + threadIdx.x; i < k; i += blockDim.x) G[i + j * k] /= piv;
    __syncthreads();
    // trailing update of the lower triangle: G(a, b) -= L(a, j) L(b, j), b > j, a >= b
    const int64_t rem = k - j - 1;
    for (int64_t q = threadIdx.x; q < rem * rem; q += blockDim.x) {
      const int64_t a = j + 1 + q % rem, b = j + 1 + q / rem;
      if (a >= b) G[a + b * k] -= G[a + j * k] * G[b + j * k];
    }
    __syncthreads();
  }
  if (threadIdx.x == 0) status[0] = bad;
}

// R (upper, column-major k x k) = L^T from the factored lower triangle of G.
__global__ void lower_to_upper_kernel(const double* G, double* R, int64_t k) {
  for (int64_t q = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; q < k * k;
       q += (int64_t)gridDim.x * blockDim.x) {
    const int64_t i = q % k, j = q / k;
    R[i + j * k] = (i <= j) ? G[j + i * k] : 0.0;
  }
}

// Solve R X = B in place for upper-triangular R (column-major k x k) and B
// (k x nrhs, column stride ldb): one warp per right-hand side.
__global__ void trsm_upper_kernel(const double* __restrict__ R, int64_t k, double* B, int64_t ldb,
                                  int64_t nrhs) {
  const int lane = threadIdx.x & 31;
  const int64_t col = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  if (col >= nrhs) return;
  double* x = B + col * ldb;
  for (int64_t i = k - 1; i >= 0; --i) {
    double s = 0.0;
    for (int64_t l = i + 1 + lane; l < k; l += 32) s += R[i + l * k] * x[l];
    for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
    if (lane == 0) x[i] = (x[i] - s) / R[i + i * k];
    __syncwarp();
  }
}

// Packed triangles in shared memory. Upper: column j holds rows 0..j from
// j (j + 1) / 2. Lower: column j holds rows j..k-1 from j k - j (j - 1) / 2.
__device__ __forceinline__ int up_off(int j) { return j * (j + 1) / 2; }
__device__ __forceinline__ int lo_off(int j, int k) { return j * k - j * (j - 1) / 2; }

// Largest k for which a packed triangle and one warp's right-hand sides fit
// shared memory (217,800 bytes at 225).
constexpr int kPackedMaxK = 225;
size_t packed_smem_bytes(int64_t k) { return sizeof(double) * (size_t)(k * (k + 1) / 2); }
// Row stride of a warp's right-hand sides: k rounded up to 16, plus 4, so that
// the 4 x 8 fragment reads hit distinct banks.
__host__ __device__ __forceinline__ int tri_ld(int k) { return (k + 15) / 16 * 16 + 4; }

// Solve R X = B, R upper triangular (column-major k x k), B k x nrhs (column
// stride ldb) in place, or with B the identity (its columns are not read: X =
// R^{-1}). R packed in shared memory with its 8 x 8 diagonal blocks inverted in
// place; a warp (nw of them) takes eight right-hand sides and goes up by block rows,
//   X_I = inv(R_II) (B_I - sum_{K > I} R_IK X_K),
// every product on the FP64 tensor cores (m8n8k4), so a step is a few MMAs
// instead of eight dependent eliminations. The right-hand sides are spread over
// the grid, so the inverse of a Cholesky factor no longer runs in one CTA.
// k = 201, nrhs = 201: 44 us, 35 for the identity (a column at a time in
// registers took 75; 114 when only the solving warps filled shared memory).
// Returns at once when *status (may be null) is not 0.
constexpr int kTriThreads = 512;
__global__ void __launch_bounds__(kTriThreads)
    tri_solve_kernel(const double* __restrict__ R, int k, double* B, int64_t ldb, int nrhs, int nw, int identity,
                     const int* __restrict__ status) {
  if (status && *status != 0) return;
  extern __shared__ __align__(16) double ts_smem[];
  double* Rp = ts_smem;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, lr = lane & 3, lc = lane >> 2;
  const int ld = tri_ld(k), nblk = (k + 7) >> 3;
  double* X = Rp + k * (k + 1) / 2 + (size_t)warp * 8 * ld;  // column c, row i at X[c * ld + i]
  const int nall = blockDim.x >> 5;  // all warps fill shared memory, nw solve
#pragma unroll 4
  for (int j = warp; j < k; j += nall)
#pragma unroll
    for (int v = 0; v < 8; ++v) {  // k <= 225 rows
      const int i = lane + 32 * v;
      if (i <= j) Rp[up_off(j) + i] = R[i + j * k];
    }
  __syncthreads();
  for (int t = warp; t < nblk; t += nall) {
    const int o = 8 * t, nb = min(8, k - o);
    double x[8];
    if (lane < nb) {  // column `lane` of the block's inverse
#pragma unroll
      for (int i = 7; i >= 0; --i) {
        x[i] = 0.0;
        if (i >= nb || i > lane) continue;
        double v = i == lane ? 1.0 : 0.0;
#pragma unroll
        for (int l = i + 1; l < 8; ++l)
          if (l <= lane && l < nb) v = fma(-Rp[up_off(o + l) + o + i], x[l], v);
        x[i] = v / Rp[up_off(o + i) + o + i];
      }
    }
    __syncwarp();
    if (lane < nb) {
#pragma unroll
      for (int i = 0; i < 8; ++i)
        if (i <= lane) Rp[up_off(o + lane) + o + i] = x[i];
    }
  }
  __syncthreads();
  const int c0 = ((int)blockIdx.x * nw + warp) * 8;
  if (warp >= nw || c0 >= nrhs) return;
  const int nc = min(8, nrhs - c0);
  for (int q = lane; q < 8 * ld; q += 32) {
    const int c = q / ld, i = q - c * ld;
    X[q] = (c >= nc || i >= k) ? 0.0 : identity ? (i == c0 + c ? 1.0 : 0.0) : B[(int64_t)(c0 + c) * ldb + i];
  }
  __syncwarp();
  // columns of the identity start at their own block row
  for (int I = identity ? min(nblk - 1, c0 >> 3) : nblk - 1; I >= 0; --I) {
    const int row = 8 * I + lc;
    double s0[2] = {0.0, 0.0}, s1[2] = {0.0, 0.0};
    const int Kend = identity ? min(nblk - 1, c0 >> 3) : nblk - 1;
#pragma unroll 4
    for (int K = I + 1; K <= Kend; ++K) {
      const int ca = 8 * K + lr, cb = ca + 4;
      const double a0 = ca < k ? Rp[up_off(ca) + row] : 0.0, a1 = cb < k ? Rp[up_off(cb) + row] : 0.0;
      dmma(s0, a0, X[lc * ld + ca]);
      dmma(s1, a1, X[lc * ld + cb]);
    }
    __syncwarp();
#pragma unroll
    for (int h = 0; h < 2; ++h) X[(2 * lr + h) * ld + row] -= s0[h] + s1[h];
    __syncwarp();
    const int ca = 8 * I + lr, cb = ca + 4;
    const double a0 = (ca < k && row <= ca) ? Rp[up_off(ca) + row] : 0.0;
    const double a1 = (cb < k && row <= cb) ? Rp[up_off(cb) + row] : 0.0;
    double y[2] = {0.0, 0.0};
    dmma(y, a0, X[lc * ld + ca]);
    dmma(y, a1, X[lc * ld + cb]);
    __syncwarp();
#pragma unroll
    for (int h = 0; h < 2; ++h) X[(2 * lr + h) * ld + row] = y[h];
    __syncwarp();
  }
  for (int c = 0; c < nc; ++c)
    for (int i = lane; i < k; i += 32) B[(int64_t)(c0 + c) * ldb + i] = X[c * ld + i];
}

// Cholesky G = L L^T of the symmetric positive definite G (column-major k x k,
// lower triangle read), R = L^T (upper, column-major, zeros below the
// diagonal). One CTA, the lower triangle packed in shared memory, in panels of
// eight columns: every thread that owns a row factors the panel's 8 x 8
// diagonal block in registers for itself (no barrier per column), solves its
// row against it, and then all warps subtract the panel's rank-8 product from
// the trailing triangle, four columns at a time with their 32 panel values in
// registers. Two barriers per panel; bound by the chain of 8 reciprocal square
// roots per panel and the FP64 FMAs of the update (k = 201: 128 us, and
// 35 us for the inverse by tri_solve_kernel; one column at a time with a barrier
// each, and the inverse column by column in the same CTA, took 690). INV (k up to
// kCholInvMaxK): Rinv, the inverse of R, from the first warp, lane c column c
// of L^-1 by forward substitution in registers, which for a small k is shorter
// than a launch of tri_solve_kernel (k = 9, 300 x 300: the approximation's
// eight factorisations took 30 us longer). Rinv may be G. status[0] = 0, or j + 1
// when the j-th pivot is not positive (R and Rinv are then not written).
constexpr int kCholThreads = 512, kCholInvMaxK = 32;
template <bool INV>
__global__ void __launch_bounds__(kCholThreads) chol_factor_kernel(const double* G, int k, double* R, double* Rinv,
                                                                   int* status) {
  extern __shared__ double cf_smem[];
  double* L = cf_smem;
  __shared__ int bad;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  if (threadIdx.x == 0) bad = 0;
#pragma unroll 4
  for (int j = warp; j < k; j += kCholThreads / 32)
#pragma unroll
    for (int v = 0; v < 8; ++v) {  // k <= 225 rows
      const int i = lane + 32 * v;
      if (i >= j && i < k) L[lo_off(j, k) + i - j] = G[i + j * k];
    }
  __syncthreads();
  for (int j0 = 0; j0 < k; j0 += 8) {
    const int nb = min(8, k - j0);
    const int i = j0 + threadIdx.x;  // this thread's row
    double x[8];
    if (i < k) {
      // the diagonal block, a pad of the identity past k
      double d[8][8], inv[8];
#pragma unroll
      for (int c = 0; c < 8; ++c)
#pragma unroll
        for (int e = c; e < 8; ++e)
          d[e][c] = (e < nb && c < nb) ? L[lo_off(j0 + c, k) + e - c] : (e == c ? 1.0 : 0.0);
#pragma unroll
      for (int c = 0; c < 8; ++c) x[c] = (c < nb && i >= j0 + c) ? L[lo_off(j0 + c, k) + i - j0 - c] : 0.0;
      int wrong = 0;
#pragma unroll
      for (int c = 0; c < 8; ++c) {
        double p = d[c][c];
        if (!(p > 0.0)) {
          if (!wrong) wrong = j0 + c + 1;
          p = 1.0;
        }
        inv[c] = rsqrt(p);
        d[c][c] = p * inv[c];
#pragma unroll
        for (int e = c + 1; e < 8; ++e) d[e][c] *= inv[c];
#pragma unroll
        for (int f = c + 1; f < 8; ++f)
#pragma unroll
          for (int e = f; e < 8; ++e) d[e][f] = fma(-d[e][c], d[f][c], d[e][f]);
      }
      if (wrong && threadIdx.x == 0) bad = wrong;
      if (threadIdx.x < 8) {
        // a row of the diagonal block
#pragma unroll
        for (int e = 0; e < 8; ++e)
          if (e == (int)threadIdx.x) {
#pragma unroll
            for (int c = 0; c < 8; ++c) x[c] = c <= e ? d[e][c] : 0.0;
          }
      } else {
#pragma unroll
        for (int c = 0; c < 8; ++c) {
#pragma unroll
          for (int e = 0; e < c; ++e) x[c] = fma(-x[e], d[c][e], x[c]);
          x[c] *= inv[c];
        }
      }
    }
    __syncthreads();  // every thread has read the panel
    if (bad) break;
    if (i < k) {
#pragma unroll
      for (int c = 0; c < 8; ++c)
        if (c < nb && i >= j0 + c) L[lo_off(j0 + c, k) + i - j0 - c] = x[c];
    }
    __syncthreads();
    const double* pc[8];  // pc[c][a] = L(a, j0 + c)
#pragma unroll
    for (int c = 0; c < 8; ++c) pc[c] = L + lo_off(j0 + c, k) - (j0 + c);
    // nb < 8 only in the last panel, which has no trailing columns
    for (int b0 = j0 + 8 + 4 * warp; b0 < k; b0 += 4 * (kCholThreads / 32)) {
      double lb[4][8];
#pragma unroll
      for (int q = 0; q < 4; ++q)
#pragma unroll
        for (int c = 0; c < 8; ++c) lb[q][c] = b0 + q < k ? pc[c][b0 + q] : 0.0;
      for (int a = b0 + lane; a < k; a += 32) {
        double la[8];
#pragma unroll
        for (int c = 0; c < 8; ++c) la[c] = pc[c][a];
#pragma unroll
        for (int q = 0; q < 4; ++q) {
          if (b0 + q >= k || a < b0 + q) continue;
          double* g = L + lo_off(b0 + q, k) + a - b0 - q;
          double v = *g;
#pragma unroll
          for (int c = 0; c < 8; ++c) v = fma(-la[c], lb[q][c], v);
          *g = v;
        }
      }
    }
    __syncthreads();
  }
  if (bad) {
    if (threadIdx.x == 0) status[0] = bad;
    return;
  }
  for (int j = warp; j < k; j += kCholThreads / 32)
#pragma unroll
    for (int v = 0; v < 8; ++v) {
      const int i = lane + 32 * v;
      if (i < k) R[i + j * k] = (i <= j) ? L[lo_off(i, k) + j - i] : 0.0;
    }
  if (threadIdx.x == 0) status[0] = 0;
  if (!INV || warp != 0) return;
  const double inv = lane < k ? 1.0 / L[lo_off(lane, k)] : 0.0;
  double x[kCholInvMaxK];
#pragma unroll
  for (int i = 0; i < kCholInvMaxK; ++i) x[i] = i == lane ? 1.0 : 0.0;
#pragma unroll
  for (int l = 0; l < kCholInvMaxK; ++l) {
    if (l >= k) break;
    x[l] *= __shfl_sync(0xffffffffu, inv, l);
    const double* c = L + lo_off(l, k) - l;
#pragma unroll
    for (int i = l + 1; i < kCholInvMaxK; ++i)
      if (i < k) x[i] = fma(-c[i], x[l], x[i]);
  }
  if (lane < k)
#pragma unroll
    for (int i = 0; i < kCholInvMaxK; ++i)
      if (i < k) Rinv[lane + i * k] = x[i];
}

// D = S^T for column-major k x k matrices.
__global__ void dtranspose_kernel(const double* __restrict__ S, double* __restrict__ D, int64_t k) {
  for (int64_t q = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; q < k * k;
       q += (int64_t)gridDim.x * blockDim.x) {
    const int64_t i = q % k, j = q / k;
    D[i + j * k] = S[j + i * k];
  }
}

__global__ void identity_kernel(double* I, int64_t k) {
  for (int64_t q = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; q < k * k;
       q += (int64_t)gridDim.x * blockDim.x)
    I[q] = (q % k == q / k) ? 1.0 : 0.0;
}

// G(j, j) += shift
__global__ void shift_diag_kernel(double* G, int64_t k, const double* fro2, double factor) {
  const int64_t j = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (j < k) G[j + j * k] += factor * fro2[0];
}

__global__ void trace_kernel(const double* G, int64_t k, double* out) {
  __shared__ double red[256];
  double s = 0.0;
  for (int64_t j = threadIdx.x; j < k; j += blockDim.x) s += G[j + j * k];
  red[threadIdx.x] = s;
  __syncthreads();
  for (int st = 128; st > 0; st >>= 1) {
    if (threadIdx.x < st) red[threadIdx.x] += red[threadIdx.x + st];
    __syncthreads();
  }
  if (threadIdx.x == 0) out[0] = red[0];
}

// --------------------------------------------------- sparse-sign maps ------
// out(r, :) = sum_t sign_rt Q(c_rt, :) for a row-sparse map (R x m, zeta per
// row); Q is m x k column-major (ldq), out R x k column-major (ldo).
__global__ void rowsparse_apply_kernel(const uint32_t* __restrict__ mp, int zeta, int64_t R,
                                       const double* __restrict__ Q, int64_t ldq, int64_t k,
                                       double* __restrict__ out, int64_t ldo, int64_t q0, int64_t qrows) {
  // Q holds rows [q0, q0 + qrows) of the operand; map entries elsewhere
  // belong to other row blocks
  for (int64_t q = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; q < R * k;
       q += (int64_t)gridDim.x * blockDim.x) {
    const int64_t r = q % R, j = q / R;
    double a = 0.0;
    for (int t = 0; t < zeta; ++t) {
      const uint32_t w = mp[r * zeta + t];
      const int64_t row = (int64_t)(w & 0x7fffffffu) - q0;
      if ((uint64_t)row >= (uint64_t)qrows) continue;
      const double v = Q[row + j * ldq];
      a += (w >> 31) ? -v : v;
    }
    out[r + j * ldo] = a;
  }
}

// out(c_jt, :) += sign_jt P(j, :) for a stored-transposed map (n rows, zeta
// entries over R columns); out is R x k column-major, zeroed by the caller.
__global__ void colsparse_apply_kernel(const uint32_t* __restrict__ mp, int zeta, int64_t n,
                                       const double* __restrict__ P, int64_t ldp, int64_t k,
                                       double* __restrict__ out, int64_t ldo) {
  for (int64_t q = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; q < n * k;
       q += (int64_t)gridDim.x * blockDim.x) {
    const int64_t j = q % n, col = q / n;
    const double v = P[j + col * ldp];
    for (int t = 0; t < zeta; ++t) {
      const uint32_t w = mp[j * zeta + t];
      atomicAdd(out + (int64_t)(w & 0x7fffffffu) + col * ldo, (w >> 31) ? -v : v);
    }
  }
}

// The same product with a private copy of out per CTA in shared memory: the
// CTA's stored rows add into it with shared-memory atomics (few collisions:
// out has R x k entries), then each entry goes to out with one global atomic
// per CTA. Used when out fits in shared memory; the kernel above turns every
// map entry into a global atomic on out's few entries.
__global__ void colsparse_apply_smem_kernel(const uint32_t* __restrict__ mp, int zeta, int64_t n,
                                            const double* __restrict__ P, int64_t ldp, int64_t k,
                                            double* __restrict__ out, int64_t ldo, int64_t R) {
  extern __shared__ double priv[];  // R x k, column-major (ld R)
  for (int64_t q = threadIdx.x; q < R * k; q += blockDim.x) priv[q] = 0.0;
  __syncthreads();
  const int64_t per = (n + gridDim.x - 1) / gridDim.x;
  const int64_t j0 = (int64_t)blockIdx.x * per, j1 = min(n, j0 + per);
  const int64_t span = j1 > j0 ? j1 - j0 : 0;
  for (int64_t q = threadIdx.x; q < span * k; q += blockDim.x) {
    const int64_t j = j0 + q % span, col = q / span;  // consecutive threads: consecutive rows j
    const double v = P[j + col * ldp];
    for (int t = 0; t < zeta; ++t) {
      const uint32_t w = mp[j * zeta + t];
      atomicAdd(priv + (int64_t)(w & 0x7fffffffu) + col * R, (w >> 31) ? -v : v);
    }
  }
  __syncthreads();
  for (int64_t q = threadIdx.x; q < R * k; q += blockDim.x) {
    const double a = priv[q];
    if (a != 0.0) atomicAdd(out + (q % R) + (q / R) * ldo, a);
  }
}

// ------------------------------------------------------ Jacobi SVD ---------
// The rotation of a pair of columns with squared norms al, be and product ga:
// tan of the angle is the smaller root of t^2 + 2 zeta t - 1 with zeta = d / h,
// d = beta - alpha, h = 2 gamma, t = sign(d) h / (|d| + sqrt(d^2 + h^2)). It is
// on the chain that every round waits for, and a dependent FP64 operation takes
// 9 cycles with up to four warps on the SM, 13 with 16 and 25 with 32 (a square
// root or a division many of them), so (c0, s0) comes from FP32 (d and h scaled by
// a power of two) and one Newton step corrects it in FP64: the rotated product is
//   F = (c0^2 - s0^2) h / 2 - c0 s0 d,  delta = F / (sign(d) sqrt(d^2 + h^2)),
// the angle moves by delta (1e-7, so its square is FP64 rounding) and the pair
// is normalised by 1 - e / 2 + 3 e^2 / 8 - delta^2 / 2, e = c0^2 + s0^2 - 1, which
// needs neither the corrected values nor a square root. cs^2 + sn^2 is one to
// 4e-16, as by FP64 square roots; the product falls to 1e-12 of itself or less
// (3e-15 by them), and the next sweep, which there is unless every pair is within
// tol, sees the rest. False: the pair is orthogonal to tol and stays.
__device__ __forceinline__ bool jacobi_angle(double al, double be, double ga, double tol2, double& cs, double& sn) {
  cs = 1.0, sn = 0.0;
  if (ga == 0.0 || ga * ga <= tol2 * (al * be)) return false;
  double d = be - al, h = ga + ga;
  const int e = max(__double2hiint(d) & 0x7ff00000, __double2hiint(h) & 0x7ff00000);
  const double sc = __hiloint2double(0x7fe00000 - e, 0);  // 2^-exponent, a normal number
  d *= sc;
  h *= sc;
  const float df = (float)d, hf = (float)h;
  const float w2 = fmaf(df, df, hf * hf), rw = rsqrtf(w2);  // w2 is at least 1
  const float sg = df < 0.f ? -1.f : 1.f;
  const float t = sg * __fdividef(hf, fabsf(df) + w2 * rw);
  const float cf = rsqrtf(fmaf(t, t, 1.f));
  const double c0 = (double)cf, s0 = (double)(cf * t), rwd = (double)(sg * rw);
  const double cc = c0 * c0, ss = s0 * s0;
  const double delta = fma(0.5 * h, cc - ss, -(d * (c0 * s0))) * rwd;
  const double eps = (cc - 1.0) + ss;
  const double f0 = fma(fma(0.375, eps, -0.5), eps, 1.0), c1 = c0 * f0, s1 = s0 * f0;
  const double hd = -0.5 * delta;
  cs = fma(delta, fma(hd, c1, -s1), c1);
  sn = fma(delta, fma(hd, s1, c1), s1);
  return true;
}

// Players p < q of pair pr in a round of a round-robin among np (even) players:
// the last stays, the others rotate.
__device__ __forceinline__ void robin_pair(int np, int round, int pr, int& p, int& q) {
  if (pr == 0) {
    p = round;
    q = np - 1;
    return;
  }
  p = round + pr;
  if (p >= np - 1) p -= np - 1;
  q = round - pr;
  if (q < 0) q += np - 1;
}

// One-sided Jacobi on the column-major k x k A (overwritten by A V = U S),
// V accumulated (column-major k x k), k <= 114. A cluster of two CTAs: CTA 0
// holds A in shared memory and rotates the pairs of each round of a round-robin,
// a half-warp per pair with the pair's columns in registers (EPL values of each
// per lane), writing every (cs, sn) of the sweep to rot; CTA 1 holds V and
// applies the sweep before, rows along the threads and the round's pairs over
// groups of threads. So a round is one read and one write of A, its dot products
// and one angle; V's traffic and FP64 work (as much again) are off that chain. A
// sweep without a rotation (every pair within tol of orthogonal) ends the loop.
// rot: two buffers of (kp - 1) (kp / 2) double2, kp = k rounded up to even, and
// two flags after them. k = 81, 11 sweeps: 1.18 ms (2,500 cycles a round: the
// chain of dependent FP64 operations and 1,000 cycles of shared memory); one CTA
// with A and V took 1.80.
constexpr int kJacMaxK = 114;
constexpr size_t kJacRotBytes = sizeof(double2) * 2 * (kJacMaxK - 1) * (kJacMaxK / 2) + 16;

template <int EPL>
__global__ void __launch_bounds__(EPL == 8 ? 960 : 128 * EPL)
    jacobi_svd_kernel(double* __restrict__ Ag, double* __restrict__ Vg, int k, int max_sweeps, double tol, double2* rot,
                      int* sweeps_out) {
  namespace cg = cooperative_groups;
  cg::cluster_group cl = cg::this_cluster();
  extern __shared__ __align__(16) double jac_smem[];
  __shared__ int any;
  const int kp = (k + 1) & ~1, npair = kp / 2, nrot = (kp - 1) * npair;
  volatile int* flags = reinterpret_cast<int*>(rot + 2 * nrot);
  const bool is_v = cl.block_rank() == 1;
  double* M = jac_smem;  // A or V
  for (int q = threadIdx.x; q < k * k; q += blockDim.x) M[q] = is_v ? ((q % k == q / k) ? 1.0 : 0.0) : Ag[q];
  double2* rs = reinterpret_cast<double2*>(jac_smem + ((size_t)k * k + 1) / 2 * 2);  // CTA 1: a sweep's rotations
  __syncthreads();
  const int hl = threadIdx.x & 15, pr = threadIdx.x >> 4;
  const unsigned hmask = (threadIdx.x & 16) ? 0xffff0000u : 0x0000ffffu;
  const double tol2 = tol * tol;
  // rows of V along the threads, the pairs of a round over the groups of rows
  const int rk = (k + 31) & ~31, grp = threadIdx.x / rk, ngrp = blockDim.x / rk, row = threadIdx.x - grp * rk;
  auto apply_v = [&](const double2* src) {
    for (int q = threadIdx.x; q < nrot; q += blockDim.x) rs[q] = __ldcg(src + q);
    __syncthreads();
    for (int round = 0; round < kp - 1; ++round) {
      if (grp < ngrp && row < k)
        for (int g = grp; g < npair; g += 2 * ngrp) {
          int p[2], q[2];
          double x[2], y[2];
          double2 r[2];
#pragma unroll
          for (int u = 0; u < 2; ++u) {
            const int pp = min(g + u * ngrp, npair - 1);
            robin_pair(kp, round, pp, p[u], q[u]);
            if (p[u] > q[u]) {
              const int t = p[u];
              p[u] = q[u];
              q[u] = t;
            }
            if (g + u * ngrp >= npair || q[u] >= k) p[u] = -1;
            if (p[u] >= 0) x[u] = M[p[u] * k + row], y[u] = M[q[u] * k + row], r[u] = rs[round * npair + pp];
          }
#pragma unroll
          for (int u = 0; u < 2; ++u)
            if (p[u] >= 0) {
              M[p[u] * k + row] = r[u].x * x[u] - r[u].y * y[u];
              M[q[u] * k + row] = r[u].y * x[u] + r[u].x * y[u];
            }
        }
      __syncthreads();
    }
  };
  int sweep = 0;
  bool more = true;
  for (; sweep < max_sweeps; ++sweep) {
    if (!is_v) {
      if (threadIdx.x == 0) any = 0;
      __syncthreads();
      double2* out = rot + (sweep & 1) * nrot;
      for (int round = 0; round < kp - 1; ++round) {
        int p, q;
        robin_pair(kp, round, min(pr, npair - 1), p, q);
        if (p > q) {
          const int t = p;
          p = q;
          q = t;
        }
        if (pr < npair && q < k) {  // q == k: a bye
          double* ap = M + p * k;
          double* aq = M + q * k;
          // two sums of each product: the chains of dependent FMAs are half as long
          double x[EPL], y[EPL], sa[2] = {0.0, 0.0}, sb[2] = {0.0, 0.0}, sg[2] = {0.0, 0.0};
#pragma unroll
          for (int e = 0; e < EPL; ++e) {
            const int i = hl + 16 * e;
            x[e] = i < k ? ap[i] : 0.0;
            y[e] = i < k ? aq[i] : 0.0;
          }
#pragma unroll
          for (int e = 0; e < EPL; ++e) {
            sa[e & 1] = fma(x[e], x[e], sa[e & 1]);
            sb[e & 1] = fma(y[e], y[e], sb[e & 1]);
            sg[e & 1] = fma(x[e], y[e], sg[e & 1]);
          }
          // lanes 0-7 of the half-warp go on with al and ga, lanes 8-15 with be:
          // fewer FP64 additions than three full butterflies
          double al = sa[0] + sa[1], be = sb[0] + sb[1], ga = sg[0] + sg[1];
          const bool up = hl & 8;
          double n1 = (up ? be : al) + __shfl_xor_sync(hmask, up ? al : be, 8);
          ga += __shfl_xor_sync(hmask, ga, 8);
          // then lanes 4-7 (mod 8) take ga, the others the norm
          const bool up2 = hl & 4;
          double n2 = (up2 ? ga : n1) + __shfl_xor_sync(hmask, up2 ? n1 : ga, 4);
#pragma unroll
          for (int o = 2; o > 0; o >>= 1) n2 += __shfl_xor_sync(hmask, n2, o);
          const int l0 = threadIdx.x & 16;
          al = __shfl_sync(hmask, n2, l0);
          ga = __shfl_sync(hmask, n2, l0 + 4);
          be = __shfl_sync(hmask, n2, l0 + 8);
          double cs, sn;
          if (jacobi_angle(al, be, ga, tol2, cs, sn)) {
            if (hl == 0) any = 1;
#pragma unroll
            for (int e = 0; e < EPL; ++e) {
              const int i = hl + 16 * e;
              if (i < k) {
                ap[i] = cs * x[e] - sn * y[e];
                aq[i] = sn * x[e] + cs * y[e];
              }
            }
          }
          if (hl == 0) __stcg(out + round * npair + pr, make_double2(cs, sn));
        }
        __syncthreads();
      }
      if (threadIdx.x == 0) flags[sweep & 1] = any;
    } else if (sweep > 0) {
      apply_v(rot + ((sweep - 1) & 1) * nrot);
    }
    cl.sync();  // releases the sweep's rotations and flag to CTA 1
    more = flags[sweep & 1] != 0;
    if (!more) break;
  }
  // CTA 1 is one sweep behind; a sweep without rotations leaves nothing to do
  if (is_v && more && sweep > 0) apply_v(rot + ((sweep - 1) & 1) * nrot);
  if (!is_v && threadIdx.x == 0) sweeps_out[0] = sweep;
  __syncthreads();
  double* out = is_v ? Vg : Ag;
  for (int q = threadIdx.x; q < k * k; q += blockDim.x) out[q] = M[q];
}

// Block one-sided Jacobi, 114 < k <= 256: the columns are cut into nb blocks of
// eight, an outer round pairs the blocks round-robin and a CTA takes a pair of
// blocks (16 columns); nb / 2 CTAs form one cluster and meet at its barrier
// after every round, so all sweeps are one launch. Per round a CTA forms the
// Gram matrix of its 16 columns (FP64 tensor cores), runs one inner sweep of
// rotations on it (the two-sided update of 16 x 16 values, one barrier per inner
// round, no pass over the columns), and multiplies its columns of A and V by the
// accumulated 16 x 16 rotation. The Gram matrix is formed afresh in every
// round, so what its updates lose early is corrected later, and a round without
// rotations leaves the columns as they are; sweeps go on until one makes none.
// k = 201, 13 sweeps: 4.0 ms, four fifths of it the chain of angles (about 1,000
// cycles per inner round). With every rotation passing over the columns and a
// launch per round it took 10.
constexpr int kJacClusterMaxK = 256;
__global__ void __launch_bounds__(256, 1) jacobi_cluster_kernel(double* Ag, double* Vg, int k, int nb, int max_sweeps,
                                                             double tol, int* sweeps_out) {
  namespace cg = cooperative_groups;
  cg::cluster_group cl = cg::this_cluster();
  constexpr int P = 16, LG = 17;
  extern __shared__ __align__(16) double jc_smem[];
  __shared__ double G[2][P * LG], J[2][P * LG], part[8][3][64];
  __shared__ int any_round, any_sweep;
  const int ld = tri_ld(k);
  double* Ac = jc_smem;           // column c at Ac + c * ld, rows past k zero
  double* Vc = jc_smem + P * ld;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, lr = lane & 3, lc = lane >> 2;
  const int kr = (k + 7) & ~7;  // rows in whole MMA blocks
  const double tol2 = tol * tol;
  int sweep = 0;
  for (; sweep < max_sweeps; ++sweep) {
    if (tid == 0) any_sweep = 0;
    for (int round = 0; round < nb - 1; ++round) {
      int bi, bj;
      robin_pair(nb, round, (int)blockIdx.x, bi, bj);
      auto gcol = [&](int c) { return c < 8 ? bi * 8 + c : bj * 8 + (c - 8); };
      for (int c = warp; c < P; c += 8) {
        const int g = gcol(c);
        double x[8], y[8];  // k <= 256: a column of each in flight
#pragma unroll
        for (int v = 0; v < 8; ++v) {
          const int i = lane + 32 * v;
          const bool in = g < k && i < k;
          x[v] = in ? __ldcg(Ag + (size_t)g * k + i) : 0.0;
          y[v] = in ? __ldcg(Vg + (size_t)g * k + i) : 0.0;
        }
#pragma unroll
        for (int v = 0; v < 8; ++v) {
          const int i = lane + 32 * v;
          if (i < kr) Ac[c * ld + i] = x[v], Vc[c * ld + i] = y[v];
        }
      }
      if (tid == 0) any_round = 0;
      __syncthreads();
      {  // Gram matrix: a warp per K steps of four rows, then a sum in warp order
        double s00[2] = {0.0, 0.0}, s01[2] = {0.0, 0.0}, s11[2] = {0.0, 0.0};
        for (int r = 4 * warp; r < kr; r += 32) {
          const double a0 = Ac[lc * ld + r + lr], a1 = Ac[(8 + lc) * ld + r + lr];
          dmma(s00, a0, a0);
          dmma(s01, a0, a1);
          dmma(s11, a1, a1);
        }
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          const int e = lc * 8 + 2 * lr + h;
          part[warp][0][e] = s00[h];
          part[warp][1][e] = s01[h];
          part[warp][2][e] = s11[h];
        }
      }
      __syncthreads();
      if (tid < 192) {
        const int blk = tid >> 6, e = tid & 63, i = e >> 3, j = e & 7;
        double v = 0.0;
#pragma unroll
        for (int w = 0; w < 8; ++w) v += part[w][blk][e];
        if (blk == 0) {
          G[0][i * LG + j] = v;
        } else if (blk == 1) {
          G[0][i * LG + 8 + j] = v;
          G[0][(8 + j) * LG + i] = v;
        } else {
          G[0][(8 + i) * LG + 8 + j] = v;
        }
      }
      J[0][(tid >> 4) * LG + (tid & 15)] = (tid >> 4) == (tid & 15) ? 1.0 : 0.0;
      __syncthreads();
      int cur = 0;
      for (int r = 0; r < P - 1; ++r, cur ^= 1) {
        // threads 0-63: the 2 x 2 block of pairs (a, b); 64-191: row i of J in
        // pair b. Each works out the angles that it needs.
        const double* Gc = G[cur];
        if (tid < 192) {
          const int b = tid & 7;
          int p2, q2;
          robin_pair(P, r, b, p2, q2);
          double c2, s2;
          const bool rot =
              jacobi_angle(Gc[p2 * LG + p2], Gc[q2 * LG + q2], Gc[p2 * LG + q2], tol2, c2, s2);
          if (tid < 64) {
            int p1, q1;
            robin_pair(P, r, tid >> 3, p1, q1);
            double c1, s1;
            jacobi_angle(Gc[p1 * LG + p1], Gc[q1 * LG + q1], Gc[p1 * LG + q1], tol2, c1, s1);
            const double pp = Gc[p1 * LG + p2], pq = Gc[p1 * LG + q2], qp = Gc[q1 * LG + p2], qq = Gc[q1 * LG + q2];
            const double rp = c1 * pp - s1 * qp, rq = c1 * pq - s1 * qq;
            const double tp = s1 * pp + c1 * qp, tq = s1 * pq + c1 * qq;
            double* Gn = G[cur ^ 1];
            Gn[p1 * LG + p2] = c2 * rp - s2 * rq;
            Gn[p1 * LG + q2] = s2 * rp + c2 * rq;
            Gn[q1 * LG + p2] = c2 * tp - s2 * tq;
            Gn[q1 * LG + q2] = s2 * tp + c2 * tq;
            if (rot) any_round = 1;
          } else {
            const int i = (tid - 64) >> 3;
            const double x = J[cur][i * LG + p2], y = J[cur][i * LG + q2];
            J[cur ^ 1][i * LG + p2] = c2 * x - s2 * y;
            J[cur ^ 1][i * LG + q2] = s2 * x + c2 * y;
          }
        }
        __syncthreads();
      }
      if (any_round) {
        if (tid == 0) any_sweep = 1;
        const double* Jc = J[cur];
        double jb[4][2];
#pragma unroll
        for (int t = 0; t < 4; ++t)
#pragma unroll
          for (int n = 0; n < 2; ++n) jb[t][n] = Jc[(4 * t + lr) * LG + 8 * n + lc];
        for (int w = warp; w < kr / 4; w += 8) {  // row blocks of A, then of V
          const bool v = w >= kr / 8;
          const int row = 8 * (v ? w - kr / 8 : w) + lc;
          const double* S = v ? Vc : Ac;
          double* D = v ? Vg : Ag;
          double o[2][2] = {{0.0, 0.0}, {0.0, 0.0}};
#pragma unroll
          for (int t = 0; t < 4; ++t) {
            const double a = S[(4 * t + lr) * ld + row];
            dmma(o[0], a, jb[t][0]);
            dmma(o[1], a, jb[t][1]);
          }
          if (row < k) {
#pragma unroll
            for (int n = 0; n < 2; ++n)
#pragma unroll
              for (int h = 0; h < 2; ++h) {
                const int g = gcol(8 * n + 2 * lr + h);
                if (g < k) __stcg(D + (size_t)g * k + row, o[n][h]);
              }
          }
        }
      }
      cl.sync();  // the round's columns are in place for the next round's CTAs
    }
    bool more = false;
    for (unsigned b = 0; b < cl.num_blocks(); ++b) more |= *cl.map_shared_rank(&any_sweep, b) != 0;
    cl.sync();  // every CTA has read every flag
    if (!more) break;
  }
  if (blockIdx.x == 0 && tid == 0) sweeps_out[0] = sweep;
}

// Block one-sided Jacobi for k above the cluster form, or where the device has
// no room for its cluster: one launch per outer round. The columns are cut into
// nb blocks of bs (the last ones short or empty). An outer round pairs the blocks round-robin; each CTA takes one
// pair (I, J), copies the up to 2 bs columns of A and V into shared memory,
// runs one inner sweep of the one-sided Jacobi rotations over all pairs of
// those columns (a half-warp per pair, as in jacobi_svd_kernel), and
// writes them back. rotated[0] is set when any rotation was made. nb - 1
// outer rounds make an outer sweep, after which every pair of columns has
// met; sweeps continue until one makes no rotation.
__global__ void __launch_bounds__(1024) jacobi_block_kernel(double* __restrict__ Ag, double* __restrict__ Vg, int k,
                                                            int bs, int nb, int round, double tol,
                                                            int* __restrict__ rotated) {
  extern __shared__ double jb_smem[];
  __shared__ int any;
  // this CTA's pair of blocks in the round-robin round
  const int pr = blockIdx.x;
  int bi, bj;
  if (pr == 0) {
    bi = round;
    bj = nb - 1;
  } else {
    bi = round + pr;
    if (bi >= nb - 1) bi -= nb - 1;
    bj = round - pr;
    if (bj < 0) bj += nb - 1;
  }
  // local column c < 2 bs: block bi's columns, then block bj's
  auto gcol = [&](int c) { return c < bs ? bi * bs + c : bj * bs + (c - bs); };
  double* A = jb_smem;                       // 2 bs columns of length k
  double* V = jb_smem + (size_t)2 * bs * k;  // same for V
  for (int q = threadIdx.x; q < 2 * bs * k; q += blockDim.x) {
    const int c = q / k, i = q - c * k, g = gcol(c);
    const bool in = g < k;
    A[q] = in ? Ag[(size_t)g * k + i] : 0.0;
    V[q] = in ? Vg[(size_t)g * k + i] : 0.0;
  }
  if (threadIdx.x == 0) any = 0;
  __syncthreads();
  const int hl = threadIdx.x & 15, slot = threadIdx.x >> 4, nslot = blockDim.x >> 4;
  const unsigned hmask = (threadIdx.x & 16) ? 0xffff0000u : 0x0000ffffu;
  const int np = 2 * bs;  // even number of local players
  for (int r = 0; r < np - 1; ++r) {
    for (int pp = slot; pp < np / 2; pp += nslot) {
      int p, q;
      if (pp == 0) {
        p = r;
        q = np - 1;
      } else {
        p = r + pp;
        if (p >= np - 1) p -= np - 1;
        q = r - pp;
        if (q < 0) q += np - 1;
      }
      if (gcol(p) >= k || gcol(q) >= k) continue;  // an absent column
      double* ap = A + (size_t)p * k;
      double* aq = A + (size_t)q * k;
      double al = 0.0, be = 0.0, ga = 0.0;
      for (int i = hl; i < k; i += 16) {
        const double x = ap[i], y = aq[i];
        al = fma(x, x, al);
        be = fma(y, y, be);
        ga = fma(x, y, ga);
      }
#pragma unroll
      for (int o = 8; o > 0; o >>= 1) {
        al += __shfl_xor_sync(hmask, al, o);
        be += __shfl_xor_sync(hmask, be, o);
        ga += __shfl_xor_sync(hmask, ga, o);
      }
      if (ga == 0.0 || ga * ga <= (tol * tol) * (al * be)) continue;
      if (hl == 0) any = 1;
      const double d = be - al, h = 2.0 * ga;
      const double t = (d >= 0.0 ? h : -h) / (fabs(d) + sqrt(fma(d, d, h * h)));
      const double cs = rsqrt(fma(t, t, 1.0)), sn = cs * t;
      for (int i = hl; i < k; i += 16) {
        const double x = ap[i], y = aq[i];
        ap[i] = cs * x - sn * y;
        aq[i] = sn * x + cs * y;
      }
      double* vp = V + (size_t)p * k;
      double* vq = V + (size_t)q * k;
      for (int i = hl; i < k; i += 16) {
        const double x = vp[i], y = vq[i];
        vp[i] = cs * x - sn * y;
        vq[i] = sn * x + cs * y;
      }
    }
    __syncthreads();
  }
  for (int q = threadIdx.x; q < 2 * bs * k; q += blockDim.x) {
    const int c = q / k, i = q - c * k, g = gcol(c);
    if (g < k) {
      Ag[(size_t)g * k + i] = A[q];
      Vg[(size_t)g * k + i] = V[q];
    }
  }
  if (threadIdx.x == 0 && any) atomicExch(rotated, 1);
}

__global__ void store_int_kernel(int* dst, int v) { *dst = v; }

// One-sided Jacobi by jacobi_block_kernel: block sweeps driven
// from the host, each outer sweep's rotation flag read back once.
void jacobi_svd_blocked(skema_ctx* c, double* A, double* V, int64_t k, int max_sweeps, double tol,
                        int* sweeps_out) {
  // columns per block: 8, or fewer where two blocks of A and V would not fit
  // about 200 KB. Small blocks put more CTAs on each round (nb / 2) for the
  // same pairs per outer sweep: at k = 201, 8 columns (13 CTAs a round) took
  // 10.5 ms against 15.1 ms for 31 columns (4 CTAs), 12 and 16 about 11.2 ms,
  // 6 and 4 11.1 and 11.8 ms.
  const int bs = (int)std::max<int64_t>(
      2, std::min<int64_t>(8, (200 * 1024) / (4 * (int64_t)sizeof(double) * k)));
  int nb = (int)((k + bs - 1) / bs);
  nb += nb & 1;  // an even number of players
  const size_t smem = sizeof(double) * (size_t)(4 * bs * k);
  SKEMA_CUDA(cudaFuncSetAttribute(jacobi_block_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
  identity_kernel<<<(unsigned)std::min<int64_t>((k * k + 255) / 256, 4096), 256, 0, c->stream>>>(V, k);
  SKEMA_LAUNCHED(c);
  int* flag = sweeps_out + 2;  // the caller's status block has room after the sweep count
  int sweep = 0;
  for (; sweep < max_sweeps; ++sweep) {
    SKEMA_CUDA(cudaMemsetAsync(flag, 0, sizeof(int), c->stream));
    for (int r = 0; r < nb - 1; ++r) {
      jacobi_block_kernel<<<nb / 2, 1024, smem, c->stream>>>(A, V, (int)k, bs, nb, r, tol, flag);
      SKEMA_LAUNCHED(c);
    }
    int h = 0;
    SKEMA_CUDA(cudaMemcpyAsync(&h, flag, sizeof(int), cudaMemcpyDeviceToHost, c->stream));
    SKEMA_CUDA(cudaStreamSynchronize(c->stream));
    if (!h) break;
  }
  store_int_kernel<<<1, 1, 0, c->stream>>>(sweeps_out, sweep);
  SKEMA_LAUNCHED(c);
}

// One cluster of `ctas` CTAs; false when the device cannot place it.
template <typename Kern, typename... Args>
bool launch_one_cluster(skema_ctx* c, Kern kern, int ctas, int threads, size_t smem, Args... args) {
  SKEMA_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
  if (ctas > 8) SKEMA_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeNonPortableClusterSizeAllowed, 1));
  cudaLaunchAttribute at;
  at.id = cudaLaunchAttributeClusterDimension;
  at.val.clusterDim.x = ctas;
  at.val.clusterDim.y = at.val.clusterDim.z = 1;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(ctas);
  cfg.blockDim = dim3(threads);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = c->stream;
  cfg.attrs = &at;
  cfg.numAttrs = 1;
  int n = 0;
  if (cudaOccupancyMaxActiveClusters(&n, kern, &cfg) != cudaSuccess || n < 1) {
    (void)cudaGetLastError();
    return false;
  }
  SKEMA_CUDA(cudaLaunchKernelEx(&cfg, kern, args...));
  SKEMA_LAUNCHED(c);
  return true;
}

// The SVD kernel for a k x k problem: one pair of CTAs while A and V fit their
// shared memory, block sweeps in one cluster up to k = 256, else block sweeps
// driven from the host.
// st: the caller's status block of kStatusBytes; st[1] gets the sweeps, st[3] is
// the host-driven form's flag, and the rotations that the pair of CTAs exchanges
// follow at st + 64.
constexpr size_t kStatusBytes = 64 * sizeof(int) + kJacRotBytes;
void jacobi_svd(skema_ctx* c, double* A, double* V, int64_t k, int max_sweeps, double tol, int* st) {
  int* sweeps_out = st + 1;
  double2* rot = reinterpret_cast<double2*>(st + 64);
  if (k <= kJacMaxK) {
    const int kp = (int)((k + 1) & ~1);
    const size_t smem = sizeof(double) * ((size_t)(k * k + 1) / 2 * 2) + sizeof(double2) * (size_t)(kp - 1) * (kp / 2);
    const int threads = std::max(128, (kp / 2 * 16 + 31) / 32 * 32);
    auto go = [&](auto kern) {
      return launch_one_cluster(c, kern, 2, threads, smem, A, V, (int)k, max_sweeps, tol, rot, sweeps_out);
    };
    if (k <= 32   ? go(jacobi_svd_kernel<2>)
        : k <= 64 ? go(jacobi_svd_kernel<4>)
        : k <= 96 ? go(jacobi_svd_kernel<6>)
                  : go(jacobi_svd_kernel<8>))
      return;
  } else if (k <= kJacClusterMaxK) {
    const int nb = (int)((k + 15) / 16 * 2);
    const size_t smem = sizeof(double) * 2 * 16 * (size_t)tri_ld((int)k);
    identity_kernel<<<(unsigned)std::min<int64_t>((k * k + 255) / 256, 4096), 256, 0, c->stream>>>(V, k);
    SKEMA_LAUNCHED(c);
    if (launch_one_cluster(c, jacobi_cluster_kernel, nb / 2, 256, smem, A, V, (int)k, nb, max_sweeps, tol, sweeps_out))
      return;
  }
  jacobi_svd_blocked(c, A, V, k, max_sweeps, tol, sweeps_out);
}

// sigma_j = ||a_j||, ranks by descending sigma (ties by index), then
// U(:, rank) = a_j / sigma_j, Vout(:, rank) = v_j, S(rank) = sigma_j.
// One CTA, a warp per column (a thread per column walked k^2 values 8 k bytes
// apart: 108 us at k = 201).
constexpr int kFinishThreads = 1024;
__global__ void __launch_bounds__(kFinishThreads) svd_finish_kernel(const double* A, const double* V, int64_t k,
                                                                    double* U, double* Vout, double* S, double* sig) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  for (int64_t j = warp; j < k; j += kFinishThreads / 32) {
    double s = 0.0;
    for (int64_t i = lane; i < k; i += 32) s = fma(A[i + j * k], A[i + j * k], s);
    for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
    if (lane == 0) sig[j] = sqrt(s);
  }
  __syncthreads();
  for (int64_t j = warp; j < k; j += kFinishThreads / 32) {
    const double sj = sig[j];
    int rank = 0;
    for (int64_t l = lane; l < k; l += 32) rank += (sig[l] > sj || (sig[l] == sj && l < j)) ? 1 : 0;
    rank = __reduce_add_sync(0xffffffffu, rank);
    const double inv = sj > 0.0 ? 1.0 / sj : 0.0;
    if (lane == 0) S[rank] = sj;
    for (int64_t i = lane; i < k; i += 32) {
      U[i + rank * k] = A[i + j * k] * inv;
      Vout[i + rank * k] = V[i + j * k];
    }
  }
}

// ------------------------------------------------------------ helpers ------
// Buffers of one approximation call, carved from the context's workspace
// (grown once, then reused by every later call: no allocation per call).
class Carve {
 public:
  Carve(skema_ctx* c, std::initializer_list<size_t> bytes) {
    size_t total = 0;
    for (size_t b : bytes) total += round(b);
    base_ = static_cast<char*>(workspace(c, total));
    at_ = base_;
  }
  double* take(size_t bytes) {
    char* p = at_;
    at_ += round(bytes);
    return reinterpret_cast<double*>(p);
  }

 private:
  static size_t round(size_t b) { return (std::max<size_t>(b, 16) + 255) / 256 * 256; }
  char* base_;
  char* at_;
};

int g1(const skema_ctx* c, int64_t total) {
  return (int)std::max<int64_t>(1, std::min<int64_t>((total + 255) / 256, (int64_t)c->sm_count * 16));
}

// R X = B in place (identity: X = R^{-1}) for upper-triangular R (k x k) and
// B (k x nrhs, ld ldb): the packed shared-memory kernel when R fits, else one
// warp per right-hand side reading R from global memory.
void tri_solve(skema_ctx* c, const double* R, int64_t k, double* B, int64_t ldb, int64_t nrhs, bool identity,
               const int* status) {
  // up to four warps a CTA, as many as have room for their right-hand sides
  const size_t warp_bytes = sizeof(double) * 8 * (size_t)tri_ld((int)k);
  const size_t room = (226 * 1024 - packed_smem_bytes(k)) / warp_bytes;
  const int warps = (int)std::max<size_t>(1, std::min<size_t>({4, (size_t)(nrhs + 7) / 8, room}));
  const size_t smem = packed_smem_bytes(k) + warps * warp_bytes;
  SKEMA_CUDA(cudaFuncSetAttribute(tri_solve_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
  const int grid = (int)((nrhs + 8 * warps - 1) / (8 * warps));
  tri_solve_kernel<<<grid, kTriThreads, smem, c->stream>>>(R, (int)k, B, ldb, (int)nrhs, warps, identity ? 1 : 0,
                                                          status);
  SKEMA_LAUNCHED(c);
}
void trsm_upper(skema_ctx* c, const double* R, int64_t k, double* B, int64_t ldb, int64_t nrhs) {
  if (nrhs <= 0 || k <= 0) return;
  if (k <= kPackedMaxK) {
    tri_solve(c, R, k, B, ldb, nrhs, false, nullptr);
    return;
  }
  trsm_upper_kernel<<<(int)((nrhs * 32 + 255) / 256), 256, 0, c->stream>>>(R, k, B, ldb, nrhs);
  SKEMA_LAUNCHED(c);
}

// Cholesky G = L L^T of the k x k G with R = L^T and Rinv = R^{-1} (Rinv may
// alias G); st[0] as chol_factor_kernel sets it, read by the caller. G is
// consumed. When the factorisation fails R and Rinv hold no meaning.
void chol_inverse(skema_ctx* c, double* G, int64_t k, double* R, double* Rinv, int* st) {
  if (k <= kPackedMaxK) {
    const size_t smem = packed_smem_bytes(k);
    const bool small = k <= kCholInvMaxK;
    auto kern = small ? chol_factor_kernel<true> : chol_factor_kernel<false>;
    SKEMA_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    kern<<<1, kCholThreads, smem, c->stream>>>(G, (int)k, R, Rinv, st);
    SKEMA_LAUNCHED(c);
    if (!small) tri_solve(c, R, k, Rinv, k, k, true, st);
    return;
  }
  cholesky_kernel<<<1, 1024, 0, c->stream>>>(G, k, st);
  SKEMA_LAUNCHED(c);
  lower_to_upper_kernel<<<g1(c, k * k), 256, 0, c->stream>>>(G, R, k);
  SKEMA_LAUNCHED(c);
  identity_kernel<<<g1(c, k * k), 256, 0, c->stream>>>(Rinv, k);
  SKEMA_LAUNCHED(c);
  trsm_upper(c, R, k, Rinv, k, k);
}

// In-place CholeskyQR2 (+ shifted pre-pass if needed) of the column-major
// rows x k matrix Qm (ld = rows). On return Rout (k x k, upper, column-major)
// holds R with Q_in = Q_out R. False when a Cholesky failed even after the
// shifted pass (the columns are numerically dependent); Qm then holds the
// input times an invertible upper-triangular matrix (the same column space).
bool cholqr_try(skema_ctx* c, double* Qm, int64_t rows, int64_t k, double* Rout, double* work,
                int* dstatus) {
  double* G = work;            // k x k
  double* R = work + k * k;    // k x k
  double* Racc = work + 2 * k * k;
  double* fro2 = work + 3 * k * k;
  identity_kernel<<<g1(c, k * k), 256, 0, c->stream>>>(Racc, k);
  SKEMA_LAUNCHED(c);
  int passes_left = 2;
  bool shifted = false;
  // each pass writes Q R^{-1} into the other of the two buffers
  double* cur = Qm;
  double* nxt = work + 3 * k * k + 8;
  while (passes_left > 0) {
    // G = Q^T Q
    gram(c, cur, rows, rows, k, G);
    chol_inverse(c, G, k, R, G, dstatus);
    int st = 0;
    SKEMA_CUDA(cudaMemcpyAsync(&st, dstatus, sizeof(int), cudaMemcpyDeviceToHost, c->stream));
    SKEMA_CUDA(cudaStreamSynchronize(c->stream));
    if (st != 0) {
      if (shifted) {
        if (cur != Qm)
          SKEMA_CUDA(cudaMemcpyAsync(Qm, cur, sizeof(double) * (size_t)(rows * k), cudaMemcpyDeviceToDevice,
                                     c->stream));
        return false;
      }
      // shifted CholeskyQR: G + s I with s = 11 (rows*k + k(k+1)) u ||Q||_F^2
      gram(c, cur, rows, rows, k, G);
      trace_kernel<<<1, 256, 0, c->stream>>>(G, k, fro2);
      SKEMA_LAUNCHED(c);
      const double u = 1.1102230246251565e-16;
      shift_diag_kernel<<<(int)((k + 255) / 256), 256, 0, c->stream>>>(
          G, k, fro2, 11.0 * ((double)rows * k + (double)k * (k + 1)) * u);
      SKEMA_LAUNCHED(c);
      chol_inverse(c, G, k, R, G, dstatus);
      SKEMA_CUDA(cudaMemcpyAsync(&st, dstatus, sizeof(int), cudaMemcpyDeviceToHost, c->stream));
      SKEMA_CUDA(cudaStreamSynchronize(c->stream));
      if (st != 0) {
        if (cur != Qm)
          SKEMA_CUDA(cudaMemcpyAsync(Qm, cur, sizeof(double) * (size_t)(rows * k), cudaMemcpyDeviceToDevice,
                                     c->stream));
        return false;
      }
      shifted = true;
      passes_left = 3;  // shifted pass + CholeskyQR2
    }
    // Q <- Q R^{-1} with G = R^{-1} (upper): next <- cur * Rinv (rows x k)
    tall_times_small(c, cur, rows, rows, k, G, k, k, nxt, rows, true);
    std::swap(cur, nxt);
    // Racc <- R * Racc
    double* tmp = Rout;
    dgemm<double, double>(c, k, k, k, 1.0, R, 1, k, Racc, 1, k, 0.0, tmp, 1, k, false);
    SKEMA_CUDA(cudaMemcpyAsync(Racc, tmp, sizeof(double) * (size_t)(k * k),
                               cudaMemcpyDeviceToDevice, c->stream));
    --passes_left;
  }
  if (cur != Qm)
    SKEMA_CUDA(cudaMemcpyAsync(Qm, cur, sizeof(double) * (size_t)(rows * k), cudaMemcpyDeviceToDevice, c->stream));
  SKEMA_CUDA(cudaMemcpyAsync(Rout, Racc, sizeof(double) * (size_t)(k * k), cudaMemcpyDeviceToDevice,
                             c->stream));
  return true;
}

void cholqr(skema_ctx* c, double* Qm, int64_t rows, int64_t k, double* Rout, double* work, int* dstatus) {
  if (!cholqr_try(c, Qm, rows, k, Rout, work, dstatus))
    fail(SKEMA_ENOTPD, "Cholesky of the Gram matrix failed after the shifted pass");
}

// 3 k^2 + 8 for cholqr's small matrices, rows x k for its second buffer,
// 3 k^2 + 8 more for orth's eigen-decomposition.
size_t cholqr_work_doubles(int64_t rows, int64_t k) { return (size_t)(6 * k * k + 16 + rows * k); }

// Uniform values on [-1, 1) from SplitMix64 (Steele, Lea and Flood, OOPSLA
// 2014) of (seed + index): the completion directions of orth.
__global__ void fill_uniform_kernel(double* __restrict__ W, int64_t cnt, uint64_t seed) {
  for (int64_t q = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; q < cnt; q += (int64_t)gridDim.x * blockDim.x) {
    uint64_t z = seed + 0x9e3779b97f4a7c15ull * (uint64_t)(q + 1);
    z = (z ^ (z >> 30)) * 0xbf58476d1ce4e5b9ull;
    z = (z ^ (z >> 27)) * 0x94d049bb133111ebull;
    z ^= z >> 31;
    W[q] = (double)(z >> 11) * (2.0 / 9007199254740992.0) - 1.0;
  }
}

// An orthonormal basis Q (rows x k, in place) whose first columns span the
// column space of the input, as dgeqrf + dorgqr give (src/Skema_SketchySVD.cpp:
// 355-357, 381-383) also for inputs of rank below k. CholeskyQR2 first; when
// the columns are numerically dependent, the eigen-decomposition of the
// Gram matrix gives the independent directions (eigenvalues above 1e-12 of
// the largest), which are orthonormalised, and the remaining columns are
// completed with pseudo-random directions orthogonalised against them twice
// (block Gram-Schmidt) and then among themselves. Householder QR completes
// the basis with other orthonormal columns of the same complement; the
// fixed-rank approximation does not depend on that choice beyond the rank
// of the sketch.
void orth(skema_ctx* c, double* Qm, int64_t rows, int64_t k, double* Rscratch, double* work, int* dstatus) {
  if (cholqr_try(c, Qm, rows, k, Rscratch, work, dstatus)) return;
  double* T = work + 3 * k * k + 8;              // rows x k
  double* G = T + rows * k;                      // k x k
  double* V = G + k * k;                         // k x k
  double* Vs = V + k * k;                        // k x k (sorted)
  double* Sv = Vs + k * k;                       // k
  double* sig = Sv + k;                          // k
  dgemm<double, double>(c, k, k, rows, 1.0, Qm, rows, 1, Qm, 1, rows, 0.0, G, 1, k);
  jacobi_svd(c, G, V, k, 60, 1e-15, dstatus);
  // G V = U diag(lambda) with U = V for the symmetric positive semidefinite G
  svd_finish_kernel<<<1, kFinishThreads, 0, c->stream>>>(G, V, k, Rscratch /*U, unused*/, Vs, Sv, sig);
  SKEMA_LAUNCHED(c);
  std::vector<double> lam(k), vs((size_t)(k * k));
  SKEMA_CUDA(cudaMemcpyAsync(lam.data(), Sv, sizeof(double) * (size_t)k, cudaMemcpyDeviceToHost, c->stream));
  SKEMA_CUDA(cudaMemcpyAsync(vs.data(), Vs, sizeof(double) * (size_t)(k * k), cudaMemcpyDeviceToHost, c->stream));
  SKEMA_CUDA(cudaStreamSynchronize(c->stream));
  int64_t r = 0;
  while (r < k && lam[r] > 1e-12 * lam[0]) ++r;
  if (r == 0) fail(SKEMA_ENOTPD, "the sketch is zero: no direction to orthonormalise");
  // B = V_r diag(lambda_r^-1/2): Q V_r B has orthonormal columns up to rounding
  for (int64_t j = 0; j < r; ++j) {
    const double sc = 1.0 / std::sqrt(lam[j]);
    for (int64_t i = 0; i < k; ++i) vs[i + j * k] *= sc;
  }
  SKEMA_CUDA(cudaMemcpyAsync(G, vs.data(), sizeof(double) * (size_t)(k * r), cudaMemcpyHostToDevice, c->stream));
  dgemm<double, double>(c, rows, r, k, 1.0, Qm, 1, rows, G, 1, k, 0.0, T, 1, rows, false);
  SKEMA_CUDA(cudaMemcpyAsync(Qm, T, sizeof(double) * (size_t)(rows * r), cudaMemcpyDeviceToDevice, c->stream));
  // stream order keeps the host vectors' copies complete before they go out of scope
  SKEMA_CUDA(cudaStreamSynchronize(c->stream));
  cholqr(c, Qm, rows, r, Rscratch, work, dstatus);  // well conditioned now
  if (r == k) return;
  double* W = Qm + r * rows;  // columns r .. k-1
  const int64_t kr = k - r;
  fill_uniform_kernel<<<g1(c, rows * kr), 256, 0, c->stream>>>(W, rows * kr, 0x5eed5eedull + (uint64_t)k);
  SKEMA_LAUNCHED(c);
  for (int pass = 0; pass < 2; ++pass) {
    // W <- W - Q2 (Q2^T W)
    dgemm<double, double>(c, r, kr, rows, 1.0, Qm, rows, 1, W, 1, rows, 0.0, G, 1, r);
    dgemm<double, double>(c, rows, kr, r, -1.0, Qm, 1, rows, G, 1, r, 1.0, W, 1, rows, false);
  }
  cholqr(c, W, rows, kr, Rscratch, work, dstatus);
}

// In-place sum over the ranks of a row-block sharded sketch (device
// memory, after the context's stream has finished writing it), through the
// caller's all-reduce; nothing for a single context.
struct RankSum {
  skema_allreduce_fn fn = nullptr;
  void* user = nullptr;
  bool on() const { return fn != nullptr; }
  void operator()(skema_ctx* c, double* buf, int64_t count) const {
    if (!fn) return;
    SKEMA_CUDA(cudaStreamSynchronize(c->stream));
    if (fn(buf, count, user) != 0) fail(SKEMA_ECOLLECTIVE, "the all-reduce callback reported a failure");
  }
};

// The orthonormal basis of orth() for the FP32 sketch S (rows x k,
// column-major ld lds), left as Qm Tout with Tout upper triangular (k x k):
// the first CholeskyQR pass reads S itself (its products are exact in
// FP64) and writes Qm = S R1^{-1}; the second pass only factors
// Qm^T Qm = R2^T R2 and returns Tout = R2^{-1}, so the last product with
// the tall matrix is folded by the caller into the small matrices it
// multiplies the basis by anyway. When a Cholesky factor does not exist,
// orth() makes the basis explicit in Qm from the FP64 matrix at hand and
// Tout = I. With a rank sum, S is this rank's row block of a sharded
// sketch: both Gram matrices are summed over the ranks before their
// Cholesky, Qm is the block's rows of the basis, and a missing factor
// fails (SKEMA_ENOTPD) on every rank alike, since the explicit fallback
// needs the whole matrix.
void orth_lazy(skema_ctx* c, const float* S, int64_t lds, double* Qm, int64_t rows, int64_t k, double* Tout,
               double* Rscratch, double* work, int* dstatus, const RankSum& rsum = RankSum{}) {
  double* G = work;
  double* R = work + k * k;
  auto factor = [&] {
    chol_inverse(c, G, k, R, G, dstatus);
    int st = 0;
    SKEMA_CUDA(cudaMemcpyAsync(&st, dstatus, sizeof(int), cudaMemcpyDeviceToHost, c->stream));
    SKEMA_CUDA(cudaStreamSynchronize(c->stream));
    return st == 0;
  };
  auto explicit_basis = [&] {
    if (rsum.on())
      fail(SKEMA_ENOTPD, "the sharded sketch is rank deficient: CholeskyQR needs full column rank");
    orth(c, Qm, rows, k, Rscratch, work, dstatus);
    identity_kernel<<<g1(c, k * k), 256, 0, c->stream>>>(Tout, k);
    SKEMA_LAUNCHED(c);
  };
  if (k <= kTallMaxK || rows <= 0) {
    gram_t<float>(c, S, lds, rows, k, G);
  } else {
    dgemm<float, float>(c, k, k, rows, 1.0, S, lds, 1, S, 1, lds, 0.0, G, 1, k);
  }
  rsum(c, G, k * k);
  if (!factor()) {
    f2d_kernel<<<g1(c, rows * k), 256, 0, c->stream>>>(S, 1, lds, Qm, 1, rows, rows, k);
    SKEMA_LAUNCHED(c);
    explicit_basis();
    return;
  }
  // Qm = S R1^{-1} (G holds R1^{-1})
  if (rows <= 0) {
  } else if (k <= kTallMaxK) {
    tall_times_small_t<float>(c, S, lds, rows, k, G, k, k, Qm, rows, true);
  } else {
    dgemm<float, double>(c, rows, k, k, 1.0, S, 1, lds, G, 1, k, 0.0, Qm, 1, rows, false);
  }
  gram(c, Qm, rows, rows, k, G);
  rsum(c, G, k * k);
  if (!factor()) {
    explicit_basis();
    return;
  }
  SKEMA_CUDA(cudaMemcpyAsync(Tout, G, sizeof(double) * (size_t)(k * k), cudaMemcpyDeviceToDevice, c->stream));
}

// out (R x k, column-major ld R) = Map~ (R x cols) * Qm (cols x k, column-major ld cols)
// out (R x k, column-major) = M Q for the map's logical R x cols matrix M
// and rows [q0, q0 + qrows) of Q held in Qm (column-major, ld qrows): the
// block's share of M Q, which sums over the row blocks to the whole.
void apply_map_rows(skema_ctx* c, const Map& mp, const double* Qm, int64_t q0, int64_t qrows, int64_t k,
                    double* out) {
  const int64_t R = mp.lrows;
  if (qrows <= 0) {
    SKEMA_CUDA(cudaMemsetAsync(out, 0, sizeof(double) * (size_t)(R * k), c->stream));
    return;
  }
  if (mp.kind == SKEMA_MAP_GAUSS) {
    if (mp.cs == 1 && R <= kTallMaxK * 4 && k <= kTallMaxK) {
      // M(:, rows) Q = (M(:, rows)^T)^T Q: the map's logical rows are
      // contiguous over the operand's rows, a tall column-major matrix
      SKEMA_CUDA(cudaMemsetAsync(out, 0, sizeof(double) * (size_t)(R * k), c->stream));
      launch_atb_mma<float, double>(c, mp.f32 + q0, mp.rs, R, Qm, qrows, k, qrows, out);
      return;
    }
    dgemm<float, double>(c, R, k, qrows, 1.0, mp.f32 + q0 * mp.cs, mp.rs, mp.cs, Qm, 1, qrows, 0.0, out, 1, R);
    return;
  }
  if (!mp.transposed) {
    rowsparse_apply_kernel<<<g1(c, R * k), 256, 0, c->stream>>>(mp.packed, mp.zeta, R, Qm, qrows, k, out, R, q0,
                                                                 qrows);
    SKEMA_LAUNCHED(c);
  } else {
    // stored rows are the operand's rows: the block's stored rows only
    const uint32_t* mpb = mp.packed + q0 * mp.zeta;
    SKEMA_CUDA(cudaMemsetAsync(out, 0, sizeof(double) * (size_t)(R * k), c->stream));
    const size_t priv = sizeof(double) * (size_t)(R * k);
    if (priv <= 200 * 1024) {
      SKEMA_CUDA(cudaFuncSetAttribute(colsparse_apply_smem_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                      (int)priv));
      colsparse_apply_smem_kernel<<<c->sm_count, 1024, priv, c->stream>>>(mpb, mp.zeta, qrows, Qm, qrows, k, out,
                                                                            R, R);
    } else {
      colsparse_apply_kernel<<<g1(c, qrows * k), 256, 0, c->stream>>>(mpb, mp.zeta, qrows, Qm, qrows, k, out, R);
    }
    SKEMA_LAUNCHED(c);
  }
}

void apply_map(skema_ctx* c, const Map& mp, const double* Qm, int64_t cols, int64_t k, double* out) {
  apply_map_rows(c, mp, Qm, 0, cols, k, out);
}

// ---- SketchySPD pieces -----------------------------------------------------
// Stored SparseSign rows (zeta entries: column | sign << 31) -> dense n x k
// (column-major, ld n, zeroed beforehand); duplicate entries add up.
__global__ void ssign_dense_kernel(const uint32_t* __restrict__ packed, int zeta, int64_t n, double* __restrict__ D) {
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x)
    for (int t = 0; t < zeta; ++t) {
      const uint32_t w = packed[i * zeta + t];
      D[i + (int64_t)(w & 0x7fffffffu) * n] += (w >> 31) ? -1.0 : 1.0;
    }
}
// SparseSignDimRedux::axpy as the reference runs it (`*=`): each stored entry
// multiplies its Y entry by eta * sign, a duplicate entry twice.
__global__ void ssign_scale_kernel(const uint32_t* __restrict__ packed, int zeta, int64_t n, double* __restrict__ Y,
                                   int64_t ldy, double eta) {
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x)
    for (int t = 0; t < zeta; ++t) {
      const uint32_t w = packed[i * zeta + t];
      Y[i + (int64_t)(w & 0x7fffffffu) * ldy] *= eta * ((w >> 31) ? -1.0 : 1.0);
    }
}
__global__ void daxpy_kernel(double* __restrict__ Y, const double* __restrict__ X, int64_t cnt, double a) {
  for (int64_t q = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; q < cnt; q += (int64_t)gridDim.x * blockDim.x)
    Y[q] += a * X[q];
}
// C = (B + B^T) / 2, column-major k x k.
__global__ void symmetrize_kernel(const double* __restrict__ B, double* __restrict__ C, int64_t k) {
  for (int64_t q = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; q < k * k; q += (int64_t)gridDim.x * blockDim.x) {
    const int64_t i = q % k, j = q / k;
    C[q] = 0.5 * (B[i + j * k] + B[j + i * k]);
  }
}
// out_j = max(0, S_j^2 - sub): squared singular values of E less the shift.
__global__ void spd_eig_kernel(const double* __restrict__ S, double* __restrict__ out, int64_t r, double sub) {
  for (int64_t j = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; j < r; j += (int64_t)gridDim.x * blockDim.x)
    out[j] = fmax(0.0, S[j] * S[j] - sub);
}

}  // namespace

// SketchySPD::low_rank_approx (src/Skema_SketchySVD.cpp:935-1151) in FP64 on
// the device, with Omega the stored n x k map and Y the m x k sketch (m = n):
//   nu = ||Y||_2 (from the largest eigenvalue of Y^T Y), eta = eps nu (below)
//   Y_eta = Y + eta Omega   (REFERENCE_STEPS with SparseSign: each stored map
//                            entry multiplies its Y entry by eta * sign)
//   B = Omega^T Y_eta, R^T R = (B + B^T) / 2 (upper Cholesky, as dpotrf 'U')
//   E = Y_eta R^{-1}        (REFERENCE_STEPS: the unshifted Y, :1094-1103)
//   U S V^T = svd(E)        (CholeskyQR2 of E, then a Jacobi SVD of its R)
//   U <- U(:, 1:r), S_j <- max(0, S_j^2 - eta)   (REFERENCE_STEPS: - nu)
// The reference takes eta from the norm of a buffer dgesvd has already
// overwritten (:964-965), a value that depends on the LAPACK build; its
// steps here use eps ||Y||_2, the value its comment states, which enters at
// the level of eps. The Nystrom form shifts by the FP32 epsilon times
// ||Y||_2, because Y is held in FP32: a shift below the rounding of Y leaves
// B indefinite for spectra that decay to zero.
void spd_low_rank_approx(skema_ctx* c, double* Uout, double* Sout) {
  const int64_t m = c->m, n = c->n, k = c->k, r = c->p.rank;
  const bool ref_steps = c->p.spd_approx == SKEMA_SPD_REFERENCE_STEPS;
  const Map& O = c->omg;
  y_materialize(c);
  const size_t b_mk = sizeof(double) * (size_t)(m * k), b_nk = sizeof(double) * (size_t)(n * k);
  const size_t b_w = sizeof(double) * cholqr_work_doubles(m, k);
  const size_t b_small = sizeof(double) * (size_t)(8 * k * k + 4 * k + 64);
  Carve cv(c, {b_mk, b_mk, b_nk, b_w, b_small, kStatusBytes});
  double* Yd = cv.take(b_mk);
  double* Ye = cv.take(b_mk);
  double* Od = cv.take(b_nk);
  double* W = cv.take(b_w);
  double* G = cv.take(b_small);  // k x k
  double* R = G + k * k;        // k x k
  double* Rinv = R + k * k;     // k x k
  double* Cw = Rinv + k * k;    // k x k
  double* Vc = Cw + k * k;      // k x k
  double* Uc = Vc + k * k;      // k x k
  double* Vt = Uc + k * k;      // k x k
  double* RE = Vt + k * k;      // k x k
  double* Sv = RE + k * k;      // k
  double* sig = Sv + k;         // k
  int* st = reinterpret_cast<int*>(cv.take(kStatusBytes));

  f2d_kernel<<<g1(c, m * k), 256, 0, c->stream>>>(c->Y, 1, m, Yd, 1, m, m, k);
  SKEMA_LAUNCHED(c);
  if (O.kind == SKEMA_MAP_GAUSS) {
    // stored (i, j) = logical (j, i)
    f2d_kernel<<<g1(c, n * k), 256, 0, c->stream>>>(O.f32, O.cs, O.rs, Od, 1, n, n, k);
  } else {
    SKEMA_CUDA(cudaMemsetAsync(Od, 0, sizeof(double) * (size_t)(n * k), c->stream));
    ssign_dense_kernel<<<g1(c, n), 256, 0, c->stream>>>(O.packed, O.zeta, n, Od);
  }
  SKEMA_LAUNCHED(c);

  // nu = ||Y||_2 = sqrt(lambda_max(Y^T Y))
  dgemm<double, double>(c, k, k, m, 1.0, Yd, m, 1, Yd, 1, m, 0.0, G, 1, k);
  jacobi_svd(c, G, Vc, k, 60, 1e-15, st);
  svd_finish_kernel<<<1, kFinishThreads, 0, c->stream>>>(G, Vc, k, Uc, Vt, Sv, sig);
  SKEMA_LAUNCHED(c);
  double lmax = 0.0;
  SKEMA_CUDA(cudaMemcpyAsync(&lmax, Sv, sizeof(double), cudaMemcpyDeviceToHost, c->stream));
  SKEMA_CUDA(cudaStreamSynchronize(c->stream));
  const double nu = std::sqrt(std::max(lmax, 0.0));
  // the Nystrom shift covers the rounding of Y, which is held in FP32 here
  // (the reference holds Y in FP64 and shifts by the FP64 epsilon)
  const double eta =
      (ref_steps ? std::numeric_limits<double>::epsilon() : (double)std::numeric_limits<float>::epsilon()) * nu;

  // Y_eta
  SKEMA_CUDA(cudaMemcpyAsync(Ye, Yd, sizeof(double) * (size_t)(m * k), cudaMemcpyDeviceToDevice, c->stream));
  if (ref_steps && O.kind == SKEMA_MAP_SPARSE_SIGN) {
    ssign_scale_kernel<<<g1(c, n), 256, 0, c->stream>>>(O.packed, O.zeta, n, Ye, m, eta);
  } else {
    daxpy_kernel<<<g1(c, m * k), 256, 0, c->stream>>>(Ye, Od, m * k, eta);
  }
  SKEMA_LAUNCHED(c);
  // B = Omega^T Y_eta; R^T R = (B + B^T) / 2
  dgemm<double, double>(c, k, k, n, 1.0, Od, n, 1, Ye, 1, m, 0.0, Cw, 1, k);
  symmetrize_kernel<<<g1(c, k * k), 256, 0, c->stream>>>(Cw, G, k);
  SKEMA_LAUNCHED(c);
  chol_inverse(c, G, k, R, Rinv, st);
  int bad = 0;
  SKEMA_CUDA(cudaMemcpyAsync(&bad, st, sizeof(int), cudaMemcpyDeviceToHost, c->stream));
  SKEMA_CUDA(cudaStreamSynchronize(c->stream));
  if (bad != 0) fail(SKEMA_ENOTPD, "SketchySPD: (B + B^T) / 2 is not positive definite (dpotrf would fail)");
  // E = (Y_eta or Y) R^{-1}, into Yd's buffer when it is no longer needed
  double* E = ref_steps ? Ye : Yd;
  const double* src = ref_steps ? Yd : Ye;
  dgemm<double, double>(c, m, k, k, 1.0, src, 1, m, Rinv, 1, k, 0.0, E, 1, m, false);
  // svd(E) = Q svd(R_E)
  cholqr(c, E, m, k, RE, W, st);
  SKEMA_CUDA(cudaMemcpyAsync(Cw, RE, sizeof(double) * (size_t)(k * k), cudaMemcpyDeviceToDevice, c->stream));
  jacobi_svd(c, Cw, Vc, k, 60, 1e-15, st);
  svd_finish_kernel<<<1, kFinishThreads, 0, c->stream>>>(Cw, Vc, k, Uc, Vt, Sv, sig);
  SKEMA_LAUNCHED(c);
  if (Uout) dgemm<double, double>(c, m, r, k, 1.0, E, 1, m, Uc, 1, k, 0.0, Uout, 1, m, false);
  if (Sout) {
    spd_eig_kernel<<<1, 256, 0, c->stream>>>(Sv, Sout, r, ref_steps ? nu : eta);
    SKEMA_LAUNCHED(c);
  }
  SKEMA_CUDA(cudaStreamSynchronize(c->stream));
}

void dgemm_f32_f64(skema_ctx* c, int64_t M, int64_t N, int64_t K, double alpha, const float* A, int64_t ars,
                   int64_t acs, const double* B, int64_t brs, int64_t bcs, double beta, double* C, int64_t crs,
                   int64_t ccs) {
  dgemm<float, double>(c, M, N, K, alpha, A, ars, acs, B, brs, bcs, beta, C, crs, ccs);
}

// The fixed-rank approximation from Y's rows [row0, row0 + nrows) with
// the sums over row blocks taken by rsum (a row-block sharded sketch whose
// X and Z are already summed), or from all of Y (rsum off, the whole
// range). U (nrows x rank, column-major ld nrows) gets the block's rows.
void low_rank_approx_rows(skema_ctx* c, int64_t row0, int64_t nrows, const RankSum& rsum, double* Uout,
                          double* Sout, double* Vout) {
  const int64_t m = nrows, n = c->n, k = c->k, s = c->s, r = c->p.rank;
  y_materialize(c);
  const size_t b_q = sizeof(double) * (size_t)(m * k), b_p = sizeof(double) * (size_t)(n * k);
  const size_t b_w = sizeof(double) * cholqr_work_doubles(std::max(m, std::max(n, s)), k);
  const size_t b_u = sizeof(double) * (size_t)(s * k);
  const size_t b_small = sizeof(double) * (size_t)(12 * k * k + s * s + k * s + 4 * k + 64);
  Carve cv(c, {b_q, b_p, b_w, b_u, b_u, b_small, kStatusBytes});
  double* Q = cv.take(b_q);
  double* P = cv.take(b_p);
  double* W = cv.take(b_w);
  double* U1 = cv.take(b_u);
  double* U2 = cv.take(b_u);
  double* T1 = cv.take(b_small);
  double* T2 = T1 + k * k;
  double* Z1 = T2 + k * k;         // k x s
  double* Z2 = Z1 + k * s;         // k x k
  double* Z2t = Z2 + k * k;        // k x k
  double* Uc = Z2t + k * k;        // k x k
  double* Vc = Uc + k * k;         // k x k
  double* Sv = Vc + k * k;         // k
  double* sig = Sv + k;            // k
  double* Zd = sig + k;            // s x s
  double* TQ = Zd + s * s;         // k x k: the basis of Y is Q TQ
  double* TP = TQ + k * k;         // k x k: the basis of X^T is P TP
  double* WU = TP + k * k;         // k x r
  double* WV = WU + k * k;         // k x r
  int* st = reinterpret_cast<int*>(cv.take(kStatusBytes));

  auto orth_scope = std::make_unique<StageScope>(c, ST_A_ORTH);
  f2d_kernel<<<g1(c, s * s), 256, 0, c->stream>>>(c->Z, s, 1, Zd, 1, s, s, s);
  SKEMA_LAUNCHED(c);
  // bases of Y (m x k, column-major) and X^T (n x k: X is k x n row-major),
  // as Q TQ and P TP
  orth_lazy(c, c->X, n, P, n, k, TP, T1, W, st);  // T1 used as scratch R here
  orth_lazy(c, c->Y + row0, c->m, Q, m, k, TQ, T1, W, st, rsum);
  orth_scope.reset();
  auto core_scope = std::make_unique<StageScope>(c, ST_A_CORE);
  // U1 = Phi~ Q TQ (s x k), U2 = Psi~ P TP (s x k); W holds Phi~ Q, Psi~ P
  apply_map_rows(c, c->phi, Q, row0, m, k, W);
  rsum(c, W, s * k);
  tall_times_small(c, W, s, s, k, TQ, k, k, U1, s, true);
  apply_map(c, c->psi, P, n, k, W);
  tall_times_small(c, W, s, s, k, TP, k, k, U2, s, true);
  cholqr(c, U1, s, k, T1, W, st);
  cholqr(c, U2, s, k, T2, W, st);
  // Z1 = U1^T Z (k x s); Z2 = Z1 U2 (k x k)
  dgemm<double, double>(c, k, s, s, 1.0, U1, s, 1, Zd, 1, s, 0.0, Z1, 1, k);
  dgemm<double, double>(c, k, k, s, 1.0, Z1, 1, k, U2, 1, s, 0.0, Z2, 1, k);
  // Z2 = T1 \ Z2
  trsm_upper(c, T1, k, Z2, k, k);
  // C^T = T2 \ Z2^T
  dtranspose_kernel<<<g1(c, k * k), 256, 0, c->stream>>>(Z2, Z2t, k);
  SKEMA_LAUNCHED(c);
  trsm_upper(c, T2, k, Z2t, k, k);
  // C = (Z2t)^T: copy into Uc's slot as the Jacobi working matrix
  double* C = Uc;
  core_scope.reset();
  {
    StageScope sc(c, ST_A_SVD);
    double* Cw = W;  // k x k working copy
    dtranspose_kernel<<<g1(c, k * k), 256, 0, c->stream>>>(Z2t, Cw, k);
    SKEMA_LAUNCHED(c);
    jacobi_svd(c, Cw, Vc, k, 60, 1e-15, st);
    svd_finish_kernel<<<1, kFinishThreads, 0, c->stream>>>(Cw, Vc, k, C, Z2 /*Vout*/, Sv, sig);
    SKEMA_LAUNCHED(c);
  }
  {
    StageScope sc(c, ST_A_VECTORS);
    // U = Q TQ Uc(:, 1:r), V = P TP Vc(:, 1:r), S = S(1:r)
    if (Uout) {
      tall_times_small(c, TQ, k, k, k, C, k, r, WU, k);
      tall_times_small(c, Q, m, m, k, WU, k, r, Uout, m);
    }
    if (Vout) {
      tall_times_small(c, TP, k, k, k, Z2, k, r, WV, k);
      tall_times_small(c, P, n, n, k, WV, k, r, Vout, n);
    }
    if (Sout)
      SKEMA_CUDA(cudaMemcpyAsync(Sout, Sv, sizeof(double) * (size_t)r, cudaMemcpyDeviceToDevice, c->stream));
  }
  int sweeps = 0;
  SKEMA_CUDA(cudaMemcpyAsync(&sweeps, st + 1, sizeof(int), cudaMemcpyDeviceToHost, c->stream));
  SKEMA_CUDA(cudaStreamSynchronize(c->stream));
  c->svd_sweeps = sweeps;
}

void low_rank_approx(skema_ctx* c, double* Uout, double* Sout, double* Vout) {
  low_rank_approx_rows(c, 0, c->m, RankSum{}, Uout, Sout, Vout);
}

void low_rank_approx_sharded(skema_ctx* c, int64_t row0, int64_t nrows, skema_allreduce_fn fn, void* user,
                             double* Uout, double* Sout, double* Vout) {
  RankSum rs;
  rs.fn = fn;
  rs.user = user;
  low_rank_approx_rows(c, row0, nrows, rs, Uout, Sout, Vout);
}

}  // namespace skema
