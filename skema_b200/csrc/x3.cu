// x3.cu -- the FP32 form of the dense and kernel sketch on the tensor cores
// (update(dense, Gauss), src/Skema_SketchySVD.cpp:256-268, and the Gauss-RBF
// window), by three BF16 planes per FP32 operand (tc_x3.cuh).
//
// Per block of rows [R0, R0 + wr) of the input:
//   planes of A_w        row-blocked (64-row blocks, a 128-byte line of 64
//                        rows per column), written once, read by both products
//   [Y_w | T] = A_w [Omega~; Psi~]^T   M = wr, N = k + s, K = n
//   X^T += eta A_w^T Upsilon~_w^T      M = n,  N = k,     K = wr
//   Z^T += eta T^T Phi~_w^T            M = s,  N = s,     K = wr
// T stays in planes. Blocks need not follow the windows: with
// X = nu X + eta x_w after each of G windows, X = nu^G X + eta sum_w
// nu^(G-1-w) x_w, so the weights go into the converted columns of Upsilon~
// and Phi~, and a call of many short windows is one block.
#include <cuda_bf16.h>
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>

#include "internal.h"
#include "tc_host.h"
#include "tc_x3.cuh"
#include "x3.h"

namespace skema {

namespace {

__device__ __forceinline__ void store_planes8(const float* v, __nv_bfloat16* d, int64_t pstride) {
  __nv_bfloat162 q[3][4];
#pragma unroll
  for (int t = 0; t < 4; ++t) tc::split3x2(v[2 * t], v[2 * t + 1], q[0][t], q[1][t], q[2][t]);
#pragma unroll
  for (int p = 0; p < 3; ++p) *reinterpret_cast<uint4*>(d + p * pstride) = *reinterpret_cast<const uint4*>(q[p]);
}

// A window block into row-blocked planes; rows past `rows` in the last 64 are
// zeros. VEC: rows contiguous and 16-byte aligned (a thread: 8 rows of one
// column, two 16-byte loads, three 16-byte stores). 10 bytes per element, HBM
// bound.
__global__ void __launch_bounds__(256)
    x3_block_vec_kernel(const float* __restrict__ S, int64_t scs, int64_t rows, int64_t cols,
                        __nv_bfloat16* __restrict__ D, int64_t nrb, int64_t pstride, uint32_t big,
                        uint32_t small, uint32_t* __restrict__ flag) {
  const int64_t total = nrb * 8 * cols;
  float top = 0.f;
  for (int64_t q = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; q < total; q += (int64_t)gridDim.x * blockDim.x) {
    // 64-row block outermost, then columns, then the 8 groups of a line: a
    // warp's stores are 512 contiguous bytes per plane
    const int64_t rb = q / (8 * cols), w = q - rb * 8 * cols, j = w >> 3, i = rb * 64 + (w & 7) * 8;
    const float* sp = S + i + j * scs;
    float v[8];
    if (i + 8 <= rows) {
      const float4 a = __ldcs(reinterpret_cast<const float4*>(sp));
      const float4 b = __ldcs(reinterpret_cast<const float4*>(sp + 4));
      v[0] = a.x, v[1] = a.y, v[2] = a.z, v[3] = a.w, v[4] = b.x, v[5] = b.y, v[6] = b.z, v[7] = b.w;
    } else {
#pragma unroll
      for (int t = 0; t < 8; ++t) v[t] = (i + t < rows) ? sp[t] : 0.f;
    }
#pragma unroll
    for (int t = 0; t < 8; ++t) x3_note(top, v[t]);
    store_planes8(v, D + (rb * cols + j) * 64 + (w & 7) * 8, pstride);
  }
  x3_report(top, big, flag, small);
}

// The same from any strides, by 64 x 32 tiles through shared memory.
__global__ void __launch_bounds__(256)
    x3_block_tiled_kernel(const float* __restrict__ S, int64_t srs, int64_t scs, int64_t rows, int64_t cols,
                          __nv_bfloat16* __restrict__ D, int64_t nrb, int64_t pstride, uint32_t big,
                          uint32_t small, uint32_t* __restrict__ flag) {
  __shared__ float tile[32][65];
  const int tx = threadIdx.x & 31, ty = threadIdx.x >> 5;
  const int64_t tj = (cols + 31) / 32;
  const bool rowfast = srs <= scs;
  float top = 0.f;
  for (int64_t t = blockIdx.x; t < nrb * tj; t += gridDim.x) {
    const int64_t rb = t / tj, j0 = (t - rb * tj) * 32;
#pragma unroll
    for (int q = 0; q < 8; ++q) {
      const int e = ty + 8 * q;  // 0 .. 63: (32-row half, column) or row
      const int r = rowfast ? tx + 32 * (e >> 5) : e, j = rowfast ? (e & 31) : tx;
      const int64_t gi = rb * 64 + r, gj = j0 + j;
      const float v = (gi < rows && gj < cols) ? S[gi * srs + gj * scs] : 0.f;
      x3_note(top, v);
      tile[j][r] = v;
    }
    __syncthreads();
    const int j = threadIdx.x >> 3, g8 = (threadIdx.x & 7) * 8;
    if (j0 + j < cols) {
      float v[8];
#pragma unroll
      for (int e = 0; e < 8; ++e) v[e] = tile[j][g8 + e];
      store_planes8(v, D + (rb * cols + j0 + j) * 64 + g8, pstride);
    }
    __syncthreads();
  }
  x3_report(top, big, flag, small);
}

// Map columns [0, cols) of up to two row-contiguous FP32 sources into one
// stack of K-major planes, row r of plane q at D[q * pstride + r * ld]. Column
// j is scaled by nu^(nwin - 1 - (j0 + j) / W) (nu = 1: unscaled).
struct X3Src {
  const float* p;
  int64_t rs, rows;
};
__global__ void __launch_bounds__(256)
    x3_maps_kernel(X3Src a, X3Src b, int64_t cols, __nv_bfloat16* __restrict__ D, int64_t ld, int64_t pstride, float nu,
                   int64_t W, int64_t nwin, int64_t j0, uint32_t big, uint32_t* __restrict__ flag) {
  const int64_t c8 = ld / 8, total = (a.rows + b.rows) * c8;
  float top = 0.f;
  for (int64_t q = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; q < total; q += (int64_t)gridDim.x * blockDim.x) {
    const int64_t r = q / c8, j = (q - r * c8) * 8;
    const float* sp = (r < a.rows ? a.p + r * a.rs : b.p + (r - a.rows) * b.rs) + j;
    float v[8];
#pragma unroll
    for (int t = 0; t < 8; ++t) v[t] = (j + t < cols) ? sp[t] : 0.f;
    if (nu != 1.f) {
      int64_t w = -1;
      float s = 1.f;
#pragma unroll
      for (int t = 0; t < 8; ++t) {
        const int64_t wt = (j0 + j + t) / W;
        if (wt != w) w = wt, s = (float)pow((double)nu, (double)max((int64_t)0, nwin - 1 - wt));
        v[t] *= s;
      }
    }
    if (flag) {
#pragma unroll
      for (int t = 0; t < 8; ++t) x3_note(top, v[t]);
    }
    store_planes8(v, D + r * ld + j, pstride);
  }
  if (flag) x3_report(top, big, flag);
}

// The products of X3Plain3 for the rare block that is refused (returns at once
// otherwise): 128 x 128 tiles, 8 x 8 per thread, K steps of 16 through two
// buffers, and K cut into g.split parts that are added to C with atomics when
// the tiles alone would leave the chip idle. Bound by FP32 issue, as
// sgemm_kernel is (36 TFLOP/s): 50,000 x 20,000 (k = 201, s = 403) with an
// infinity in every block takes 59.5 ms in all, 12,000 x 5,000 (k = 81, s = 163)
// 3.1; SIMT calls take 52.3 and 5.5 (64 x 64 tiles with 4 x 4 per thread and a pow
// per weighted value took 174 and 7.8, 228 and 11.6 for nu = 0.95).
constexpr int kPlBM = 128, kPlBK = 16, kPlLd = kPlBM + 4;
// What a thread stages of one operand, element (r, k) with r < R: value q < 8 is
// (r, k + 2 q) where the rows are the contiguous ones, else (r + 16 q, k).
struct PlainSrc {
  const float* p;
  const __nv_bfloat16* pl;  // or the sum of three planes, ps apart, k along the rows
  int64_t ps, dq, adv;      // from value to value, from K step to K step
  int r, k, left, R;        // in the tile; K left from this thread's k on; rows of the tile
  bool rfast;
  __device__ __forceinline__ void init(const float* P, int64_t rs, int64_t ks, const __nv_bfloat16* Pl, int64_t ld,
                                       int64_t planes, int64_t r0, int64_t rows, int64_t k0, int64_t k1) {
    rfast = !Pl && rs <= ks;
    r = rfast ? threadIdx.x & 127 : threadIdx.x >> 4;
    k = rfast ? threadIdx.x >> 7 : threadIdx.x & 15;
    R = (int)min((int64_t)kPlBM, rows - r0);
    left = (int)min((int64_t)0x7fffffff, k1 - k0 - k);
    p = P + (r0 + r) * rs + (k0 + k) * ks;
    pl = Pl ? Pl + (r0 + r) * ld + k0 + k : nullptr;
    ps = planes;
    dq = Pl ? 16 * ld : rfast ? 2 * ks : 16 * rs;
    adv = Pl ? kPlBK : kPlBK * ks;
  }
  __device__ __forceinline__ void load(float (&v)[8]) {
    const int n = rfast ? (r < R ? (left + 1) / 2 : 0) : (left > 0 ? (R - r + 15) / 16 : 0);
    if (pl) {
#pragma unroll
      for (int q = 0; q < 8; ++q) {
        const __nv_bfloat16* t = pl + q * dq;
        v[q] = q < n ? (__bfloat162float(t[0]) + __bfloat162float(t[ps])) + __bfloat162float(t[2 * ps]) : 0.f;
      }
      pl += adv;
    } else {
#pragma unroll
      for (int q = 0; q < 8; ++q) v[q] = q < n ? p[q * dq] : 0.f;
      p += adv;
    }
    left -= kPlBK;
  }
  __device__ __forceinline__ void store(const float (&v)[8], float (*sm)[kPlLd]) const {
    float* s = &sm[k][r];
    const int d = rfast ? 2 * kPlLd : 16;
#pragma unroll
    for (int q = 0; q < 8; ++q) s[q * d] = v[q];
  }
};
__global__ void __launch_bounds__(256, 1) x3_plain_kernel(X3Plain3 a, const uint32_t* __restrict__ flag) {
  if (!x3_refused(*flag)) return;
  __shared__ __align__(16) float As[2][kPlBK][kPlLd], Bs[2][kPlBK][kPlLd];
  const int tx = threadIdx.x & 15, ty = threadIdx.x >> 4;
  for (int64_t q = blockIdx.x * 256 + threadIdx.x; q < a.nscale; q += (int64_t)gridDim.x * 256)
    a.scale[q] = a.by == 0.f ? 0.f : a.by * a.scale[q];
  int64_t t = blockIdx.x;  // tiles of all the products, one after another
  for (int w = 0; w < a.n; ++w) {
    const X3Plain& g = a.g[w];
    const int64_t tn = (g.N + kPlBM - 1) / kPlBM, tiles = (g.M + kPlBM - 1) / kPlBM * tn;
    const int64_t kc = (g.K + g.split - 1) / g.split;
    for (; t < tiles * g.split; t += gridDim.x) {
      const int64_t part = t / tiles, q = t - part * tiles;
      const int64_t m0 = (q / tn) * kPlBM, n0 = (q % tn) * kPlBM, kb = part * kc, ke = min(g.K, kb + kc);
      float acc[8][8] = {}, ra[8], rb[8];
      PlainSrc sa, sb;
      sa.init(g.A, g.ars, g.acs, g.Apl, g.ald, g.aps, m0, g.M, kb, ke);
      sb.init(g.B, g.bcs, g.brs, nullptr, 0, 0, n0, g.N, kb, ke);
      sa.load(ra);
      sb.load(rb);
      sa.store(ra, As[0]);
      sb.store(rb, Bs[0]);
      __syncthreads();
      int buf = 0;
      for (int64_t k0 = kb; k0 < ke; k0 += kPlBK, buf ^= 1) {
        const bool more = k0 + kPlBK < ke;
        if (more) {
          sa.load(ra);
          sb.load(rb);
        }
#pragma unroll
        for (int kk = 0; kk < kPlBK; ++kk) {
          float x[8], y[8];
#pragma unroll
          for (int h = 0; h < 2; ++h) {
            *reinterpret_cast<float4*>(x + 4 * h) = *reinterpret_cast<const float4*>(&As[buf][kk][4 * tx + 64 * h]);
            *reinterpret_cast<float4*>(y + 4 * h) = *reinterpret_cast<const float4*>(&Bs[buf][kk][4 * ty + 64 * h]);
          }
#pragma unroll
          for (int i = 0; i < 8; ++i)
#pragma unroll
            for (int j = 0; j < 8; ++j) acc[i][j] = fmaf(x[i], y[j], acc[i][j]);
        }
        if (more) {  // the other buffer was read last a step ago, before the barrier
          sa.store(ra, As[buf ^ 1]);
          sb.store(rb, Bs[buf ^ 1]);
        }
        __syncthreads();
      }
#pragma unroll
      for (int i = 0; i < 8; ++i)
#pragma unroll
        for (int j = 0; j < 8; ++j) {
          const int64_t m = m0 + 4 * tx + 64 * (i >> 2) + (i & 3), n = n0 + 4 * ty + 64 * (j >> 2) + (j & 3);
          if (m >= g.M || n >= g.N) continue;
          float* p = g.C + m * g.crs + n * g.ccs;
          if (g.split > 1)
            atomicAdd(p, g.alpha * acc[i][j]);
          else
            *p = g.beta == 0.f ? g.alpha * acc[i][j] : fmaf(g.beta, *p, g.alpha * acc[i][j]);
        }
    }
    t -= tiles * g.split;
  }
}

// K-major planes D[q * pstride + c * ld + i] of a row-major source (rows i of
// `cols` values, rs apart), turned by kTrRows x 32 tiles; columns i past `rows`
// up to ld are zeros. Row i is scaled by nu^(nwin - 1 - (j0 + i) / W), which a
// lane forms for each of its warp's rows (a pow in FP64 by every lane took 110 us
// longer). Bound by memory: 100,000 x 163 in 68 us with 64 rows per tile, 34
// with 128, whose stores are runs of 256 bytes.
constexpr int kTrRows = 128;
__global__ void __launch_bounds__(256)
    x3_transposed_kernel(const float* __restrict__ S, int64_t rs, int64_t rows, int64_t cols,
                         __nv_bfloat16* __restrict__ D, int64_t ld, int64_t pstride, float nu, int64_t W, int64_t nwin,
                         int64_t j0, uint32_t big, uint32_t* __restrict__ flag) {
  constexpr int NR = kTrRows / 8;  // rows per warp
  __shared__ float tile[32][kTrRows + 1];
  float top = 0.f;
  const int tx = threadIdx.x & 31, ty = threadIdx.x >> 5;
  const int64_t ti = (ld + kTrRows - 1) / kTrRows, tj = (cols + 31) / 32;
  for (int64_t t = blockIdx.x; t < ti * tj; t += gridDim.x) {
    const int64_t i0 = (t / tj) * kTrRows, c0 = (t % tj) * 32;
    float v[NR];
#pragma unroll
    for (int q = 0; q < NR; ++q) {
      const int r = ty + 8 * q;
      v[q] = (i0 + r < rows && c0 + tx < cols) ? S[(i0 + r) * rs + c0 + tx] : 0.f;
    }
    float w = 1.f;
    if (nu != 1.f && tx < NR && i0 + ty + 8 * tx < rows)
      w = (float)pow((double)nu, (double)(nwin - 1 - (j0 + i0 + ty + 8 * tx) / W));
#pragma unroll
    for (int q = 0; q < NR; ++q) {
      if (nu != 1.f) v[q] *= __shfl_sync(0xffffffffu, w, q);
      x3_note(top, v[q]);
      tile[tx][ty + 8 * q] = v[q];
    }
    __syncthreads();
#pragma unroll
    for (int h = 0; h < kTrRows / 64; ++h) {
      const int item = threadIdx.x + 256 * h, j = item / NR, g8 = (item % NR) * 8;
      if (c0 + j < cols && i0 + g8 < ld) {
        float x[8];
#pragma unroll
        for (int e = 0; e < 8; ++e) x[e] = tile[j][g8 + e];
        store_planes8(x, D + (c0 + j) * ld + i0 + g8, pstride);
      }
    }
    __syncthreads();
  }
  if (flag) x3_report(top, big, flag);
}

int grid_1d(const skema_ctx* c, int64_t items, int per_sm) {
  return (int)std::max<int64_t>(1, std::min<int64_t>((items + 255) / 256, (int64_t)c->sm_count * per_sm));
}

size_t up256(size_t b) { return (b + 255) / 256 * 256; }

CUtensorMap tmap_planes_k(const __nv_bfloat16* p, int64_t K, int64_t rows, int64_t ld, int64_t pstride, uint32_t brows,
                          uint32_t bplanes) {
  return tmap_3d(CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, p, (uint64_t)K, (uint64_t)rows, 3, (uint64_t)ld * 2,
                 (uint64_t)pstride * 2, tc::kX3BK, brows, bplanes, CU_TENSOR_MAP_SWIZZLE_64B);
}

constexpr size_t kX3Smem = 226 * 1024;

}  // namespace

size_t x3_part_bytes(const skema_ctx* c) {
  return (size_t)2 * c->sm_count * 256 * tc::BM * sizeof(float);
}

void x3_gemm(skema_ctx* c, const X3A& a, const X3B& b, int64_t M, int64_t N, int64_t K, const tc::X3Out& o, float* part,
             X3Words words) {
  if (M <= 0 || N <= 0 || K <= 0) return;
  tc::X3Grid g;
  g.mtiles = (int)((M + tc::BM - 1) / tc::BM);
  g.ntiles = (int)((N + 255) / 256);
  g.nt = (int)((N + (int64_t)g.ntiles * 16 - 1) / ((int64_t)g.ntiles * 16) * 16);
  g.ksteps = (int)((K + tc::kX3BK - 1) / tc::kX3BK);
  const size_t stage = tc::kX3ABytes + (size_t)3 * g.nt * tc::kX3BK * 2;
  g.stages = (int)std::min<size_t>(tc::kX3MaxStages, (kX3Smem - 2048) / stage);
  const int64_t tiles = (int64_t)g.mtiles * g.ntiles;
  // runs of at least four K steps (so that none is empty), or a tile: a K of one
  // to three steps leaves nothing to cut
  const int G = (int)std::max<int64_t>(1, std::min<int64_t>(c->sm_count, std::max(tiles, tiles * g.ksteps / 4)));
  g.full = (int)(tiles / G * G);
  if ((tiles - g.full) * g.ksteps < 4 * (int64_t)G) g.full = (int)tiles;  // too little to cut
  CUtensorMap ta;
  if (a.blocked)
    ta = tmap_3d(CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, a.p, 64, (uint64_t)a.cols, (uint64_t)(3 * a.nrb), 128,
                 (uint64_t)a.cols * 128, a.mn ? 64 : tc::kX3BK, a.mn ? tc::kX3BK : tc::BM, 1,
                 a.mn ? CU_TENSOR_MAP_SWIZZLE_128B : CU_TENSOR_MAP_SWIZZLE_64B);
  else
    ta = tmap_planes_k(a.p, K, M, a.ld, a.pstride, tc::BM, 1);
  const CUtensorMap tb = tmap_planes_k(b.p, K, N, b.ld, b.pstride, (uint32_t)g.nt, 3);
  auto kern = a.mn ? tc::gemm_x3_kernel<true> : tc::gemm_x3_kernel<false>;
  SKEMA_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kX3Smem));
  kern<<<G, tc::kX3Threads, kX3Smem, c->stream>>>(ta, tb, g, o, a.blocked ? 1 : 0, (int)a.nrb, part, words, c->dev_err);
  SKEMA_LAUNCHED(c);
  c->dev_err_armed = std::max(c->dev_err_armed, 1);
  const int rem = (int)(tiles - g.full);
  if (rem > 0) {
    if (rem * (g.nt / 8) >= 2 * c->sm_count)
      tc::x3_reduce_kernel<4><<<dim3(rem, g.nt / 8), 256, 0, c->stream>>>(g, o, G, part, words);
    else
      tc::x3_reduce_kernel<1><<<dim3(rem, g.nt / 2), 256, 0, c->stream>>>(g, o, G, part, words);
    SKEMA_LAUNCHED(c);
  }
}

void x3_block_planes(skema_ctx* c, Mat src, int64_t rows, int64_t cols, __nv_bfloat16* D, int64_t pstride, int top,
                     int bottom, uint32_t* flag) {
  const int64_t nrb = (rows + 63) / 64;
  if (src.rs == 1 && src.cs % 4 == 0 && reinterpret_cast<uintptr_t>(src.p) % 16 == 0)
    x3_block_vec_kernel<<<grid_1d(c, nrb * 8 * cols, 16), 256, 0, c->stream>>>(src.p, src.cs, rows, cols, D, nrb,
                                                                               pstride, x3_bits(top), x3_bits(bottom),
                                                                               flag);
  else
    x3_block_tiled_kernel<<<grid_1d(c, nrb * ((cols + 31) / 32) * 256, 16), 256, 0, c->stream>>>(
        src.p, src.rs, src.cs, rows, cols, D, nrb, pstride, x3_bits(top), x3_bits(bottom), flag);
  SKEMA_LAUNCHED(c);
}

void x3_transposed_planes(skema_ctx* c, const float* S, int64_t rs, int64_t rows, int64_t cols, __nv_bfloat16* D,
                          int64_t ld, int64_t pstride, float nu, int64_t W, int64_t nwin, int64_t j0, int top,
                          uint32_t* flag) {
  const int64_t tiles = ((ld + kTrRows - 1) / kTrRows) * ((cols + 31) / 32);
  x3_transposed_kernel<<<grid_1d(c, tiles * 256, 16), 256, 0, c->stream>>>(S, rs, rows, cols, D, ld, pstride, nu, W,
                                                                          nwin, j0, x3_bits(top), flag);
  SKEMA_LAUNCHED(c);
}

void x3_row_planes(skema_ctx* c, const float* S, int64_t rs, int64_t rows, int64_t cols, __nv_bfloat16* D, int64_t ld,
                   int64_t pstride, int top, uint32_t* flag) {
  x3_maps_kernel<<<grid_1d(c, rows * ld / 8, 16), 256, 0, c->stream>>>(X3Src{S, rs, rows}, X3Src{S, rs, 0}, cols, D, ld,
                                                                      pstride, 1.f, 1, 1, 0, x3_bits(top), flag);
  SKEMA_LAUNCHED(c);
}

// K parts of an s x s product, of 256 or more, that fill the chip.
int x3_plain_split(const skema_ctx* c, int64_t s, int64_t K) {
  const int64_t tiles = ((s + kPlBM - 1) / kPlBM) * ((s + kPlBM - 1) / kPlBM);
  return (int)std::max<int64_t>(2, std::min<int64_t>(c->sm_count / tiles, K / 256));
}

void x3_plain(skema_ctx* c, const X3Plain3& p, const uint32_t* flag) {
  x3_plain_kernel<<<c->sm_count, 256, 0, c->stream>>>(p, flag);
  SKEMA_LAUNCHED(c);
}

// The exponent of the bound on A's values for sums over n columns and up to
// `rows` rows of nwin windows: T = A Psi, and the three sketches' sums over the
// block with the window weights (of nu > 1: 2^40 at most) in the maps, stay below
// 2^126.
static int x3_top(const skema_ctx* c, int64_t rows, int64_t nwin) {
  const int ln = x3_log2(c->n), lr = x3_log2(rows);
  int top = std::min(100, 126 - ln - x3_exp(c->omg));
  if (c->spd) return top;
  const double nu = c->p.sketch_nu;
  const int lw = nu > 1.0 ? (int)std::ceil(std::log2(nu) * (double)(nwin - 1)) : 0;
  const int t = ln + x3_exp(c->psi);
  return std::min({top, 126 - t, 126 - lr - x3_exp(c->ups) - lw, 126 - t - lr - x3_exp(c->phi) - lw});
}

// nrows <= wsrows, which sizes the blocks and the workspace. top: x3_top.
static bool x3_windows(skema_ctx* c, const X3Input& in, int64_t row0, int64_t nrows, int64_t wsrows, int top) {
  const int64_t n = c->n, k = c->k, s = c->spd ? 0 : c->s, W = c->w;
  const float eta = (float)c->p.sketch_eta, nu = (float)c->p.sketch_nu;
  const int64_t ldn = pad8(n);
  const size_t b_op = up256(sizeof(__nv_bfloat16) * (size_t)(3 * (k + s) * ldn));
  const size_t b_part = up256(x3_part_bytes(c));
  // rows per block: all of them, or equal blocks whose planes fit the budget
  int64_t rb = 0;
  char* ws = nullptr;
  size_t b_a = 0, b_uf = 0, b_t = 0, b_t32 = 0, b_flag = 0;
  for (size_t budget = (size_t)2 << 30; budget >= ((size_t)64 << 20) && !ws; budget >>= 2) {
    const int64_t cap = std::max<int64_t>(64, (int64_t)(budget / (size_t)(6 * n)) / 64 * 64);
    const int64_t nb = (wsrows + cap - 1) / cap;
    rb = ((wsrows + nb - 1) / nb + 63) / 64 * 64;
    b_a = up256(sizeof(__nv_bfloat16) * (size_t)(3 * rb * n));
    b_uf = up256(sizeof(__nv_bfloat16) * (size_t)(3 * (k + s) * rb));
    b_t = up256(sizeof(__nv_bfloat16) * (size_t)(3 * s * rb));
    b_t32 = in.A.p ? up256(sizeof(float) * (size_t)(s * rb)) : 0;
    b_flag = up256(sizeof(uint32_t) * (size_t)((wsrows + rb - 1) / rb));
    ws = static_cast<char*>(try_workspace(c, b_op + b_part + b_a + b_uf + b_t + b_t32 + b_flag, in.otherwise));
    if (cap == 64) break;
  }
  if (!ws) return false;
  auto take = [&](size_t bytes) {
    char* p = ws;
    ws += bytes;
    return p;
  };
  __nv_bfloat16* op = reinterpret_cast<__nv_bfloat16*>(take(b_op));
  float* part = reinterpret_cast<float*>(take(b_part));
  __nv_bfloat16* Ap = reinterpret_cast<__nv_bfloat16*>(take(b_a));
  __nv_bfloat16* uf = reinterpret_cast<__nv_bfloat16*>(take(b_uf));
  __nv_bfloat16* Tp = reinterpret_cast<__nv_bfloat16*>(take(b_t));
  float* T32 = reinterpret_cast<float*>(take(b_t32));
  uint32_t* flags = in.A.p ? reinterpret_cast<uint32_t*>(take(b_flag)) : nullptr;

  const int64_t nwin = (nrows + W - 1) / W;
  const float ybeta = y_beta(c, row0, row0 + nrows, nu);
  const float xbeta = (float)std::pow((double)nu, (double)nwin);
  if (flags) SKEMA_CUDA(cudaMemsetAsync(flags, 0, b_flag, c->stream));
  {
    StageScope st(c, ST_WINDOW);
    const X3Src so{c->omg.f32, c->omg.rs, k}, sp{c->psi.f32, c->psi.rs, s};
    x3_maps_kernel<<<grid_1d(c, (k + s) * ldn / 8, 16), 256, 0, c->stream>>>(so, sp, n, op, ldn, (k + s) * ldn, 1.f, 1,
                                                                            1, 0, 0, nullptr);
    SKEMA_LAUNCHED(c);
  }
  for (int64_t r = 0, i = 0; r < nrows; r += rb, ++i) {
    const int64_t wr = std::min(rb, nrows - r), R0 = row0 + r;
    const int64_t nrb = (wr + 63) / 64, ldw = pad8(wr), ps = nrb * 64 * n;
    uint32_t* flag = flags ? flags + i : nullptr;
    const X3Words words{flag, nullptr};
    const Mat Aw{in.A.p ? in.A.p + r * in.A.rs : nullptr, in.A.rs, in.A.cs};
    {
      StageScope st(c, ST_WINDOW);
      if (in.A.p)
        x3_block_planes(c, Aw, wr, n, Ap, ps, top, s > 0 ? std::max(-90, -102 - x3_exp(c->psi)) : -90, flag);
      else
        in.fill(R0, wr, Ap, ps);
      if (s > 0) {
        const X3Src su{c->ups.f32 + R0, c->ups.rs, k}, sf{c->phi.f32 + R0, c->phi.rs, s};  // cs = 1
        x3_maps_kernel<<<grid_1d(c, (k + s) * ldw / 8, 16), 256, 0, c->stream>>>(su, sf, wr, uf, ldw, (k + s) * ldw, nu,
                                                                                W, nwin, r, 0, nullptr);
        SKEMA_LAUNCHED(c);
      }
    }
    const X3A an{Ap, true, true, n, nrb, 0, 0}, at{Ap, true, false, n, nrb, 0, 0};
    {
      StageScope st(c, s > 0 ? ST_FUSED : ST_OMEGA);
      x3_gemm(c, an, X3B{op, ldn, (k + s) * ldn}, wr, k + s, n,
              tc::X3Out{c->Y + R0, 1, c->m, eta, ybeta, Tp, ldw, s * ldw, wr, k, k + s}, part, words);
    }
    if (s > 0) {
      const float xb = i == 0 ? xbeta : 1.f;
      {
        StageScope st(c, ST_UPSILON);
        x3_gemm(c, at, X3B{uf, ldw, (k + s) * ldw}, n, k, wr, tc::X3Out{c->X, 1, n, eta, xb, nullptr, 0, 0, n, k, k},
                part, words);
      }
      StageScope st(c, ST_PHI);
      x3_gemm(c, X3A{Tp, false, false, 0, 0, ldw, s * ldw}, X3B{uf + k * ldw, ldw, (k + s) * ldw}, s, s, wr,
              tc::X3Out{c->Z, 1, s, eta, xb, nullptr, 0, 0, s, s, s}, part, words);
    }
    if (flag) {
      const float xb = i == 0 ? xbeta : 1.f;
      X3Plain3 p{};
      p.g[0] = X3Plain{Aw.p, Aw.rs, Aw.cs, nullptr, 0, 0, c->omg.f32, c->omg.cs, c->omg.rs, c->Y + R0, 1, c->m,
                       wr, k, n, eta, ybeta, 1};
      p.n = 1;
      if (s > 0) {
        p.g[1] = X3Plain{Aw.p, Aw.rs, Aw.cs, nullptr, 0, 0, c->psi.f32, c->psi.cs, c->psi.rs, T32, 1, wr,
                         wr, s, n, 1.f, 0.f, 1};
        p.g[2] = X3Plain{nullptr, 0, 0, uf, ldw, (k + s) * ldw, Aw.p, Aw.rs, Aw.cs, c->X, n, 1, k, n, wr, eta, xb, 1};
        p.n = 3;
        p.scale = c->Z, p.nscale = s * s, p.by = xb;
      }
      x3_plain(c, p, flag);
      if (s > 0) {
        X3Plain3 z{};
        z.g[0] = X3Plain{nullptr, 0, 0, uf + k * ldw, ldw, (k + s) * ldw, T32, 1, wr, c->Z, s, 1, s, s, wr, eta, 1.f,
                         x3_plain_split(c, s, wr)};
        z.n = 1;
        x3_plain(c, z, flag);
      }
    }
  }
  y_rows_mark(c, row0, row0 + nrows);
  return true;
}

bool x3_update(skema_ctx* c, const X3Input& in, int64_t row0, int64_t nrows) {
  const float nu = (float)c->p.sketch_nu;
  if (nrows <= 0 || !(nu > 0.f)) return false;
  for (const Map* mp : {&c->ups, &c->omg, &c->phi, &c->psi})
    if (!x3_carries(*mp)) return false;
  // below this the launches and conversions cost more than the products
  if ((double)nrows * (double)c->n * (double)(2 * c->k + (c->spd ? 0 : c->s)) < 2e7) return false;
  const int64_t W = c->w, nwin = std::min((nrows + W - 1) / W, weight_windows(nu)), step = nwin * W;
  // maps so large that ordinary values (2^40) would be refused; kernel values are
  // at most one
  const int top = x3_top(c, std::min(step, nrows), nwin);
  if (top < (in.A.p ? 40 : 1)) return false;
  for (int64_t r = 0; r < nrows; r += step) {
    X3Input part = in;
    if (part.A.p) part.A.p += r * part.A.rs;
    // false at r = 0 only: every run asks for the same workspace
    if (!x3_windows(c, part, row0 + r, std::min(step, nrows - r), std::min(step, nrows), top)) return false;
  }
  return true;
}

}  // namespace skema
