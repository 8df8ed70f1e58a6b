// rbf.cu -- the Gauss RBF kernel input (GaussRBFWindow::get +
// GaussRBF::compute, src/Skema_Window.hpp:90-107, src/Skema_Kernel.cpp:6-81)
// and the standalone kernel-sketch forward/VJP pair.
//
// K(i, j) = exp(-gamma * sum_f (x_if - x_jf)^2) with explicit differences
// (the reference's formula, src/Skema_Kernel.cpp:37-44), and K(i, i) = 1
// (src/Skema_Kernel.cpp:62-74). Kernel rows are made a block at a time and
// consumed by the sketch products of the same block, so K never exists as a
// whole: as BF16 planes for the tensor-core FP32 form (rbf_planes_kernel, blocks
// of up to 2 GB that need not follow the windows), or as FP32 rows, a window at
// a time, for the SIMT form (rbf_tile_kernel).
//
// VJP of Y = K Omega~^T with respect to gamma and the points, given
// Ybar = dL/dY:  M = Ybar Omega~,  E = M o K,
//   dL/dgamma = -sum_ij E_ij d_ij^2,
//   dL/dx_i   = -2 gamma sum_j (E_ij + E_ji)(x_i - x_j)
//             = -2 gamma [ (rowsum(E)_i + colsum(E)_i) x_i - (E X)_i - (E^T X)_i ].
// Kernel tiles are recomputed in the backward pass, never stored.
#include <cuda_runtime.h>

#include <algorithm>

#include "internal.h"
#include "x3.h"

namespace skema {

size_t dense_scratch_bytes(const skema_ctx* c, int64_t wr);
void dense_window(skema_ctx* c, Mat Aw, int64_t R0, int64_t wr, float* T);

namespace {

constexpr int TT = 64;  // tile edge
constexpr int TD = 16;  // feature chunk

// MODE 0: out(i, j) = K.  MODE 1: out(i, j) <- out(i, j) * K (E = M o K) and
// accumulate -sum E d^2 into *dgamma, rowsum(E) into rsum[R0+i] and
// colsum(E) into csum[j].
template <int MODE>
__global__ void __launch_bounds__(256)
    rbf_tile_kernel(const float* __restrict__ P, int64_t prs, int64_t pcs, int64_t N, int64_t d,
                    float gamma, int64_t R0, int64_t wr, float* __restrict__ out, int64_t ldo,
                    double* __restrict__ dgamma, float* __restrict__ rsum, float* __restrict__ csum,
                    const uint32_t* __restrict__ run_if) {
  if (run_if && !x3_refused(*run_if)) return;
  __shared__ float xi[TD][TT + 1];
  __shared__ float xj[TD][TT + 1];
  __shared__ float red[256];
  const int tx = threadIdx.x & 15, ty = threadIdx.x >> 4;
  const int64_t tiles_j = (N + TT - 1) / TT;
  const int64_t tiles_i = (wr + TT - 1) / TT;
  for (int64_t tile = blockIdx.x; tile < tiles_i * tiles_j; tile += gridDim.x) {
    const int64_t i0 = (tile / tiles_j) * TT, j0 = (tile % tiles_j) * TT;
    float acc[4][4];
#pragma unroll
    for (int a = 0; a < 4; ++a)
#pragma unroll
      for (int b = 0; b < 4; ++b) acc[a][b] = 0.f;
    for (int64_t f0 = 0; f0 < d; f0 += TD) {
      for (int q = threadIdx.x; q < TD * TT; q += 256) {
        const int ff = q / TT, rr = q % TT;
        const int64_t f = f0 + ff;
        const int64_t gi = R0 + i0 + rr, gj = j0 + rr;
        xi[ff][rr] = (f < d && i0 + rr < wr) ? P[gi * prs + f * pcs] : 0.f;
        xj[ff][rr] = (f < d && gj < N) ? P[gj * prs + f * pcs] : 0.f;
      }
      __syncthreads();
#pragma unroll
      for (int ff = 0; ff < TD; ++ff) {
        float a[4], b[4];
#pragma unroll
        for (int u = 0; u < 4; ++u) {
          a[u] = xi[ff][ty + 16 * u];
          b[u] = xj[ff][tx + 16 * u];
        }
#pragma unroll
        for (int u = 0; u < 4; ++u)
#pragma unroll
          for (int v = 0; v < 4; ++v) {
            const float df = a[u] - b[v];
            acc[u][v] = fmaf(df, df, acc[u][v]);
          }
      }
      __syncthreads();
    }
    float gpart = 0.f;
    float rpart[4] = {0.f, 0.f, 0.f, 0.f};
    float cpart[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      const int64_t li = i0 + ty + 16 * u;
#pragma unroll
      for (int v = 0; v < 4; ++v) {
        const int64_t gj = j0 + tx + 16 * v;
        if (li < wr && gj < N) {
          const bool diag = (gj == R0 + li);
          const float kv = diag ? 1.f : expf(-gamma * acc[u][v]);
          float* op = out + li * ldo + gj;
          if (MODE == 0) {
            *op = kv;
          } else {
            const float e = *op * kv;
            *op = e;
            if (!diag) gpart += e * acc[u][v];
            rpart[u] += e;
            cpart[v] += e;
          }
        }
      }
    }
    if (MODE == 1) {
      // block reduction of the gamma partial
      red[threadIdx.x] = gpart;
      __syncthreads();
      for (int st = 128; st > 0; st >>= 1) {
        if (threadIdx.x < st) red[threadIdx.x] += red[threadIdx.x + st];
        __syncthreads();
      }
      if (threadIdx.x == 0) atomicAdd(dgamma, -(double)red[0]);
      __syncthreads();
#pragma unroll
      for (int u = 0; u < 4; ++u) {
        const int64_t li = i0 + ty + 16 * u;
        float r = rpart[u];
        // reduce over tx (16 lanes of one half-warp share ty)
        for (int o = 8; o > 0; o >>= 1) r += __shfl_xor_sync(0xffffffffu, r, o);
        if (tx == 0 && li < wr) atomicAdd(rsum + R0 + li, r);
      }
#pragma unroll
      for (int v = 0; v < 4; ++v) {
        const int64_t gj = j0 + tx + 16 * v;
        if (gj < N && cpart[v] != 0.f) atomicAdd(csum + gj, cpart[v]);
      }
    }
  }
}

// Kernel rows as the row-blocked BF16 planes of the tensor-core FP32 form
// (x3.h): K is split where it is made, so it is written once (6 bytes) and
// never as FP32. 64 rows x 128 points per CTA of 128 threads, 8 x 8 per thread
// (rows 4 t .. 4 t + 3 and 32 more on: eight lanes write 64 bytes of a plane's
// line), so four 16-byte shared loads feed 64 differences. Features go 16 at a time
// through two buffers, the next ones loaded during the current ones' sums; the
// last chunk stops at a multiple of four. FCONTIG: a point's features are
// contiguous (pcs = 1). Bound by the two FP32 instructions per difference:
// 40,000^2 kernel entries of d = 100 take 12.7 ms (8.8 at the FP32 rate; 17.5
// with scalar instructions, one buffer and whole chunks, 14.9 with the packed
// pairs of J kept in shared memory, whose reads then bound it, 13.3 with 4 x 8
// entries per thread).
//
// GRAD: the planes hold E = M o K with M = Ybar Omega~ formed beside the
// distances (k more FP32 instructions per entry; as a product of its own it
// cost an FP32 block written and read back: forward and adjoint at N = 20,000,
// d = 24, k = 65 took 8.0 ms, now 6.1, this kernel 3.1 of them), E_ii = 0 (the
// diagonal's terms of the gradient cancel), and the sums -E d^2, rowsum(E) and
// colsum(E) as rbf_tile_kernel<1> adds them; E's magnitudes are noted in *word.
struct RbfGrad {
  const float* Ybar;   // N x k row-major
  const float* omega;  // k x N row-major
  int64_t k;
  double* dgamma;
  float* rsum;
  float* csum;
  uint32_t big;  // x3_report's
  uint32_t* word;
};
// s += (a + b)^2, and s += a b, on two packed FP32 values, each rounded as FADD
// and FFMA do.
__device__ __forceinline__ void add_sq(unsigned long long& s, unsigned long long a, unsigned long long b) {
  unsigned long long t;
  asm("add.rn.f32x2 %0, %1, %2;" : "=l"(t) : "l"(a), "l"(b));
  asm("fma.rn.f32x2 %0, %1, %1, %0;" : "+l"(s) : "l"(t));
}
__device__ __forceinline__ void add_mul(unsigned long long& s, unsigned long long a, unsigned long long b) {
  asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(s) : "l"(a), "l"(b));
}
__device__ __forceinline__ unsigned long long twice(float x) {
  unsigned long long r;
  asm("mov.b64 %0, {%1, %1};" : "=l"(r) : "f"(x));
  return r;
}

constexpr int kTI = 64, kTJ = 128, kTF = 16, kPlThreads = 128;
struct RbfTile {
  float xi[2][kTF][kTI + 4];
  float xj[2][kTF][kTJ + 4];
};
// Over f < d: acc += (I(f, i) - J(f, j))^2 (DIST) or I(f, i) J(f, j) for this
// thread's 8 x 8 entries, packed by two rows. I(f, i) = Ip[i * irs + f * ics] for
// i < ni, else 0; J alike. FI, FJ: the f run is the contiguous one. What a thread
// stages: feature f + q (step) of point r + q (step), the offsets of the q
// constants. All threads are past the tile's last use when it returns.
template <bool FI, bool FJ, bool DIST>
__device__ __forceinline__ void rbf_pass(RbfTile& t, unsigned long long (&acc)[4][8], const float* __restrict__ Ip,
                                         int64_t irs, int64_t ics, int ni, const float* __restrict__ Jp, int64_t jrs,
                                         int64_t jcs, int nj, int64_t d) {
  constexpr int NI = kTF * kTI / kPlThreads, NJ = kTF * kTJ / kPlThreads;
  const int tid = threadIdx.x, tx = tid & 7, ty = tid >> 3;
  const int fi = FI ? tid & 15 : tid >> 6, ri = FI ? tid >> 4 : tid & 63;
  const int fj = FJ ? tid & 15 : 0, rj = FJ ? tid >> 4 : tid;
  const int64_t qi = FI ? 8 * irs : 2 * ics, qj = FJ ? 8 * jrs : jcs;
  const float* pi = Ip + ri * irs + fi * ics;
  const float* pj = Jp + rj * jrs + fj * jcs;
  float vi[NI], vj[NJ];
  auto load = [&](int64_t f0) {
    const int left = (int)min((int64_t)kTF, d - f0);
    const float* a = pi + f0 * ics;
    const float* b = pj + f0 * jcs;
#pragma unroll
    for (int q = 0; q < NI; ++q, a += qi)
      vi[q] = (fi + (FI ? 0 : 2 * q) < left && ri + (FI ? 8 * q : 0) < ni) ? __ldg(a) : 0.f;
#pragma unroll
    for (int q = 0; q < NJ; ++q, b += qj)
      vj[q] = (fj + (FJ ? 0 : q) < left && rj + (FJ ? 8 * q : 0) < nj) ? __ldg(b) : 0.f;
  };
  auto store = [&](int b) {
#pragma unroll
    for (int q = 0; q < NI; ++q) t.xi[b][fi + (FI ? 0 : 2 * q)][ri + (FI ? 8 * q : 0)] = vi[q];
#pragma unroll
    for (int q = 0; q < NJ; ++q) t.xj[b][fj + (FJ ? 0 : q)][rj + (FJ ? 8 * q : 0)] = DIST ? -vj[q] : vj[q];
  };
  load(0);
  store(0);
  __syncthreads();
  int buf = 0;
  for (int64_t f0 = 0; f0 < d; f0 += kTF, buf ^= 1) {
    if (f0 + kTF < d) load(f0 + kTF);
    const int nf = (int)min((int64_t)kTF, d - f0);
    for (int f4 = 0; f4 < nf; f4 += 4) {
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        const ulonglong2 a2 = *reinterpret_cast<const ulonglong2*>(&t.xi[buf][f4 + q][4 * tx]);
        const ulonglong2 h2 = *reinterpret_cast<const ulonglong2*>(&t.xi[buf][f4 + q][32 + 4 * tx]);
        const float4 b4 = *reinterpret_cast<const float4*>(&t.xj[buf][f4 + q][8 * ty]);
        const float4 c4 = *reinterpret_cast<const float4*>(&t.xj[buf][f4 + q][8 * ty + 4]);
        const unsigned long long a[4] = {a2.x, a2.y, h2.x, h2.y};
        const float b[8] = {b4.x, b4.y, b4.z, b4.w, c4.x, c4.y, c4.z, c4.w};
#pragma unroll
        for (int v = 0; v < 8; ++v) {
          const unsigned long long bb = twice(b[v]);
#pragma unroll
          for (int u = 0; u < 4; ++u) {
            if (DIST)
              add_sq(acc[u][v], a[u], bb);
            else
              add_mul(acc[u][v], a[u], bb);
          }
        }
      }
    }
    if (f0 + kTF < d) store(buf ^ 1);  // read last a chunk ago, before the barrier
    __syncthreads();
  }
}
__device__ __forceinline__ float half_of(unsigned long long x, int h) {
  return __uint_as_float((uint32_t)(x >> (32 * h)));
}

template <bool FCONTIG, bool GRAD>
__global__ void __launch_bounds__(kPlThreads, GRAD ? 2 : 3)
    rbf_planes_kernel(const float* __restrict__ P, int64_t prs, int64_t pcs, int64_t N, int64_t d, float gamma,
                      int64_t R0, int64_t wr, __nv_bfloat16* __restrict__ out, int64_t pstride, RbfGrad g) {
  __shared__ __align__(16) RbfTile t;
  const int tx = threadIdx.x & 7, ty = threadIdx.x >> 3;
  const int64_t tiles_j = (N + kTJ - 1) / kTJ, tiles_i = (wr + kTI - 1) / kTI;
  float top = 0.f;
  double gsum = 0.0;
  for (int64_t tile = blockIdx.x; tile < tiles_i * tiles_j; tile += gridDim.x) {
    const int64_t ib = tile / tiles_j, i0 = ib * kTI, j0 = (tile - ib * tiles_j) * kTJ;
    const int ni = (int)min((int64_t)kTI, wr - i0), nj = (int)min((int64_t)kTJ, N - j0);
    // two adjacent rows per 64-bit register: packed FP32 has the rate of the
    // scalar instructions at half their issue slots, which the loads and the
    // exponentials need
    unsigned long long acc[4][8], mac[GRAD ? 4 : 1][8];
#pragma unroll
    for (int a = 0; a < 4; ++a)
#pragma unroll
      for (int b = 0; b < 8; ++b) {
        acc[a][b] = 0ull;
        if (GRAD) mac[GRAD ? a : 0][b] = 0ull;
      }
    rbf_pass<FCONTIG, FCONTIG, true>(t, acc, P + (R0 + i0) * prs, prs, pcs, ni, P + j0 * prs, prs, pcs, nj, d);
    if constexpr (GRAD)
      rbf_pass<true, false, false>(t, mac, g.Ybar + (R0 + i0) * g.k, g.k, 1, ni, g.omega + j0, 1, N, nj, g.k);
    float rpart[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f}, gpart = 0.f;
    const int64_t dg = R0 + i0 - j0;  // the diagonal: j = i + dg within the tile
#pragma unroll
    for (int v = 0; v < 8; ++v) {
      const int lj = 8 * ty + v;
      const bool in = lj < nj;
      float cpart = 0.f;
      __nv_bfloat162 q[3][4];
#pragma unroll
      for (int u = 0; u < 4; ++u) {
        float kk[2];
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          const int li = 4 * tx + 32 * (u >> 1) + 2 * (u & 1) + h;
          const bool diag = (int64_t)lj == li + dg;
          const float d2 = half_of(acc[u][v], h);
          float kv = expf(-gamma * d2);
          if (GRAD) {
            kv = (in && li < ni && !diag) ? half_of(mac[GRAD ? u : 0][v], h) * kv : 0.f;
            x3_note(top, kv);
            gpart = fmaf(kv, d2, gpart);
            rpart[2 * u + h] += kv;
            cpart += kv;
          } else {
            kv = li >= ni ? 0.f : diag ? 1.f : kv;
          }
          kk[h] = kv;
        }
        tc::split3x2(kk[0], kk[1], q[0][u], q[1][u], q[2][u]);
      }
      if (in) {
        __nv_bfloat16* dp = out + (ib * N + j0 + lj) * 64 + 4 * tx;
#pragma unroll
        for (int p = 0; p < 3; ++p) {
          *reinterpret_cast<uint2*>(dp + p * pstride) = *reinterpret_cast<const uint2*>(&q[p][0]);
          *reinterpret_cast<uint2*>(dp + p * pstride + 32) = *reinterpret_cast<const uint2*>(&q[p][2]);
        }
      }
      if (GRAD) {  // eight lanes hold the column's 64 rows
#pragma unroll
        for (int o = 4; o > 0; o >>= 1) cpart += __shfl_xor_sync(0xffffffffu, cpart, o);
        if (tx == 0 && in) atomicAdd(g.csum + j0 + lj, cpart);
      }
    }
    if (GRAD) {
      gsum += (double)gpart;
      // row sums over the 16 groups of columns
      float* red = &t.xj[0][0][0];
#pragma unroll
      for (int e = 0; e < 8; ++e) red[ty * kTI + 4 * tx + 32 * (e >> 2) + (e & 3)] = rpart[e];
      __syncthreads();
      if (threadIdx.x < kTI && (int)threadIdx.x < ni) {
        float r = 0.f;
#pragma unroll
        for (int q = 0; q < 16; ++q) r += red[q * kTI + threadIdx.x];
        atomicAdd(g.rsum + R0 + i0 + threadIdx.x, r);
      }
      __syncthreads();
    }
  }
  if (GRAD) {
    x3_report(top, g.big, g.word);
    for (int o = 16; o > 0; o >>= 1) gsum += __shfl_xor_sync(0xffffffffu, gsum, o);
    if ((threadIdx.x & 31) == 0) atomicAdd(g.dgamma, -gsum);
  }
}

// dX = -2 gamma * (r o X - S), r = rsum + csum (N), S = S1 + S2 (N x d).
__global__ void rbf_dx_kernel(const float* __restrict__ P, int64_t prs, int64_t pcs, int64_t N,
                              int64_t d, float gamma, const float* __restrict__ rsum,
                              const float* __restrict__ csum, const float* __restrict__ S,
                              float* __restrict__ dX) {
  const int64_t total = N * d;
  for (int64_t q = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; q < total;
       q += (int64_t)gridDim.x * blockDim.x) {
    const int64_t i = q / d, f = q - i * d;
    const float r = rsum[i] + csum[i];
    dX[q] = -2.f * gamma * (r * P[i * prs + f * pcs] - S[q]);
  }
}

int grid_cap(const skema_ctx* c, int64_t want, int per_sm) {
  return (int)std::max<int64_t>(1, std::min<int64_t>(want, (int64_t)c->sm_count * per_sm));
}

void launch_tile(skema_ctx* c, int mode, Mat P, int64_t N, int64_t d, float gamma, int64_t R0,
                 int64_t wr, float* out, int64_t ldo, double* dg, float* rs, float* cs) {
  const int64_t tiles = ((wr + TT - 1) / TT) * ((N + TT - 1) / TT);
  const int grid = grid_cap(c, tiles, 8);
  if (mode == 0)
    rbf_tile_kernel<0><<<grid, 256, 0, c->stream>>>(P.p, P.rs, P.cs, N, d, gamma, R0, wr, out, ldo,
                                                    dg, rs, cs, c->run_if);
  else
    rbf_tile_kernel<1><<<grid, 256, 0, c->stream>>>(P.p, P.rs, P.cs, N, d, gamma, R0, wr, out, ldo,
                                                    dg, rs, cs, c->run_if);
  SKEMA_LAUNCHED(c);
}

// Rows per scratch block so that a w x N FP32 block stays near 1 GiB.
int64_t rows_per_block(int64_t N, int64_t cap_rows) {
  const int64_t budget = (int64_t)1 << 28;  // floats
  return std::max<int64_t>(1, std::min<int64_t>(cap_rows, budget / std::max<int64_t>(N, 1)));
}

}  // namespace

void rbf_window_block(skema_ctx* c, Mat P, int64_t N, int64_t d, float gamma, int64_t R0,
                      int64_t wr, float* out, int64_t ldo) {
  launch_tile(c, 0, P, N, d, gamma, R0, wr, out, ldo, nullptr, nullptr, nullptr);
}

void rbf_update(skema_ctx* c, Mat P, int64_t npts, int64_t d, int64_t row0, int64_t nrows) {
  if (c->residual_pass) {
    residual_rbf(c, P, npts, d, row0, nrows);
    return;
  }
  if (!c->spd && c->p.precision == SKEMA_PREC_BF16 && rbf_tc_supported(c, d)) {
    // tensor-core form: kernel tiles regenerated inside the sketch kernels
    rbf_tc_update(c, P, npts, d, row0, nrows);
    return;
  }
  const int64_t W = c->w;
  const int64_t N = npts;
  const float gamma = (float)c->p.kernel_gamma;
  const int64_t wmax = std::min(W, nrows);
  const size_t kbytes = (sizeof(float) * (size_t)(wmax * N) + 255) / 256 * 256;
  if (c->p.precision == SKEMA_PREC_FP32 && c->p.dim_redux == SKEMA_MAP_GAUSS && gamma >= 0.f) {
    X3Input in{Mat{nullptr, 0, 0}, [&](int64_t R0, int64_t wr, __nv_bfloat16* planes, int64_t pstride) {
                 const int64_t tiles = ((wr + 63) / 64) * ((N + 127) / 128);
                 auto kern = P.cs == 1 ? rbf_planes_kernel<true, false> : rbf_planes_kernel<false, false>;
                 kern<<<grid_cap(c, tiles, 3), kPlThreads, 0, c->stream>>>(P.p, P.rs, P.cs, N, d, gamma, R0, wr,
                                                                           planes, pstride, RbfGrad{});
                 SKEMA_LAUNCHED(c);
               },
               kbytes + dense_scratch_bytes(c, wmax)};
    if (x3_update(c, in, row0, nrows)) return;
  }
  char* ws = (char*)workspace(c, kbytes + dense_scratch_bytes(c, wmax));
  float* Kw = (float*)ws;
  float* T = (float*)(ws + kbytes);
  for (int64_t r = 0; r < nrows; r += W) {
    const int64_t wr = std::min(W, nrows - r);
    const int64_t R0 = row0 + r;
    {
      StageScope st(c, ST_WINDOW);
      launch_tile(c, 0, P, N, d, gamma, R0, wr, Kw, N, nullptr, nullptr, nullptr);
    }
    dense_window(c, Mat{Kw, N, 1}, R0, wr, T);
  }
}

// Room for the K-split partial products of the FP32 forward and adjoint
// (a window's rows times k or d, at most 16 splits).
constexpr int64_t kRbfPartFloats = (int64_t)4 << 20;

size_t up256(size_t b) { return (b + 255) / 256 * 256; }

// Y = K Omega~^T by kernel blocks of wb rows in Kw and SIMT products.
static void rbf_fwd_plain(skema_ctx* c, const float* pts, int64_t N, int64_t d, float gamma, const float* omega,
                          int64_t k, float* Y, int64_t wb, float* Kw, float* part) {
  for (int64_t r = 0; r < N; r += wb) {
    const int64_t wr = std::min(wb, N - r);
    launch_tile(c, 0, Mat{pts, d, 1}, N, d, gamma, r, wr, Kw, N, nullptr, nullptr, nullptr);
    // Y(r:r+wr, :) = K_w Omega~^T ; B(kk=j, col=q) = omega[q*N + j]
    sgemm_split(c, wr, k, N, 1.f, Mat{Kw, N, 1}, Mat{omega, 1, N}, 0.f, MatOut{Y + r * k, k, 1}, part,
                kRbfPartFloats);
  }
}

// The adjoint's sums (rs, cs, S, *dgamma, zeroed beforehand) by blocks of wb
// rows of M and E in one buffer.
static void rbf_vjp_plain(skema_ctx* c, const float* pts, int64_t N, int64_t d, float gamma, const float* omega,
                          int64_t k, const float* Ybar, double* dgamma, float* rs, float* cs, float* S, int64_t wb,
                          float* E, float* part) {
  const Mat P{pts, d, 1};
  for (int64_t r = 0; r < N; r += wb) {
    const int64_t wr = std::min(wb, N - r);
    // M_w = Ybar_w Omega~   (wr x N)
    sgemm(c, wr, N, k, 1.f, Mat{Ybar + r * k, k, 1}, Mat{omega, N, 1}, 0.f, MatOut{E, N, 1});
    // E_w = M_w o K_w, with the gamma / row / column partial sums
    launch_tile(c, 1, P, N, d, gamma, r, wr, E, N, dgamma, rs, cs);
    // S(r:r+wr, :) += E_w X ;  S += E_w^T X_w
    sgemm_split(c, wr, d, N, 1.f, Mat{E, N, 1}, Mat{pts, d, 1}, 1.f, MatOut{S + r * d, d, 1}, part, kRbfPartFloats);
    sgemm(c, N, d, wr, 1.f, Mat{E, 1, N}, Mat{pts + r * d, d, 1}, 1.f, MatOut{S, d, 1});
  }
}

// Below this many kernel entries times columns the conversions and launches of
// the tensor-core form cost more than its products save.
static bool rbf_pair_small(int64_t N, int64_t d, int64_t k) { return (double)N * N * (double)(k + d) < 2e8; }

// Rows per block of the tensor-core forms, `bytes` per kernel entry: equal
// blocks, a multiple of 64, within about 1 GB.
static int64_t rbf_rows_x3(int64_t N, int64_t bytes) {
  const int64_t cap = std::max<int64_t>(64, ((int64_t)1 << 30) / (bytes * N) / 64 * 64);
  const int64_t nb = (N + cap - 1) / cap;
  return ((N + nb - 1) / nb + 63) / 64 * 64;
}

struct RunIf {  // the SIMT kernels launched in this scope run when *flag is refused
  skema_ctx* c;
  RunIf(skema_ctx* ctx, const uint32_t* flag) : c(ctx) { c->run_if = flag; }
  ~RunIf() { c->run_if = nullptr; }
};

static void launch_planes(skema_ctx* c, const float* pts, int64_t N, int64_t d, float gamma, int64_t r, int64_t wr,
                          __nv_bfloat16* planes, int64_t pstride, const RbfGrad* g) {
  const int64_t tiles = ((wr + 63) / 64) * ((N + 127) / 128);
  if (g)
    rbf_planes_kernel<true, true><<<grid_cap(c, tiles, 2), kPlThreads, 0, c->stream>>>(pts, d, 1, N, d, gamma, r, wr,
                                                                                       planes, pstride, *g);
  else
    rbf_planes_kernel<true, false><<<grid_cap(c, tiles, 3), kPlThreads, 0, c->stream>>>(pts, d, 1, N, d, gamma, r, wr,
                                                                                        planes, pstride, RbfGrad{});
  SKEMA_LAUNCHED(c);
}

// The forward product on the tensor cores: kernel planes a block of rows at a
// time, Y_w = K_w Omega~^T. When Omega~ is refused (x3.h), the SIMT form behind it
// runs (K has ones on its diagonal). False when the workspace is not to be had.
static bool rbf_fwd_x3(skema_ctx* c, const float* pts, int64_t N, int64_t d, float gamma, const float* omega, int64_t k,
                       float* Y) {
  if (rbf_pair_small(N, 0, k)) return false;
  const int64_t ldN = (N + 7) / 8 * 8, rb = rbf_rows_x3(N, 6);
  const size_t b_o = up256(2 * (size_t)(3 * k * ldN)), b_k = up256(2 * (size_t)(3 * rb * N)),
               b_p = up256(std::max(x3_part_bytes(c), sizeof(float) * (size_t)kRbfPartFloats));
  char* ws = static_cast<char*>(try_workspace(c, b_o + b_k + b_p + 256));
  if (!ws) return false;
  __nv_bfloat16* Op = reinterpret_cast<__nv_bfloat16*>(ws);
  __nv_bfloat16* Kp = reinterpret_cast<__nv_bfloat16*>(ws + b_o);
  float* part = reinterpret_cast<float*>(ws + b_o + b_k);
  uint32_t* flag = reinterpret_cast<uint32_t*>(ws + b_o + b_k + b_p);
  const X3Words words{flag, nullptr};
  SKEMA_CUDA(cudaMemsetAsync(flag, 0, sizeof(uint32_t), c->stream));
  // sums of N products with values of K, at most one
  x3_row_planes(c, omega, N, k, N, Op, ldN, k * ldN, std::min(100, 126 - x3_log2(N)), flag);
  for (int64_t r = 0; r < N; r += rb) {
    const int64_t wr = std::min(rb, N - r), nrb = (wr + 63) / 64;
    launch_planes(c, pts, N, d, gamma, r, wr, Kp, nrb * 64 * N, nullptr);
    x3_gemm(c, X3A{Kp, true, true, N, nrb, 0, 0}, X3B{Op, ldN, k * ldN}, wr, k, N,
            tc::X3Out{Y + r * k, k, 1, 1.f, 0.f, nullptr, 0, 0, wr, k, k}, part, words);
  }
  RunIf second(c, flag);
  rbf_fwd_plain(c, pts, N, d, gamma, omega, k, Y, std::max<int64_t>(1, (int64_t)(b_k / 4) / N),
                reinterpret_cast<float*>(Kp), part);
  return true;
}

// The adjoint's sums on the tensor cores, a block of rows at a time: E_w = M_w o
// K_w as planes with the sums, then E_w X and E_w^T X_w from the same planes. As
// for the forward, the SIMT form follows when X or a block's E is refused, over
// zeroed sums.
static bool rbf_vjp_x3(skema_ctx* c, const float* pts, int64_t N, int64_t d, float gamma, const float* omega, int64_t k,
                       const float* Ybar, float* dpts, double* dgamma) {
  if (rbf_pair_small(N, d, k)) return false;
  const int64_t ldN = (N + 7) / 8 * 8, rb = rbf_rows_x3(N, 6);
  const size_t b_x = up256(2 * (size_t)(3 * d * ldN)), b_e = up256(2 * (size_t)(3 * rb * N)),
               b_p = up256(std::max(x3_part_bytes(c), sizeof(float) * (size_t)kRbfPartFloats)),
               b_v = up256(4 * (size_t)N), b_s = up256(4 * (size_t)(N * d)),
               b_w = up256(4 * (size_t)(1 + (N + rb - 1) / rb));
  char* ws = static_cast<char*>(try_workspace(c, b_x + b_e + b_p + 2 * b_v + b_s + b_w));
  if (!ws) return false;
  auto take = [&](size_t b) {
    char* q = ws;
    ws += b;
    return q;
  };
  __nv_bfloat16* Xp = reinterpret_cast<__nv_bfloat16*>(take(b_x));
  __nv_bfloat16* Ep = reinterpret_cast<__nv_bfloat16*>(take(b_e));
  float* part = reinterpret_cast<float*>(take(b_p));
  float* rs = reinterpret_cast<float*>(take(b_v));
  float* cs = reinterpret_cast<float*>(take(b_v));
  float* S = reinterpret_cast<float*>(take(b_s));
  uint32_t* flag = reinterpret_cast<uint32_t*>(take(b_w));  // X's and the call's word, then one per block
  // the sums and the words behind them
  SKEMA_CUDA(cudaMemsetAsync(rs, 0, 2 * b_v + b_s + b_w, c->stream));
  SKEMA_CUDA(cudaMemsetAsync(dgamma, 0, sizeof(double), c->stream));
  // sums of N products of E and X: points far below 2^36, cotangents anywhere
  const int top_x = 36, top_e = std::min(100, 126 - x3_log2(N) - top_x);
  x3_transposed_planes(c, pts, d, N, d, Xp, ldN, d * ldN, 1.f, 1, 1, 0, top_x, flag);
  for (int64_t r = 0, i = 1; r < N; r += rb, ++i) {
    const int64_t wr = std::min(rb, N - r), nrb = (wr + 63) / 64;
    const X3Words words{flag + i, flag};
    const RbfGrad g{Ybar, omega, k, dgamma, rs, cs, x3_bits(top_e), flag + i};
    launch_planes(c, pts, N, d, gamma, r, wr, Ep, nrb * 64 * N, &g);
    x3_gemm(c, X3A{Ep, true, true, N, nrb, 0, 0}, X3B{Xp, ldN, d * ldN}, wr, d, N,
            tc::X3Out{S + r * d, d, 1, 1.f, 1.f, nullptr, 0, 0, wr, d, d}, part, words);
    x3_gemm(c, X3A{Ep, true, false, N, nrb, 0, 0}, X3B{Xp + r, ldN, d * ldN}, N, d, wr,
            tc::X3Out{S, d, 1, 1.f, 1.f, nullptr, 0, 0, N, d, d}, part, words);
  }
  {
    RunIf second(c, flag);
    scale_block(c, MatOut{rs, (int64_t)(2 * b_v + b_s) / 4, 1}, 1, (int64_t)(2 * b_v + b_s) / 4, 0.f);
    scale_block(c, MatOut{reinterpret_cast<float*>(dgamma), 2, 1}, 1, 2, 0.f);
    rbf_vjp_plain(c, pts, N, d, gamma, omega, k, Ybar, dgamma, rs, cs, S, std::max<int64_t>(1, (int64_t)(b_e / 4) / N),
                  reinterpret_cast<float*>(Ep), part);
  }
  rbf_dx_kernel<<<grid_cap(c, (N * d + 255) / 256, 16), 256, 0, c->stream>>>(pts, d, 1, N, d, gamma, rs, cs, S, dpts);
  SKEMA_LAUNCHED(c);
  return true;
}

void rbf_fwd(skema_ctx* c, const float* pts, int64_t N, int64_t d, double gamma,
             const float* omega, int64_t k, float* Y) {
  if (rbf_pair_tc_supported(c, d, k, gamma)) {
    rbf_fwd_tc(c, pts, N, d, gamma, omega, k, Y);
    return;
  }
  if (rbf_fwd_x3(c, pts, N, d, (float)gamma, omega, k, Y)) return;
  const int64_t wb = rows_per_block(N, N);
  const size_t kb = up256(sizeof(float) * (size_t)(wb * N));
  char* ws = (char*)workspace(c, kb + sizeof(float) * (size_t)kRbfPartFloats);
  rbf_fwd_plain(c, pts, N, d, (float)gamma, omega, k, Y, wb, (float*)ws, (float*)(ws + kb));
}

void rbf_vjp(skema_ctx* c, const float* pts, int64_t N, int64_t d, double gamma,
             const float* omega, int64_t k, const float* Ybar, float* dpts, double* dgamma) {
  if (rbf_pair_tc_supported(c, d, k, gamma)) {
    rbf_vjp_tc(c, pts, N, d, gamma, omega, k, Ybar, dpts, dgamma);
    return;
  }
  if (rbf_vjp_x3(c, pts, N, d, (float)gamma, omega, k, Ybar, dpts, dgamma)) return;
  const int64_t wb = rows_per_block(N, N);
  const size_t eb = up256(sizeof(float) * (size_t)(wb * N)), vb = up256(sizeof(float) * (size_t)N),
               sb = up256(sizeof(float) * (size_t)(N * d));
  char* ws = (char*)workspace(c, eb + 2 * vb + sb + sizeof(float) * (size_t)kRbfPartFloats);
  float* rs = (float*)(ws + eb);
  float* cs = (float*)(ws + eb + vb);
  float* S = (float*)(ws + eb + 2 * vb);
  float* part = (float*)(ws + eb + 2 * vb + sb);  // K-split partial products
  SKEMA_CUDA(cudaMemsetAsync(rs, 0, 2 * vb + sb, c->stream));
  SKEMA_CUDA(cudaMemsetAsync(dgamma, 0, sizeof(double), c->stream));
  rbf_vjp_plain(c, pts, N, d, (float)gamma, omega, k, Ybar, dgamma, rs, cs, S, wb, (float*)ws, part);
  rbf_dx_kernel<<<grid_cap(c, (N * d + 255) / 256, 16), 256, 0, c->stream>>>(
      pts, d, 1, N, d, (float)gamma, rs, cs, S, dpts);
  SKEMA_LAUNCHED(c);
}

}  // namespace skema
