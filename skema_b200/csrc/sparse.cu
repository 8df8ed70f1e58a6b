// sparse.cu -- the sparse-map and sparse-input forms of the sketch update.
//
//   CSR x SparseSign (update(crs, SparseSign), src/Skema_SketchySVD.cpp:319-335):
//     y_i  = sum_j a_ij Omega(j, :)      Omega stored n x k, zeta per row
//     X(r,:) += sign * A(c, :)           for each Upsilon entry (r, c) in the window
//     Z(r,:) += sign * A(c, :) Psi       for each Phi entry (r, c) in the window
//   The reference forms these with spgemm + densify
//   (src/Skema_DimRedux_SparseSign.cpp:53-111) after a serial col_subview
//   (:125-155). Here all windows of a call are handled by two launches: a
//   streaming kernel for Y (the HBM-bound part: every nonzero read once, every
//   Y element written once) and a tiny kernel for the X/Z entries, whose window
//   weights eta*nu^(W-1-w) reproduce the per-window axpy sequence.
//   CSR x Gauss (src/Skema_SketchySVD.cpp:296-316), dense x SparseSign
//   (:271-293) and the SketchySPD updates (:896-932) follow.
//
// Y is column-major (m x k, ld = m), the reference's LayoutLeft.
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>

#include "internal.h"
#include "tc_x3.cuh"
#include "x3.h"

namespace skema {

namespace {

int grid_cap(const skema_ctx* c, int64_t want, int per_sm) {
  return (int)std::max<int64_t>(1, std::min<int64_t>(want, (int64_t)c->sm_count * per_sm));
}

// ---------------------------------------------------------------------------
// Y rows of a CSR block times a stored-transposed SparseSign map (n rows of
// zeta entries over k columns).
//
// One thread per input row. Each warp owns 32 consecutive rows and a
// bin-major accumulator acc[r * 32 + lane] in shared memory: lane l adds
// +-a_ij into the k bins of its own row only, so the updates need no
// atomics and every shared access of a warp hits 32 distinct banks. After
// the rows are done, bin r of the 32 rows is one coalesced 128-byte store
// into the column-major Y. Nonzeros go through the read-only path (the
// warp's 32 rows are contiguous in col/val, so L1 serves the lanes' strided
// walk). This general form reads zeta 32-bit map words per input column
// (column | sign << 31); csr_ssign_y16_kernel below is the form for zeta = 8
// and k <= 256.
// ---------------------------------------------------------------------------
__device__ __forceinline__ void ssign_apply(float* __restrict__ my, const uint32_t* __restrict__ omg32, int zeta,
                                            int32_t j, float a) {
  for (int t = 0; t < zeta; ++t) {
    const uint32_t w = __ldg(omg32 + (int64_t)j * zeta + t);
    my[(w & 0x7fffffffu) * 32] += (w >> 31) ? -a : a;
  }
}

template <int UNR>
__global__ void __launch_bounds__(128)
    csr_ssign_y_kernel(const int64_t* __restrict__ rowptr, const int32_t* __restrict__ col,
                       const float* __restrict__ val, int64_t col_offset, int64_t nrows,
                       const uint32_t* __restrict__ omg32,
                       int zeta, int k, int ncol, float* __restrict__ Y, int64_t ldy, float alpha,
                       float beta) {
  extern __shared__ float acc_all[];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
  float* my = acc_all + (size_t)warp * k * 32 + lane;  // bins of this lane's row: my[r * 32]
  for (int r = 0; r < k; ++r) my[r * 32] = 0.f;
  const int64_t ntiles = (nrows + 31) / 32;
  for (int64_t tile = (int64_t)blockIdx.x * nw + warp; tile < ntiles;
       tile += (int64_t)gridDim.x * nw) {
    const int64_t i = tile * 32 + lane;
    const bool live = i < nrows;
    int64_t b = live ? __ldg(rowptr + i) - col_offset : 0;
    int64_t e = __shfl_down_sync(0xffffffffu, b, 1);
    if (lane == 31 || i + 1 >= nrows) e = live ? __ldg(rowptr + i + 1) - col_offset : 0;
    int64_t p = b;
    for (; p + UNR <= e; p += UNR) {
      int32_t jj[UNR];
      float aa[UNR];
#pragma unroll
      for (int u = 0; u < UNR; ++u) {
        jj[u] = __ldg(col + p + u);
        aa[u] = __ldg(val + p + u);
      }
#pragma unroll
      for (int u = 0; u < UNR; ++u)
        if ((unsigned)jj[u] < (unsigned)ncol) ssign_apply(my, omg32, zeta, jj[u], aa[u]);
    }
    for (; p < e; ++p) {
      const int32_t j = __ldg(col + p);
      if ((unsigned)j < (unsigned)ncol) ssign_apply(my, omg32, zeta, j, __ldg(val + p));
    }
    if (live) {
      float* yp = Y + i;
      for (int r = 0; r < k; ++r) {
        const float v = my[r * 32];
        my[r * 32] = 0.f;
        if (beta == 0.f)
          __stcs(yp + r * ldy, alpha * v);
        else
          yp[r * ldy] = fmaf(beta, yp[r * ldy], alpha * v);
      }
    }
  }
}

// The same Y rows for the map's 16-bit offset form (zeta = 8, k <= 256):
// each entry is the byte offset of its bin in the warp's accumulator, the
// sign in bit 15 and a same-bin-as-previous flag in bit 0 (pack16_kernel).
// Per nonzero the eight bin loads are issued together, then the eight stores
// in entry order; a flagged entry adds to the previous entry's sum instead of
// its own (stale) load, so every bin still sees its additions in entry order
// and Y is bit-identical to one read-modify-write per entry.
// The work is pipelined across each warp's tiles: the next tile's row range
// is loaded when a tile starts and its first U nonzeros with the current
// tile's last batch, so their latency overlaps the apply and the write-out.
// Map rows are gathered through L2 only (.cg): 1e7 random 16-byte gathers
// would otherwise evict the col/val lines that the lanes' row walks reuse
// from L1. The write-out moves four bins per 16-byte access (lane -> bin
// r0 + lane / 8, rows 4 (lane % 8) .. + 3) and clears them in the same pass.
// The launch keeps about 128 KB of bins per SM and gives the rest of the
// unified L1 / shared memory to L1, which the row walks need (measured on the
// 1e6 x 1e5, 1e7-nonzero case: 48 KB less L1 cost 8 %, 96 KB less 34 %).
__device__ __forceinline__ float bin_ld(uint32_t addr) {
  float x;
  asm volatile("ld.shared.f32 %0, [%1];" : "=f"(x) : "r"(addr) : "memory");
  return x;
}
__device__ __forceinline__ void bin_st(uint32_t addr, float v) {
  asm volatile("st.shared.f32 [%0], %1;" ::"r"(addr), "f"(v) : "memory");
}

__device__ __forceinline__ void ssign_apply8(uint32_t base, uint4 wv, float a) {
  const uint32_t abits = __float_as_uint(a);
  const uint32_t e[8] = {wv.x & 0xffffu, wv.x >> 16, wv.y & 0xffffu, wv.y >> 16,
                         wv.z & 0xffffu, wv.z >> 16, wv.w & 0xffffu, wv.w >> 16};
  float v[8];
#pragma unroll
  for (int t = 0; t < 8; ++t) v[t] = bin_ld(base + (e[t] & 0x7f80u));
  float prev = 0.f;
#pragma unroll
  for (int t = 0; t < 8; ++t) {
    const float nv = ((e[t] & 1u) ? prev : v[t]) + __uint_as_float(abits ^ ((e[t] << 16) & 0x80000000u));
    bin_st(base + (e[t] & 0x7f80u), nv);
    prev = nv;
  }
}

// (A form with one red.shared.add per map entry instead of the load and
// store measured 30 % slower: 0.170 against 0.131 ms on the 1e6 x 1e5 case.)
//
// S = 4: a row is cut into four equal runs of nonzeros in four adjacent lanes,
// whose bins are added at the write-out, (0 + 1) + (2 + 3). For calls of few
// rows, whose time is the walk along the longest row: 2,000 rows of 0 to 200
// entries take 16 us against 35. (A warp per row with the bins in its lanes took
// 42 to 62.) The line between the two is at launch_csr_ssign_y.
template <int U, int S>
__global__ void __launch_bounds__(128)
    csr_ssign_y16_kernel(const int64_t* __restrict__ rowptr, const int32_t* __restrict__ col,
                         const float* __restrict__ val, int64_t col_offset, int64_t nrows,
                         const uint4* __restrict__ omg16, int k, int ncol, float* __restrict__ Y, int64_t ldy,
                         float alpha, float beta) {
  extern __shared__ __align__(16) float acc_all[];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
  float* bins = acc_all + (size_t)warp * k * 32;
  const uint32_t base = (uint32_t)__cvta_generic_to_shared(bins + lane);
  float4* bins4 = reinterpret_cast<float4*>(bins);
  const float4 z4 = make_float4(0.f, 0.f, 0.f, 0.f);
  for (int q = lane; q < k * 8; q += 32) bins4[q] = z4;
  __syncwarp();
  constexpr int R = 32 / S;  // rows per tile
  const int64_t ntiles = (nrows + R - 1) / R;
  const int64_t tstride = (int64_t)gridDim.x * nw;
  const bool vec = (reinterpret_cast<uintptr_t>(Y) & 15) == 0 && ldy % 4 == 0;
  int64_t tile = (int64_t)blockIdx.x * nw + warp;
  auto row_range = [&](int64_t t, int64_t& b, int64_t& e) {
    const int64_t i = t * R + lane / S;
    b = 0, e = 0;
    if (t < ntiles && i < nrows) b = __ldg(rowptr + i) - col_offset, e = __ldg(rowptr + i + 1) - col_offset;
    if (S > 1) {
      const int64_t len = (e - b + S - 1) / S;
      b = min(e, b + (lane % S) * len);
      e = min(e, b + len);
    }
  };
  auto load_batch = [&](int64_t q0, int64_t q1, int32_t* jj, float* aa) {
#pragma unroll
    for (int u = 0; u < U; ++u) {
      jj[u] = -1, aa[u] = 0.f;
      if (q0 + u < q1) jj[u] = __ldcs(col + q0 + u), aa[u] = __ldcs(val + q0 + u);
    }
  };
  int64_t b, e;
  row_range(tile, b, e);
  int32_t jj[U];
  float aa[U];
  load_batch(b, e, jj, aa);
  for (; tile < ntiles; tile += tstride) {
    int64_t nb, ne;
    row_range(tile + tstride, nb, ne);
    for (int64_t p = b;; p += U) {
      uint4 ww[U];
#pragma unroll
      for (int u = 0; u < U; ++u)
        ww[u] = (unsigned)jj[u] < (unsigned)ncol ? __ldcg(omg16 + jj[u]) : make_uint4(0u, 0u, 0u, 0u);
      // the next batch: the rest of this row, else the next tile's first
      const bool more = p + U < e;
      int32_t j2[U];
      float a2[U];
      load_batch(more ? p + U : nb, more ? e : ne, j2, a2);
#pragma unroll
      for (int u = 0; u < U; ++u)
        if ((unsigned)jj[u] < (unsigned)ncol) ssign_apply8(base, ww[u], aa[u] * alpha);
#pragma unroll
      for (int u = 0; u < U; ++u) jj[u] = j2[u], aa[u] = a2[u];
      if (!more) break;
    }
    __syncwarp();
    const int64_t r0 = tile * R;
    if (S == 4) {
      // row lane % 8, bins lane / 8, + 4, ..: four lanes' bins lie side by side
      // (four at a time: what beta scales is loaded ahead of the stores)
      const int64_t i = r0 + (lane & 7);
      const bool in = i < nrows, last = tile + tstride >= ntiles;
      float* yp = Y + i + (lane >> 3) * ldy;
      for (int r = lane >> 3; r < k; r += 16, yp += 16 * ldy) {
        float4* bp = bins4 + r * 8 + (lane & 7);
        float4 q[4];
        float o[4];
#pragma unroll
        for (int u = 0; u < 4; ++u) {
          q[u] = r + 4 * u < k ? bp[32 * u] : z4;
          o[u] = beta != 0.f && in && r + 4 * u < k ? yp[4 * u * ldy] : 0.f;
        }
#pragma unroll
        for (int u = 0; u < 4; ++u) {
          if (r + 4 * u >= k) continue;
          if (!last) bp[32 * u] = z4;
          const float v = (q[u].x + q[u].y) + (q[u].z + q[u].w);
          if (in) yp[4 * u * ldy] = beta == 0.f ? v : fmaf(beta, o[u], v);
        }
      }
    } else if (vec && r0 + 32 <= nrows) {
      const int sub = lane >> 3, q4 = lane & 7;
      float* yp = Y + r0 + 4 * q4 + (int64_t)sub * ldy;
      for (int r = sub; r < k; r += 4, yp += 4 * ldy) {
        float4* bp = bins4 + r * 8 + q4;
        float4 v = *bp;
        *bp = z4;
        float4* y4 = reinterpret_cast<float4*>(yp);
        if (beta == 0.f) {
          __stcs(y4, v);
        } else {
          const float4 o = *y4;
          v.x = fmaf(beta, o.x, v.x), v.y = fmaf(beta, o.y, v.y), v.z = fmaf(beta, o.z, v.z),
          v.w = fmaf(beta, o.w, v.w);
          *y4 = v;
        }
      }
    } else {
      const int64_t i = r0 + lane;
      if (i < nrows) {
        float* yp = Y + i;
        if (beta == 0.f) {
          for (int r = 0; r < k; ++r, yp += ldy) __stcs(yp, bins[r * 32 + lane]);
        } else {
          for (int r = 0; r < k; ++r, yp += ldy) *yp = fmaf(beta, *yp, bins[r * 32 + lane]);
        }
      }
      __syncwarp();
      for (int q = lane; q < k * 8; q += 32) bins4[q] = z4;
    }
    __syncwarp();
    b = nb, e = ne;
  }
}

// X and Z contributions of the Upsilon / Phi entries whose input row lies
// in the call's rows. One warp per entry. (Z: the zeta_s = 8 entries of a
// nonzero's Psi row lie along the lanes; with a 64-bit division per pair the
// longest rows took 17 us.)
__global__ void csr_ssign_entries_kernel(
    const int64_t* __restrict__ rowptr, const int32_t* __restrict__ col,
    const float* __restrict__ val, int64_t col_offset, int64_t row0, int64_t W, int64_t nwin,
    float eta, float nu, const int64_t* __restrict__ u_row, const uint32_t* __restrict__ u_rs,
    int64_t nu_ent, const int64_t* __restrict__ p_row, const uint32_t* __restrict__ p_rs,
    int64_t np_ent, const uint32_t* __restrict__ psi, int zeta_s, float* __restrict__ X, int64_t n,
    float* __restrict__ Z, int64_t s) {
  const int lane = threadIdx.x & 31;
  const int64_t gw = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const int64_t nwarps = ((int64_t)gridDim.x * blockDim.x) >> 5;
  for (int64_t e = gw; e < nu_ent + np_ent; e += nwarps) {
    const bool is_u = e < nu_ent;
    const int64_t ee = is_u ? e : e - nu_ent;
    const int64_t li = (is_u ? u_row[ee] : p_row[ee]) - row0;
    const uint32_t rsw = is_u ? u_rs[ee] : p_rs[ee];
    const int64_t r = rsw & 0x7fffffffu;
    const int64_t wi = li / W;
    float wgt = eta;
    if (nu != 1.f) wgt = (float)((double)eta * pow((double)nu, (double)(nwin - 1 - wi)));
    if (rsw >> 31) wgt = -wgt;
    const int64_t b = rowptr[li] - col_offset, en = rowptr[li + 1] - col_offset;
    if (is_u) {
      for (int64_t q = b + lane; q < en; q += 32)
        if ((uint64_t)col[q] < (uint64_t)n) atomicAdd(X + r * n + col[q], wgt * val[q]);
    } else {
      // zeta_s <= 8: 32 / 8 nonzeros at a time, lane t of eight the entry t
      const int t = lane & 7;
      for (int64_t p = b + (lane >> 3); p < en; p += 16) {
        int32_t j[4];
        float v[4];
        uint32_t w[4];
#pragma unroll
        for (int q = 0; q < 4; ++q) {
          const bool in = p + 4 * q < en && t < zeta_s;
          j[q] = in ? col[p + 4 * q] : -1;
          v[q] = in ? wgt * val[p + 4 * q] : 0.f;
        }
#pragma unroll
        for (int q = 0; q < 4; ++q)
          if ((uint64_t)(int64_t)j[q] < (uint64_t)n) w[q] = psi[(int64_t)j[q] * zeta_s + t];
#pragma unroll
        for (int q = 0; q < 4; ++q)
          if ((uint64_t)(int64_t)j[q] < (uint64_t)n)
            atomicAdd(Z + r * s + (w[q] & 0x7fffffffu), (w[q] >> 31) ? -v[q] : v[q]);
      }
    }
  }
}

// ---------------------------------------------------------------------------
// CSR x Gauss: Y rows by a warp-per-row SpMM against the stored n x k map
// (rows contiguous); X^T / W^T by atomic scatter of map rows.
// ---------------------------------------------------------------------------
__global__ void csr_gauss_y_kernel(const int64_t* __restrict__ rowptr,
                                   const int32_t* __restrict__ col, const float* __restrict__ val,
                                   int64_t col_offset, int64_t nrows, int64_t ncol,
                                   const float* __restrict__ mapT /* n x k rows */, int64_t k,
                                   float* __restrict__ Y, int64_t ldy, float alpha, float beta) {
  const int lane = threadIdx.x & 31;
  const int64_t gw = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const int64_t nwarps = ((int64_t)gridDim.x * blockDim.x) >> 5;
  for (int64_t i = gw; i < nrows; i += nwarps) {
    const int64_t b = rowptr[i] - col_offset, e = rowptr[i + 1] - col_offset;
    for (int64_t c0 = 0; c0 < k; c0 += 128) {
      float a[4] = {0.f, 0.f, 0.f, 0.f};
      for (int64_t p = b; p < e; ++p) {
        if ((uint64_t)col[p] >= (uint64_t)ncol) continue;
        const float v = val[p];
        const float* mrow = mapT + (int64_t)col[p] * k;
#pragma unroll
        for (int u = 0; u < 4; ++u) {
          const int64_t cc = c0 + lane + 32 * u;
          if (cc < k) a[u] = fmaf(v, __ldg(mrow + cc), a[u]);
        }
      }
#pragma unroll
      for (int u = 0; u < 4; ++u) {
        const int64_t cc = c0 + lane + 32 * u;
        if (cc < k) {
          float* yp = Y + i + cc * ldy;
          *yp = (beta == 0.f) ? alpha * a[u] : fmaf(beta, *yp, alpha * a[u]);
        }
      }
    }
  }
}

// out^T(j, :) += alpha * a_ij * map_rows(R0 + i, :) for every nonzero; out is
// stored with (row stride ors, col stride ocs) for logical out(r, j).
__global__ void csr_gauss_scatter_kernel(const int64_t* __restrict__ rowptr,
                                         const int32_t* __restrict__ col,
                                         const float* __restrict__ val, int64_t col_offset,
                                         int64_t nrows, int64_t ncol,
                                         const float* __restrict__ maprows, int64_t kk,
                                         float* __restrict__ out, int64_t ors, int64_t ocs,
                                         float alpha) {
  const int lane = threadIdx.x & 31;
  const int64_t gw = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const int64_t nwarps = ((int64_t)gridDim.x * blockDim.x) >> 5;
  for (int64_t i = gw; i < nrows; i += nwarps) {
    const int64_t b = rowptr[i] - col_offset, e = rowptr[i + 1] - col_offset;
    const float* mrow = maprows + i * kk;
    for (int64_t p = b; p < e; ++p) {
      const float v = alpha * val[p];
      const int64_t j = col[p];
      if ((uint64_t)j >= (uint64_t)ncol) continue;
      for (int64_t r = lane; r < kk; r += 32) atomicAdd(out + r * ors + j * ocs, v * mrow[r]);
    }
  }
}

// CSR x Gauss for all windows of a call: rows of [Y | T] = A [Omega Psi], 32
// rows per CTA. A warp takes a row of the tile at a time (from a counter, so
// a long row holds up one warp only) and its lanes hold up to 192 output
// columns, six each. The tile is turned in shared memory, so that Y (column
// major) and T leave as lines of 32 rows. T goes out as the three BF16 planes
// of the tensor-core product Z += Phi^T T (T32 null), or as FP32 columns of
// ldt when T is refused (x3.h; run again under *cond).
// Bound by the gathered bytes, 4 (k + s) per nonzero out of L2: 100,000 x
// 20,000 with 1e6 nonzeros at k = 81, s = 163 takes 178 us, 5.4 TB/s, with rows of
// log-normal lengths, and 135 with rows of ten entries. With all
// 244 columns in one pass of eight slots it took 338 (the loads of a group not
// all in flight) and 588 us (144 registers, one CTA per SM); 64 registers and
// four CTAs per SM are what pays.
struct GaussGather {
  const int64_t* rowptr;
  const int32_t* col;
  const float* val;
  int64_t col_offset, nrows, ncol;
  int tile;          // rows per CTA, up to 32
  const float* omg;  // ncol x k
  const float* psi;  // ncol x s
  int64_t k, s;
  float* Y;  // column-major; null: T only
  int64_t ldy;
  float alpha, beta;
  __nv_bfloat16* T;
  float* T32;
  int64_t ldt, pstride;
  uint32_t big;    // x3_report's
  uint32_t* word;  // T's magnitudes are noted here
  float* scale;    // nscale values to be scaled by `by`: Z before a split product
  int64_t nscale;
  float by;
};
// One row against NU x 32 columns of a map: acc[u] = sum_p a_p map(j_p, c0 +
// lane + 32 u), cols columns left from c0 on. 32 entries are loaded at once,
// one per lane, and go through four at a time: 4 NU loads per lane in flight,
// at one address and constant offsets per entry.
template <int NU>
__device__ __forceinline__ void gauss_row(const GaussGather& g, int64_t b, int64_t e, const float* __restrict__ map,
                                          int64_t stride, int cols, int lane, float* acc) {
  constexpr int Q = NU > 4 ? 2 : 4;
  const bool last = lane + 32 * (NU - 1) < cols;
#pragma unroll
  for (int u = 0; u < NU; ++u) acc[u] = 0.f;
  for (int64_t p0 = b; p0 < e; p0 += 32) {
    const int cnt = (int)min((int64_t)32, e - p0);
    int32_t jl = -1;
    float al = 0.f;
    if (lane < cnt) jl = __ldg(g.col + p0 + lane), al = __ldg(g.val + p0 + lane);
    if ((uint64_t)(int64_t)jl >= (uint64_t)g.ncol) jl = -1;
    for (int p = 0; p < cnt; p += Q) {
      float m[Q][NU], a[Q];
      int32_t j[Q];
#pragma unroll
      for (int q = 0; q < Q; ++q) {
        j[q] = __shfl_sync(0xffffffffu, jl, p + q);
        a[q] = __shfl_sync(0xffffffffu, al, p + q);
        const float* mp = map + (int64_t)max(j[q], 0) * stride + lane;
#pragma unroll
        for (int u = 0; u < NU; ++u) m[q][u] = (u < NU - 1 || last) ? __ldg(mp + 32 * u) : 0.f;
      }
#pragma unroll
      for (int q = 0; q < Q; ++q)
        if (j[q] >= 0) {  // an entry outside the matrix adds nothing
#pragma unroll
          for (int u = 0; u < NU; ++u) acc[u] = fmaf(a[q], m[q][u], acc[u]);
        }
    }
  }
}

template <int NU>
__device__ __forceinline__ void gauss_tile(const GaussGather& g, int64_t r0, int nr, const float* map, int64_t stride,
                                           int cols, int lane, int* next, float* tile) {
  while (true) {
    int i = 0;
    if (lane == 0) i = atomicAdd(next, 1);
    i = __shfl_sync(0xffffffffu, i, 0);
    if (i >= nr) return;
    float acc[NU];
    gauss_row<NU>(g, g.rowptr[r0 + i] - g.col_offset, g.rowptr[r0 + i + 1] - g.col_offset, map, stride, cols, lane,
                  acc);
#pragma unroll
    for (int u = 0; u < NU; ++u) tile[(lane + 32 * u) * 33 + i] = acc[u];
  }
}

__global__ void __launch_bounds__(256, 4) csr_gauss_gather_kernel(GaussGather g, const uint32_t* __restrict__ cond) {
  if (cond && !x3_refused(*cond)) return;
  constexpr int CH = 192;  // columns per pass
  extern __shared__ float gg_tile[];  // CH x 33
  __shared__ int next;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int64_t r0 = (int64_t)blockIdx.x * g.tile;
  const int nr = (int)min((int64_t)g.tile, g.nrows - r0);
  for (int64_t q = (int64_t)blockIdx.x * 256 + threadIdx.x; q < g.nscale; q += (int64_t)gridDim.x * 256)
    g.scale[q] = g.by == 0.f ? 0.f : g.by * g.scale[q];
  float top = 0.f;
  // the columns of Omega, then those of Psi
  for (int64_t c = g.Y ? 0 : g.k; c < g.k + g.s;) {
    const bool om = c < g.k;
    const int64_t c0 = om ? c : c - g.k, width = om ? g.k : g.s;
    const int cols = (int)min((int64_t)CH, width - c0);
    const float* map = (om ? g.omg : g.psi) + c0;
    if (threadIdx.x == 0) next = 0;
    __syncthreads();
    switch ((cols + 31) / 32) {
      case 1: gauss_tile<1>(g, r0, nr, map, width, cols, lane, &next, gg_tile); break;
      case 2: gauss_tile<2>(g, r0, nr, map, width, cols, lane, &next, gg_tile); break;
      case 3: gauss_tile<3>(g, r0, nr, map, width, cols, lane, &next, gg_tile); break;
      case 4: gauss_tile<4>(g, r0, nr, map, width, cols, lane, &next, gg_tile); break;
      case 5: gauss_tile<5>(g, r0, nr, map, width, cols, lane, &next, gg_tile); break;
      default: gauss_tile<6>(g, r0, nr, map, width, cols, lane, &next, gg_tile); break;
    }
    __syncthreads();
    // what beta scales is loaded ahead of the stores
    for (int cl = warp; om && cl < cols && lane < nr; cl += 32) {
      float* yp = g.Y + r0 + lane + (c0 + cl) * g.ldy;
      float o[4];
#pragma unroll
      for (int u = 0; u < 4; ++u) o[u] = g.beta != 0.f && cl + 8 * u < cols ? yp[8 * u * g.ldy] : 0.f;
#pragma unroll
      for (int u = 0; u < 4; ++u) {
        if (cl + 8 * u >= cols) continue;
        const float v = g.alpha * gg_tile[(cl + 8 * u) * 33 + lane];
        yp[8 * u * g.ldy] = g.beta == 0.f ? v : fmaf(g.beta, o[u], v);
      }
    }
    for (int cl = warp; !om && cl < cols; cl += 8) {
      const float v = gg_tile[cl * 33 + lane];
      if (lane >= nr) continue;
      if (g.T32) {
        g.T32[(c0 + cl) * g.ldt + r0 + lane] = v;
      } else {
        x3_note(top, v);
        __nv_bfloat16 h, m, l;
        tc::split3(v, h, m, l);
        __nv_bfloat16* tp = g.T + (c0 + cl) * g.ldt + r0 + lane;
        tp[0] = h, tp[g.pstride] = m, tp[2 * g.pstride] = l;
      }
    }
    __syncthreads();
    c += cols;
  }
  if (g.word) x3_report(top, g.big, g.word);
}

// X^T(j, :) += w_i a_ij Upsilon(i, :) into a zeroed n x kp scratch (kp a
// multiple of 4), w_i = nu^(windows after row i): a warp per row, one 16-byte
// reduction per four columns and nonzero. The rows of X itself are n apart, so
// its columns would take one 4-byte reduction in a sector of its own each
// (that form, with the same for Phi, took 174 us per 10,000 rows; this one
// takes 83 us for 100,000).
__global__ void __launch_bounds__(256)
    csr_gauss_xt_kernel(const int64_t* __restrict__ rowptr, const int32_t* __restrict__ col,
                        const float* __restrict__ val, int64_t col_offset, int64_t nrows, int64_t ncol,
                        const float* __restrict__ ups, int64_t k, int64_t kp, float* __restrict__ XT, float nu,
                        int64_t W, int64_t nwin) {
  const int lane = threadIdx.x & 31;
  const int64_t gw = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const int64_t nwarps = ((int64_t)gridDim.x * blockDim.x) >> 5;
  for (int64_t i = gw; i < nrows; i += nwarps) {
    const int64_t b = rowptr[i] - col_offset, e = rowptr[i + 1] - col_offset;
    if (b >= e) continue;
    float w = 1.f;
    if (nu != 1.f) w = (float)pow((double)nu, (double)(nwin - 1 - i / W));
    for (int64_t c = 4 * lane; c < kp; c += 128) {
      float u[4];
#pragma unroll
      for (int q = 0; q < 4; ++q) u[q] = c + q < k ? w * __ldg(ups + i * k + c + q) : 0.f;
      for (int64_t p = b; p < e; ++p) {
        const int32_t j = __ldg(col + p);
        if ((uint64_t)(int64_t)j >= (uint64_t)ncol) continue;
        const float a = __ldg(val + p);
        asm volatile("red.global.add.v4.f32 [%0], {%1, %2, %3, %4};" ::"l"(XT + (int64_t)j * kp + c), "f"(a * u[0]),
                     "f"(a * u[1]), "f"(a * u[2]), "f"(a * u[3])
                     : "memory");
      }
    }
  }
}

// X(r, j) = beta X + alpha XT(j, r), by 32 x 32 tiles.
__global__ void __launch_bounds__(256) xt_add_kernel(const float* __restrict__ XT, int64_t kp, int64_t k, int64_t n,
                                                     float* __restrict__ X, float alpha, float beta) {
  __shared__ float t[32][33];
  const int tx = threadIdx.x & 31, ty = threadIdx.x >> 5;
  const int64_t tk = (k + 31) / 32, tn = (n + 31) / 32;
  for (int64_t q = blockIdx.x; q < tk * tn; q += gridDim.x) {
    const int64_t r0 = (q % tk) * 32, j0 = (q / tk) * 32;
    for (int y = ty; y < 32; y += 8)
      if (j0 + y < n && r0 + tx < k) t[y][tx] = XT[(j0 + y) * kp + r0 + tx];
    __syncthreads();
    for (int y = ty; y < 32; y += 8)
      if (r0 + y < k && j0 + tx < n) {
        float* p = X + (r0 + y) * n + j0 + tx;
        *p = beta == 0.f ? alpha * t[tx][y] : fmaf(beta, *p, alpha * t[tx][y]);
      }
    __syncthreads();
  }
}

// ---------------------------------------------------------------------------
// Dense window x SparseSign (three-sketch, dense input, update(dense,
// SparseSign) src/Skema_SketchySVD.cpp:271-293).
// Y(R0+i, r) = beta*Y + alpha * sum_t sign_rt A_w(i, c_rt) for the k x n
// row-sparse Omega~: thread (row, map row), consecutive threads on
// consecutive rows (coalesced gathers from a column-major window and
// coalesced stores into the column-major Y).
// ---------------------------------------------------------------------------
__global__ void dense_ssign_y_kernel(const float* __restrict__ A, int64_t ars, int64_t acs,
                                     int64_t wr, const uint32_t* __restrict__ omg, int zeta,
                                     int64_t k, float* __restrict__ Y, int64_t ldy, float alpha,
                                     float beta) {
  const int64_t total = wr * k;
  for (int64_t q = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; q < total;
       q += (int64_t)gridDim.x * blockDim.x) {
    const int64_t r = q / wr, i = q - r * wr;
    float a = 0.f;
    for (int t = 0; t < zeta; ++t) {
      const uint32_t w = __ldg(omg + r * zeta + t);
      const float v = __ldg(A + i * ars + (int64_t)(w & 0x7fffffffu) * acs);
      a += (w >> 31) ? -v : v;
    }
    float* yp = Y + i + r * ldy;
    *yp = (beta == 0.f) ? alpha * a : fmaf(beta, *yp, alpha * a);
  }
}

// X(r, :) += wgt * A_w(li, :) for the Upsilon entries in the window, and
// Z(r, :) += wgt * sum_u sign A_w(li, c_{r'' u}) for the Phi entries.
__global__ void dense_ssign_entries_kernel(const float* __restrict__ A, int64_t ars, int64_t acs,
                                           int64_t R0, float eta, const int64_t* __restrict__ u_row,
                                           const uint32_t* __restrict__ u_rs, int64_t nu_ent,
                                           const int64_t* __restrict__ p_row,
                                           const uint32_t* __restrict__ p_rs, int64_t np_ent,
                                           const uint32_t* __restrict__ psi, int zeta_s,
                                           float* __restrict__ X, int64_t n, float* __restrict__ Z,
                                           int64_t s) {
  const int lane = threadIdx.x & 31;
  const int64_t gw = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const int64_t nwarps = ((int64_t)gridDim.x * blockDim.x) >> 5;
  for (int64_t e = gw; e < nu_ent + np_ent; e += nwarps) {
    const bool is_u = e < nu_ent;
    const int64_t ee = is_u ? e : e - nu_ent;
    const int64_t li = (is_u ? u_row[ee] : p_row[ee]) - R0;
    const uint32_t rsw = is_u ? u_rs[ee] : p_rs[ee];
    const int64_t r = rsw & 0x7fffffffu;
    const float wgt = (rsw >> 31) ? -eta : eta;
    const float* arow = A + li * ars;
    if (is_u) {
      for (int64_t j = lane; j < n; j += 32) atomicAdd(X + r * n + j, wgt * arow[j * acs]);
    } else {
      for (int64_t r2 = lane; r2 < s; r2 += 32) {
        float a = 0.f;
        for (int t = 0; t < zeta_s; ++t) {
          const uint32_t w = psi[r2 * zeta_s + t];
          const float v = arow[(int64_t)(w & 0x7fffffffu) * acs];
          a += (w >> 31) ? -v : v;
        }
        atomicAdd(Z + r * s + r2, wgt * a);
      }
    }
  }
}

// SketchySPD with a SparseSign Omega stored n x k (zeta per input column):
// Y(R0+i, :) = beta*Y + alpha * sum_j A_w(i, j) Omega(j, :). One thread per
// row with bin-major accumulators acc[r * blockDim + tid] (conflict free).
__global__ void dense_colsparse_y_kernel(const float* __restrict__ A, int64_t ars, int64_t acs,
                                         int64_t wr, int64_t n, const uint32_t* __restrict__ omg,
                                         int zeta, int64_t k, float* __restrict__ Y, int64_t ldy,
                                         float alpha, float beta) {
  extern __shared__ float acc[];
  float* my = acc + threadIdx.x;
  const int nt = blockDim.x;
  for (int64_t i0 = (int64_t)blockIdx.x * nt; i0 < wr; i0 += (int64_t)gridDim.x * nt) {
    const int64_t i = i0 + threadIdx.x;
    for (int64_t r = 0; r < k; ++r) my[r * nt] = 0.f;
    if (i < wr) {
      for (int64_t j = 0; j < n; ++j) {
        const float v = __ldg(A + i * ars + j * acs);
        for (int t = 0; t < zeta; ++t) {
          const uint32_t w = __ldg(omg + j * zeta + t);
          my[(int64_t)(w & 0x7fffffffu) * nt] += (w >> 31) ? -v : v;
        }
      }
      for (int64_t r = 0; r < k; ++r) {
        float* yp = Y + i + r * ldy;
        *yp = (beta == 0.f) ? alpha * my[r * nt] : fmaf(beta, *yp, alpha * my[r * nt]);
      }
    }
  }
}

// Index range of the sorted inverse entries with input row in [a, b).
std::pair<int64_t, int64_t> entry_range(const Map& mp, int64_t a, int64_t b) {
  const auto lo = std::lower_bound(mp.inv_row.begin(), mp.inv_row.end(), a);
  const auto hi = std::lower_bound(mp.inv_row.begin(), mp.inv_row.end(), b);
  return {lo - mp.inv_row.begin(), hi - mp.inv_row.begin()};
}

}  // namespace

template <int UNR>
void launch_csr_ssign_y_variant(skema_ctx* c, int warps_per_block, const int64_t* rowptr,
                                const int32_t* col, const float* val, int64_t col_offset,
                                int64_t nrows, const Map& O, float* Y, int64_t ldy, float alpha,
                                float beta) {
  const int k = (int)c->k;
  const size_t smem = sizeof(float) * 32 * (size_t)k * warps_per_block;
  auto kern = csr_ssign_y_kernel<UNR>;
  SKEMA_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
  int per_sm = 1;
  SKEMA_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kern, 32 * warps_per_block, smem));
  const int64_t tiles = (nrows + 31) / 32;
  const int grid = grid_cap(c, (tiles + warps_per_block - 1) / warps_per_block, std::max(1, per_sm));
  kern<<<grid, 32 * warps_per_block, smem, c->stream>>>(rowptr, col, val, col_offset, nrows, O.packed, O.zeta,
                                                        k, (int)c->n, Y, ldy, alpha, beta);
  SKEMA_LAUNCHED(c);
}

template <int U, int S>
static void launch_csr_ssign_y16(skema_ctx* c, const int64_t* rowptr, const int32_t* col, const float* val,
                                 int64_t col_offset, int64_t nrows, const Map& O, float* Y, int64_t ldy, float alpha,
                                 float beta) {
  const int k = (int)c->k;
  // warps per block: the most warps within the bin budget per SM (about
  // 128 KB), in the fewest blocks (k = 81: 4 x 3 = 12 warps; k = 161:
  // 2 x 3 = 6; k = 256: 4 x 1)
  const size_t budget = (size_t)c->ssign_bin_kb * 1024;
  int wpb = 1;
  {
    const size_t per_warp = sizeof(float) * 32 * (size_t)k;
    int best = 0;
    for (int w = 4; w >= 1; w >>= 1) {
      const int warps = w * (int)(budget / (per_warp * w));
      if (warps > best) best = warps, wpb = w;
    }
  }
  const size_t smem = sizeof(float) * 32 * (size_t)k * wpb;
  auto kern = csr_ssign_y16_kernel<U, S>;
  SKEMA_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
  // the bin budget per SM; the carve-out leaves the rest of the unified
  // L1 / shared memory to L1
  int smem_sm = 0;
  SKEMA_CUDA(cudaDeviceGetAttribute(&smem_sm, cudaDevAttrMaxSharedMemoryPerMultiprocessor, c->dev));
  const int per_sm = (int)std::max<size_t>(1, budget / smem);
  const int carve = (int)std::min<size_t>(100, (per_sm * (smem + 1024) * 100 + smem_sm - 1) / std::max(1, smem_sm) + 2);
  SKEMA_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributePreferredSharedMemoryCarveout, carve));
  const int64_t tiles = (nrows + 32 / S - 1) / (32 / S);
  const int grid = grid_cap(c, (tiles + wpb - 1) / wpb, per_sm);
  kern<<<grid, 32 * wpb, smem, c->stream>>>(rowptr, col, val, col_offset, nrows,
                                            static_cast<const uint4*>(O.packed16), k, (int)c->n, Y, ldy, alpha,
                                            beta);
  SKEMA_LAUNCHED(c);
}

static void launch_csr_ssign_y(skema_ctx* c, const int64_t* rowptr, const int32_t* col,
                               const float* val, int64_t col_offset, int64_t nrows, const Map& O,
                               float* Y, int64_t ldy, float alpha, float beta) {
  // Four lanes per row while the eight-row tiles of the call all fit on the chip
  // at once (1024 / k warps of bins per SM within 128 KB, and no more than 48).
  // Measured from 32 rows to the line, k = 9 to 253, after a reset: log-normal
  // row lengths (mean 10) take 0.40 to 0.62 of the time of a lane per row, rows
  // of 10 entries 0.74 to 1.05 (k = 201: 1.0 to 1.13), rows of 2 or 4 0.8 to
  // 1.3, which is 8 to 10 us +- 2 either way, and at 49,152 rows and k = 21 10
  // against 11 to 16 us, where log-normal ones take 40 against 23. Past the cap,
  // at k = 9 and 131,072 rows, short rows would take 12 to 17 against 17 to 20.
  // (Added to a Y that is not empty: 0.26 to 1.1.)
  if (O.packed16) {  // zeta = 8, k <= 256: at most 32 KB of bins per warp
    const bool few = nrows <= 8 * c->sm_count * std::min<int64_t>(48, std::max<int64_t>(1, 1024 / c->k));
    auto go = [&](auto one, auto four) {
      (few ? four : one)(c, rowptr, col, val, col_offset, nrows, O, Y, ldy, alpha, beta);
    };
    switch (c->ssign_batch) {
      case 2: go(launch_csr_ssign_y16<2, 1>, launch_csr_ssign_y16<2, 4>); break;
      case 6: go(launch_csr_ssign_y16<6, 1>, launch_csr_ssign_y16<6, 4>); break;
      case 8: go(launch_csr_ssign_y16<8, 1>, launch_csr_ssign_y16<8, 4>); break;
      default: go(launch_csr_ssign_y16<4, 1>, launch_csr_ssign_y16<4, 4>); break;
    }
    return;
  }
  // general form: up to 4 warps within 96 KB of bins per block; one warp's
  // bins (32 k floats) must fit the 200 KB limit
  int wpb = 4;
  while (wpb > 1 && sizeof(float) * 32 * (size_t)c->k * wpb > 96 * 1024) wpb >>= 1;
  if (sizeof(float) * 32 * (size_t)c->k * wpb > 200 * 1024)
    fail(SKEMA_EUNSUPPORTED, "sketch range too large for the sparse-sign kernel");
  launch_csr_ssign_y_variant<4>(c, wpb, rowptr, col, val, col_offset, nrows, O, Y, ldy, alpha, beta);
}

// CSR x Gauss over all windows of a call (src/Skema_SketchySVD.cpp:296-316):
// Z = nu^G Z + eta sum_i w_i Phi(i, :)^T T(i, :) with T = A Psi, the
// association of the dense form, instead of an n x s scatter and an n-deep
// product per window: 3.64 -> 0.44 ms for 100,000 x 20,000, 1e6 nonzeros, ten
// windows, k = 81, s = 163. False when the workspace is not to be had.
static bool csr_gauss_update(skema_ctx* c, const int64_t* rowptr, const int32_t* col, const float* val,
                             int64_t col_offset, int64_t row0, int64_t nrows, float ybeta) {
  const float eta = (float)c->p.sketch_eta, nu = (float)c->p.sketch_nu;
  const int64_t n = c->n, k = c->k, s = c->spd ? 0 : c->s, W = c->w, nwin = (nrows + W - 1) / W;
  auto up = [](size_t b) { return (b + 255) / 256 * 256; };
  // a row per warp where 32 rows per CTA would leave SMs idle: 20 rows of 20
  // entries (k = 201) 246 -> 78 us a call, 500 of 300 (k = 281) 817 -> 328, 3,000
  // of 10 (k = 81) 81 -> 76; 9,000 (k = 41) 85 against 90
  const int tile = nrows < (int64_t)32 * c->sm_count ? 8 : 32;
  GaussGather g{rowptr, col, val, col_offset, nrows, n, tile, c->omg.f32, c->psi.f32, k, s, c->Y + row0, c->m,
                eta, ybeta, nullptr, nullptr, 0, 0, 0, nullptr, nullptr, 0, 0.f};
  const size_t smem = sizeof(float) * 192 * 33;
  auto gather = [&](const GaussGather& q, const uint32_t* cond) {
    csr_gauss_gather_kernel<<<(unsigned)((q.nrows + q.tile - 1) / q.tile), 256, smem, c->stream>>>(q, cond);
    SKEMA_LAUNCHED(c);
  };
  if (c->spd) {
    StageScope st(c, ST_OMEGA);
    gather(g, nullptr);
    y_rows_mark(c, row0, row0 + nrows);
    return true;
  }
  // imported maps beyond the range of the planes, or of a weight on top
  const int lw = nu > 1.f ? (int)std::ceil(std::log2((double)nu) * (double)(nwin - 1)) : 0;
  if (!x3_carries(c->phi) || !x3_carries(c->ups) || x3_exp(c->ups) + lw > 126) return false;
  const int64_t kp = (k + 3) / 4 * 4;
  // rows per block: T, its FP32 form and Phi's planes within 512 MB
  const int64_t rb = std::min<int64_t>(nrows, std::max<int64_t>(32, ((int64_t)512 << 20) / (16 * s) / 32 * 32));
  const int64_t ldt = (rb + 7) / 8 * 8, nblk = (nrows + rb - 1) / rb;
  // T's bound: sums over a block's rows with Phi's weights stay below 2^126
  const int top = std::min(100, 126 - x3_log2(rb) - x3_exp(c->phi) - lw);
  if (top < 40) return false;
  const size_t b_xt = up(sizeof(float) * (size_t)(n * kp)), b_pl = up(sizeof(__nv_bfloat16) * (size_t)(3 * s * ldt)),
               b_t32 = up(sizeof(float) * (size_t)(s * ldt)), b_flag = up(sizeof(uint32_t) * (size_t)nblk);
  char* ws = static_cast<char*>(try_workspace(c, b_xt + 2 * b_pl + b_t32 + x3_part_bytes(c) + b_flag,
                                             sizeof(float) * (size_t)(n * s)));
  if (!ws) return false;
  float* XT = reinterpret_cast<float*>(ws);
  __nv_bfloat16* Tp = reinterpret_cast<__nv_bfloat16*>(ws + b_xt);
  __nv_bfloat16* Fp = reinterpret_cast<__nv_bfloat16*>(ws + b_xt + b_pl);
  float* T32 = reinterpret_cast<float*>(ws + b_xt + 2 * b_pl);
  float* part = reinterpret_cast<float*>(ws + b_xt + 2 * b_pl + b_t32);
  uint32_t* flags = reinterpret_cast<uint32_t*>(ws + b_xt + 2 * b_pl + b_t32 + x3_part_bytes(c));
  const float wn = (float)std::pow((double)nu, (double)nwin);
  {
    StageScope st(c, ST_UPSILON);
    SKEMA_CUDA(cudaMemsetAsync(XT, 0, b_xt, c->stream));
    SKEMA_CUDA(cudaMemsetAsync(flags, 0, b_flag, c->stream));
    csr_gauss_xt_kernel<<<grid_cap(c, (nrows + 7) / 8, 16), 256, 0, c->stream>>>(
        rowptr, col, val, col_offset, nrows, n, c->ups.f32 + row0 * k, k, kp, XT, nu, W, nwin);
    SKEMA_LAUNCHED(c);
    xt_add_kernel<<<grid_cap(c, ((k + 31) / 32) * ((n + 31) / 32), 16), 256, 0, c->stream>>>(XT, kp, k, n, c->X, eta,
                                                                                            wn);
    SKEMA_LAUNCHED(c);
  }
  for (int64_t r = 0, i = 0; r < nrows; r += rb, ++i) {
    const int64_t wr = std::min(rb, nrows - r), ps = s * ldt;
    GaussGather q = g;
    q.rowptr += r, q.nrows = wr, q.Y += r, q.T = Tp, q.ldt = ldt, q.pstride = ps;
    q.big = x3_bits(top), q.word = flags + i;
    {
      StageScope st(c, ST_OMEGA);
      gather(q, nullptr);
    }
    StageScope st(c, ST_PHI);
    const float* F = c->phi.f32 + (row0 + r) * s;
    const float zb = i == 0 ? wn : 1.f;
    x3_transposed_planes(c, F, s, wr, s, Fp, ldt, ps, nu, W, nwin, r, 0, nullptr);
    x3_gemm(c, X3A{Tp, false, false, 0, 0, ldt, ps}, X3B{Fp, ldt, ps}, s, s, wr,
            tc::X3Out{c->Z, 1, s, eta, zb, nullptr, 0, 0, s, s, s}, part, X3Words{flags + i, nullptr});
    q.Y = nullptr, q.T32 = T32, q.word = nullptr;
    q.scale = c->Z, q.nscale = s * s, q.by = zb;
    gather(q, flags + i);
    X3Plain3 z{};
    z.n = 1;
    z.g[0] = X3Plain{nullptr, 0, 0, Fp, ldt, ps, T32, 1, ldt, c->Z, s, 1, s, s, wr, eta, 1.f,
                     x3_plain_split(c, s, wr)};
    x3_plain(c, z, flags + i);
  }
  y_rows_mark(c, row0, row0 + nrows);
  return true;
}

// ---------------------------------------------------------------------------
void csr_update(skema_ctx* c, const int64_t* rowptr, const int32_t* col, const float* val,
                int64_t col_offset, int64_t row0, int64_t nrows) {
  if (c->residual_pass) {
    residual_csr(c, rowptr, col, val, col_offset, row0, nrows);
    return;
  }
  const float eta = (float)c->p.sketch_eta, nu = (float)c->p.sketch_nu;
  const int64_t W = c->w;
  const int64_t nwin = (nrows + W - 1) / W;
  const float ybeta = y_beta(c, row0, row0 + nrows, nu);

  if (c->p.dim_redux == SKEMA_MAP_SPARSE_SIGN) {
    // X / Z (zeroing after a reset, the nu scaling and the Upsilon / Phi
    // entries) touch neither Y nor anything the Y kernel reads: they run on
    // the side stream, forked before the Y launch and joined after it,
    // beside the Y kernel.
    const auto ur = entry_range(c->ups, row0, row0 + nrows);
    const auto pr = entry_range(c->phi, row0, row0 + nrows);
    const int64_t nue = c->spd ? 0 : ur.second - ur.first, npe = c->spd ? 0 : pr.second - pr.first;
    const bool side = c->xz_pending || (!c->spd && (nu != 1.f || nue + npe > 0));
    if (side) SKEMA_CUDA(cudaEventRecord(c->fork_ev, c->stream));
    {
      StageScope st(c, ST_OMEGA);
      launch_csr_ssign_y(c, rowptr, col, val, col_offset, nrows, c->omg, c->Y + row0, c->m, eta, ybeta);
    }
    y_rows_mark(c, row0, row0 + nrows);
    if (!side) return;
    SKEMA_CUDA(cudaStreamWaitEvent(c->side, c->fork_ev, 0));
    xz_materialize(c, c->side);
    if (c->spd) {
      SKEMA_CUDA(cudaEventRecord(c->join_ev, c->side));
      SKEMA_CUDA(cudaStreamWaitEvent(c->stream, c->join_ev, 0));
      return;
    }
    if (nu != 1.f) {
      StageScope st(c, ST_DAXPY, c->side);
      const float sc = (float)std::pow((double)nu, (double)nwin);
      scale_block(c, MatOut{c->X, c->n, 1}, c->k, c->n, sc, c->side);
      scale_block(c, MatOut{c->Z, c->s, 1}, c->s, c->s, sc, c->side);
    }
    if (nue + npe > 0) {
      StageScope st(c, ST_ENTRIES, c->side);
      const int grid = grid_cap(c, (nue + npe + 7) / 8, 8);
      csr_ssign_entries_kernel<<<grid, 256, 0, c->side>>>(
          rowptr, col, val, col_offset, row0, W, nwin, eta, nu, c->ups.d_inv_row + ur.first,
          c->ups.d_inv_rs + ur.first, nue, c->phi.d_inv_row + pr.first, c->phi.d_inv_rs + pr.first,
          npe, c->psi.packed, c->psi.zeta, c->X, c->n, c->Z, c->s);
      SKEMA_LAUNCHED(c);
    }
    SKEMA_CUDA(cudaEventRecord(c->join_ev, c->side));
    SKEMA_CUDA(cudaStreamWaitEvent(c->stream, c->join_ev, 0));
    return;
  }

  xz_materialize(c, c->stream);
  int64_t done = 0;
  const int64_t L = c->spd ? nwin : std::min(nwin, weight_windows(nu));
  while (done < nrows) {
    const int64_t wr = std::min(L * W, nrows - done);
    if (!csr_gauss_update(c, rowptr + done, col, val, col_offset, row0 + done, wr, ybeta)) break;
    done += wr;
  }
  // The same window by window, for a workspace limit that has no room for
  // the call's T and X^T (SPD calls need none).
  // Gauss maps, all stored transposed (src/Skema_SketchySVD.cpp:296-316):
  // stored rows contiguous, logical (r, j) at f32[r + j*lrows].
  const int threads = 256;
  for (int64_t r = done; r < nrows; r += W) {
    const int64_t wr = std::min(W, nrows - r);
    const int64_t R0 = row0 + r;
    const float yb = y_beta(c, R0, R0 + wr, nu);
    {
      StageScope st(c, ST_OMEGA);
      csr_gauss_y_kernel<<<grid_cap(c, (wr + 7) / 8, 16), threads, 0, c->stream>>>(
          rowptr + r, col, val, col_offset, wr, c->n, c->omg.f32, c->k, c->Y + R0, c->m, eta, yb);
      SKEMA_LAUNCHED(c);
    }
    y_rows_mark(c, R0, R0 + wr);
    {  // X = nu X + eta (A_w^T Upsilon_stored(R0:R0+wr, :))^T
      StageScope st(c, ST_UPSILON);
      scale_block(c, MatOut{c->X, c->n, 1}, c->k, c->n, nu);
      csr_gauss_scatter_kernel<<<grid_cap(c, (wr + 7) / 8, 16), threads, 0, c->stream>>>(
          rowptr + r, col, val, col_offset, wr, c->n, c->ups.f32 + R0 * c->k, c->k, c->X, c->n, 1, eta);
      SKEMA_LAUNCHED(c);
    }
    // W^T = A_w^T Phi_stored(R0:R0+wr, :) in scratch (n x s), then
    // Z = nu Z + eta W Psi_stored.
    StageScope st(c, ST_PHI);
    float* Wt = (float*)workspace(c, sizeof(float) * (size_t)(c->n * c->s));
    SKEMA_CUDA(cudaMemsetAsync(Wt, 0, sizeof(float) * (size_t)(c->n * c->s), c->stream));
    csr_gauss_scatter_kernel<<<grid_cap(c, (wr + 7) / 8, 16), threads, 0, c->stream>>>(
        rowptr + r, col, val, col_offset, wr, c->n, c->phi.f32 + R0 * c->s, c->s, Wt, 1, c->s, 1.f);
    SKEMA_LAUNCHED(c);
    scale_block(c, MatOut{c->Z, c->s, 1}, c->s, c->s, nu);
    const int64_t tiles = ((c->s + 127) / 128) * ((c->s + 127) / 128);
    int sk = (int)std::max<int64_t>(1, std::min<int64_t>((2 * c->sm_count + tiles - 1) / tiles, c->n / 256));
    sgemm(c, c->s, c->s, c->n, eta, Mat{Wt, 1, c->s}, Mat{c->psi.f32, c->psi.cs, c->psi.rs}, 1.f,
          MatOut{c->Z, c->s, 1}, std::max(1, sk));
  }
}

void dense_ssign_window(skema_ctx* c, Mat Aw, int64_t R0, int64_t wr) {
  const float eta = (float)c->p.sketch_eta, nu = (float)c->p.sketch_nu;
  const float ybeta = y_beta(c, R0, R0 + wr, nu);
  {
    StageScope st(c, ST_OMEGA);
    dense_ssign_y_kernel<<<grid_cap(c, (wr * c->k + 255) / 256, 16), 256, 0, c->stream>>>(
        Aw.p, Aw.rs, Aw.cs, wr, c->omg.packed, c->omg.zeta, c->k, c->Y + R0, c->m, eta, ybeta);
    SKEMA_LAUNCHED(c);
  }
  y_rows_mark(c, R0, R0 + wr);
  scale_block(c, MatOut{c->X, c->n, 1}, c->k, c->n, nu);
  scale_block(c, MatOut{c->Z, c->s, 1}, c->s, c->s, nu);
  const auto ur = entry_range(c->ups, R0, R0 + wr);
  const auto pr = entry_range(c->phi, R0, R0 + wr);
  const int64_t nue = ur.second - ur.first, npe = pr.second - pr.first;
  if (nue + npe == 0) return;
  StageScope st(c, ST_ENTRIES);
  dense_ssign_entries_kernel<<<grid_cap(c, (nue + npe + 7) / 8, 8), 256, 0, c->stream>>>(
      Aw.p, Aw.rs, Aw.cs, R0, eta, c->ups.d_inv_row + ur.first, c->ups.d_inv_rs + ur.first, nue,
      c->phi.d_inv_row + pr.first, c->phi.d_inv_rs + pr.first, npe, c->psi.packed, c->psi.zeta, c->X,
      c->n, c->Z, c->s);
  SKEMA_LAUNCHED(c);
}

void spd_ssign_window(skema_ctx* c, Mat Aw, int64_t R0, int64_t wr) {
  const float eta = (float)c->p.sketch_eta, nu = (float)c->p.sketch_nu;
  const float ybeta = y_beta(c, R0, R0 + wr, nu);
  int threads = 128;
  while (threads > 32 && sizeof(float) * (size_t)(threads * c->k) > 200 * 1024) threads >>= 1;
  const size_t smem = sizeof(float) * (size_t)(threads * c->k);
  if (smem > 200 * 1024) fail(SKEMA_EUNSUPPORTED, "sketch range too large for the SPD sparse-sign kernel");
  SKEMA_CUDA(cudaFuncSetAttribute(dense_colsparse_y_kernel,
                                  cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
  StageScope st(c, ST_OMEGA);
  dense_colsparse_y_kernel<<<grid_cap(c, (wr + threads - 1) / threads, 4), threads, smem, c->stream>>>(
      Aw.p, Aw.rs, Aw.cs, wr, c->n, c->omg.packed, c->omg.zeta, c->k, c->Y + R0, c->m, eta, ybeta);
  SKEMA_LAUNCHED(c);
  y_rows_mark(c, R0, R0 + wr);
}

}  // namespace skema
