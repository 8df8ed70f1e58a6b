// tc_x3.cuh -- FP32 products on the BF16 tensor cores of sm_100a.
//
// An FP32 value is the sum of three BF16 values (8 + 8 + 8 significant bits):
//   x0 = bf16(x), x1 = bf16(x - x0), x2 = bf16(x - x0 - x1),
// exact up to 2^-24 |x| down to |x| = 2^-109 and to half of BF16's smallest step,
// 2^-134, below (x3.h says what becomes of such values). A product of two
// such sums keeps six of its nine BF16 products,
//   a b = a0 b0 + (a0 b1 + a1 b0) + (a1 b1 + a0 b2 + a2 b0) + O(2^-24 |a b|),
// each of which the tensor core forms exactly and adds in FP32. The split is
// carried as three planes per operand.
//
// What bounds it: six BF16 MMAs per FP32 one, so 1/6 of the BF16 tensor rate
// (about 230 TFLOP/s of FP32 work at the measured sustained 1400) against 74
// nominal and 31-37 measured for the SIMT kernel. Whole sketch updates: 50,000
// x 20,000 at k = 201, s = 403 in 52.4 -> 11.1 ms; the RBF kernel of 40,000
// points (d = 100, k = 129, s = 259) in 102.5 -> 24.6 ms; 3001 x 1003 in six
// windows in 2.42 -> 0.12 ms.
//
// Accuracy. tcgen05 accumulates in FP32 without round-to-nearest, so a long
// run of MMAs on one accumulator drifts towards zero. Each K step of 32 is
// therefore a run of its own (12 MMAs, the five small products first, a0 b0
// last, so only the last two meet the full sum); epilogue warps take the
// run's result out of TMEM and add it in registers with FP32 round-to-nearest
// while the MMAs of the next step go into the other TMEM accumulator. Against
// FP64 the sketches of those cases are 4.6e-7, 5.3e-7 and 1.6e-7 off, those of
// the SIMT kernel 1.3e-6, 1.2e-6 and 7.4e-7.
//
// Work: tiles of 128 x nt outputs (nt <= 256, a multiple of 16, chosen at
// launch). The first floor(tiles / G) G tiles go whole, one CTA each, N
// fastest so that the CTAs of one row block read the same A tiles together.
// The K steps of the remaining tiles are cut into G equal runs (at most two
// tiles per run); a CTA writes its part of a tile to a slot of its own and a
// second kernel adds a tile's slots in K order, so results do not depend on
// scheduling.
//
// Roles (320 threads): warps 0-7 epilogue (warp w: TMEM lanes 32 (w % 4) ..,
// half w / 4 of the columns: at most 128 sums per thread), warp 8 TMA
// producer, warp 9 MMA issuer. One stage holds a K step of 32 of all six
// planes (24 KB + 192 nt bytes): with all planes of a step on chip each is
// loaded once for its three (or two, or one) products.
#pragma once
#include "tc_gemm.cuh"
#include "x3.h"

namespace skema {
namespace tc {

constexpr int kX3Threads = 320;
constexpr int kX3BK = 32;        // K per stage (a 64-byte swizzle row of BF16)
constexpr int kX3MaxStages = 8;
constexpr uint32_t kX3ABytes = 3 * BM * kX3BK * 2;  // 24 KB

struct X3Grid {
  int mtiles, ntiles, ksteps, nt, stages;
  int full;  // tiles [0, full) go whole; the rest is cut into gridDim.x runs
};

// K-major operand descriptor, 64-byte swizzle: lines of 32 K-elements, 512
// bytes per 8 lines.
__device__ __forceinline__ uint64_t sdesc64(uint32_t saddr) {
  uint64_t d = 0;
  d |= (uint64_t)((saddr & 0x3FFFFu) >> 4);
  d |= (uint64_t)1 << 16;
  d |= (uint64_t)(512 >> 4) << 32;
  d |= (uint64_t)1 << 46;
  d |= (uint64_t)4 << 61;  // SWIZZLE_64B
  return d;
}

struct X3Seg {
  int mt, nt, kt0, kt1;
  int slot;  // >= 0: part of a tile, to this slot; -1: a whole tile
};
struct X3Sched {
  int t;
  int64_t pos, end;
  int seg;
};
__host__ __device__ __forceinline__ int64_t x3_run(const X3Grid& g, int64_t b, int64_t G) {
  return ((int64_t)(g.mtiles * g.ntiles - g.full) * g.ksteps) * b / G;
}
__device__ __forceinline__ void x3_init(const X3Grid& g, X3Sched& s) {
  s.t = blockIdx.x;
  s.pos = x3_run(g, blockIdx.x, gridDim.x);
  s.end = x3_run(g, blockIdx.x + 1, gridDim.x);
  s.seg = 0;
}
__device__ __forceinline__ bool x3_next(const X3Grid& g, X3Sched& s, X3Seg& u) {
  int tile;
  if (s.t < g.full) {
    tile = s.t;
    s.t += gridDim.x;
    u.kt0 = 0, u.kt1 = g.ksteps, u.slot = -1;
  } else {
    if (s.pos >= s.end) return false;
    const int q = (int)(s.pos / g.ksteps);
    u.kt0 = (int)(s.pos - (int64_t)q * g.ksteps);
    u.kt1 = (int)min((int64_t)g.ksteps, u.kt0 + (s.end - s.pos));
    s.pos += u.kt1 - u.kt0;
    u.slot = (u.kt0 == 0 && u.kt1 == g.ksteps) ? -1 : 2 * (int)blockIdx.x + s.seg;
    ++s.seg;
    tile = g.full + q;
  }
  u.nt = tile % g.ntiles;
  u.mt = tile / g.ntiles;
  return true;
}

__device__ __forceinline__ void x3_store(const X3Out& o, int64_t row, int64_t col, float v) {
  if (col >= o.ncols) return;
  if (col < o.split) {
    float* p = o.p0 + row * o.rs0 + col * o.cs0;
    *p = (o.beta == 0.f) ? o.alpha * v : fmaf(o.beta, *p, o.alpha * v);
  } else {
    __nv_bfloat16 h, m, l;
    split3(v, h, m, l);
    __nv_bfloat16* p = o.pl + (col - o.split) * o.ld + row;
    p[0] = h, p[o.pstride] = m, p[2 * o.pstride] = l;
  }
}

// Eight columns. What beta scales is loaded ahead of the stores, which the
// compiler cannot move it past: one after another, a tile of 208 columns and one K
// step took 55 us, and a call of 16 x 20,000 (k = 201, s = 403) 605; 146 now.
__device__ __forceinline__ void x3_store8(const X3Out& o, int64_t row, int64_t col, const float* v) {
  if (o.beta != 0.f && col + 8 <= o.split) {
    float* p = o.p0 + row * o.rs0 + col * o.cs0;
    float old[8];
#pragma unroll
    for (int e = 0; e < 8; ++e) old[e] = p[e * o.cs0];
#pragma unroll
    for (int e = 0; e < 8; ++e) p[e * o.cs0] = fmaf(o.beta, old[e], o.alpha * v[e]);
  } else {
#pragma unroll
    for (int e = 0; e < 8; ++e) x3_store(o, row, col + e, v[e]);
  }
}

// AMN = true:  A planes row-blocked {64, K, 3 nrb}, read MN-major (rows of
//              the output are the block's contiguous rows);
// AMN = false: the same layout {64, M, 3 nrb}, read K-major (K runs along the
//              contiguous rows), or any 3-D map {K, M, 3} with a_blk = 0.
// words: nothing is written when an operand is refused (x3.h).
template <bool AMN>
__global__ void __launch_bounds__(kX3Threads, 1)
    gemm_x3_kernel(const __grid_constant__ CUtensorMap tmA, const __grid_constant__ CUtensorMap tmB, X3Grid g, X3Out o,
                   int a_blk, int nrb, float* __restrict__ part, X3Words words, int* err) {
  extern __shared__ __align__(1024) unsigned char smem_raw[];
  if (x3_skip(words)) {
    if (blockIdx.x == 0 && threadIdx.x == 0 && words.all) atomicOr(words.all, kX3Big);
    return;
  }
  unsigned char* smem = reinterpret_cast<unsigned char*>(
      (reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~(uintptr_t)1023);
  const uint32_t bplane = (uint32_t)g.nt * kX3BK * 2;
  const uint32_t stage_bytes = kX3ABytes + 3 * bplane;
  const int S = g.stages;
  uint64_t* full = reinterpret_cast<uint64_t*>(smem + (size_t)S * stage_bytes);
  uint64_t* empty = full + kX3MaxStages;
  uint64_t* tfull = empty + kX3MaxStages;
  uint64_t* tempty = tfull + 2;
  uint32_t* tbase = reinterpret_cast<uint32_t*>(tempty + 2);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;

  if (threadIdx.x == 0) {
    for (int s = 0; s < S; ++s) {
      mbar_init(full + s, 1);
      mbar_init(empty + s, 1);
    }
    for (int a = 0; a < 2; ++a) {
      mbar_init(tfull + a, 1);
      mbar_init(tempty + a, 8 * 32);
    }
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == 9) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tbase)), "r"(512)
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = *tbase;

  X3Sched sc;
  x3_init(g, sc);
  X3Seg u;
  if (warp == 8 && lane == 0) {
    // ---------------- TMA producer ----------------
    int s = 0;
    uint32_t ph = 1;
    bool ok = true;
    while (ok && x3_next(g, sc, u)) {
      for (int kt = u.kt0; kt < u.kt1; ++kt) {
        if (!mbar_wait(empty + s, ph, err)) {
          ok = false;
          break;
        }
        unsigned char* sa = smem + (size_t)s * stage_bytes;
        mbar_expect_tx(full + s, stage_bytes);
        const int kc = kt * kX3BK;
#pragma unroll
        for (int q = 0; q < 3; ++q) {
          if (AMN) {
            tma_load_3d(&tmA, full + s, sa + q * 8192, 0, kc, q * nrb + 2 * u.mt);
            tma_load_3d(&tmA, full + s, sa + q * 8192 + 4096, 0, kc, q * nrb + 2 * u.mt + 1);
          } else if (a_blk) {
            tma_load_3d(&tmA, full + s, sa + q * 8192, kc & 32, u.mt * BM, q * nrb + (kc >> 6));
          } else {
            tma_load_3d(&tmA, full + s, sa + q * 8192, kc, u.mt * BM, q);
          }
        }
        tma_load_3d(&tmB, full + s, sa + kX3ABytes, kc, u.nt * g.nt, 0);
        if (++s == S) s = 0, ph ^= 1;
      }
    }
  } else if (warp == 9 && lane == 0) {
    // ---------------- MMA issuer ----------------
    const uint32_t idesc = idesc_bf16(g.nt, AMN, false);
    int s = 0;
    uint32_t ph = 0, cnt = 0;
    bool ok = true;
    while (ok && x3_next(g, sc, u)) {
      for (int kt = u.kt0; kt < u.kt1; ++kt, ++cnt) {
        const uint32_t acc = cnt & 1, aph = (cnt >> 1) & 1;
        if (!mbar_wait(tempty + acc, aph ^ 1, err) || !mbar_wait(full + s, ph, err)) {
          ok = false;
          break;
        }
        tc_fence_after();
        const uint32_t d = tmem + acc * 256;
        const uint32_t sa = smem_u32(smem + (size_t)s * stage_bytes), sb = sa + kX3ABytes;
        constexpr int pa[6] = {0, 2, 1, 0, 1, 0}, pb[6] = {2, 0, 1, 1, 0, 0};
#pragma unroll
        for (int q = 0; q < 6; ++q)
#pragma unroll
          for (int kk = 0; kk < 2; ++kk) {
            const uint64_t ad = AMN ? sdesc(sa + pa[q] * 8192 + kk * 2048, 4096, 1024)
                                    : sdesc64(sa + pa[q] * 8192 + kk * 32);
            umma(d, ad, sdesc64(sb + pb[q] * bplane + kk * 32), idesc, (q > 0 || kk > 0) ? 1u : 0u);
          }
        umma_commit(empty + s);
        umma_commit(tfull + acc);
        if (++s == S) s = 0, ph ^= 1;
      }
    }
  } else if (warp < 8) {
    // ---------------- epilogue ----------------
    const int nch = g.nt >> 4, h0 = (nch + 1) >> 1;
    const int c0 = warp >= 4 ? h0 : 0, nc = warp >= 4 ? nch - h0 : h0;  // 16-column chunks of this warp
    const int r = (warp & 3) * 32 + lane;
    const uint32_t taddr = tmem + ((uint32_t)((warp & 3) * 32) << 16) + c0 * 16;
    uint32_t cnt = 0;
    bool ok = true;
    while (ok && x3_next(g, sc, u)) {
      float sum[128];
#pragma unroll
      for (int i = 0; i < 128; ++i) sum[i] = 0.f;
      for (int kt = u.kt0; kt < u.kt1; ++kt, ++cnt) {
        const uint32_t acc = cnt & 1, aph = (cnt >> 1) & 1;
        // tcgen05.ld is warp-collective: the whole warp reads TMEM or none of it
        if (!__all_sync(0xffffffffu, mbar_wait(tfull + acc, aph, err))) {
          ok = false;
          break;
        }
        tc_fence_after();
#pragma unroll
        for (int i = 0; i < 8; i += 2) {
          float v[32];
          if (i + 1 < nc) {
            tmem_ld32(taddr + acc * 256 + i * 16, v);
#pragma unroll
            for (int e = 0; e < 32; ++e) sum[i * 16 + e] += v[e];
          } else if (i < nc) {
            tmem_ld16(taddr + acc * 256 + i * 16, v);
#pragma unroll
            for (int e = 0; e < 16; ++e) sum[i * 16 + e] += v[e];
          }
        }
        tc_fence_before();
        mbar_arrive(tempty + acc);
      }
      if (!ok) break;
      const int64_t row = (int64_t)u.mt * BM + r;
      if (u.slot >= 0) {
        float* pp = part + ((int64_t)u.slot * g.nt + c0 * 16) * BM + r;
#pragma unroll
        for (int i = 0; i < 8; ++i) {
          if (i >= nc) break;
#pragma unroll
          for (int e = 0; e < 16; ++e) pp[(i * 16 + e) * BM] = sum[i * 16 + e];
        }
      } else if (row < o.rows) {
        const int64_t col = (int64_t)u.nt * g.nt + c0 * 16;
#pragma unroll
        for (int i = 0; i < 8; ++i) {
          if (i >= nc) break;
          x3_store8(o, row, col + i * 16, sum + i * 16);
          x3_store8(o, row, col + i * 16 + 8, sum + i * 16 + 8);
        }
      }
    }
  }
  drain_on_error(err);
  if (warp == 9) {
    __syncwarp();
    tc_fence_after();
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(512) : "memory");
  }
}

// Adds the parts of the tiles that were cut, in K order, and stores them.
// blockIdx.x: tile, blockIdx.y: 2 COLS columns; G: the product's grid; a
// thread per row and COLS columns. A product of few tiles cuts each into as
// many as G parts: COLS = 1, eight parts loaded at a time (one after another took 79
// us, this way 22, for two tiles of 74 parts). One of many tiles has two or
// three parts per tile, and finding them (64-bit divisions) cost more than
// adding them: COLS = 4, 60 -> 17 us for 97 tiles of 208 columns.
template <int COLS>
static __global__ void __launch_bounds__(256) x3_reduce_kernel(X3Grid g, X3Out o, int G, const float* __restrict__ part,
                                                        X3Words words) {
  if (x3_skip(words)) return;
  const int64_t q = blockIdx.x;
  const int64_t kb = q * g.ksteps, ke = kb + g.ksteps;
  const int64_t T = (int64_t)(g.mtiles * g.ntiles - g.full) * g.ksteps;
  int64_t b = kb * G / T;
  while (b > 0 && x3_run(g, b, G) > kb) --b;
  while (x3_run(g, b + 1, G) <= kb) ++b;
  if (x3_run(g, b, G) <= kb && x3_run(g, b + 1, G) >= ke) return;  // one run: stored by the product
  int64_t e = (ke - 1) * G / T;  // the run that holds the tile's last step
  while (x3_run(g, e, G) > ke - 1) --e;
  while (x3_run(g, e + 1, G) <= ke - 1) ++e;
  const int tile = g.full + (int)q;
  const int r = threadIdx.x & 127, cl = (blockIdx.y * 2 + (threadIdx.x >> 7)) * COLS;
  const int64_t row = (int64_t)(tile / g.ntiles) * BM + r;
  const float* pp = part + (int64_t)cl * BM + r;
  const int64_t slot = (int64_t)g.nt * BM;
  // the first run may begin in the tile before: its part of this tile is its
  // second; every other run begins inside the tile (runs are never empty)
  float sum[COLS];
  const float* p0 = pp + (2 * b + (x3_run(g, b, G) < kb ? 1 : 0)) * slot;
#pragma unroll
  for (int q = 0; q < COLS; ++q) sum[q] = p0[q * BM];
  pp += 2 * slot;
  constexpr int U = 8 / COLS;
  for (int64_t i = b; i < e; i += U) {
    float v[U][COLS];
#pragma unroll
    for (int u = 0; u < U; ++u)
#pragma unroll
      for (int q = 0; q < COLS; ++q) v[u][q] = i + u < e ? pp[2 * (i + u) * slot + q * BM] : 0.f;
#pragma unroll
    for (int u = 0; u < U; ++u)
#pragma unroll
      for (int q = 0; q < COLS; ++q) sum[q] += v[u][q];
  }
  if (row >= o.rows) return;
#pragma unroll
  for (int q = 0; q < COLS; ++q) x3_store(o, row, (int64_t)(tile % g.ntiles) * g.nt + cl + q, sum[q]);
}

}  // namespace tc
}  // namespace skema
