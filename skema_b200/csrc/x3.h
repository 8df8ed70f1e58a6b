// x3.h -- FP32 products on the tensor cores through three BF16 planes per
// operand (x3.cu, tc_x3.cuh).
#pragma once
#include <cuda_bf16.h>

#include <algorithm>
#include <cmath>
#include <functional>

#include "internal.h"

namespace skema {

// The range of the planes. The low planes of a value below about 2^-109 reach
// BF16's smallest step (2^-133) and lose bits, so what counts is the largest
// magnitude of a block of values: from 2^-90 on, what the smaller ones lose is
// below 2^-44 of it. (A block of A that meets a map of small values needs as much
// more as leaves T = A Psi at 2^-102.) Upwards, what counts is that the sums stay
// within FP32's range: an infinity, or one in a plane, turns into a NaN where FP32
// arithmetic has an infinity. The bound, 2^100 at most, follows from the length of
// the sums and the other operand's largest value (x3_top).
// A kernel that makes planes notes in a device word which kinds it met; a block
// that is all tiny, or holds a value from the bound on, is refused, and FP32
// arithmetic forms its products. A NaN is a NaN in its planes too and counts for
// nothing here.
constexpr uint32_t kX3Normal = 1, kX3Tiny = 2, kX3Big = 4;
constexpr uint32_t kX3SmallBits = (uint32_t)(127 - 90) << 23;
inline uint32_t x3_bits(int e) { return (uint32_t)(127 + e) << 23; }  // 2^e
// Least e with 2^e >= n
inline int x3_log2(int64_t n) {
  int e = 0;
  while (((int64_t)1 << e) < n) ++e;
  return e;
}
// A bound 2^e on a map's magnitudes, and whether planes carry the map: its
// largest value is finite, and far enough up that a weight of 2^-40 leaves it
// all its bits.
inline int x3_exp(const Map& mp) { return mp.amax > 0.f ? std::max(-50, std::ilogb(mp.amax) + 1) : -50; }
inline bool x3_carries(const Map& mp) { return mp.amax == 0.f || (mp.amax >= 0x1p-50f && mp.amax <= 0x1p100f); }
__host__ __device__ __forceinline__ bool x3_refused(uint32_t w) {
  return (w & kX3Big) || (w & (kX3Normal | kX3Tiny)) == kX3Tiny;
}
// m: the largest of this thread's magnitudes (fmaxf passes a NaN over)
__device__ __forceinline__ void x3_note(float& m, float x) { m = fmaxf(m, fabsf(x)); }
// Notes the block's largest magnitude in *word, big from the bits `big` on, tiny
// below the bits `small`; called by all its threads.
__device__ __forceinline__ void x3_report(float top, uint32_t big, uint32_t* word, uint32_t small = kX3SmallBits) {
  const uint32_t m = __float_as_uint(top);
  uint32_t kind = 0;
  if (__syncthreads_or(m >= big))
    kind = kX3Big;
  else if (__syncthreads_or(m >= small))
    kind = kX3Normal;
  else if (__syncthreads_or(m > 0))
    kind = kX3Tiny;
  // most blocks find their kind noted
  if (threadIdx.x == 0 && kind && !(*(volatile uint32_t*)word & kind)) atomicOr(word, kind);
}

namespace tc {
// Two values as sums of three BF16 values each (split3), whose parts lie side
// by side.
__device__ __forceinline__ void split3x2(float x, float y, __nv_bfloat162& h, __nv_bfloat162& m, __nv_bfloat162& l) {
  h = __floats2bfloat162_rn(x, y);
  const float rx = x - __low2float(h), ry = y - __high2float(h);
  m = __floats2bfloat162_rn(rx, ry);
  l = __floats2bfloat162_rn(rx - __low2float(m), ry - __high2float(m));
}
// Where an x3_gemm product goes.
struct X3Out {
  // columns [0, split): FP32, p0[row * rs0 + col * cs0] = beta p0 + alpha acc
  float* p0;
  int64_t rs0, cs0;
  float alpha, beta;
  // columns [split, ncols): the three planes of acc, plane q of column c at
  // pl[q * pstride + (c - split) * ld + row]
  __nv_bfloat16* pl;
  int64_t ld, pstride;
  int64_t rows, split, ncols;
};

// x as the sum of three BF16 values
__device__ __forceinline__ void split3(float x, __nv_bfloat16& h, __nv_bfloat16& m, __nv_bfloat16& l) {
  h = __float2bfloat16(x);
  const float r = x - __bfloat162float(h);
  m = __float2bfloat16(r);
  l = __float2bfloat16(r - __bfloat162float(m));
}
}  // namespace tc

// The M-side operand. blocked: the row-blocked window planes (element (i, j)
// of plane q at p[((q nrb + i / 64) cols + j) 64 + i % 64]), with the output's
// rows along i (mn) or along j; else K-major rows of ld elements, pstride
// between planes.
struct X3A {
  const __nv_bfloat16* p;
  bool blocked, mn;
  int64_t cols, nrb, ld, pstride;
};
// The N-side operand: K-major rows.
struct X3B {
  const __nv_bfloat16* p;
  int64_t ld, pstride;
};
// Room for the parts of cut tiles.
size_t x3_part_bytes(const skema_ctx* c);
// The words that decide a product: word, of its own operands (null: no check),
// and all (may be null), of the call, which a refused word marks as refused.
struct X3Words {
  const uint32_t* word;
  uint32_t* all;
};
__device__ __forceinline__ bool x3_skip(const X3Words& w) {
  return (w.word && x3_refused(*w.word)) || (w.all && x3_refused(*w.all));
}
// acc(i, j) = sum_kk A(i, kk) B(j, kk) into o; nothing when refused.
void x3_gemm(skema_ctx* c, const X3A& a, const X3B& b, int64_t M, int64_t N, int64_t K, const tc::X3Out& o, float* part,
             X3Words words);
// A strided FP32 block into row-blocked planes (zero rows up to a multiple of
// 64); its magnitudes are noted in *flag, 2^top and above as big, here and below
// (null: not), those below 2^bottom (-90 elsewhere) as tiny.
void x3_block_planes(skema_ctx* c, Mat src, int64_t rows, int64_t cols, __nv_bfloat16* D, int64_t pstride, int top,
                     int bottom, uint32_t* flag);

// K-major planes of a row-major source's transpose: row i of S (rows x cols,
// rs apart), scaled by nu^(nwin - 1 - (j0 + i) / W), is K index i; D holds
// cols rows of ld (a multiple of 8) per plane.
void x3_transposed_planes(skema_ctx* c, const float* S, int64_t rs, int64_t rows, int64_t cols, __nv_bfloat16* D,
                          int64_t ld, int64_t pstride, float nu, int64_t W, int64_t nwin, int64_t j0, int top,
                          uint32_t* flag);
// K-major planes of a row-major source (rows x cols, rs apart): D holds rows of
// ld (a multiple of 8) per plane.
void x3_row_planes(skema_ctx* c, const float* S, int64_t rs, int64_t rows, int64_t cols, __nv_bfloat16* D, int64_t ld,
                   int64_t pstride, int top, uint32_t* flag);

// Up to three FP32 products C = alpha A B + beta C by plain FMA, run when
// *flag is refused: the form of a block whose values the planes cannot carry.
struct X3Plain {
  const float* A;
  int64_t ars, acs;
  const __nv_bfloat16* Apl;  // A null: the sum of its planes (aps apart), rows of ald with K along them
  int64_t ald, aps;
  const float* B;
  int64_t brs, bcs;
  float* C;
  int64_t crs, ccs;
  int64_t M, N, K;
  float alpha, beta;
  int split;  // above 1: K in so many parts, added to C (beta not applied)
};
struct X3Plain3 {
  X3Plain g[3];
  int n;
  float* scale;  // nscale values are scaled by `by`: the C of a split product to follow
  int64_t nscale;
  float by;
};
int x3_plain_split(const skema_ctx* c, int64_t s, int64_t K);
void x3_plain(skema_ctx* c, const X3Plain3& p, const uint32_t* flag);

// One call's input: a dense matrix, or a filler of window planes (A.p null)
// whose values are at most 1 in magnitude or NaN.
struct X3Input {
  Mat A;
  std::function<void(int64_t R0, int64_t wr, __nv_bfloat16* planes, int64_t pstride)> fill;
  size_t otherwise;  // the SIMT form's workspace (try_workspace)
};
// All windows of one call of a Gauss-map FP32 context. False (and nothing
// done) when the call is small, its workspace is not to be had, or nu or the
// maps are outside the form's range: the caller then takes the SIMT form.
bool x3_update(skema_ctx* c, const X3Input& in, int64_t row0, int64_t nrows);

}  // namespace skema
