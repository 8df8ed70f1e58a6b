// x3.h -- FP32 products on the tensor cores through three BF16 planes per
// operand (x3.cu, tc_x3.cuh).
#pragma once
#include <cuda_bf16.h>

#include <functional>

#include "internal.h"

namespace skema {

namespace tc {
// The same for two values, whose BF16 parts lie side by side.
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
// acc(i, j) = sum_kk A(i, kk) B(j, kk) into o; nothing when *flag (may be
// null) is set.
void x3_gemm(skema_ctx* c, const X3A& a, const X3B& b, int64_t M, int64_t N, int64_t K, const tc::X3Out& o, float* part,
             const uint32_t* flag);
// A strided FP32 block into row-blocked planes (zero rows up to a multiple of
// 64); sets *flag when a value is out of the planes' range.
void x3_block_planes(skema_ctx* c, Mat src, int64_t rows, int64_t cols, __nv_bfloat16* D, int64_t pstride,
                     uint32_t* flag);

// K-major planes of a row-major source's transpose: row i of S (rows x cols,
// rs apart), scaled by nu^(nwin - 1 - (j0 + i) / W), is K index i; D holds
// cols rows of ld (a multiple of 8) per plane. *flag (may be null) is set when
// a value is out of the planes' range.
void x3_transposed_planes(skema_ctx* c, const float* S, int64_t rs, int64_t rows, int64_t cols, __nv_bfloat16* D,
                          int64_t ld, int64_t pstride, float nu, int64_t W, int64_t nwin, int64_t j0, uint32_t* flag);
// K-major planes of a row-major source (rows x cols, rs apart): D holds rows of
// ld (a multiple of 8) per plane.
void x3_row_planes(skema_ctx* c, const float* S, int64_t rs, int64_t rows, int64_t cols, __nv_bfloat16* D, int64_t ld,
                   int64_t pstride, uint32_t* flag);

// Up to three FP32 products C = alpha A B + beta C by plain FMA, run when
// *flag is set: the form of a block whose values the planes cannot carry.
// A(i, kk) is scaled by nu^(nwin - 1 - (j0 + kk) / W).
struct X3Plain {
  const float* A;
  int64_t ars, acs;
  const float* B;
  int64_t brs, bcs;
  float* C;
  int64_t crs, ccs;
  int64_t M, N, K;
  float alpha, beta, nu;
  int64_t W, nwin, j0;
};
struct X3Plain3 {
  X3Plain g[3];
  int n;
};
void x3_plain(skema_ctx* c, const X3Plain3& p, const uint32_t* flag);

// One call's input: a dense matrix, or a filler of window planes (A.p null)
// whose values are at most 1 in magnitude or NaN.
struct X3Input {
  Mat A;
  std::function<void(int64_t R0, int64_t wr, __nv_bfloat16* planes, int64_t pstride)> fill;
};
// All windows of one call of a Gauss-map FP32 context. False (and nothing
// done) when the call is small, its workspace is not to be had, or nu or the
// maps are outside the form's range: the caller then takes the SIMT form.
bool x3_update(skema_ctx* c, const X3Input& in, int64_t row0, int64_t nrows);

}  // namespace skema
