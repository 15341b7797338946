// The dense tail of the batched V-cycle as a digit product (tail_product.cu).
#pragma once

#include <cuda_bf16.h>

#include "common.cuh"

namespace afp {

// The n x n inverse cut into digits (ten of 2 bytes a number, rows padded to
// 128 and columns to 512), laid out once per hierarchy for the tensor cores;
// ex: row and column i scaled by 2^ex[i] first.
struct TailDigits {
  int64_t n = 0, np = 0;
  int chunks = 0;
  DevBuf<int> ex;
  DevBuf<__nv_bfloat16> dig;
  DevBuf<double> scale;
};

constexpr double kTailEntryBytes = 20.0;  // of an entry's digits

// Work space of one batch width: the block's digits and the partial sums.
struct TailWork {
  int splits = 1;
  DevBuf<__nv_bfloat16> dig;
  DevBuf<double> scale, part;
};

// From the inverse of a symmetric positive definite matrix in FP64 (row stride
// ld), or from its FP32 pair hi + lo.  False, with nothing allocated that
// counts, if its diagonal is not positive, of extreme size or of too wide a
// range (a factor above 2^34) for a column's digits.
bool tail_digits(const afp_context* ctx, int64_t n, const double* inv, const float* hi, const float* lo, int64_t ld,
                 TailDigits& D);
void tail_work(const afp_context* ctx, const TailDigits& D, int k, TailWork& W);

// X = T R for n x k row-major blocks, k <= 64; *error |= 1 if a bounded wait
// ran out.
template <class X>
void tail_product(const afp_context* ctx, const TailDigits& D, TailWork& W, const X* R, X* out, int k, int* error);

}  // namespace afp
