// The dense tail of the batched V-cycle as a digit product (tail_product.cu).
#pragma once

#include <cuda_bf16.h>

#include "common.cuh"

namespace afp {

// The n x n inverse cut into digits (2 bytes each, 9 a number in FP64, 7 in
// mixed precision), laid out once per hierarchy for the tensor cores.
struct TailDigits {
  int64_t n = 0, np = 0;
  int chunks = 0, digits = 0;
  DevBuf<__nv_bfloat16> dig;
  DevBuf<double> scale;
};

// Work space of one batch width: the block's digits and the partial sums.
struct TailWork {
  int splits = 1;
  DevBuf<__nv_bfloat16> dig;
  DevBuf<double> scale, part;
};

// From the FP64 inverse (row stride ld), or from its FP32 pair hi + lo.
void tail_digits(const afp_context* ctx, int64_t n, const double* inv, const float* hi, const float* lo, int64_t ld,
                 TailDigits& D);
void tail_work(const afp_context* ctx, const TailDigits& D, int k, TailWork& W);

// X = T R for n x k row-major blocks, k <= 64; *error |= 1 if a bounded wait
// ran out.  FP64 digits take double blocks, mixed-precision ones float blocks.
template <class X>
void tail_product(const afp_context* ctx, const TailDigits& D, TailWork& W, const X* R, X* out, int k, int* error);

}  // namespace afp
