// Products of FP64 accuracy on the tensor cores.
//
// Every row of an operand is scaled by a power of two and cut into S signed
// digits of 7 bits (|d| <= 64; the cut rounds at 2^-7S of the row's scale),
// digit i stored times 2^-7i in BF16, which holds it exactly (the splitting of
// Ozaki, Ogita, Oishi, Rump, Numer. Algorithms 59, 2012).  A product is the sum
// over digit pairs; pairs of one weight i + j share an FP32 accumulator.  In
// units of their weight a product of two digits is at most 2^12 and a sum over
// up to 512 inner indices and 8 pairs at most 2^24, so the accumulators are
// exact.  An entry's sums are put together in 64-bit integers and FP64.
#pragma once

#include <cuda_bf16.h>

#include <cstdint>

namespace afp {

constexpr int kKC = 32;  // inner indices per pipeline stage

// Digit arrays: [stage kc][digit][8-row group][octet of kKC][8 rows][8
// inner], BF16: any run of row groups of one stage and digit is contiguous in
// the core-matrix order the tensor cores read (8 rows x 16 bytes, next octet
// 128 bytes on, next row group 512 bytes on), so a tile is one bulk copy.
template <int S>
__device__ __forceinline__ size_t digit_offset(int64_t groups, int64_t kc, int s, int64_t row, int octet) {
  return ((((size_t)kc * S + s) * groups + row / 8) * (kKC / 8) + octet) * 64 + (row % 8) * 8;
}

// One warp cuts 256 H inner indices of one row, stages kc0 on: lane l holds
// the inner indices 256 h + 8 l .. 256 h + 8 l + 7 in v[h].
template <int S, int H>
__device__ __forceinline__ void cut_row(const double (&v)[H][8], int lane, int64_t groups, int64_t row, int64_t kc0,
                                        __nv_bfloat16* __restrict__ dig, double* __restrict__ scale) {
  double mx = 0.0;
#pragma unroll
  for (int h = 0; h < H; ++h)
#pragma unroll
    for (int e = 0; e < 8; ++e) mx = fmax(mx, fabs(v[h][e]));
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) mx = fmax(mx, __shfl_xor_sync(0xffffffffu, mx, o));
  // 2^ex > mx, from the exponent bits; a row below 2^-900 counts as zeros
  const int ex = min(900, max(-900, (int)((__double2hiint(mx) >> 20) & 0x7ff) - 1022));
  const double up = __hiloint2double((1023 + 7 * S - 1 - ex) << 20, 0);
#pragma unroll
  for (int h = 0; h < H; ++h) {
    long long w[8];
#pragma unroll
    for (int e = 0; e < 8; ++e) w[e] = __double2ll_rn(v[h][e] * up);
#pragma unroll
    for (int s = S - 1; s >= 0; --s) {
      __align__(16) __nv_bfloat16 d[8];
      const float unit = __int_as_float((127 - 7 * s) << 23);  // 2^-7s
#pragma unroll
      for (int e = 0; e < 8; ++e) {
        long long g = w[e];
        if (s > 0) {
          g = ((w[e] + 64) & 127) - 64;
          w[e] = (w[e] - g) >> 7;
        }
        d[e] = __float2bfloat16_rn((float)(int)g * unit);
      }
      *reinterpret_cast<uint4*>(dig + digit_offset<S>(groups, kc0 + h * 8 + lane / 4, s, row, lane % 4)) =
          *reinterpret_cast<const uint4*>(d);
    }
  }
  if (lane == 0) *scale = __hiloint2double((1023 + ex) << 20, 0);
}

__device__ __forceinline__ uint32_t smem_u32(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }

__device__ __forceinline__ void bar_init(uint64_t* b, int count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(b)), "r"(count) : "memory");
}
__device__ __forceinline__ void bar_expect(uint64_t* b, uint32_t bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_u32(b)), "r"(bytes) : "memory");
}
// false when the phase does not complete within the bound (seconds at most)
__device__ __forceinline__ bool bar_wait(uint64_t* b, uint32_t phase) {
  for (int it = 0; it < (1 << 22); ++it) {
    uint32_t ok;
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
        "selp.b32 %0, 1, 0, p;\n\t}"
        : "=r"(ok)
        : "r"(smem_u32(b)), "r"(phase)
        : "memory");
    if (ok) return true;
  }
  return false;
}
__device__ __forceinline__ void bulk_load(uint32_t dst, const void* src, uint32_t bytes, uint64_t* b) {
  asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(dst),
               "l"(src), "r"(bytes), "r"(smem_u32(b))
               : "memory");
}
// Shared-memory matrix descriptor: no swizzle, K-major, next octet 128 bytes
// on (leading offset), next 8-row group 512 bytes on (stride offset).
__device__ __forceinline__ uint64_t mat_desc(uint32_t addr) {
  return (uint64_t)((addr >> 4) & 0x3fff) | ((uint64_t)(128 >> 4) << 16) | ((uint64_t)(512 >> 4) << 32) |
         ((uint64_t)1 << 46);
}
// FP32 accumulators, both operands BF16 and K-major, m x n
constexpr uint32_t instr_desc(int m, int n) {
  return (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(n / 8) << 17) | ((uint32_t)(m / 16) << 24);
}

__device__ __forceinline__ void mma(uint32_t d, uint64_t a, uint64_t b, uint32_t instr, bool accumulate) {
  asm volatile(
      "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}" ::"r"(d),
      "l"(a), "l"(b), "r"(instr), "r"((uint32_t)accumulate)
      : "memory");
}
__device__ __forceinline__ void mma_commit(uint64_t* b) {
  asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(smem_u32(b))
               : "memory");
}
__device__ __forceinline__ void tmem_ld8(uint32_t addr, float (&v)[8]) {
  uint32_t r[8];
  asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7])
               : "r"(addr));
#pragma unroll
  for (int i = 0; i < 8; ++i) v[i] = __uint_as_float(r[i]);
}

// an integer below 2^51 as a double: placed in the fraction of 3 * 2^51, which is then taken off
__device__ __forceinline__ double exact_double(long long v) {
  return __longlong_as_double(0x4338000000000000LL + v) - 0x1.8p52;
}

}  // namespace afp
