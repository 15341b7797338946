// Products of FP64 accuracy on the tensor cores.
//
// Every row of an operand is scaled by a power of two and cut into kDigits = 10
// signed digits of 7 bits (|d| <= 64; the cut rounds at 2^-70 of the row's
// scale), digit i stored times 2^-7i in BF16, which holds it exactly (the
// splitting of Ozaki, Ogita, Oishi, Rump, Numer. Algorithms 59, 2012).  A
// product is the sum over the digit pairs i + j < kDigits; pairs of one weight
// i + j share an FP32 accumulator.  In units of their weight a product of two
// digits is at most 2^12 and a sum over up to 512 inner indices and 7 pairs
// below 2^24, so the accumulators of the weights 0 to 6 are exact.  Tensor
// memory has no room for more than eight of them: the weights 7, 8 and 9 share
// the last one, which rounds at 2^-24 of its own sum -- 2^-61 of the scales'
// product at the very worst, a few units of weight 9 (2^-63) for digits of
// random sign.  An entry's sums are put together in 64-bit integers and FP64.
//
// A row's scale is that of its largest entry, so an entry that is 2^-17 of it
// still has FP64's 53 bits and a smaller one fewer; callers scale rows and
// columns of graded matrices first (by powers of two, which is exact).
//
// A row that holds an infinity or a NaN gets a NaN for its scale, so that every
// result made from it is NaN.
#pragma once

#include <cuda_bf16.h>

#include <cstdint>

namespace afp {

constexpr int kDigits = 10;
constexpr int kAcc = 8;     // accumulators of an output tile: the weights 0..6, and 7 on
constexpr int kKC = 16;     // inner indices per pipeline stage: the depth of one tensor-core product
constexpr int kStages = 3;  // stages of a block's ring
constexpr int kTM = 128;    // rows of an output tile

// The products of a stage are issued for i = 0.., and for each i for j = 0.. .
constexpr int accumulator(int i, int j) { return i + j < kAcc ? i + j : kAcc - 1; }
// Whether the product of digits i and j is the first into its accumulator, the
// only one that may overwrite what an earlier tile left there.
constexpr bool first_into(int i, int j) { return i == 0 && j < kAcc; }
constexpr bool first_into_is_right() {
  bool seen[kAcc] = {};
  for (int i = 0; i < kDigits; ++i)
    for (int j = 0; i + j < kDigits; ++j) {
      if (first_into(i, j) == seen[accumulator(i, j)]) return false;
      seen[accumulator(i, j)] = true;
    }
  for (bool s : seen)
    if (!s) return false;
  return true;
}
static_assert(first_into_is_right(), "each accumulator is overwritten by its first product and by no other");

// Digit arrays: [stage kc][digit][8-row group][octet of kKC][8 rows][8
// inner], BF16: any run of row groups of one stage and digit is contiguous in
// the core-matrix order the tensor cores read (8 rows x 16 bytes, next octet
// 128 bytes on, next row group 256 bytes on), so a tile is one bulk copy.
__device__ __forceinline__ size_t digit_offset(int64_t groups, int64_t kc, int s, int64_t row, int octet) {
  return ((((size_t)kc * kDigits + s) * groups + row / 8) * (kKC / 8) + octet) * 64 + (row % 8) * 8;
}

// 2^e for a normal result
__device__ __forceinline__ double pow2(int e) { return __hiloint2double((1023 + e) << 20, 0); }

// The scaling of a row and a column whose diagonal entry is d: 2^e d 2^e in
// [1/2, 2) for a positive normal d.
__device__ __forceinline__ int balance(double d) { return -((((__double2hiint(d) >> 20) & 0x7ff) - 1022) >> 1); }

// One warp cuts 256 H inner indices of one row, stages kc0 on: lane l holds
// the inner indices 256 h + 8 l .. 256 h + 8 l + 7 in v[h].  The row's values are
// the digits' sum times *scale; the caller's own factor 2^shift goes in there.
// The top four digits are cut from v, the others from what they leave of it
// (exact); a number is rounded to an integer by adding 3 * 2^51 to it.
template <int H>
__device__ __forceinline__ void cut_row(const double (&v)[H][8], int lane, int64_t groups, int64_t row, int64_t kc0,
                                        __nv_bfloat16* __restrict__ dig, double* __restrict__ scale, int shift = 0) {
  int top = 0;  // high word of the largest |v|; infinities and NaNs are above all numbers
#pragma unroll
  for (int h = 0; h < H; ++h)
#pragma unroll
    for (int e = 0; e < 8; ++e) top = max(top, __double2hiint(v[h][e]) & 0x7fffffff);
  top = __reduce_max_sync(0xffffffffu, top) >> 20;
  const bool finite = top < 0x7ff;
  // 2^ex > |v|; a row below 2^-900 counts as zeros
  const int ex = finite ? max(-900, top - 1022) : 0;
  constexpr double magic = 0x1.8p52;
  const double up = pow2(27 - ex), down = pow2(ex - 27), up2 = pow2(7 * kDigits - 1 - ex);
#pragma unroll
  for (int h = 0; h < H; ++h) {
    int hi[8];
    long long lo[8];
#pragma unroll
    for (int e = 0; e < 8; ++e) {
      const double x = finite ? v[h][e] : 0.0;
      const double t = fma(x, up, magic);
      hi[e] = __double2loint(t);
      lo[e] = __double_as_longlong(fma(fma(-(t - magic), down, x), up2, magic)) - __double_as_longlong(magic);
    }
#pragma unroll
    for (int s = kDigits - 1; s >= 0; --s) {
      __align__(16) __nv_bfloat16 d[8];
      const float unit = __int_as_float((127 - 7 * s) << 23);  // 2^-7s
#pragma unroll
      for (int e = 0; e < 8; ++e) {
        int g;
        if (s >= 4) {
          g = ((int)(lo[e] + 64) & 127) - 64;
          lo[e] = (lo[e] - g) >> 7;
          if (s == 4) hi[e] += (int)lo[e];
        } else {
          g = hi[e];
          if (s > 0) {
            g = ((hi[e] + 64) & 127) - 64;
            hi[e] = (hi[e] - g) >> 7;
          }
        }
        d[e] = __float2bfloat16_rn((float)g * unit);
      }
      *reinterpret_cast<uint4*>(dig + digit_offset(groups, kc0 + h * (256 / kKC) + lane / 2, s, row, lane % 2)) =
          *reinterpret_cast<const uint4*>(d);
    }
  }
  // (a scale beyond the range of normal numbers is taken to its end: below it the row counts for nothing either way)
  if (lane == 0)
    *scale = finite ? pow2(min(1023, max(-1022, ex - 6 + shift))) : __longlong_as_double(0x7ff8000000000000LL);
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
// on (leading offset), next 8-row group 256 bytes on (stride offset).
__device__ __forceinline__ uint64_t mat_desc(uint32_t addr) {
  return (uint64_t)((addr >> 4) & 0x3fff) | ((uint64_t)(128 >> 4) << 16) | ((uint64_t)(256 >> 4) << 32) |
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

// Digit sums of one entry (an accumulator each) as hi 2^34 + lo, in units of
// 2^-62 of the scales' product.  At 512 inner indices a sum of weight s < 7 is
// an integer of at most (s + 1) 2^21 units; the last accumulator is taken apart
// into units of weight 7 (at most 2^24.2) and the rest, rounded at 2^-62.
struct DigitSum {
  double hi, lo;
};
__device__ __forceinline__ DigitSum put_together(const float (&v)[kAcc]) {
  int w[kAcc];
#pragma unroll
  for (int s = 0; s < kAcc; ++s) w[s] = __float2int_rn(v[s] * __int_as_float((127 + 7 * s) << 23));
  const int rest = __float2int_rn(fmaf(-(float)w[7], 0x1p-49f, v[7]) * 0x1p62f);
  const long long hi = ((long long)(w[0] * 128 + w[1]) * 16384 + (w[2] * 128 + w[3])) * 128 + w[4];  // < 2^49.1
  const long long lo = ((long long)(w[5] * 128 + w[6]) * 128 + w[7]) * 8192 + rest;                  // < 2^50.7
  return {exact_double(hi), exact_double(lo)};
}

// ------------------------------------------------- the products of one block
// A block of 192 threads forms a kTM x N tile of A B^T: thread 0 of warp 4
// streams the digits of both operands through a ring of stages, thread 0 of
// warp 5 issues the products, warps 0-3 put the sums together.  Every wait is
// bounded; one that runs out ends its thread's part, and the caller reports it.
constexpr int kDigitThreads = 192;

template <int N>
struct DigitTile {
  static constexpr uint32_t kA = kTM * kKC * 2, kB = N * kKC * 2;  // one digit's rows of a stage
  static constexpr uint32_t kStage = kDigits * (kA + kB);
  static constexpr uint32_t kCols = kAcc * N;  // tensor memory columns
  static constexpr size_t kSmem = kStages * kStage + 1024;
  static_assert(kCols <= 512 && (kCols & (kCols - 1)) == 0 && kSmem > 114 * 1024, "one block per SM");
};

struct DigitPipe {  // in shared memory
  uint64_t full[kStages], empty[kStages], done, flushed;
  uint32_t tmem;
};

// Whole block: barriers and tensor memory; returns the accumulators' address.
template <int N>
__device__ __forceinline__ uint32_t pipe_begin(DigitPipe& p) {
  if (threadIdx.x == 0) {
    for (int s = 0; s < kStages; ++s) {
      bar_init(&p.full[s], 1);
      bar_init(&p.empty[s], 1);
    }
    bar_init(&p.done, 1);
    bar_init(&p.flushed, 128);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
  }
  if (threadIdx.x >> 5 == 5) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&p.tmem)),
                 "n"(DigitTile<N>::kCols)
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  return p.tmem;
}

// Whole block, the warps that read tensor memory after their fence.
template <int N>
__device__ __forceinline__ void pipe_end(uint32_t tmem) {
  __syncthreads();
  if (threadIdx.x >> 5 == 5) {
    __syncwarp();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "n"(DigitTile<N>::kCols)
                 : "memory");
  }
}

// The block's stage number `it` into the ring (base: its address): digit 0 of
// the tile's rows at a and b, the next digits stride_a and stride_b elements on.
template <int N>
__device__ __forceinline__ bool pipe_load(DigitPipe& p, uint32_t base, int it, const __nv_bfloat16* a, size_t stride_a,
                                          const __nv_bfloat16* b, size_t stride_b) {
  using T = DigitTile<N>;
  const int st = it % kStages;
  if (it >= kStages && !bar_wait(&p.empty[st], ((it / kStages) - 1) & 1)) return false;
  bar_expect(&p.full[st], T::kStage);
  const uint32_t dst = base + st * T::kStage;
  for (int s = 0; s < kDigits; ++s) {
    bulk_load(dst + s * T::kA, a + s * stride_a, T::kA, &p.full[st]);
    bulk_load(dst + kDigits * T::kA + s * T::kB, b + s * stride_b, T::kB, &p.full[st]);
  }
  return true;
}

// After `issued` stages: the copies in flight end before the block does.
__device__ __forceinline__ bool pipe_drain(DigitPipe& p, int issued) {
  bool ok = true;
  for (int it = issued > kStages ? issued - kStages : 0; it < issued; ++it)
    ok &= bar_wait(&p.full[it % kStages], (it / kStages) & 1);
  return ok;
}

// The products of stage number `it`; fresh: the accumulators start from them.
template <int N>
__device__ __forceinline__ bool pipe_issue(DigitPipe& p, uint32_t base, uint32_t tmem, int it, bool fresh) {
  using T = DigitTile<N>;
  const int st = it % kStages;
  if (!bar_wait(&p.full[st], (it / kStages) & 1)) return false;
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  const uint32_t ab = base + st * T::kStage, bb = ab + kDigits * T::kA;
#pragma unroll
  for (int i = 0; i < kDigits; ++i)
#pragma unroll
    for (int j = 0; j < kDigits - i; ++j)
      mma(tmem + accumulator(i, j) * N, mat_desc(ab + i * T::kA), mat_desc(bb + j * T::kB), instr_desc(kTM, N),
          !(fresh && first_into(i, j)));
  mma_commit(&p.empty[st]);
  return true;
}

// The accumulators of columns c .. c + 7 of the calling warp's 32 rows.
template <int N>
__device__ __forceinline__ void pipe_read8(uint32_t tmem, int c, float (&v)[kAcc][8]) {
#pragma unroll
  for (int s = 0; s < kAcc; ++s) tmem_ld8(tmem + ((uint32_t)((threadIdx.x >> 5) * 32) << 16) + s * N + c, v[s]);
  asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
}

}  // namespace afp
