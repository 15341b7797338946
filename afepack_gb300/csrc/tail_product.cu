// X = T R for the dense coarsest solve of the batched V-cycle: T the n x n
// inverse, R an n x k block, by digit products on the tensor cores
// (digits.cuh).  T is cut once per hierarchy, R every time, both with a scale
// per row (column) and 512 inner indices, so that every 512 inner indices'
// exact sums are put together and added up in FP64.  FP64 hierarchies take 9
// digits a number, mixed-precision ones 7: 49 bits for an inverse held as a
// pair of 48 and a residual of 24.
//
// One block takes 128 rows, all columns (N >= k, 16, 32 or 64) and a run of
// 512-index chunks; partial sums of the runs meet in k_tail_add in order.  A
// product of 128 x N x 16 reads 4 KB of T's digits and 32 N bytes of R's from
// shared memory, 36 to 48 clocks; a chunk is 45 (28) x 32 of them and then
// 128 N entries of five FP64 operations (20K clocks at N = 64).
//
// Measured (GB300), against a double-float product on the FP32 pipe (11
// operations a term) and, in FP64, a warp per row: see tail_product().
#include <algorithm>

#include "common.cuh"
#include "digits.cuh"
#include "kernels.cuh"
#include "tail_product.cuh"

namespace afp {
namespace {

constexpr int kTM = 128;
constexpr int kChunk = 512, kChunkStages = kChunk / kKC;
constexpr int kStages = 2;
constexpr int kThreads = 192;

template <int S>
__global__ void __launch_bounds__(256) k_tail_cut(int64_t n, int64_t np, const double* __restrict__ inv,
                                                  const float* __restrict__ hi, const float* __restrict__ lo,
                                                  int64_t ld, __nv_bfloat16* __restrict__ dig,
                                                  double* __restrict__ scale) {
  const int lane = threadIdx.x & 31;
  const int64_t row = (int64_t)blockIdx.x * 8 + (threadIdx.x >> 5), chunk = blockIdx.y;
  double v[2][8];
#pragma unroll
  for (int h = 0; h < 2; ++h)
#pragma unroll
    for (int e = 0; e < 8; ++e) {
      const int64_t j = chunk * kChunk + 256 * h + 8 * lane + e;
      const bool on = row < n && j < n;
      v[h][e] = !on ? 0.0 : inv != nullptr ? inv[row * ld + j] : (double)hi[row * ld + j] + (double)lo[row * ld + j];
    }
  cut_row<S>(v, lane, np / 8, row, chunk * kChunkStages, dig, scale + chunk * np + row);
}

// The columns of R as rows of N: a warp per column and chunk
template <int S, class X>
__global__ void __launch_bounds__(256) k_tail_cut_rhs(int64_t n, int k, int N, const X* __restrict__ R,
                                                      __nv_bfloat16* __restrict__ dig, double* __restrict__ scale) {
  const int lane = threadIdx.x & 31;
  const int c = blockIdx.x * 8 + (threadIdx.x >> 5);
  const int64_t chunk = blockIdx.y;
  double v[2][8];
#pragma unroll
  for (int h = 0; h < 2; ++h)
#pragma unroll
    for (int e = 0; e < 8; ++e) {
      const int64_t j = chunk * kChunk + 256 * h + 8 * lane + e;
      v[h][e] = c < k && j < n ? (double)R[j * k + c] : 0.0;
    }
  cut_row<S>(v, lane, N / 8, c, chunk * kChunkStages, dig, scale + chunk * N + c);
}

template <int S, int N>
struct Shape {
  static constexpr int kAcc = S < 8 ? S : 8;
  static constexpr uint32_t kA = kTM * kKC * 2, kBb = N * kKC * 2;  // a digit's tile of a stage
  static constexpr uint32_t kStage = S * (kA + kBb);
  static constexpr uint32_t kCols = N >= 64 ? 512 : N >= 32 ? 256 : 128;  // tensor memory columns
  static constexpr size_t kSmem = kStages * kStage + 1024;
};

// Digit sums of one accumulator set -> the entry, times 2^55 (S = 9) or 2^42
// (S = 7).  At 512 inner indices a sum of weight s < 7 is an integer of at most
// (s + 1) 2^21 units; the last accumulator of S = 9 holds the weights 7 and 8,
// rounded here to half a unit of weight 8 (at most 2^30.1 of those).
template <int S, int ACC>
__device__ __forceinline__ double put_together(const float (&v)[ACC]) {
  int w[ACC];
#pragma unroll
  for (int s = 0; s < ACC; ++s)
    w[s] = __float2int_rn(v[s] * __int_as_float((127 + (S == 9 && s == 7 ? 55 : 7 * s)) << 23));
  const long long four = (long long)(w[0] * 128 + w[1]) * 16384 + (long long)(w[2] * 128 + w[3]);  // < 2^42.1
  if constexpr (S == 9) {
    const long long hi = four * 128 + w[4];                                                // < 2^49.1
    const long long lo = (long long)w[5] * 1048576 + ((long long)w[6] * 8192 + w[7]);      // < 2^44
    return fma(exact_double(hi), 0x1p27, exact_double(lo));
  } else {
    const long long lo = (long long)(w[4] * 128 + w[5]) * 128 + w[6];
    return fma(exact_double(four), 0x1p21, exact_double(lo));
  }
}

template <int S, int N>
__global__ void __launch_bounds__(kThreads, 1) k_tail_product(int64_t n, int64_t np, int k, int chunks, int splits,
                                                              const __nv_bfloat16* __restrict__ T,
                                                              const double* __restrict__ st,
                                                              const __nv_bfloat16* __restrict__ R,
                                                              const double* __restrict__ sr,
                                                              double* __restrict__ part, int* __restrict__ error) {
  using Sh = Shape<S, N>;
  constexpr int ACC = Sh::kAcc;
  const int64_t i0 = (int64_t)blockIdx.x * kTM;
  const int split = blockIdx.y;
  const int ch0 = split * chunks / splits, ch1 = (split + 1) * chunks / splits;
  const int64_t groups = np / 8;
  extern __shared__ unsigned char tail_raw[];
  __shared__ uint64_t full[kStages], empty[kStages], done, flushed;
  __shared__ uint32_t tmem_slot;
  const uint32_t base = (smem_u32(tail_raw) + 1023u) & ~1023u;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  // stages of a chunk: the last one's end with n
  auto stages_of = [&](int ch) { return (int)min((int64_t)kChunkStages, (n - (int64_t)ch * kChunk + kKC - 1) / kKC); };
  if (threadIdx.x == 0) {
    for (int s = 0; s < kStages; ++s) {
      bar_init(&full[s], 1);
      bar_init(&empty[s], 1);
    }
    bar_init(&done, 1);
    bar_init(&flushed, 128);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
  }
  if (warp == 5) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&tmem_slot)),
                 "n"(Sh::kCols)
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  const uint32_t tmem = tmem_slot;
  if (warp == 4 && lane == 0) {
    int it = 0;
    bool ok = true;
    for (int ch = ch0; ch < ch1 && ok; ++ch) {
      const int ns = stages_of(ch);
      for (int kc = 0; kc < ns; ++kc, ++it) {
        const int b = it % kStages;
        if (it >= kStages && !bar_wait(&empty[b], ((it / kStages) - 1) & 1)) {
          atomicOr(error, 1);
          ok = false;
          break;
        }
        bar_expect(&full[b], Sh::kStage);
        const uint32_t dst = base + b * Sh::kStage;
        const size_t stage = (size_t)ch * kChunkStages + kc;
        for (int s = 0; s < S; ++s) {
          bulk_load(dst + s * Sh::kA, T + ((stage * S + s) * groups + i0 / 8) * (kKC * 8), Sh::kA, &full[b]);
          bulk_load(dst + S * Sh::kA + s * Sh::kBb, R + (stage * S + s) * (N / 8) * (kKC * 8), Sh::kBb, &full[b]);
        }
      }
    }
    // copies in flight end before the block does
    for (int q = it > kStages ? it - kStages : 0; q < it; ++q)
      if (!bar_wait(&full[q % kStages], (q / kStages) & 1)) atomicOr(error, 1);
  } else if (warp == 5 && lane == 0) {
    int it = 0;
    bool ok = true;
    for (int ch = ch0; ch < ch1; ++ch) {
      const int ns = stages_of(ch);
      // the accumulators of the chunk before have been read
      if (ok && ch > ch0 && !bar_wait(&flushed, (ch - ch0 - 1) & 1)) {
        atomicOr(error, 1);
        ok = false;
      }
      if (ok) asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
      for (int kc = 0; kc < ns && ok; ++kc, ++it) {
        const int b = it % kStages;
        if (!bar_wait(&full[b], (it / kStages) & 1)) {
          atomicOr(error, 1);
          ok = false;
          break;
        }
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        const uint32_t ab = base + b * Sh::kStage, bb = ab + S * Sh::kA;
#pragma unroll 1
        for (int i = 0; i < S; ++i)
          for (int j = 0; i + j < S; ++j)
#pragma unroll
            for (int q = 0; q < kKC / 16; ++q)
              mma(tmem + min(i + j, ACC - 1) * N, mat_desc(ab + i * Sh::kA + q * 256),
                  mat_desc(bb + j * Sh::kBb + q * 256), instr_desc(kTM, N),
                  kc > 0 || i > 0 || j >= ACC || q > 0);  // each accumulator's first product overwrites
        mma_commit(&empty[b]);
      }
      mma_commit(&done);
    }
  } else if (warp < 4) {
    const int64_t row = i0 + warp * 32 + lane;
    double acc[N];
#pragma unroll
    for (int c = 0; c < N; ++c) acc[c] = 0.0;
    for (int ch = ch0; ch < ch1; ++ch) {
      const double rs = st[(int64_t)ch * np + row] * (S == 9 ? 0x1p-67 : 0x1p-54);  // 2^-12 of the digits' scale, the sums' unit
      const double* cs = sr + (int64_t)ch * N;
      if (!bar_wait(&done, (ch - ch0) & 1)) {
        atomicOr(error, 1);
        break;
      }
      asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
#pragma unroll
      for (int c = 0; c < N; c += 8) {
        float v[ACC][8];
#pragma unroll
        for (int s = 0; s < ACC; ++s) tmem_ld8(tmem + ((uint32_t)(warp * 32) << 16) + s * N + c, v[s]);
        asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
        for (int e = 0; e < 8; ++e) {
          float w[ACC];
#pragma unroll
          for (int s = 0; s < ACC; ++s) w[s] = v[s][e];
          acc[c + e] = fma(put_together<S, ACC>(w), rs * cs[c + e], acc[c + e]);
        }
      }
      asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
      asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_u32(&flushed)) : "memory");
    }
    if (row < n) {
      double* o = part + ((int64_t)split * n + row) * k;
#pragma unroll
      for (int c = 0; c < N; ++c)
        if (c < k) o[c] = acc[c];
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  }
  __syncthreads();
  if (warp == 5) {
    __syncwarp();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "n"(Sh::kCols) : "memory");
  }
}

template <class X>
__global__ void k_tail_add(int64_t nk, int parts, const double* __restrict__ part, X* __restrict__ out) {
  const int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= nk) return;
  double s = part[t];
  for (int p = 1; p < parts; ++p) s += part[p * nk + t];
  out[t] = (X)s;
}

int pad_cols(int k) { return k <= 16 ? 16 : k <= 32 ? 32 : 64; }

template <int S, class X>
void product(const afp_context* ctx, const TailDigits& D, TailWork& W, const X* R, X* out, int k, int* error) {
  const int N = pad_cols(k);
  k_tail_cut_rhs<S, X><<<dim3(N / 8, D.chunks), 256, 0, ctx->stream>>>(D.n, k, N, R, W.dig.get(), W.scale.get());
  check_launch(ctx, "tail right-hand side digits");
  auto go = [&](auto Nc) {
    constexpr int NN = decltype(Nc)::value;
    AFP_CUDA(cudaFuncSetAttribute(k_tail_product<S, NN>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                  (int)Shape<S, NN>::kSmem));
    k_tail_product<S, NN><<<dim3((unsigned)(D.np / kTM), W.splits), kThreads, Shape<S, NN>::kSmem, ctx->stream>>>(
        D.n, D.np, k, D.chunks, W.splits, D.dig.get(), D.scale.get(), W.dig.get(), W.scale.get(), W.part.get(),
        error);
  };
  if (N == 16) go(std::integral_constant<int, 16>());
  else if (N == 32) go(std::integral_constant<int, 32>());
  else go(std::integral_constant<int, 64>());
  check_launch(ctx, "tail product");
  k_tail_add<X><<<grid_for(D.n * k, 256), 256, 0, ctx->stream>>>(D.n * k, W.splits, W.part.get(), out);
  check_launch(ctx, "tail sums");
}

}  // namespace

void tail_digits(const afp_context* ctx, int64_t n, const double* inv, const float* hi, const float* lo, int64_t ld,
                 TailDigits& D) {
  D.n = n;
  D.np = (n + kTM - 1) / kTM * kTM;
  D.chunks = (int)((n + kChunk - 1) / kChunk);
  D.digits = inv != nullptr ? 9 : 7;
  D.dig.alloc(ctx, (size_t)D.np * D.chunks * kChunk * D.digits);
  D.scale.alloc(ctx, (size_t)D.np * D.chunks);
  const dim3 grid((unsigned)(D.np / 8), (unsigned)D.chunks);
  if (D.digits == 9)
    k_tail_cut<9><<<grid, 256, 0, ctx->stream>>>(n, D.np, inv, hi, lo, ld, D.dig.get(), D.scale.get());
  else
    k_tail_cut<7><<<grid, 256, 0, ctx->stream>>>(n, D.np, inv, hi, lo, ld, D.dig.get(), D.scale.get());
  check_launch(ctx, "tail digits");
}

void tail_work(const afp_context* ctx, const TailDigits& D, int k, TailWork& W) {
  const int N = pad_cols(k);
  W.dig.alloc(ctx, (size_t)N * D.chunks * kChunk * D.digits);
  W.scale.alloc(ctx, (size_t)N * D.chunks);
  // runs of chunks: as many as give the fewest chunks one after the other on
  // an SM (a block fills one), then the fewest
  const int64_t tiles = D.np / kTM;
  int64_t best = INT64_MAX;
  W.splits = 1;
  for (int s = 1; s <= D.chunks; ++s) {
    const int64_t waves = (tiles * s + ctx->sm_count - 1) / ctx->sm_count;
    const int64_t cost = waves * ((D.chunks + s - 1) / s);
    if (cost < best) {
      best = cost;
      W.splits = s;
    }
  }
  W.part.alloc(ctx, (size_t)W.splits * D.n * k);
}

template <>
void tail_product<double>(const afp_context* ctx, const TailDigits& D, TailWork& W, const double* R, double* X, int k,
                          int* error) {
  product<9, double>(ctx, D, W, R, X, k, error);
}
template <>
void tail_product<float>(const afp_context* ctx, const TailDigits& D, TailWork& W, const float* R, float* X, int k,
                         int* error) {
  product<7, float>(ctx, D, W, R, X, k, error);
}

}  // namespace afp
