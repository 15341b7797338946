// X = T R for the dense coarsest solve of the batched V-cycle: T the n x n
// inverse of a symmetric positive definite matrix, R an n x k block, by digit
// products on the tensor cores (digits.cuh).  T's rows and columns are scaled
// by powers of two to a diagonal near one, which bounds its other entries, and
// R's rows against it (exact); T is cut once per hierarchy, R every time, both
// with a scale per row (column) and 512 inner indices, so that every 512 inner
// indices' sums are put together and added up in FP64.
//
// Error against extended precision, the largest entry in units of sum |T||R|
// (GB300, 729 rows, 7-point matrices with random cell coefficients of contrast
// 1e2, 1e4 and 1e8): 1.3e-16, 2.0e-16 and 2.1e-15; the FP64 sums of the row
// kernel 2.7e-15, 4.7e-15 and 4.8e-15.  In mixed precision (T a pair of 48 bits, R
// FP32) the same digits: the result's own rounding to FP32 is all that shows.
// With nine digits, unscaled, it was 1e-11 at 1e8, with seven for mixed precision
// 2e-7 of the entries at 1e4 and 1e-4 at 1e8.
//
// One block takes 128 rows, all columns (N >= k, 16, 32 or 64) and a run of
// 512-index chunks; partial sums of the runs meet in k_tail_add in order.  A
// product of 128 x N x 16 reads 4 KB of T's digits and 32 N bytes of R's from
// shared memory, 36 to 48 clocks; a chunk is 55 x 32 of them and then 128 N
// entries of five FP64 operations (20K clocks at N = 64).  Times against the row
// kernels: digit_tail_rows in mrhs.cu.
#include <algorithm>

#include "common.cuh"
#include "digits.cuh"
#include "kernels.cuh"
#include "tail_product.cuh"

namespace afp {
namespace {

constexpr int kChunk = 512, kChunkStages = kChunk / kKC;
static_assert(kTailEntryBytes == 2.0 * kDigits, "kTailEntryBytes");

// The largest difference of the rows' exponents with which the digits are used.
// A residual whose entries are of their matrix rows' size spreads, scaled, by as
// many bits as the exponents do; a column's digits count from its largest
// entry, and of their 70 bits FP64's 53 are to be left to the smallest.
constexpr int kSpread = 7 * kDigits - 53;

// e[i] with 2^e T_ii 2^e in [1/2, 2) (T from inv, or from hi + lo).  *flag (3
// words, zeros): not zero unless every T_ii is a number in [2^-400, 2^400]; the
// largest of 512 + e and of 512 - e.
__global__ void k_tail_exponents(int64_t n, const double* __restrict__ inv, const float* __restrict__ hi,
                                 const float* __restrict__ lo, int64_t ld, int* __restrict__ e,
                                 int* __restrict__ flag) {
  const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const int64_t q = i * ld + i;
  const double d = inv != nullptr ? inv[q] : (double)hi[q] + (double)lo[q];
  if (!(d >= 0x1p-400 && d <= 0x1p400)) flag[0] = 1;
  const int b = balance(d);
  e[i] = b;
  atomicMax(flag + 1, 512 + b);
  atomicMax(flag + 2, 512 - b);
}

// T scaled and cut: rows and columns by 2^e; the rows' own 2^-e into their scales
__global__ void __launch_bounds__(256) k_tail_cut(int64_t n, int64_t np, const double* __restrict__ inv,
                                                  const float* __restrict__ hi, const float* __restrict__ lo,
                                                  int64_t ld, const int* __restrict__ ex,
                                                  __nv_bfloat16* __restrict__ dig, double* __restrict__ scale) {
  const int lane = threadIdx.x & 31;
  const int64_t row = (int64_t)blockIdx.x * 8 + (threadIdx.x >> 5), chunk = blockIdx.y;
  const int er = row < n ? ex[row] : 0;
  double v[2][8];
#pragma unroll
  for (int h = 0; h < 2; ++h)
#pragma unroll
    for (int e = 0; e < 8; ++e) {
      const int64_t j = chunk * kChunk + 256 * h + 8 * lane + e;
      v[h][e] = 0.0;
      if (row < n && j < n) {
        const double t = inv != nullptr ? inv[row * ld + j] : (double)hi[row * ld + j] + (double)lo[row * ld + j];
        v[h][e] = t * pow2(er + ex[j]);
      }
    }
  cut_row(v, lane, np / 8, row, chunk * kChunkStages, dig, scale + chunk * np + row, -er);
}

// The columns of R as rows of N, its rows scaled by 2^-e: a warp per column and chunk
template <class X>
__global__ void __launch_bounds__(256) k_tail_cut_rhs(int64_t n, int k, int N, const X* __restrict__ R,
                                                      const int* __restrict__ ex, __nv_bfloat16* __restrict__ dig, double* __restrict__ scale) {
  const int lane = threadIdx.x & 31;
  const int c = blockIdx.x * 8 + (threadIdx.x >> 5);
  const int64_t chunk = blockIdx.y;
  double v[2][8];
#pragma unroll
  for (int h = 0; h < 2; ++h)
#pragma unroll
    for (int e = 0; e < 8; ++e) {
      const int64_t j = chunk * kChunk + 256 * h + 8 * lane + e;
      v[h][e] = c < k && j < n ? (double)R[j * k + c] * pow2(-ex[j]) : 0.0;
    }
  cut_row(v, lane, N / 8, c, chunk * kChunkStages, dig, scale + chunk * N + c);
}

template <int N>
__global__ void __launch_bounds__(kDigitThreads, 1) k_tail_product(int64_t n, int64_t np, int k, int chunks, int splits,
                                                                const __nv_bfloat16* __restrict__ T,
                                                                const double* __restrict__ st,
                                                                const __nv_bfloat16* __restrict__ R,
                                                                const double* __restrict__ sr,
                                                                double* __restrict__ part, int* __restrict__ error) {
  const int64_t i0 = (int64_t)blockIdx.x * kTM;
  const int split = blockIdx.y;
  const int ch0 = split * chunks / splits, ch1 = (split + 1) * chunks / splits;
  extern __shared__ unsigned char tail_raw[];
  __shared__ DigitPipe pipe;
  const uint32_t base = (smem_u32(tail_raw) + 1023u) & ~1023u;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  // stages of a chunk: the last one's end with n
  auto stages_of = [&](int ch) { return (int)min((int64_t)kChunkStages, (n - (int64_t)ch * kChunk + kKC - 1) / kKC); };
  const uint32_t tmem = pipe_begin<N>(pipe);
  if (warp == 4 && lane == 0) {
    int it = 0;
    bool ok = true;
    for (int ch = ch0; ch < ch1 && ok; ++ch) {
      const int ns = stages_of(ch);
      for (int kc = 0; kc < ns && ok; ++kc) {
        const int64_t stage = (int64_t)ch * kChunkStages + kc;
        ok = pipe_load<N>(pipe, base, it, T + digit_offset(np / 8, stage, 0, i0, 0), np * kKC,
                          R + digit_offset(N / 8, stage, 0, 0, 0), N * kKC);
        it += ok;
      }
    }
    if (!pipe_drain(pipe, it) || !ok) atomicOr(error, 1);
  } else if (warp == 5 && lane == 0) {
    int it = 0;
    bool ok = true;
    for (int ch = ch0; ch < ch1; ++ch) {
      // the accumulators of the chunk before have been read
      if (ok && ch > ch0) ok = bar_wait(&pipe.flushed, (ch - ch0 - 1) & 1);
      asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
      const int ns = stages_of(ch);
      for (int kc = 0; kc < ns && ok; ++kc, ++it) ok = pipe_issue<N>(pipe, base, tmem, it, kc == 0);
      mma_commit(&pipe.done);
    }
    if (!ok) atomicOr(error, 1);
  } else if (warp < 4) {
    const int64_t row = i0 + warp * 32 + lane;
    double acc[N];
#pragma unroll
    for (int c = 0; c < N; ++c) acc[c] = 0.0;
    for (int ch = ch0; ch < ch1; ++ch) {
      const double rs = st[(int64_t)ch * np + row] * 0x1p-62;  // put_together's unit
      const double* cs = sr + (int64_t)ch * N;
      if (!bar_wait(&pipe.done, (ch - ch0) & 1)) {
        atomicOr(error, 1);
        break;
      }
      asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
#pragma unroll
      for (int c = 0; c < N; c += 8) {
        float v[kAcc][8];
        pipe_read8<N>(tmem, c, v);
#pragma unroll
        for (int e = 0; e < 8; ++e) {
          float w[kAcc];
#pragma unroll
          for (int s = 0; s < kAcc; ++s) w[s] = v[s][e];
          const DigitSum sum = put_together(w);
          acc[c + e] = fma(fma(sum.hi, 0x1p34, sum.lo), rs * cs[c + e], acc[c + e]);
        }
      }
      asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
      asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_u32(&pipe.flushed)) : "memory");
    }
    if (row < n) {
      double* o = part + ((int64_t)split * n + row) * k;
#pragma unroll
      for (int c = 0; c < N; ++c)
        if (c < k) o[c] = acc[c];
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  }
  pipe_end<N>(tmem);
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

}  // namespace

bool tail_digits(const afp_context* ctx, int64_t n, const double* inv, const float* hi, const float* lo, int64_t ld,
                 TailDigits& D) {
  D.n = n;
  D.np = (n + kTM - 1) / kTM * kTM;
  D.chunks = (int)((n + kChunk - 1) / kChunk);
  D.ex.alloc(ctx, n);
  DevBuf<int> flag(ctx, 3);
  flag.zero();
  k_tail_exponents<<<grid_for(n, 256), 256, 0, ctx->stream>>>(n, inv, hi, lo, ld, D.ex.get(), flag.get());
  check_launch(ctx, "tail exponents");
  int hf[3] = {0, 0, 0};
  flag.download(hf, 3);
  sync(ctx);
  if (hf[0] || hf[1] + hf[2] - 1024 > kSpread) return false;
  D.dig.alloc(ctx, (size_t)D.np * D.chunks * kChunk * kDigits);
  D.scale.alloc(ctx, (size_t)D.np * D.chunks);
  k_tail_cut<<<dim3((unsigned)(D.np / 8), (unsigned)D.chunks), 256, 0, ctx->stream>>>(
      n, D.np, inv, hi, lo, ld, D.ex.get(), D.dig.get(), D.scale.get());
  check_launch(ctx, "tail digits");
  return true;
}

void tail_work(const afp_context* ctx, const TailDigits& D, int k, TailWork& W) {
  const int N = pad_cols(k);
  W.dig.alloc(ctx, (size_t)N * D.chunks * kChunk * kDigits);
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

template <class X>
void tail_product(const afp_context* ctx, const TailDigits& D, TailWork& W, const X* R, X* out, int k, int* error) {
  const int N = pad_cols(k);
  k_tail_cut_rhs<X><<<dim3(N / 8, D.chunks), 256, 0, ctx->stream>>>(D.n, k, N, R, D.ex.get(), W.dig.get(),
                                                                    W.scale.get());
  check_launch(ctx, "tail right-hand side digits");
  auto go = [&](auto Nc) {
    constexpr int NN = decltype(Nc)::value;
    constexpr size_t smem = DigitTile<NN>::kSmem;
    AFP_CUDA(cudaFuncSetAttribute(k_tail_product<NN>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    k_tail_product<NN><<<dim3((unsigned)(D.np / kTM), W.splits), kDigitThreads, smem, ctx->stream>>>(
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
template void tail_product<double>(const afp_context*, const TailDigits&, TailWork&, const double*, double*, int, int*);
template void tail_product<float>(const afp_context*, const TailDigits&, TailWork&, const float*, float*, int, int*);

}  // namespace afp
