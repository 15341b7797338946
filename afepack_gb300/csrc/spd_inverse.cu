// Dense inverse of a symmetric positive definite matrix (the coarsest level
// of the hierarchy), with the cubic work on the tensor cores.
//
// Block sweep in place on the lower triangle, kB pivots at a time.  With the
// pivot block P, Q = P^-1, the panel C (rows of the panel's columns; for rows
// already swept the panel's rows, transposed) and the rest S,
//   S_ij <- S_ij -+ (C_i Q) C_j^T,   C_i <- -+ C_i Q,   P <- Q
// (minus for rows below the panel, plus for rows already swept), which after
// the last panel leaves the inverse.  Symmetry halves the work; a positive
// definite matrix needs no pivoting, as every block pivot is a Schur
// complement of it.
//
// FP64 arithmetic runs at 2 multiply-adds a clock and SM here, so the n^3
// part of a 6,744-row inverse is at least 0.25 s in FP64 even with symmetry.
// The two products of a panel are therefore formed from digits (digits.cuh),
// after the matrix has been scaled by powers of two to a diagonal near one
// (exact; the inverse is scaled back).  Error against extended precision on 729
// rows of 7-point matrices with random cell coefficients of contrast 1e2, 1e4
// and 1e8: 8e-16, 6e-16 and 6e-16 of the inverse's norm (pivoted FP64 sweep:
// 10e-16, 9e-16, 8e-16), and the worst entry of the median row, against itself,
// 4e-15, 1.6e-14 and 2.5e-13 (5e-15, 1.5e-14 and 2.3e-13).  Without the scaling
// the last is three times as large, and with nine digits small entries lose
// two decimals more at 1e4 and 1e8.
//
// Measured (GB300, whole inverse): 6,744 rows 34.5 ms against 706 ms with the
// pivoted FP64 sweep of solve.cu (two launches per pivot, FP64 products);
// 2,200 rows 4.0 ms, 256 rows 0.39 ms.
#include <cuda_bf16.h>

#include <algorithm>
#include <cstdint>

#include "common.cuh"
#include "digits.cuh"
#include "launch.cuh"
#include "solve.cuh"

namespace afp {
namespace {

constexpr int kB = 256;         // panel width
constexpr int kNK = kB / kKC;   // stages of one product
constexpr int kTN = 64;         // columns of an output tile: its accumulators fill tensor memory
constexpr int kSub = 16;        // pivots per step of the panel's own inverse

// ------------------------------------------------------------- eligibility
// flag |= 1 unless the matrix is symmetric to rounding with a positive
// diagonal in [2^-400, 2^400] (the digits' scales stay normal numbers) and no
// entry above what the diagonal of a positive definite one allows
__global__ void k_spd_check(int64_t n, const double* __restrict__ M, int* __restrict__ flag) {
  __shared__ double tr[32][33];
  const int64_t i0 = (int64_t)blockIdx.y * 32, j0 = (int64_t)blockIdx.x * 32;
  if (j0 > i0) return;
  for (int r = threadIdx.y; r < 32; r += 8) {
    const int64_t i = j0 + r, j = i0 + threadIdx.x;
    tr[r][threadIdx.x] = (i < n && j < n) ? M[i * n + j] : 0.0;
  }
  __syncthreads();
  bool bad = false;
  for (int r = threadIdx.y; r < 32; r += 8) {
    const int64_t i = i0 + r, j = j0 + threadIdx.x;
    if (i >= n || j >= n || j > i) continue;
    const double a = M[i * n + j];
    const double di = M[i * n + i], dj = M[j * n + j];
    const double dd = sqrt(di * dj);
    if (!(fabs(a - tr[threadIdx.x][r]) <= 1e-12 * dd && fabs(a) <= dd * (1.0 + 1e-12))) bad = true;
    if (i == j && !(a >= 0x1p-400 && a <= 0x1p400)) bad = true;
  }
  if (__any_sync(0xffffffffu, bad) && threadIdx.x == 0) atomicOr(flag, 1);
}

// e[i] with 2^e M_ii 2^e in [1/2, 2)
__global__ void k_spd_exponents(int64_t n, const double* __restrict__ M, int* __restrict__ e) {
  const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) e[i] = balance(M[i * n + i]);
}

// The lower triangle: M_ij <- 2^(e_i + e_j) M_ij, exact
__global__ void k_spd_scale(int64_t n, const int* __restrict__ e, double* __restrict__ M) {
  const int64_t i = blockIdx.x;
  const int ei = e[i];
  for (int64_t j = threadIdx.x; j <= i; j += blockDim.x) M[i * n + j] *= pow2(ei + e[j]);
}

// ----------------------------------------------------- the panel's inverse
// P (kB x kB, full) <- the pivot block from the lower triangle, the identity
// beyond pb
__global__ void k_spd_pivot_block(int64_t n, int64_t k0, int pb, const double* __restrict__ M,
                                  double* __restrict__ P) {
  const int t = blockIdx.x * blockDim.x + threadIdx.x;
  const int r = t / kB, c = t % kB;
  double v = r == c ? 1.0 : 0.0;
  if (r < pb && c < pb) v = r >= c ? M[(k0 + r) * n + k0 + c] : M[(k0 + c) * n + k0 + r];
  P[t] = v;
}

// One step of the block Gauss-Jordan inverse of P: kSub pivots, from `in` to
// `out`.  A block owns 32 rows x kSub columns; its first warp inverts the
// kSub x kSub pivot itself, in registers (lane l: row l / 2, eight columns),
// instead of one more launch in the chain.  The 256 pivots of a panel follow
// one another, each a reciprocal and a rank-1 update whose FP64 instructions
// take 16 clocks apiece, so every entry is updated by one multiply-add, the
// pivot row and column included: 15 us a step, against 19 by four warps with
// a division and two barriers per pivot.
__global__ void __launch_bounds__(128) k_spd_sweep(int kk, const double* __restrict__ in, double* __restrict__ out,
                                                   int* __restrict__ flag) {
  __shared__ double D[kSub][kSub + 1], R[kSub][kSub + 1], T[kSub][kSub + 1], Cc[32][kSub + 1];
  const int tid = threadIdx.x;
  const int jb = blockIdx.x, ib = blockIdx.y;
  const int p0 = kk * kSub, c0 = jb * kSub, r0 = ib * 32;
  pdl_wait();
  if (*(volatile int*)flag) return;  // a pivot before was not positive: nothing of this is used
  if (tid < 32) {
    const int row = tid >> 1, half = tid & 1;
    double d[8];
#pragma unroll
    for (int e = 0; e < 8; ++e) d[e] = in[(p0 + row) * kB + p0 + half * 8 + e];
    bool bad = false;
#pragma unroll
    for (int q = 0; q < kSub; ++q) {
      const int h = q >> 3, qc = q & 7;
      const double p = __shfl_sync(0xffffffffu, d[qc], 2 * q + h);
      const double f = __shfl_sync(0xffffffffu, d[qc], (tid & ~1) + h);
      bad |= !(p > 0.0);
      const double y = 1.0 / p;
      const double g = row == q ? -y : f * y;
#pragma unroll
      for (int e = 0; e < 8; ++e) {
        double r = __shfl_sync(0xffffffffu, d[e], 2 * q + half);
        const bool pc = half == h && e == qc;  // the pivot's column
        if (pc) r = 1.0;
        d[e] = fma(-g, r, (pc || row == q) ? 0.0 : d[e]);
      }
    }
#pragma unroll
    for (int e = 0; e < 8; ++e) D[row][half * 8 + e] = d[e];
    if (bad && tid == 0) atomicOr(flag, 1);
  } else {
    for (int t = tid - 32; t < kSub * kSub; t += 96) R[t / kSub][t % kSub] = in[(p0 + t / kSub) * kB + c0 + t % kSub];
    for (int t = tid - 32; t < 32 * kSub; t += 96) Cc[t / kSub][t % kSub] = in[(r0 + t / kSub) * kB + p0 + t % kSub];
  }
  const int r = tid / kSub, c = tid % kSub;
  double old[4];
#pragma unroll
  for (int h = 0; h < 4; ++h) old[h] = in[(r0 + r + 8 * h) * kB + c0 + c];
  __syncthreads();
  // T = Q R_j, or Q itself in the pivot's own columns
#pragma unroll
  for (int h = 0; h < 2; ++h) {
    double s = 0;
#pragma unroll
    for (int q = 0; q < kSub; ++q) s += D[r + 8 * h][q] * R[q][c];
    T[r + 8 * h][c] = jb == kk ? D[r + 8 * h][c] : s;
  }
  __syncthreads();
#pragma unroll
  for (int h = 0; h < 4; ++h) {
    const int rr = r + 8 * h, row = r0 + rr;
    double v;
    if (row >= p0 && row < p0 + kSub) {
      v = T[row - p0][c];
    } else {
      v = jb == kk ? 0.0 : old[h];
#pragma unroll
      for (int q = 0; q < kSub; ++q) v -= Cc[rr][q] * T[q][c];
    }
    out[row * kB + c0 + c] = v;
  }
}

// --------------------------------------------------------------- the digits
// C of the panel [k0, k0 + pb) cut into digits; a block takes one 8-row group.
// Rows below the panel read their own columns, rows above it the panel's rows
// transposed, the panel's rows and the padding are zeros.
__global__ void __launch_bounds__(256) k_spd_cut_panel(int64_t n, int64_t k0, int pb, const double* __restrict__ M,
                                                       int64_t groups, __nv_bfloat16* __restrict__ dig,
                                                       double* __restrict__ scale) {
  __shared__ double tile[8][kB + 1];
  const int64_t i0 = (int64_t)blockIdx.x * 8;
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  const int64_t row = i0 + w;
  double v[1][8];
  if (i0 < k0) {  // k0 is a multiple of 8: the whole group is above the panel
    const int j = threadIdx.x;
    if (j < pb) {
#pragma unroll
      for (int e = 0; e < 8; ++e) tile[e][j] = M[(k0 + j) * n + i0 + e];
    } else {
#pragma unroll
      for (int e = 0; e < 8; ++e) tile[e][j] = 0.0;
    }
    __syncthreads();
#pragma unroll
    for (int e = 0; e < 8; ++e) v[0][e] = tile[w][8 * lane + e];
  } else {
    const bool on = row >= k0 + pb && row < n;
#pragma unroll
    for (int e = 0; e < 8; ++e) {
      const int j = 8 * lane + e;
      v[0][e] = (on && j < pb) ? M[row * n + k0 + j] : 0.0;
    }
  }
  cut_row(v, lane, groups, row, 0, dig, scale + row);
}

// A dense `rows` x kB array cut into digits; with M, its rows also go back
// into the panel of the lower triangle: -Z below, +Z^T into the panel's rows
// for the rows above.
__global__ void __launch_bounds__(256) k_spd_cut_dense(int64_t n, int64_t k0, int pb, const double* __restrict__ Z,
                                                       double* __restrict__ M, int64_t groups,
                                                       __nv_bfloat16* __restrict__ dig, double* __restrict__ scale) {
  __shared__ double tile[8][kB + 1];
  const int64_t i0 = (int64_t)blockIdx.x * 8;
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  const int64_t row = i0 + w;
  double v[1][8];
#pragma unroll
  for (int e = 0; e < 8; ++e) v[0][e] = Z[row * kB + 8 * lane + e];
  cut_row(v, lane, groups, row, 0, dig, scale + row);
  if (M == nullptr) return;
#pragma unroll
  for (int e = 0; e < 8; ++e) tile[w][8 * lane + e] = v[0][e];
  __syncthreads();
  const int j = threadIdx.x;
  if (i0 < k0) {
    if (j < pb)
#pragma unroll
      for (int e = 0; e < 8; ++e) M[(k0 + j) * n + i0 + e] = tile[e][j];
  } else if (j < pb) {
#pragma unroll
    for (int e = 0; e < 8; ++e)
      if (i0 + e >= k0 + pb && i0 + e < n) M[(i0 + e) * n + k0 + j] = -tile[e][j];
  }
}

// the pivot block back into the lower triangle
__global__ void k_spd_put_pivot(int64_t n, int64_t k0, int pb, const double* __restrict__ Q, double* __restrict__ M) {
  const int t = blockIdx.x * blockDim.x + threadIdx.x;
  const int r = t / kB, c = t % kB;
  if (r < pb && c <= r) M[(k0 + r) * n + k0 + c] = Q[t];
}

// M_ij <- 2^(e_i + e_j) M_ij in the lower triangle, which the upper one takes too
__global__ void k_spd_mirror(int64_t n, const int* __restrict__ e, double* __restrict__ M) {
  __shared__ double tr[32][33];
  const int64_t i0 = (int64_t)blockIdx.y * 32, j0 = (int64_t)blockIdx.x * 32;
  if (j0 > i0) return;
  for (int r = threadIdx.y; r < 32; r += 8) {
    const int64_t i = i0 + r, j = j0 + threadIdx.x;
    double v = 0.0;
    if (i < n && j <= i) {
      v = M[i * n + j] * pow2(e[i] + e[j]);
      M[i * n + j] = v;
    }
    tr[r][threadIdx.x] = v;
  }
  __syncthreads();
  for (int r = threadIdx.y; r < 32; r += 8) {
    const int64_t i = j0 + r, j = i0 + threadIdx.x;  // (i, j) above the diagonal
    if (i < n && j < n && j > i) M[i * n + j] = tr[threadIdx.x][r];
  }
}

// -------------------------------------------------------- the digit product
constexpr size_t kProdSmem = DigitTile<kTN>::kSmem;

// The sums over digit pairs of a kTM x kTN tile of A B^T (A, B digit arrays of
// kB inner indices).  UPDATE: subtracted from (rows >= k0) or added to the
// tiles of the lower triangle of `out` (row stride ld) that the panel
// [k0, k0 + kB) does not own; otherwise stored to `out`.  One tile per block
// (digits.cuh).  A tile is 880 products of 128 x 64 x 16, which read 6 KB of
// shared memory each (48 clocks, 42K in all), and then 8,192 entries of six
// FP64 operations (25K clocks); the accumulators fill tensor memory, so the two
// do not overlap.  An update of 6,744 rows takes 0.84 ms (875 us with nine digits
// whose products were issued from a rolled loop).
template <bool UPDATE>
__global__ void __launch_bounds__(kDigitThreads, 1) k_spd_product(const __nv_bfloat16* __restrict__ A, int64_t groups_a,
                                                               const double* __restrict__ sa,
                                                               const __nv_bfloat16* __restrict__ B, int64_t groups_b,
                                                               const double* __restrict__ sb, int64_t rows,
                                                               int64_t cols, int64_t k0, double* __restrict__ out,
                                                               int64_t ld, const int* __restrict__ bad,
                                                               int* __restrict__ error) {
  const int64_t i0 = (int64_t)blockIdx.x * kTM, j0 = (int64_t)blockIdx.y * kTN;
  if (*bad) return;  // not positive definite
  if (UPDATE) {
    if (j0 > i0 + kTM - 1) return;
    if ((i0 >= k0 && i0 < k0 + kB) || (j0 >= k0 && j0 < k0 + kB)) return;
  }
  extern __shared__ unsigned char prod_raw[];
  __shared__ DigitPipe pipe;
  const uint32_t base = (smem_u32(prod_raw) + 1023u) & ~1023u;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const uint32_t tmem = pipe_begin<kTN>(pipe);
  if (warp == 4 && lane == 0) {
    int it = 0;
    while (it < kNK && pipe_load<kTN>(pipe, base, it, A + digit_offset(groups_a, it, 0, i0, 0), groups_a * (kKC * 8),
                                      B + digit_offset(groups_b, it, 0, j0, 0), groups_b * (kKC * 8)))
      ++it;
    if (!pipe_drain(pipe, it) || it < kNK) atomicOr(error, 2);
  } else if (warp == 5 && lane == 0) {
    int it = 0;
    while (it < kNK && pipe_issue<kTN>(pipe, base, tmem, it, it == 0)) ++it;
    if (it < kNK) atomicOr(error, 2);
    mma_commit(&pipe.done);
  } else if (warp < 4) {
    // the entries to update, read while the products run: lane l holds columns l and 32 + l of its warp's 32 rows
    const int64_t ja = j0 + lane, jb = j0 + 32 + lane, iw = i0 + warp * 32;
    double old[32][2];
    if (UPDATE) {
#pragma unroll
      for (int r = 0; r < 32; ++r) {
        const int64_t i = iw + r;
        old[r][0] = i < rows && ja <= i ? out[i * ld + ja] : 0.0;
        old[r][1] = i < rows && jb <= i ? out[i * ld + jb] : 0.0;
      }
    }
    const double rs = sa[iw + lane] * (UPDATE && i0 >= k0 ? -0x1p-62 : 0x1p-62);  // put_together's unit
    const double ca = sb[ja], cb = sb[jb];
    if (!bar_wait(&pipe.done, 0)) {
      if (lane == 0) atomicOr(error, 2);
    } else {
      asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
      // the stages are free: warp w puts its rows' sums there
      double2* tile = reinterpret_cast<double2*>(prod_raw + (base - smem_u32(prod_raw))) + warp * 32 * (kTN + 1);
#pragma unroll 1
      for (int c = 0; c < kTN; c += 8) {
        float v[kAcc][8];
        pipe_read8<kTN>(tmem, c, v);
#pragma unroll
        for (int e = 0; e < 8; ++e) {
          float w[kAcc];
#pragma unroll
          for (int s = 0; s < kAcc; ++s) w[s] = v[s][e];
          const DigitSum sum = put_together(w);
          tile[lane * (kTN + 1) + c + e] = make_double2(sum.hi, sum.lo);
        }
      }
      __syncwarp();
#pragma unroll
      for (int r = 0; r < 32; ++r) {
        const int64_t i = iw + r;
        const double s = __shfl_sync(0xffffffffu, rs, r);
        const double2 ta = tile[r * (kTN + 1) + lane], tb = tile[r * (kTN + 1) + 32 + lane];
        const double sca = s * ca, scb = s * cb;
        const double va = fma(ta.y, sca, fma(ta.x, sca * 0x1p34, UPDATE ? old[r][0] : 0.0));
        const double vb = fma(tb.y, scb, fma(tb.x, scb * 0x1p34, UPDATE ? old[r][1] : 0.0));
        if (i < rows && (UPDATE ? ja <= i : ja < cols)) out[i * ld + ja] = va;
        if (i < rows && (UPDATE ? jb <= i : jb < cols)) out[i * ld + jb] = vb;
      }
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  }
  pipe_end<kTN>(tmem);
}

}  // namespace

bool spd_inverse(const afp_context* ctx, int64_t n, double* M) {
  DevBuf<int> flag(ctx, 2);
  flag.zero();
  const dim3 g32((unsigned)((n + 31) / 32), (unsigned)((n + 31) / 32)), b32(32, 8);
  k_spd_check<<<g32, b32, 0, ctx->stream>>>(n, M, flag.get());
  check_launch(ctx, "spd check");
  int hf[2] = {0, 0};
  flag.download(hf, 2);
  sync(ctx);
  if (hf[0]) return false;
  DevBuf<int> ex(ctx, n);
  k_spd_exponents<<<grid_for(n, 256), 256, 0, ctx->stream>>>(n, M, ex.get());
  check_launch(ctx, "spd exponents");
  k_spd_scale<<<(unsigned)n, 256, 0, ctx->stream>>>(n, ex.get(), M);
  check_launch(ctx, "spd scale");
  const int64_t np = (n + kTM - 1) / kTM * kTM, groups = np / 8;
  const bool one = n <= kB;
  DevBuf<double> P0(ctx, kB * kB), P1(ctx, kB * kB), Z, sc, sz, sq;
  DevBuf<__nv_bfloat16> dc, dz, dq;
  if (!one) {
    Z.alloc(ctx, np * kB);
    sc.alloc(ctx, np);
    sz.alloc(ctx, np);
    sq.alloc(ctx, kB);
    dc.alloc(ctx, (size_t)np * kB * kDigits);
    dz.alloc(ctx, (size_t)np * kB * kDigits);
    dq.alloc(ctx, (size_t)kB * kB * kDigits);
    AFP_CUDA(cudaFuncSetAttribute(k_spd_product<false>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kProdSmem));
    AFP_CUDA(cudaFuncSetAttribute(k_spd_product<true>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kProdSmem));
  }
  for (int64_t k0 = 0; k0 < n; k0 += kB) {
    const int pb = (int)std::min<int64_t>(kB, n - k0);
    k_spd_pivot_block<<<kB * kB / 256, 256, 0, ctx->stream>>>(n, k0, pb, M, P0.get());
    check_launch(ctx, "spd pivot block");
    double *in = P0.get(), *out = P1.get();
    for (int kk = 0; kk * kSub < pb; ++kk) {
      launch_pdl(ctx->stream, dim3(kB / kSub, kB / 32), 128, 0, k_spd_sweep, kk, (const double*)in, out, flag.get());
      check_launch(ctx, "spd panel sweep");
      std::swap(in, out);
    }
    if (!one) {
      k_spd_cut_dense<<<kB / 8, 256, 0, ctx->stream>>>(n, k0, pb, in, nullptr, kB / 8, dq.get(), sq.get());
      check_launch(ctx, "spd cut pivot inverse");
      k_spd_cut_panel<<<(unsigned)groups, 256, 0, ctx->stream>>>(n, k0, pb, M, groups, dc.get(), sc.get());
      check_launch(ctx, "spd cut panel");
      k_spd_product<false><<<dim3((unsigned)(np / kTM), kB / kTN), kDigitThreads, kProdSmem, ctx->stream>>>(
          dc.get(), groups, sc.get(), dq.get(), kB / 8, sq.get(), np, kB, k0, Z.get(), kB, flag.get(),
          flag.get() + 1);
      check_launch(ctx, "spd panel product");
      k_spd_cut_dense<<<(unsigned)groups, 256, 0, ctx->stream>>>(n, k0, pb, Z.get(), M, groups, dz.get(), sz.get());
      check_launch(ctx, "spd cut panel product");
      k_spd_product<true><<<dim3((unsigned)(np / kTM), (unsigned)(np / kTN)), kDigitThreads, kProdSmem, ctx->stream>>>(
          dz.get(), groups, sz.get(), dc.get(), groups, sc.get(), n, n, k0, M, n, flag.get(),
          flag.get() + 1);
      check_launch(ctx, "spd update");
    }
    k_spd_put_pivot<<<kB * kB / 256, 256, 0, ctx->stream>>>(n, k0, pb, in, M);
    check_launch(ctx, "spd put pivot");
  }
  k_spd_mirror<<<g32, b32, 0, ctx->stream>>>(n, ex.get(), M);
  check_launch(ctx, "spd mirror");
  flag.download(hf, 2);
  sync(ctx);
  // (a bounded wait that ran out leaves the matrix to the pivoted sweep as well)
  return hf[0] == 0 && hf[1] == 0;
}

}  // namespace afp
