// Galerkin coarse operator A_c = P A P^T on the GPU (AMGSolver::getPMPt,
// src/AMGSolver.cpp:288-358).
//
// Symbolic phase: one warp per coarse row (a block per row when there are few
// rows) collects the column set {c : c in Pt[b], b in A[a], a in P[i]} and
// writes it as [i, ascending others] -- the pattern getPMPt builds and
// compresses.  The set is a bitmap in shared memory over the row's column
// window, which the ranges of P^T's rows give beforehand: inserting is one
// load for all but the first product of a column, and reading the bitmap out
// is already sorted.  Windows too wide for that (an unordered numbering of
// more than kMaxWindow columns) take a hash set, sorted afterwards.
//
// Numeric phase: a group of lanes per coarse row walks the (j, k) pairs of
// the triple loop in the reference's order (P row ascending, A row in stored
// order), and the lanes take the entries l of the Pt row, whose columns are
// distinct, so every output entry receives its products in exactly the
// reference's order: row_entry[c] += P(i,a)*A(a,b)*Pt(b,c).  Compiled with
// -fmad=false, the result is bitwise that of getPMPt.
#include <algorithm>
#include <climits>
#include <type_traits>
#include <utility>

#include "common.cuh"
#include "kernels.cuh"

namespace afp {
namespace {

constexpr int WARP_CAP = 1024;      // hash slots of the warp-level symbolic pass
constexpr int BLOCK_CAP = 16384;    // hash slots of the block-level pass (2 x 64 KB of shared memory)
constexpr size_t NUM_SMEM_MAX = 200 * 1024;  // shared memory the numeric pass may use per block

__device__ __forceinline__ unsigned hash_slot(int key, int cap) {
  return ((unsigned)key * 2654435761u) & (unsigned)(cap - 1);
}

// Inserts key; returns 1 if it was new.  cap is a power of two.  Most products
// of a row repeat a column, so the slot is read before the atomic is tried.
__device__ __forceinline__ int hash_insert(int* table, int cap, int key) {
  unsigned s = hash_slot(key, cap);
  for (int probe = 0; probe < cap; ++probe) {
    int prev = *(volatile int*)&table[s];
    if (prev == -1) prev = atomicCAS(&table[s], -1, key);
    if (prev == -1) return 1;
    if (prev == key) return 0;
    s = (s + 1) & (unsigned)(cap - 1);
  }
  return 0;  // table full: caller checks the count against the capacity
}

template <int GROUP>
__device__ __forceinline__ void group_bitonic_sort(int* buf, int P, int tid) {
  for (int k = 2; k <= P; k <<= 1) {
    for (int j = k >> 1; j > 0; j >>= 1) {
      for (int t = tid; t < P; t += GROUP) {
        int ixj = t ^ j;
        if (ixj > t) {
          int a = buf[t], b = buf[ixj];
          bool up = (t & k) == 0;
          if ((a > b) == up) {
            buf[t] = b;
            buf[ixj] = a;
          }
        }
      }
      if (GROUP == 32) __syncwarp(); else __syncthreads();
    }
  }
}

// Collects the coarse row's column set with GROUP threads (a warp or a block).
// Returns the unique count (may exceed 0.75*cap: the caller re-routes the row).
template <int GROUP>
__device__ int collect_row(int64_t i, const int* __restrict__ prp, const int* __restrict__ pc,
                           const int* __restrict__ arp, const int* __restrict__ ac, const int* __restrict__ trp,
                           const int* __restrict__ tc, int* table, int cap, int tid, int* red) {
  for (int t = tid; t < cap; t += GROUP) table[t] = -1;
  if (GROUP == 32) __syncwarp(); else __syncthreads();
  int mine = 0;
  const int limit = (cap * 3) / 4;
  for (int j = prp[i]; j < prp[i + 1]; ++j) {
    const int a = pc[j];
    const int kb = arp[a], ke = arp[a + 1];
    for (int k = kb + tid; k < ke; k += GROUP) {
      const int b = ac[k];
      for (int l = trp[b]; l < trp[b + 1]; ++l) mine += hash_insert(table, cap, tc[l]);
    }
    if (GROUP == 32) {
      // a row that outgrows the warp's table goes to the block pass: stop
      // here instead of probing a full table for the rest of its products
      int c = mine;
      for (int o = 16; o > 0; o >>= 1) c += __shfl_xor_sync(0xffffffffu, c, o);
      if (c > limit) return c;
    }
  }
  // reduce the count
  int cnt = mine;
  if (GROUP == 32) {
    for (int o = 16; o > 0; o >>= 1) cnt += __shfl_down_sync(0xffffffffu, cnt, o);
    cnt = __shfl_sync(0xffffffffu, cnt, 0);
  } else {
    for (int o = 16; o > 0; o >>= 1) cnt += __shfl_down_sync(0xffffffffu, cnt, o);
    if ((tid & 31) == 0) atomicAdd(red, cnt);
    __syncthreads();
    cnt = *red;
    __syncthreads();
  }
  return cnt;
}

// Sorts the collected set into `out` as [i, ascending others].
template <int GROUP>
__device__ void emit_row(int64_t i, int* table, int* buf, int cap, int cnt, int tid, int* out, int* red) {
  // compact the table into buf
  if (GROUP == 32) {
    int base = 0;
    for (int t0 = 0; t0 < cap; t0 += 32) {
      int t = t0 + tid;
      int key = table[t];
      bool keep = key >= 0 && key != (int)i;
      unsigned mask = __ballot_sync(0xffffffffu, keep);
      if (keep) buf[base + __popc(mask & ((1u << tid) - 1u))] = key;
      base += __popc(mask);
    }
    __syncwarp();
  } else {
    if (tid == 0) *red = 0;
    __syncthreads();
    for (int t = tid; t < cap; t += GROUP) {
      int key = table[t];
      if (key >= 0 && key != (int)i) buf[atomicAdd(red, 1)] = key;
    }
    __syncthreads();
  }
  const int m = cnt - 1;
  int P = 1;
  while (P < m) P <<= 1;
  for (int t = m + tid; t < P; t += GROUP) buf[t] = INT_MAX;
  if (GROUP == 32) __syncwarp(); else __syncthreads();
  group_bitonic_sort<GROUP>(buf, P, tid);
  if (tid == 0) out[0] = (int)i;
  for (int t = tid; t < m; t += GROUP) out[1 + t] = buf[t];
  if (GROUP == 32) __syncwarp(); else __syncthreads();
}

// Warp-level symbolic pass over all rows.  count mode (rowptr == nullptr):
// row_len[i] = unique count, or -1 when the row needs the block-level pass.
__global__ void k_rap_symbolic_warp(int64_t n_c, const int* prp, const int* pc, const int* arp, const int* ac,
                                    const int* trp, const int* tc, int* row_len, const int* rowptr, int* cols,
                                    const unsigned char* big_flag) {
  extern __shared__ int sm_rap[];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, wpb = blockDim.x >> 5;
  int* table = sm_rap + warp * 2 * WARP_CAP;
  int* buf = table + WARP_CAP;
  for (int64_t i = (int64_t)blockIdx.x * wpb + warp; i < n_c; i += (int64_t)gridDim.x * wpb) {
    if (rowptr != nullptr && big_flag[i]) continue;  // handled by the block pass
    int cnt = collect_row<32>(i, prp, pc, arp, ac, trp, tc, table, WARP_CAP, lane, nullptr);
    if (rowptr == nullptr) {
      if (lane == 0) row_len[i] = (cnt > (WARP_CAP * 3) / 4) ? -1 : cnt;
    } else {
      emit_row<32>(i, table, buf, WARP_CAP, cnt, lane, cols + rowptr[i], nullptr);
    }
    __syncwarp();
  }
}

// Block-level symbolic pass over the rows listed in `rows`.
__global__ void k_rap_symbolic_block(const int* rows, int n_rows, int cap, const int* prp, const int* pc,
                                     const int* arp, const int* ac, const int* trp, const int* tc, int* row_len,
                                     const int* rowptr, int* cols, int* overflow) {
  extern __shared__ int sm_rapb[];
  __shared__ int red;
  int* table = sm_rapb;
  int* buf = sm_rapb + cap;
  for (int r = blockIdx.x; r < n_rows; r += gridDim.x) {
    const int64_t i = rows[r];
    if (threadIdx.x == 0) red = 0;
    __syncthreads();
    int cnt = collect_row<256>(i, prp, pc, arp, ac, trp, tc, table, cap, threadIdx.x, &red);
    if (rowptr == nullptr) {
      if (threadIdx.x == 0) {
        if (cnt > (cap * 3) / 4) atomicExch(overflow, 1);
        row_len[i] = cnt;
      }
    } else {
      emit_row<256>(i, table, buf, cap, cnt, threadIdx.x, cols + rowptr[i], &red);
    }
    __syncthreads();
  }
}

__global__ void k_collect_big(const int* row_len, int64_t n, int* rows, int* count, unsigned char* big_flag) {
  int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const bool big = row_len[i] < 0;
  big_flag[i] = big;
  if (big) rows[atomicAdd(count, 1)] = (int)i;
}

// ------------------------------------------------- bitmap symbolic pass
constexpr int kMaxWindow = 128 * 1024;  // columns of a row's window: 16 KB of bitmap per warp

// lo/hi[a] = the first and last column of {Pt[b] : b in A[a]} (INT_MAX, -1 if none)
__global__ void k_rap_fine_range(int64_t n_f, const int* __restrict__ arp, const int* __restrict__ ac,
                                 const int* __restrict__ trp, const int* __restrict__ tc, int* __restrict__ lo,
                                 int* __restrict__ hi) {
  const int64_t a = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) / 8;
  const int lane = threadIdx.x & 7;
  int l = INT_MAX, h = -1;
  if (a < n_f)
    for (int k = arp[a] + lane; k < arp[a + 1]; k += 8) {
      const int tb = trp[ac[k]], te = trp[ac[k] + 1];
      if (tb == te) continue;
      l = min(l, tc[tb]);
      h = max(h, tc[te - 1]);
    }
#pragma unroll
  for (int o = 4; o > 0; o >>= 1) {
    l = min(l, __shfl_xor_sync(0xffffffffu, l, o));
    h = max(h, __shfl_xor_sync(0xffffffffu, h, o));
  }
  if (a < n_f && lane == 0) {
    lo[a] = l;
    hi[a] = h;
  }
}

// the same over the rows a in P[i], with the row's own column when `diag`;
// *window = the widest window in 32-column words
__global__ void k_rap_coarse_range(int64_t n, const int* __restrict__ prp, const int* __restrict__ pc,
                                   const int* __restrict__ flo, const int* __restrict__ fhi, bool diag,
                                   int* __restrict__ lo, int* __restrict__ hi, int* __restrict__ window) {
  const int64_t i = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) / 8;
  const int lane = threadIdx.x & 7;
  int l = INT_MAX, h = -1;
  if (i < n) {
    if (diag) l = h = (int)i;
    for (int j = prp[i] + lane; j < prp[i + 1]; j += 8) {
      l = min(l, flo[pc[j]]);
      h = max(h, fhi[pc[j]]);
    }
  }
#pragma unroll
  for (int o = 4; o > 0; o >>= 1) {
    l = min(l, __shfl_xor_sync(0xffffffffu, l, o));
    h = max(h, __shfl_xor_sync(0xffffffffu, h, o));
  }
  if (i < n && lane == 0) {
    if (h < 0) l = h = 0;  // an empty row
    lo[i] = l;
    hi[i] = h;
  }
  int w = (i < n && h >= 0) ? (h >> 5) - (l >> 5) + 1 : 1;
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) w = max(w, __shfl_xor_sync(0xffffffffu, w, o));
  if ((threadIdx.x & 31) == 0) atomicMax(window, w);
}

// *window = the widest of the windows lo/hi in words; rows without columns get the window [0, 0]
__global__ void k_rap_fine_window(int64_t n, int* __restrict__ lo, int* __restrict__ hi, int* __restrict__ window) {
  const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  int w = 1;
  if (i < n) {
    if (hi[i] < 0) lo[i] = hi[i] = 0;
    w = (hi[i] >> 5) - (lo[i] >> 5) + 1;
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) w = max(w, __shfl_xor_sync(0xffffffffu, w, o));
  if ((threadIdx.x & 31) == 0) atomicMax(window, w);
}

template <int TPR>
__device__ __forceinline__ void row_sync() {
  if (TPR == 32) __syncwarp();
  else __syncthreads();
}

// Row i of P A P^T (pc given) or of A P^T (pc == nullptr: the row's only `a`
// is i) by TPR threads.  rowptr == nullptr: row_len[i] = number of columns.
// Else cols = [i, ascending others] with diag, the ascending columns without.
template <int TPR>
__global__ void __launch_bounds__(256) k_rap_symbolic_bits(int64_t n, int words, bool diag,
                                                           const int* __restrict__ prp, const int* __restrict__ pc,
                                                           const int* __restrict__ arp, const int* __restrict__ ac,
                                                           const int* __restrict__ trp, const int* __restrict__ tc,
                                                           const int* __restrict__ lo, const int* __restrict__ hi,
                                                           int* __restrict__ row_len, const int* __restrict__ rowptr,
                                                           int* __restrict__ cols) {
  extern __shared__ unsigned sm_bits[];
  __shared__ int red[8];
  constexpr int SUB = 8;  // lanes per row of P^T
  const int tid = threadIdx.x % TPR, lane = threadIdx.x & 31, rpb = blockDim.x / TPR;
  unsigned* bits = sm_bits + (size_t)(threadIdx.x / TPR) * words;
  for (int64_t i = (int64_t)blockIdx.x * rpb + threadIdx.x / TPR; i < n; i += (int64_t)gridDim.x * rpb) {
    const int w0 = lo[i] >> 5, nw = (hi[i] >> 5) - w0 + 1;
    for (int t = tid; t < nw; t += TPR) bits[t] = 0u;
    row_sync<TPR>();
    if (diag && tid == 0) bits[(i >> 5) - w0] = 1u << (i & 31);
    row_sync<TPR>();
    const int jb = pc ? prp[i] : 0, je = pc ? prp[i + 1] : 1;
    for (int j = jb; j < je; ++j) {
      const int a = pc ? pc[j] : (int)i;
      const int ke = arp[a + 1];
      for (int k = arp[a] + tid / SUB; k < ke; k += TPR / SUB) {
        const int b = ac[k], te = trp[b + 1];
        for (int l = trp[b] + tid % SUB; l < te; l += SUB) {
          const int c = tc[l];
          unsigned* word = bits + ((c >> 5) - w0);
          const unsigned bit = 1u << (c & 31);
          if (!(*(volatile unsigned*)word & bit)) atomicOr(word, bit);
        }
      }
    }
    row_sync<TPR>();
    if (rowptr == nullptr) {
      int cnt = 0;
      for (int t = tid; t < nw; t += TPR) cnt += __popc(bits[t]);
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) cnt += __shfl_xor_sync(0xffffffffu, cnt, o);
      if (TPR == 32) {
        if (lane == 0) row_len[i] = cnt;
      } else {
        if (lane == 0) red[threadIdx.x >> 5] = cnt;
        __syncthreads();
        if (tid == 0) {
          cnt = 0;
          for (int w = 0; w < TPR / 32; ++w) cnt += red[w];
          row_len[i] = cnt;
        }
      }
    } else if (tid < 32) {  // read out by the row's first warp
      int* out = cols + rowptr[i];
      int at = 0;
      if (diag) {
        if (lane == 0) {
          out[0] = (int)i;
          bits[(i >> 5) - w0] &= ~(1u << (i & 31));
        }
        at = 1;
        __syncwarp();
      }
      for (int t0 = 0; t0 < nw; t0 += 32) {
        unsigned v = t0 + lane < nw ? bits[t0 + lane] : 0u;
        const int c = __popc(v);
        int pre = c;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
          const int y = __shfl_up_sync(0xffffffffu, pre, o);
          if (lane >= o) pre += y;
        }
        const int total = __shfl_sync(0xffffffffu, pre, 31);
        int q = at + pre - c;
        while (v) {
          const int bpos = __ffs(v) - 1;
          v &= v - 1;
          out[q++] = ((w0 + t0 + lane) << 5) + bpos;
        }
        at += total;
      }
    }
    row_sync<TPR>();
  }
}

// out[0] = longest row, out[1] = widest column window in 32-column words of a
// pattern with rows [i, ascending others]
__global__ void k_rap_extent(int64_t n, const int* __restrict__ rowptr, const int* __restrict__ cols,
                             int* __restrict__ out) {
  const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  int len = 0, w = 1;
  if (i < n) {
    const int b = rowptr[i], e = rowptr[i + 1];
    len = e - b;
    if (len > 1) w = (max((int)i, cols[e - 1]) >> 5) - (min((int)i, cols[b + 1]) >> 5) + 1;
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    len = max(len, __shfl_xor_sync(0xffffffffu, len, o));
    w = max(w, __shfl_xor_sync(0xffffffffu, w, o));
  }
  if ((threadIdx.x & 31) == 0) {
    atomicMax(out, len);
    atomicMax(out + 1, w);
  }
}

__device__ __forceinline__ int find_slot(const int* c, int R, int key, int row) {
  if (key == row) return 0;
  int lo = 1, hi = R;
  while (lo < hi) {
    int mid = (lo + hi) >> 1;
    if (c[mid] < key) lo = mid + 1; else hi = mid;
  }
  return lo;
}

// Numeric pass: exact reference accumulation order (see file comment).
// G lanes per coarse row, 32 / G rows side by side in a warp: FP64
// instructions cost a warp 16 clocks however few lanes use them, so lanes
// idle past the end of short P^T rows (4 entries on the finest level, 13 on
// the next) are what this pass would otherwise wait for: 19 ms for the
// 31,833-row product of a 64^3 hierarchy and 1.5 ms for the 139,878-row one; a
// warp per row with one product in flight and a binary search each took 70
// and 6 ms.  The warp's groups run in lockstep: each takes the next up to G
// pairs (a, b) of its row, one per lane, then all go through them U at a time
// -- columns and weights of U rows of P^T loaded, their slots found and products formed, and only then
// added one row of P^T after the other.
// A column's slot is its rank in the row: with RANK a bitmap over the row's
// column window with the words' prefix counts (two shared loads; window <=
// `words`), else a binary search of the row's column list.  Rows accumulate
// in shared memory, or in place in global memory when the longest would not
// fit (GACC).
template <int G, bool RANK, bool GACC>
__global__ void __launch_bounds__(128) k_rap_numeric(
    int64_t n_c, const int* __restrict__ prp, const int* __restrict__ pc, const double* __restrict__ pv,
    const int* __restrict__ arp, const int* __restrict__ ac, const double* __restrict__ av,
    const int* __restrict__ trp, const int* __restrict__ tc, const double* __restrict__ tv,
    const int* __restrict__ rowptr, const int* __restrict__ cols, double* vals, int acc_cap, int words,
    int group_bytes) {
  extern __shared__ __align__(16) unsigned char sm_num[];
  constexpr int NG = 32 / G, U = 4;
  const int lane = threadIdx.x % G, grp = threadIdx.x / G, gpb = blockDim.x / G;
  unsigned char* mine = sm_num + (size_t)grp * group_bytes;
  double* sacc = reinterpret_cast<double*>(mine);
  unsigned char* rest = mine + (GACC ? 0 : (size_t)acc_cap * sizeof(double));
  unsigned* bits = reinterpret_cast<unsigned*>(rest);
  unsigned short* pre = reinterpret_cast<unsigned short*>(bits + words);
  int* scol = reinterpret_cast<int*>(rest);
  const int64_t tiles = (n_c + NG - 1) / NG;  // a warp's rows
  for (int64_t t = (int64_t)blockIdx.x * (gpb / NG) + (threadIdx.x >> 5); t < tiles;
       t += (int64_t)gridDim.x * (gpb / NG)) {
    const int64_t i = t * NG + (threadIdx.x & 31) / G;
    const bool on = i < n_c;
    const int r0 = on ? rowptr[i] : 0, R = on ? rowptr[i + 1] - r0 : 0;
    double* acc = GACC ? vals + r0 : sacc;
    int w0 = 0;
    for (int q = lane; q < R; q += G) acc[q] = 0.0;
    if (RANK) {
      const int cmin = R > 1 ? min((int)i, cols[r0 + 1]) : (int)i, cmax = R > 1 ? max((int)i, cols[r0 + R - 1]) : (int)i;
      w0 = cmin >> 5;
      const int nw = on ? (cmax >> 5) - w0 + 1 : 0;
      for (int q = lane; q < nw; q += G) bits[q] = 0u;
      __syncwarp();
      for (int q = lane; q < R; q += G) {
        const int c = cols[r0 + q];
        atomicOr(bits + ((c >> 5) - w0), 1u << (c & 31));
      }
      __syncwarp();
      int base = 0;
      const int top = __reduce_max_sync(0xffffffffu, nw);
      for (int q0 = 0; q0 < top; q0 += G) {
        const int cnt = q0 + lane < nw ? __popc(bits[q0 + lane]) : 0;
        int sc = cnt;
#pragma unroll
        for (int o = 1; o < G; o <<= 1) {
          const int y = __shfl_up_sync(0xffffffffu, sc, o, G);
          if (lane >= o) sc += y;
        }
        if (q0 + lane < nw) pre[q0 + lane] = (unsigned short)(base + sc - cnt);
        base += __shfl_sync(0xffffffffu, sc, G - 1, G);
      }
    } else {
      if (!GACC)
        for (int q = lane; q < R; q += G) scol[q] = cols[r0 + q];
    }
    __syncwarp();
    const int* rc = GACC ? cols + r0 : scol;
    auto slot_of = [&](int c) -> int {
      if (RANK) {
        const int w = (c >> 5) - w0;
        const int rank = pre[w] + __popc(bits[w] & ((1u << (c & 31)) - 1u));
        return c == (int)i ? 0 : rank + (c < (int)i ? 1 : 0);
      }
      return find_slot(rc, R, c, (int)i);
    };
    int j = on ? prp[i] : 0, k = 0, ke = 0;
    const int je = on ? prp[i + 1] : 0;
    double p = 0.0;
    for (;;) {
      while (k >= ke && j < je) {  // the next row of A that has entries
        const int a = pc[j];
        p = pv[j];
        k = arp[a];
        ke = arp[a + 1];
        ++j;
      }
      const int cnt = min(G, ke - k);
      const int most = __reduce_max_sync(0xffffffffu, cnt);
      if (most <= 0) break;
      int tb = 0, tl = 0;
      double pm = 0.0;
      if (lane < cnt) {
        const int b = ac[k + lane];
        pm = p * av[k + lane];
        tb = trp[b];
        tl = trp[b + 1] - tb;
      }
      const bool fits = !__any_sync(0xffffffffu, tl > G);
      if (fits) {
        for (int q0 = 0; q0 < most; q0 += U) {
          int sl[U];
          double pr[U];
#pragma unroll
          for (int u = 0; u < U; ++u) {
            const int q = min(q0 + u, G - 1);
            const int b0 = __shfl_sync(0xffffffffu, tb, q, G);
            const int len = __shfl_sync(0xffffffffu, tl, q, G);
            const double m = __shfl_sync(0xffffffffu, pm, q, G);
            sl[u] = -1;
            pr[u] = 0.0;
            if (q0 + u < cnt && lane < len) {
              sl[u] = tc[b0 + lane];
              pr[u] = tv[b0 + lane];
            }
            pr[u] = m * pr[u];
          }
#pragma unroll
          for (int u = 0; u < U; ++u)
            if (sl[u] >= 0) sl[u] = slot_of(sl[u]);
#pragma unroll
          for (int u = 0; u < U; ++u) {
            if (sl[u] >= 0) acc[sl[u]] += pr[u];
            __syncwarp();
          }
        }
      } else {
        for (int q = 0; q < most; ++q) {
          const int b0 = __shfl_sync(0xffffffffu, tb, q, G);
          const int len = __shfl_sync(0xffffffffu, tl, q, G);
          const double m = __shfl_sync(0xffffffffu, pm, q, G);
          if (q < cnt)
            for (int l = lane; l < len; l += G) acc[slot_of(tc[b0 + l])] += m * tv[b0 + l];
          __syncwarp();
        }
      }
      k += max(cnt, 0);
    }
    if (!GACC)
      for (int q = lane; q < R; q += G) vals[r0 + q] = sacc[q];
    __syncwarp();
  }
}

// The symbolic count of the product of n_c rows of P: row_len[i] = the unique
// columns of coarse row i.  words > 0: by bitmaps of at most that many
// 32-column words over the windows lo/hi.  Else by hash tables of warps, or of
// blocks for rows that outgrow a warp's table (listed in big, flagged in
// big_flag).
struct SymbolicCount {
  DevBuf<int> row_len, big, lo, hi;
  DevBuf<unsigned char> big_flag;
  int words = 0;
  int hbig = 0, bcap = 1;
  size_t smem_w = 0, smem_b = 0;
  unsigned grid = 1;
};
constexpr int SYM_WPB = 4;

// A bitmap pass over n rows (see k_rap_symbolic_bits): a warp per row, or a
// block where there are too few rows to fill the GPU with warps (256 sampled
// rows of the 64^3 tail: 7 ms with blocks; one warp would walk a row's 3
// million products alone).
void symbolic_bits(const afp_context* ctx, int64_t n, int words, bool diag, const int* prp, const int* pc,
                   const int* arp, const int* ac, const int* trp, const int* tc, const int* lo, const int* hi,
                   int* row_len, const int* rowptr, int* cols) {
  if (n == 0) return;
  auto go = [&](auto Tc, int threads) {
    constexpr int TPR = decltype(Tc)::value;
    const int rpb = threads / TPR;
    const size_t smem = (size_t)rpb * words * sizeof(unsigned);
    allow_smem(k_rap_symbolic_bits<TPR>);
    const unsigned grid = (unsigned)std::min<int64_t>((n + rpb - 1) / rpb, (int64_t)ctx->sm_count * 32);
    k_rap_symbolic_bits<TPR><<<grid, threads, smem, ctx->stream>>>(n, words, diag, prp, pc, arp, ac, trp, tc, lo, hi,
                                                                   row_len, rowptr, cols);
    check_launch(ctx, "rap symbolic (bitmap)");
  };
  if (n < (int64_t)ctx->sm_count * 8) go(std::integral_constant<int, 256>(), 256);
  else go(std::integral_constant<int, 32>(), words <= 1024 ? 256 : words <= 2048 ? 128 : 64);
}

// n_c rows of P over n_f fine rows; n_cols = columns of the product; diag: the
// rows are the product's own (false: a sample of them)
void symbolic_count(const afp_context* ctx, int64_t n_c, int64_t n_f, int64_t n_cols, bool diag, const int* prp,
                    const int* pc, const int* arp, const int* ac, const int* trp, const int* tc, SymbolicCount& sc) {
  sc.row_len.alloc(ctx, n_c);
  sc.lo.alloc(ctx, n_c);
  sc.hi.alloc(ctx, n_c);
  {
    DevBuf<int> flo(ctx, n_f), fhi(ctx, n_f), window(ctx, 1);
    window.zero();
    k_rap_fine_range<<<grid_for(n_f * 8, 256), 256, 0, ctx->stream>>>(n_f, arp, ac, trp, tc, flo.get(), fhi.get());
    check_launch(ctx, "rap fine range");
    k_rap_coarse_range<<<grid_for(n_c * 8, 256), 256, 0, ctx->stream>>>(n_c, prp, pc, flo.get(), fhi.get(), diag,
                                                                        sc.lo.get(), sc.hi.get(), window.get());
    check_launch(ctx, "rap coarse range");
    window.download(&sc.words, 1);
    sync(ctx);
  }
  if (sc.words * 32 <= kMaxWindow) {
    symbolic_bits(ctx, n_c, sc.words, diag, prp, pc, arp, ac, trp, tc, sc.lo.get(), sc.hi.get(), sc.row_len.get(),
                  nullptr, nullptr);
    return;
  }
  sc.words = 0;
  sc.smem_w = (size_t)SYM_WPB * 2 * WARP_CAP * sizeof(int);
  allow_smem(k_rap_symbolic_warp);
  sc.grid = (unsigned)std::min<int64_t>((n_c + SYM_WPB - 1) / SYM_WPB, (int64_t)ctx->sm_count * 16);
  k_rap_symbolic_warp<<<sc.grid, SYM_WPB * 32, sc.smem_w, ctx->stream>>>(n_c, prp, pc, arp, ac, trp, tc,
                                                                         sc.row_len.get(), nullptr, nullptr, nullptr);
  check_launch(ctx, "rap symbolic count");
  // rows whose column set does not fit the warp table go to the block pass
  DevBuf<int> nbig(ctx, 1), overflow(ctx, 1);
  sc.big.alloc(ctx, n_c);
  sc.big_flag.alloc(ctx, n_c);
  nbig.zero();
  overflow.zero();
  k_collect_big<<<grid_for(n_c, 256), 256, 0, ctx->stream>>>(sc.row_len.get(), n_c, sc.big.get(), nbig.get(),
                                                             sc.big_flag.get());
  check_launch(ctx, "rap big rows");
  nbig.download(&sc.hbig, 1);
  sync(ctx);
  while (sc.bcap < 2 * n_cols && sc.bcap < BLOCK_CAP) sc.bcap <<= 1;
  sc.smem_b = (size_t)2 * sc.bcap * sizeof(int);
  if (sc.hbig > 0) {
    allow_smem(k_rap_symbolic_block);
    k_rap_symbolic_block<<<(unsigned)std::min(sc.hbig, ctx->sm_count * 2), 256, sc.smem_b, ctx->stream>>>(
        sc.big.get(), sc.hbig, sc.bcap, prp, pc, arp, ac, trp, tc, sc.row_len.get(), nullptr, nullptr,
        overflow.get());
    check_launch(ctx, "rap symbolic count (block)");
    int hov = 0;
    overflow.download(&hov, 1);
    sync(ctx);
    AFP_REQUIRE(!hov, AFP_ERR_UNSUPPORTED, "Galerkin product row longer than the block-level table");
  }
}

// (longest row, widest window in words) of a pattern
std::pair<int, int> pattern_extent(const afp_context* ctx, int64_t n, const int* rowptr, const int* cols) {
  DevBuf<int> ext(ctx, 2);
  ext.zero();
  k_rap_extent<<<grid_for(n, 256), 256, 0, ctx->stream>>>(n, rowptr, cols, ext.get());
  check_launch(ctx, "rap extent");
  int h[2] = {0, 0};
  ext.download(h, 2);
  sync(ctx);
  return {h[0], h[1]};
}

}  // namespace

int64_t galerkin_nnz(const afp_context* ctx, int64_t n_rows, int64_t n_f, int64_t n_c, const int* prp, const int* pc,
                     const int* arp, const int* ac, const int* trp, const int* tc) {
  SymbolicCount sc;
  symbolic_count(ctx, n_rows, n_f, n_c, false, prp, pc, arp, ac, trp, tc, sc);
  DevBuf<int> rowptr(ctx, n_rows + 1);
  return exclusive_scan(ctx, sc.row_len.get(), rowptr.get(), n_rows);
}

void galerkin_product(const afp_context* ctx, int64_t n_c, int64_t n_f, const int* prp, const int* pc,
                      const double* pv, const int* arp, const int* ac, const double* av, const int* trp,
                      const int* tc, const double* tv, Pattern& out, DevBuf<double>& vals) {
  SymbolicCount sc;
  symbolic_count(ctx, n_c, n_f, n_c, true, prp, pc, arp, ac, trp, tc, sc);
  out.m = out.n = n_c;
  out.rowptr.alloc(ctx, n_c + 1);
  out.nnz = exclusive_scan(ctx, sc.row_len.get(), out.rowptr.get(), n_c);
  out.cols.alloc(ctx, out.nnz);
  if (sc.words > 0) {
    symbolic_bits(ctx, n_c, sc.words, true, prp, pc, arp, ac, trp, tc, sc.lo.get(), sc.hi.get(), nullptr,
                  out.rowptr.get(), out.cols.get());
  } else {
    DevBuf<int> overflow(ctx, 1);
    overflow.zero();
    if (sc.hbig > 0) {
      k_rap_symbolic_block<<<(unsigned)std::min(sc.hbig, ctx->sm_count * 2), 256, sc.smem_b, ctx->stream>>>(
          sc.big.get(), sc.hbig, sc.bcap, prp, pc, arp, ac, trp, tc, sc.row_len.get(), out.rowptr.get(),
          out.cols.get(), overflow.get());
      check_launch(ctx, "rap symbolic fill (block)");
    }
    k_rap_symbolic_warp<<<sc.grid, SYM_WPB * 32, sc.smem_w, ctx->stream>>>(
        n_c, prp, pc, arp, ac, trp, tc, sc.row_len.get(), out.rowptr.get(), out.cols.get(), sc.big_flag.get());
    check_launch(ctx, "rap symbolic fill");
  }
  vals.alloc(ctx, out.nnz);
  const std::pair<int, int> extent = pattern_extent(ctx, n_c, out.rowptr.get(), out.cols.get());
  const int rmax = extent.first, window = extent.second;
  AFP_REQUIRE(rmax <= (BLOCK_CAP * 3) / 4, AFP_ERR_UNSUPPORTED,
              "Galerkin product row longer than the block-level table");
  // Lanes per coarse row, by the mean row of P^T: all lanes of a group take one
  // such row's entries.  Both phases with 8, 16 and 32 lanes (ms): mean 3.3
  // 0.45, 0.50 and 0.60 (2D P2 121^2), 4.2 0.59, 0.65 and 0.93 (40^3), 4.3 2.4,
  // 2.3 and 3.4 (64^3); 5.8 1.9, 1.7 and 2.2 (2D P2 220^2), 6.9 4.9, 3.7 and 4.3
  // (3D P2 24^3); 10.6 3.0, 3.3 and 2.7 (2D P1 300^2), 11.6 6.0, 4.9 and 3.8, 12.9
  // 46, 33 and 27 (64^3), 20.1 14.4, 10.5 and 10.2.  A slot is found by rank where
  // the row windows' bitmaps fit 12 KB a group
  // (64K columns; 0.3 KB for the lattice numbering of a 64^3 mesh), else by
  // binary search.  A group's accumulator is the longest row; blocks of 4, 2
  // or 1 warps, so that two blocks fit an SM, and wider groups if not even
  // one warp's do.
  int64_t pt_nnz = 0;
  {
    int h = 0;
    copy(ctx, &h, trp + n_f, sizeof(int));
    sync(ctx);
    pt_nnz = h;
  }
  const double mean = n_f > 0 ? (double)pt_nnz / (double)n_f : 0.0;
  const bool rank = window <= 2048;
  const int acc_cap = (rmax + 1) / 2 * 2;
  const size_t search_bytes = rank ? (size_t)window * (sizeof(unsigned) + sizeof(unsigned short))
                                   : (size_t)acc_cap * sizeof(int);
  const size_t gb = ((size_t)acc_cap * sizeof(double) + search_bytes + 15) / 16 * 16;
  const bool gacc = gb > NUM_SMEM_MAX;
  const size_t group_bytes = gacc ? (rank ? (search_bytes + 15) / 16 * 16 : 16) : gb;
  int G = mean <= 5.0 ? 8 : mean <= 10.0 ? 16 : 32;
  while (G < 32 && (size_t)(32 / G) * group_bytes > NUM_SMEM_MAX / 2) G *= 2;
  if (gacc) G = 32;
  int warps = 4;
  while (warps > 1 && (size_t)warps * (32 / G) * group_bytes > NUM_SMEM_MAX / 2) warps /= 2;
  const size_t smem = (size_t)warps * (32 / G) * group_bytes;
  const int64_t tiles = (n_c + 32 / G - 1) / (32 / G);
  const unsigned grid = (unsigned)std::min<int64_t>((tiles + warps - 1) / warps, (int64_t)ctx->sm_count * 32);
  auto launch = [&](auto kernel) {
    allow_smem(kernel);
    kernel<<<grid, warps * 32, smem, ctx->stream>>>(n_c, prp, pc, pv, arp, ac, av, trp, tc, tv, out.rowptr.get(),
                                                    out.cols.get(), vals.get(), acc_cap, rank ? window : 0,
                                                    (int)group_bytes);
  };
  if (gacc && rank) launch(k_rap_numeric<32, true, true>);
  else if (gacc) launch(k_rap_numeric<32, false, true>);
  else if (rank && G == 8) launch(k_rap_numeric<8, true, false>);
  else if (rank && G == 16) launch(k_rap_numeric<16, true, false>);
  else if (rank) launch(k_rap_numeric<32, true, false>);
  else if (G == 8) launch(k_rap_numeric<8, false, false>);
  else if (G == 16) launch(k_rap_numeric<16, false, false>);
  else launch(k_rap_numeric<32, false, false>);
  check_launch(ctx, "rap numeric");
}

}  // namespace afp

// ------------------------------------------------------------------------
// Galerkin product of the dense tail.  The coarsest level is only inverted,
// never split again, so it does not need getPMPt's accumulation order and
// takes two products of two matrices, which form each row of T = A P^T once
// instead of once per coarse row that reaches it: T as a CSR matrix (a warp
// per row of A, accumulating in A's entry order in shared memory), then
// A_c = P T (a block per coarse row, P's entry order), both FP64 and
// deterministic.  The result is returned in AFEPack's CSR layout (diagonal
// first, then ascending), keeping the entries that are not exactly zero.
// T's rows are 4 to 6 times sparser than a row of n_c: on the 64^3 hierarchy's
// tail (31,833 -> 6,744 rows) the two products take 7.0 and 2.8 ms, through a
// dense n_f x n_c intermediate they took 30 and 40 ms.
namespace afp {
namespace {

// T = A P^T on the pattern trow/tcol: shared-memory accumulators over the
// row's column window [lo, hi]
__global__ void __launch_bounds__(128) k_rap_at(int64_t nf, int wmax, const int* __restrict__ arp,
                                                const int* __restrict__ ac, const double* __restrict__ av,
                                                const int* __restrict__ trp, const int* __restrict__ tc,
                                                const double* __restrict__ tv, const int* __restrict__ lo,
                                                const int* __restrict__ trow, const int* __restrict__ tcol,
                                                double* __restrict__ tval) {
  extern __shared__ double sm_at[];
  const int lane = threadIdx.x & 31, wpb = blockDim.x >> 5;
  double* acc = sm_at + (size_t)(threadIdx.x >> 5) * wmax;
  for (int64_t i = (int64_t)blockIdx.x * wpb + (threadIdx.x >> 5); i < nf; i += (int64_t)gridDim.x * wpb) {
    const int c0 = lo[i], rb = trow[i], re = trow[i + 1];
    for (int q = rb + lane; q < re; q += 32) acc[tcol[q] - c0] = 0.0;
    __syncwarp();
    const int ke = arp[i + 1];
    for (int k0 = arp[i]; k0 < ke; k0 += 32) {
      const int cnt = min(32, ke - k0);
      int tb = 0, tl = 0;
      double a = 0.0;
      if (lane < cnt) {
        const int b = ac[k0 + lane];
        a = av[k0 + lane];
        tb = trp[b];
        tl = trp[b + 1] - tb;
      }
      for (int q = 0; q < cnt; ++q) {
        const int b0 = __shfl_sync(0xffffffffu, tb, q), len = __shfl_sync(0xffffffffu, tl, q);
        const double m = __shfl_sync(0xffffffffu, a, q);
        for (int l = lane; l < len; l += 32) acc[tc[b0 + l] - c0] += m * tv[b0 + l];
        __syncwarp();
      }
    }
    for (int q = rb + lane; q < re; q += 32) tval[q] = acc[tcol[q] - c0];
    __syncwarp();
  }
}

// row c of A_c = P T into the dense D (zeros outside the row's window too)
__global__ void __launch_bounds__(256) k_rap_pt(int64_t nc, const int* __restrict__ prp, const int* __restrict__ pc,
                                                const double* __restrict__ pv, const int* __restrict__ trow,
                                                const int* __restrict__ tcol, const double* __restrict__ tval,
                                                const int* __restrict__ lo, const int* __restrict__ hi,
                                                double* __restrict__ D) {
  extern __shared__ double sm_pt[];
  const int64_t c = blockIdx.x;
  const int c0 = lo[c], w = hi[c] - c0 + 1;
  for (int t = threadIdx.x; t < w; t += blockDim.x) sm_pt[t] = 0.0;
  __syncthreads();
  for (int q = prp[c]; q < prp[c + 1]; ++q) {
    const int a = pc[q];
    const double p = pv[q];
    const int e = trow[a + 1];
    for (int l = trow[a] + threadIdx.x; l < e; l += blockDim.x) sm_pt[tcol[l] - c0] += p * tval[l];
    __syncthreads();
  }
  double* row = D + c * nc;
  for (int64_t j = threadIdx.x; j < nc; j += blockDim.x) {
    const int64_t t = j - c0;
    row[j] = (t >= 0 && t < w) ? sm_pt[t] : 0.0;
  }
}

// entries of dense row c that are kept: the diagonal always, others if != 0
__global__ void k_dense_row_count(int64_t n, const double* __restrict__ D, int* __restrict__ cnt) {
  const int64_t c = blockIdx.x;
  int local = 0;
  for (int64_t j = threadIdx.x; j < n; j += blockDim.x) local += (j == c || D[c * n + j] != 0.0) ? 1 : 0;
  __shared__ int red[256];
  red[threadIdx.x] = local;
  __syncthreads();
  for (int s = blockDim.x / 2; s > 0; s >>= 1) {
    if ((int)threadIdx.x < s) red[threadIdx.x] += red[threadIdx.x + s];
    __syncthreads();
  }
  if (threadIdx.x == 0) cnt[c] = red[0];
}

// one warp per row: the diagonal first, then the others in ascending order
__global__ void k_dense_row_fill(int64_t n, const double* __restrict__ D, const int* __restrict__ rp,
                                 int* __restrict__ ci, double* __restrict__ va) {
  const int64_t c = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) / 32;
  const int lane = threadIdx.x & 31;
  if (c >= n) return;
  int o = rp[c];
  if (lane == 0) {
    ci[o] = (int)c;
    va[o] = D[c * n + c];
  }
  ++o;
  for (int64_t j0 = 0; j0 < n; j0 += 32) {
    const int64_t j = j0 + lane;
    const double v = j < n ? D[c * n + j] : 0.0;
    const bool keep = j < n && j != c && v != 0.0;
    const unsigned m = __ballot_sync(0xffffffffu, keep);
    if (keep) {
      const int at = o + __popc(m & ((1u << lane) - 1u));
      ci[at] = (int)j;
      va[at] = v;
    }
    o += __popc(m);
  }
}

}  // namespace

// n_c <= 16384 (the caller's limit for a dense tail), so a window of columns
// fits a block's shared memory
void galerkin_product_dense(const afp_context* ctx, int64_t n_c, int64_t n_f, const int* prp, const int* pc,
                            const double* pv, const int* arp, const int* ac, const double* av, const int* trp,
                            const int* tc, const double* tv, Pattern& out, DevBuf<double>& vals) {
  DevBuf<double> D(ctx, n_c * n_c);
  {
    // T's pattern: windows of the fine rows, counted and filled by bitmaps
    DevBuf<int> flo(ctx, n_f), fhi(ctx, n_f), clo(ctx, n_c), chi(ctx, n_c), win(ctx, 2), len(ctx, n_f),
        trow(ctx, n_f + 1);
    win.zero();
    k_rap_fine_range<<<grid_for(n_f * 8, 256), 256, 0, ctx->stream>>>(n_f, arp, ac, trp, tc, flo.get(), fhi.get());
    check_launch(ctx, "rap fine range");
    k_rap_coarse_range<<<grid_for(n_c * 8, 256), 256, 0, ctx->stream>>>(n_c, prp, pc, flo.get(), fhi.get(), true,
                                                                        clo.get(), chi.get(), win.get());
    check_launch(ctx, "rap coarse range");
    k_rap_fine_window<<<grid_for(n_f, 256), 256, 0, ctx->stream>>>(n_f, flo.get(), fhi.get(), win.get() + 1);
    check_launch(ctx, "rap fine window");
    int hw[2] = {1, 1};
    win.download(hw, 2);
    sync(ctx);
    symbolic_bits(ctx, n_f, hw[1], false, nullptr, nullptr, arp, ac, trp, tc, flo.get(), fhi.get(), len.get(),
                  nullptr, nullptr);
    const int64_t tn = exclusive_scan(ctx, len.get(), trow.get(), n_f);
    DevBuf<int> tcol(ctx, tn > 0 ? tn : 1);
    DevBuf<double> tval(ctx, tn > 0 ? tn : 1);
    symbolic_bits(ctx, n_f, hw[1], false, nullptr, nullptr, arp, ac, trp, tc, flo.get(), fhi.get(), nullptr,
                  trow.get(), tcol.get());
    const int wmax = hw[1] * 32;
    int wpb = 4;
    while (wpb > 1 && (size_t)wpb * wmax * sizeof(double) > NUM_SMEM_MAX / 2) wpb /= 2;
    const size_t smem_t = (size_t)wpb * wmax * sizeof(double);
    allow_smem(k_rap_at);
    k_rap_at<<<(unsigned)std::min<int64_t>((n_f + wpb - 1) / wpb, (int64_t)ctx->sm_count * 32), wpb * 32, smem_t,
               ctx->stream>>>(n_f, wmax, arp, ac, av, trp, tc, tv, flo.get(), trow.get(), tcol.get(), tval.get());
    check_launch(ctx, "dense Galerkin A P^T");
    const size_t smem_p = (size_t)hw[0] * 32 * sizeof(double);
    allow_smem(k_rap_pt);
    k_rap_pt<<<(unsigned)n_c, 256, smem_p, ctx->stream>>>(n_c, prp, pc, pv, trow.get(), tcol.get(), tval.get(),
                                                          clo.get(), chi.get(), D.get());
    check_launch(ctx, "dense Galerkin P (A P^T)");
  }
  DevBuf<int> cnt(ctx, n_c);
  k_dense_row_count<<<(unsigned)n_c, 256, 0, ctx->stream>>>(n_c, D.get(), cnt.get());
  check_launch(ctx, "dense row count");
  out.m = out.n = n_c;
  out.rowptr.alloc(ctx, n_c + 1);
  out.nnz = exclusive_scan(ctx, cnt.get(), out.rowptr.get(), n_c);
  out.cols.alloc(ctx, out.nnz);
  vals.alloc(ctx, out.nnz);
  k_dense_row_fill<<<grid_for(n_c * 32, 128), 128, 0, ctx->stream>>>(n_c, D.get(), out.rowptr.get(), out.cols.get(),
                                                                      vals.get());
  check_launch(ctx, "dense row fill");
  sync(ctx);
}

}  // namespace afp
