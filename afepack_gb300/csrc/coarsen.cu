// C/F splitting and projection on the GPU: AMGSolver::Project
// (src/AMGSolver.cpp:18-226) with the reference's flags and P bit for bit.
//
// The reference's two passes are sequential sweeps in row order.  Both have
// a parallel restatement with the same result:
//
// * Pass 1 (lines 39-68) makes row i a C point iff no earlier C point j < i
//   holds i as a strong neighbour in its own row (|a_ji| >= beta_j).  That
//   is the lexicographically first independent set of the graph j -> i
//   (j < i, strong in row j).  It spreads as a wave: a row without such j is
//   C; a row that became C makes every row it holds F; a row that became F
//   counts down the rows it holds, and one whose count reaches zero is C.
// * Pass 2 (lines 74-126) promotes an F point i to C when some strong F
//   neighbour k > i has no C point in its row that is also a strong C
//   neighbour of i.  The C points i sees are the pass-1 C points and the
//   promoted strong neighbours j < i.  A promotion of j < i can only add to
//   that set, which can only turn i's answer from "promote" to "keep", so a
//   row that would not be promoted against the pass-1 C points alone is
//   final, and a remaining candidate is decided once its candidate strong
//   neighbours below it are decided.  Again a wave, over the (few) candidates.
//
//   A wave is up to a few hundred steps of little work each (192 on the
//   finest level of a 64^3 mesh, 512 of a 256^2 one), so each pass is one
//   kernel of one thread-block cluster: a step costs a cluster barrier
//   (hardware, well under a microsecond) and a few dependent loads, instead of a
//   launch that looks through all rows.  Only rows decided in the step
//   before are touched.  64^3 hierarchy, all levels: pass 1 5.2 ms against
//   17 ms of launches, pass 2 15 against 53 ms.
// * P and P^T (lines 127-216): every fine row's weights are accumulated by
//   one thread (a warp where rows are long) in the reference's order (the
//   same additions into the same entries), so the values are the reference's.
//
// Compiled with -fmad=false: every product and quotient rounds as on the host.
#include <cooperative_groups.h>

#include <cstdint>

#include "common.cuh"
#include "kernels.cuh"

namespace afp {

namespace {

constexpr int kRoundsPerCheck = 16;
constexpr int kWaveThreads = 1024;  // threads per block of a wave's cluster

// the reference's strength test: "if (fabs(a) < beta) continue" skips weak entries
__device__ __forceinline__ bool strong(double a, double beta) { return !(fabs(a) < beta); }

// position of column j among the off-diagonal entries of row i ([diag, ascending others]), or -1
__device__ __forceinline__ int find_offd(const int* __restrict__ rp, const int* __restrict__ ci, int i, int j) {
  int lo = rp[i] + 1, hi = rp[i + 1];
  const int end = hi;
  while (lo < hi) {
    const int mid = (lo + hi) >> 1;
    if (ci[mid] < j) lo = mid + 1;
    else hi = mid;
  }
  return (lo < end && ci[lo] == j) ? lo : -1;
}

// position of column c in a fully ascending row [b, e), or -1
__device__ __forceinline__ int find_sorted(const int* __restrict__ ci, int b, int e, int c) {
  const int end = e;
  while (b < e) {
    const int mid = (b + e) >> 1;
    if (ci[mid] < c) b = mid + 1;
    else e = mid;
  }
  return (b < end && ci[b] == c) ? b : -1;
}

__device__ __forceinline__ int vload(const int* p) { return *(const volatile int*)p; }

// beta_i = alpha * max_j |a_ij| over the off-diagonal entries; one warp per row
__global__ void k_cf_beta(int m, const int* __restrict__ rp, const double* __restrict__ va, double alpha,
                          double* __restrict__ beta) {
  const int i = (int)((blockIdx.x * (int64_t)blockDim.x + threadIdx.x) >> 5);
  const int lane = threadIdx.x & 31;
  if (i >= m) return;
  double b = 0.0;
  for (int j = rp[i] + 1 + lane; j < rp[i + 1]; j += 32) {
    const double a = fabs(va[j]);
    b = (a < b) ? b : a;
  }
  for (int o = 16; o > 0; o >>= 1) {
    const double a = __shfl_xor_sync(0xffffffffu, b, o);
    b = (a < b) ? b : a;
  }
  if (lane == 0) beta[i] = b * alpha;
}

// cnt[i] = number of rows j < i that hold i as a strong neighbour; one warp per row j
__global__ void k_cf_count_in(int m, const int* __restrict__ rp, const int* __restrict__ ci,
                              const double* __restrict__ va, const double* __restrict__ beta, int* __restrict__ cnt) {
  const int j = (int)((blockIdx.x * (int64_t)blockDim.x + threadIdx.x) >> 5);
  const int lane = threadIdx.x & 31;
  if (j >= m) return;
  const double bj = beta[j];
  for (int e = rp[j] + 1 + lane; e < rp[j + 1]; e += 32)
    if (ci[e] > j && strong(va[e], bj)) atomicAdd(cnt + ci[e], 1);
}

// Appends i of the lanes with `push` to list[*count ...]; the whole warp calls it.
__device__ __forceinline__ void push_rows(bool push, int i, int* list, int* count) {
  const unsigned b = __ballot_sync(0xffffffffu, push);
  if (b == 0) return;
  const int lane = threadIdx.x & 31;
  int base = 0;
  if (lane == __ffs(b) - 1) base = atomicAdd(count, __popc(b));
  base = __shfl_sync(0xffffffffu, base, __ffs(b) - 1);
  if (push) list[base + __popc(b & ((1u << lane) - 1u))] = i;
}

// Pass 1 as a wave.  st: 0 undecided, -1 C, 1 F; cnt from k_cf_count_in;
// list: two arrays of m rows (this step's and the next one's); counts[3]
// zeroed.  A row is listed once, when it is decided: F by the compare-and-swap
// that changed it, C by the decrement that reached zero (a row held by a C
// point never gets there, since that point does not count down).  The lists
// and counts are read past the L1 cache, and the cluster barrier orders a
// step's writes before the next step's reads.  A warp takes a row, short ones
// too: a step waits for its longest row (35,237 rows of 14 entries: the whole
// splitting 1.94 ms, with 8 lanes a row 2.52; only on steps of thousands of
// rows do 8 lanes gain, 274,625 rows of 15: 3.60 and 3.33).
__global__ void __launch_bounds__(kWaveThreads) k_cf_pass1_wave(int m, const int* __restrict__ rp,
                                                                const int* __restrict__ ci,
                                                                const double* __restrict__ va,
                                                                const double* __restrict__ beta, int* st, int* cnt,
                                                                int* list, int* counts, int* steps) {
  const cooperative_groups::cluster_group cluster = cooperative_groups::this_cluster();
  const int tid = blockIdx.x * blockDim.x + threadIdx.x, nt = gridDim.x * blockDim.x;
  const int warp = tid >> 5, lane = tid & 31, nw = nt >> 5;
  for (int i0 = 0; i0 < m; i0 += nt) {
    const int i = i0 + tid;
    const bool c = i < m && cnt[i] == 0;
    if (c) st[i] = -1;
    push_rows(c, i, list, counts);
  }
  __threadfence();
  cluster.sync();
  int step = 0;
  for (;; ++step) {
    const int n = __ldcg(counts + step % 3);
    if (n == 0) break;
    const int* cur = list + (size_t)(step & 1) * m;
    int* next = list + (size_t)((step + 1) & 1) * m;
    int* ncount = counts + (step + 1) % 3;
    if (tid == 0) counts[(step + 2) % 3] = 0;
    for (int w = warp; w < n; w += nw) {
      const int j = __ldcg(cur + w);
      const bool is_c = __ldcg(st + j) == -1;
      const double bj = beta[j];
      const int e1 = rp[j + 1];
      for (int e0 = rp[j] + 1; e0 < e1; e0 += 32) {
        const int e = e0 + lane;
        const int i = e < e1 ? ci[e] : -1;
        bool push = false;
        if (i > j && strong(va[e], bj)) {
          if (is_c) {
            push = __ldcg(st + i) == 0 && atomicCAS(st + i, 0, 1) == 0;
          } else if (atomicSub(cnt + i, 1) == 1) {
            st[i] = -1;
            push = true;
          }
        }
        push_rows(push, i, next, ncount);
      }
    }
    __threadfence();
    cluster.sync();
  }
  if (tid == 0) *steps = step;
}

// Pass 2's test for an F point i (one warp): is there a strong neighbour
// k > i, F after pass 1, whose row has no C point that is also a strong C
// neighbour of i?  C points below i are the pass-1 ones and the promoted
// (s2 == 2); above i only the pass-1 ones count (the reference has not
// reached them yet).  With s2 == nullptr no promotion is counted.
//
// i's strong C neighbours go into a hash set in shared memory (`table`,
// kSet slots of the warp's own) and four rows k at a time are looked through,
// 8 lanes each: a binary search of row i in global memory for every entry of
// every row k was 8 dependent loads instead of one shared one.  Rows of more
// strong C neighbours than the set holds are searched that way.
constexpr int kSet = 512;

__device__ __forceinline__ unsigned set_slot(int key) { return ((unsigned)key * 2654435761u) >> 23; }

__device__ __forceinline__ bool strong_c(int j, double a, double bi, int i, const int* __restrict__ st1,
                                         const int* s2) {
  return strong(a, bi) && (st1[j] == -1 || (s2 != nullptr && j < i && __ldcg(s2 + j) == 2));
}

// A block of several warps (WPR) shares the set and splits the rows k, 8 of
// i's entries to a warp at a time; each warp answers for its own.
template <int WPR>
__device__ bool cf_promote(int i, const int* __restrict__ rp, const int* __restrict__ ci,
                           const double* __restrict__ va, const double* __restrict__ beta,
                           const int* __restrict__ st1, const int* s2, int* table, int lane) {
  const double bi = beta[i];
  const int b = rp[i] + 1, e = rp[i + 1];
  const int w = WPR > 1 ? threadIdx.x >> 5 : 0;
  int n = 0;
  for (int q = b + lane; q < e; q += 32) n += strong_c(ci[q], va[q], bi, i, st1, s2);
  n = __reduce_add_sync(0xffffffffu, n);
  const bool set = n <= kSet * 3 / 4;
  if (set) {
    if (WPR > 1) __syncthreads();
    for (int t = w * 32 + lane; t < kSet; t += WPR * 32) table[t] = -1;
    if (WPR > 1) __syncthreads();
    else __syncwarp();
    for (int q = b + w * 32 + lane; q < e; q += WPR * 32) {
      const int j = ci[q];
      if (!strong_c(j, va[q], bi, i, st1, s2)) continue;
      unsigned h = set_slot(j);
      while (atomicCAS(table + h, -1, j) != -1) h = (h + 1) & (kSet - 1);
    }
    if (WPR > 1) __syncthreads();
    else __syncwarp();
  }
  const int sub = lane >> 3, sl = lane & 7;
  constexpr int CH = WPR > 1 ? 8 : 32;  // i's entries to a warp at a time
  constexpr int U = 4;                  // entries of a row k in flight per lane
  for (int q0 = b + w * CH; q0 < e; q0 += WPR * CH) {
    const int q = q0 + lane;
    const int k = lane < CH && q < e ? ci[q] : -1;
    const bool sel = k > i && st1[k] != -1 && strong(va[q], bi);
    const int kb = sel ? rp[k] + 1 : 0, ke = sel ? rp[k + 1] : 0;
    for (unsigned todo = __ballot_sync(0xffffffffu, sel); todo != 0;) {
      unsigned t = todo;
      for (int s = 0; s < sub; ++s) t &= t - 1;
      const int src = t ? __ffs(t) - 1 : 0;
      int at = __shfl_sync(0xffffffffu, kb, src) + sl;
      const int end = __shfl_sync(0xffffffffu, ke, src);
      bool open = t != 0;  // the same for a row's 8 lanes
      bool lacks = false;
      while (__any_sync(0xffffffffu, open)) {
        bool hit = false;
        int k1[U];
#pragma unroll
        for (int u = 0; u < U; ++u) k1[u] = open && at + 8 * u < end ? ci[at + 8 * u] : -1;
#pragma unroll
        for (int u = 0; u < U; ++u) {
          if (k1[u] < 0) continue;
          if (set) {
            unsigned h = set_slot(k1[u]);
            int v;
            while ((v = table[h]) != -1 && v != k1[u]) h = (h + 1) & (kSet - 1);
            hit |= v == k1[u];
          } else {
            const int p = find_offd(rp, ci, i, k1[u]);
            hit |= p >= 0 && strong_c(k1[u], va[p], bi, i, st1, s2);
          }
        }
        const unsigned any = (__ballot_sync(0xffffffffu, hit) >> (sub * 8)) & 0xffu;
        at += 8 * U;
        if (open && any) open = false;
        if (open && at - sl >= end) {
          lacks = true;
          open = false;
        }
      }
      if (__any_sync(0xffffffffu, lacks)) return true;
#pragma unroll
      for (int s = 0; s < 4; ++s) todo &= todo - 1;
    }
  }
  return false;
}

// s2 for every pass-1 F point: 1 (candidate) if it would be promoted against
// the pass-1 C points alone, else 0 (final: promotions below can only add C points)
__global__ void __launch_bounds__(256) k_cf_pass2_candidates(int m, const int* __restrict__ rp,
                                                             const int* __restrict__ ci,
                                                             const double* __restrict__ va,
                                                             const double* __restrict__ beta,
                                                             const int* __restrict__ st1, int* __restrict__ s2) {
  __shared__ int tables[8][kSet];
  const int i = (int)((blockIdx.x * (int64_t)blockDim.x + threadIdx.x) >> 5);
  const int lane = threadIdx.x & 31;
  if (i >= m) return;
  bool cand = false;
  if (st1[i] == 1) cand = cf_promote<1>(i, rp, ci, va, beta, st1, nullptr, tables[threadIdx.x >> 5], lane);
  if (lane == 0) s2[i] = cand ? 1 : 0;
}

// cnt[i] = candidate strong neighbours below candidate i
__global__ void k_cf_pass2_count(int m, const int* __restrict__ rp, const int* __restrict__ ci,
                                 const double* __restrict__ va, const double* __restrict__ beta,
                                 const int* __restrict__ s2, int* __restrict__ cnt) {
  const int i = (int)((blockIdx.x * (int64_t)blockDim.x + threadIdx.x) >> 5);
  const int lane = threadIdx.x & 31;
  if (i >= m) return;
  int n = 0;
  if (s2[i] == 1) {
    const double bi = beta[i];
    for (int e = rp[i] + 1 + lane; e < rp[i + 1]; e += 32) n += ci[e] < i && s2[ci[e]] == 1 && strong(va[e], bi);
  }
  n = __reduce_add_sync(0xffffffffu, n);
  if (lane == 0) cnt[i] = n;
}

// Pass 2 as a wave over the candidates; s2 becomes 2 (promoted) or 0 as they
// are decided.  A decided row j tells the candidates above it that hold it as
// a strong neighbour, found through its own row; where the pattern is not
// symmetric some are not found and stay 1 (*left counts them) for
// k_cf_pass2_round.  Lists and counts as in k_cf_pass1_wave.  A warp takes a
// row, or a whole block while a step has no more than `block_rows` rows: on
// levels of long rows (285 entries: 55 us a row to one warp, and 250 steps
// one after the other) a row's own time is what a step waits for (wave_block_rows).
__global__ void __launch_bounds__(kWaveThreads) k_cf_pass2_wave(int m, const int* __restrict__ rp,
                                                                const int* __restrict__ ci,
                                                                const double* __restrict__ va,
                                                                const double* __restrict__ beta,
                                                                const int* __restrict__ st1, int* s2, int* cnt,
                                                                int* list, int* counts, int* steps, int* left, int block_rows) {
  extern __shared__ int wave_sets[];
  int(*tables)[kSet] = reinterpret_cast<int(*)[kSet]>(wave_sets);
  const cooperative_groups::cluster_group cluster = cooperative_groups::this_cluster();
  const int tid = blockIdx.x * blockDim.x + threadIdx.x, nt = gridDim.x * blockDim.x;
  const int warp = tid >> 5, lane = tid & 31, nw = nt >> 5;
  int* table = tables[threadIdx.x >> 5];
  for (int i0 = 0; i0 < m; i0 += nt) {
    const int i = i0 + tid;
    push_rows(i < m && s2[i] == 1 && cnt[i] == 0, i, list, counts);
  }
  __threadfence();
  cluster.sync();
  int step = 0;
  for (;; ++step) {
    const int n = __ldcg(counts + step % 3);
    if (n == 0) break;
    const int* cur = list + (size_t)(step & 1) * m;
    int* next = list + (size_t)((step + 1) & 1) * m;
    int* ncount = counts + (step + 1) % 3;
    if (tid == 0) counts[(step + 2) % 3] = 0;
    // tells the candidates above j; `warps` warps share its row, this is number w
    auto notify = [&](int j, int w, int warps) {
      const int e1 = rp[j + 1];
      for (int e0 = rp[j] + 1 + w * 32; e0 < e1; e0 += warps * 32) {
        const int i = e0 + lane < e1 ? ci[e0 + lane] : -1;
        bool push = false;
        if (i > j && __ldcg(s2 + i) == 1) {
          const int q = find_offd(rp, ci, i, j);
          push = q >= 0 && strong(va[q], beta[i]) && atomicSub(cnt + i, 1) == 1;
        }
        push_rows(push, i, next, ncount);
      }
    };
    if (n <= block_rows) {
      for (int w = blockIdx.x; w < n; w += gridDim.x) {
        const int j = __ldcg(cur + w);
        const bool mine = cf_promote<kWaveThreads / 32>(j, rp, ci, va, beta, st1, s2, tables[0], lane);
        const bool p = __syncthreads_or(mine);
        if (threadIdx.x == 0) s2[j] = p ? 2 : 0;
        notify(j, threadIdx.x >> 5, kWaveThreads / 32);
      }
    } else {
      for (int w = warp; w < n; w += nw) {
        const int j = __ldcg(cur + w);
        const bool p = cf_promote<1>(j, rp, ci, va, beta, st1, s2, table, lane);
        if (lane == 0) s2[j] = p ? 2 : 0;
        notify(j, 0, 1);
      }
    }
    __threadfence();
    cluster.sync();
  }
  if (tid == 0) *steps = step;
  int n = 0;
  for (int i = tid; i < m; i += nt) n += __ldcg(s2 + i) == 1;
  n = __reduce_add_sync(0xffffffffu, n);
  if (lane == 0 && n) atomicAdd(left, n);
}

// one round of pass 2 over the candidates left (s2 == 1), whatever the
// pattern; s2 becomes 2 (promoted) or 0 once every candidate strong neighbour
// below i is decided
__global__ void __launch_bounds__(256) k_cf_pass2_round(int m, const int* __restrict__ rp,
                                                        const int* __restrict__ ci, const double* __restrict__ va,
                                                        const double* __restrict__ beta,
                                                        const int* __restrict__ st1, int* s2, int* undecided) {
  __shared__ int tables[8][kSet];
  const int i = (int)((blockIdx.x * (int64_t)blockDim.x + threadIdx.x) >> 5);
  const int lane = threadIdx.x & 31;
  if (i >= m || vload(s2 + i) != 1) return;
  const double bi = beta[i];
  bool wait = false;
  for (int e = rp[i] + 1 + lane; e < rp[i + 1]; e += 32) {
    const int j = ci[e];
    if (j < i && strong(va[e], bi) && vload(s2 + j) == 1) wait = true;
  }
  if (__any_sync(0xffffffffu, wait)) {
    if (lane == 0 && undecided != nullptr) atomicAdd(undecided, 1);
    return;
  }
  const bool p = cf_promote<1>(i, rp, ci, va, beta, st1, s2, tables[threadIdx.x >> 5], lane);
  if (lane == 0) s2[i] = p ? 2 : 0;
}

__global__ void k_cf_flags(int m, const int* __restrict__ st1, const int* __restrict__ s2,
                           int* __restrict__ is_c) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < m) is_c[i] = (st1[i] == -1 || s2[i] == 2) ? 1 : 0;
}

// core_point[c] = i for the C points in ascending order (core_at = scan of is_c)
__global__ void k_cf_core_points(int m, const int* __restrict__ is_c, const int* __restrict__ core_at,
                                 int* __restrict__ core_point) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < m && is_c[i]) core_point[core_at[i]] = i;
}

// P row c: the core point k and the non-C points of its row, ascending
__global__ void k_cf_p_len(int nc, const int* __restrict__ rp, const int* __restrict__ ci,
                           const int* __restrict__ core_point, const int* __restrict__ is_c, int* __restrict__ len) {
  const int c = blockIdx.x * blockDim.x + threadIdx.x;
  if (c >= nc) return;
  const int k = core_point[c];
  int n = 1;
  for (int e = rp[k] + 1; e < rp[k + 1]; ++e) n += !is_c[ci[e]];
  len[c] = n;
}

__global__ void k_cf_p_fill(int nc, const int* __restrict__ rp, const int* __restrict__ ci,
                            const int* __restrict__ core_point, const int* __restrict__ is_c,
                            const int* __restrict__ p_rp, int* __restrict__ p_ci, int* __restrict__ pt_len) {
  const int c = blockIdx.x * blockDim.x + threadIdx.x;
  if (c >= nc) return;
  const int k = core_point[c];
  int q = p_rp[c];
  bool placed = false;
  for (int e = rp[k] + 1; e < rp[k + 1]; ++e) {
    const int l = ci[e];
    if (is_c[l]) continue;
    if (!placed && l > k) {
      p_ci[q++] = k;
      placed = true;
    }
    p_ci[q++] = l;
    atomicAdd(pt_len + l, 1);
  }
  if (!placed) p_ci[q++] = k;
  atomicAdd(pt_len + k, 1);
}

// P^T pattern: counted, filled in any order, then each row sorted (the rows
// are short) -- the result does not depend on the order of the fill
__global__ void k_cf_pt_fill(int nc, const int* __restrict__ p_rp, const int* __restrict__ p_ci,
                             int* __restrict__ cursor, int* __restrict__ pt_ci) {
  const int c = blockIdx.x * blockDim.x + threadIdx.x;
  if (c >= nc) return;
  for (int q = p_rp[c]; q < p_rp[c + 1]; ++q) pt_ci[atomicAdd(cursor + p_ci[q], 1)] = c;
}

__global__ void k_cf_pt_sort(int m, const int* __restrict__ pt_rp, int* __restrict__ pt_ci) {
  const int l = blockIdx.x * blockDim.x + threadIdx.x;
  if (l >= m) return;
  const int b = pt_rp[l], e = pt_rp[l + 1];
  for (int q = b + 1; q < e; ++q) {
    const int v = pt_ci[q];
    int r = q - 1;
    while (r >= b && pt_ci[r] > v) {
      pt_ci[r + 1] = pt_ci[r];
      --r;
    }
    pt_ci[r + 1] = v;
  }
}

// a_lc[q] = M(l, core_point[c]) for the P^T entry q = (l, c)
__global__ void k_cf_a_lc(int m, const int* __restrict__ rp, const int* __restrict__ ci, const double* __restrict__ va,
                          const int* __restrict__ pt_rp, const int* __restrict__ pt_ci,
                          const int* __restrict__ core_point, double* __restrict__ a_lc) {
  const int l = blockIdx.x * blockDim.x + threadIdx.x;
  if (l >= m) return;
  for (int q = pt_rp[l]; q < pt_rp[l + 1]; ++q) {
    const int k = core_point[pt_ci[q]];
    double a = 0.0;
    if (rp[l] < rp[l + 1] && ci[rp[l]] == k) a = va[rp[l]];
    else {
      const int p = find_offd(rp, ci, l, k);
      if (p >= 0) a = va[p];
    }
    a_lc[q] = a;
  }
}

// P^T values of fine row i, one thread per row, in the reference's order
__global__ void k_cf_weights(int m, const int* __restrict__ rp, const int* __restrict__ ci,
                             const double* __restrict__ va, const double* __restrict__ beta,
                             const int* __restrict__ is_c, const int* __restrict__ core_at,
                             const int* __restrict__ pt_rp, const int* __restrict__ pt_ci,
                             const double* __restrict__ a_lc, double* __restrict__ pt_va) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= m) return;
  const int tb = pt_rp[i], te = pt_rp[i + 1];
  if (is_c[i]) {
    const int q = find_sorted(pt_ci, tb, te, core_at[i]);
    if (q >= 0) pt_va[q] += 1.0;
    return;
  }
  const double bi = beta[i];
  double aii = rp[i] < rp[i + 1] ? va[rp[i]] : 0.0;
  for (int e = rp[i] + 1; e < rp[i + 1]; ++e)
    if (fabs(va[e]) < bi) aii += va[e];
  for (int e = rp[i] + 1; e < rp[i + 1]; ++e) {
    const int l = ci[e];
    if (fabs(va[e]) < bi) continue;
    if (is_c[l]) {
      const int q = find_sorted(pt_ci, tb, te, core_at[l]);
      if (q >= 0) pt_va[q] += fabs(va[e] / aii);
    } else {
      double d = 0.0;
      for (int i1 = pt_rp[l]; i1 < pt_rp[l + 1]; ++i1)
        if (find_sorted(pt_ci, tb, te, pt_ci[i1]) >= 0) d += a_lc[i1];
      if (fabs(d * aii) < 1e-16) continue;
      for (int i1 = pt_rp[l]; i1 < pt_rp[l + 1]; ++i1) {
        const int q = find_sorted(pt_ci, tb, te, pt_ci[i1]);
        if (q >= 0) pt_va[q] += fabs(va[e] * a_lc[i1] / (d * aii));
      }
    }
  }
}

// The same with a warp per row, for long rows (a thread per row walks the
// P^T row of every strong F neighbour alone: 43 ms on the 31,833-row level of
// a 64^3 hierarchy, 285 entries a row; 4.2 ms this way).  The lanes take a P^T row's entries;
// the sums whose order is the reference's (aii, d, and an entry's own
// additions) are still added one term at a time: matched terms of a 32-entry
// chunk are passed round in order.  Rows of P^T longer than kPtCap accumulate
// and search in global memory.
constexpr int kPtCap = 256;
// Mean row length above which a warp takes a row.  The whole splitting with a
// warp and with a thread (ms): 7.0 entries 8.99 and 8.66 (361,201 rows), 14.5 2.31
// and 2.19 (48^3), 14.6 4.03 and 3.69 (64^3); 21 1.86 and 1.97 (2D P2 220^2), 24
// 0.98 and 1.29 (121^2), 41 1.39 and 2.07, 131 2.7 and 10.2 (3D P2 20^3).
constexpr double kWarpWeightsLen = 18.0;

// acc + the values v of the lanes in `which`, added in lane order
__device__ __forceinline__ double add_in_order(double acc, double v, unsigned which) {
  while (which) {
    const int src = __ffs(which) - 1;
    which &= which - 1;
    acc += __shfl_sync(0xffffffffu, v, src);
  }
  return acc;
}

__global__ void __launch_bounds__(128) k_cf_weights_warp(int m, const int* __restrict__ rp,
                                                         const int* __restrict__ ci, const double* __restrict__ va,
                                                         const double* __restrict__ beta,
                                                         const int* __restrict__ is_c,
                                                         const int* __restrict__ core_at,
                                                         const int* __restrict__ pt_rp,
                                                         const int* __restrict__ pt_ci,
                                                         const double* __restrict__ a_lc, double* pt_va) {
  __shared__ int scol[4][kPtCap];
  __shared__ double sacc[4][kPtCap];
  const int i = (int)((blockIdx.x * (int64_t)blockDim.x + threadIdx.x) >> 5);
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  if (i >= m) return;
  const int tb = pt_rp[i], tn = pt_rp[i + 1] - tb;
  if (is_c[i]) {
    if (lane == 0) {
      const int q = find_sorted(pt_ci, tb, tb + tn, core_at[i]);
      if (q >= 0) pt_va[q] += 1.0;
    }
    return;
  }
  const bool in_smem = tn <= kPtCap;
  const int* tcol = in_smem ? scol[w] : pt_ci + tb;
  double* acc = in_smem ? sacc[w] : pt_va + tb;
  if (in_smem)
    for (int q = lane; q < tn; q += 32) {
      scol[w][q] = pt_ci[tb + q];
      sacc[w][q] = pt_va[tb + q];
    }
  __syncwarp();
  const double bi = beta[i];
  const int b = rp[i] + 1, e1 = rp[i + 1];
  double aii = rp[i] < e1 ? va[rp[i]] : 0.0;
  for (int e0 = b; e0 < e1; e0 += 32) {
    const int e = e0 + lane;
    const double v = e < e1 ? va[e] : 0.0;
    aii = add_in_order(aii, v, __ballot_sync(0xffffffffu, e < e1 && fabs(v) < bi));
  }
  for (int e0 = b; e0 < e1; e0 += 32) {
    const int e = e0 + lane;
    const double v = e < e1 ? va[e] : 0.0;
    const int l = e < e1 ? ci[e] : 0;
    const bool st = e < e1 && !(fabs(v) < bi);
    const int core = st && is_c[l] ? core_at[l] : -1;
    const int lb = st && core < 0 ? pt_rp[l] : 0, le = st && core < 0 ? pt_rp[l + 1] : 0;
    for (unsigned todo = __ballot_sync(0xffffffffu, st); todo != 0; todo &= todo - 1) {
      const int src = __ffs(todo) - 1;
      const double ve = __shfl_sync(0xffffffffu, v, src);
      const int c = __shfl_sync(0xffffffffu, core, src);
      const int pb = __shfl_sync(0xffffffffu, lb, src), pe = __shfl_sync(0xffffffffu, le, src);
      if (c >= 0) {
        if (lane == 0) {
          const int q = find_sorted(tcol, 0, tn, c);
          if (q >= 0) acc[q] += fabs(ve / aii);
        }
        __syncwarp();
        continue;
      }
      double d = 0.0, a0 = 0.0;
      int q0 = -1;  // the first chunk's match is kept for the second pass
      for (int p0 = pb; p0 < pe; p0 += 32) {
        const bool on = p0 + lane < pe;
        const double a = on ? a_lc[p0 + lane] : 0.0;
        const int q = on ? find_sorted(tcol, 0, tn, pt_ci[p0 + lane]) : -1;
        if (p0 == pb) {
          a0 = a;
          q0 = q;
        }
        d = add_in_order(d, a, __ballot_sync(0xffffffffu, q >= 0));
      }
      if (fabs(d * aii) < 1e-16) continue;
      for (int p0 = pb; p0 < pe; p0 += 32) {
        double a = a0;
        int q = q0;
        if (p0 != pb) {
          const bool on = p0 + lane < pe;
          a = on ? a_lc[p0 + lane] : 0.0;
          q = on ? find_sorted(tcol, 0, tn, pt_ci[p0 + lane]) : -1;
        }
        if (q >= 0) acc[q] += fabs(ve * a / (d * aii));
      }
      __syncwarp();
    }
  }
  if (in_smem)
    for (int q = lane; q < tn; q += 32) pt_va[tb + q] = sacc[w][q];
}

// P(c, i) received the same additions as P^T(i, c)
__global__ void k_cf_p_vals(int nc, const int* __restrict__ p_rp, const int* __restrict__ p_ci,
                            const int* __restrict__ pt_rp, const int* __restrict__ pt_ci,
                            const double* __restrict__ pt_va, double* __restrict__ p_va) {
  const int c = blockIdx.x * blockDim.x + threadIdx.x;
  if (c >= nc) return;
  for (int q = p_rp[c]; q < p_rp[c + 1]; ++q) {
    const int i = p_ci[q];
    const int t = find_sorted(pt_ci, pt_rp[i], pt_rp[i + 1], c);
    p_va[q] = t >= 0 ? pt_va[t] : 0.0;
  }
}

// launches `launch(counter)` in batches, the last of each batch counting the
// rows left, until none are; returns the number of rounds run
template <class F>
int run_rounds(const afp_context* ctx, int m, DevBuf<int>& counter, F launch, const char* what) {
  int rounds = 0;
  for (;;) {
    counter.zero();
    for (int r = 0; r < kRoundsPerCheck; ++r) launch(r + 1 == kRoundsPerCheck ? counter.get() : nullptr);
    rounds += kRoundsPerCheck;
    check_launch(ctx, what);
    int left = 0;
    copy(ctx, &left, counter.get(), sizeof(int));
    sync(ctx);
    if (left == 0) return rounds;
    // the lowest undecided row decides in every round
    if (rounds > m + kRoundsPerCheck) fail(AFP_ERR_CUDA, std::string(what) + ": rounds did not settle");
  }
}

// Pass 2: a step of at most so many rows gives each a whole block.  The whole
// splitting with 0, 96 and 512 (ms), by mean row length: 15 entries 2.18, 2.66
// and 4.37 (48^3), 28 2.17, 2.29 and 2.80 (3D P2 20^3), 56 2.83, 2.83 and 2.94;
// 68 1.77, 1.64 and 1.80, 73 3.56, 3.40 and 3.83 (40^3), 76 8.6, 8.9 and 9.2 (64^3),
// 131 2.67, 2.69 and 3.01; 273 14.0, 10.7 and 10.9 (48^3), 285 20.2, 17.5 and 17.9.
int wave_block_rows(double len) { return len > 64.0 ? 96 : 0; }

// Launches a wave kernel as one cluster, of 16 blocks where the device can
// place one that large, else of the portable 8.
template <class... K, class... Args>
void launch_wave(const afp_context* ctx, const char* what, size_t smem, void (*kernel)(K...), Args... args) {
  cudaLaunchConfig_t cfg = {};
  cfg.dynamicSmemBytes = smem;
  AFP_CUDA(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
  cfg.blockDim = kWaveThreads;
  cfg.stream = ctx->stream;
  cudaLaunchAttribute at[1];
  at[0].id = cudaLaunchAttributeClusterDimension;
  cfg.attrs = at;
  cfg.numAttrs = 1;
  AFP_CUDA(cudaFuncSetAttribute(kernel, cudaFuncAttributeNonPortableClusterSizeAllowed, 1));
  for (unsigned size : {16u, 8u}) {
    at[0].val.clusterDim = {size, 1, 1};
    cfg.gridDim = size;
    int fit = 0;
    if (size > 8 && (cudaOccupancyMaxActiveClusters(&fit, kernel, &cfg) != cudaSuccess || fit < 1)) {
      cudaGetLastError();
      continue;
    }
    AFP_CUDA(cudaLaunchKernelEx(&cfg, kernel, args...));
    break;
  }
  check_launch(ctx, what);
}

}  // namespace

int gpu_project(const afp_context* ctx, int64_t m64, const int* rp, const int* ci, const double* va, double alpha,
                GpuProjection& out) {
  const int m = (int)m64;
  const cudaStream_t s = ctx->stream;
  int nnz = 0;
  copy(ctx, &nnz, rp + m, sizeof(int));
  sync(ctx);
  const unsigned warp_grid = grid_for((int64_t)m * 32, 256);
  DevBuf<double> beta(ctx, m);
  DevBuf<int> st1(ctx, m), s2(ctx, m), cnt(ctx, m), list(ctx, 2 * (size_t)m);
  DevBuf<int> waves(ctx, 9);  // list counts of both passes, steps of both, candidates left
  k_cf_beta<<<warp_grid, 256, 0, s>>>(m, rp, va, alpha, beta.get());
  st1.zero();
  cnt.zero();
  waves.zero();
  k_cf_count_in<<<warp_grid, 256, 0, s>>>(m, rp, ci, va, beta.get(), cnt.get());
  const double len = (double)nnz / (double)m;  // mean row
  launch_wave(ctx, "C/F pass 1", 0, k_cf_pass1_wave, m, rp, ci, va, (const double*)beta.get(), st1.get(), cnt.get(),
              list.get(), waves.get(), waves.get() + 6);
  k_cf_pass2_candidates<<<warp_grid, 256, 0, s>>>(m, rp, ci, va, beta.get(), st1.get(), s2.get());
  k_cf_pass2_count<<<warp_grid, 256, 0, s>>>(m, rp, ci, va, beta.get(), s2.get(), cnt.get());
  launch_wave(ctx, "C/F pass 2", kWaveThreads / 32 * kSet * sizeof(int), k_cf_pass2_wave, m, rp, ci, va, (const double*)beta.get(), (const int*)st1.get(),
              s2.get(), cnt.get(), list.get(), waves.get() + 3, waves.get() + 7, waves.get() + 8, wave_block_rows(len));
  int hw[3] = {0, 0, 0};
  copy(ctx, hw, waves.get() + 6, sizeof(hw));
  sync(ctx);
  out.rounds1 = hw[0];
  out.rounds2 = hw[1];
  if (hw[2] != 0) {
    DevBuf<int> counter(ctx, 1);
    out.rounds2 += run_rounds(
        ctx, m, counter,
        [&](int* left) {
          k_cf_pass2_round<<<warp_grid, 256, 0, s>>>(m, rp, ci, va, beta.get(), st1.get(), s2.get(), left);
        },
        "C/F pass 2 (nonsymmetric pattern)");
  }
  DevBuf<int> is_c(ctx, m), core_at(ctx, m + 1);
  k_cf_flags<<<grid_for(m, 256), 256, 0, s>>>(m, st1.get(), s2.get(), is_c.get());
  const int nc = (int)exclusive_scan(ctx, is_c.get(), core_at.get(), m);
  out.cf.alloc(ctx, m);
  AFP_CUDA(cudaMemcpyAsync(out.cf.get(), is_c.get(), sizeof(int) * m, cudaMemcpyDeviceToDevice, s));
  DevBuf<int> core_point(ctx, nc > 0 ? nc : 1);
  k_cf_core_points<<<grid_for(m, 256), 256, 0, s>>>(m, is_c.get(), core_at.get(), core_point.get());

  DevCSR& P = out.P;
  DevCSR& T = out.Pt;
  P.m = nc;
  P.n = m;
  T.m = m;
  T.n = nc;
  DevBuf<int> plen(ctx, nc > 0 ? nc : 1);
  k_cf_p_len<<<grid_for(nc, 256), 256, 0, s>>>(nc, rp, ci, core_point.get(), is_c.get(), plen.get());
  P.rp.alloc(ctx, nc + 1);
  P.nnz = exclusive_scan(ctx, plen.get(), P.rp.get(), nc);
  P.ci.alloc(ctx, P.nnz);
  DevBuf<int> tlen(ctx, m);
  tlen.zero();
  k_cf_p_fill<<<grid_for(nc, 256), 256, 0, s>>>(nc, rp, ci, core_point.get(), is_c.get(), P.rp.get(), P.ci.get(),
                                                tlen.get());
  T.rp.alloc(ctx, m + 1);
  T.nnz = exclusive_scan(ctx, tlen.get(), T.rp.get(), m);
  T.ci.alloc(ctx, T.nnz);
  DevBuf<int> cursor(ctx, m);
  AFP_CUDA(cudaMemcpyAsync(cursor.get(), T.rp.get(), sizeof(int) * m, cudaMemcpyDeviceToDevice, s));
  k_cf_pt_fill<<<grid_for(nc, 256), 256, 0, s>>>(nc, P.rp.get(), P.ci.get(), cursor.get(), T.ci.get());
  k_cf_pt_sort<<<grid_for(m, 128), 128, 0, s>>>(m, T.rp.get(), T.ci.get());
  DevBuf<double> a_lc(ctx, T.nnz > 0 ? T.nnz : 1);
  k_cf_a_lc<<<grid_for(m, 128), 128, 0, s>>>(m, rp, ci, va, T.rp.get(), T.ci.get(), core_point.get(), a_lc.get());
  T.va.alloc(ctx, T.nnz);
  T.va.zero();
  if ((double)nnz > kWarpWeightsLen * (double)m)
    k_cf_weights_warp<<<grid_for((int64_t)m * 32, 128), 128, 0, s>>>(m, rp, ci, va, beta.get(), is_c.get(),
                                                                     core_at.get(), T.rp.get(), T.ci.get(),
                                                                     a_lc.get(), T.va.get());
  else
    k_cf_weights<<<grid_for(m, 128), 128, 0, s>>>(m, rp, ci, va, beta.get(), is_c.get(), core_at.get(), T.rp.get(),
                                                  T.ci.get(), a_lc.get(), T.va.get());
  P.va.alloc(ctx, P.nnz);
  k_cf_p_vals<<<grid_for(nc, 128), 128, 0, s>>>(nc, P.rp.get(), P.ci.get(), T.rp.get(), T.ci.get(), T.va.get(),
                                                P.va.get());
  check_launch(ctx, "GPU C/F splitting");
  return nc;
}

}  // namespace afp
