// Long rows of the persistent sweep: one row (or one hub chunk) on T threads,
// with the community table in shared memory.  Parallel accumulation only: the
// modes that come here accept a row's additions in any order (integral
// weights, where every order is exact, and fast mode).
//
// What bounds it: not bytes but the chain of dependent steps of one row, and
// within it the instructions of a round of 32 entries.  Measured on B200
// (cycles): __match_any_sync 379 with 32 distinct keys and about 12 per
// distinct key, a shared f64 add 103 (and as much again for every further lane
// on the same address), a shared CAS 52, an L2 gather 450.  So:
//
// * the row's own community and its self-loops are summed in registers;
// * a round groups equal communities with __match_any_sync only while the row
//   repeats communities (folding a group by pointer jumping, log2 of its size);
//   where a round finds mostly different ones the next rounds insert every
//   entry by itself;
// * the table is empty between rows: a thread remembers the slots it filled
//   first (`fill`, one 16-bit entry per entry of the row), scans only those for
//   the best gain, and empties them.  Clearing and scanning whole tables (twice
//   the row's length and up) went with that.
#pragma once

#include "sweep.cuh"

namespace glv {

constexpr uint16_t kNoSlot = 0xffffu;

// Team of T threads (T/32 warps; T == blockDim.x or a named-barrier slice of
// the block, or one warp).
template <int T>
__device__ __forceinline__ void team_sync(int team) {
  if (T == 32) __syncwarp();
  else if (T == 512) __syncthreads();
  else asm volatile("bar.sync %0, %1;" ::"r"(team + 1), "r"(T) : "memory");
}

__device__ __forceinline__ void prefetch_l1(const void *p) {
  asm volatile("prefetch.global.L1 [%0];" ::"l"(p));
}

// Sums x over the lanes of each group (m: the lanes with this lane's key);
// the group's lowest lane holds the group's sum.
__device__ __forceinline__ double group_sum(double x, unsigned m) {
  const int lane = threadIdx.x & 31;
  const unsigned above = m & (0xfffffffeu << lane);
  int nx = above ? __ffs(above) - 1 : 32;
  while (__any_sync(FULL, nx < 32)) {
    const int src = nx < 32 ? nx : lane;
    const double y = __shfl_sync(FULL, x, src);
    const int nn = __shfl_sync(FULL, nx, src);
    if (nx < 32) {
      x = __dadd_rn(x, y);
      nx = nn;
    }
  }
  return x;
}

__device__ __forceinline__ double warp_sum(double x) {
#pragma unroll
  for (int off = 16; off >= 1; off >>= 1) x = __dadd_rn(x, __shfl_xor_sync(FULL, x, off));
  return x;
}

// Adds the `len` entries from rb on (of v's row) to the table, T at a time.
// Entries of the row's own community go to own_w, self-loops to self_w (both
// per lane).  fill[r * T] is this thread's slot of round r (kNoSlot: none
// filled).  Returns the rounds of this warp.
template <int T>
__device__ __forceinline__ int row_accumulate(const SweepArgs &a, int32_t v, int32_t own,
                                              int64_t rb, int len, int32_t *keys, double *vals,
                                              uint32_t mask, uint16_t *fill, double &self_w,
                                              double &own_w) {
  const int tt = threadIdx.x % T, lane = threadIdx.x & 31;
  const int32_t *const tail = a.tail + rb;
  const double *const w = a.w + rb;
  // Software pipeline, two rounds deep: while this round is folded, the next
  // round's communities are gathered and the round after's entries load.
  // Neighbours' communities do not change during the sweep of one step.  The
  // entries are read once per sweep: streaming loads keep them from pushing the
  // gathered per-vertex arrays out of L2.
  int32_t t_cur = (tt < len) ? __ldcs(tail + tt) : -1;
  double w_cur = (tt < len) ? __ldcs(w + tt) : 0.0;
  int32_t t_next = (tt + T < len) ? __ldcs(tail + tt + T) : -1;
  double w_next = (tt + T < len) ? __ldcs(w + tt + T) : 0.0;
  int32_t c_cur = (tt < len) ? a.C[t_cur] : -1;
  bool group = true;  // the row repeats communities: group a round's equal ones
  int r = 0;
  for (int j = tt; j - lane < len; j += T, ++r) {
    const int32_t t = t_cur, c = c_cur;
    const double wt = w_cur;
    c_cur = (j + T < len) ? a.C[t_next] : -1;
    t_cur = t_next;
    w_cur = w_next;
    t_next = (j + 2 * T < len) ? __ldcs(tail + j + 2 * T) : -1;
    w_next = (j + 2 * T < len) ? __ldcs(w + j + 2 * T) : 0.0;
    if (t == v) self_w = __dadd_rn(self_w, wt);
    if (c == own) own_w = __dadd_rn(own_w, wt);
    bool put = j < len && c != own;
    const int n = __popc(__ballot_sync(FULL, put));
    double x = wt;
    const bool grouped = group;
    if (group) {
      const unsigned m = __match_any_sync(FULL, put ? c : -1);
      x = group_sum(wt, put ? m : 0u);
      put = put && lane == __ffs(m) - 1;
      group = 4 * __popc(__ballot_sync(FULL, put)) <= 3 * n;
    }
    uint32_t slot = kNoSlot;
    if (put) {
      uint32_t s = hash_slot(c, mask);
      while (true) {
        const int32_t k = atomicCAS(&keys[s], -1, c);
        if (k == -1) slot = s;
        if (k == -1 || k == c) break;
        s = (s + 1) & mask;
      }
      atomicAdd(&vals[s], x);
    }
    fill[r * T] = (uint16_t)slot;
    if (!grouped) group = 2 * __popc(__ballot_sync(FULL, slot != kNoSlot)) < n;
  }
  return r;
}

// Best (gain, id) over the slots this thread filled, which are emptied.  Four
// slots per thread are in flight: their cDeg gathers overlap.
template <int T>
__device__ __forceinline__ void row_scan(const SweepArgs &a, int32_t *keys, double *vals,
                                         const uint16_t *fill, int rounds, double eix, double ax,
                                         double degree, double cst, double &g, int32_t &bc) {
  for (int r0 = 0; r0 < rounds; r0 += 4) {
    int32_t k[4];
    double val[4], cd[4];
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      const uint16_t s = (r0 + q < rounds) ? fill[(r0 + q) * T] : kNoSlot;
      k[q] = -1;
      if (s != kNoSlot) {
        k[q] = keys[s];
        val[q] = vals[s];
        keys[s] = -1;
        vals[s] = 0.0;
      }
    }
#pragma unroll
    for (int q = 0; q < 4; ++q) cd[q] = (k[q] >= 0) ? a.cDeg[k[q]] : 0.0;
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      if (k[q] < 0) continue;
      const double gain = louvain_gain(val[q], eix, degree, cd[q], ax, cst);
      if (gain > 0.0 && better(gain, k[q], g, bc)) { g = gain; bc = k[q]; }
    }
  }
}

// One row on T threads (all of the team call).  keys/vals: the team's table,
// empty on entry and on exit; fill: room for the row's entries rounded up to T;
// s_self, s_own, s_g, s_c: one entry per warp of the team.  The caller
// synchronises the team between rows.
template <int T>
__device__ __forceinline__ void row_vertex(const SweepArgs &a, int64_t pos, int32_t *keys,
                                           double *vals, uint16_t *fill, int team, double *s_self,
                                           double *s_own, double *s_g, int32_t *s_c) {
  constexpr int NW = T / 32;
  const int tt = threadIdx.x % T, lane = tt & 31, tw = tt >> 5;
  const int32_t v = a.members[pos];
  if (skipped(a, v)) {  // team-uniform
    if (tt == 0) emit_stay(a, pos, v, a.C[v]);
    return;
  }
  const int64_t rb = a.ptr[v];
  const int len = (int)(a.ptr[v + 1] - rb);
  const int32_t own = a.C[v];
  // the vertex's and its community's totals come into L1 while the row
  // accumulates (no registers held for them)
  prefetch_l1(&a.vDeg[v]);
  prefetch_l1(&a.cDeg[own]);
  if (tt == 0) prefetch_l1(&a.cSize[own]);
  double self_w = 0.0, own_w = 0.0;
  const int rounds = row_accumulate<T>(a, v, own, rb, len, keys, vals, table_cap(len) - 1,
                                       fill + tt, self_w, own_w);
  const double degree = a.vDeg[v];
  const double cdeg_own = a.cDeg[own];
  if (__any_sync(FULL, self_w != 0.0)) self_w = warp_sum(self_w);
  if (__any_sync(FULL, own_w != 0.0)) own_w = warp_sum(own_w);
  if (NW > 1) {
    if (lane == 0) { s_self[tw] = self_w; s_own[tw] = own_w; }
    team_sync<T>(team);
    self_w = own_w = 0.0;
    for (int k = 0; k < NW; ++k) {
      self_w = __dadd_rn(self_w, s_self[k]);
      own_w = __dadd_rn(own_w, s_own[k]);
    }
  } else {
    __syncwarp();
  }
  const double eix = __dsub_rn(own_w, self_w);
  const double ax = __dsub_rn(cdeg_own, degree);
  double g = 0.0;
  int32_t bc = INT32_MAX;
  row_scan<T>(a, keys, vals, fill + tt, rounds, eix, ax, degree, cst_of(a, v), g, bc);
  warp_argmax(g, bc);
  if (NW > 1) {
    if (lane == 0) { s_g[tw] = g; s_c[tw] = bc; }
    team_sync<T>(team);
  }
  if (tt == 0) {
    for (int k = 1; k < NW; ++k)
      if (better(s_g[k], s_c[k], g, bc)) { g = s_g[k]; bc = s_c[k]; }
    emit_decision(a, pos, v, own, finish_choice(a, own, a.cSize[own], g, bc), degree, own_w, g);
  }
  if (NW == 1) __syncwarp();
}

}  // namespace glv
