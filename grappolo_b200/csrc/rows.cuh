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

// ---------------------------------------------------------------------------
// Rows of at most 32 entries: G lanes per row, 32 / G rows per warp and item,
// everything in registers.  A warp runs its items of a bin one after another
// (item k, k + stride, ...), and an item is a chain of four dependent loads
// (member, row bounds, entries, communities), so the loads run ahead: while an
// item is decided, the next one's entries, the one after's row bounds and the
// third's members are on their way.
struct SmallRow {
  int32_t v;       // -1: no row
  int deg;
  int64_t rb;
};

__device__ __forceinline__ void small_bounds(const SweepArgs &a, SmallRow &r) {
  r.rb = 0;
  r.deg = 0;
  if (r.v >= 0) {
    r.rb = a.ptr[r.v];
    r.deg = (int)(a.ptr[r.v + 1] - r.rb);
  }
}

// Decides the 32 / G rows of an item: row r, entry (t, w) of this lane, own =
// community of r.v (-1 for an empty row).
template <int G>
__device__ __forceinline__ void small_decide(const SweepArgs &a, int pos, const SmallRow &r,
                                             int32_t t, double w, int32_t own) {
  const int lane = threadIdx.x & 31, gl = lane & (G - 1);
  const bool skip = r.deg > 0 && skipped(a, r.v);
  const bool has = !skip && gl < r.deg;
  const int32_t c = has ? a.C[t] : -1;
  // the community's and the vertex's totals, while the entries are compared
  const double degree = r.deg > 0 ? a.vDeg[r.v] : 0.0;
  const double cdeg_own = r.deg > 0 ? a.cDeg[own] : 0.0;
  const double cdeg = (has && c != own) ? a.cDeg[c] : 0.0;
  const int32_t own_size = (r.deg > 0 && gl == 0) ? a.cSize[own] : 0;
  double sum, own_w = 0.0, self_w = 0.0;  // Counter[c], Counter[own], self-loops
  bool cand;                              // this lane offers community c
  if (G <= 8) {
    // every lane sees all entries of its row in order (3 shuffles each; a match
    // over the warp takes up to 379 cycles); the top bit marks self-loops.  In
    // order, so that every lane of the row has the same sums on any weights:
    // from each lane's own entry on, candidates of equal gain differed in the
    // last bit.
    const int32_t mark = (has && t == r.v) ? (c | INT32_MIN) : (has ? c : 0x7fffffff);
    sum = 0.0;
#pragma unroll
    for (int q = 0; q < G; ++q) {
      const int src = (lane & ~(G - 1)) | q;
      const int32_t oc = __shfl_sync(FULL, mark, src);
      const double ow = __shfl_sync(FULL, w, src);
      const int32_t id = oc & 0x7fffffff;
      if (id == c) sum = __dadd_rn(sum, ow);
      if (id == own) own_w = __dadd_rn(own_w, ow);
      if (oc < 0) self_w = __dadd_rn(self_w, ow);
    }
    cand = has && c != own;
  } else {
    const unsigned gmask = (G == 32) ? FULL : (((1u << (G & 31)) - 1u) << (lane & ~(G - 1)));
    const unsigned m = __match_any_sync(FULL, c) & gmask;
    sum = group_sum(has ? w : 0.0, has ? m : 0u);
    const bool leader = has && lane == __ffs(m) - 1;
    const unsigned om = __ballot_sync(FULL, leader && c == own) & gmask;
    own_w = __shfl_sync(FULL, sum, om ? __ffs(om) - 1 : lane);
    if (!om) own_w = 0.0;
    const unsigned sm = __ballot_sync(FULL, has && t == r.v) & gmask;
    if (__any_sync(FULL, sm != 0)) {
      self_w = group_sum((has && t == r.v) ? w : 0.0, (has && t == r.v) ? sm : 0u);
      self_w = __shfl_sync(FULL, self_w, sm ? __ffs(sm) - 1 : lane);
      if (!sm) self_w = 0.0;
    }
    cand = leader && c != own;
  }
  double g = 0.0;
  int32_t bc = INT32_MAX;
  if (cand) {
    const double eix = __dsub_rn(own_w, self_w);
    const double ax = __dsub_rn(cdeg_own, degree);
    const double gain = louvain_gain(sum, eix, degree, cdeg, ax, cst_of(a, r.v));
    if (gain > 0.0) { g = gain; bc = c; }
  }
#pragma unroll
  for (int off = G / 2; off >= 1; off >>= 1) {
    const double og = __shfl_xor_sync(FULL, g, off);
    const int32_t oc = __shfl_xor_sync(FULL, bc, off);
    if (better(og, oc, g, bc)) { g = og; bc = oc; }
  }
  if (r.v >= 0 && gl == 0) {
    if (skip) {
      emit_stay(a, pos, r.v, own);
    } else {
      const int32_t tgt = (r.deg == 0) ? -1 : finish_choice(a, own, own_size, g, bc);
      emit_decision(a, pos, r.v, own, tgt, degree, own_w, g);
    }
  }
}

// This warp's items k, k + stride, ... of the rows at member positions
// [begin, end); returns the first item number past the bin's, for the next bin.
template <int G>
__device__ __forceinline__ int small_rows(const SweepArgs &a, int begin, int end, int k,
                                          int stride) {
  constexpr int VPW = 32 / G;
  const int n = (end - begin + VPW - 1) / VPW;
  if (k < n) {
    const int grp = (threadIdx.x & 31) / G, gl = threadIdx.x & (G - 1);
    const int hop = VPW * stride;
    int pos = begin + VPW * k + grp;
    SmallRow cur, nxt;
    cur.v = (pos < end) ? a.members[pos] : -1;
    nxt.v = (pos + hop < end) ? a.members[pos + hop] : -1;
    int32_t v3 = (pos + 2 * hop < end) ? a.members[pos + 2 * hop] : -1;
    small_bounds(a, cur);
    small_bounds(a, nxt);
    int32_t t = (gl < cur.deg) ? __ldcs(&a.tail[cur.rb + gl]) : -1;
    double w = (gl < cur.deg) ? __ldcs(&a.w[cur.rb + gl]) : 0.0;
    int32_t own = cur.deg > 0 ? a.C[cur.v] : -1;
    for (;;) {
      // ahead: the next item's entries, the one after's bounds, a third's members
      const int32_t t2 = (gl < nxt.deg) ? __ldcs(&a.tail[nxt.rb + gl]) : -1;
      const double w2 = (gl < nxt.deg) ? __ldcs(&a.w[nxt.rb + gl]) : 0.0;
      const int32_t own2 = nxt.deg > 0 ? a.C[nxt.v] : -1;
      SmallRow after;
      after.v = v3;
      small_bounds(a, after);
      v3 = (pos + 3 * hop < end) ? a.members[pos + 3 * hop] : -1;
      small_decide<G>(a, pos, cur, t, w, own);
      k += stride;
      if (k >= n) break;
      pos += hop;
      cur = nxt;
      nxt = after;
      t = t2;
      w = w2;
      own = own2;
    }
  }
  return k - n;
}

}  // namespace glv
