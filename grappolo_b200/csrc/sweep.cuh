// Local-moving sweep kernels (one launch per colour class and degree bin).
//
// Per vertex v with community own = C[v] and weighted degree k = vDeg[v] the
// kernels compute what Grappolo's buildLocalMapCounter + max compute
// (Utility/utilityClusteringFunctions.cpp:172-194, 226-259):
//   Counter[c] = sum of w(v,t) over neighbours t with C[t] = c, in CSR order,
//   selfLoop   = sum of w(v,v) entries,
//   eix = Counter[own] - selfLoop,  ax = cDeg[own] - k,
//   gain(c) = 2*(Counter[c] - eix) - 2*k*(cDeg[c] - ax)*constant  (c != own),
// and move to the strictly positive best gain (ties: lower id), with the
// reference's swap protection for two singletons.  Every per-community sum is
// folded in CSR order (leader lanes add their group's weights lane by lane,
// chunks in row order), so the sums are bit-identical to the reference's.
#pragma once

#include <cooperative_groups.h>

#include "glv_common.cuh"

namespace glv {

struct SweepArgs {
  const int64_t *ptr;
  const int32_t *tail;
  const double *w;
  int32_t *C;            // communities read; colour phases also write decisions here
  int32_t *target;       // Jacobi phases: decisions (nullptr in colour phases)
  double *own_w;         // Jacobi phases: Counter[own] per vertex (cluster weight internal)
  const double *vDeg;
  const double *cDeg;
  const int32_t *cSize;
  double constant;
  const int32_t *members;  // vertices ordered by (colour, bin, id)
  int32_t *move_old;       // per member slot: old community if it moved, else -1
  int32_t *move_new;       // per member slot: decision
  double *dDeg;            // community-degree deltas (atomic accumulation)
  int32_t *dSize;
  int atomic_deltas;       // 1: accumulate deltas here; 0: ordered fold after the class
  int32_t *hub_keys;       // BIN_HUB global tables
  double *hub_vals;
  const int64_t *hub_off;  // per member slot: table offset
  // learned gating (colour phases of the persistent path; nullptr = off)
  const uint8_t *skip;     // per vertex: 1 = not evaluated this sweep (stays)
  double *rec_own;         // per vertex: Counter[own] of its last evaluation
  float *rec_gain;         // per vertex: best positive gain of its last evaluation
  int32_t *last_move;      // per vertex: iteration of its last move
  int32_t iter;            // this sweep's iteration number within the phase
  // batches of graphs (one level holds many graphs; nullptr = one graph)
  const int32_t *gid;      // per vertex: its graph
  const double *gcst;      // per graph: 1 / (2m) of that graph
  // per block: sum over the moves of 2 (e_iy - e_ix), the change each move
  // makes to the modularity's internal-weight term (nullptr = not tracked)
  double *exx_delta;
  // colour phases whose classes include batches of the core: decisions reach
  // C only after their step (the apply stage), so every member of a step
  // decides against the communities its step started from
  int defer_c;
};

__device__ __forceinline__ bool skipped(const SweepArgs &a, int32_t v) {
  return a.skip && a.skip[v];
}

// The modularity constant that vertex v's gains use: its own graph's.
__device__ __forceinline__ double cst_of(const SweepArgs &a, int32_t v) {
  return a.gid ? a.gcst[a.gid[v]] : a.constant;
}

// Set when a vertex that this block decided moves (read and cleared by the
// persistent kernel at the end of a step).
__device__ __forceinline__ int &block_moved() {
  __shared__ int moved;
  return moved;
}

// A vertex the gate left out keeps its community and moves nothing.
__device__ __forceinline__ void emit_stay(const SweepArgs &a, int64_t pos, int32_t v,
                                          int32_t own) {
  if (a.target) a.target[v] = own;
  a.move_old[pos] = -1;
  a.move_new[pos] = own;
}

// Writes the decision of vertex v (member slot pos) and its delta records.
__device__ __forceinline__ void emit_decision(const SweepArgs &a, int64_t pos, int32_t v,
                                              int32_t own, int32_t target, double degree,
                                              double own_w, double best_g = 0.0) {
  if (a.rec_own) {
    a.rec_own[v] = own_w;
    a.rec_gain[v] = (float)best_g;
  }
  if (a.target) {
    a.target[v] = target;
    if (a.own_w) a.own_w[v] = own_w;
  } else if (!a.defer_c) {
    a.C[v] = target;
  }
  bool moved = (target != own) && (target != -1);
  a.move_old[pos] = moved ? own : -1;
  a.move_new[pos] = target;
  if (moved && a.exx_delta) {
    // the move's gain is t1 - t2 with t1 = 2 (e_iy - e_ix) (louvain_gain):
    // recover t1 from it and t2, computed as the gain computed it
    const double ax = __dsub_rn(a.cDeg[own], degree);
    const double t2 = __dmul_rn(__dmul_rn(__dmul_rn(2.0, degree), __dsub_rn(a.cDeg[target], ax)),
                                cst_of(a, v));
    atomicAdd(&a.exx_delta[blockIdx.x], __dadd_rn(best_g, t2));
  }
  if (moved && a.last_move) a.last_move[v] = a.iter;
  if (moved && a.atomic_deltas) {
    block_moved() = 1;
    atomicAdd(&a.dDeg[target], degree);
    atomicAdd(&a.dDeg[own], -degree);
    atomicAdd(&a.dSize[target], 1);
    atomicAdd(&a.dSize[own], -1);
  }
}

// Final choice: best strictly positive gain or stay; swap protection
// (utilityClusteringFunctions.cpp:254-256).
__device__ __forceinline__ int32_t finish_choice(const SweepArgs &a, int32_t own, double best_g,
                                                 int32_t best_c) {
  int32_t t = (best_g > 0.0) ? best_c : own;
  if (t != own && a.cSize[t] == 1 && a.cSize[own] == 1 && t > own) t = own;
  return t;
}

// The same with cSize[own] loaded by the caller ahead of time: only a move
// out of a singleton reads the target's size.
__device__ __forceinline__ int32_t finish_choice(const SweepArgs &a, int32_t own, int32_t own_size,
                                                 double best_g, int32_t best_c) {
  int32_t t = (best_g > 0.0) ? best_c : own;
  if (t != own && own_size == 1 && t > own && a.cSize[t] == 1) t = own;
  return t;
}

// ---------------------------------------------------------------------------
// Rows of at most G entries: G lanes per vertex, one entry per lane, no table.
// One warp handles the 32/G member slots starting at `base` (all lanes call).
template <int G>
__device__ __forceinline__ void small_item(const SweepArgs &a, int64_t base, int64_t end) {
  const int lane = threadIdx.x & 31;
  const int grp = lane / G;
  const int gl = lane & (G - 1);
  const unsigned gmask = (G == 32) ? FULL : (((1u << G) - 1u) << (grp * G));
  const int64_t pos = base + grp;
  const bool valid = pos < end;
  const int32_t v = valid ? a.members[pos] : 0;
  const int64_t rb = valid ? a.ptr[v] : 0;
  const int deg = valid ? (int)(a.ptr[v + 1] - rb) : 0;
  const int32_t own = (valid && deg > 0) ? a.C[v] : -1;
  const bool skip = valid && deg > 0 && skipped(a, v);
  const bool has = !skip && gl < deg;
  const int32_t t = has ? __ldcs(&a.tail[rb + gl]) : -1;
  const double wt = has ? __ldcs(&a.w[rb + gl]) : 0.0;
  const int32_t c = has ? a.C[t] : -1;
  const unsigned long long key =
      has ? (((unsigned long long)grp << 32) | (uint32_t)c) : (0xFFFFFFFF00000000ull | lane);
  const unsigned m = __match_any_sync(FULL, key);
  const bool leader = has && (lane == __ffs(m) - 1);
  // Ordered fold of each community group (lane order == CSR order).
  unsigned rem = leader ? m : 0u;
  const int rounds = __reduce_max_sync(FULL, (unsigned)__popc(rem));
  double sum = 0.0;
  for (int it = 0; it < rounds; ++it) {
    const int src = rem ? __ffs(rem) - 1 : lane;
    const double x = __shfl_sync(FULL, wt, src);
    if (rem) { sum = __dadd_rn(sum, x); rem &= rem - 1; }
  }
  // Self-loop weight, in CSR order.
  unsigned sm = __ballot_sync(FULL, has && t == v) & gmask;
  const int srounds = __reduce_max_sync(FULL, (unsigned)__popc(sm));
  double self_loop = 0.0;
  for (int it = 0; it < srounds; ++it) {
    const int src = sm ? __ffs(sm) - 1 : lane;
    const double x = __shfl_sync(FULL, wt, src);
    if (sm) { self_loop = __dadd_rn(self_loop, x); sm &= sm - 1; }
  }
  // Counter[own]
  const unsigned om = __ballot_sync(FULL, leader && c == own) & gmask;
  const double osum = __shfl_sync(FULL, sum, om ? __ffs(om) - 1 : lane);
  const double own_w = om ? osum : 0.0;
  const double degree = (valid && deg > 0) ? a.vDeg[v] : 0.0;
  double g = 0.0;
  int32_t bc = INT32_MAX;
  if (leader && c != own) {
    const double eix = __dsub_rn(own_w, self_loop);
    const double ax = __dsub_rn(a.cDeg[own], degree);
    const double gain = louvain_gain(sum, eix, degree, a.cDeg[c], ax, cst_of(a, v));
    if (gain > 0.0) { g = gain; bc = c; }
  }
#pragma unroll
  for (int off = G / 2; off >= 1; off >>= 1) {
    const double og = __shfl_xor_sync(FULL, g, off);
    const int32_t oc = __shfl_xor_sync(FULL, bc, off);
    if (better(og, oc, g, bc)) { g = og; bc = oc; }
  }
  if (valid && gl == 0) {
    if (skip) {
      emit_stay(a, pos, v, own);
    } else {
      const int32_t tgt = (deg == 0) ? -1 : finish_choice(a, own, g, bc);
      emit_decision(a, pos, v, own, tgt, degree, own_w, g);
    }
  }

}

template <int G>
__global__ void __launch_bounds__(256) k_sweep_small(SweepArgs a, int64_t begin, int64_t end) {
  constexpr int VPW = 32 / G;
  const int64_t wid = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const int64_t nw = ((int64_t)gridDim.x * blockDim.x) >> 5;
  for (int64_t base = begin + wid * VPW; base < end; base += nw * VPW) small_item<G>(a, base, end);
}

// ---------------------------------------------------------------------------
// Shared/global open-addressing table helpers.  Keys are community ids (>= 0),
// -1 marks an empty slot; values start at 0.0.

// Find or insert `key`, returning its slot.  Safe under concurrent inserts.
__device__ __forceinline__ uint32_t table_slot(int32_t *keys, uint32_t mask, int32_t key) {
  uint32_t s = hash_slot(key, mask);
  while (true) {
    int32_t k = keys[s];
    if (k == key) return s;
    if (k == -1) {
      int32_t old = atomicCAS(&keys[s], -1, key);
      if (old == -1 || old == key) return s;
    }
    s = (s + 1) & mask;
  }
}

// One warp accumulates row [rb, re) into the table in CSR order.  Leaders
// fold their group's weights starting from the table value, so each
// community's sum is the sequential CSR-order sum.  Returns the self-loop sum
// (same value in every lane).  With `atomic_add` the group sums are added with
// atomics instead (used when several warps share one table).
__device__ __forceinline__ double warp_accumulate(const SweepArgs &a, int32_t v, int64_t rb,
                                                  int64_t re, int64_t stride, int32_t *keys,
                                                  double *vals, uint32_t mask, bool atomic_add) {
  const int lane = threadIdx.x & 31;
  double self_loop = 0.0;
  // Software pipeline, two rounds deep: while this round is folded, the next
  // round's communities are gathered and the round after's entries load.
  // Neighbours' communities do not change during the sweep of one step.  The
  // row's entries are read once per sweep: streaming loads (evict-first in
  // L1 and L2) keep them from pushing the gathered per-vertex arrays out of L2.
  const int64_t j0 = rb + lane, j1 = j0 + stride;
  int32_t t_cur = (j0 < re) ? __ldcs(&a.tail[j0]) : -1;
  double w_cur = (j0 < re) ? __ldcs(&a.w[j0]) : 0.0;
  int32_t t_next = (j1 < re) ? __ldcs(&a.tail[j1]) : -1;
  double w_next = (j1 < re) ? __ldcs(&a.w[j1]) : 0.0;
  int32_t c_cur = (j0 < re) ? a.C[t_cur] : -1;
  for (int64_t base = rb; base < re; base += stride) {
    const int64_t j = base + lane;
    const bool has = j < re;
    const int32_t t = t_cur;
    const double wt = w_cur;
    const int32_t c = c_cur;
    const int64_t jn = j + stride, jnn = j + 2 * stride;
    c_cur = (jn < re) ? a.C[t_next] : -1;
    t_cur = t_next;
    w_cur = w_next;
    t_next = (jnn < re) ? __ldcs(&a.tail[jnn]) : -1;
    w_next = (jnn < re) ? __ldcs(&a.w[jnn]) : 0.0;
    const uint32_t key = has ? (uint32_t)c : (0x80000000u | lane);
    const unsigned m = __match_any_sync(FULL, key);
    const bool leader = has && (lane == __ffs(m) - 1);
    uint32_t slot = 0;
    double acc = 0.0;
    if (leader) {
      slot = table_slot(keys, mask, c);
      if (!atomic_add) acc = vals[slot];
    }
    unsigned rem = leader ? m : 0u;
    const int rounds = __reduce_max_sync(FULL, (unsigned)__popc(rem));
    for (int it = 0; it < rounds; ++it) {
      const int src = rem ? __ffs(rem) - 1 : lane;
      const double x = __shfl_sync(FULL, wt, src);
      if (rem) { acc = __dadd_rn(acc, x); rem &= rem - 1; }
    }
    if (leader) {
      if (atomic_add) atomicAdd(&vals[slot], acc);
      else vals[slot] = acc;
    }
    unsigned sm = __ballot_sync(FULL, has && t == v);
    while (sm) {  // warp-uniform
      const int src = __ffs(sm) - 1;
      self_loop = __dadd_rn(self_loop, __shfl_sync(FULL, wt, src));
      sm &= sm - 1;
    }
    __syncwarp();
  }
  return self_loop;
}

// Best (gain, id) over table slots [first, cap) with stride.
__device__ __forceinline__ void scan_table(const SweepArgs &a, const int32_t *keys,
                                           const double *vals, uint32_t first, uint32_t cap,
                                           uint32_t stride, int32_t own, double eix, double ax,
                                           double degree, double cst, double &g, int32_t &bc) {
  // four slots per thread in flight: their cDeg gathers overlap
  for (uint32_t s0 = first; s0 < cap; s0 += 4 * stride) {
    int32_t k[4];
    double cd[4];
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      const uint32_t s = s0 + q * stride;
      k[q] = (s < cap) ? keys[s] : -1;
    }
#pragma unroll
    for (int q = 0; q < 4; ++q) cd[q] = (k[q] >= 0 && k[q] != own) ? a.cDeg[k[q]] : 0.0;
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      if (k[q] < 0 || k[q] == own) continue;
      const double gain =
          louvain_gain(vals[s0 + q * stride], eix, degree, cd[q], ax, cst);
      if (gain > 0.0 && better(gain, k[q], g, bc)) { g = gain; bc = k[q]; }
    }
  }
}

__device__ __forceinline__ void warp_argmax(double &g, int32_t &bc) {
#pragma unroll
  for (int off = 16; off >= 1; off >>= 1) {
    const double og = __shfl_xor_sync(FULL, g, off);
    const int32_t oc = __shfl_xor_sync(FULL, bc, off);
    if (better(og, oc, g, bc)) { g = og; bc = oc; }
  }
}

// ---------------------------------------------------------------------------
// Rows of 33..warp_max entries: one warp per vertex, table (capacity <= 256)
// in the warp's slice of shared memory.
__device__ __forceinline__ void warp_table_vertex(const SweepArgs &a, int64_t pos, int32_t *keys,
                                                  double *vals) {
  const int lane = threadIdx.x & 31;
  const int32_t v = a.members[pos];
  if (skipped(a, v)) {
    if (lane == 0) emit_stay(a, pos, v, a.C[v]);
    return;
  }
  const int64_t rb = a.ptr[v], re = a.ptr[v + 1];
  const int32_t own = a.C[v];
  const double degree = a.vDeg[v];
  const double cdeg_own = a.cDeg[own];
  const int32_t own_size = (lane == 0) ? a.cSize[own] : 0;
  const uint32_t cap = table_cap(re - rb);
  const uint32_t mask = cap - 1;
  for (uint32_t s = lane; s < cap; s += 32) { keys[s] = -1; vals[s] = 0.0; }
  __syncwarp();
  if (lane == 0) keys[hash_slot(own, mask)] = own;
  __syncwarp();
  const double self_loop = warp_accumulate(a, v, rb, re, 32, keys, vals, mask, false);
  const double own_w = vals[hash_slot(own, mask)];
  const double eix = __dsub_rn(own_w, self_loop);
  const double ax = __dsub_rn(cdeg_own, degree);
  double g = 0.0;
  int32_t bc = INT32_MAX;
  scan_table(a, keys, vals, lane, cap, 32, own, eix, ax, degree, cst_of(a, v), g, bc);
  warp_argmax(g, bc);
  if (lane == 0)
    emit_decision(a, pos, v, own, finish_choice(a, own, own_size, g, bc), degree, own_w, g);
  __syncwarp();
}

template <int CAP>
__global__ void __launch_bounds__(256) k_sweep_warp(SweepArgs a, int64_t begin, int64_t end) {
  extern __shared__ unsigned char smem_raw[];
  const int warp = threadIdx.x >> 5;
  const int nwb = blockDim.x >> 5;
  double *vals = reinterpret_cast<double *>(smem_raw) + (size_t)warp * CAP;
  int32_t *keys = reinterpret_cast<int32_t *>(reinterpret_cast<double *>(smem_raw) + (size_t)nwb * CAP) +
                  (size_t)warp * CAP;
  const int64_t wid = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const int64_t nw = ((int64_t)gridDim.x * blockDim.x) >> 5;
  for (int64_t pos = begin + wid; pos < end; pos += nw) warp_table_vertex(a, pos, keys, vals);
}

// ---------------------------------------------------------------------------
// Large rows without the persistent kernel (parallel accumulation): one block
// per vertex, the table in shared memory; all warps take rounds of 32 entries
// and add group sums with atomics.  All threads call.
__device__ __forceinline__ void block_vertex(const SweepArgs &a, int64_t pos, int32_t *keys,
                                             double *vals, double *s_self, double *s_g,
                                             int32_t *s_c) {
  const int lane = threadIdx.x & 31;
  const int warp = threadIdx.x >> 5;
  const int nwb = blockDim.x >> 5;
  const int32_t v = a.members[pos];
  const int64_t rb = a.ptr[v], re = a.ptr[v + 1];
  const uint32_t cap = table_cap(re - rb);
  const uint32_t mask = cap - 1;
  for (uint32_t s = threadIdx.x; s < cap; s += blockDim.x) { keys[s] = -1; vals[s] = 0.0; }
  __syncthreads();
  const int32_t own = a.C[v];
  if (threadIdx.x == 0) keys[hash_slot(own, mask)] = own;
  __syncthreads();
  const double sl =
      warp_accumulate(a, v, rb + 32 * warp, re, 32 * nwb, keys, vals, mask, true);
  if (lane == 0) s_self[warp] = sl;
  __syncthreads();
  double self_loop = 0.0;
  for (int k = 0; k < nwb; ++k) self_loop = __dadd_rn(self_loop, s_self[k]);
  const double degree = a.vDeg[v];
  const double own_w = vals[hash_slot(own, mask)];
  const double eix = __dsub_rn(own_w, self_loop);
  const double ax = __dsub_rn(a.cDeg[own], degree);
  double g = 0.0;
  int32_t bc = INT32_MAX;
  scan_table(a, keys, vals, threadIdx.x, cap, blockDim.x, own, eix, ax, degree, cst_of(a, v), g, bc);
  warp_argmax(g, bc);
  if (lane == 0) { s_g[warp] = g; s_c[warp] = bc; }
  __syncthreads();
  if (threadIdx.x == 0) {
    for (int k = 1; k < nwb; ++k)
      if (better(s_g[k], s_c[k], g, bc)) { g = s_g[k]; bc = s_c[k]; }
    emit_decision(a, pos, v, own, finish_choice(a, own, g, bc), degree, own_w, g);
  }
  __syncthreads();
}

__global__ void __launch_bounds__(512) k_sweep_block(SweepArgs a, int64_t begin, int64_t end) {
  extern __shared__ unsigned char smem_raw[];
  __shared__ double s_self[32];
  __shared__ double s_g[32];
  __shared__ int32_t s_c[32];
  for (int64_t pos = begin + blockIdx.x; pos < end; pos += gridDim.x) {
    const int32_t v = a.members[pos];
    const uint32_t cap = table_cap(a.ptr[v + 1] - a.ptr[v]);
    double *vals = reinterpret_cast<double *>(smem_raw);
    int32_t *keys = reinterpret_cast<int32_t *>(vals + cap);
    block_vertex(a, pos, keys, vals, s_self, s_g, s_c);
  }
}

// ---------------------------------------------------------------------------
// Hubs in the parallel-accumulation modes (hub.cuh): the hubs of a schedule,
// numbered densely, with their chunks and partitions.
constexpr int kHubChunk = 2048;     // most CSR entries per chunk
constexpr int kHubChunkMin = 512;   // fewest the schedule cuts rows into

struct HubInfo {
  int32_t pos;              // member slot
  int32_t chunk0, nchunks;  // its chunks
  int32_t part0, nparts;    // its partitions (nparts a power of two)
  int32_t inline_pairs;     // most pairs the last chunk's block merges itself
};
struct HubChunk {
  int64_t beg;              // CSR range [beg, beg + len)
  int64_t out;              // its pairs in out_c / out_w
  int64_t off;              // its nparts + 1 partition offsets in part_off
  int32_t len, hub;
};
struct HubState {
  double self_w, own_w;     // row sums: self-loops, own community
  int32_t cnt;              // pairs written
  int32_t chunks_left, parts_left;
  uint32_t state;           // 4 * epoch + 1 decided, + 2 its partitions decide
};
struct HubWork {
  const HubInfo *hubs;
  const HubChunk *chunks;
  const int32_t *part_hub;  // partition task -> hub
  HubState *state;
  int32_t *out_c;           // pairs of the step's chunks
  double *out_w;
  uint16_t *part_off;
  double *part_g;           // per partition task: best gain
  int32_t *part_c;          //                     and its community
  uint32_t epoch;           // this launch of the persistent kernel (0: a launch per kernel)
  int32_t *err;             // set when a partition's wait gives up
  // persistent kernel on thread-block clusters (cluster_row_tasks): the hub
  // rows' tasks, one per (row, community partition); a partitioned row's
  // partial bests are ct_g/ct_c[task], and ct_left[its first task] counts its
  // partitions not yet done
  const int32_t *ct_pos;    // task -> member slot
  const int32_t *ct_part;   // task -> partition index
  const int32_t *ct_nparts; // task -> partitions of its row (a power of two)
  double *ct_g;             // task -> best gain of its partition
  int32_t *ct_c;            //         and its community
  int32_t *ct_left;
};

// ---------------------------------------------------------------------------
// Hub rows on thread-block clusters (persistent kernel, parallel modes).  The
// CL blocks of a cluster hold one open-addressing table in their shared
// memory, reached through distributed shared memory: slot s lives in block
// s mod CL at local slot s / CL, up to CL x kClusterBlockSlots slots.  A row
// whose table would need more is split by community: partition p of P takes
// the neighbours whose community c has mix32(c) mod P = p, each partition a
// separate task that reads the whole row; the partitions' best moves are
// folded by the last one to finish.  Nothing of a hub table touches HBM.

constexpr int kClusterBlockSlots = 8192;  // table slots in one block's shared region
constexpr int kClusterMax = 16;           // largest cluster the tasks support
constexpr int kClusterMaxParts = 2;       // most partitions of a cluster row (each reads the row)

// Per-block scratch of the cluster tasks; rank 0's copy is the one read.
struct ClusterShared {
  double acc[2][2];              // by task parity: the row's self-loop weight, Counter[own]
  double g[kClusterMax];         // per block: best gain
  int32_t c[kClusterMax];        //            and its community
  int64_t next;                  // next task of the step (set by rank 0)
};

// Partitions of a row of `deg` entries on a cluster of `cl` blocks, and the
// slots of each partition's table (both powers of two).
__host__ __device__ inline void cluster_row_shape(int64_t deg, int cl, uint32_t *nparts,
                                                  uint32_t *cap) {
  const uint32_t need = table_cap(deg);
  const uint32_t full = (uint32_t)cl * kClusterBlockSlots;
  *nparts = need > full ? need / full : 1u;
  *cap = need / *nparts;
}

// Find or insert `key` in the cluster table; returns the slot, or UINT32_MAX
// when every slot holds another key (a partition far above its expected
// load; the caller raises the error flag).
__device__ __forceinline__ uint32_t cluster_table_slot(cooperative_groups::cluster_group &cl,
                                                       int32_t *keys, uint32_t mask,
                                                       unsigned cl_bits, int32_t key) {
  uint32_t s = hash_slot(key, mask);
  const uint32_t rank_mask = (1u << cl_bits) - 1u;
  for (uint32_t probe = 0; probe <= mask; ++probe) {
    int32_t *k = cl.map_shared_rank(keys, s & rank_mask) + (s >> cl_bits);
    const int32_t old = atomicCAS(k, -1, key);
    if (old == -1 || old == key) return s;
    s = (s + 1) & mask;
  }
  return UINT32_MAX;
}

// Warp gw of the cluster's nw warps adds its entries of row [rb, rb + deg) that
// fall in partition `part` to the cluster table, and sums (per lane) the row's
// self-loop weight and the weight to the row's own community.
__device__ __forceinline__ void cluster_accumulate(const SweepArgs &a,
                                                   cooperative_groups::cluster_group &cl,
                                                   int32_t v, int32_t own, int64_t rb, int64_t re,
                                                   int64_t gw, int64_t nw, int32_t *keys,
                                                   double *vals, uint32_t mask, unsigned cl_bits,
                                                   uint32_t part, uint32_t part_mask,
                                                   double &self_w, double &own_w, bool &overflow) {
  const int lane = threadIdx.x & 31;
  const int64_t stride = 32 * nw;
  const uint32_t rank_mask = (1u << cl_bits) - 1u;
  // two rounds in flight, as in warp_accumulate
  const int64_t j0 = rb + 32 * gw + lane, j1 = j0 + stride;
  int32_t t_cur = (j0 < re) ? __ldcs(&a.tail[j0]) : -1;
  double w_cur = (j0 < re) ? __ldcs(&a.w[j0]) : 0.0;
  int32_t t_next = (j1 < re) ? __ldcs(&a.tail[j1]) : -1;
  double w_next = (j1 < re) ? __ldcs(&a.w[j1]) : 0.0;
  int32_t c_cur = (j0 < re) ? a.C[t_cur] : -1;
  for (int64_t base = rb + 32 * gw; base < re; base += stride) {
    const int64_t j = base + lane;
    const bool has = j < re;
    const int32_t t = t_cur;
    const double wt = w_cur;
    const int32_t c = c_cur;
    const int64_t jn = j + stride, jnn = j + 2 * stride;
    c_cur = (jn < re) ? a.C[t_next] : -1;
    t_cur = t_next;
    w_cur = w_next;
    t_next = (jnn < re) ? __ldcs(&a.tail[jnn]) : -1;
    w_next = (jnn < re) ? __ldcs(&a.w[jnn]) : 0.0;
    if (has && t == v) self_w += wt;
    if (has && c == own) own_w += wt;
    const bool mine = has && (mix32((uint32_t)c) & part_mask) == part;
    const uint32_t key = mine ? (uint32_t)c : (0x80000000u | lane);
    const unsigned m = __match_any_sync(FULL, key);
    const bool leader = mine && (lane == __ffs(m) - 1);
    double acc = 0.0;
    unsigned rem = leader ? m : 0u;
    const int rounds = __reduce_max_sync(FULL, (unsigned)__popc(rem));
    for (int it = 0; it < rounds; ++it) {
      const int src = rem ? __ffs(rem) - 1 : lane;
      const double x = __shfl_sync(FULL, wt, src);
      if (rem) { acc += x; rem &= rem - 1; }
    }
    if (leader) {
      const uint32_t s = cluster_table_slot(cl, keys, mask, cl_bits, c);
      if (s == UINT32_MAX) overflow = true;
      else atomicAdd(cl.map_shared_rank(vals, s & rank_mask) + (s >> cl_bits), acc);
    }
  }
}

// The hub tasks [tb, tb + ntask) of one step, run by every thread of every
// block of the cluster.  `keys`/`vals` are this block's table region (at
// least kClusterBlockSlots slots), `cs` its ClusterShared, `red` 32 doubles
// and `redc` 32 ints of block scratch (every block of the cluster calls with
// the same tb, ntask and ctr).  Two cluster barriers per task: after
// the inserts (row sums complete), and after the scan (every block's best in
// rank 0, its own slots cleared again, the next task published).  The row
// sums alternate between two slots by task parity, so rank 0 clears one pair
// while the blocks may already add to the other.
__device__ __forceinline__ void cluster_row_tasks(const SweepArgs &a, const HubWork &h, int64_t tb,
                                               int64_t ntask, unsigned *ctr, int32_t *keys,
                                               double *vals, ClusterShared *cs, double *red,
                                               int32_t *redc) {
  namespace cgx = cooperative_groups;
  cgx::cluster_group cl = cgx::this_cluster();
  const unsigned ncl = cl.num_blocks(), rank = cl.block_rank();
  const unsigned cl_bits = __ffs(ncl) - 1;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nwb = blockDim.x >> 5;
  ClusterShared *cs0 = cl.map_shared_rank(cs, 0);
  for (uint32_t q = threadIdx.x; q < kClusterBlockSlots; q += blockDim.x) {
    keys[q] = -1;
    vals[q] = 0.0;
  }
  if (rank == 0 && threadIdx.x == 0) {
    cs->next = (int64_t)atomicAdd(ctr, 1u);
    cs->acc[0][0] = cs->acc[0][1] = cs->acc[1][0] = cs->acc[1][1] = 0.0;
  }
  cl.sync();
  for (unsigned it = 0;; ++it) {
    const int64_t t = cs0->next;
    if (t >= ntask) break;
    const int64_t ti = tb + t;
    const int32_t pos = h.ct_pos[ti];
    const uint32_t part = (uint32_t)h.ct_part[ti], nparts = (uint32_t)h.ct_nparts[ti];
    const int32_t v = a.members[pos];
    const int32_t own = a.C[v];
    if (skipped(a, v)) {  // cluster-uniform
      if (rank == 0 && threadIdx.x == 0 && part == 0) emit_stay(a, pos, v, own);
      cl.sync();  // every block has read `next`
      if (rank == 0 && threadIdx.x == 0)
        cs->next = (int64_t)atomicAdd(ctr, 1u);
      cl.sync();
      continue;
    }
    double *acc = cs0->acc[it & 1];
    const int64_t rb = a.ptr[v], re = a.ptr[v + 1];
    uint32_t np, cap;
    cluster_row_shape(re - rb, (int)ncl, &np, &cap);
    const uint32_t local = cap >> cl_bits;  // this block's slots of the table
    double self_w = 0.0, own_w = 0.0;
    bool overflow = false;
    cluster_accumulate(a, cl, v, own, rb, re, (int64_t)rank * nwb + warp, (int64_t)ncl * nwb, keys,
                       vals, cap - 1, cl_bits, part, nparts - 1, self_w, own_w, overflow);
    if (overflow) atomicExch(h.err, 2);
#pragma unroll
    for (int off = 16; off >= 1; off >>= 1) {
      self_w += __shfl_xor_sync(FULL, self_w, off);
      own_w += __shfl_xor_sync(FULL, own_w, off);
    }
    if (lane == 0) {
      if (self_w != 0.0) atomicAdd(&acc[0], self_w);
      if (own_w != 0.0) atomicAdd(&acc[1], own_w);
    }
    cl.sync();  // every entry is in the table, the row sums are complete
    const double degree = a.vDeg[v];
    const double row_own = acc[1];
    const double eix = __dsub_rn(row_own, acc[0]);
    const double ax = __dsub_rn(a.cDeg[own], degree);
    double g = 0.0;
    int32_t bc = INT32_MAX;
    scan_table(a, keys, vals, threadIdx.x, local, blockDim.x, own, eix, ax, degree, cst_of(a, v),
               g, bc);
    warp_argmax(g, bc);
    if (lane == 0) { red[warp] = g; redc[warp] = bc; }
    __syncthreads();  // the block's scan is done: its slots are cleared below
    if (threadIdx.x == 0) {
      for (int k = 1; k < nwb; ++k)
        if (better(red[k], redc[k], g, bc)) { g = red[k]; bc = redc[k]; }
      cs0->g[rank] = g;
      cs0->c[rank] = bc;
      if (rank == 0) cs->next = (int64_t)atomicAdd(ctr, 1u);
    }
    for (uint32_t q = threadIdx.x; q < local; q += blockDim.x) {
      keys[q] = -1;
      vals[q] = 0.0;
    }
    cl.sync();  // bests in rank 0, tables clear, next task published
    if (rank == 0 && threadIdx.x == 0) {
      g = cs->g[0];
      bc = cs->c[0];
      for (unsigned k = 1; k < ncl; ++k)
        if (better(cs->g[k], cs->c[k], g, bc)) { g = cs->g[k]; bc = cs->c[k]; }
      cs->acc[it & 1][0] = 0.0;  // read by every block before the barrier above
      cs->acc[it & 1][1] = 0.0;
      bool decide = true;
      if (nparts > 1) {
        // the last partition of the row to finish folds the others' bests
        h.ct_g[ti] = g;
        h.ct_c[ti] = bc;
        __threadfence();
        decide = atomicSub(&h.ct_left[ti - part], 1) == 1;
        if (decide) {
          __threadfence();
          const int64_t t0 = ti - part;
          for (uint32_t k = 0; k < nparts; ++k) {
            const double pg = __ldcg(&h.ct_g[t0 + k]);
            const int32_t pc = __ldcg(&h.ct_c[t0 + k]);
            if (better(pg, pc, g, bc)) { g = pg; bc = pc; }
          }
          h.ct_left[t0] = (int32_t)nparts;
        }
      }
      if (decide) emit_decision(a, pos, v, own, finish_choice(a, own, g, bc), degree, row_own, g);
    }
  }
}

}  // namespace glv
