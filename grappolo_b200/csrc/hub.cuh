// Hub rows (longer than the block bin) in the parallel-accumulation modes:
// many blocks per row, two kinds of block tasks.
//
//   chunk      at most kHubChunk entries: folded into the block's shared table,
//              then written out as (community, weight) pairs grouped by
//              partition (mix32(community) mod nparts) with the partitions'
//              offsets.  The block that finishes a hub's last chunk merges all
//              pairs and decides the hub when they are few (inline_pairs);
//   partition  one partition's pairs of all the hub's chunks, merged in the
//              block's shared table and scanned for the best gain; the last
//              partition to finish folds the partitions' bests and decides.
//
// What bounds it: a step is as long as its slowest row, and a hub was that row.
// Global hash tables took a chain of compare-and-swaps on L2 (785 cycles each,
// as many as the longest probe sequence of a batch of keys) and then a scan of
// the filled slots (three dependent gathers): on R-MAT 18, whose hub steps hold
// 3 to 13 chunks, 9 us of inserts and 21 us of scan after 8 us of folding.  Pairs are
// written and read once, in runs, and every table access stays on chip.
#pragma once

#include "rows.cuh"

namespace glv {

constexpr int kHubThreads = 512;
constexpr int kHubTableCap = 8192;   // the block's table
constexpr int kHubList = 4096;       // filled slots a merge may hold at once
constexpr int kHubInline = 2048;     // pairs the last chunk's block merges itself; in full
constexpr int kHubInlineFull = 4096; // steps (HubInfo::inline_pairs)
constexpr int kHubMaxParts = 512;
constexpr int kHubRuns = 512;        // chunks a merge looks up at a time
constexpr uint32_t kSpinLimit = 1u << 22;  // polls of a partition's wait (>= 128 ns each)
static_assert(kHubInlineFull <= kHubList, "an inline merge fits the list");
static_assert(kHubChunk <= 2048 && kHubChunk <= kHubTableCap / 2, "a chunk fits the table");
static_assert(kHubRuns <= kHubThreads && kHubRuns <= kHubMaxParts, "one thread per run");
static_assert(kHubChunk < 65536 && kHubTableCap <= kNoSlot, "16-bit offsets and slots");

// Partitions of a row (a power of two, at least 2) of about `entries` row
// entries each (more only past kHubMaxParts).
__host__ __device__ inline int hub_parts(int64_t deg, int entries) {
  int p = 2;
  while (p < kHubMaxParts && (int64_t)p * entries < deg) p <<= 1;
  return p;
}

// Block scratch of the hub tasks.
struct HubShared {
  int hist[kHubMaxParts + 1];  // pairs per partition, then running offsets; merge: run starts
  int base[kHubRuns];          // merge: the runs' first pairs, from the hub's first
  int wsum[kHubThreads / 32];
  int count;                   // merge: filled slots listed
  int over;                    // merge: more distinct communities than the list holds
  int flag;
  uint32_t word;
};

__device__ __forceinline__ uint32_t ld_acquire(const uint32_t *p) {
  uint32_t v;
  asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
  return v;
}

// Best (gain, id) of this thread over the communities of partitions [p0, p1)
// of hub `hb`.  All threads of the block call; the table is empty on entry and
// on exit.  When the partitions hold more distinct communities than the list,
// they are merged in several passes over disjoint shares of the communities
// (further bits of mix32), twice as many shares after every overflow.
__device__ __forceinline__ void hub_merge(const SweepArgs &a, const HubWork &h, const HubInfo &hb,
                                          int p0, int p1, double eix, double ax, double degree,
                                          double cst, int32_t *keys, double *vals, uint16_t *list,
                                          HubShared *sh, double &g, int32_t &bc) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  constexpr int NW = kHubThreads / 32;
  const uint32_t mask = kHubTableCap - 1;
  const int64_t out0 = h.chunks[hb.chunk0].out;
  int bits = 0;
  for (uint32_t share = 0; share < (1u << bits);) {
    if (threadIdx.x == 0) { sh->count = 0; sh->over = 0; }
    __syncthreads();
    const uint32_t smask = (1u << bits) - 1u;
    // The chunks' runs of these partitions as one sequence, kHubRuns chunks at
    // a time: every thread looks one chunk up, then all threads share the pairs
    // (a warp per chunk left most lanes idle: runs are short and few).
    for (int k0 = 0; k0 < hb.nchunks; k0 += kHubRuns) {
      const int nk = min(kHubRuns, hb.nchunks - k0);
      int mine = 0;
      if (threadIdx.x < nk) {
        const HubChunk &ch = h.chunks[hb.chunk0 + k0 + threadIdx.x];
        const uint16_t *off = h.part_off + ch.off;
        const int b = __ldcg(&off[p0]);
        mine = __ldcg(&off[p1]) - b;
        sh->base[threadIdx.x] = (int)(ch.out - out0) + b;
      }
      // exclusive prefix of the run lengths: within the warp, then over warps
      int incl = mine;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const int y = __shfl_up_sync(FULL, incl, o);
        if (lane >= o) incl += y;
      }
      if (lane == 31) sh->wsum[warp] = incl;
      __syncthreads();
      int before = 0, total = 0;
#pragma unroll
      for (int q = 0; q < NW; ++q) {
        before += q < warp ? sh->wsum[q] : 0;
        total += sh->wsum[q];
      }
      if (threadIdx.x < nk) sh->hist[threadIdx.x] = before + incl - mine;
      __syncthreads();
      for (int i = threadIdx.x; i - lane < total; i += kHubThreads) {
        const bool has = i < total;
        int lo = 0, hi = nk - 1;  // the last run starting at or before i
        while (lo < hi) {
          const int mid = (lo + hi + 1) >> 1;
          if (sh->hist[mid] <= i) lo = mid; else hi = mid - 1;
        }
        const int64_t at = out0 + sh->base[lo] + (i - sh->hist[lo]);
        const int32_t c = has ? __ldcg(&h.out_c[at]) : -1;
        const double w = has ? __ldcg(&h.out_w[at]) : 0.0;
        bool fresh = false;
        uint32_t s = hash_slot(c, mask);
        if (has && ((mix32((uint32_t)c) >> 12) & smask) == share &&
            *(volatile int *)&sh->over == 0) {
          while (true) {
            const int32_t x = atomicCAS(&keys[s], -1, c);
            fresh = x == -1;
            if (x == -1 || x == c) break;
            s = (s + 1) & mask;
          }
          atomicAdd(&vals[s], w);
        }
        const unsigned fm = __ballot_sync(FULL, fresh);
        if (fm) {
          int n = 0;
          if (lane == 0) n = atomicAdd(&sh->count, __popc(fm));
          n = __shfl_sync(FULL, n, 0) + __popc(fm & ((1u << lane) - 1u));
          if (fresh) {
            if (n < kHubList) list[n] = (uint16_t)s;
            else sh->over = 1;
          }
        }
      }
      __syncthreads();  // the pairs are in the table, the runs' offsets read
    }
    if (sh->over) {  // block-uniform: start over with twice the shares
      __syncthreads();
      for (int q = threadIdx.x; q < kHubTableCap; q += kHubThreads) {
        keys[q] = -1;
        vals[q] = 0.0;
      }
      ++bits;
      share = 0;
      continue;
    }
    const int n = sh->count;
    for (int q0 = threadIdx.x; q0 < n; q0 += 4 * kHubThreads) {
      int32_t k[4];
      double val[4], cd[4];
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        const int i = q0 + q * kHubThreads;
        k[q] = -1;
        if (i < n) {
          const uint16_t s = list[i];
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
    ++share;
    __syncthreads();
  }
}

// The block's best into thread 0's (g, bc); one barrier.
__device__ __forceinline__ void hub_block_best(double &g, int32_t &bc, double *s_g, int32_t *s_c) {
  warp_argmax(g, bc);
  if ((threadIdx.x & 31) == 0) { s_g[threadIdx.x >> 5] = g; s_c[threadIdx.x >> 5] = bc; }
  __syncthreads();
  if (threadIdx.x == 0)
    for (int k = 1; k < kHubThreads / 32; ++k)
      if (better(s_g[k], s_c[k], g, bc)) { g = s_g[k]; bc = s_c[k]; }
}

// The hub's state for its next sweep (the one thread that decided it calls).
__device__ __forceinline__ void hub_reset(HubState *hs, const HubInfo &hb) {
  hs->cnt = 0;
  hs->self_w = 0.0;
  hs->own_w = 0.0;
  hs->chunks_left = hb.nchunks;
  hs->parts_left = hb.nparts;
}

// One chunk as a block task (all threads call).
__device__ __forceinline__ void hub_chunk_task(const SweepArgs &a, const HubWork &h, int64_t ci,
                                               int32_t *keys, double *vals, uint16_t *fill,
                                               HubShared *sh, double *s_g, int32_t *s_c) {
  const int lane = threadIdx.x & 31;
  const HubChunk ch = h.chunks[ci];
  const HubInfo hb = h.hubs[ch.hub];
  HubState *hs = &h.state[ch.hub];
  const int32_t v = a.members[hb.pos];
  const bool skip = skipped(a, v);  // block-uniform
  const uint32_t pmask = (uint32_t)hb.nparts - 1u;
  if (!skip) {
    for (int q = threadIdx.x; q <= hb.nparts; q += kHubThreads) sh->hist[q] = 0;
    double self_w = 0.0, own_w = 0.0;
    const int rounds =
        row_accumulate<kHubThreads>(a, v, a.C[v], ch.beg, ch.len, keys, vals, kHubTableCap - 1,
                                    fill + threadIdx.x, self_w, own_w);
    if (__any_sync(FULL, self_w != 0.0)) self_w = warp_sum(self_w);
    if (__any_sync(FULL, own_w != 0.0)) own_w = warp_sum(own_w);
    if (lane == 0) {
      if (self_w != 0.0) atomicAdd(&hs->self_w, self_w);
      if (own_w != 0.0) atomicAdd(&hs->own_w, own_w);
    }
    __syncthreads();
    for (int r = 0; r < rounds; ++r) {
      const uint16_t s = fill[threadIdx.x + r * kHubThreads];
      if (s != kNoSlot) atomicAdd(&sh->hist[mix32((uint32_t)keys[s]) & pmask], 1);
    }
    __syncthreads();
    if (threadIdx.x < 32) {  // exclusive scan; offsets out, and kept as running counters
      uint16_t *off = h.part_off + ch.off;
      int sum = 0;
      for (int q = lane; q - lane < hb.nparts; q += 32) {
        const int x = (q < hb.nparts) ? sh->hist[q] : 0;
        int incl = x;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
          const int y = __shfl_up_sync(FULL, incl, o);
          if (lane >= o) incl += y;
        }
        if (q < hb.nparts) {
          sh->hist[q] = sum + incl - x;
          off[q] = (uint16_t)(sum + incl - x);
        }
        sum += __shfl_sync(FULL, incl, 31);
      }
      if (lane == 0) {
        off[hb.nparts] = (uint16_t)sum;
        atomicAdd(&hs->cnt, sum);
      }
    }
    __syncthreads();
    for (int r = 0; r < rounds; ++r) {
      const uint16_t s = fill[threadIdx.x + r * kHubThreads];
      if (s == kNoSlot) continue;
      const int32_t c = keys[s];
      const int at = atomicAdd(&sh->hist[mix32((uint32_t)c) & pmask], 1);
      h.out_c[ch.out + at] = c;
      h.out_w[ch.out + at] = vals[s];
      keys[s] = -1;
      vals[s] = 0.0;
    }
  }
  // every thread publishes its pairs before the countdown
  __threadfence();
  __syncthreads();
  if (threadIdx.x == 0) sh->flag = (atomicSub(&hs->chunks_left, 1) == 1) ? 1 : 0;
  __syncthreads();
  if (!sh->flag) return;
  __threadfence();
  const uint32_t decided = 4u * h.epoch + 1u;
  const int32_t own = a.C[v];
  if (skip) {
    if (threadIdx.x == 0) {
      emit_stay(a, hb.pos, v, own);
      hs->chunks_left = hb.nchunks;
      if (h.epoch) {
        __threadfence();
        atomicExch(&hs->state, decided);
      }
    }
    return;
  }
  if (__ldcg(&hs->cnt) > hb.inline_pairs) {
    if (threadIdx.x == 0) atomicExch(&hs->state, decided + 1u);  // its partitions decide it
    return;
  }
  const double degree = a.vDeg[v];
  const double own_w = __ldcg(&hs->own_w);
  const double eix = __dsub_rn(own_w, __ldcg(&hs->self_w));
  const double ax = __dsub_rn(a.cDeg[own], degree);
  double g = 0.0;
  int32_t bc = INT32_MAX;
  hub_merge(a, h, hb, 0, hb.nparts, eix, ax, degree, cst_of(a, v), keys, vals, fill, sh, g, bc);
  hub_block_best(g, bc, s_g, s_c);
  if (threadIdx.x == 0) {
    emit_decision(a, hb.pos, v, own, finish_choice(a, own, g, bc), degree, own_w, g);
    hub_reset(hs, hb);
    if (h.epoch) {
      __threadfence();
      atomicExch(&hs->state, decided);
    }
  }
}

// One partition as a block task (all threads call).  In the persistent kernel
// partitions are queued after every chunk of their step and a chunk never
// waits, so the wait for the hub's chunks ends.  With a launch per kernel
// (epoch 0) the chunks are done, and state 2 marks the hubs that need this.
__device__ __forceinline__ void hub_part_task(const SweepArgs &a, const HubWork &h, int64_t si,
                                              int32_t *keys, double *vals, uint16_t *fill,
                                              HubShared *sh, double *s_g, int32_t *s_c) {
  const int lane = threadIdx.x & 31;
  const int32_t hub = h.part_hub[si];
  const HubInfo hb = h.hubs[hub];
  HubState *hs = &h.state[hub];
  const uint32_t decided = 4u * h.epoch + 1u;
  if (threadIdx.x == 0) {
    uint32_t st, it = 0;
    while ((st = ld_acquire(&hs->state)) < decided && h.epoch) {
      if (++it > kSpinLimit) {
        atomicExch(h.err, 1);
        st = 0;
        break;
      }
      __nanosleep(128);
    }
    sh->word = st;
  }
  __syncthreads();
  const uint32_t st = sh->word;
  __syncthreads();
  if (st != decided + 1u) return;  // decided by its last chunk (block-uniform)
  const int32_t v = a.members[hb.pos];
  const int32_t own = a.C[v];
  const double degree = a.vDeg[v];
  const double own_w = __ldcg(&hs->own_w);
  const double eix = __dsub_rn(own_w, __ldcg(&hs->self_w));
  const double ax = __dsub_rn(a.cDeg[own], degree);
  const int p = (int)(si - hb.part0);
  double g = 0.0;
  int32_t bc = INT32_MAX;
  hub_merge(a, h, hb, p, p + 1, eix, ax, degree, cst_of(a, v), keys, vals, fill, sh, g, bc);
  hub_block_best(g, bc, s_g, s_c);
  if (threadIdx.x == 0) {
    h.part_g[si] = g;
    h.part_c[si] = bc;
    __threadfence();
    sh->flag = (atomicSub(&hs->parts_left, 1) == 1) ? 1 : 0;
  }
  __syncthreads();
  const bool last = sh->flag != 0;
  __syncthreads();
  if (!last || threadIdx.x >= 32) return;
  __threadfence();
  g = 0.0;
  bc = INT32_MAX;
  for (int k = lane; k < hb.nparts; k += 32) {
    const double pg = __ldcg(&h.part_g[hb.part0 + k]);
    const int32_t pc = __ldcg(&h.part_c[hb.part0 + k]);
    if (better(pg, pc, g, bc)) { g = pg; bc = pc; }
  }
  warp_argmax(g, bc);
  if (lane == 0) {
    emit_decision(a, hb.pos, v, own, finish_choice(a, own, g, bc), degree, own_w, g);
    hub_reset(hs, hb);
    if (!h.epoch) hs->state = 0;
  }
}

// The launch-per-kernel path: all chunks of a step, then all partitions.
constexpr int kHubSmem = kHubTableCap * (int)(sizeof(double) + sizeof(int32_t)) +
                         kHubList * (int)sizeof(uint16_t);
static_assert(kHubList >= kHubChunk, "a chunk's filled slots fit the list");

template <bool kParts>
__global__ void __launch_bounds__(kHubThreads) k_hub_tasks(SweepArgs a, HubWork h, int64_t b,
                                                           int64_t e) {
  extern __shared__ unsigned char smem_raw[];
  __shared__ HubShared sh;
  __shared__ double s_g[32];
  __shared__ int32_t s_c[32];
  double *vals = reinterpret_cast<double *>(smem_raw);
  int32_t *keys = reinterpret_cast<int32_t *>(vals + kHubTableCap);
  uint16_t *fill = reinterpret_cast<uint16_t *>(keys + kHubTableCap);
  for (int q = threadIdx.x; q < kHubTableCap; q += kHubThreads) {
    keys[q] = -1;
    vals[q] = 0.0;
  }
  for (int64_t t = b + blockIdx.x; t < e; t += gridDim.x) {
    __syncthreads();
    if (kParts) hub_part_task(a, h, t, keys, vals, fill, &sh, s_g, s_c);
    else hub_chunk_task(a, h, t, keys, vals, fill, &sh, s_g, s_c);
  }
}

}  // namespace glv
