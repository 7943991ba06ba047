// Distance-1 colouring in priority order as a dataflow (Jones-Plassmann).
//
// A vertex takes the smallest colour that none of its higher-priority
// neighbours has.  With priority "lower id first" this is exactly the
// sequential first-fit pass of Coloring/coloringDistanceOne.cpp:137-150 at one
// thread; with hashed priorities it is the parallel independent-set form.  The
// result is a function of the priorities alone, whatever the order in which
// the vertices become ready.
//
// What bounds it: the longest chain of dependent vertices (R-MAT 20 in id
// order: 1,233 links, a planted partition of 100k vertices: 1,816), each link
// a few L2 round trips; the bytes (4 B per entry and direction) are minor.
// Rounds with a grid barrier, one warp scanning a whole row twice per round,
// made a round as long as its longest row: R-MAT 20, whose rows on that chain
// sum to 5.8 M entries, took 182 ms, R-MAT 22 (edge factor 14) 583 ms, the
// 100k partition 10.6 ms.  Here nothing waits for a round; the same colourings
// take 7.5, 13.9 and 3.7 ms:
//
// * one 64-bit word per vertex holds the higher-priority neighbours not yet
//   coloured (high half) and the colours 0..31 they took (low half).  A vertex
//   that got colour c sends every lower-priority neighbour an OR of bit c and a
//   subtraction of 1 << 32.  Both go to one address, so the subtraction that
//   takes the count to zero returns every colour below 32: no fence and no scan
//   of the row.  Colours from 32 up go to a bitmap word beside it (`ext`),
//   ordered before the subtraction by a fence;
// * the warp that made a vertex ready colours it at once, keeps one such vertex
//   as its own next one and publishes the others in a queue, rows cut into
//   tasks of kFlowChunk entries so that a hub's row is sent by many warps.  A
//   task word holds vertex, colour and part, so publishing needs no fence;
// * a vertex without lower-priority neighbours is finished by the lane that
//   made it ready.
//
// Waiting: a warp polls the queue slot of its ticket.  It leaves when every
// published task is finished (nothing can become ready any more), and gives up
// with status[1] when neither counter moved for kFlowStallNs.  A warp holds no
// task while it waits, so the launch needs no co-residency.
#pragma once

#include "glv_common.cuh"
#include "phase_kernels.cuh"

namespace glv {

constexpr int kFlowThreads = 256;
// Blocks per SM of the dataflow kernel.  Idle warps poll, and polling slows the
// atomics of the others: 4 blocks took 17.3 ms on R-MAT 20's second level, 2 or 1
// 12.0; a batch of 200 graphs, with work for every warp, 18.4 ms with 2 and
// 22.1 with 1.
constexpr int kFlowBlocks = 2;
constexpr int kFlowChunk = 512;                         // fewest entries of a split row's task
constexpr int64_t kFlowMaxParts = (int64_t)1 << 20;     // tasks of one row (21 bits of a task word)
constexpr int kFlowCtr = 16;                            // counters on lines of their own (128 B)
constexpr int kFlowChain = 64;                          // own next vertices before one is published
constexpr unsigned long long kFlowEmpty = ~0ull;
constexpr unsigned long long kFlowStallNs = 5000000000ull;

struct ColorFlow {
  int64_t nv;
  const int64_t *ptr;
  const int32_t *tail;
  int hashed;
  uint32_t seed;
  unsigned long long *word;   // per vertex: waiting-for count << 32 | colours 0..31 seen
  int32_t *start;             // per vertex: first entry with a lower-priority tail, row-relative
  uint32_t *ext;              // colours of all neighbours, (deg + 32) / 32 words from ext_base
  int32_t *color;
  unsigned long long *queue;  // task words (kFlowEmpty = not yet published)
  unsigned long long qcap;
  unsigned long long *ctr;    // next ticket, tasks published, tasks finished, kFlowCtr apart
  int32_t *status;            // [0] a vertex needs more than kMaxColors, [1] no progress
};

// Tasks of a row with `len` entries from its first lower-priority one on.
__host__ __device__ inline int64_t flow_parts(int64_t len) {
  const int64_t n = (len + kFlowChunk - 1) / kFlowChunk;
  return n < kFlowMaxParts ? n : kFlowMaxParts;
}

// Bitmap words start at floor(ptr / 32) + v: consecutive rows are at least
// floor(deg / 32) + 1 words apart, the words a row of deg entries needs.
__device__ __forceinline__ int64_t flow_ext_base(int64_t rb, int32_t v) { return (rb >> 5) + v; }

__device__ __forceinline__ unsigned long long flow_task(int32_t v, int32_t c, int64_t part) {
  return ((unsigned long long)part << 43) | ((unsigned long long)c << 31) |
         (unsigned long long)(uint32_t)v;
}

// Per row: higher-priority entries (into word's high half, zero on entry) and
// the place of the first lower-priority one (start, INT32_MAX-like on entry:
// any value at or past the row's length means none).  Merge-path tiles, as in
// k_row_sums_tiles: every entry read once with coalesced loads, rows that span
// tiles folded with atomics.
struct FlowTileSmem {
  int32_t cnt[kMergeTile + 1];
  int32_t first[kMergeTile + 1];
  TileRows rows;
};

__global__ void __launch_bounds__(kFlowThreads) k_flow_counts(ColorFlow f, int64_t nnz,
                                                              const int64_t *split_row) {
  extern __shared__ unsigned char smem_raw[];
  FlowTileSmem &sm = *reinterpret_cast<FlowTileSmem *>(smem_raw);
  const int lane = threadIdx.x & 31;
  const int64_t nv = f.nv;
  const int64_t ntiles = merge_tiles(nv, nnz);
  for (int64_t tile = blockIdx.x; tile < ntiles; tile += gridDim.x) {
    const int64_t d0 = tile * (int64_t)kMergeTile;
    const int64_t d1 = min(d0 + (int64_t)kMergeTile, nv + nnz);
    const int64_t i0 = split_row[tile], i1 = split_row[tile + 1];
    const int64_t j0 = d0 - i0, j1 = d1 - i1;
    if (j1 <= j0) continue;  // only row ends (tile-uniform)
    const int64_t ih = min(i1, nv - 1);
    const int nr = (int)(ih - i0 + 1);
    const int ne = (int)(j1 - j0);
    for (int k = threadIdx.x; k < nr; k += kFlowThreads) {
      sm.cnt[k] = 0;
      sm.first[k] = INT32_MAX;
    }
    tile_rows_fill(&sm.rows, f.ptr, i0, nr, j0, ne);
    for (int q0 = 0; q0 < ne; q0 += kFlowThreads) {  // ne is the tile's: warp-uniform
      const int q = q0 + (int)threadIdx.x;
      const bool has = q < ne;
      const int lo = tile_row(&sm.rows, q, ne);
      bool before = false, after = false;
      if (has) {
        const int32_t v = (int32_t)(i0 + lo), u = f.tail[j0 + q];
        if (u != v) {
          before = prio_before(u, v, f.hashed, f.seed);
          after = !before;
        }
      }
      const unsigned m = __match_any_sync(FULL, has ? lo : -1 - lane);
      const unsigned mb = m & __ballot_sync(FULL, before), ma = m & __ballot_sync(FULL, after);
      if (has && lane == __ffs(m) - 1) {
        if (mb) atomicAdd(&sm.cnt[lo], __popc(mb));
        if (ma) atomicMin(&sm.first[lo], q - lane + __ffs(ma) - 1);
      }
    }
    __syncthreads();
    for (int k = threadIdx.x; k < nr; k += kFlowThreads) {
      const int64_t i = i0 + k, rb = f.ptr[i];
      const bool whole = rb >= j0 && i < i1;  // starts and ends in this tile
      const unsigned long long cnt = (unsigned long long)sm.cnt[k] << 32;
      const int32_t first =
          (sm.first[k] == INT32_MAX) ? INT32_MAX : (int32_t)(j0 + sm.first[k] - rb);
      if (whole) {
        f.word[i] = cnt;
        f.start[i] = first;
      } else {
        if (cnt) atomicAdd(&f.word[i], cnt);
        if (first != INT32_MAX) atomicMin(&f.start[i], first);
      }
    }
    __syncthreads();  // the next tile reuses the shared arrays
  }
}

// Warp-collective: every lane publishes parts [p0, n) of its vertex v (n <= p0:
// nothing).  The counter moves once per warp, from lane 0.
__device__ __forceinline__ void flow_publish(const ColorFlow &f, int32_t v, int32_t c, int64_t p0,
                                             int64_t n) {
  const int lane = threadIdx.x & 31;
  const int mine = (int)max((int64_t)0, n - p0);
  int incl = mine;
#pragma unroll
  for (int off = 1; off < 32; off <<= 1) {
    const int y = __shfl_up_sync(FULL, incl, off);
    if (lane >= off) incl += y;
  }
  const int total = __shfl_sync(FULL, incl, 31);
  if (total == 0) return;
  unsigned long long base = 0;
  if (lane == 0) base = atomicAdd(&f.ctr[kFlowCtr], (unsigned long long)total);
  base = __shfl_sync(FULL, base, 0) + (unsigned long long)(incl - mine);
  for (int64_t p = 0; p < mine; ++p)
    if (base + p < f.qcap)
      *(volatile unsigned long long *)&f.queue[base + p] = flow_task(v, c, p0 + p);
}

// The vertices without a higher-priority neighbour: colour 0, their rows the
// first tasks.  The other colours start at -1.
__global__ void __launch_bounds__(256) k_flow_seed(ColorFlow f) {
  const int64_t step = (int64_t)gridDim.x * blockDim.x;
  for (int64_t b = (int64_t)blockIdx.x * blockDim.x; b < f.nv; b += step) {
    const int64_t v = b + threadIdx.x;
    int64_t n = 0;
    if (v < f.nv) {
      const bool ready = (f.word[v] >> 32) == 0;
      f.color[v] = ready ? 0 : -1;
      const int64_t len = f.ptr[v + 1] - f.ptr[v] - f.start[v];
      if (ready && len > 0) n = flow_parts(len);
    }
    flow_publish(f, (int32_t)v, 0, 0, n);
  }
}

// First colour not set in `fb` (colours 0..31) or the vertex's bitmap words
// from word 1 on.  Warp-collective over one vertex; all lanes get the result.
__device__ __forceinline__ int flow_first_free(const ColorFlow &f, int32_t u, int64_t rb,
                                               int64_t deg) {
  const int lane = threadIdx.x & 31;
  const int words = (int)min((deg + 32) / 32, (int64_t)(kMaxColors / 32));
  const uint32_t *bm = f.ext + flow_ext_base(rb, u);
  int first = INT32_MAX;
  for (int q = 1 + lane; q < words; q += 32) {
    const uint32_t fr = ~__ldcg(&bm[q]);
    if (fr) { first = q * 32 + __ffs(fr) - 1; break; }
  }
  first = __reduce_min_sync(FULL, first);
  return first == INT32_MAX ? words * 32 : first;
}

__global__ void __launch_bounds__(kFlowThreads) k_color_flow(ColorFlow f) {
  const int lane = threadIdx.x & 31;
  while (true) {
    // next task: lane 0 polls its ticket's slot
    unsigned long long task = kFlowEmpty;
    if (lane == 0) {
      const unsigned long long t = atomicAdd(&f.ctr[0], 1ull);
      unsigned long long seen = 0, since = 0;
      unsigned pause = 20;
      for (unsigned it = 0;; ++it) {
        if (t < f.qcap) {
          task = *(volatile unsigned long long *)&f.queue[t];
          if (task != kFlowEmpty) break;
        }
        if ((it & 15u) == 15u) {
          // finished first: it never passes the published count, so equal
          // values mean that no task is running or waiting
          const unsigned long long fin = *(volatile unsigned long long *)&f.ctr[2 * kFlowCtr];
          __threadfence();
          const unsigned long long pub = *(volatile unsigned long long *)&f.ctr[kFlowCtr];
          if (fin == pub) break;
          unsigned long long now;
          asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(now));
          if (since == 0 || fin + pub != seen) {
            seen = fin + pub;
            since = now;
          } else if (now - since > kFlowStallNs) {
            atomicExch(&f.status[1], 1);
            break;
          }
          // Tasks come in ticket order: the warps next in line poll, the
          // others sleep longer the more tickets are before theirs.
          const unsigned long long ahead = t >= pub ? t - pub : 0;
          pause = ahead < 16 ? 20u : (ahead < 512 ? 20u + (unsigned)ahead : 512u);
        }
        __nanosleep(pause);
      }
    }
    task = __shfl_sync(FULL, task, 0);
    if (task == kFlowEmpty) return;
    int32_t v = (int32_t)(task & 0x7FFFFFFFull), c = (int32_t)((task >> 31) & 0xFFFull);
    int64_t part = (int64_t)(task >> 43);
    int64_t rb = f.ptr[v], deg = f.ptr[v + 1] - rb, s0 = f.start[v];
    for (int chain = 0;; ++chain) {
      const int64_t len = deg - s0, np = flow_parts(len), per = (len + np - 1) / np;
      const int64_t jb = rb + s0 + part * per, je = min(jb + per, rb + deg);
      const unsigned long long bit = 1ull << (c & 31);
      int32_t nv_ = -1, nc = 0;  // the ready vertex this warp keeps
      int64_t nrb = 0, ndeg = 0, ns0 = 0;
      for (int64_t base = jb; base < je; base += 32) {
        const int32_t u = (base + lane < je) ? f.tail[base + lane] : v;
        const bool low = u != v && prio_before(v, u, f.hashed, f.seed);
        if (c < 32) {
          if (low) atomicOr(&f.word[u], bit);
        } else {
          if (low) {
            const int64_t p0 = f.ptr[u], p1 = f.ptr[u + 1];
            if ((c >> 5) < (p1 - p0 + 32) / 32)  // colours past the degree never block u
              atomicOr(&f.ext[flow_ext_base(p0, u) + (c >> 5)], (uint32_t)bit);
          }
          __threadfence();
        }
        const unsigned long long old = low ? atomicAdd(&f.word[u], 0xFFFFFFFF00000000ull) : 0ull;
        const bool ready = (old >> 32) == 1ull;
        if (!__any_sync(FULL, ready)) continue;
        const int64_t p0 = ready ? f.ptr[u] : 0;
        const int64_t dg = ready ? f.ptr[u + 1] - p0 : 0;
        const int32_t st = ready ? f.start[u] : 0;
        const uint32_t fr = ~(uint32_t)old;
        int cu = fr ? __ffs(fr) - 1 : 0;
        unsigned full = __ballot_sync(FULL, ready && fr == 0);
        if (full) __threadfence();  // the bitmap words ordered before the count
        while (full) {  // warp-uniform
          const int src = __ffs(full) - 1;
          full &= full - 1;
          const int x = flow_first_free(f, __shfl_sync(FULL, u, src), __shfl_sync(FULL, p0, src),
                                        __shfl_sync(FULL, dg, src));
          if (lane == src) cu = x;
        }
        if (cu >= kMaxColors) {
          atomicExch(&f.status[0], 1);
          cu = kMaxColors - 1;
        }
        if (ready) f.color[u] = cu;
        const int64_t n = (ready && dg > st) ? flow_parts(dg - st) : 0;
        const unsigned pm = __ballot_sync(FULL, n > 0);
        int64_t first = 0;
        if (base + 32 >= je && chain < kFlowChain && pm) {
          // keep the first ready vertex with a row to send
          const int src = __ffs(pm) - 1;
          nv_ = __shfl_sync(FULL, u, src);
          nc = __shfl_sync(FULL, cu, src);
          nrb = __shfl_sync(FULL, p0, src);
          ndeg = __shfl_sync(FULL, dg, src);
          ns0 = __shfl_sync(FULL, st, src);
          if (lane == src) first = 1;
        }
        flow_publish(f, u, cu, first, n);
      }
      if (nv_ < 0) break;
      v = nv_; c = nc; part = 0;
      rb = nrb; deg = ndeg; s0 = ns0;
    }
    __syncwarp();
    if (lane == 0) {
      __threadfence();  // this task's publications before its end
      atomicAdd(&f.ctr[2 * kFlowCtr], 1ull);
    }
  }
}

}  // namespace glv
