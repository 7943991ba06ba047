// Ordered accumulation (verify mode on non-integral weights): every
// per-community sum is folded in CSR order, every community total in vertex
// order, as the reference's one-thread loop adds them.  A colour class is two
// launches, the rows of all degree bins and the totals; bins of many short rows
// (kOrdOwnItems) have a launch of their own.
//
// What bounds it: latency, launch by launch.  With a launch per degree bin, long
// rows walked by one warp (a round of 32 entries about 1 us), and a radix sort
// of several kernels for the totals of each class, a class of R-MAT 15 took
// 118 us, of its coarse level 90; now 20 (a run 126 -> 47.5 ms).
//
// Long rows: the block loads kOrdChunk entries and their communities into
// shared memory, then warp w lists, in order, the entries whose community hashes
// to it and adds them: every community belongs to one warp, so its sum is
// sequential and the table needs no atomic adds, while eight communities' sums
// advance at once.
#pragma once

#include "phase_kernels.cuh"
#include "sweep.cuh"

namespace glv {

constexpr int kOrdThreads = 256;
constexpr int kOrdWarps = kOrdThreads / 32;
constexpr int kOrdChunk = 512;
constexpr int kOrdTableCap = 8192;      // table_cap(4095): rows up to the block bin
constexpr int kOrdWarpCap = 256;        // table_cap(127)
// Rows of a bin for each warp of k_sweep_ordered from which the bin has a launch of
// its own, with 64 warps per SM instead of 16: a step of all vertices (the basic
// driver, 1M vertices of 20 entries) 93.8 -> 73.3 ms a run (75.5 with a launch per
// bin everywhere), 300k 28.6 -> 23.9; limits of 1 to 8 measure the same, 16 takes 3 %
// more.  Below it the launches cost more than the warps: classes of R-MAT 15.
constexpr int64_t kOrdOwnItems = 2;

struct OrderedShared {
  int32_t c[kOrdChunk];
  double w[kOrdChunk];
  uint32_t self[kOrdChunk / 32];        // entries that are self-loops
  uint32_t mask[kOrdWarps][kOrdChunk / 32];  // entries of each warp
  uint16_t list[kOrdWarps][kOrdChunk];  // the same in order
  int any_self;
};
constexpr int kOrdSmem =
    kOrdTableCap * (int)(sizeof(double) + sizeof(int32_t)) + (int)sizeof(OrderedShared);
static_assert(kOrdWarps * kOrdWarpCap <= kOrdTableCap, "warp tables tile the block table");
static_assert(kOrdWarps * (kOrdChunk / 32) <= kOrdThreads && kOrdChunk / 32 <= 32,
              "one thread per mask word, one lane per word of a warp");

// One row by the whole block; keys/vals are the block's shared table or, for
// hub rows, a global one (written by this block alone).
__device__ __forceinline__ void ordered_row(const SweepArgs &a, int64_t pos, int32_t *keys,
                                            double *vals, OrderedShared *sh, double *s_g,
                                            int32_t *s_c) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int32_t v = a.members[pos];
  const int64_t rb = a.ptr[v], re = a.ptr[v + 1];
  const uint32_t cap = table_cap(re - rb), mask = cap - 1;
  for (uint32_t s = threadIdx.x; s < cap; s += kOrdThreads) { keys[s] = -1; vals[s] = 0.0; }
  constexpr int kWords = kOrdChunk / 32;
  if (threadIdx.x < kWords) sh->self[threadIdx.x] = 0u;
  if (threadIdx.x < kOrdWarps * kWords) sh->mask[threadIdx.x / kWords][threadIdx.x % kWords] = 0u;
  if (threadIdx.x == 0) sh->any_self = 0;
  __syncthreads();
  const int32_t own = a.C[v];
  if (threadIdx.x == 0) keys[hash_slot(own, mask)] = own;
  double self_loop = 0.0;  // thread 0's
  for (int64_t b = rb; b < re; b += kOrdChunk) {
    const int n = (int)min((int64_t)kOrdChunk, re - b);
    for (int i = threadIdx.x; i < n; i += kOrdThreads) {
      const int32_t t = __ldcs(&a.tail[b + i]);
      sh->w[i] = __ldcs(&a.w[b + i]);
      const int32_t c = a.C[t];
      sh->c[i] = c;
      atomicOr(&sh->mask[(mix32((uint32_t)c) >> 8) & (kOrdWarps - 1)][i >> 5], 1u << (i & 31));
      if (t == v) {
        atomicOr(&sh->self[i >> 5], 1u << (i & 31));
        sh->any_self = 1;
      }
    }
    __syncthreads();
    // this warp's entries in order: lane q expands word q of its mask
    uint32_t word = (lane < kWords) ? sh->mask[warp][lane] : 0u;
    int at = __popc(word);
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int y = __shfl_up_sync(FULL, at, o);
      if (lane >= o) at += y;
    }
    const int cnt = __shfl_sync(FULL, at, 31);
    at -= __popc(word);
    for (; word; word &= word - 1) sh->list[warp][at++] = (uint16_t)(32 * lane + __ffs(word) - 1);
    if (lane < kWords) sh->mask[warp][lane] = 0u;
    __syncwarp();
    for (int r = 0; r < cnt; r += 32) {
      const int32_t c = (r + lane < cnt) ? sh->c[sh->list[warp][r + lane]] : -1;
      const unsigned m = __match_any_sync(FULL, c);
      if (c >= 0 && lane == __ffs(m) - 1) {
        const uint32_t slot = table_slot(keys, mask, c);
        double acc = vals[slot];
        for (unsigned rem = m; rem; rem &= rem - 1)
          acc = __dadd_rn(acc, sh->w[sh->list[warp][r + __ffs(rem) - 1]]);
        vals[slot] = acc;
      }
      __syncwarp();
    }
    if (threadIdx.x == 0 && sh->any_self) {
      for (int q = 0; q < kWords; ++q) {
        for (uint32_t rem = sh->self[q]; rem; rem &= rem - 1)
          self_loop = __dadd_rn(self_loop, sh->w[32 * q + __ffs(rem) - 1]);
        sh->self[q] = 0u;
      }
      sh->any_self = 0;
    }
    __syncthreads();
  }
  if (threadIdx.x == 0) s_g[0] = self_loop;
  __syncthreads();
  self_loop = s_g[0];
  __syncthreads();
  const double degree = a.vDeg[v];
  const double own_w = vals[hash_slot(own, mask)];
  const double eix = __dsub_rn(own_w, self_loop);
  const double ax = __dsub_rn(a.cDeg[own], degree);
  double g = 0.0;
  int32_t bc = INT32_MAX;
  scan_table(a, keys, vals, threadIdx.x, cap, kOrdThreads, own, eix, ax, degree, cst_of(a, v), g,
             bc);
  warp_argmax(g, bc);
  if (lane == 0) { s_g[warp] = g; s_c[warp] = bc; }
  __syncthreads();
  if (threadIdx.x == 0) {
    for (int k = 1; k < kOrdWarps; ++k)
      if (better(s_g[k], s_c[k], g, bc)) { g = s_g[k]; bc = s_c[k]; }
    emit_decision(a, pos, v, own, finish_choice(a, own, g, bc), degree, own_w, g);
  }
  __syncthreads();
}

// The member positions of each degree bin that a launch decides.
struct BinRanges {
  int64_t lo[NBINS], hi[NBINS];
};

// Blocks [0, nlong) take the rows above the warp bin (longest bins first), the
// others the shorter rows, a warp at a time.
__global__ void __launch_bounds__(kOrdThreads) k_sweep_ordered(SweepArgs a, BinRanges r,
                                                               int nlong) {
  extern __shared__ unsigned char smem_raw[];
  __shared__ double s_g[32];
  __shared__ int32_t s_c[32];
  double *vals = reinterpret_cast<double *>(smem_raw);
  int32_t *keys = reinterpret_cast<int32_t *>(vals + kOrdTableCap);
  OrderedShared *sh = reinterpret_cast<OrderedShared *>(keys + kOrdTableCap);
  if ((int)blockIdx.x < nlong) {
    int64_t k = blockIdx.x;  // number of this block's next row, longest bins first
    for (int b = BIN_HUB; b >= BIN_T128; --b) {
      const int64_t n = r.hi[b] - r.lo[b];
      for (; k < n; k += nlong) {
        const int64_t pos = r.lo[b] + k;
        if (b == BIN_HUB)
          ordered_row(a, pos, a.hub_keys + a.hub_off[pos], a.hub_vals + a.hub_off[pos], sh, s_g,
                      s_c);
        else
          ordered_row(a, pos, keys, vals, sh, s_g, s_c);
      }
      k -= n;
    }
    return;
  }
  const int warp = threadIdx.x >> 5;
  const int64_t nw = (int64_t)(gridDim.x - nlong) * kOrdWarps;
  int64_t k = (int64_t)warp * (gridDim.x - nlong) + (blockIdx.x - nlong);
  auto small = [&](int b, int vpw, auto item) {
    const int64_t n = (r.hi[b] - r.lo[b] + vpw - 1) / vpw;
    for (; k < n; k += nw) item(r.lo[b] + vpw * k, r.hi[b]);
    k -= n;
  };
  small(BIN_WARP, 1, [&](int64_t pos, int64_t) {
    warp_table_vertex(a, pos, keys + warp * kOrdWarpCap, vals + warp * kOrdWarpCap);
  });
  small(BIN_G32, 1, [&](int64_t pos, int64_t end) { small_item<32>(a, pos, end); });
  small(BIN_G16, 2, [&](int64_t pos, int64_t end) { small_item<16>(a, pos, end); });
  small(BIN_G8, 4, [&](int64_t pos, int64_t end) { small_item<8>(a, pos, end); });
  small(BIN_G4, 8, [&](int64_t pos, int64_t end) { small_item<4>(a, pos, end); });
}

// Community totals after a class of at most kOrdApplyMax members, in one block:
// the moves' records (community, vertex) sorted in shared memory, each
// community's deltas folded from 0.0 in vertex order (k_delta_records and
// k_fold_deltas with a device-wide sort do the same for larger classes; that is
// about eight launches, 25 us a class against 7).
constexpr int kOrdApplyThreads = 1024;
constexpr int64_t kOrdApplyMax = 4096;
constexpr int kOrdApplyRecs = 2 * (int)kOrdApplyMax;
constexpr int kOrdApplySmem = kOrdApplyRecs * (int)(sizeof(uint64_t) + sizeof(double));

__global__ void __launch_bounds__(kOrdApplyThreads) k_apply_ordered(
    int64_t begin, int64_t end, const int32_t *members, const int32_t *move_old,
    const int32_t *move_new, const double *vDeg, double *cDeg, int32_t *cSize) {
  extern __shared__ unsigned char smem_raw[];
  uint64_t *key = reinterpret_cast<uint64_t *>(smem_raw);  // community, vertex, leaving
  double *d = reinterpret_cast<double *>(key + kOrdApplyRecs);
  __shared__ int s_n;
  if (threadIdx.x == 0) s_n = 0;
  __syncthreads();
  for (int64_t pos = begin + threadIdx.x; pos < end; pos += kOrdApplyThreads) {
    const int32_t o = move_old[pos];
    if (o < 0) continue;
    const uint64_t v = (uint32_t)members[pos], n = (uint32_t)move_new[pos];
    const int at = atomicAdd(&s_n, 2);
    key[at] = (n << 32) | (v << 1);
    key[at + 1] = ((uint64_t)(uint32_t)o << 32) | (v << 1) | 1u;
  }
  __syncthreads();
  const int n = s_n;
  if (n == 0) return;
  int size = 2;
  while (size < n) size <<= 1;
  for (int i = n + threadIdx.x; i < size; i += kOrdApplyThreads) key[i] = ~0ull;
  __syncthreads();
  for (int k = 2; k <= size; k <<= 1) {  // bitonic: ascending
    for (int j = k >> 1; j > 0; j >>= 1) {
      for (int i = threadIdx.x; i < size; i += kOrdApplyThreads) {
        const int p = i ^ j;
        if (p <= i) continue;
        const uint64_t x = key[i], y = key[p];
        if ((x > y) == ((i & k) == 0)) { key[i] = y; key[p] = x; }
      }
      __syncthreads();
    }
  }
  for (int i = threadIdx.x; i < n; i += kOrdApplyThreads) {
    const uint64_t x = key[i];
    const double dg = vDeg[(uint32_t)x >> 1];
    d[i] = (x & 1) ? -dg : dg;
  }
  __syncthreads();
  for (int i = threadIdx.x; i < n; i += kOrdApplyThreads) {
    const uint32_t c = (uint32_t)(key[i] >> 32);
    if (i > 0 && (uint32_t)(key[i - 1] >> 32) == c) continue;
    double s = 0.0;
    int32_t cnt = 0;
    for (int j = i; j < n && (uint32_t)(key[j] >> 32) == c; ++j) {
      s = __dadd_rn(s, d[j]);
      cnt += (key[j] & 1) ? -1 : 1;
    }
    cDeg[c] = __dadd_rn(cDeg[c], s);
    cSize[c] += cnt;
  }
}

}  // namespace glv
