// One Louvain iteration in one cooperative launch (parallel-accumulation modes).
//
// The colour classes of an iteration depend on each other (a class decides
// against the community totals left by the classes before it), and R-MAT-like
// graphs need hundreds of classes, most of them small and made of high-degree
// vertices.  Launching a few kernels per class leaves the GPU waiting on
// launches and on the single largest row of each class.  Here every block of
// a persistent grid takes part in every class:
//   stage 1  hub rows on thread-block clusters (one table over the shared
//            memory of a cluster's blocks) or, without clusters, hub chunks
//            and partitions (hub.cuh); rows of 1024..4095 entries per
//            block; rows of 128..1023 entries per 128-thread team (shared
//            tables); then warp items (rows <= 32 entries, and 33..127-entry
//            rows with a per-warp shared table)                  -> grid barrier
//            (a hub whose last chunk's block does not decide it is decided by
//            partition tasks of the same queue)
//   stage 2  community totals += the class's deltas             -> grid barrier
// (stage 2 after the class's last sublevel), then the modularity pass of the
// iteration.
#pragma once

#include <cooperative_groups.h>

#include "phase_kernels.cuh"
#include "hub.cuh"
#include "rows.cuh"
#include "sweep.cuh"

namespace glv {

// 32-bit: member positions and work items stay below 2^31.
struct StepDesc {
  int32_t seg[NBINS + 1];  // member positions of each degree bin
  int32_t hub_chunk[2];    // hub chunks
  int32_t hub_segs[2];     // hub partitions
  int32_t apply[2];        // member range whose deltas are applied after this step
  int32_t cls;             // colour class of the step
  int32_t ctask[2];        // hub tasks on thread-block clusters (cluster_row_tasks)
};
constexpr int kStepWords = sizeof(StepDesc) / sizeof(int32_t);

struct IterArgs {
  SweepArgs a;
  HubWork h;
  const StepDesc *steps;
  int nsteps;
  int jacobi;              // 1: Q on the state before the moves, totals updated after
  int64_t nv;
  const int32_t *C_mod;    // communities the modularity pass compares (colour phases)
  const double *own_w_mod; // Jacobi phases: Counter[own] per vertex
  double *part_e, *part_a; // per 256-vertex tile partials
  const double *cst;       // {constant, 2m}
  double *mod_out;         // {Q, e_xx, a2_x}
  double *cDeg;
  int32_t *cSize;
  uint64_t *trace;         // optional: globaltimer at each barrier, 4 per step + 2
  unsigned *task_ctr;      // per step: next block, team and cluster task (zero at launch)
  int *moved;              // per colour class: some vertex moved (zero at launch)
  const int32_t *kept;     // gated or batched sweeps: k_steps_kept's flags (NULL = all steps run)
  int64_t nnz;
  const int64_t *split_row;   // merge-path tile boundaries of the level
  // batches of graphs: per-graph modularity sums instead of one Q
  const int32_t *gid;
  double *gacc;
  // The internal-weight term e_xx: 0 = a full pass over the level (stored in
  // exx_state); 1 = exx_state plus this sweep's moves' changes (a.exx_delta),
  // with only sum cDeg^2 taken in full; 2 = both, Q from the carried value
  // and the full pass's e_xx in mod_out[3] (a self-check)
  int exx_mode;
  double *exx_state;
  // Carried e_xx with classes that are not independent sets (core batches):
  // the CSR entries (member slot of u, member slot of t, w) whose two ends
  // run in the same step.  Each move's change 2 (e_iy - e_ix) assumes its
  // neighbours stay; for such an entry whose two ends both moved the carried
  // sum is corrected by w ([y_u == y_t] + [x_u == x_t] - [y_u == x_t] - [x_u == y_t]).
  const int32_t *pair_u, *pair_t;
  const double *pair_w;
  int64_t npairs;
};

// Gated or batched sweeps: kept[s] & 2 when some member of step s is evaluated,
// kept[s] & 1 at the last step of a class when some member of the class is
// (kept must be zero on entry).  With per_class a class runs all its steps or
// none.  Member positions are strided over the grid; a position's step is found
// by binary search in step_begin; [step_first, step_last] are its class's.
__global__ void k_steps_kept(int nsteps, const int64_t *step_begin, const int32_t *step_first,
                             const int32_t *step_last, int per_class, int64_t nmem,
                             const int32_t *members, const uint8_t *skip, int32_t *kept) {
  for (int64_t pos = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; pos < nmem;
       pos += (int64_t)gridDim.x * blockDim.x) {
    if (skip[members[pos]]) continue;
    int lo = 0, hi = nsteps - 1;  // last step starting at or before pos
    while (lo < hi) {
      const int mid = (lo + hi + 1) >> 1;
      if (step_begin[mid] <= pos) lo = mid; else hi = mid - 1;
    }
    const int last = step_last[lo];
    for (int q = per_class ? step_first[lo] : lo; q <= (per_class ? last : lo); ++q)
      if (!(kept[q] & 2)) atomicOr(&kept[q], 2);
    if (!(kept[last] & 1)) atomicOr(&kept[last], 1);
  }
}

__device__ __forceinline__ uint64_t global_ns() {
  uint64_t t;
  asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
  return t;
}

#define GLV_TRACE(slot)                                                  \
  do {                                                                   \
    if (p.trace && blockIdx.x == 0 && threadIdx.x == 0) p.trace[slot] = global_ns(); \
  } while (0)

// Debug traces, 4 slots per step after the 4 per step + 2: the latest time
// over the grid at which a queue of step s ran dry (q = 0 block queue, 1 team
// queue, 2 warp items, 3 cluster tasks).
#define GLV_QTRACE(s, q, cond)                                                       \
  do {                                                                               \
    if (p.trace && (cond))                                                           \
      atomicMax((unsigned long long *)&p.trace[4 * p.nsteps + 2 + 4 * (s) + (q)],    \
                (unsigned long long)global_ns());                                    \
  } while (0)

constexpr int kPersistThreads = 512;
constexpr int kPersistTableCap = 8192;  // BIN_BLOCK rows: degree <= 4095
constexpr int kPersistWarpCap = 256;    // warp-table rows: degree <= 127
constexpr int kTeamThreads = 128;      // team of the 128..1023-entry rows
constexpr int kTeamCap = 2048;         // its table: table_cap(1023)
constexpr int kPersistFill = 4096;      // filled-slot entries of a block: BIN_BLOCK rows
// table values, table keys, filled slots
constexpr size_t kPersistTableBytes =
    (size_t)kPersistTableCap * (sizeof(double) + sizeof(int32_t));
constexpr size_t kPersistSmem = kPersistTableBytes + kPersistFill * sizeof(uint16_t);
static_assert(kPersistThreads / kTeamThreads * kTeamCap == kPersistTableCap,
              "team tables tile the block table");
static_assert(kTeamThreads / 32 * kPersistWarpCap <= kTeamCap,
              "warp tables tile their team's table");
static_assert(kPersistSmem >= sizeof(MergeSmem), "merge tiles must fit");
static_assert(kPersistTableCap >= kClusterBlockSlots, "a cluster table part must fit");
static_assert(kPersistTableCap == kHubTableCap && kPersistFill >= kHubList &&
                  kPersistThreads == kHubThreads,
              "hub tasks use the block's table and list");
static_assert(kPersistTableBytes >= (size_t)(kPersistThreads / 32) * kPersistWarpCap *
                                        (sizeof(double) + sizeof(int32_t)),
              "warp tables must fit in the block-table region");
static_assert(kPersistFill / (kPersistThreads / kTeamThreads) >= 1024 && 127 < 4 * 32 &&
                  kPersistFill >= 4096,
              "every entry of a row has a filled-slot entry");

// Community totals += the deltas the sweep accumulated (see k_apply_deltas).
// The whole stage sits between two grid barriers, so what counts is its chain
// of dependent accesses: a position's records load together, and both
// communities' claims and totals are in flight together (one claim at a time,
// each an L2 round trip, took 4.3 us a step on R-MAT 20's second level; now
// 2.2).  Only the thread that claimed a nonzero delta writes a total, and
// stage 1 is over, so a total read beside the claim is still current.
__device__ __forceinline__ void apply_deltas_range(const IterArgs &p, int b, int e, int gt,
                                                   int ngt) {
  for (int pos = b + gt; pos < e; pos += ngt) {
    const int32_t o = p.a.move_old[pos], n = p.a.move_new[pos];
    if (p.a.defer_c) {
      // deferred decisions: moves, and isolated vertices leaving every community
      if (o >= 0 || n < 0) p.a.C[p.a.members[pos]] = n;
    }
    if (o < 0) continue;
    const unsigned long long dn = atomicExch((unsigned long long *)&p.a.dDeg[n], 0ull);
    const unsigned long long od = atomicExch((unsigned long long *)&p.a.dDeg[o], 0ull);
    const int32_t sn = atomicExch(&p.a.dSize[n], 0), so = atomicExch(&p.a.dSize[o], 0);
    const double cn = __ldcg(&p.cDeg[n]), co = __ldcg(&p.cDeg[o]);
    const int32_t zn = __ldcg(&p.cSize[n]), zo = __ldcg(&p.cSize[o]);
    if (dn) p.cDeg[n] = __dadd_rn(cn, __longlong_as_double((long long)dn));
    if (od) p.cDeg[o] = __dadd_rn(co, __longlong_as_double((long long)od));
    if (sn) p.cSize[n] = zn + sn;
    if (so) p.cSize[o] = zo + so;
  }
}

// Q from the per-block partials (block 0, all threads).
__device__ __forceinline__ void modularity_fold(const IterArgs &p, int64_t nparts, double *sh) {
  double e = 0.0, a = 0.0, d = 0.0;
  const int64_t per = (nparts + blockDim.x - 1) / blockDim.x;
  const int64_t b = threadIdx.x * per, en = min(nparts, b + per);
  for (int64_t i = b; i < en; ++i) {
    e = __dadd_rn(e, p.part_e[i]);
    a = __dadd_rn(a, p.part_a[i]);
    if (p.exx_mode == 2) d = __dadd_rn(d, p.a.exx_delta[i]);
  }
  e = block_sum<kPersistThreads>(e, sh);
  a = block_sum<kPersistThreads>(a, sh);
  if (p.exx_mode == 2) d = block_sum<kPersistThreads>(d, sh);
  if (threadIdx.x == 0) {
    const double c = p.cst[0];
    double exx = e;  // mode 0: the full pass
    if (p.exx_mode == 1) exx = __dadd_rn(p.exx_state[0], e);  // e holds the moves' changes
    if (p.exx_mode == 2) {
      exx = __dadd_rn(p.exx_state[0], d);
      p.mod_out[3] = e;
    }
    if (p.exx_state) p.exx_state[0] = exx;
    p.mod_out[0] = __dsub_rn(__dmul_rn(exx, c), __dmul_rn(__dmul_rn(a, c), c));
    p.mod_out[1] = exx;
    p.mod_out[2] = a;
  }
}

// threadIdx.x read anew: indexes derived from it are not kept (and spilled)
// across a step's tasks, whose reloads after a grid barrier miss in L1.
__device__ __forceinline__ int thread_id() {
  int t;
  asm volatile("mov.u32 %0, %%tid.x;" : "=r"(t));
  return t;
}

// kClusters: the instantiation launched with a cluster dimension, which runs
// the steps' cluster tasks; the other one leaves that code out entirely (its
// registers go to the other paths).
template <bool kClusters>
__global__ void __launch_bounds__(kPersistThreads, 2) k_sweep_iteration(IterArgs p) {
  cg::grid_group grid = cg::this_grid();
  extern __shared__ unsigned char smem_raw[];
  __shared__ double s_self[32], s_own[32], s_g[32], sh[32];
  __shared__ int32_t s_c[32];
  // shared table region: one 8192-slot table (block tasks), four 2048-slot
  // team tables, or a 256-slot table per warp inside its team's table; the
  // filled slots likewise: the block's, a quarter of it per team, 128 of that
  // per warp
  double *const tvals = reinterpret_cast<double *>(smem_raw);
  int32_t *const tkeys = reinterpret_cast<int32_t *>(tvals + kPersistTableCap);
  uint16_t *const fill = reinterpret_cast<uint16_t *>(smem_raw + kPersistTableBytes);
  // tables are empty between tasks; every task empties the slots it filled
  for (int q = threadIdx.x; q < kPersistTableCap; q += kPersistThreads) {
    tkeys[q] = -1;
    tvals[q] = 0.0;
  }
  __syncthreads();
  GLV_TRACE(4 * p.nsteps);
  // next task of the block and team queues, by task parity: the following
  // task is fetched when a task starts and published after it ends
  __shared__ int s_task[2];
  __shared__ int s_team_task[kPersistThreads / kTeamThreads][2];
  __shared__ HubShared s_hub;
  __shared__ ClusterShared s_cluster;
  // this block's slot of the moves' e_xx changes (only this block writes it)
  if (p.a.exx_delta && threadIdx.x == 0) p.a.exx_delta[blockIdx.x] = 0.0;
  // The step's description in shared memory, loaded a step ahead: its values
  // cost no registers across the tasks and no L2 round trip after a barrier.
  // Three of them, so that a step's may be read until the next step's barrier.
  __shared__ StepDesc s_step[3];
  __shared__ int s_keep[3];
  if (threadIdx.x < kStepWords && p.nsteps > 0)
    reinterpret_cast<int32_t *>(&s_step[0])[threadIdx.x] =
        reinterpret_cast<const int32_t *>(&p.steps[0])[threadIdx.x];
  if (threadIdx.x == kStepWords && p.nsteps > 0) s_keep[0] = p.kept ? p.kept[0] : 3;
  if (threadIdx.x == 0) block_moved() = 0;
  __syncthreads();
  for (int s = 0, cur = 0; s < p.nsteps; ++s, cur = (cur == 2) ? 0 : cur + 1) {
    const StepDesc &st = s_step[cur];
    {
      const int nx = (cur == 2) ? 0 : cur + 1, t = thread_id();
      if (t < kStepWords && s + 1 < p.nsteps)
        reinterpret_cast<int32_t *>(&s_step[nx])[t] =
            reinterpret_cast<const int32_t *>(&p.steps[s + 1])[t];
      if (t == kStepWords && s + 1 < p.nsteps) s_keep[nx] = p.kept ? p.kept[s + 1] : 3;
    }
    // a step with nothing to evaluate is skipped (no work, no grid barrier)
    if (!(s_keep[cur] & 2)) {
      __syncthreads();
    } else {
    // Stage 1 in three parts, each from its own queue: (A) hub chunks and
    // rows of 1024..4095 entries, whole blocks with an 8192-slot table;
    // (B) rows of 128..1023 entries, 128-thread teams (four per block, each
    // fetching its own rows, 2048-slot tables); (C) warp items (rows of up to
    // 32 entries, several per warp; rows of 33..127 entries, one per warp),
    // item t to warp t mod (warps of the grid), in the warp's slice of its
    // team's table region.
    const int t_hub = st.hub_chunk[1] - st.hub_chunk[0];
    const int t_blk = st.seg[BIN_BLOCK + 1] - st.seg[BIN_BLOCK];
    const int t_seg = st.hub_segs[1] - st.hub_segs[0];
    const int t_ct = kClusters ? st.ctask[1] - st.ctask[0] : 0;
    if constexpr (kClusters) if (t_ct > 0) {
      // hub rows on clusters (launches with a cluster dimension): every block
      // of a cluster takes part in every task of its cluster
      cluster_row_tasks(p.a, p.h, st.ctask[0], t_ct, &p.task_ctr[3 * s + 2],
                        tkeys, tvals, &s_cluster, s_g, s_c);
      GLV_QTRACE(s, 3, threadIdx.x == 0);
    }
    // The rows of 128..1023 entries of a step with few of them (at most
    // gridDim / 4, and no more than the blocks left) go to whole blocks: 1 or 2
    // rounds instead of up to 8.  With more, four rows per block are better:
    // R-MAT 20, whose steps hold 50 to 800, took 3% longer with as many on
    // blocks as the grid could take, while steps of a row or two (the last
    // levels of a planted partition) go from 12.3 to 9.5 us.
    const int nteam = st.seg[BIN_T256 + 1] - st.seg[BIN_T128];
    const int n_up = (4 * nteam <= (int)gridDim.x &&
                      nteam + t_hub + t_blk + t_seg <= (int)gridDim.x) ? nteam : 0;
    if (t_hub + t_blk + n_up + t_seg > 0) {
      // hub chunks, block rows, team rows, then hub partitions (which wait for
      // their hub's chunks: every chunk is handed out before any partition)
      unsigned *ctr = &p.task_ctr[3 * s];
      if (thread_id() == 0) s_task[0] = (int)atomicAdd(ctr, 1u);
      __syncthreads();
      for (unsigned it = 0;; ++it) {
        int t = s_task[it & 1];
        if (t >= t_hub + t_blk + n_up + t_seg) break;
        const int nxt = (thread_id() == 0) ? (int)atomicAdd(&p.task_ctr[3 * s], 1u) : 0;
        if (t < t_hub) {
          hub_chunk_task(p.a, p.h, st.hub_chunk[0] + t, tkeys, tvals, fill, &s_hub, s_g, s_c);
        } else if ((t -= t_hub) < t_blk + n_up) {
          const int n256 = st.seg[BIN_T256 + 1] - st.seg[BIN_T256];
          int pos = st.seg[BIN_BLOCK] + t;
          if ((t -= t_blk) >= 0)
            pos = (t < n256) ? st.seg[BIN_T256] + t : st.seg[BIN_T128] + (t - n256);
          row_vertex<512>(p.a, pos, tkeys, tvals, fill, 0, s_self, s_own, s_g, s_c);
        } else {
          hub_part_task(p.a, p.h, st.hub_segs[0] + (t - t_blk - n_up), tkeys, tvals, fill, &s_hub,
                        s_g, s_c);
        }
        if (thread_id() == 0) s_task[(it + 1) & 1] = nxt;
        __syncthreads();
      }
      GLV_QTRACE(s, 0, threadIdx.x == 0);
    }
    if (nteam > n_up) {
      const int team = thread_id() / kTeamThreads, tt = thread_id() % kTeamThreads;
      if (tt == 0) s_team_task[team][0] = n_up + (int)atomicAdd(&p.task_ctr[3 * s + 1], 1u);
      team_sync<128>(team);
      for (unsigned it = 0;; ++it) {
        const int t = s_team_task[team][it & 1];
        // the longer rows (the T256 bin, after the T128 bin in member order) first
        const int n256 = st.seg[BIN_T256 + 1] - st.seg[BIN_T256];
        if (t >= nteam) break;
        const int nxt = (tt == 0) ? n_up + (int)atomicAdd(&p.task_ctr[3 * s + 1], 1u) : 0;
        const int pos = (t < n256) ? st.seg[BIN_T256] + t : st.seg[BIN_T128] + (t - n256);
        row_vertex<128>(p.a, pos, tkeys + team * kTeamCap, tvals + team * kTeamCap,
                        fill + team * (kPersistFill * kTeamThreads / kPersistThreads), team,
                        s_self + 4 * team, s_own + 4 * team, s_g + 4 * team, s_c + 4 * team);
        if (tt == 0) s_team_task[team][(it + 1) & 1] = nxt;
        team_sync<128>(team);
      }
      GLV_QTRACE(s, 1, tt == 0);
    }
    {
      // warps numbered across blocks first: a step with few warp items spreads over SMs
      const int warp = thread_id() >> 5, ngw = gridDim.x * (kPersistThreads / 32);
      const int gwi = warp * gridDim.x + blockIdx.x;
      int k = small_rows<4>(p.a, st.seg[0], st.seg[1], gwi, ngw);
      k = small_rows<8>(p.a, st.seg[1], st.seg[2], k, ngw);
      k = small_rows<16>(p.a, st.seg[2], st.seg[3], k, ngw);
      k = small_rows<32>(p.a, st.seg[3], st.seg[4], k, ngw);
      for (int pos = st.seg[4] + k; pos < st.seg[5]; pos += ngw)
        row_vertex<32>(p.a, pos, tkeys + (warp >> 2) * kTeamCap + (warp & 3) * kPersistWarpCap,
                       tvals + (warp >> 2) * kTeamCap + (warp & 3) * kPersistWarpCap,
                       fill + (warp >> 2) * (kPersistFill * kTeamThreads / kPersistThreads) +
                           (warp & 3) * 128,
                       0, nullptr, nullptr, nullptr, nullptr);
      GLV_QTRACE(s, 2, (threadIdx.x & 31) == 0);
    }
    __syncthreads();
    if (thread_id() == 0 && block_moved()) {
      p.moved[st.cls] = 1;
      block_moved() = 0;
    }
    grid.sync();
    GLV_TRACE(4 * s);
    }
    // A class that moved nothing has no totals to update (in a phase's first
    // sweep the apply stage also takes isolated vertices out of C).
    if (!p.jacobi && st.apply[1] > st.apply[0] && (s_keep[cur] & 1) &&
        (p.a.iter <= 1 || __ldcg(&p.moved[st.cls]))) {
      apply_deltas_range(p, st.apply[0], st.apply[1], blockIdx.x * kPersistThreads + thread_id(),
                         gridDim.x * kPersistThreads);
      grid.sync();
      GLV_TRACE(4 * s + 3);
    }
  }
  const int gt = blockIdx.x * kPersistThreads + threadIdx.x, ngt = gridDim.x * kPersistThreads;
  {
    // merge-path tiles, one partial pair per block
    double ex = 0.0, a2 = 0.0;
    const int64_t ntiles = merge_tiles(p.nv, p.nnz);
    MergeSmem *msm = reinterpret_cast<MergeSmem *>(smem_raw);
    __syncthreads();  // stage-1 tables in the same shared memory are done
    if (p.exx_mode >= 1 && p.npairs > 0) {
      // same-step entries whose two ends both moved (see IterArgs::pair_u)
      double corr = 0.0;
      for (int64_t k = gt; k < p.npairs; k += ngt) {
        const int32_t pu = p.pair_u[k], pt = p.pair_t[k];
        const int32_t xu = p.a.move_old[pu], xt = p.a.move_old[pt];
        if (xu < 0 || xt < 0) continue;
        const int32_t yu = p.a.move_new[pu], yt = p.a.move_new[pt];
        const int f = (yu == yt) + (xu == xt) - (yu == xt) - (xu == yt);
        if (f != 0) corr = __dadd_rn(corr, __dmul_rn((double)f, p.pair_w[k]));
      }
      corr = block_sum<kPersistThreads>(corr, sh);
      if (threadIdx.x == 0 && corr != 0.0) p.a.exx_delta[blockIdx.x] += corr;
      __syncthreads();
    }
    if (p.exx_mode == 1) {
      // e_xx is carried: only a2 = sum of cDeg^2 over the level
      for (int64_t c = gt; c < p.nv; c += ngt) a2 = __dadd_rn(a2, __dmul_rn(p.cDeg[c], p.cDeg[c]));
      if (threadIdx.x == 0) ex = p.a.exx_delta[blockIdx.x];
    } else if (p.gid) {
      // contiguous tile ranges, so a thread's running pair changes graph rarely
      GraphAcc acc;
      const int64_t tb = ntiles * blockIdx.x / gridDim.x;
      const int64_t te = ntiles * (blockIdx.x + 1) / gridDim.x;
      for (int64_t tile = tb; tile < te; ++tile)
        modularity_merge_tile_graphs<kPersistThreads>(tile, p.nv, p.nnz, p.a.ptr, p.a.tail, p.a.w,
                                                      p.C_mod, p.own_w_mod, p.cDeg, p.split_row,
                                                      p.gid, p.gacc, msm, acc);
      graph_acc_flush(acc, p.gacc);
    } else {
      for (int64_t tile = blockIdx.x; tile < ntiles; tile += gridDim.x)
        modularity_merge_tile<kPersistThreads>(tile, p.nv, p.nnz, p.a.ptr, p.a.tail, p.a.w,
                                               p.C_mod, p.own_w_mod, p.cDeg, p.split_row, msm, ex,
                                               a2);
    }
    ex = block_sum<kPersistThreads>(ex, sh);
    a2 = block_sum<kPersistThreads>(a2, sh);
    if (threadIdx.x == 0) { p.part_e[blockIdx.x] = ex; p.part_a[blockIdx.x] = a2; }
  }
  grid.sync();
  GLV_TRACE(4 * p.nsteps + 1);
  if (blockIdx.x == 0) {
    if (!p.gid) modularity_fold(p, gridDim.x, sh);
    if (threadIdx.x == 0) p.mod_out[4] = (double)__ldcg(p.h.err);
  }
  if (p.jacobi && p.nsteps > 0) {
    // Q above used the totals before the moves; now take the moves' deltas.
    apply_deltas_range(p, p.steps[0].apply[0], p.steps[p.nsteps - 1].apply[1], gt, ngt);
  }
}

}  // namespace glv
