// Edge lists to CSR on the device, and Grappolo's binary graph files.
//
// The reference builds its graphs on the host: removeEdges drops self-loops
// and repeated (head, tail) pairs (Utility/utilityFunctions.cpp:416-460), the
// loaders (e.g. InputsOutput/loadPajekFormat.cpp:94-150) and
// SortEdgesUndirected (utilityFunctions.cpp:463-498) store every edge in the
// rows of both its ends in list order, and SortNodeEdgesByIndex
// (:501-531) sorts each row by tail.  Here each of those is a handful of
// grid-stride kernels around CUB radix sorts and scans, with the exact output
// order of the reference's one-thread code:
//
//  * kept edges: a stable sort of (head, tail) keys marks the first of each
//    run; removeEdges' compaction fills the dropped slots below NGE, in
//    ascending order, with the kept edges above NGE from the top down, which
//    two scans and two scatters reproduce;
//  * rows: entry 2k + d (kept edge k, d = 0 head side, 1 tail side) is
//    stable-sorted by row, which is the loaders' fill order;
//  * sorted rows: the reference's bottom-up merge takes the right run on equal
//    tails, so equal tails end in descending position; a stable sort by
//    (row, tail) of the entries listed in reverse gives exactly that;
//  * both at once: sorted rows are merged from the kept edges as they stand
//    (by head) and sorted by tail.
//
// Included into engine.cu after the C ABI helpers (Call, fail, CK, TRY).

namespace glv {

constexpr int kIdBits = 31;
constexpr uint64_t kIdMask = (1ull << kIdBits) - 1;

// Bits that hold every id below nv: sort keys (row, col) take 2 * id_bits(nv)
// bits, so the radix sorts make only the passes the graph needs.
static int id_bits(int64_t nv) {
  int b = 1;
  while (b < kIdBits && (int64_t(1) << b) < nv) ++b;
  return b;
}

// Edge arrays as the kernels read them: AoS glv_edge (stride 3 words) or
// separate int64 heads / tails and double weights (stride 1).  A null weight
// array reads as 1.0.
struct EdgeView {
  const int64_t *head, *tail;
  const double *w;
  int64_t stride;
  __device__ __forceinline__ int64_t h(int64_t i) const { return head[i * stride]; }
  __device__ __forceinline__ int64_t t(int64_t i) const { return tail[i * stride]; }
  __device__ __forceinline__ double wt(int64_t i) const { return w ? w[i * stride] : 1.0; }
};

static EdgeView aos_view(const glv_edge *e) {
  static_assert(sizeof(glv_edge) == 24, "glv_edge is three 8-byte words");
  const int64_t *base = reinterpret_cast<const int64_t *>(e);
  return EdgeView{base, base + 1, reinterpret_cast<const double *>(base + 2), 3};
}

__global__ void k_edge_pair_keys(int64_t ne, EdgeView ev, int64_t nv, int bits, uint64_t *keys,
                                 int64_t *idx, int32_t *bad) {
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < ne;
       i += (int64_t)gridDim.x * blockDim.x) {
    int64_t h = ev.h(i), t = ev.t(i);
    if (h < 0 || h >= nv || t < 0 || t >= nv) {
      atomicOr(bad, 1);
      h = t = 0;
    }
    keys[i] = ((uint64_t)h << bits) | (uint64_t)t;
    idx[i] = i;
  }
}

// After the stable sort: the first edge of each (head, tail) run is kept
// unless it is a self-loop.
__global__ void k_mark_kept(int64_t ne, int bits, const uint64_t *skeys, const int64_t *sidx,
                            uint8_t *kept, unsigned long long *count) {
  unsigned int mine = 0;
  for (int64_t s = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; s < ne;
       s += (int64_t)gridDim.x * blockDim.x) {
    const uint64_t k = skeys[s];
    const bool first = s == 0 || skeys[s - 1] != k;
    const bool loop = (k >> bits) == (k & ((1ull << bits) - 1));
    const bool g = first && !loop;
    kept[sidx[s]] = g ? 1 : 0;
    mine += g ? 1u : 0u;
  }
  mine = __reduce_add_sync(FULL, mine);
  if ((threadIdx.x & 31) == 0 && mine) atomicAdd(count, (unsigned long long)mine);
}

// Scan input of the compaction: below NGE the dropped slots, from NGE on the
// kept edges.
__global__ void k_slot_flags(int64_t ne, int64_t nge, const uint8_t *kept, int64_t *f) {
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < ne;
       i += (int64_t)gridDim.x * blockDim.x)
    f[i] = (i < nge) ? (kept[i] ? 0 : 1) : (kept[i] ? 1 : 0);
}

__global__ void k_order_low(int64_t nge, const uint8_t *kept, const int64_t *scan, int64_t *order,
                            int64_t *holes) {
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < nge;
       i += (int64_t)gridDim.x * blockDim.x) {
    if (kept[i]) order[i] = i;
    else holes[scan[i]] = i;
  }
}

// Kept edge i >= NGE is the r-th from the top (r = nholes - 1 - its rank
// above NGE) and fills the r-th hole.
__global__ void k_order_high(int64_t ne, int64_t nge, int64_t nholes, const uint8_t *kept,
                             const int64_t *scan, const int64_t *holes, int64_t *order) {
  for (int64_t i = nge + (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < ne;
       i += (int64_t)gridDim.x * blockDim.x) {
    if (!kept[i]) continue;
    const int64_t r = nholes - 1 - (scan[i] - nholes);
    order[holes[r]] = i;
  }
}

__device__ __forceinline__ void entry_of(int64_t e, const int64_t *order, const EdgeView &ev,
                                         int64_t *src, int64_t *row, int64_t *col) {
  const int64_t k = e >> 1;
  const int64_t i = order ? order[k] : k;
  const int64_t h = ev.h(i), t = ev.t(i);
  *src = i;
  *row = (e & 1) ? t : h;
  *col = (e & 1) ? h : t;
}

// Sort records of the 2 * nk directed entries, one per entry e = 2k + d.
// sorted_rows: listed in reverse, key (row, col), sorted on all 2 * bits;
// otherwise in order, key (col above row), sorted on the row bits only, so
// the column rides along in the key's upper bits.  The weight is the sort
// value: the sorted records are the CSR, with nothing left to gather.
__global__ void k_entry_keys(int64_t m, bool sorted_rows, int bits, int64_t nv,
                             const int64_t *order, EdgeView ev, uint64_t *keys, double *vals,
                             int32_t *bad) {
  for (int64_t q = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; q < m;
       q += (int64_t)gridDim.x * blockDim.x) {
    const int64_t e = sorted_rows ? m - 1 - q : q;
    int64_t src, row, col;
    entry_of(e, order, ev, &src, &row, &col);
    if (row < 0 || row >= nv || col < 0 || col >= nv) {
      atomicOr(bad, 1);
      row = col = 0;
    }
    keys[q] = sorted_rows ? (((uint64_t)row << bits) | (uint64_t)col)
                          : (((uint64_t)col << bits) | (uint64_t)row);
    vals[q] = ev.wt(src);
  }
}

__device__ __forceinline__ int64_t key_row(uint64_t k, bool sorted_rows, int bits) {
  return sorted_rows ? (int64_t)(k >> bits) : (int64_t)(k & ((1ull << bits) - 1));
}

__device__ __forceinline__ int64_t key_col(uint64_t k, bool sorted_rows, int bits) {
  return sorted_rows ? (int64_t)(k & ((1ull << bits) - 1)) : (int64_t)(k >> bits);
}

// Row offsets from the sorted records: position s opens every row after the
// previous record's row up to its own (s = m closes the rest).
__global__ void k_row_bounds(int64_t m, int64_t nv, bool sorted_rows, int bits,
                             const uint64_t *skeys, int64_t *ptr) {
  for (int64_t s = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; s <= m;
       s += (int64_t)gridDim.x * blockDim.x) {
    const int64_t here = s < m ? key_row(skeys[s], sorted_rows, bits) : nv;
    const int64_t prev = s > 0 ? key_row(skeys[s - 1], sorted_rows, bits) : -1;
    for (int64_t r = prev + 1; r <= here; ++r) ptr[r] = s;
  }
}

__global__ void k_emit_entries(int64_t m, bool sorted_rows, int bits, const uint64_t *skeys,
                               const double *svals, int32_t *otail, double *ow, glv_edge *oaos) {
  for (int64_t s = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; s < m;
       s += (int64_t)gridDim.x * blockDim.x) {
    const uint64_t k = skeys[s];
    const int64_t col = key_col(k, sorted_rows, bits);
    const double w = svals[s];
    if (otail) otail[s] = (int32_t)col;
    if (ow) ow[s] = w;
    if (oaos) oaos[s] = glv_edge{(long)key_row(k, sorted_rows, bits), (long)col, w};
  }
}

__global__ void k_gather_edges(int64_t n, const int64_t *order, const glv_edge *in, glv_edge *out) {
  for (int64_t k = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; k < n;
       k += (int64_t)gridDim.x * blockDim.x)
    out[k] = in[order[k]];
}

// Row id of every entry of a CSR (one warp per row).
__global__ void k_row_ids(int64_t nv, const int64_t *ptr, int64_t *rowid) {
  const int lane = threadIdx.x & 31;
  for (int64_t v = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5; v < nv;
       v += ((int64_t)gridDim.x * blockDim.x) >> 5)
    for (int64_t j = ptr[v] + lane; j < ptr[v + 1]; j += 32) rowid[j] = v;
}

// SortNodeEdgesByIndex keys: positions listed in reverse, keyed (row, tail).
__global__ void k_row_sort_keys(int64_t nnz, const int64_t *rowid, const glv_edge *e,
                                uint64_t *keys, int64_t *vals, int32_t *bad) {
  // the row above the tail's 31 bits: tails of a given CSR are not bounded by
  // its row count
  for (int64_t q = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; q < nnz;
       q += (int64_t)gridDim.x * blockDim.x) {
    const int64_t p = nnz - 1 - q;
    int64_t t = e[p].tail;
    if (t < 0 || t > (int64_t)kIdMask) {
      atomicOr(bad, 1);
      t = 0;
    }
    keys[q] = ((uint64_t)rowid[p] << kIdBits) | (uint64_t)t;
    vals[q] = p;
  }
}

// Binary files: ids of each entry checked against NV while splitting.
__global__ void k_split_checked(int64_t n, const glv_edge *aos, int64_t nv, int32_t *tail,
                                double *w, int32_t *bad) {
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n;
       i += (int64_t)gridDim.x * blockDim.x) {
    const int64_t t = aos[i].tail;
    if (t < 0 || t >= nv) atomicOr(bad, 1);
    tail[i] = (int32_t)t;
    w[i] = aos[i].weight;
  }
}

// Pool allocations released (stream-ordered) when the owner goes out of scope.
struct DevScratch {
  cudaStream_t s;
  std::vector<void *> held;
  explicit DevScratch(cudaStream_t st) : s(st) {}
  ~DevScratch() {
    for (void *p : held) cudaFreeAsync(p, s);
  }
  template <class T>
  int get(T **p, int64_t n) {
    cudaError_t e = cudaMallocFromPoolAsync((void **)p, std::max<int64_t>(n, 1) * sizeof(T),
                                            engine_pool(), s);
    if (e == cudaErrorMemoryAllocation) {
      // hand the pool's unused blocks back and retry once
      cudaGetLastError();
      cudaStreamSynchronize(s);
      cudaMemPoolTrimTo(engine_pool(), 0);
      e = cudaMallocFromPoolAsync((void **)p, std::max<int64_t>(n, 1) * sizeof(T), engine_pool(), s);
    }
    if (e != cudaSuccess) {
      cudaGetLastError();
      return fail(GLV_ERR_OOM, "device allocation failed while building a CSR");
    }
    held.push_back(*p);
    return GLV_OK;
  }
};

static int csr_grid(int64_t n) { return grid_for(n, 256, 148 * 16); }

// removeEdges on the device: *order[k] = index of the edge that ends in slot
// k < *nge.
static int kept_order(cudaStream_t s, int64_t nv, int64_t ne, EdgeView ev, DevScratch &d,
                      int64_t **order, int64_t *nge, long *launches) {
  uint64_t *k1, *k2;
  int64_t *v1, *v2, *scan, *flags, *holes;
  uint8_t *kept;
  int32_t *bad;
  unsigned long long *cnt;
  TRY(d.get(&k1, ne));
  TRY(d.get(&k2, ne));
  TRY(d.get(&v1, ne));
  TRY(d.get(&v2, ne));
  TRY(d.get(&kept, ne));
  TRY(d.get(&bad, 1));
  TRY(d.get(&cnt, 1));
  CK(cudaMemsetAsync(bad, 0, sizeof(int32_t), s));
  CK(cudaMemsetAsync(cnt, 0, sizeof(unsigned long long), s));
  const int bits = id_bits(nv);
  k_edge_pair_keys<<<csr_grid(ne), 256, 0, s>>>(ne, ev, nv, bits, k1, v1, bad);
  ++*launches;
  CK(cudaGetLastError());
  size_t tb = 0;
  CK(cub::DeviceRadixSort::SortPairs(nullptr, tb, k1, k2, v1, v2, ne, 0, 2 * bits, s));
  void *temp;
  TRY(d.get((char **)&temp, (int64_t)tb));
  CK(cub::DeviceRadixSort::SortPairs(temp, tb, k1, k2, v1, v2, ne, 0, 2 * bits, s));
  k_mark_kept<<<csr_grid(ne), 256, 0, s>>>(ne, bits, k2, v2, kept, cnt);
  ++*launches;
  CK(cudaGetLastError());
  int32_t hbad = 0;
  unsigned long long hcnt = 0;
  CK(cudaMemcpyAsync(&hbad, bad, sizeof(hbad), cudaMemcpyDeviceToHost, s));
  CK(cudaMemcpyAsync(&hcnt, cnt, sizeof(hcnt), cudaMemcpyDeviceToHost, s));
  CK(cudaStreamSynchronize(s));
  if (hbad) return fail(GLV_ERR_ARG, "an edge end is outside [0, NV)");
  *nge = (int64_t)hcnt;
  // keys and sort values are free again: reuse them for the compaction
  flags = reinterpret_cast<int64_t *>(k1);
  scan = reinterpret_cast<int64_t *>(k2);
  holes = v1;
  *order = v2;
  k_slot_flags<<<csr_grid(ne), 256, 0, s>>>(ne, *nge, kept, flags);
  ++*launches;
  CK(cudaGetLastError());
  size_t tb2 = 0;
  CK(cub::DeviceScan::ExclusiveSum(nullptr, tb2, flags, scan, ne, s));
  if (tb2 > tb) TRY(d.get((char **)&temp, (int64_t)tb2));
  CK(cub::DeviceScan::ExclusiveSum(temp, tb2, flags, scan, ne, s));
  int64_t nholes = 0;
  if (*nge < ne) {
    CK(cudaMemcpyAsync(&nholes, scan + *nge, sizeof(nholes), cudaMemcpyDeviceToHost, s));
    CK(cudaStreamSynchronize(s));
  }
  if (*nge > 0) {
    k_order_low<<<csr_grid(*nge), 256, 0, s>>>(*nge, kept, scan, *order, holes);
    ++*launches;
    CK(cudaGetLastError());
  }
  if (nholes > 0) {
    k_order_high<<<csr_grid(ne - *nge), 256, 0, s>>>(ne, *nge, nholes, kept, scan, holes, *order);
    ++*launches;
    CK(cudaGetLastError());
  }
  return GLV_OK;
}

// The 2 * nk directed entries of the kept edges in row order (sorted_rows:
// rows sorted by tail, equal tails latest first), written as a CSR: d_ptr[nv
// + 1] and any of otail / ow (SoA) and oaos (glv_edge records).  Ids outside
// [0, nv) are GLV_ERR_ARG.
static int row_entries(cudaStream_t s, int64_t nv, int64_t nk, const int64_t *order, EdgeView ev,
                       bool sorted_rows, DevScratch &d, int64_t *d_ptr, int32_t *otail, double *ow,
                       glv_edge *oaos, long *launches) {
  const int64_t m = 2 * nk;
  const int ib = id_bits(nv);
  uint64_t *k1, *k2;
  double *v1, *v2;
  int32_t *bad;
  TRY(d.get(&k1, m));
  TRY(d.get(&k2, m));
  TRY(d.get(&v1, m));
  TRY(d.get(&v2, m));
  TRY(d.get(&bad, 1));
  CK(cudaMemsetAsync(bad, 0, sizeof(int32_t), s));
  if (m > 0) {
    k_entry_keys<<<csr_grid(m), 256, 0, s>>>(m, sorted_rows, ib, nv, order, ev, k1, v1, bad);
    ++*launches;
    CK(cudaGetLastError());
    const int bits = sorted_rows ? 2 * ib : ib;
    size_t tb = 0;
    CK(cub::DeviceRadixSort::SortPairs(nullptr, tb, k1, k2, v1, v2, m, 0, bits, s));
    void *temp;
    TRY(d.get((char **)&temp, (int64_t)tb));
    CK(cub::DeviceRadixSort::SortPairs(temp, tb, k1, k2, v1, v2, m, 0, bits, s));
  }
  k_row_bounds<<<csr_grid(m + 1), 256, 0, s>>>(m, nv, sorted_rows, ib, k2, d_ptr);
  ++*launches;
  CK(cudaGetLastError());
  if (m > 0) {
    k_emit_entries<<<csr_grid(m), 256, 0, s>>>(m, sorted_rows, ib, k2, v2, otail, ow, oaos);
    ++*launches;
    CK(cudaGetLastError());
  }
  int32_t hb = 0;
  CK(cudaMemcpyAsync(&hb, bad, sizeof(hb), cudaMemcpyDeviceToHost, s));
  CK(cudaStreamSynchronize(s));
  if (hb) return fail(GLV_ERR_ARG, "an edge end is outside [0, NV)");
  return GLV_OK;
}

// ---- removeEdges and sorted rows together --------------------------------
// The sort that finds repeats leaves the kept edges in (head, tail) order, which
// is the order of their head-side entries.  Their tail-side entries need only a
// stable sort of that list on the tail's bits (half the passes over half the
// records of a new sort of all directed entries), and the rows are the merge of
// the two lists: both are ordered by (row, column) over the whole graph.
// R-MAT 22 (67M edges): 15.7 ms by sorting all entries anew, 9.15 this way, of
// which the two sorts 5.1, the weights' gathers 1.7, the rest of the merge 1.2.
//
// Equal entries come latest first, by the slots removeEdges leaves the edges in:
// an edge below NGE keeps its slot, and the q-th kept edge from NGE on fills the
// q-th hole from the end.  Only ties need slots; they come from a bitmap of the
// dropped places with the count before every 128 (two loads a count, both from
// L2), and the holes, the dropped places below NGE, in order.  (A sorted list of
// all dropped places, searched for every tie, cost more than it saved where most
// edges are repeats: 20M edges over 1000 vertices 1.39 ms by sorting all entries,
// 1.59 that way, 1.07 this way.)
constexpr int kDropBlock = 128;  // places to a count
// Counts that one block makes alone, in one launch for three: with the three
// 300,000 edges took 237.8 us for 234.5, 20,463 edges 6 % more; a million edges
// take the same either way.
constexpr int kDropOneBlock = 4096;
struct KeptSorted {
  int64_t nge = 0, ndrop = 0;
  uint64_t *key = nullptr;    // kept edges by (head, tail): head << bits | tail
  int32_t *idx = nullptr;     // their places in the list
  uint32_t *dropped = nullptr;  // bitmap over the list
  int32_t *before = nullptr;  // dropped places before each kDropBlock
  int32_t *hole = nullptr;    // the holes, ascending
};

__device__ __forceinline__ int drop_count(const uint4 &w) {
  return __popc(w.x) + __popc(w.y) + __popc(w.z) + __popc(w.w);
}

struct DropCount {  // dropped places of each kDropBlock
  const uint4 *words;
  __device__ int32_t operator()(int32_t b) const { return drop_count(words[b]); }
};

constexpr int kPickItems = 8;            // records a lane of k_pick
constexpr int kPickTile = 256 * kPickItems;
constexpr int kRunItems = 7;  // entries a thread of k_merge_runs; odd: the threads'
constexpr int kRunThreads = 256;
constexpr int kRunTile = kRunThreads * kRunItems;  // runs start in different banks

__global__ void k_pair_keys32(int64_t ne, EdgeView ev, int64_t nv, int bits, uint64_t *keys,
                              int32_t *idx, int32_t *bad, int64_t words, uint32_t *dropped) {
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < words;
       i += (int64_t)gridDim.x * blockDim.x)
    dropped[i] = 0;
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < ne;
       i += (int64_t)gridDim.x * blockDim.x) {
    int64_t h = ev.h(i), t = ev.t(i);
    if (h < 0 || h >= nv || t < 0 || t >= nv) {
      atomicOr(bad, 1);
      h = t = 0;
    }
    keys[i] = ((uint64_t)h << bits) | (uint64_t)t;
    idx[i] = (int32_t)i;
  }
}

// Whether sorted record s is the first of its (head, tail) run and no self-loop.
__device__ __forceinline__ bool run_first(const uint64_t *skeys, int64_t s, int bits, uint64_t k) {
  return (k >> bits) != (k & ((1ull << bits) - 1)) && (s == 0 || skeys[s - 1] != k);
}

// One block per tile of sorted records.  Not kWrite: kept[tile] = its kept
// records; otherwise they go to key / idx from kept[tile] (the tile's offset)
// on, in order, and the other records' places are set in dropped.  A warp takes 256
// records in a row, so its writes are coalesced (two passes over the keys,
// 8 + 24 bytes a record, 0.58 ms for 67M; a scatter of one flag byte per record
// to its place in the list and selections from those flags took 1.3).
template <bool kWrite>
__global__ void __launch_bounds__(256) k_pick(int64_t ne, int bits, const uint64_t *skeys,
                                              const int32_t *sidx, int64_t *kept, uint64_t *key,
                                              int32_t *idx, uint32_t *dropped) {
  __shared__ int s_n[8];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int64_t s0 = (int64_t)blockIdx.x * kPickTile + warp * (32 * kPickItems);
  uint64_t k[kPickItems];
  unsigned m[kPickItems];
  int n = 0;
#pragma unroll
  for (int u = 0; u < kPickItems; ++u) {
    const int64_t s = s0 + u * 32 + lane;
    k[u] = s < ne ? skeys[s] : 0;
    m[u] = __ballot_sync(0xffffffffu, s < ne && run_first(skeys, s, bits, k[u]));
    n += __popc(m[u]);
  }
  if (lane == 0) s_n[warp] = n;
  __syncthreads();
  int before = 0, all = 0;
  for (int w = 0; w < 8; ++w) {
    if (w < warp) before += s_n[w];
    all += s_n[w];
  }
  if constexpr (!kWrite) {
    if (threadIdx.x == 0) kept[blockIdx.x] = all;
  } else {
    int64_t at = kept[blockIdx.x] + before;
#pragma unroll
    for (int u = 0; u < kPickItems; ++u) {
      const int64_t s = s0 + u * 32 + lane;
      const int64_t p = at + __popc(m[u] & ((1u << lane) - 1));
      at += __popc(m[u]);
      if (s >= ne) continue;
      if (m[u] >> lane & 1) {
        key[p] = k[u];
        idx[p] = sidx[s];
      } else {
        const int32_t i = sidx[s];
        atomicOr(&dropped[i >> 5], 1u << (i & 31));
      }
    }
  }
}

// The holes among the places of count b (bits w), of which `at` stand before.
__device__ __forceinline__ void emit_holes(int64_t b, const uint4 &w, int64_t at, int64_t nge,
                                           int32_t *hole) {
  const uint32_t part[4] = {w.x, w.y, w.z, w.w};
#pragma unroll
  for (int q = 0; q < 4; ++q)
    for (uint32_t rem = part[q]; rem; rem &= rem - 1) {
      const int64_t place = b * kDropBlock + 32 * q + __ffs(rem) - 1;
      if (place < nge) hole[at++] = (int32_t)place;
    }
}

// The holes in order; one thread per kDropBlock places.
__global__ void k_holes(int64_t nge, const uint4 *words, const int32_t *before, int32_t *hole) {
  const int64_t nb = (nge + kDropBlock - 1) / kDropBlock;
  for (int64_t b = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; b < nb;
       b += (int64_t)gridDim.x * blockDim.x)
    emit_holes(b, words[b], before[b], nge, hole);
}

// Counts and holes of a short list (nb <= kDropOneBlock) by one block.
__global__ void __launch_bounds__(1024) k_drop_index(int nb, int64_t nge, const uint4 *words,
                                                     int32_t *before, int32_t *hole) {
  constexpr int kPer = kDropOneBlock / 1024;
  __shared__ int s_n[32];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int b0 = threadIdx.x * kPer;
  uint4 w[kPer];
  int n = 0;
#pragma unroll
  for (int k = 0; k < kPer; ++k) {
    w[k] = b0 + k < nb ? words[b0 + k] : make_uint4(0, 0, 0, 0);
    n += drop_count(w[k]);
  }
  int incl = n;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const int y = __shfl_up_sync(0xffffffffu, incl, o);
    if (lane >= o) incl += y;
  }
  if (lane == 31) s_n[warp] = incl;
  __syncthreads();
  int at = incl - n;
  for (int k = 0; k < warp; ++k) at += s_n[k];
#pragma unroll
  for (int k = 0; k < kPer; ++k) {
    if (b0 + k < nb) {
      before[b0 + k] = at;
      emit_holes(b0 + k, w[k], at, nge, hole);
    }
    at += drop_count(w[k]);
  }
}

__device__ __forceinline__ int64_t drops_below(const KeptSorted &ks, int64_t place) {
  const int64_t b = place / kDropBlock;
  uint4 w = reinterpret_cast<const uint4 *>(ks.dropped)[b];
  const int q = (int)(place % kDropBlock) >> 5;
  const uint32_t low = (1u << (place & 31)) - 1u;  // of the word that holds place
  w.x &= q > 0 ? ~0u : low;
  w.y &= q > 1 ? ~0u : (q == 1 ? low : 0u);
  w.z &= q > 2 ? ~0u : (q == 2 ? low : 0u);
  w.w &= q == 3 ? low : 0u;
  return ks.before[b] + drop_count(w);
}

// The slot that removeEdges leaves the kept list edge i in.
__device__ __forceinline__ int64_t kept_slot(const KeptSorted &ks, int32_t i) {
  if (i < ks.nge) return i;
  const int64_t holes = drops_below(ks, ks.nge);
  const int64_t q = (i - ks.nge) - (drops_below(ks, i) - holes);
  return ks.hole[holes - 1 - q];
}

// The two lists of directed entries: by head as the kept edges stand, by tail
// as sorted on the tail's bits (still head << bits | tail).
struct EntryRuns {
  KeptSorted ks;
  const uint64_t *tkey;
  const int32_t *tidx;
  int bits;
  __device__ __forceinline__ uint64_t tail_side(int64_t j) const {
    const uint64_t k = tkey[j];
    return ((k & ((1ull << bits) - 1)) << bits) | (k >> bits);
  }
};

// Whether the head-side entry (ka, edge ia) comes before the tail-side (kb, ib).
__device__ __forceinline__ bool head_first(const KeptSorted &ks, uint64_t ka, uint64_t kb,
                                           int32_t ia, int32_t ib) {
  return ka != kb ? ka < kb : kept_slot(ks, ia) > kept_slot(ks, ib);
}

// split[t] = head-side entries among the first t * kRunTile merged ones.
__global__ void k_run_splits(EntryRuns r, int64_t ntiles, int64_t *split) {
  const int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (t > ntiles) return;
  const int64_t n = r.ks.nge, d = min(t * (int64_t)kRunTile, 2 * n);
  int64_t lo = max((int64_t)0, d - n), hi = min(d, n);
  while (lo < hi) {
    const int64_t mid = (lo + hi) >> 1, j = d - 1 - mid;
    if (head_first(r.ks, r.ks.key[mid], r.tail_side(j), r.ks.idx[mid], r.tidx[j]))
      lo = mid + 1;
    else
      hi = mid;
  }
  split[t] = lo;
}

// One tile of the merged entries per block: both lists' parts to shared memory,
// each thread merges kRunItems entries, and the merged tile is written out
// coalesced, with the row offsets.  The weights are gathered by the edge's
// place in the list, which is what bounds it (32-byte sectors for 8 bytes): 2.9
// ms for 131M entries, 1.2 of it without weights.  Tiles of 3 to 7 entries a
// thread and 128 or 256 threads measure the same to 1%, 11 and 15 entries 24%
// more of the whole build.  A search of every entry in the other list's row
// took 5.9 ms.
__global__ void __launch_bounds__(kRunThreads) k_merge_runs(EntryRuns r, EdgeView ev, int64_t nv,
                                                    const int64_t *split, int64_t *ptr,
                                                    int32_t *otail, double *ow, glv_edge *oaos) {
  __shared__ uint64_t s_key[kRunTile];
  __shared__ int32_t s_idx[kRunTile];
  __shared__ uint16_t s_from[kRunTile];  // where the merged tile's entries stand
  const int64_t m = 2 * r.ks.nge;
  const int64_t d0 = (int64_t)blockIdx.x * kRunTile;
  const int n = (int)min((int64_t)kRunTile, m - d0);
  const int64_t a0 = split[blockIdx.x], b0 = d0 - a0;
  const int na = (int)(split[blockIdx.x + 1] - a0), nb = n - na;
  const int bits = r.bits;
#pragma unroll
  for (int u = 0; u < kRunItems; ++u) {
    const int q = u * kRunThreads + threadIdx.x;
    if (q < na) {
      s_key[q] = r.ks.key[a0 + q];
      s_idx[q] = r.ks.idx[a0 + q];
    } else if (q < n) {
      s_key[q] = r.tail_side(b0 + q - na);
      s_idx[q] = r.tidx[b0 + q - na];
    }
  }
  __syncthreads();
  const int d = min((int)threadIdx.x * kRunItems, n);
  int lo = max(0, d - nb), hi = min(d, na);
  while (lo < hi) {
    const int mid = (lo + hi) >> 1, j = na + d - 1 - mid;
    if (head_first(r.ks, s_key[mid], s_key[j], s_idx[mid], s_idx[j])) lo = mid + 1; else hi = mid;
  }
  int a = lo, b = na + d - lo;
  uint64_t ka = a < na ? s_key[a] : ~0ull, kb = b < n ? s_key[b] : ~0ull;  // ~0: after any key
#pragma unroll
  for (int u = 0; u < kRunItems; ++u) {
    if (d + u < n) {
      const bool left = ka != kb ? ka < kb : head_first(r.ks, ka, kb, s_idx[a], s_idx[b]);
      s_from[d + u] = (uint16_t)(left ? a : b);
      if (left) {
        ++a;
        ka = a < na ? s_key[a] : ~0ull;
      } else {
        ++b;
        kb = b < n ? s_key[b] : ~0ull;
      }
    }
  }
  __syncthreads();
  double w[kRunItems];
#pragma unroll
  for (int u = 0; u < kRunItems; ++u) {
    const int q = u * kRunThreads + threadIdx.x;
    w[u] = q < n ? ev.wt(s_idx[s_from[q]]) : 0;
  }
  const uint64_t low = (1ull << bits) - 1;
#pragma unroll
  for (int u = 0; u < kRunItems; ++u) {
    const int q = u * kRunThreads + threadIdx.x;
    if (q >= n) continue;
    const int64_t at = d0 + q;
    const uint64_t k = s_key[s_from[q]];
    const int64_t row = (int64_t)(k >> bits), col = (int64_t)(k & low);
    if (otail) otail[at] = (int32_t)col;
    if (ow) ow[at] = w[u];
    if (oaos) oaos[at] = glv_edge{(long)row, (long)col, w[u]};
    int64_t prev = -1;  // the row of the entry before
    if (q > 0) {
      prev = (int64_t)(s_key[s_from[q - 1]] >> bits);
    } else {
      if (a0 > 0) prev = (int64_t)(r.ks.key[a0 - 1] >> bits);
      if (b0 > 0) prev = max(prev, (int64_t)(r.tail_side(b0 - 1) >> bits));
    }
    for (int64_t x = prev + 1; x <= row; ++x) ptr[x] = at;
    if (at == m - 1)
      for (int64_t x = row + 1; x <= nv; ++x) ptr[x] = m;
  }
}

// Whether a build takes this way: both options, and list places in 32 bits.  It
// is the faster one at every size measured: 128 edges 147 -> 138 us, 130k 285 ->
// 249, 8M 2036 -> 1254, 67M 15700 -> 9150.
static bool merges_rows(int flags, int64_t ne) {
  return ne > 0 && ne < (int64_t(1) << 31) - 1 && (flags & GLV_CSR_REMOVE_EDGES) &&
         (flags & GLV_CSR_SORT_ROWS);
}

static bool overlap(const void *a, int64_t na, const void *b, int64_t nb) {
  const uintptr_t x = (uintptr_t)a, y = (uintptr_t)b;
  return a && b && x < y + (uintptr_t)nb && y < x + (uintptr_t)na;
}

// The kept edges in (head, tail) order.
static int kept_sorted(cudaStream_t s, int64_t nv, int64_t ne, EdgeView ev, DevScratch &d,
                       KeptSorted *ks, long *launches) {
  uint64_t *k1, *k2;
  int32_t *v1, *v2, *bad;
  int64_t *cnt;
  const int64_t tiles = (ne + kPickTile - 1) / kPickTile;
  TRY(d.get(&k1, ne)); TRY(d.get(&k2, ne)); TRY(d.get(&v1, ne)); TRY(d.get(&v2, ne));
  TRY(d.get(&bad, 1)); TRY(d.get(&cnt, tiles + 1));
  CK(cudaMemsetAsync(bad, 0, sizeof(int32_t), s));
  CK(cudaMemsetAsync(cnt + tiles, 0, sizeof(int64_t), s));
  const int64_t nb = (ne + kDropBlock - 1) / kDropBlock, nw = nb * (kDropBlock / 32);
  TRY(d.get(&ks->dropped, nw));
  const int bits = id_bits(nv);
  k_pair_keys32<<<csr_grid(ne), 256, 0, s>>>(ne, ev, nv, bits, k1, v1, bad, nw, ks->dropped);
  CK(cudaGetLastError());
  size_t tb = 0, t2 = 0;
  CK(cub::DeviceRadixSort::SortPairs(nullptr, tb, k1, k2, v1, v2, ne, 0, 2 * bits, s));
  CK(cub::DeviceScan::ExclusiveSum(nullptr, t2, cnt, cnt, tiles + 1, s));
  void *temp;
  TRY(d.get((char **)&temp, (int64_t)std::max(tb, t2)));
  CK(cub::DeviceRadixSort::SortPairs(temp, tb, k1, k2, v1, v2, ne, 0, 2 * bits, s));
  k_pick<false><<<(unsigned)tiles, 256, 0, s>>>(ne, bits, k2, v2, cnt, nullptr, nullptr, nullptr);
  CK(cudaGetLastError());
  CK(cub::DeviceScan::ExclusiveSum(temp, t2, cnt, cnt, tiles + 1, s));
  int32_t hbad = 0;
  CK(cudaMemcpyAsync(&hbad, bad, sizeof(hbad), cudaMemcpyDeviceToHost, s));
  CK(cudaMemcpyAsync(&ks->nge, cnt + tiles, sizeof(int64_t), cudaMemcpyDeviceToHost, s));
  CK(cudaStreamSynchronize(s));
  if (hbad) return fail(GLV_ERR_ARG, "an edge end is outside [0, NV)");
  ks->key = k1;
  ks->idx = v1;
  ks->ndrop = ne - ks->nge;
  k_pick<true><<<(unsigned)tiles, 256, 0, s>>>(ne, bits, k2, v2, cnt, k1, v1, ks->dropped);
  CK(cudaGetLastError());
  *launches += 3;
  if (ks->ndrop > 0 && ks->nge > 0) {
    const uint4 *words = reinterpret_cast<const uint4 *>(ks->dropped);
    TRY(d.get(&ks->before, nb)); TRY(d.get(&ks->hole, std::min(ks->nge, ks->ndrop)));
    if (nb <= kDropOneBlock) {
      k_drop_index<<<1, 1024, 0, s>>>((int)nb, ks->nge, words, ks->before, ks->hole);
    } else {
      const auto count = thrust::make_transform_iterator(thrust::counting_iterator<int32_t>(0),
                                                         DropCount{words});
      CK(cub::DeviceScan::ExclusiveSum(nullptr, t2, count, ks->before, nb, s));
      TRY(d.get((char **)&temp, (int64_t)t2));
      CK(cub::DeviceScan::ExclusiveSum(temp, t2, count, ks->before, nb, s));
      k_holes<<<csr_grid(nb), 256, 0, s>>>(ks->nge, words, ks->before, ks->hole);
    }
    ++*launches;
    CK(cudaGetLastError());
  }
  return GLV_OK;
}

// The CSR of the kept edges, both directions, rows sorted.
static int merged_rows(cudaStream_t s, int64_t nv, const KeptSorted &ks, EdgeView ev,
                       DevScratch &d, int64_t *d_ptr, int32_t *otail, double *ow, glv_edge *oaos,
                       long *launches) {
  const int64_t n = ks.nge;
  if (n == 0) {
    CK(cudaMemsetAsync(d_ptr, 0, (nv + 1) * sizeof(int64_t), s));
  } else {
    EntryRuns r{ks, nullptr, nullptr, id_bits(nv)};
    const int64_t tiles = (2 * n + kRunTile - 1) / kRunTile;
    uint64_t *tkey;
    int32_t *tidx;
    int64_t *split;
    TRY(d.get(&tkey, n)); TRY(d.get(&tidx, n)); TRY(d.get(&split, tiles + 1));
    size_t tb = 0;
    CK(cub::DeviceRadixSort::SortPairs(nullptr, tb, ks.key, tkey, ks.idx, tidx, n, 0, r.bits, s));
    void *temp;
    TRY(d.get((char **)&temp, (int64_t)tb));
    CK(cub::DeviceRadixSort::SortPairs(temp, tb, ks.key, tkey, ks.idx, tidx, n, 0, r.bits, s));
    r.tkey = tkey;
    r.tidx = tidx;
    k_run_splits<<<(unsigned)(tiles / 256 + 1), 256, 0, s>>>(r, tiles, split);
    k_merge_runs<<<(unsigned)tiles, kRunThreads, 0, s>>>(r, ev, nv, split, d_ptr, otail, ow, oaos);
    *launches += 2;
    CK(cudaGetLastError());
  }
  CK(cudaStreamSynchronize(s));
  return GLV_OK;
}

// Device-to-host copy of a large result into ordinary (pageable, possibly
// never touched) host memory, such as the malloc'd arrays the reference's API
// returns.  A plain cudaMemcpy into such memory runs at the speed of one
// thread faulting pages in; here the data moves by DMA into two pinned
// staging buffers while a team of host threads copies the previous chunk out
// (and takes the page faults in parallel).
static bool page_locked(const void *p) {
  cudaPointerAttributes a;
  if (cudaPointerGetAttributes(&a, p) != cudaSuccess) {
    cudaGetLastError();
    return false;
  }
  return a.type == cudaMemoryTypeHost;
}

static void parallel_memcpy(char *dst, const char *src, int64_t n) {
  const int nthreads = (int)std::max(1u, std::min(16u, std::thread::hardware_concurrency()));
  std::vector<std::thread> team;
  const int64_t part = (n + nthreads - 1) / nthreads;
  for (int t = 0; t < nthreads; ++t) {
    const int64_t a = t * part, b = std::min(n, a + part);
    if (a >= b) break;
    team.emplace_back([=] { memcpy(dst + a, src + a, b - a); });
  }
  for (auto &th : team) th.join();
}

static int d2h_large(cudaStream_t s, void *host, const void *dev, int64_t bytes) {
  if (bytes <= 0) return GLV_OK;
  if (bytes < (int64_t(64) << 20) || page_locked(host)) {
    CK(cudaMemcpyAsync(host, dev, bytes, cudaMemcpyDeviceToHost, s));
    CK(cudaStreamSynchronize(s));
    return GLV_OK;
  }
  const int64_t chunk = int64_t(128) << 20;
  char *stage[2] = {nullptr, nullptr};
  cudaEvent_t ev[2] = {nullptr, nullptr};
  struct Guard {
    char **st;
    cudaEvent_t *ev;
    ~Guard() {
      for (int k = 0; k < 2; ++k) {
        if (ev[k]) {
          cudaEventSynchronize(ev[k]);
          cudaEventDestroy(ev[k]);
        }
        if (st[k]) cudaFreeHost(st[k]);
      }
    }
  } guard{stage, ev};
  for (int k = 0; k < 2; ++k) {
    CK(cudaHostAlloc((void **)&stage[k], chunk, cudaHostAllocDefault));
    CK(cudaEventCreateWithFlags(&ev[k], cudaEventDisableTiming));
  }
  auto copy_out = [](const char *src, char *dst, int64_t n) { parallel_memcpy(dst, src, n); };
  const char *d = static_cast<const char *>(dev);
  char *h = static_cast<char *>(host);
  int64_t prev_off = -1, prev_n = 0;
  int k = 0;
  for (int64_t off = 0; off < bytes; off += chunk, k ^= 1) {
    const int64_t n = std::min(chunk, bytes - off);
    CK(cudaMemcpyAsync(stage[k], d + off, n, cudaMemcpyDeviceToHost, s));
    CK(cudaEventRecord(ev[k], s));
    if (prev_off >= 0) {  // the previous chunk's DMA is done: copy it out meanwhile
      CK(cudaEventSynchronize(ev[k ^ 1]));
      copy_out(stage[k ^ 1], h + prev_off, prev_n);
    }
    prev_off = off;
    prev_n = n;
    // stage[k ^ 1] is free again for the next chunk's DMA
  }
  CK(cudaEventSynchronize(ev[k ^ 1]));
  copy_out(stage[k ^ 1], h + prev_off, prev_n);
  return GLV_OK;
}

// Host-to-device counterpart of d2h_large for pageable sources: host threads
// copy chunk i + 1 into a pinned staging buffer while chunk i moves by DMA.
static int h2d_large(cudaStream_t s, void *dev, const void *host, int64_t bytes) {
  if (bytes <= 0) return GLV_OK;
  if (bytes < (int64_t(64) << 20) || page_locked(host)) {
    CK(cudaMemcpyAsync(dev, host, bytes, cudaMemcpyHostToDevice, s));
    return GLV_OK;
  }
  const int64_t chunk = int64_t(128) << 20;
  char *stage[2] = {nullptr, nullptr};
  cudaEvent_t ev[2] = {nullptr, nullptr};
  struct Guard {
    char **st;
    cudaEvent_t *ev;
    ~Guard() {
      for (int k = 0; k < 2; ++k) {
        if (ev[k]) {
          cudaEventSynchronize(ev[k]);
          cudaEventDestroy(ev[k]);
        }
        if (st[k]) cudaFreeHost(st[k]);
      }
    }
  } guard{stage, ev};
  for (int k = 0; k < 2; ++k) {
    CK(cudaHostAlloc((void **)&stage[k], chunk, cudaHostAllocDefault));
    CK(cudaEventCreateWithFlags(&ev[k], cudaEventDisableTiming));
  }
  const char *h = static_cast<const char *>(host);
  char *d = static_cast<char *>(dev);
  int k = 0;
  for (int64_t off = 0; off < bytes; off += chunk, k ^= 1) {
    const int64_t n = std::min(chunk, bytes - off);
    CK(cudaEventSynchronize(ev[k]));  // this buffer's previous DMA has finished
    parallel_memcpy(stage[k], h + off, n);
    CK(cudaMemcpyAsync(d + off, stage[k], n, cudaMemcpyHostToDevice, s));
    CK(cudaEventRecord(ev[k], s));
  }
  return GLV_OK;  // the guard waits for both buffers' last DMA
}

static int upload_edges(cudaStream_t s, const glv_edge *host, int64_t n, DevScratch &d,
                        glv_edge **dev) {
  TRY(d.get(dev, n));
  return h2d_large(s, *dev, host, n * (int64_t)sizeof(glv_edge));
}

static int open_stream(Call &c) {
  TRY(device_ready());
  if (!engine_pool()) return fail(GLV_ERR_CUDA, "could not create the device memory pool");
  CK(engine_stream(&c.s));
  return GLV_OK;
}

static FILE *open_binary(const char *path, const char *how) {
  return path ? fopen(path, how) : nullptr;
}

// Header of a binary graph file (InputsOutput/loadBinary.cpp:26-30).
static int read_binary_header(FILE *f, long *nv, long *ne, long *weighted) {
  long h[3];
  if (fread(h, sizeof(long), 3, f) != 3) return fail(GLV_ERR_IO, "short binary header");
  if (h[0] < 0 || h[1] < 0) return fail(GLV_ERR_IO, "negative sizes in the binary header");
  *nv = h[0];
  *ne = h[1];
  *weighted = h[2];
  return GLV_OK;
}

}  // namespace glv

extern "C" {

int glv_remove_edges(long NV, long NE, glv_edge *edgeList, long *numGoodEdges) {
  if (NV < 0 || NE < 0 || (!edgeList && NE > 0)) return fail(GLV_ERR_ARG, "bad arguments");
  if (NV > (long)kIdMask) return fail(GLV_ERR_TOO_LARGE, "NV >= 2^31");
  Call c;
  TRY(open_stream(c));
  DevScratch d(c.s);
  glv_edge *din, *dout;
  TRY(upload_edges(c.s, edgeList, NE, d, &din));
  int64_t *order = nullptr, nge = 0;
  if (NE > 0) TRY(kept_order(c.s, NV, NE, aos_view(din), d, &order, &nge, &c.launches));
  if (nge > 0) {
    TRY(d.get(&dout, nge));
    k_gather_edges<<<csr_grid(nge), 256, 0, c.s>>>(nge, order, din, dout);
    ++c.launches;
    CK(cudaGetLastError());
    TRY(d2h_large(c.s, edgeList, dout, nge * (int64_t)sizeof(glv_edge)));
  }
  CK(cudaStreamSynchronize(c.s));
  g_launches += c.launches;
  if (numGoodEdges) *numGoodEdges = (long)nge;
  return GLV_OK;
}

int glv_sort_edges_undirected(long NV, long NE, const glv_edge *list1, glv_edge *list2,
                              long *ptrs) {
  if (NV < 0 || NE < 0 || !ptrs || (NE > 0 && (!list1 || !list2)))
    return fail(GLV_ERR_ARG, "bad arguments");
  if (NV > (long)kIdMask) return fail(GLV_ERR_TOO_LARGE, "NV >= 2^31");
  Call c;
  TRY(open_stream(c));
  DevScratch d(c.s);
  glv_edge *din, *dout;
  int64_t *dptr;
  TRY(upload_edges(c.s, list1, NE, d, &din));
  TRY(d.get(&dptr, NV + 1));
  TRY(d.get(&dout, 2 * NE));
  TRY(row_entries(c.s, NV, NE, nullptr, aos_view(din), false, d, dptr, nullptr, nullptr, dout,
                  &c.launches));
  TRY(d2h_large(c.s, list2, dout, 2 * NE * (int64_t)sizeof(glv_edge)));
  CK(cudaMemcpyAsync(ptrs, dptr, (NV + 1) * sizeof(long), cudaMemcpyDeviceToHost, c.s));
  CK(cudaStreamSynchronize(c.s));
  ptrs[NV + 1] = 2 * NE;  // the reference's shifted histogram leaves 2*NE here
  g_launches += c.launches;
  return GLV_OK;
}

int glv_sort_node_edges_by_index(long NV, glv_edge *list1, glv_edge *list2, const long *ptrs) {
  (void)list2;
  TRY(check_ptr(NV, ptrs));
  const int64_t nnz = ptrs[NV];
  if (nnz > 0 && !list1) return fail(GLV_ERR_ARG, "list1 is NULL");
  Call c;
  TRY(open_stream(c));
  DevScratch d(c.s);
  glv_edge *din, *dout;
  int64_t *dptr, *rowid, *v1, *v2;
  uint64_t *k1, *k2;
  int32_t *bad;
  TRY(upload_edges(c.s, list1, nnz, d, &din));
  TRY(d.get(&dptr, NV + 1));
  TRY(d.get(&rowid, nnz));
  TRY(d.get(&k1, nnz));
  TRY(d.get(&k2, nnz));
  TRY(d.get(&v1, nnz));
  TRY(d.get(&v2, nnz));
  TRY(d.get(&bad, 1));
  TRY(d.get(&dout, nnz));
  CK(cudaMemsetAsync(bad, 0, sizeof(int32_t), c.s));
  CK(cudaMemcpyAsync(dptr, ptrs, (NV + 1) * sizeof(long), cudaMemcpyHostToDevice, c.s));
  if (nnz > 0) {
    k_row_ids<<<grid_for(NV * 32, 256, 148 * 16), 256, 0, c.s>>>(NV, dptr, rowid);
    k_row_sort_keys<<<csr_grid(nnz), 256, 0, c.s>>>(nnz, rowid, din, k1, v1, bad);
    c.launches += 2;
    CK(cudaGetLastError());
    size_t tb = 0;
    const int bits = kIdBits + id_bits(NV);
    CK(cub::DeviceRadixSort::SortPairs(nullptr, tb, k1, k2, v1, v2, nnz, 0, bits, c.s));
    void *temp;
    TRY(d.get((char **)&temp, (int64_t)tb));
    CK(cub::DeviceRadixSort::SortPairs(temp, tb, k1, k2, v1, v2, nnz, 0, bits, c.s));
    k_gather_edges<<<csr_grid(nnz), 256, 0, c.s>>>(nnz, v2, din, dout);
    ++c.launches;
    CK(cudaGetLastError());
    int32_t hb = 0;
    CK(cudaMemcpyAsync(&hb, bad, sizeof(hb), cudaMemcpyDeviceToHost, c.s));
    CK(cudaStreamSynchronize(c.s));
    if (hb) return fail(GLV_ERR_ARG, "a tail is outside [0, 2^31)");
    TRY(d2h_large(c.s, list1, dout, nnz * (int64_t)sizeof(glv_edge)));
  }
  CK(cudaStreamSynchronize(c.s));
  g_launches += c.launches;
  return GLV_OK;
}

int glv_build_csr(long NV, long NE, const glv_edge *edges, int flags, glv_graph *Gout) {
  if (NV < 0 || NE < 0 || !Gout || (!edges && NE > 0)) return fail(GLV_ERR_ARG, "bad arguments");
  if (NV > (long)kIdMask) return fail(GLV_ERR_TOO_LARGE, "NV >= 2^31");
  if (flags & ~(GLV_CSR_REMOVE_EDGES | GLV_CSR_SORT_ROWS)) return fail(GLV_ERR_ARG, "bad flags");
  Call c;
  TRY(open_stream(c));
  DevScratch d(c.s);
  glv_edge *din, *dout;
  int64_t *dptr, *order = nullptr, nk = NE;
  TRY(upload_edges(c.s, edges, NE, d, &din));
  TRY(d.get(&dptr, NV + 1));
  const bool merge = merges_rows(flags, NE);
  KeptSorted ks;
  if (merge) {
    TRY(kept_sorted(c.s, NV, NE, aos_view(din), d, &ks, &c.launches));
    nk = ks.nge;
  } else if (NE > 0 && (flags & GLV_CSR_REMOVE_EDGES)) {
    TRY(kept_order(c.s, NV, NE, aos_view(din), d, &order, &nk, &c.launches));
  }
  const int64_t m = 2 * nk;
  TRY(d.get(&dout, m));
  if (merge)
    TRY(merged_rows(c.s, NV, ks, aos_view(din), d, dptr, nullptr, nullptr, dout, &c.launches));
  else
    TRY(row_entries(c.s, NV, nk, order, aos_view(din), (flags & GLV_CSR_SORT_ROWS) != 0, d, dptr,
                    nullptr, nullptr, dout, &c.launches));
  long *hp = (long *)malloc((NV + 1) * sizeof(long));
  glv_edge *he = (glv_edge *)malloc(std::max<int64_t>(m, 1) * sizeof(glv_edge));
  if (!hp || !he) {
    free(hp);
    free(he);
    return fail(GLV_ERR_OOM, "host allocation failed");
  }
  int rc = d2h_large(c.s, hp, dptr, (NV + 1) * sizeof(long));
  if (rc == GLV_OK) rc = d2h_large(c.s, he, dout, m * (int64_t)sizeof(glv_edge));
  if (rc != GLV_OK) {
    free(hp);
    free(he);
    return rc;
  }
  g_launches += c.launches;
  Gout->numVertices = NV;
  Gout->sVertices = NV;
  Gout->numEdges = nk;
  Gout->edgeListPtrs = hp;
  Gout->edgeList = he;
  return GLV_OK;
}

int glv_dev_build_csr(long NV, long NE, const long *d_head, const long *d_tail,
                      const double *d_weight, int flags, long *d_ptr, int *d_tail_out,
                      double *d_weight_out, long *nnz, void *stream) {
  if (NV < 0 || NE < 0 || !d_ptr || (NE > 0 && (!d_head || !d_tail || !d_tail_out || !d_weight_out)))
    return fail(GLV_ERR_ARG, "bad arguments");
  if (NV > (long)kIdMask) return fail(GLV_ERR_TOO_LARGE, "NV >= 2^31");
  if (flags & ~(GLV_CSR_REMOVE_EDGES | GLV_CSR_SORT_ROWS)) return fail(GLV_ERR_ARG, "bad flags");
  TRY(device_ready());
  if (!engine_pool()) return fail(GLV_ERR_CUDA, "could not create the device memory pool");
  cudaStream_t s = (cudaStream_t)stream;
  long launches = 0;
  int64_t *order = nullptr, nk = NE;
  const EdgeView ev{reinterpret_cast<const int64_t *>(d_head),
                    reinterpret_cast<const int64_t *>(d_tail), d_weight, 1};
  {
    DevScratch d(s);
    // the merge reads the weights while it writes: not in place
    const bool in_place = overlap(d_weight, NE * 8, d_ptr, (NV + 1) * 8) ||
                          overlap(d_weight, NE * 8, d_tail_out, 2 * NE * 4) ||
                          overlap(d_weight, NE * 8, d_weight_out, 2 * NE * 8);
    if (merges_rows(flags, NE) && !in_place) {
      KeptSorted ks;
      TRY(kept_sorted(s, NV, NE, ev, d, &ks, &launches));
      nk = ks.nge;
      TRY(merged_rows(s, NV, ks, ev, d, reinterpret_cast<int64_t *>(d_ptr), d_tail_out,
                      d_weight_out, nullptr, &launches));
    } else {
      if (NE > 0 && (flags & GLV_CSR_REMOVE_EDGES))
        TRY(kept_order(s, NV, NE, ev, d, &order, &nk, &launches));
      TRY(row_entries(s, NV, nk, order, ev, (flags & GLV_CSR_SORT_ROWS) != 0, d,
                      reinterpret_cast<int64_t *>(d_ptr), d_tail_out, d_weight_out, nullptr,
                      &launches));
    }
  }
  CK(cudaStreamSynchronize(s));
  g_launches += launches;
  if (nnz) *nnz = 2 * nk;
  return GLV_OK;
}

int glv_binary_header(const char *path, long *numVertices, long *numEdges, long *weighted) {
  FILE *f = open_binary(path, "rb");
  if (!f) return fail(GLV_ERR_IO, "cannot open the binary file");
  long nv, ne, wt;
  const int rc = read_binary_header(f, &nv, &ne, &wt);
  fclose(f);
  TRY(rc);
  if (numVertices) *numVertices = nv;
  if (numEdges) *numEdges = ne;
  if (weighted) *weighted = wt;
  return GLV_OK;
}

int glv_load_binary(const char *path, glv_graph *G) {
  if (!G) return fail(GLV_ERR_ARG, "G is NULL");
  FILE *f = open_binary(path, "rb");
  if (!f) return fail(GLV_ERR_IO, "cannot open the binary file");
  long nv, ne, wt;
  int rc = read_binary_header(f, &nv, &ne, &wt);
  if (rc != GLV_OK) {
    fclose(f);
    return rc;
  }
  long *p = (long *)malloc((nv + 1) * sizeof(long));
  glv_edge *e = (glv_edge *)malloc(std::max<long>(2 * ne, 1) * sizeof(glv_edge));
  if (!p || !e) {
    fclose(f);
    free(p);
    free(e);
    return fail(GLV_ERR_OOM, "host allocation failed");
  }
  const bool ok = fread(p, sizeof(long), nv + 1, f) == (size_t)(nv + 1) &&
                  fread(e, sizeof(glv_edge), 2 * ne, f) == (size_t)(2 * ne);
  fclose(f);
  if (!ok) {
    free(p);
    free(e);
    return fail(GLV_ERR_IO, "binary file shorter than its header says");
  }
  G->numVertices = nv;
  G->sVertices = nv;
  G->numEdges = ne;
  G->edgeListPtrs = p;
  G->edgeList = e;
  return GLV_OK;
}

int glv_write_binary(const glv_graph *G, const char *path, long weighted) {
  if (!G || G->numVertices < 0 || !G->edgeListPtrs) return fail(GLV_ERR_ARG, "bad graph");
  FILE *f = open_binary(path, "wb");
  if (!f) return fail(GLV_ERR_IO, "cannot create the binary file");
  const long h[3] = {G->numVertices, G->numEdges, weighted};
  const long n2 = 2 * G->numEdges;  // the reference writes 2 * numEdges entries
  bool ok = fwrite(h, sizeof(long), 3, f) == 3 &&
            fwrite(G->edgeListPtrs, sizeof(long), G->numVertices + 1, f) ==
                (size_t)(G->numVertices + 1) &&
            (n2 == 0 || fwrite(G->edgeList, sizeof(glv_edge), n2, f) == (size_t)n2);
  ok = (fclose(f) == 0) && ok;
  return ok ? GLV_OK : fail(GLV_ERR_IO, "write to the binary file failed");
}

int glv_dev_load_binary(const char *path, long numVertices, long nnz, long *d_ptr, int *d_tail,
                        double *d_weight, void *stream) {
  if (numVertices < 0 || nnz < 0 || !d_ptr || (nnz > 0 && (!d_tail || !d_weight)))
    return fail(GLV_ERR_ARG, "bad arguments");
  if (numVertices > (long)kIdMask) return fail(GLV_ERR_TOO_LARGE, "numVertices >= 2^31");
  TRY(device_ready());
  if (!engine_pool()) return fail(GLV_ERR_CUDA, "could not create the device memory pool");
  FILE *f = open_binary(path, "rb");
  if (!f) return fail(GLV_ERR_IO, "cannot open the binary file");
  struct Closer {
    FILE *f;
    ~Closer() { fclose(f); }
  } closer{f};
  long nv, ne, wt;
  TRY(read_binary_header(f, &nv, &ne, &wt));
  if (nv != numVertices || 2 * ne != nnz)
    return fail(GLV_ERR_ARG, "numVertices / nnz differ from the file's header");
  cudaStream_t s = (cudaStream_t)stream;
  std::vector<long> ptr(nv + 1);
  if (fread(ptr.data(), sizeof(long), nv + 1, f) != (size_t)(nv + 1))
    return fail(GLV_ERR_IO, "binary file shorter than its header says");
  if (ptr[0] != 0 || ptr[nv] != nnz) return fail(GLV_ERR_IO, "row offsets do not span 2*NE");
  for (long v = 0; v < nv; ++v)
    if (ptr[v + 1] < ptr[v]) return fail(GLV_ERR_IO, "row offsets decrease");
  CK(cudaMemcpyAsync(d_ptr, ptr.data(), (nv + 1) * sizeof(long), cudaMemcpyHostToDevice, s));
  // Entries stream through two pinned buffers: the file read of one chunk
  // overlaps the copy and split of the previous one.
  const int64_t chunk = std::min<int64_t>(std::max<int64_t>(nnz, 1), int64_t(1) << 22);
  glv_edge *pin[2] = {nullptr, nullptr};
  cudaEvent_t done[2] = {nullptr, nullptr};
  struct PinGuard {
    glv_edge **p;
    cudaEvent_t *ev;
    ~PinGuard() {
      for (int k = 0; k < 2; ++k) {
        if (ev[k]) {
          cudaEventSynchronize(ev[k]);
          cudaEventDestroy(ev[k]);
        }
        if (p[k]) cudaFreeHost(p[k]);
      }
    }
  } guard{pin, done};
  for (int k = 0; k < 2; ++k) {
    CK(cudaHostAlloc((void **)&pin[k], chunk * sizeof(glv_edge), cudaHostAllocDefault));
    CK(cudaEventCreateWithFlags(&done[k], cudaEventDisableTiming));
  }
  long launches = 0;
  int32_t hbad = 0;
  {
    DevScratch d(s);
    glv_edge *stage[2];
    int32_t *bad;
    TRY(d.get(&stage[0], chunk));
    TRY(d.get(&stage[1], chunk));
    TRY(d.get(&bad, 1));
    CK(cudaMemsetAsync(bad, 0, sizeof(int32_t), s));
    int k = 0;
    for (int64_t b = 0; b < nnz; b += chunk, k ^= 1) {
      const int64_t n = std::min(chunk, nnz - b);
      CK(cudaEventSynchronize(done[k]));  // the buffer's previous copy has finished
      if (fread(pin[k], sizeof(glv_edge), n, f) != (size_t)n)
        return fail(GLV_ERR_IO, "binary file shorter than its header says");
      CK(cudaMemcpyAsync(stage[k], pin[k], n * sizeof(glv_edge), cudaMemcpyHostToDevice, s));
      CK(cudaEventRecord(done[k], s));
      k_split_checked<<<csr_grid(n), 256, 0, s>>>(n, stage[k], nv, d_tail + b, d_weight + b, bad);
      ++launches;
      CK(cudaGetLastError());
    }
    CK(cudaMemcpyAsync(&hbad, bad, sizeof(hbad), cudaMemcpyDeviceToHost, s));
    CK(cudaStreamSynchronize(s));
  }
  g_launches += launches;
  if (hbad) return fail(GLV_ERR_IO, "a tail in the binary file is outside [0, NV)");
  return GLV_OK;
}

}  // extern "C"
