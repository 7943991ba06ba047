// Comparing two community assignments (Utility/utilityClusterComparisonMetrics.cpp).
//
// computeCommunityComparisons (:50-307) counts, over every pair of vertices
// in one community of C1 (the truth), those in one community of C2 too
// (SameSame, true positives) or not (SameDiff, false negatives), and over
// every pair in one community of C2, those split by C1 (DiffSame, false
// positives) -- by enumerating the pairs, quadratic in community size.  The
// same integers come from the contingency table of (C1, C2) labels:
//
//   SameSame = sum over label pairs (a, b) of C(n_ab, 2)
//   SameDiff = sum over a of C(n_a, 2) - SameSame
//   DiffSame = sum over b of C(n_b, 2) - SameSame
//
// Here: one kernel relabels as the reference does (-1 entries, 0- or 1-based
// ids) and histograms both sides; the n_ab are counted community by community in
// shared memory, or, where communities are too large or too many, by a radix
// sort of the (a, b) keys and a run-length encode.  The Gini coefficient of each side's
// community sizes (computeGiniCoefficient, :310-330) sorts the sizes and takes
// sum (i + 1) * size_i in exact 64-bit integers (the reference's FP64 running
// sum is exact, and so equal, while it stays below 2^53).
//
// Included into engine.cu after csr_build.cuh (DevScratch, staged copies).

namespace glv {

// Max, zero and -1 presence, and ids below -1, of one label array.  When
// `minus_one_as` >= 0 a -1 counts as that value (C2's rule, :92-93).
__global__ void k_label_stats(int64_t n, const int64_t *C, int64_t minus_one_as,
                              long long *mx, int32_t *flags) {
  long long m = LLONG_MIN;
  int f = 0;
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n;
       i += (int64_t)gridDim.x * blockDim.x) {
    int64_t c = C[i];
    if (c == -1) {
      f |= 2;
      if (minus_one_as < 0) continue;
      c = minus_one_as;
    } else if (c < -1) {
      f |= 4;
      continue;
    }
    if (c == 0) f |= 1;
    m = c > m ? c : m;
  }
  for (int off = 16; off; off >>= 1) {
    m = max(m, (long long)__shfl_xor_sync(FULL, m, off));
    f |= __shfl_xor_sync(FULL, f, off);
  }
  if ((threadIdx.x & 31) == 0) {
    if (m != LLONG_MIN) atomicMax(mx, m);
    if (f) atomicOr(flags, f);
  }
}

// One more vertex in each lane's community: hist[g] grows, the old values are
// returned (lanes without a vertex pass valid = false).  The vertices of the
// community the warp has met most often (hot, kept between calls) are added at
// once: one address takes its adds one after another, and labels come in runs
// or with one community that holds a large part (20M vertices of one community:
// the comparison 25 ms with an add per vertex, 1.4 with these).
__device__ __forceinline__ unsigned long long label_count(unsigned long long *hist, int64_t g,
                                                          bool valid, int64_t &hot) {
  const int lane = threadIdx.x & 31;
  const int64_t g0 = __shfl_sync(FULL, g, 0);
  const unsigned m0 = __ballot_sync(FULL, valid && g == g0);
  unsigned mh = __ballot_sync(FULL, valid && g == hot);
  if (__popc(m0) > __popc(mh)) {
    hot = g0;
    mh = m0;
  }
  const bool in_hot = mh >> lane & 1;
  const int leader = __ffs(mh) - 1;  // -1: no lane meets it
  unsigned long long r = 0;
  if (valid && (!in_hot || lane == leader))
    r = atomicAdd(&hist[g], in_hot ? (unsigned long long)__popc(mh) : 1ull);
  const unsigned long long base = __shfl_sync(FULL, r, max(leader, 0));
  return in_hot ? base + __popc(mh & ((1u << lane) - 1)) : r;
}

// Relabel in place as the reference does (C1: -1 -> fill1, C2: -1 -> fill2),
// map ids to community indices (minus one for 1-based ids) and histogram them;
// either the contingency keys (a above b) go to keys, or the vertices' places
// in their communities of one side (by2: C2's) to rank.
__global__ void k_label_pairs(int64_t n, int64_t *C1, int64_t *C2, int64_t fill1, int64_t fill2,
                              int64_t base1, int64_t base2, int bits2,
                              unsigned long long *hist1, unsigned long long *hist2,
                              uint64_t *keys, int32_t *rank, bool by2) {
  const int lane = threadIdx.x & 31;
  int64_t hot1 = -1, hot2 = -1;
  for (int64_t i0 = (int64_t)blockIdx.x * blockDim.x + threadIdx.x - lane; i0 < n;
       i0 += (int64_t)gridDim.x * blockDim.x) {
    const int64_t i = i0 + lane;
    const bool valid = i < n;
    int64_t a = base1, b = base2;
    if (valid) {
      a = C1[i];
      b = C2[i];
      if (a == -1) C1[i] = a = fill1;
      if (b == -1) C2[i] = b = fill2;
    }
    a -= base1;
    b -= base2;
    const unsigned long long r1 = label_count(hist1, a, valid, hot1);
    const unsigned long long r2 = label_count(hist2, b, valid, hot2);
    if (!valid) continue;
    if (rank) rank[i] = (int32_t)(by2 ? r2 : r1);
    else keys[i] = ((uint64_t)a << bits2) | (uint64_t)b;
  }
}

// ---- n_ab by community ----------------------------------------------------
// The label pairs of one community a of a side are counted where the other
// side's labels b of its vertices stand together: a pair's count grows by one at
// a time, and the old counts sum to C(n_ab, 2).  Bound by the label pass's
// atomics and the random 4-byte writes of the grouping; a radix sort of all
// (a, b) keys and a run-length encode moved five times the bytes (20M vertices in
// communities of 150, labels shuffled: 1.88 ms, this way 1.04).
constexpr int kGroupWarp = 384;    // most vertices of a community on one warp: 512 slots
constexpr int kGroupBlock = 6144;  // on a block: 8192 slots; larger ones are sorted

// other[off[g] + rank] = the other side's community of each vertex.
__global__ void k_group_labels(int64_t n, const int64_t *Cg, const int64_t *Co, int64_t baseg,
                               int64_t baseo, const int64_t *off, const int32_t *rank,
                               int32_t *other) {
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n;
       i += (int64_t)gridDim.x * blockDim.x)
    other[off[Cg[i] - baseg] + rank[i]] = (int32_t)(Co[i] - baseo);
}

// Counts one label per lane (b < 0: none) in an open table; returns the pairs
// it closed.  Lanes with lane 0's label count as one: most of a community's
// vertices usually share theirs.
__device__ __forceinline__ unsigned long long group_add(int32_t b, int32_t *key, uint32_t *cnt,
                                                        uint32_t mask) {
  const int32_t b0 = __shfl_sync(FULL, b, 0);
  const unsigned same = __ballot_sync(FULL, b >= 0 && b == b0);
  const int lane = threadIdx.x & 31;
  if (b < 0 || ((same >> lane & 1) && lane != 0)) return 0;
  const uint32_t m = lane == 0 ? (uint32_t)__popc(same) : 1u;
  uint32_t h = hash_slot((uint32_t)b, mask);
  for (;;) {  // ends: the table has more slots than the community has vertices
    const int32_t k = atomicCAS(&key[h], -1, b);
    if (k == -1 || k == b) break;
    h = (h + 1) & mask;
  }
  const unsigned long long old = atomicAdd(&cnt[h], m);
  return old * m + (unsigned long long)m * (m - 1) / 2;
}

// A power of two of slots, at least 4/3 of the vertices.
__device__ __forceinline__ int group_slots(int size) {
  int s = 64;
  while (3 * s < 4 * size) s <<= 1;
  return s;
}

// Communities of up to kGroupWarp vertices, one per warp; larger ones are
// listed: *nblock for blocks; for sorting with the vertices listed before, and
// *total counts both the communities (from kSortCount up) and their vertices.
constexpr int kSortShift = 34;  // vertices stay below 2^30
constexpr unsigned long long kSortCount = 1ull << kSortShift;

__global__ void __launch_bounds__(256) k_group_pairs_warp(
    int64_t nC, const unsigned long long *size, const int64_t *off, const int32_t *other,
    unsigned long long *out, int32_t *list_block, int32_t *list_sort, int32_t *sort_start,
    int32_t *nblock, unsigned long long *total) {
  __shared__ int32_t s_key[8][512];
  __shared__ uint32_t s_cnt[8][512];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  int32_t *key = s_key[warp];
  uint32_t *cnt = s_cnt[warp];
  unsigned long long acc = 0;
  for (int64_t c = (int64_t)blockIdx.x * 8 + warp; c < nC; c += (int64_t)gridDim.x * 8) {
    const unsigned long long n = size[c];
    if (n < 2) continue;
    if (n > kGroupWarp) {
      if (lane == 0) {
        if (n <= kGroupBlock) {
          list_block[atomicAdd(nblock, 1)] = (int32_t)c;
        } else {
          const unsigned long long at = atomicAdd(total, kSortCount | n);
          list_sort[at >> kSortShift] = (int32_t)c;
          sort_start[at >> kSortShift] = (int32_t)(at & (kSortCount - 1));
        }
      }
      continue;
    }
    const int m = (int)n, slots = group_slots(m);
    for (int k = lane; k < slots; k += 32) {
      key[k] = -1;
      cnt[k] = 0;
    }
    __syncwarp();
    const int32_t *lab = other + off[c];
    for (int k = 0; k < m; k += 32)
      acc += group_add(k + lane < m ? lab[k + lane] : -1, key, cnt, slots - 1);
    __syncwarp();
  }
  for (int o = 16; o; o >>= 1) acc += __shfl_xor_sync(FULL, acc, o);
  if (lane == 0 && acc) atomicAdd(out, acc);
}

// The listed communities of up to kGroupBlock vertices, one per block.
__global__ void __launch_bounds__(512) k_group_pairs_block(
    const unsigned long long *size, const int64_t *off, const int32_t *other,
    const int32_t *list, const int32_t *nblock, unsigned long long *out) {
  extern __shared__ int32_t s_table[];
  unsigned long long acc = 0;
  const int lane = threadIdx.x & 31, nl = *nblock;
  for (int t = blockIdx.x; t < nl; t += gridDim.x) {
    const int32_t c = list[t];
    const int m = (int)size[c], slots = group_slots(m);
    int32_t *key = s_table;
    uint32_t *cnt = reinterpret_cast<uint32_t *>(s_table + slots);
    for (int k = threadIdx.x; k < slots; k += 512) {
      key[k] = -1;
      cnt[k] = 0;
    }
    __syncthreads();
    const int32_t *lab = other + off[c];
    for (int k = threadIdx.x - lane; k < m; k += 512)
      acc += group_add(k + lane < m ? lab[k + lane] : -1, key, cnt, slots - 1);
    __syncthreads();
  }
  for (int o = 16; o; o >>= 1) acc += __shfl_xor_sync(FULL, acc, o);
  if (lane == 0 && acc) atomicAdd(out, acc);
}

// The keys (community above label) of the nl communities listed for sorting, of
// `left` vertices: a block takes 8192 places of the whole list, which are at most
// three communities.  (All blocks over each community in turn left one or two
// of them busy: 20M vertices in communities of 3000 to 9000 13.9 ms, now 1.25.)
__global__ void __launch_bounds__(512) k_group_keys(const unsigned long long *size,
                                                    const int64_t *off, const int32_t *other,
                                                    const int32_t *list, const int32_t *start,
                                                    int nl, int64_t left, int bits,
                                                    uint64_t *keys) {
  for (int64_t p0 = (int64_t)blockIdx.x * 8192; p0 < left; p0 += (int64_t)gridDim.x * 8192) {
    const int64_t p1 = min(left, p0 + 8192);
    int lo = 0, hi = nl - 1;  // the community that holds place p0
    while (lo < hi) {
      const int mid = (lo + hi + 1) >> 1;
      if (start[mid] <= p0) lo = mid; else hi = mid - 1;
    }
    for (int t = lo; t < nl && start[t] < p1; ++t) {
      const int32_t c = list[t];
      const int64_t b = start[t], e = b + (int64_t)size[c];
      const int32_t *lab = other + off[c];
      for (int64_t p = max(b, p0) + threadIdx.x; p < min(e, p1); p += 512)
        keys[p] = ((uint64_t)c << bits) | (uint32_t)lab[p - b];
    }
  }
}

// sum of C(n_k, 2) over counts n_k (32- or 64-bit counts).
template <class T>
__global__ void k_pair_sum(int64_t m, const T *counts, unsigned long long *out) {
  unsigned long long acc = 0;
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < m;
       i += (int64_t)gridDim.x * blockDim.x) {
    const unsigned long long c = (unsigned long long)counts[i];
    acc += c * (c - (c > 0 ? 1 : 0)) / 2;
  }
  for (int off = 16; off; off >>= 1) acc += __shfl_xor_sync(FULL, acc, off);
  if ((threadIdx.x & 31) == 0 && acc) atomicAdd(out, acc);
}

// out[0] += sum over the ascending sizes of (i + 1) * size_i, out[1] += the
// sum of the sizes.
__global__ void k_gini_sums(int64_t m, const unsigned long long *sorted, unsigned long long *out) {
  unsigned long long num = 0, den = 0;
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < m;
       i += (int64_t)gridDim.x * blockDim.x) {
    num += (unsigned long long)(i + 1) * sorted[i];
    den += sorted[i];
  }
  for (int off = 16; off; off >>= 1) {
    num += __shfl_xor_sync(FULL, num, off);
    den += __shfl_xor_sync(FULL, den, off);
  }
  if ((threadIdx.x & 31) == 0) {
    if (num) atomicAdd(out, num);
    if (den) atomicAdd(out + 1, den);
  }
}

// computeGiniCoefficient's closing expression (:323), on the exact sums.
static double gini_from(unsigned long long num, unsigned long long den, int numColors) {
  const double numFunc = (double)num, denFunc = (double)den;
  return ((2 * numFunc) / (numColors * denFunc)) - ((double)(numColors + 1) / (double)numColors);
}

// Sizes sorted ascending (into *sorted) and the Gini sums of them
// (device sums[0] += numerator, sums[1] += total); sizes take at most `bits` bits.
static int gini_sums(cudaStream_t s, const unsigned long long *sizes, int64_t m, int bits,
                     DevScratch &d, unsigned long long **sorted, unsigned long long *sums,
                     long *launches) {
  TRY(d.get(sorted, m));
  size_t tb = 0;
  CK(cub::DeviceRadixSort::SortKeys(nullptr, tb, sizes, *sorted, m, 0, bits, s));
  void *temp;
  TRY(d.get((char **)&temp, (int64_t)tb));
  CK(cub::DeviceRadixSort::SortKeys(temp, tb, sizes, *sorted, m, 0, bits, s));
  k_gini_sums<<<csr_grid(m), 256, 0, s>>>(m, *sorted, sums);
  ++*launches;
  CK(cudaGetLastError());
  return GLV_OK;
}

// acc[0] += sum of C(n, 2) over the m keys' multiplicities; *keys is used up.
static int sorted_pairs(cudaStream_t s, int64_t m, int bits, uint64_t *keys, DevScratch &d,
                        unsigned long long *acc, long *launches) {
  uint64_t *k2, *uniq;
  int64_t *counts, *nruns;
  TRY(d.get(&k2, m));
  TRY(d.get(&uniq, m));
  TRY(d.get(&counts, m));
  TRY(d.get(&nruns, 1));
  size_t tb = 0, tb2 = 0;
  CK(cub::DeviceRadixSort::SortKeys(nullptr, tb, keys, k2, m, 0, bits, s));
  CK(cub::DeviceRunLengthEncode::Encode(nullptr, tb2, k2, uniq, counts, nruns, m, s));
  void *temp;
  TRY(d.get((char **)&temp, (int64_t)std::max(tb, tb2)));
  CK(cub::DeviceRadixSort::SortKeys(temp, tb, keys, k2, m, 0, bits, s));
  CK(cub::DeviceRunLengthEncode::Encode(temp, tb2, k2, uniq, counts, nruns, m, s));
  int64_t hr = 0;
  CK(cudaMemcpyAsync(&hr, nruns, sizeof(hr), cudaMemcpyDeviceToHost, s));
  CK(cudaStreamSynchronize(s));
  k_pair_sum<<<csr_grid(hr), 256, 0, s>>>(hr, counts, acc);
  ++*launches;
  CK(cudaGetLastError());
  return GLV_OK;
}

// Whether the pairs are counted by a side's nC communities.  Not
// with less than two vertices an id (singletons, ids with gaps), where both ways
// take the same time and this one the memory of an offset per id; not where a
// community is too large for a block even on average; and below 2^30 vertices,
// so that sorting every community after all still fits the scratch that
// sorting all keys takes at 2^31.  20M vertices, 20 % noise: communities of 20 1.91
// -> 1.09 ms, of 150 1.93 -> 0.70, of 5000 1.95 -> 0.75; skewed sizes (k-th label
// by u^6, most vertices sorted after all) 4.80 -> 3.21, 3000 to 9000 2.03 -> 1.25.
static bool counts_by_community(int64_t n, int64_t nC) {
  return n < (int64_t(1) << 30) && nC <= n / 2 && n / nC <= kGroupBlock;
}

// One side's vertices by community.
struct LabelGroups {
  int64_t nC = 0;
  const unsigned long long *size = nullptr;
  int64_t *off = nullptr;
  int32_t *other = nullptr, *list_block = nullptr, *nblock = nullptr;
  int32_t *list_sort = nullptr, *sort_start = nullptr;
};

// *pairs += sum of C(n_ab, 2) over the communities of up to kGroupBlock vertices of
// the side with g->nC communities of g->size (labels Cg); rank from
// k_label_pairs.  *total counts the larger ones (k_group_pairs_warp).
static int grouped_pairs(cudaStream_t s, int64_t n, const int64_t *Cg, const int64_t *Co,
                         int64_t baseg, int64_t baseo, const int32_t *rank, DevScratch &d,
                         LabelGroups *g, unsigned long long *pairs, unsigned long long *total,
                         long *launches) {
  const int64_t most_block = n / (kGroupWarp + 1) + 1;
  TRY(d.get(&g->off, g->nC));
  TRY(d.get(&g->other, n));
  TRY(d.get(&g->list_block, most_block));
  TRY(d.get(&g->list_sort, n / (kGroupBlock + 1) + 1));
  TRY(d.get(&g->sort_start, n / (kGroupBlock + 1) + 1));
  TRY(d.get(&g->nblock, 1));
  CK(cudaMemsetAsync(g->nblock, 0, sizeof(int32_t), s));
  const int64_t *size = reinterpret_cast<const int64_t *>(g->size);
  size_t tb = 0;
  CK(cub::DeviceScan::ExclusiveSum(nullptr, tb, size, g->off, g->nC, s));
  void *temp;
  TRY(d.get((char **)&temp, (int64_t)tb));
  CK(cub::DeviceScan::ExclusiveSum(temp, tb, size, g->off, g->nC, s));
  k_group_labels<<<csr_grid(n), 256, 0, s>>>(n, Cg, Co, baseg, baseo, g->off, rank, g->other);
  k_group_pairs_warp<<<(unsigned)std::min<int64_t>((g->nC + 7) / 8, 148 * 6), 256, 0, s>>>(
      g->nC, g->size, g->off, g->other, pairs, g->list_block, g->list_sort, g->sort_start,
      g->nblock, total);
  const int smem = 8192 * 8;
  CK(cudaFuncSetAttribute(k_group_pairs_block, cudaFuncAttributeMaxDynamicSharedMemorySize, smem));
  k_group_pairs_block<<<(unsigned)std::min<int64_t>(most_block, 148 * 3), 512, smem, s>>>(
      g->size, g->off, g->other, g->list_block, g->nblock, pairs);
  *launches += 3;
  CK(cudaGetLastError());
  return GLV_OK;
}

// The comparison on device-resident label arrays (int64, relabelled in place).
static int compare_device(cudaStream_t s, int64_t n, int64_t *dC1, int64_t *dC2, DevScratch &d,
                          glv_comparison *out, long *launches) {
  long long *mx;
  int32_t *fl;
  TRY(d.get(&mx, 2));
  TRY(d.get(&fl, 2));
  const long long lo[2] = {LLONG_MIN, LLONG_MIN};
  CK(cudaMemcpyAsync(mx, lo, sizeof(lo), cudaMemcpyHostToDevice, s));
  CK(cudaMemsetAsync(fl, 0, 2 * sizeof(int32_t), s));
  k_label_stats<<<csr_grid(n), 256, 0, s>>>(n, dC1, -1, mx, fl);
  k_label_stats<<<csr_grid(n), 256, 0, s>>>(n, dC2, n + 1, mx + 1, fl + 1);
  *launches += 2;
  CK(cudaGetLastError());
  long long hmx[2];
  int32_t hfl[2];
  CK(cudaMemcpyAsync(hmx, mx, sizeof(hmx), cudaMemcpyDeviceToHost, s));
  CK(cudaMemcpyAsync(hfl, fl, sizeof(hfl), cudaMemcpyDeviceToHost, s));
  CK(cudaStreamSynchronize(s));
  if ((hfl[0] | hfl[1]) & 4) return fail(GLV_ERR_ARG, "a community id below -1");
  // The -1 entries of the two sides get different values, and the labels are read
  // again after that: arrays that share memory (a labelling against itself) are
  // compared in copies.  Without -1 entries nothing is written.
  int64_t *const home1 = dC1, *const home2 = dC2;
  const bool copies = ((hfl[0] | hfl[1]) & 2) && overlap(dC1, n * 8, dC2, n * 8);
  if (copies) {
    TRY(d.get(&dC1, n));
    TRY(d.get(&dC2, n));
    CK(cudaMemcpyAsync(dC1, home1, n * sizeof(int64_t), cudaMemcpyDeviceToDevice, s));
    CK(cudaMemcpyAsync(dC2, home2, n * sizeof(int64_t), cudaMemcpyDeviceToDevice, s));
  }
  // C1 (:63-87): nC1 = largest id, plus one when 0 is an id; -1 entries
  // become nC1, which then grows by one
  const bool z1 = hfl[0] & 1, z2 = hfl[1] & 1;
  int64_t nC1 = (hmx[0] == LLONG_MIN ? -1 : hmx[0]) + (z1 ? 1 : 0);
  const int64_t fill1 = nC1;
  if (hfl[0] & 2) ++nC1;
  // C2 (:89-113): -1 entries become N2 + 1 before the count
  const int64_t nC2 = (int64_t)hmx[1] + (z2 ? 1 : 0);
  if (nC1 <= 0 || nC2 <= 0) return fail(GLV_ERR_ARG, "no community ids in C1 or C2");
  const int64_t base1 = z1 ? 0 : 1, base2 = z2 ? 0 : 1;
  if (nC1 > (int64_t)kIdMask + 1 || nC2 > (int64_t)kIdMask + 1)
    return fail(GLV_ERR_TOO_LARGE, "community ids >= 2^31");
  const int bits1 = id_bits(nC1), bits2 = id_bits(nC2);
  unsigned long long *h1, *h2, *acc;
  TRY(d.get(&h1, nC1));
  TRY(d.get(&h2, nC2));
  TRY(d.get(&acc, 8));  // pairs, pairs of C1, of C2, Gini sums of both, left to sort
  CK(cudaMemsetAsync(h1, 0, nC1 * sizeof(*h1), s));
  CK(cudaMemsetAsync(h2, 0, nC2 * sizeof(*h2), s));
  CK(cudaMemsetAsync(acc, 0, 8 * sizeof(*acc), s));
  // the side with more ids has the smaller communities; a -1 in C2 becomes id n +
  // 1, and then C1's ids may still be dense
  const bool ok1 = counts_by_community(n, nC1), ok2 = counts_by_community(n, nC2);
  const bool grouped = ok1 || ok2, by2 = ok2 && (nC2 > nC1 || !ok1);
  uint64_t *keys = nullptr;
  int32_t *rank = nullptr;
  if (grouped) TRY(d.get(&rank, n)); else TRY(d.get(&keys, n));
  k_label_pairs<<<csr_grid(n), 256, 0, s>>>(n, dC1, dC2, fill1, n + 1, base1, base2, bits2, h1,
                                            h2, keys, rank, by2);
  if (copies) {  // C2's values last, as each entry's two stores stand
    CK(cudaMemcpyAsync(home1, dC1, n * sizeof(int64_t), cudaMemcpyDeviceToDevice, s));
    CK(cudaMemcpyAsync(home2, dC2, n * sizeof(int64_t), cudaMemcpyDeviceToDevice, s));
  }
  k_pair_sum<<<csr_grid(nC1), 256, 0, s>>>(nC1, h1, acc + 1);
  k_pair_sum<<<csr_grid(nC2), 256, 0, s>>>(nC2, h2, acc + 2);
  *launches += 3;
  CK(cudaGetLastError());
  unsigned long long *srt, pairs[8];
  // community sizes are at most n: sort only the bits that can be set
  const int size_bits = id_bits(n + 1);
  TRY(gini_sums(s, h1, nC1, size_bits, d, &srt, acc + 3, launches));
  TRY(gini_sums(s, h2, nC2, size_bits, d, &srt, acc + 5, launches));
  LabelGroups g;
  if (grouped) {
    g.nC = by2 ? nC2 : nC1;
    g.size = by2 ? h2 : h1;
    TRY(grouped_pairs(s, n, by2 ? dC2 : dC1, by2 ? dC1 : dC2, by2 ? base2 : base1,
                      by2 ? base1 : base2, rank, d, &g, acc, acc + 7, launches));
  } else {
    TRY(sorted_pairs(s, n, bits1 + bits2, keys, d, acc, launches));
  }
  CK(cudaMemcpyAsync(pairs, acc, sizeof(pairs), cudaMemcpyDeviceToHost, s));
  CK(cudaStreamSynchronize(s));
  if (pairs[7] > 0) {
    const int64_t left = (int64_t)(pairs[7] & (kSortCount - 1));
    TRY(d.get(&keys, left));
    k_group_keys<<<(unsigned)std::min<int64_t>((left + 8191) / 8192, 148 * 4), 512, 0, s>>>(
        g.size, g.off, g.other, g.list_sort, g.sort_start, (int)(pairs[7] >> kSortShift), left,
        by2 ? bits1 : bits2, keys);
    ++*launches;
    CK(cudaGetLastError());
    TRY(sorted_pairs(s, left, bits1 + bits2, keys, d, acc, launches));
    CK(cudaMemcpyAsync(pairs, acc, sizeof(pairs[0]), cudaMemcpyDeviceToHost, s));
    CK(cudaStreamSynchronize(s));
  }
  const long SameSame = (long)pairs[0];
  const long SameDiff = (long)(pairs[1] - pairs[0]);
  const long DiffSame = (long)(pairs[2] - pairs[0]);
  // :258-263, :265-266
  const double precision = (double)SameSame / (double)(SameSame + DiffSame);
  const double recall = (double)SameSame / (double)(SameSame + SameDiff);
  out->n1 = n;
  out->n2 = n;
  out->num_communities1 = nC1;
  out->num_communities2 = nC2;
  out->same_same = SameSame;
  out->same_diff = SameDiff;
  out->diff_same = DiffSame;
  out->precision = precision;
  out->recall = recall;
  out->f_score = 2 * ((precision * recall) / (precision + recall));
  out->gini1 = gini_from(pairs[3], pairs[4], (int)nC1);
  out->gini2 = gini_from(pairs[5], pairs[6], (int)nC2);
  return GLV_OK;
}

}  // namespace glv

extern "C" {

int glv_compare_communities(long *C1, long N1, long *C2, long N2, glv_comparison *out) {
  if (!out || N1 <= 0 || N2 <= 0 || !C1 || !C2) return fail(GLV_ERR_ARG, "bad arguments");
  if (N1 != N2) return fail(GLV_ERR_ARG, "C1 and C2 label different numbers of vertices");
  if (N1 >= (1L << 31) - 2) return fail(GLV_ERR_TOO_LARGE, "N >= 2^31");
  Call c;
  TRY(open_stream(c));
  DevScratch d(c.s);
  int64_t *d1, *d2;
  TRY(d.get(&d1, N1));
  TRY(d.get(&d2, N1));
  TRY(h2d_large(c.s, d1, C1, N1 * (int64_t)sizeof(long)));
  TRY(h2d_large(c.s, d2, C2, N1 * (int64_t)sizeof(long)));
  TRY(compare_device(c.s, N1, d1, d2, d, out, &c.launches));
  TRY(d2h_large(c.s, C1, d1, N1 * (int64_t)sizeof(long)));
  TRY(d2h_large(c.s, C2, d2, N1 * (int64_t)sizeof(long)));
  g_launches += c.launches;
  return GLV_OK;
}

int glv_dev_compare_communities(long n, long *d_C1, long *d_C2, glv_comparison *out,
                                void *stream) {
  if (!out || n <= 0 || !d_C1 || !d_C2) return fail(GLV_ERR_ARG, "bad arguments");
  if (n >= (1L << 31) - 2) return fail(GLV_ERR_TOO_LARGE, "n >= 2^31");
  TRY(device_ready());
  if (!engine_pool()) return fail(GLV_ERR_CUDA, "could not create the device memory pool");
  cudaStream_t s = (cudaStream_t)stream;
  long launches = 0;
  {
    DevScratch d(s);
    TRY(compare_device(s, n, reinterpret_cast<int64_t *>(d_C1), reinterpret_cast<int64_t *>(d_C2),
                       d, out, &launches));
  }
  CK(cudaStreamSynchronize(s));
  g_launches += launches;
  return GLV_OK;
}

int glv_gini_coefficient(long *colorSize, int numColors, double *gini) {
  if (!gini || numColors <= 0 || !colorSize) return fail(GLV_ERR_ARG, "bad arguments");
  Call c;
  TRY(open_stream(c));
  DevScratch d(c.s);
  unsigned long long *dh, *sorted, *acc, sums[2];
  TRY(d.get(&dh, numColors));
  TRY(d.get(&acc, 2));
  CK(cudaMemsetAsync(acc, 0, 2 * sizeof(*acc), c.s));
  CK(cudaMemcpyAsync(dh, colorSize, numColors * sizeof(long), cudaMemcpyHostToDevice, c.s));
  // sizes are counts; a negative one would sort as a huge unsigned value
  long long *mn;
  int32_t *fl;
  TRY(d.get(&mn, 1));
  TRY(d.get(&fl, 1));
  const long long lo = LLONG_MIN;
  CK(cudaMemcpyAsync(mn, &lo, sizeof(lo), cudaMemcpyHostToDevice, c.s));
  CK(cudaMemsetAsync(fl, 0, sizeof(int32_t), c.s));
  k_label_stats<<<csr_grid(numColors), 256, 0, c.s>>>(numColors, (const int64_t *)dh, -1, mn, fl);
  ++c.launches;
  CK(cudaGetLastError());
  int32_t hf = 0;
  CK(cudaMemcpyAsync(&hf, fl, sizeof(hf), cudaMemcpyDeviceToHost, c.s));
  CK(cudaStreamSynchronize(c.s));
  if (hf & 6) return fail(GLV_ERR_ARG, "a negative size");
  TRY(gini_sums(c.s, dh, numColors, 64, d, &sorted, acc, &c.launches));
  CK(cudaMemcpyAsync(sums, acc, sizeof(sums), cudaMemcpyDeviceToHost, c.s));
  // the reference sorts colorSize in place
  CK(cudaMemcpyAsync(colorSize, sorted, numColors * sizeof(long), cudaMemcpyDeviceToHost, c.s));
  CK(cudaStreamSynchronize(c.s));
  *gini = gini_from(sums[0], sums[1], numColors);
  g_launches += c.launches;
  return GLV_OK;
}

}  // extern "C"
