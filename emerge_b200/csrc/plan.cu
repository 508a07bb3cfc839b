// plan.cu -- sparsity pattern and column-gather plan of the Nedelec-2 system.
//
// Replaces CSCMapping.from_rowcol / precompute_csc_pattern (mth/csc_cast.py:51-160)
// for the structured Nedelec-2 pattern: the rows of the columns of entity x
// (edge or face) are the DoFs of every entity that shares an assembled tet
// with x, in four sorted blocks [edges | edges+E | faces+2E | faces+2E+F]
// (the DoF numbering of elements/nedelec2.py:65-79).
#include "common.cuh"

namespace emg {
namespace {

__global__ void k_status_reset(int64_t *st) {
  st[0] = 0;
  st[1] = INT64_MAX;
}

// ---------------------------------------------------------------------------
// exclusive scan int32 counts -> int32 offsets (n + 1 entries), int64 guard
// ---------------------------------------------------------------------------
constexpr int SCAN_THREADS = 1024;
constexpr int SCAN_PER_THREAD = 4;
constexpr int SCAN_BLOCK = SCAN_THREADS * SCAN_PER_THREAD;

__device__ __forceinline__ long long block_exclusive_scan(long long v, long long *warp_sums, long long *total) {
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  long long x = v;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    long long y = __shfl_up_sync(0xffffffffu, x, o);
    if (lane >= o) x += y;
  }
  if (lane == 31) warp_sums[w] = x;
  __syncthreads();
  if (w == 0) {
    long long s = (lane < (int)(blockDim.x >> 5)) ? warp_sums[lane] : 0;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      long long y = __shfl_up_sync(0xffffffffu, s, o);
      if (lane >= o) s += y;
    }
    warp_sums[lane] = s;  // inclusive
  }
  __syncthreads();
  long long base = (w > 0) ? warp_sums[w - 1] : 0;
  *total = warp_sums[(blockDim.x >> 5) - 1];
  __syncthreads();
  return base + x - v;
}

__global__ void __launch_bounds__(SCAN_THREADS) k_scan_reduce(const int32_t *in, int64_t n, long long *bsum) {
  __shared__ long long ws[32];
  int64_t base = (int64_t)blockIdx.x * SCAN_BLOCK + (int64_t)threadIdx.x * SCAN_PER_THREAD;
  long long s = 0;
#pragma unroll
  for (int k = 0; k < SCAN_PER_THREAD; ++k)
    if (base + k < n) s += in[base + k];
  long long tot;
  block_exclusive_scan(s, ws, &tot);
  if (threadIdx.x == 0) bsum[blockIdx.x] = tot;
}

__global__ void __launch_bounds__(SCAN_THREADS) k_scan_bsums(long long *bsum, int64_t nb) {
  __shared__ long long ws[32];
  long long carry = 0;
  for (int64_t b0 = 0; b0 < nb; b0 += SCAN_THREADS) {
    int64_t i = b0 + threadIdx.x;
    long long v = (i < nb) ? bsum[i] : 0;
    long long tot;
    long long ex = block_exclusive_scan(v, ws, &tot);
    if (i < nb) bsum[i] = carry + ex;
    carry += tot;
    __syncthreads();
  }
  if (threadIdx.x == 0) bsum[nb] = carry;
}

__global__ void __launch_bounds__(SCAN_THREADS) k_scan_apply(const int32_t *in, int64_t n, const long long *bsum,
                                                             int32_t *out, int64_t *st) {
  __shared__ long long ws[32];
  int64_t base = (int64_t)blockIdx.x * SCAN_BLOCK + (int64_t)threadIdx.x * SCAN_PER_THREAD;
  long long v[SCAN_PER_THREAD];
  long long s = 0;
#pragma unroll
  for (int k = 0; k < SCAN_PER_THREAD; ++k) {
    v[k] = (base + k < n) ? in[base + k] : 0;
    s += v[k];
  }
  long long tot;
  long long ex = block_exclusive_scan(s, ws, &tot) + bsum[blockIdx.x];
#pragma unroll
  for (int k = 0; k < SCAN_PER_THREAD; ++k) {
    if (base + k < n) {
      if (ex > INT32_MAX) flag(st, EMG_ST_CAPACITY, base + k);
      out[base + k] = (int32_t)ex;
    }
    ex += v[k];
  }
  if (blockIdx.x == gridDim.x - 1 && threadIdx.x == 0) {
    long long total = bsum[gridDim.x];
    if (total > INT32_MAX) flag(st, EMG_ST_CAPACITY, n);
    out[n] = (int32_t)total;
  }
}

// in and out may alias (in-place scan of counts stored in out[0..n))
int exclusive_scan(const int32_t *in, int64_t n, int32_t *out, long long *bsum, int64_t *st, cudaStream_t s) {
  int64_t nb = (n + SCAN_BLOCK - 1) / SCAN_BLOCK;
  if (nb == 0) nb = 1;
  k_scan_reduce<<<(unsigned)nb, SCAN_THREADS, 0, s>>>(in, n, bsum);
  k_scan_bsums<<<1, SCAN_THREADS, 0, s>>>(bsum, nb);
  k_scan_apply<<<(unsigned)nb, SCAN_THREADS, 0, s>>>(in, n, bsum, out, st);
  return launch_check("exclusive_scan");
}

size_t scan_bsum_bytes(int64_t n) { return (size_t)((n + SCAN_BLOCK - 1) / SCAN_BLOCK + 2) * sizeof(long long); }

// ---------------------------------------------------------------------------
// plan: entity -> incident (tet, slot) items and column positions
// ---------------------------------------------------------------------------
constexpr int MAX_ADJ = 255;  // adjacent edges (faces) per entity: uint8 positions

__device__ __forceinline__ int64_t tet_of(const int32_t *tetids, int64_t ia) { return tetids ? tetids[ia] : ia; }


__global__ void k_count_incidence(const int32_t *t2e, const int32_t *t2t, const int32_t *tetids, int64_t nT,
                                  int64_t nA, int64_t E, int64_t F, int32_t *cnt, int64_t *st) {
  int64_t g = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (g >= nA * 10) return;
  int64_t ia = g / 10;
  int s = (int)(g % 10);
  int64_t it = tet_of(tetids, ia);
  if (it < 0 || it >= nT) {
    flag(st, EMG_ST_INDEX, ia);
    return;
  }
  int64_t raw = s < 6 ? (int64_t)t2e[(int64_t)s * nT + it] : (int64_t)t2t[(int64_t)(s - 6) * nT + it];
  if (raw < 0 || raw >= (s < 6 ? E : F)) {
    flag(st, EMG_ST_INDEX, ia);
    return;
  }
  atomicAdd(&cnt[s < 6 ? raw : E + raw], 1);
}

__global__ void k_fill_items(const int32_t *tets, const int32_t *t2e, const int32_t *t2t, const int32_t *tetids,
                             int64_t nT, int64_t nA, int64_t E, int64_t F, const int32_t *ent_ptr, int32_t *cursor,
                             Item *items) {
  int64_t g = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (g >= nA * 10) return;
  int64_t ia = g / 10;
  int s = (int)(g % 10);
  int64_t it = tet_of(tetids, ia);
  if (it < 0 || it >= nT) return;
  int64_t raw = s < 6 ? (int64_t)t2e[(int64_t)s * nT + it] : (int64_t)t2t[(int64_t)(s - 6) * nT + it];
  if (raw < 0 || raw >= (s < 6 ? E : F)) return;
  int64_t x = s < 6 ? raw : E + raw;
  int32_t p = ent_ptr[x] + atomicAdd(&cursor[x], 1);
  Item rec;
  rec.ia = (int32_t)ia;
  rec.slot = (uint8_t)s;
#pragma unroll
  for (int k = 0; k < 10; ++k) rec.pos[k] = 0;
  // vertex ranks by global id (a repeated vertex is caught by the element kernel)
  int32_t v[4];
#pragma unroll
  for (int q = 0; q < 4; ++q) v[q] = tets[(int64_t)q * nT + it];
  uint32_t ranks = 0;
#pragma unroll
  for (int q = 0; q < 4; ++q) {
    int r = 0;
#pragma unroll
    for (int o = 0; o < 4; ++o) r += (v[o] < v[q] || (v[o] == v[q] && o < q)) ? 1 : 0;
    ranks |= (uint32_t)r << (2 * q);
  }
  rec.ranks = (uint8_t)ranks;
  items[p] = rec;
}

// insertion sort of each entity's items by assembled tet index (deterministic order)
__global__ void k_sort_items(const int32_t *ent_ptr, int64_t n_ent, Item *items) {
  int64_t x = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (x >= n_ent) return;
  int32_t b = ent_ptr[x], e = ent_ptr[x + 1];
  for (int32_t i = b + 1; i < e; ++i) {
    Item v = items[i];
    int32_t j = i - 1;
    while (j >= b && items[j].ia > v.ia) {
      items[j + 1] = items[j];
      --j;
    }
    items[j + 1] = v;
  }
}

// Warp per entity. Candidates = the 6 edges and 4 faces of every incident tet,
// faces marked to come after all edges: sorted with their place (in registers; in
// shared memory past 120), so that a candidate's rank among the distinct values,
// its position in the item, is the number of first ones up to it. k_entity_rows
// does this for the column lengths and the positions; k_entity_indices then
// writes the rows. Comparing all candidates with each other, once to count and
// once to rank, took 152 + 313 us at 103,680 tets; this 154 + 106. Bound: latency
// (item -> tet -> candidate).
constexpr int ROWS_WARPS = 4;
constexpr int MAX_ITEMS = 106;  // incident tets of an entity
constexpr int BIG_ITEMS = 12;   // up to here its candidates are sorted in registers

// ranks sorted candidates, 32 a round (key = face << 63 | value << 32 | place), into
// the items; counts the distinct edges and faces
struct CandRank {
  int ue, uf;
  uint32_t last;
  __device__ __forceinline__ void round(uint64_t key, bool in, bool start, Item *items) {
    const int lane = threadIdx.x & 31;
    const uint32_t v = (uint32_t)(key >> 32), place = (uint32_t)key;
    uint32_t before = __shfl_up_sync(0xffffffffu, v, 1);
    if (lane == 0) before = last;
    const bool first = in && ((start && lane == 0) || v != before), face = v >> 31;
    const unsigned me = __ballot_sync(0xffffffffu, first && !face), mf = __ballot_sync(0xffffffffu, first && face);
    const unsigned upto = 0xffffffffu >> (31 - lane);
    // a rank over MAX_ADJ does not fit: the caller flags it
    if (in) items[place / 10].pos[place % 10] = (uint8_t)((face ? uf + __popc(mf & upto) : ue + __popc(me & upto)) - 1);
    ue += __popc(me);
    uf += __popc(mf);
    last = __shfl_sync(0xffffffffu, v, 31);
  }
};

template <int K, typename Load>
__device__ __forceinline__ void rank_candidates(int n, Item *items, CandRank &c, Load load) {
  const int lane = threadIdx.x & 31;
  uint64_t k[K];
#pragma unroll
  for (int r = 0; r < K; ++r) k[r] = r * 32 + lane < n ? load(r * 32 + lane) : ~0ull;
  warp_sort<K>(k);
#pragma unroll
  for (int r = 0; r < K; ++r) c.round(k[r], r * 32 + lane < n, r == 0, items);
}

// one entity, up to 10 BIG_ITEMS candidates in registers or, `buf`, any number
struct RowsArgs {
  const int32_t *t2e, *t2t, *tetids;
  int64_t nT, E, F;
  const int32_t *ent_ptr;
  Item *items;
  int64_t n_ent;
  int32_t *col_len;
  uint32_t *ent_cnt;
  int64_t *st;
};

template <bool BIG>
__device__ __forceinline__ void entity_rows(const RowsArgs &a, int64_t x, uint64_t *buf) {
  const int lane = threadIdx.x & 31;
  const int32_t b = a.ent_ptr[x];
  const int nitem = a.ent_ptr[x + 1] - b, n = 10 * nitem;
  if (!BIG && nitem > BIG_ITEMS) return;  // k_big_entity_rows
  if (BIG && nitem > MAX_ITEMS) {
    if (lane == 0) flag(a.st, EMG_ST_CAPACITY, x);
    return;
  }
  Item *own = a.items + b;
  auto load = [&](int i) {
    const int s = i % 10;
    const int64_t it = tet_of(a.tetids, own[i / 10].ia);
    const uint32_t v =
        s < 6 ? (uint32_t)a.t2e[(int64_t)s * a.nT + it] : 0x80000000u | (uint32_t)a.t2t[(int64_t)(s - 6) * a.nT + it];
    return ((uint64_t)v << 32) | (uint32_t)i;
  };
  CandRank c{0, 0, 0};
  if constexpr (!BIG) {
    if (n <= 32) rank_candidates<1>(n, own, c, load);
    else if (n <= 64) rank_candidates<2>(n, own, c, load);
    else rank_candidates<4>(n, own, c, load);
  } else {
    for (int i = lane; i < n; i += 32) buf[i] = load(i);
    __syncwarp();
    // comparators that all put the smaller key first: those past the end are left out
    for (int size = 2; (size >> 1) < n; size <<= 1)
      for (int j = size >> 1; j > 0; j >>= 1) {
        for (int k = lane; k < (n + 2 * j - 1) / (2 * j) * j; k += 32) {
          const int block = k / j * (2 * j), at = k % j;
          const int i = block + at, o = j == (size >> 1) ? block + 2 * j - 1 - at : i + j;
          if (o < n && buf[i] > buf[o]) {
            const uint64_t t = buf[i];
            buf[i] = buf[o];
            buf[o] = t;
          }
        }
        __syncwarp();
      }
    for (int i0 = 0; i0 < n; i0 += 32) c.round(i0 + lane < n ? buf[i0 + lane] : ~0ull, i0 + lane < n, i0 == 0, own);
    __syncwarp();
  }
  if (lane != 0) return;
  if (c.ue > MAX_ADJ || c.uf > MAX_ADJ) {
    flag(a.st, EMG_ST_CAPACITY, x);
    return;
  }
  const bool is_edge = x < a.E;
  const int32_t L = 2 * (c.ue + c.uf);
  a.col_len[is_edge ? x : a.E + x] = L;              // 2E + (x - E)
  a.col_len[is_edge ? x + a.E : a.E + a.F + x] = L;  // 2E + F + (x - E)
  a.ent_cnt[x] = (uint32_t)c.ue | ((uint32_t)c.uf << 16);
}

__global__ void __launch_bounds__(ROWS_WARPS * 32) k_entity_rows(const RowsArgs a) {
  const int64_t x = (int64_t)blockIdx.x * ROWS_WARPS + (threadIdx.x >> 5);
  if (x < a.n_ent) entity_rows<false>(a, x, nullptr);
}

// the entities with more than BIG_ITEMS incident tets, few in any mesh: a warp
// looks through 32 entities at a time
__global__ void __launch_bounds__(ROWS_WARPS * 32) k_big_entity_rows(const RowsArgs a) {
  __shared__ uint64_t bufs[ROWS_WARPS][10 * MAX_ITEMS];
  const int lane = threadIdx.x & 31;
  const int64_t step = (int64_t)gridDim.x * ROWS_WARPS * 32;
  for (int64_t x0 = ((int64_t)blockIdx.x * ROWS_WARPS + (threadIdx.x >> 5)) * 32; x0 < a.n_ent; x0 += step) {
    const int64_t x = x0 + lane;
    unsigned big = __ballot_sync(0xffffffffu, x < a.n_ent && a.ent_ptr[x + 1] - a.ent_ptr[x] > BIG_ITEMS);
    for (; big; big &= big - 1) entity_rows<true>(a, x0 + __ffs(big) - 1, bufs[threadIdx.x >> 5]);
  }
}

// the rows of the four column blocks: every candidate writes its value at its rank
__global__ void __launch_bounds__(ROWS_WARPS * 32)
    k_entity_indices(const int32_t *t2e, const int32_t *t2t, const int32_t *tetids, int64_t nT, int64_t E, int64_t F,
                     const int32_t *ent_ptr, const Item *items, int64_t n_ent, const uint32_t *ent_cnt,
                     const int32_t *indptr, int32_t *indices) {
  const int lane = threadIdx.x & 31;
  const int64_t x = (int64_t)blockIdx.x * ROWS_WARPS + (threadIdx.x >> 5);
  if (x >= n_ent) return;
  const int32_t b = ent_ptr[x];
  const int n = 10 * (ent_ptr[x + 1] - b);
  const uint32_t c = ent_cnt[x];
  const int ue = (int)(c & 0xffffu), uf = (int)(c >> 16);
  const bool is_edge = x < E;
  const int64_t s0 = indptr[is_edge ? x : E + x], s1 = indptr[is_edge ? x + E : E + F + x];
  for (int i = lane; i < n; i += 32) {
    const int k = i / 10, s = i % 10;
    const Item &rec = items[b + k];
    const int64_t it = tet_of(tetids, rec.ia);
    const int r = rec.pos[s];
    const bool e = s < 6;
    const int32_t v = e ? t2e[(int64_t)s * nT + it] : t2t[(int64_t)(s - 6) * nT + it];
    const int at = e ? r : 2 * ue + r, part = e ? ue : uf;
    const int32_t r0 = e ? v : v + 2 * (int32_t)E, r1 = e ? v + (int32_t)E : v + 2 * (int32_t)E + (int32_t)F;
    indices[s0 + at] = indices[s1 + at] = r0;
    indices[s0 + at + part] = indices[s1 + at + part] = r1;
  }
}

__global__ void k_max_col(const int32_t *col_len, int64_t n, int32_t *out) {
  int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  int32_t m = 0;
  for (; i < n; i += (int64_t)gridDim.x * blockDim.x) m = max(m, col_len[i]);
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) m = max(m, __shfl_xor_sync(0xffffffffu, m, o));
  if ((threadIdx.x & 31) == 0) atomicMax(out, m);
}

// Packed gather lists, warp per chunk: every (item, row) of the chunk contributes to
// one position of the chunk's first-DoF run (and the same position of its
// second-DoF run). Count per position, scan, then place the contributions in
// item order (items of an entity are sorted by tet), so each output sums its
// contributions in a fixed order.
constexpr int CC_WARPS = 8;

__global__ void __launch_bounds__(CC_WARPS * 32)
    k_chunk_contrib(const int32_t *ent_ptr, const Item *items, const uint32_t *ent_cnt, int64_t E, int64_t F,
                    const int32_t *indptr, uint16_t *posoff, void *pidx_v, bool compact, int64_t *st) {
  __shared__ int32_t cnt_all[CC_WARPS][CHUNK_MAX_POS];
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  const int64_t chunk = (int64_t)blockIdx.x * CC_WARPS + w;
  const int64_t nec = n_edge_chunks(E);
  if (chunk >= n_chunks(E, F)) return;
  const bool edges = chunk < nec;
  const int64_t x0 = edges ? chunk * CHUNK : E + (chunk - nec) * CHUNK;
  const int nx = (int)min((int64_t)CHUNK, (edges ? E : E + F) - x0);
  const int64_t cb0 = edges ? x0 : E + x0;
  const int32_t my_ptr = lane <= nx ? ent_ptr[x0 + lane] : 0;
  const int32_t my_c0 = lane <= nx ? indptr[cb0 + lane] : 0;
  const uint32_t my_cnt = lane < nx ? ent_cnt[x0 + lane] : 0u;
  const int32_t I0 = __shfl_sync(0xffffffffu, my_ptr, 0), I1 = __shfl_sync(0xffffffffu, my_ptr, nx);
  const int32_t A0 = __shfl_sync(0xffffffffu, my_c0, 0), A0e = __shfl_sync(0xffffffffu, my_c0, nx);
  const int Lsum = A0e - A0;
  if (Lsum > CHUNK_MAX_POS || I1 - I0 > CHUNK_MAX_ITEMS) {
    if (lane == 0) flag(st, EMG_ST_CAPACITY, x0);
    return;
  }
  const int64_t hbase = edges ? (int64_t)A0 : (int64_t)indptr[E] + (A0 - indptr[2 * E]);
  int32_t *cnt = cnt_all[w];
  for (int i = lane; i < Lsum; i += 32) cnt[i] = 0;
  const int r = lane;
  const int sl = r < 6 ? r : (r < 12 ? r - 6 : (r < 16 ? r - 6 : r - 10));
  const int blk = r < 6 ? 0 : (r < 12 ? 1 : (r < 16 ? 2 : 3));
  __syncwarp();
  for (int pass = 0; pass < 2; ++pass) {
    if (pass == 1) {
      // exclusive scan of the counts into start offsets (lane-serial blocks of 32)
      int32_t carry = 0;
      for (int b0 = 0; b0 < Lsum; b0 += 32) {
        const int i = b0 + lane;
        const int32_t v = i < Lsum ? cnt[i] : 0;
        int32_t x = v;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
          const int32_t y = __shfl_up_sync(0xffffffffu, x, o);
          if (lane >= o) x += y;
        }
        if (i < Lsum) {
          cnt[i] = carry + x - v;  // becomes the cursor
          posoff[hbase + i] = (uint16_t)(carry + x - v);
        }
        carry += __shfl_sync(0xffffffffu, x, 31);
      }
      __syncwarp();
    }
    for (int32_t k = I0; k < I1; ++k) {
      if (r < 20) {
        int e = 0;
        for (int q = 1; q < nx; ++q)
          if (k >= __shfl_sync(0x000fffffu, my_ptr, q)) e = q;
        const int32_t ce = __shfl_sync(0x000fffffu, my_c0, e);
        const uint32_t c = __shfl_sync(0x000fffffu, my_cnt, e);
        const int ne = (int)(c & 0xffffu), nf = (int)(c >> 16);
        const int off = blk == 0 ? 0 : (blk == 1 ? ne : (blk == 2 ? 2 * ne : 2 * ne + nf));
        const Item rec = items[k];
        const int p = (ce - A0) + off + rec.pos[sl];
        if (pass == 0) {
          cnt[p] += 1;  // distinct p across the 20 lanes of one item
        } else {
          const int32_t at = cnt[p]++;
          const int s = rec.slot;
          const int a0 = s < 6 ? s : 12 + (s - 6), a1 = s < 6 ? s + 6 : 16 + (s - 6);
          const int al = canon_dof(rec.ranks, r);
          const int b0 = canon_dof(rec.ranks, a0), b1 = canon_dof(rec.ranks, a1);
          const int64_t base = (int64_t)rec.ia * 210;
          if (compact)
            static_cast<uint32_t *>(pidx_v)[(int64_t)20 * I0 + at] =
                (uint32_t)(base + packed_index(min(al, b0), max(al, b0))) | (al <= b0 ? 0x80000000u : 0u);
          else
            static_cast<int2 *>(pidx_v)[(int64_t)20 * I0 + at] =
                make_int2((int)(base + packed_index(min(al, b0), max(al, b0))),
                          (int)(base + packed_index(min(al, b1), max(al, b1))));
        }
      }
      __syncwarp();
    }
  }
}

// Block gather records (EMG_LAYOUT_BLOCK), warp per chunk, lane per (item, row
// entity): the tet's block of that entity pair goes to one row pair (the row
// entity's first-DoF row and its partner row, which hold the same tets). The
// items of the chunk entity that hold the same row entity (the same position
// byte) give the length of the row pair's list and the block's place in it, in
// item order, so each output sums its contributions in the order of the packed
// lists. Layout of the records: common.cuh. A tet's canonical entities come from
// a table of its vertex ranks that each CTA lays out once for all its chunks.
// 103,680 tets: 192 us (683 with them worked out per lane, 351 for a serial walk
// over the items).
__device__ __forceinline__ uint32_t item_byte(const uint4 &o, int i) {  // byte i of an item
  const uint32_t w = i < 8 ? (i < 4 ? o.x : o.y) : (i < 12 ? o.z : o.w);
  return (w >> (8 * (i & 3))) & 0xffu;
}

__global__ void __launch_bounds__(CC_WARPS * 32)
    k_chunk_blocks(const int32_t *ent_ptr, const Item *items, const uint32_t *ent_cnt, int64_t E, int64_t F,
                   const int32_t *indptr, uint32_t *brec, int64_t *st) {
  struct Meta {
    int32_t ptr[CHUNK + 1], c0[CHUNK + 1], ne[CHUNK], n_long;
  };
  __shared__ Meta meta[CC_WARPS];
  __shared__ uint8_t canon[256][12];  // canonical entity of slot s (0..9) by the tet's ranks byte
  for (int i = threadIdx.x; i < 2560; i += CC_WARPS * 32) {
    const int ranks = i / 10, s = i % 10;
    canon[ranks][s] = (uint8_t)(s < 6 ? canon_dof(ranks, s) : canon_dof(ranks, 12 + (s - 6)) - 6);
  }
  __syncthreads();
  const int lane = threadIdx.x & 31;
  Meta &m = meta[threadIdx.x >> 5];
  const int64_t nec = n_edge_chunks(E), nch = n_chunks(E, F);
  const uint4 *raw = reinterpret_cast<const uint4 *>(items);
  // block number of item o for row slot r, bit 31 when it is stored transposed
  auto word_of = [&](const uint4 &o, int r) {
    const uint8_t *of = canon[item_byte(o, 15)];
    const int ca = of[r], cb = of[item_byte(o, 4)];
    const int lo = min(ca, cb), hi = max(ca, cb);
    return (o.x * 55u + (uint32_t)block_index(lo, hi)) | (ca > cb ? 0x80000000u : 0u);
  };
  for (int64_t chunk = (int64_t)blockIdx.x * CC_WARPS + (threadIdx.x >> 5); chunk < nch;
       chunk += (int64_t)gridDim.x * CC_WARPS) {
    const bool edges = chunk < nec;
    const int64_t x0 = edges ? chunk * CHUNK : E + (chunk - nec) * CHUNK;
    const int nx = (int)min((int64_t)CHUNK, (edges ? E : E + F) - x0);
    const int64_t cb0 = edges ? x0 : E + x0;
    __syncwarp();
    if (lane <= CHUNK) {  // past the chunk's last entity: its end
      m.ptr[lane] = ent_ptr[x0 + min(lane, nx)];
      m.c0[lane] = indptr[cb0 + min(lane, nx)];
    }
    if (lane < nx) m.ne[lane] = (int32_t)(ent_cnt[x0 + lane] & 0xffffu);
    if (lane == 0) m.n_long = 0;
    __syncwarp();
    const int32_t I0 = m.ptr[0], nI = m.ptr[CHUNK] - I0, A0 = m.c0[0];
    const int Lsum = m.c0[CHUNK] - A0, H = Lsum / 2;
    if (Lsum > CHUNK_MAX_POS || nI > CHUNK_MAX_ITEMS) {
      if (lane == 0) flag(st, EMG_ST_CAPACITY, x0);
      continue;
    }
    uint32_t *words = brec + (int64_t)kPairWords * I0;
    uint2 *pairs = reinterpret_cast<uint2 *>(words);
    for (int t = lane; t < 10 * nI; t += 32) {
      const int k = I0 + t / 10, r = t % 10;
      int e = k >= m.ptr[4] ? 4 : 0;
      e += k >= m.ptr[e + 2] ? 2 : 0;
      e += k >= m.ptr[e + 1] ? 1 : 0;
      const uint4 own = raw[k];
      const uint32_t pos = item_byte(own, 5 + r), same = pos * 0x01010101u;
      // bytes of an item: slot at 4, pos[0..9] at 5..14 (edges, then faces), ranks at 15
      const uint32_t my = r < 6 ? 0xffffff00u : 0u, mz = r < 6 ? 0x00ffffffu : 0xff000000u, mw = r < 6 ? 0u : 0x00ffffffu;
      // the first row slot of item o that holds this row entity, -1 if none does:
      // the first matching byte, less the five before pos
      auto slot_in = [&](const uint4 &o) {
        const uint32_t hy = __vcmpeq4(o.y, same) & my, hz = __vcmpeq4(o.z, same) & mz, hw = __vcmpeq4(o.w, same) & mw;
        if (!(hy | hz | hw)) return -1;
        return (hy ? __ffs(hy) / 8 : (hz ? 4 + __ffs(hz) / 8 : 8 + __ffs(hw) / 8)) - 1;
      };
      const uint32_t word = word_of(own, r);
      const int slot = (int)item_byte(own, 4);
      if (r == slot) words[2 * H + (k - I0)] = word;
      // a tet that lists a row entity twice, which only inconsistent topology arrays
      // do, counts once: more would not fit the chunk's words
      if (slot_in(own) != r) continue;
      const int i0 = m.ptr[e], i1 = m.ptr[e + 1];
      int total = 0, rank = 0, other = k, other_r = r;
      for (int i = i0; i < i1; ++i) {
        const int at = slot_in(raw[i]);
        if (at >= 0) {
          ++total;
          rank += i < k ? 1 : 0;
          if (i != k) {
            other = i;
            other_r = at;
          }
        }
      }
      const int h = (m.c0[e] - A0) / 2 + (r < 6 ? 0 : m.ne[e]) + (int)pos;
      // the entity's pair with itself: every item has one
      const bool self = (r < 6) == (slot < 6) && item_byte(own, 5 + slot) == pos;
      // two blocks stored different ways round: only with inconsistent topology arrays
      const bool differ = total == 2 && ((word_of(raw[other], other_r) ^ word) >> 31);
      if (total <= 2 && !differ) {
        if (total == 1) pairs[h] = make_uint2(word, kBlockNone);
        else words[2 * h + rank] = word;
      } else if (rank == 0) {  // one lane writes the whole list
        int off = 0;
        if (!self) {
          off = 2 * H + nI + atomicAdd(&m.n_long, total);
          uint32_t *list = words + off;
          for (int i = i0; i < i1; ++i) {
            const uint4 o = raw[i];
            for (int p = r < 6 ? 0 : 6; p < (r < 6 ? 6 : 10); ++p)
              if (item_byte(o, 5 + p) == pos) {
                *list++ = word_of(o, p);
                break;
              }
          }
        }
        pairs[h] = make_uint2(self ? 0u : (uint32_t)off | ((uint32_t)total << 16), kBlockLong);
      }
    }
  }
}

// chunk descriptors in processing order (common.cuh)
__global__ void k_chunk_desc(const int32_t *ent_ptr, const Item *items, const uint32_t *ent_cnt, int64_t E, int64_t F,
                             const int32_t *indptr, const int32_t *order, ChunkDesc *desc) {
  const int64_t g = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  const int64_t nec = n_edge_chunks(E), nch = n_chunks(E, F);
  if (g >= nch) return;
  const int64_t chunk = order[g];
  ChunkDesc d = {};
  if (chunk >= 0 && chunk < nch) {
    const bool edges = chunk < nec;
    const int64_t x0 = edges ? chunk * CHUNK : E + (chunk - nec) * CHUNK;
    const int nx = (int)min((int64_t)CHUNK, (edges ? E : E + F) - x0);
    const int64_t cb0 = edges ? x0 : E + x0, cb1 = edges ? x0 + E : E + F + x0;
    d.I0 = ent_ptr[x0];
    d.A0 = indptr[cb0];
    d.A1 = indptr[cb1];
    d.faces = edges ? 0 : 1;
    const int rows = indptr[cb0 + nx] - d.A0, n = ent_ptr[x0 + nx] - d.I0;
    if (rows <= CHUNK_MAX_POS && n <= CHUNK_MAX_ITEMS) {  // else the build was flagged
      d.H = (uint16_t)(rows / 2);
      d.nI = (uint16_t)n;
      for (int e = 0; e < CHUNK; ++e) {
        d.hs[e] = d.H;
        if (e >= nx) continue;
        const int32_t i0 = ent_ptr[x0 + e], i1 = ent_ptr[x0 + e + 1];
        d.hs[e] = (uint16_t)((indptr[cb0 + e] - d.A0) / 2);
        d.ne[e] = (uint8_t)(ent_cnt[x0 + e] & 0xffu);
        d.cnt[e] = (uint8_t)(i1 - i0);
        if (i1 > i0) d.self[e] = items[i0].pos[items[i0].slot];
      }
    }
  }
  desc[g] = d;
}

int write_chunk_desc(const emg_plan *p, char *plan, const int32_t *indptr, cudaStream_t s) {
  const int64_t nch = n_chunks(p->n_edges, p->n_tris);
  k_chunk_desc<<<grid_for(nch, 128), 128, 0, s>>>(
      reinterpret_cast<const int32_t *>(plan + p->off_ent_ptr), reinterpret_cast<const Item *>(plan + p->off_item),
      reinterpret_cast<const uint32_t *>(plan + p->off_ent_cnt), p->n_edges, p->n_tris, indptr,
      reinterpret_cast<const int32_t *>(plan + p->off_order), reinterpret_cast<ChunkDesc *>(plan + p->off_hoff));
  return launch_check("k_chunk_desc");
}

__global__ void k_default_order(int32_t *order, int64_t nec, int64_t nch) {
  const int64_t g = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (g < nch) order[g] = (int32_t)chunk_at(g, nec, nch);
}

// bounding box of the nodes (SoA [3][nN]): per-block partials, then one block
__global__ void __launch_bounds__(256) k_bbox_partial(const double *nodes, int64_t nN, double *part) {
  __shared__ double sm[6][256];
  double lo[3] = {INFINITY, INFINITY, INFINITY}, hi[3] = {-INFINITY, -INFINITY, -INFINITY};
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < nN; i += (int64_t)gridDim.x * blockDim.x)
    for (int d = 0; d < 3; ++d) {
      const double x = nodes[d * nN + i];
      lo[d] = fmin(lo[d], x);
      hi[d] = fmax(hi[d], x);
    }
  for (int d = 0; d < 3; ++d) {
    sm[d][threadIdx.x] = lo[d];
    sm[3 + d][threadIdx.x] = hi[d];
  }
  __syncthreads();
  for (int st = 128; st > 0; st >>= 1) {
    if ((int)threadIdx.x < st)
      for (int d = 0; d < 3; ++d) {
        sm[d][threadIdx.x] = fmin(sm[d][threadIdx.x], sm[d][threadIdx.x + st]);
        sm[3 + d][threadIdx.x] = fmax(sm[3 + d][threadIdx.x], sm[3 + d][threadIdx.x + st]);
      }
    __syncthreads();
  }
  if (threadIdx.x < 6) part[blockIdx.x * 6 + threadIdx.x] = sm[threadIdx.x][0];
}

// a warp per bound
__global__ void k_bbox_final(const double *part, int nblk, double *box) {
  const int d = threadIdx.x >> 5, lane = threadIdx.x & 31;
  double v = d < 3 ? INFINITY : -INFINITY;
  for (int b = lane; b < nblk; b += 32) v = d < 3 ? fmin(v, part[b * 6 + d]) : fmax(v, part[b * 6 + d]);
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    const double x = __shfl_xor_sync(0xffffffffu, v, o);
    v = d < 3 ? fmin(v, x) : fmax(v, x);
  }
  if (lane == 0) box[d] = v;
}

__device__ __forceinline__ uint32_t spread_bits10(uint32_t x) {  // bit i -> bit 3i
  x &= 0x3ffu;
  x = (x | (x << 16)) & 0x030000ffu;
  x = (x | (x << 8)) & 0x0300f00fu;
  x = (x | (x << 4)) & 0x030c30c3u;
  x = (x | (x << 2)) & 0x09249249u;
  return x;
}

// key of chunk c = Morton code of the centroid of its first incident tet in
// the high 32 bits, c in the low 32 bits; chunks without items and the
// padding up to the power of two sort last
__global__ void k_chunk_keys(const int32_t *ent_ptr, const Item *items, const double *nodes, int64_t nN,
                             const int32_t *tets, int64_t nT, const int32_t *tetids, int64_t nA, const double *box,
                             int64_t E, int64_t F, int64_t nch, int64_t n2, uint64_t *keys) {
  const int64_t c = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (c >= n2) return;
  uint64_t key = ~0ull;
  if (c < nch) {
    const int64_t nec = n_edge_chunks(E);
    const int64_t x0 = c < nec ? c * CHUNK : E + (c - nec) * CHUNK;
    const int64_t xe = min(x0 + CHUNK, c < nec ? E : E + F);
    const int32_t i0 = ent_ptr[x0], i1 = ent_ptr[xe];
    uint32_t code = 0xffffffffu;
    if (i1 > i0) {
      const int64_t ia = items[i0].ia;
      const int64_t t = (ia >= 0 && ia < nA) ? (tetids ? (int64_t)tetids[ia] : ia) : -1;
      if (t >= 0 && t < nT) {
        const double ext = fmax(fmax(box[3] - box[0], box[4] - box[1]), fmax(box[5] - box[2], 1e-300));
        uint32_t q[3];
        for (int d = 0; d < 3; ++d) {
          double x = 0.0;
          for (int k = 0; k < 4; ++k) {
            const int64_t v = tets[k * nT + t];
            x += (v >= 0 && v < nN) ? nodes[d * nN + v] : box[d];
          }
          const double u = (0.25 * x - box[d]) / ext * 1024.0;
          q[d] = (uint32_t)fmin(fmax(u, 0.0), 1023.0);
        }
        code = spread_bits10(q[0]) | (spread_bits10(q[1]) << 1) | (spread_bits10(q[2]) << 2);
      }
    }
    key = ((uint64_t)code << 32) | (uint64_t)c;
  }
  keys[c] = key;
}

// Bitonic sort of n2 = 2^m keys. A CTA does every step within a tile of
// SORT_TILE keys in shared memory: all stages up to the tile (k_sort_tile<true>), or
// the steps j < SORT_TILE of stage k (k_sort_tile<false>). The steps between tiles go
// three to a launch, on the 8 keys a thread exchanges among themselves. 2^14 keys
// (a port's forcing vector) take 7 launches and 40 us instead of 105 and 176, 2^16
// and 2^17 30 and 160 us instead of 289 and 510. Tiles of 8,192 keys and 1,024
// threads: fewer launches, but 87 and 293 us on the few SMs that have a tile.
constexpr int SORT_TILE = 2048;
constexpr int SORT_THREADS = 512;

__device__ __forceinline__ void sort_tile_steps(uint64_t *t, int tile, int64_t base, int64_t k, int j0) {
  for (int j = j0; j > 0; j >>= 1) {
    __syncthreads();
    for (int c = threadIdx.x; c < tile / 2; c += SORT_THREADS) {
      const int i = ((c & ~(j - 1)) << 1) | (c & (j - 1)), l = i | j;
      const uint64_t a = t[i], b = t[l];
      if ((a > b) == (((base + i) & k) == 0)) {
        t[i] = b;
        t[l] = a;
      }
    }
  }
}

// ALL: sort the tile (all n2 keys, if fewer) from scratch; else stage k's last steps
template <bool ALL>
__global__ void __launch_bounds__(SORT_THREADS) k_sort_tile(uint64_t *keys, int64_t n2, int64_t k) {
  extern __shared__ uint64_t sort_keys[];
  const int tile = (int)min((int64_t)SORT_TILE, n2);
  const int64_t base = (int64_t)blockIdx.x * tile;
  for (int i = threadIdx.x; i < tile; i += SORT_THREADS) sort_keys[i] = keys[base + i];
  if (ALL) {
    for (int s = 2; s <= tile; s <<= 1) sort_tile_steps(sort_keys, tile, base, s, s >> 1);
  } else {
    sort_tile_steps(sort_keys, tile, base, k, tile >> 1);
  }
  __syncthreads();
  for (int i = threadIdx.x; i < tile; i += SORT_THREADS) keys[base + i] = sort_keys[i];
}

// steps j, j/2, ..., j/2^(STEPS-1) of stage k: a thread's 2^STEPS keys lie j/2^(STEPS-1) apart
template <int STEPS>
__global__ void __launch_bounds__(256) k_sort_steps(uint64_t *keys, int64_t n2, int64_t j, int64_t k) {
  constexpr int M = 1 << STEPS;
  const int64_t lo = j >> (STEPS - 1);  // the smallest of the steps
  const int64_t c = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (c >= n2 / M) return;
  const int64_t i0 = (c / lo) * (lo * M) + c % lo;
  uint64_t v[M];
#pragma unroll
  for (int m = 0; m < M; ++m) v[m] = keys[i0 + m * lo];
  const bool up = (i0 & k) == 0;  // k > j: the same for all of them
#pragma unroll
  for (int h = M / 2; h > 0; h >>= 1)
#pragma unroll
    for (int m = 0; m < M; ++m)
      if (!(m & h) && (v[m] > v[m | h]) == up) {
        const uint64_t t = v[m];
        v[m] = v[m | h];
        v[m | h] = t;
      }
#pragma unroll
  for (int m = 0; m < M; ++m) keys[i0 + m * lo] = v[m];
}

// the new order; block layout: the chunk descriptors (by_chunk: in chunk
// order) follow it
__global__ void k_write_order(const uint64_t *keys, int64_t nch, int32_t *order, const ChunkDesc *by_chunk,
                              ChunkDesc *desc) {
  const int64_t g = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (g >= nch) return;
  const int64_t c = (int64_t)(keys[g] & 0xffffffffu);
  order[g] = (int32_t)c;
  if (desc && c < nch) desc[g] = by_chunk[c];
}

__global__ void k_desc_by_chunk(const int32_t *order, const ChunkDesc *desc, int64_t nch, ChunkDesc *by_chunk) {
  const int64_t g = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (g < nch && order[g] >= 0 && order[g] < nch) by_chunk[order[g]] = desc[g];
}

}  // namespace

int status_reset(int64_t *st, cudaStream_t s) {
  k_status_reset<<<1, 1, 0, s>>>(st);
  return launch_check("k_status_reset");
}

int scan_i32(const int32_t *in, int64_t n, int32_t *out, long long *bsum, int64_t *st, cudaStream_t s) {
  return exclusive_scan(in, n, out, bsum, st, s);
}
size_t scan_i32_bsum_bytes(int64_t n) { return scan_bsum_bytes(n); }

size_t plan_layout(emg_plan *p) {
  size_t o = 0;
  p->off_ent_ptr = o;
  o = align_up(o + (size_t)(p->n_ent + 1) * 4, 256);
  p->off_item = o;
  o = align_up(o + (size_t)p->n_items * sizeof(Item), 256);
  p->off_item_pos = p->off_item;  // positions live inside the item records
  p->off_ent_cnt = o;
  o = align_up(o + (size_t)p->n_ent * 4, 256);
  // packed layout: one uint16 list start per first-DoF output position; a column
  // of entity x has 2 (n_adj_edges + n_adj_faces) <= 20 * items(x) entries, so 20
  // per item bounds the positions before nnz is known
  const bool block = p->value_layout == EMG_LAYOUT_BLOCK;
  p->off_contrib = p->off_posoff = o;
  o = align_up(o + (block ? 0 : (size_t)p->n_items * 20 * 2), 256);
  // packed layout: per contribution the indices of its two values (first- and
  // second-DoF column); block layout: the row
  // pairs' two-block records and the long lists, kPairWords words per item
  p->off_pidx = o;
  o = align_up(o + (size_t)p->n_items * (block ? kPairWords * 4 : 20 * (p->record_bytes == 4 ? 4 : 8)), 256);
  p->off_hoff = o;  // block layout: the chunk descriptors
  o = align_up(o + (block ? (size_t)n_chunks(p->n_edges, p->n_tris) * sizeof(ChunkDesc) : 0), 256);
  // the gather's chunk processing order
  p->off_order = o;
  o = align_up(o + (size_t)n_chunks(p->n_edges, p->n_tris) * 4, 256);
  p->plan_bytes = o;
  return o;
}

// chunk-order scratch: bounding-box partials, the sort keys (power of two) and
// the chunk descriptors
constexpr int BBOX_BLOCKS = 296;
static size_t order_desc_offset(const emg_plan *p) {
  return align_up(align_up((size_t)BBOX_BLOCKS * 6 * 8 + 64, 256) +
                      (size_t)pow2_at_least(n_chunks(p->n_edges, p->n_tris)) * 8,
                  256);
}
static size_t order_workspace_bytes(const emg_plan *p) {
  return order_desc_offset(p) + (size_t)n_chunks(p->n_edges, p->n_tris) * sizeof(ChunkDesc);
}

// workspace: per-entity counters, per-column lengths, scan block sums, max
// (plan build); bounding box and sort keys (chunk order); the larger of both
size_t plan_workspace_bytes(const emg_plan *p) {
  size_t w = 0;
  w = align_up(w + (size_t)p->n_ent * 4, 256);
  w = align_up(w + (size_t)(p->N + 1) * 4, 256);
  w = align_up(w + scan_bsum_bytes(p->N > p->n_ent ? p->N : p->n_ent), 256);
  w = align_up(w + 16, 256);
  const size_t wo = order_workspace_bytes(p);
  return w > wo ? w : wo;
}

int plan_build(emg_plan *p, const int32_t *d_tets, const int32_t *d_t2e, const int32_t *d_t2t,
               const int32_t *d_tetids, void *d_plan, void *d_ws, int32_t *d_indptr, int64_t *d_status,
               cudaStream_t s) {
  char *plan = static_cast<char *>(d_plan);
  char *ws = static_cast<char *>(d_ws);
  int32_t *ent_ptr = reinterpret_cast<int32_t *>(plan + p->off_ent_ptr);
  Item *items = reinterpret_cast<Item *>(plan + p->off_item);
  uint32_t *ent_cnt = reinterpret_cast<uint32_t *>(plan + p->off_ent_cnt);
  size_t o = 0;
  int32_t *cnt = reinterpret_cast<int32_t *>(ws + o);
  o = align_up(o + (size_t)p->n_ent * 4, 256);
  int32_t *col_len = reinterpret_cast<int32_t *>(ws + o);
  o = align_up(o + (size_t)(p->N + 1) * 4, 256);
  long long *bsum = reinterpret_cast<long long *>(ws + o);
  o = align_up(o + scan_bsum_bytes(p->N > p->n_ent ? p->N : p->n_ent), 256);
  int32_t *maxc = reinterpret_cast<int32_t *>(ws + o);
  int rc;
  if ((rc = status_reset(d_status, s))) return rc;
  if (p->n_ent > 0) CUDA_TRY(cudaMemsetAsync(cnt, 0, (size_t)p->n_ent * 4, s));
  CUDA_TRY(cudaMemsetAsync(maxc, 0, 4, s));
  const int64_t nI = p->n_items;
  if (nI > 0) {
    k_count_incidence<<<grid_for(nI, 256), 256, 0, s>>>(d_t2e, d_t2t, d_tetids, p->n_tets, p->n_assy, p->n_edges,
                                                         p->n_tris, cnt, d_status);
    if ((rc = launch_check("k_count_incidence"))) return rc;
  }
  if ((rc = exclusive_scan(cnt, p->n_ent, ent_ptr, bsum, d_status, s))) return rc;
  if (p->n_ent > 0) CUDA_TRY(cudaMemsetAsync(cnt, 0, (size_t)p->n_ent * 4, s));
  if (nI > 0) {
    k_fill_items<<<grid_for(nI, 256), 256, 0, s>>>(d_tets, d_t2e, d_t2t, d_tetids, p->n_tets, p->n_assy,
                                                    p->n_edges, p->n_tris, ent_ptr, cnt, items);
    if ((rc = launch_check("k_fill_items"))) return rc;
  }
  CUDA_TRY(cudaMemsetAsync(col_len, 0, (size_t)(p->N + 1) * 4, s));
  if (p->n_ent > 0) {
    k_sort_items<<<grid_for(p->n_ent, 256), 256, 0, s>>>(ent_ptr, p->n_ent, items);
    if ((rc = launch_check("k_sort_items"))) return rc;
    const RowsArgs ra{d_t2e, d_t2t, d_tetids, p->n_tets, p->n_edges, p->n_tris, ent_ptr, items, p->n_ent, col_len,
                      ent_cnt, d_status};
    k_entity_rows<<<grid_for(p->n_ent, ROWS_WARPS), ROWS_WARPS * 32, 0, s>>>(ra);
    if ((rc = launch_check("k_entity_rows"))) return rc;
    const int g = grid_for(p->n_ent, ROWS_WARPS * 32);
    k_big_entity_rows<<<g < persistent_ctas(4) ? g : persistent_ctas(4), ROWS_WARPS * 32, 0, s>>>(ra);
    if ((rc = launch_check("k_big_entity_rows"))) return rc;
    k_max_col<<<296, 256, 0, s>>>(col_len, p->N, maxc);
    if ((rc = launch_check("k_max_col"))) return rc;
  }
  if ((rc = exclusive_scan(col_len, p->N, d_indptr, bsum, d_status, s))) return rc;
  int32_t h_nnz = 0, h_max = 0;
  int64_t h_st[2] = {0, 0};
  CUDA_TRY(cudaMemcpyAsync(&h_nnz, d_indptr + p->N, 4, cudaMemcpyDeviceToHost, s));
  CUDA_TRY(cudaMemcpyAsync(&h_max, maxc, 4, cudaMemcpyDeviceToHost, s));
  CUDA_TRY(cudaMemcpyAsync(h_st, d_status, 16, cudaMemcpyDeviceToHost, s));
  CUDA_TRY(cudaStreamSynchronize(s));
  if (h_st[0])
    return fail(EMG_EMESH, "plan build: status flags 0x%llx at index %lld", (long long)h_st[0], (long long)h_st[1]);
  p->nnz = h_nnz;
  p->max_col = h_max;
  return EMG_OK;
}

int plan_finish(const emg_plan *p, const int32_t *d_t2e, const int32_t *d_t2t, const int32_t *d_tetids,
                void *d_plan, const int32_t *d_indptr, int32_t *d_indices, int64_t *d_status, cudaStream_t s) {
  char *plan = static_cast<char *>(d_plan);
  const int64_t nch = n_chunks(p->n_edges, p->n_tris);
  if (nch > 0) {
    k_default_order<<<grid_for(nch, 256), 256, 0, s>>>(reinterpret_cast<int32_t *>(plan + p->off_order),
                                                        n_edge_chunks(p->n_edges), nch);
    const int rc = launch_check("k_default_order");
    if (rc) return rc;
  }
  if (p->n_ent == 0) return EMG_OK;
  if (p->n_assy == 0)  // empty columns; the block gather still walks the chunks
    return p->value_layout == EMG_LAYOUT_BLOCK ? write_chunk_desc(p, plan, d_indptr, s) : EMG_OK;
  const int32_t *ent_ptr = reinterpret_cast<const int32_t *>(plan + p->off_ent_ptr);
  Item *items = reinterpret_cast<Item *>(plan + p->off_item);
  uint32_t *ent_cnt = reinterpret_cast<uint32_t *>(plan + p->off_ent_cnt);
  k_entity_indices<<<grid_for(p->n_ent, ROWS_WARPS), ROWS_WARPS * 32, 0, s>>>(
      d_t2e, d_t2t, d_tetids, p->n_tets, p->n_edges, p->n_tris, ent_ptr, items, p->n_ent, ent_cnt, d_indptr, d_indices);
  int rc = launch_check("k_entity_indices");
  if (rc) return rc;
  void *pidx = plan + p->off_pidx;
  if (p->value_layout != EMG_LAYOUT_BLOCK) {
    k_chunk_contrib<<<grid_for(n_chunks(p->n_edges, p->n_tris), CC_WARPS), CC_WARPS * 32, 0, s>>>(
        ent_ptr, items, ent_cnt, p->n_edges, p->n_tris, d_indptr, reinterpret_cast<uint16_t *>(plan + p->off_posoff),
        pidx, p->record_bytes == 4, d_status);
    return launch_check("k_chunk_contrib");
  }
  const int64_t block_ctas = (n_chunks(p->n_edges, p->n_tris) + CC_WARPS - 1) / CC_WARPS;
  k_chunk_blocks<<<(int)(block_ctas < persistent_ctas(8) ? block_ctas : persistent_ctas(8)), CC_WARPS * 32, 0, s>>>(
      ent_ptr, items, ent_cnt, p->n_edges, p->n_tris, d_indptr, static_cast<uint32_t *>(pidx), d_status);
  if ((rc = launch_check("k_chunk_blocks"))) return rc;
  return write_chunk_desc(p, plan, d_indptr, s);
}

int sort_u64(uint64_t *keys, int64_t n2, cudaStream_t s) {
  if (n2 & (n2 - 1)) return fail(EMG_EINVAL, "sort length %lld is not a power of two", (long long)n2);
  if (n2 < 2) return EMG_OK;
  constexpr int smem = SORT_TILE * 8;
  const int tiles = grid_for(n2, SORT_TILE);
  k_sort_tile<true><<<tiles, SORT_THREADS, smem, s>>>(keys, n2, 0);
  int rc = launch_check("k_sort_tile");
  for (int64_t k = 2 * SORT_TILE; k <= n2 && !rc; k <<= 1) {
    for (int64_t j = k >> 1; j >= SORT_TILE && !rc;) {
      const int steps = j >= 4 * SORT_TILE ? 3 : (j >= 2 * SORT_TILE ? 2 : 1);
      const int g = grid_for(n2 >> steps, 256);
      if (steps == 3) k_sort_steps<3><<<g, 256, 0, s>>>(keys, n2, j, k);
      else if (steps == 2) k_sort_steps<2><<<g, 256, 0, s>>>(keys, n2, j, k);
      else k_sort_steps<1><<<g, 256, 0, s>>>(keys, n2, j, k);
      rc = launch_check("k_sort_steps");
      j >>= steps;
    }
    if (rc) return rc;
    k_sort_tile<false><<<tiles, SORT_THREADS, smem, s>>>(keys, n2, k);
    rc = launch_check("k_sort_tile");
  }
  return rc;
}

int plan_order(const emg_plan *p, void *d_plan, const double *nodes, int64_t nN, const int32_t *tets,
               const int32_t *tetids, void *d_ws, cudaStream_t s) {
  const int64_t nch = n_chunks(p->n_edges, p->n_tris);
  if (nch == 0 || p->n_assy == 0 || nN == 0) return EMG_OK;
  char *plan = static_cast<char *>(d_plan);
  char *ws = static_cast<char *>(d_ws);
  double *part = reinterpret_cast<double *>(ws);
  double *box = part + (size_t)BBOX_BLOCKS * 6;
  uint64_t *keys = reinterpret_cast<uint64_t *>(ws + align_up((size_t)BBOX_BLOCKS * 6 * 8 + 64, 256));
  const int64_t n2 = pow2_at_least(nch);
  k_bbox_partial<<<BBOX_BLOCKS, 256, 0, s>>>(nodes, nN, part);
  int rc = launch_check("k_bbox_partial");
  if (rc) return rc;
  k_bbox_final<<<1, 6 * 32, 0, s>>>(part, BBOX_BLOCKS, box);
  if ((rc = launch_check("k_bbox_final"))) return rc;
  k_chunk_keys<<<grid_for(n2, 256), 256, 0, s>>>(
      reinterpret_cast<const int32_t *>(plan + p->off_ent_ptr), reinterpret_cast<const Item *>(plan + p->off_item),
      nodes, nN, tets, p->n_tets, tetids, p->n_assy, box, p->n_edges, p->n_tris, nch, n2, keys);
  if ((rc = launch_check("k_chunk_keys"))) return rc;
  if ((rc = sort_u64(keys, n2, s))) return rc;
  int32_t *order = reinterpret_cast<int32_t *>(plan + p->off_order);
  ChunkDesc *by_chunk = reinterpret_cast<ChunkDesc *>(ws + order_desc_offset(p)), *desc = nullptr;
  if (p->value_layout == EMG_LAYOUT_BLOCK) {
    desc = reinterpret_cast<ChunkDesc *>(plan + p->off_hoff);
    k_desc_by_chunk<<<grid_for(nch, 256), 256, 0, s>>>(order, desc, nch, by_chunk);
    if ((rc = launch_check("k_desc_by_chunk"))) return rc;
  }
  k_write_order<<<grid_for(nch, 256), 256, 0, s>>>(keys, nch, order, by_chunk, desc);
  return launch_check("k_write_order");
}

}  // namespace emg
