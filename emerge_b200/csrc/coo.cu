// coo.cu -- a general COO -> CSC mapping on the device.
//
// Replaces CSCMapping.from_rowcol / precompute_csc_pattern / to_csc for any
// (rows, cols) slot list (mth/csc_cast.py:51-177), as the heat-conduction
// assembly calls them (physics/heatconduction/assembly/grad.py:403-460).
// Pattern: slots counted per column, scattered into column buckets, each
// bucket sorted by (row, slot) -- a fixed order, whatever order the scatter
// left them in -- and its distinct rows become the column's entries; the value
// of an entry is the sum of its slots in that order. Slots that are the D x D blocks
// of elements are counted and scattered as the D columns of each element, and
// their rows read from the elements' DoFs.
#include "common.cuh"

namespace emg {
namespace {

// Where the slots' rows and columns come from. An item is what is counted and
// scattered: width() slots of one column.
struct SlotList {  // any list: slot s has row rows[s] and column cols[s]
  const int32_t *rows, *cols;
  __device__ __forceinline__ int width() const { return 1; }
  __device__ __forceinline__ int32_t col(int64_t item) const { return cols[item]; }
  __device__ __forceinline__ int32_t slot(int64_t item) const { return (int32_t)item; }
  __device__ __forceinline__ int32_t row(int32_t slot) const { return rows[slot]; }
  // slot q of a column's list whose items' first slots are scattered
  __device__ __forceinline__ int32_t listed(const int32_t *perm, int q) const { return perm[q]; }
};

// Element blocks: slot D^2 t + D i + j has row dofs[t][i] and column dofs[t][j]; an
// item is column j of element t, its D slots D apart. A tenth of the atomics of a
// list of 10 x 10 blocks and no row and column arrays: at 99,900 tets 8 + 15 us
// for count and scatter, where the lists took 44 (k_coo_rowcol) + 166 + 216, and
// k_coo_fill 32 instead of 48.
template <int D_>
struct BlockList {
  const int32_t *dofs;  // [n_elements][D]
  int d;
  __device__ __forceinline__ int D() const { return D_ ? D_ : d; }
  __device__ __forceinline__ int width() const { return D(); }
  __device__ __forceinline__ int32_t col(int64_t item) const { return dofs[item]; }
  __device__ __forceinline__ int32_t slot(int64_t item) const {
    return (int32_t)(item / D() * (D() * (int64_t)D()) + item % D());
  }
  __device__ __forceinline__ int32_t row(int32_t slot) const {
    const int32_t col_of = slot / D();  // D t + i
    return dofs[col_of];
  }
  __device__ __forceinline__ int32_t listed(const int32_t *perm, int q) const {
    return perm[q / D() * D()] + q % D() * D();
  }
};

template <typename List>
__global__ void k_coo_count(List list, int64_t items, int64_t N, int32_t *cnt, int64_t *st) {
  const int64_t k = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (k >= items) return;
  const int32_t c = list.col(k);
  if (c < 0 || c >= N) {
    flag(st, EMG_ST_INDEX, list.slot(k));
    return;
  }
  atomicAdd(&cnt[c], list.width());
}

// each item's first slot to the start of its part of the column's list
template <typename List>
__global__ void k_coo_scatter(List list, int64_t items, int64_t N, const int32_t *col_off, int32_t *cursor,
                              int32_t *perm) {
  const int64_t k = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (k >= items) return;
  const int32_t c = list.col(k);
  if (c < 0 || c >= N) return;
  perm[col_off[c] + atomicAdd(&cursor[c], list.width())] = list.slot(k);
}

// Sort each column's slots by (row, slot) and count its distinct rows: a warp per
// column, its keys in registers (bitonic network, 32 K keys). An element's node
// columns hold 10 slots of some 24 tets, its edge columns of 5. A thread per
// column that inserted its slots one by one in global memory took 8,481 us at
// 99,900 tets (9.99M slots); this 120 us (k_coo_fill 191 -> 48). Bound: the gather
// of the slots' rows.
constexpr int SORT_WARPS = 8;

template <typename List>
__device__ __forceinline__ uint64_t coo_key(const List &list, int32_t slot) {
  return ((uint64_t)(uint32_t)list.row(slot) << 32) | (uint32_t)slot;
}

// sorts the column's n <= 32 K slots perm[0..n); returns its distinct rows
template <int K, typename List>
__device__ __forceinline__ int32_t sort_column(const List &list, int64_t N, int32_t *perm, int n, int64_t *st) {
  const int lane = threadIdx.x & 31;
  uint64_t k[K];
#pragma unroll
  for (int r = 0; r < K; ++r) k[r] = r * 32 + lane < n ? coo_key(list, list.listed(perm, r * 32 + lane)) : ~0ull;
  __syncwarp();  // every lane has read the list before any writes it
  warp_sort<K>(k);
  int32_t distinct = 0;
#pragma unroll
  for (int r = 0; r < K; ++r) {
    const int32_t row = (int32_t)(k[r] >> 32), slot = (int32_t)(uint32_t)k[r];
    int32_t before = __shfl_up_sync(0xffffffffu, row, 1);
    if (r > 0) {
      const int32_t last = __shfl_sync(0xffffffffu, (int32_t)(k[r > 0 ? r - 1 : 0] >> 32), 31);
      if (lane == 0) before = last;
    }
    const bool in = r * 32 + lane < n;
    if (in) {
      perm[r * 32 + lane] = slot;
      if (row < 0 || row >= N) flag(st, EMG_ST_INDEX, slot);
    }
    distinct += __popc(__ballot_sync(0xffffffffu, in && (r * 32 + lane == 0 || row != before)));
  }
  return distinct;
}

// the same for a column of any length, in global memory: a bitonic network
// whose comparators all put the smaller key first, so that those past the end
// of the column can be left out
template <typename List>
__device__ int32_t sort_long_column(const List &list, int64_t N, int32_t *perm, int64_t n, int64_t *st) {
  const int lane = threadIdx.x & 31, width = list.width();
  for (int64_t q = (int64_t)lane * width; width > 1 && q < n; q += 32 * (int64_t)width)  // an item's slots, in its part
    for (int i = 1; i < width; ++i) perm[q + i] = perm[q] + i * width;
  __syncwarp();
  for (int64_t size = 2; (size >> 1) < n; size <<= 1)
    for (int64_t j = size >> 1; j > 0; j >>= 1) {
      const bool flip = j == (size >> 1);
      for (int64_t c = lane; c < (n + 2 * j - 1) / (2 * j) * j; c += 32) {
        const int64_t block = c / j * (2 * j), at = c % j;
        const int64_t i = block + at, o = flip ? block + 2 * j - 1 - at : i + j;
        if (o < n) {
          const int32_t a = perm[i], b = perm[o];
          if (coo_key(list, a) > coo_key(list, b)) {
            perm[i] = b;
            perm[o] = a;
          }
        }
      }
      __syncwarp();
    }
  int32_t distinct = 0;
  for (int64_t i = lane; i < n; i += 32) {
    const int32_t r = list.row(perm[i]);
    if (r < 0 || r >= N) flag(st, EMG_ST_INDEX, perm[i]);
    distinct += i == 0 || r != list.row(perm[i - 1]) ? 1 : 0;
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) distinct += __shfl_xor_sync(0xffffffffu, distinct, o);
  return distinct;
}

// one warp, a column of any length
template <typename List>
__device__ int32_t sort_any_column(const List &list, int64_t N, int32_t *perm, int n, int64_t *st) {
  if (n <= 32) return sort_column<1>(list, N, perm, n, st);
  if (n <= 64) return sort_column<2>(list, N, perm, n, st);
  if (n <= 128) return sort_column<4>(list, N, perm, n, st);
  if (n <= 256) return sort_column<8>(list, N, perm, n, st);
  if (n <= 512) return sort_column<16>(list, N, perm, n, st);
  return sort_long_column(list, N, perm, n, st);
}

// indices (distinct rows) and, per entry, the first of its sorted slots: a warp
// per column
template <typename List>
__device__ __forceinline__ void fill_column(const List &list, int64_t b, int64_t e, int32_t q, const int32_t *perm,
                                            int32_t *indices, int32_t *run) {
  const int lane = threadIdx.x & 31;
  int32_t last = -1;
  for (int64_t i0 = b; i0 < e; i0 += 32) {  // i0 passes e, which may be nearly the last int32
    const int64_t i = i0 + lane;
    const int32_t r = i < e ? list.row(perm[i]) : -1;
    int32_t before = __shfl_up_sync(0xffffffffu, r, 1);
    if (lane == 0) before = last;
    const bool first = i < e && (i == b || r != before);
    const unsigned m = __ballot_sync(0xffffffffu, first);
    if (first) {
      const int32_t at = q + __popc(m & ((1u << lane) - 1u));
      indices[at] = r;
      run[at] = (int32_t)i;
    }
    q += __popc(m);
    last = __shfl_sync(0xffffffffu, r, 31);
  }
}

template <typename List>
__global__ void __launch_bounds__(SORT_WARPS * 32)
    k_coo_sort_count(List list, const int32_t *col_off, int64_t N, int32_t *perm, int32_t *col_nnz,
                     int64_t *st) {
  const int64_t c = (int64_t)blockIdx.x * SORT_WARPS + (threadIdx.x >> 5);
  if (c >= N) return;
  const int32_t b = col_off[c], n = col_off[c + 1] - b;
  const int32_t distinct = sort_any_column(list, N, perm + b, n, st);
  if ((threadIdx.x & 31) == 0) col_nnz[c] = distinct;
}

template <typename List>
__global__ void __launch_bounds__(SORT_WARPS * 32)
    k_coo_fill(List list, const int32_t *col_off, int64_t N, const int32_t *perm, const int32_t *indptr,
               int32_t *indices, int32_t *run) {
  const int64_t c = (int64_t)blockIdx.x * SORT_WARPS + (threadIdx.x >> 5);
  if (c >= N) return;
  fill_column(list, col_off[c], col_off[c + 1], indptr[c], perm, indices, run);
}

// Columns that hold few slots on average (a list of scattered entries, empty
// columns): a lane per column, and the warp together for those of its 32 that are
// longer than COO_LANE slots. The whole mapping of random slots, a warp per column
// -> this: 2M columns, no slots 0.75 -> 0.18 ms, 2M slots 0.97 -> 0.24, 6M 1.17 ->
// 0.37; 1M columns, 8M 0.77 -> 0.52, 10M 0.86 -> 0.64, 16M 1.11 -> 0.92. But 20,000
// columns, 200,000 slots 0.152 -> 0.183: from 10 slots per column on there are longer
// columns in every warp, and few columns leave it too few warps.
constexpr int COO_LANE = 8;
constexpr int COO_SHORT = 10;  // slots per column, on average

// one lane, n <= COO_LANE slots
template <typename List>
__device__ __forceinline__ int32_t sort_short_column(const List &list, int64_t N, int32_t *perm, int n, int64_t *st) {
  uint64_t k[COO_LANE];
#pragma unroll
  for (int q = 0; q < COO_LANE; ++q) k[q] = q < n ? coo_key(list, list.listed(perm, q)) : ~0ull;
#pragma unroll
  for (int round = 0; round < COO_LANE; ++round)
#pragma unroll
    for (int q = round & 1; q + 1 < COO_LANE; q += 2) {
      const uint64_t lo = k[q] < k[q + 1] ? k[q] : k[q + 1], hi = k[q] < k[q + 1] ? k[q + 1] : k[q];
      k[q] = lo;
      k[q + 1] = hi;
    }
  int32_t distinct = 0;
#pragma unroll
  for (int q = 0; q < COO_LANE; ++q) {
    if (q >= n) continue;
    const int32_t row = (int32_t)(k[q] >> 32), slot = (int32_t)(uint32_t)k[q];
    perm[q] = slot;
    if (row < 0 || row >= N) flag(st, EMG_ST_INDEX, slot);
    distinct += q == 0 || row != (int32_t)(k[q > 0 ? q - 1 : 0] >> 32) ? 1 : 0;
  }
  return distinct;
}

template <typename List>
__global__ void __launch_bounds__(SORT_WARPS * 32)
    k_coo_sort_count_short(List list, const int32_t *col_off, int64_t N, int32_t *perm, int32_t *col_nnz,
                           int64_t *st) {
  const int64_t c = (int64_t)blockIdx.x * (SORT_WARPS * 32) + threadIdx.x;
  const int32_t b = c < N ? col_off[c] : 0, n = c < N ? col_off[c + 1] - b : 0;
  int32_t distinct = n <= COO_LANE ? sort_short_column(list, N, perm + b, n, st) : 0;
  for (unsigned more = __ballot_sync(0xffffffffu, n > COO_LANE); more; more &= more - 1) {
    const int src = __ffs(more) - 1;
    const int32_t bs = __shfl_sync(0xffffffffu, b, src), ns = __shfl_sync(0xffffffffu, n, src);
    const int32_t d = sort_any_column(list, N, perm + bs, ns, st);
    if ((threadIdx.x & 31) == src) distinct = d;
  }
  if (c < N) col_nnz[c] = distinct;
}

template <typename List>
__global__ void __launch_bounds__(SORT_WARPS * 32)
    k_coo_fill_short(List list, const int32_t *col_off, int64_t N, const int32_t *perm, const int32_t *indptr,
                     int32_t *indices, int32_t *run) {
  const int64_t c = (int64_t)blockIdx.x * (SORT_WARPS * 32) + threadIdx.x;
  const int32_t b = c < N ? col_off[c] : 0, e = c < N ? col_off[c + 1] : 0, n = e - b;
  int32_t q = c < N ? indptr[c] : 0;
  for (unsigned more = __ballot_sync(0xffffffffu, n > COO_LANE); more; more &= more - 1) {
    const int src = __ffs(more) - 1;
    fill_column(list, __shfl_sync(0xffffffffu, b, src), __shfl_sync(0xffffffffu, e, src),
                __shfl_sync(0xffffffffu, q, src), perm, indices, run);
  }
  if (n > COO_LANE) return;
  int32_t before = -1;
#pragma unroll
  for (int i = 0; i < COO_LANE; ++i) {
    if (i >= n) break;
    const int32_t r = list.row(perm[b + i]);
    if (i == 0 || r != before) {
      indices[q] = r;
      run[q++] = b + i;
    }
    before = r;
  }
}

__global__ void k_coo_run_end(const int32_t *run, int64_t nnz, int64_t S, int32_t *run_end) {
  if (blockIdx.x == 0 && threadIdx.x == 0) run_end[nnz] = (int32_t)S;
}

// the value index of slot s: s itself, or, for values stored as transposed
// D x D blocks (slot D^2 t + D i + j at D^2 t + D j + i), the swapped one
template <int D>
__device__ __forceinline__ int64_t value_index(int32_t s) {
  if constexpr (D == 0) {
    return s;
  } else {
    const int32_t t = s / (D * D), r = s - t * (D * D);
    const int32_t i = r / D, j = r - i * D;
    return (int64_t)t * (D * D) + j * D + i;
  }
}

template <int D>
__global__ void __launch_bounds__(256, 8) k_coo_gather_f8(const int32_t *perm, const int32_t *run, int64_t nnz,
                                                          int64_t S, const double *vals, double *out) {
  // the run bounds of this thread's next entry are loaded while the current
  // entry is summed (one dependent load off each entry's chain)
  const int64_t stride = (int64_t)gridDim.x * blockDim.x;
  int64_t p = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  int32_t nb = 0, ne = 0;
  if (p < nnz) {
    nb = run[p];
    ne = run[p + 1];
  }
  for (; p < nnz; p += stride) {
    const int32_t b = nb, e = min((int64_t)ne, S);
    if (p + stride < nnz) {
      nb = run[p + stride];
      ne = run[p + stride + 1];
    }
    double s = 0.0;
    int32_t i = b;
    for (; e - i >= 4; i += 4) {  // four loads in flight, summed in slot order
      const int32_t p0 = perm[i], p1 = perm[i + 1], p2 = perm[i + 2], p3 = perm[i + 3];
      const double v0 = vals[value_index<D>(p0)], v1 = vals[value_index<D>(p1)];
      const double v2 = vals[value_index<D>(p2)], v3 = vals[value_index<D>(p3)];
      s += v0;
      s += v1;
      s += v2;
      s += v3;
    }
    if (e - i >= 2) {
      const int32_t p0 = perm[i], p1 = perm[i + 1];
      const double v0 = vals[value_index<D>(p0)], v1 = vals[value_index<D>(p1)];
      s += v0;
      s += v1;
      i += 2;
    }
    if (i < e) s += vals[value_index<D>(perm[i])];
    out[p] = s;
  }
}

template <int D>
__global__ void __launch_bounds__(256) k_coo_gather_c16(const int32_t *perm, const int32_t *run, int64_t nnz,
                                                        int64_t S, const double2 *vals, double2 *out) {
  for (int64_t p = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; p < nnz; p += (int64_t)gridDim.x * blockDim.x) {
    const int32_t b = run[p], e = run[p + 1];
    double sr = 0.0, si = 0.0;
    for (int32_t i = b; i < e && i < S; ++i) {
      const double2 v = vals[value_index<D>(perm[i])];
      sr += v.x;
      si += v.y;
    }
    out[p] = make_double2(sr, si);
  }
}

// rows/cols of an element with D DoFs per tet in the reference layout
// (femdata.py:58-73, grad.py:350-354): slot p = D^2 t + D ii + jj
__global__ void k_coo_rowcol(const int32_t *t2f, int D, int64_t nT, int32_t *rows, int32_t *cols) {
  const int64_t s = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  const int64_t D2 = (int64_t)D * D;
  if (s >= D2 * nT) return;
  const int64_t t = s / D2;
  const int r = (int)(s % D2);
  rows[s] = t2f[(int64_t)(r / D) * nT + t];
  cols[s] = t2f[(int64_t)(r % D) * nT + t];
}

struct CooWs {
  int32_t *cnt, *col_off, *cursor, *col_nnz;
  long long *bsum;
};

CooWs coo_ws(void *d_ws, int64_t N) {
  char *w = static_cast<char *>(d_ws);
  CooWs r;
  size_t o = 0;
  r.cnt = reinterpret_cast<int32_t *>(w + o);
  o = align_up(o + (size_t)(N + 1) * 4, 256);
  r.col_off = reinterpret_cast<int32_t *>(w + o);
  o = align_up(o + (size_t)(N + 1) * 4, 256);
  r.cursor = reinterpret_cast<int32_t *>(w + o);
  o = align_up(o + (size_t)(N + 1) * 4, 256);
  r.col_nnz = reinterpret_cast<int32_t *>(w + o);
  o = align_up(o + (size_t)(N + 1) * 4, 256);
  r.bsum = reinterpret_cast<long long *>(w + o);
  return r;
}

template <typename List>
int coo_build(const List &list, int64_t items, emg_coo_map *m, int32_t *d_perm, void *d_ws, int32_t *d_indptr,
              int64_t *d_status, cudaStream_t s) {
  CooWs w = coo_ws(d_ws, m->N);
  int rc;
  if ((rc = status_reset(d_status, s))) return rc;
  CUDA_TRY(cudaMemsetAsync(w.cnt, 0, (size_t)(m->N + 1) * 4, s));
  CUDA_TRY(cudaMemsetAsync(w.cursor, 0, (size_t)(m->N + 1) * 4, s));
  if (items > 0) {
    k_coo_count<<<grid_for(items, 256), 256, 0, s>>>(list, items, m->N, w.cnt, d_status);
    if ((rc = launch_check("k_coo_count"))) return rc;
  }
  if ((rc = scan_i32(w.cnt, m->N, w.col_off, w.bsum, d_status, s))) return rc;
  if (items > 0) {
    k_coo_scatter<<<grid_for(items, 256), 256, 0, s>>>(list, items, m->N, w.col_off, w.cursor, d_perm);
    if ((rc = launch_check("k_coo_scatter"))) return rc;
  }
  if (m->N > 0) {
    if (m->S < COO_SHORT * m->N)
      k_coo_sort_count_short<<<grid_for(m->N, SORT_WARPS * 32), SORT_WARPS * 32, 0, s>>>(list, w.col_off, m->N, d_perm,
                                                                                         w.col_nnz, d_status);
    else
      k_coo_sort_count<<<grid_for(m->N, SORT_WARPS), SORT_WARPS * 32, 0, s>>>(list, w.col_off, m->N, d_perm, w.col_nnz,
                                                                              d_status);
    if ((rc = launch_check("k_coo_sort_count"))) return rc;
  }
  if ((rc = scan_i32(w.col_nnz, m->N, d_indptr, w.bsum, d_status, s))) return rc;
  int32_t nnz = 0;
  int64_t h_st[2] = {0, 0};
  CUDA_TRY(cudaMemcpyAsync(&nnz, d_indptr + m->N, 4, cudaMemcpyDeviceToHost, s));
  CUDA_TRY(cudaMemcpyAsync(h_st, d_status, 16, cudaMemcpyDeviceToHost, s));
  CUDA_TRY(cudaStreamSynchronize(s));
  if (h_st[0]) return fail(EMG_EMESH, "COO pattern: index out of range at slot %lld", (long long)h_st[1]);
  m->nnz = nnz;
  return EMG_OK;
}

template <typename List>
int coo_finish(const List &list, const emg_coo_map *m, const int32_t *d_perm, void *d_ws, const int32_t *d_indptr,
               int32_t *d_indices, int32_t *d_run, cudaStream_t s) {
  CooWs w = coo_ws(d_ws, m->N);
  if (m->N > 0) {
    if (m->S < COO_SHORT * m->N)
      k_coo_fill_short<<<grid_for(m->N, SORT_WARPS * 32), SORT_WARPS * 32, 0, s>>>(list, w.col_off, m->N, d_perm,
                                                                                   d_indptr, d_indices, d_run);
    else
      k_coo_fill<<<grid_for(m->N, SORT_WARPS), SORT_WARPS * 32, 0, s>>>(list, w.col_off, m->N, d_perm, d_indptr,
                                                                        d_indices, d_run);
    const int rc = launch_check("k_coo_fill");
    if (rc) return rc;
  }
  k_coo_run_end<<<1, 32, 0, s>>>(d_run, m->nnz, m->S, d_run);
  return launch_check("k_coo_run_end");
}

}  // namespace
}  // namespace emg

using namespace emg;

extern "C" {

int emg_coo_init(int64_t S, int64_t N, emg_coo_map *m) {
  if (!m) return fail(EMG_EINVAL, "null descriptor");
  if (S < 0 || N < 0) return fail(EMG_EINVAL, "negative size");
  if (S >= INT32_MAX || N >= INT32_MAX) return fail(EMG_ERANGE, "more than 2^31 slots or columns");
  memset(m, 0, sizeof(*m));
  m->S = S;
  m->N = N;
  m->perm_bytes = align_up((size_t)(S > 0 ? S : 1) * 4, 256);
  m->run_bytes = align_up((size_t)(S + 1) * 4, 256);
  m->workspace_bytes = align_up((size_t)(N + 1) * 4, 256) * 4 + scan_i32_bsum_bytes(N + 1);
  return EMG_OK;
}

int emg_coo_rowcol(const int32_t *d_tet_to_field, int dofs_per_tet, int64_t n_tets, int32_t *d_rows, int32_t *d_cols,
                   emg_stream_t stream) {
  if (dofs_per_tet <= 0 || n_tets < 0) return fail(EMG_EINVAL, "bad sizes");
  const int64_t n = (int64_t)dofs_per_tet * dofs_per_tet * n_tets;
  if (n == 0) return EMG_OK;
  if (n >= INT32_MAX) return fail(EMG_ERANGE, "more than 2^31 slots");
  if (!d_tet_to_field || !d_rows || !d_cols) return fail(EMG_EINVAL, "null pointer");
  k_coo_rowcol<<<grid_for(n, 256), 256, 0, S(stream)>>>(d_tet_to_field, dofs_per_tet, n_tets, d_rows, d_cols);
  return launch_check("k_coo_rowcol");
}

int emg_coo_build(emg_coo_map *m, const int32_t *d_rows, const int32_t *d_cols, int32_t *d_perm, void *d_ws,
                  int32_t *d_indptr, int64_t *d_status, emg_stream_t stream) {
  if (!m || !d_perm || !d_ws || !d_indptr || !d_status || (m->S > 0 && (!d_rows || !d_cols)))
    return fail(EMG_EINVAL, "null pointer");
  return coo_build(SlotList{d_rows, d_cols}, m->S, m, d_perm, d_ws, d_indptr, d_status, S(stream));
}

int emg_coo_finish(const emg_coo_map *m, const int32_t *d_rows, const int32_t *d_perm, void *d_ws,
                   const int32_t *d_indptr, int32_t *d_indices, int32_t *d_run, emg_stream_t stream) {
  if (!m || !d_perm || !d_ws || !d_indptr || !d_run) return fail(EMG_EINVAL, "null pointer");
  if (m->nnz > 0 && (!d_indices || !d_rows)) return fail(EMG_EINVAL, "null pointer");
  return coo_finish(SlotList{d_rows, nullptr}, m, d_perm, d_ws, d_indptr, d_indices, d_run, S(stream));
}

int emg_coo_build_blocks(emg_coo_map *m, const int32_t *d_dofs, int dofs_per_tet, int32_t *d_perm, void *d_ws,
                         int32_t *d_indptr, int64_t *d_status, emg_stream_t stream) {
  if (!m || !d_perm || !d_ws || !d_indptr || !d_status || (m->S > 0 && !d_dofs))
    return fail(EMG_EINVAL, "null pointer");
  const int64_t D = dofs_per_tet;
  if (D <= 0 || m->S % (D * D)) return fail(EMG_EINVAL, "slot count is not a multiple of the block size");
  if (D == 10) return coo_build(BlockList<10>{d_dofs, 10}, m->S / 10, m, d_perm, d_ws, d_indptr, d_status, S(stream));
  return coo_build(BlockList<0>{d_dofs, dofs_per_tet}, m->S / D, m, d_perm, d_ws, d_indptr, d_status, S(stream));
}

int emg_coo_finish_blocks(const emg_coo_map *m, const int32_t *d_dofs, int dofs_per_tet, const int32_t *d_perm,
                          void *d_ws, const int32_t *d_indptr, int32_t *d_indices, int32_t *d_run,
                          emg_stream_t stream) {
  if (!m || !d_perm || !d_ws || !d_indptr || !d_run || dofs_per_tet <= 0) return fail(EMG_EINVAL, "null pointer");
  if (m->nnz > 0 && (!d_indices || !d_dofs)) return fail(EMG_EINVAL, "null pointer");
  if (dofs_per_tet == 10)
    return coo_finish(BlockList<10>{d_dofs, 10}, m, d_perm, d_ws, d_indptr, d_indices, d_run, S(stream));
  return coo_finish(BlockList<0>{d_dofs, dofs_per_tet}, m, d_perm, d_ws, d_indptr, d_indices, d_run, S(stream));
}

int emg_coo_gather(const emg_coo_map *m, const int32_t *d_perm, const int32_t *d_run, int is_complex, int block_dofs,
                   const void *d_values, void *d_out, emg_stream_t stream) {
  if (!m) return fail(EMG_EINVAL, "null descriptor");
  if (block_dofs != 0 && block_dofs != 10) return fail(EMG_EINVAL, "block_dofs must be 0 or 10");
  if (block_dofs && m->S % 100) return fail(EMG_EINVAL, "slot count is not a multiple of the block size");
  if (m->nnz == 0) return EMG_OK;
  if (!d_perm || !d_run || !d_values || !d_out) return fail(EMG_EINVAL, "null pointer");
  const int g = persistent_ctas(8);
  cudaStream_t s = S(stream);
  const int64_t n = m->nnz, S_ = m->S;
  if (is_complex) {
    auto v = static_cast<const double2 *>(d_values);
    auto o = static_cast<double2 *>(d_out);
    if (block_dofs)
      k_coo_gather_c16<10><<<g, 256, 0, s>>>(d_perm, d_run, n, S_, v, o);
    else
      k_coo_gather_c16<0><<<g, 256, 0, s>>>(d_perm, d_run, n, S_, v, o);
  } else {
    auto v = static_cast<const double *>(d_values);
    auto o = static_cast<double *>(d_out);
    if (block_dofs)
      k_coo_gather_f8<10><<<g, 256, 0, s>>>(d_perm, d_run, n, S_, v, o);
    else
      k_coo_gather_f8<0><<<g, 256, 0, s>>>(d_perm, d_run, n, S_, v, o);
  }
  return launch_check("k_coo_gather");
}

}  // extern "C"
