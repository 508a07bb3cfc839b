// gather.cu -- column gather + segmented sum, and the frequency-sweep form.
//
// Replaces CSCMapping.to_csc / scatter_to_csc_c16 (mth/csc_cast.py:55-63,
// 162-177) and the caller's COO combination Evec - Bvec*k0^2
// (physics/microwave/assembly/assembler.py:494).
#include <type_traits>
#include "common.cuh"

namespace emg {
namespace {

struct C64 {
  double re, im;
};


// L2 eviction priority "evict last" for the element values: each
// off-diagonal block is read twice, by the chunks of its two entities, and
// the second read comes after some of A and of the records have streamed
// through L2. Marking the value reads evict-last (createpolicy, a per-load
// hint; no device setting changes) keeps more of them resident for that
// second read (1.008M tets: complex128 gather 1,628 -> 1,598 us, complex64 1,425 ->
// 1,398); evict-first on A's stores: 1,610 / 1,440.
__device__ __forceinline__ uint64_t policy_evict_last() {
  uint64_t p;
  asm volatile("createpolicy.fractional.L2::evict_last.b64 %0, 1.0;" : "=l"(p));
  return p;
}

template <typename R>
__device__ __forceinline__ C64 load_val_last(const void *p, int64_t idx, uint64_t pol) {
  if constexpr (sizeof(R) == 8) {
    double2 v;
    asm volatile("ld.global.nc.L2::cache_hint.v2.f64 {%0, %1}, [%2], %3;"
                 : "=d"(v.x), "=d"(v.y)
                 : "l"(reinterpret_cast<const double2 *>(p) + idx), "l"(pol));
    return {v.x, v.y};
  } else {
    float2 v;
    asm volatile("ld.global.nc.L2::cache_hint.v2.f32 {%0, %1}, [%2], %3;"
                 : "=f"(v.x), "=f"(v.y)
                 : "l"(reinterpret_cast<const float2 *>(p) + idx), "l"(pol));
    return {(double)v.x, (double)v.y};
  }
}

template <typename R>
__device__ __forceinline__ C64 load_val(const void *p, int64_t idx) {
  if constexpr (sizeof(R) == 8) {
    double2 v = reinterpret_cast<const double2 *>(p)[idx];
    return {v.x, v.y};
  } else {
    float2 v = reinterpret_cast<const float2 *>(p)[idx];
    return {(double)v.x, (double)v.y};
  }
}

// Packed gather. A warp owns one entity chunk (CHUNK consecutive entities of one
// kind, see common.cuh); its two output runs are contiguous. Lane l owns
// positions l, l+32, ... of the runs: it reads the position's contribution list
// from the plan, sums the contributing element values in that fixed order (items
// ascending, so tets ascending), and writes the first-DoF and second-DoF entries
// once. No shared memory, no atomics; each nonzero is produced by exactly one
// lane.
constexpr int PG_WARPS = 8;

// element slots (row r, column a0) and (row r, column a1) of the reference COO
// block: the item's contributions to its entity's two columns
template <typename R>
__device__ __forceinline__ void load_coo_pair(const void *v, int ia, int slot, int r, C64 &u0, C64 &u1) {
  const int a0 = slot < 6 ? slot : 12 + (slot - 6);
  const int a1 = slot < 6 ? slot + 6 : 16 + (slot - 6);
  const int64_t base = (int64_t)ia * 400 + r * 20;
  u0 = load_val<R>(v, base + a0);
  u1 = load_val<R>(v, base + a1);
}

struct ChunkMeta {
  int32_t I0, I1, A0, A1, Lsum;
  int64_t hbase;
  int64_t x0, cb0;  // first entity of the chunk and its first-DoF column
  int nx;           // entities in the chunk
};

// Processing position g -> chunk through the plan's order array (the default
// interleave, or a spatial order from emg_plan_order), so that the element
// values of a region's tets are read while still in L2.
__device__ __forceinline__ bool chunk_meta(const int32_t *ent_ptr, const int32_t *order, const int32_t *indptr,
                                           int64_t E, int64_t F, int64_t g, ChunkMeta &m) {
  const int lane = threadIdx.x & 31;
  const int64_t nec = n_edge_chunks(E);
  const int64_t nch = n_chunks(E, F);
  if (g >= nch) return false;
  const int64_t chunk = __ldg(order + g);
  if (chunk < 0 || chunk >= nch) return false;  // only a corrupted plan can hold this
  const bool edges = chunk < nec;
  const int64_t x0 = edges ? chunk * CHUNK : E + (chunk - nec) * CHUNK;
  const int nx = (int)min((int64_t)CHUNK, (edges ? E : E + F) - x0);
  const int64_t cb0 = edges ? x0 : E + x0;          // first-DoF column of x0 (faces: 2E + (x0 - E))
  const int64_t cb1 = edges ? x0 + E : E + F + x0;  // second-DoF column of x0
  int32_t meta = 0;
  if (lane == 0) meta = ent_ptr[x0];
  else if (lane == 1) meta = ent_ptr[x0 + nx];
  else if (lane == 2) meta = indptr[cb0];
  else if (lane == 3) meta = indptr[cb0 + nx];
  else if (lane == 4) meta = indptr[cb1];
  else if (lane == 5) meta = edges ? 0 : indptr[E];
  else if (lane == 6) meta = edges ? 0 : indptr[2 * E];
  m.I0 = __shfl_sync(0xffffffffu, meta, 0);
  m.I1 = __shfl_sync(0xffffffffu, meta, 1);
  m.A0 = __shfl_sync(0xffffffffu, meta, 2);
  m.Lsum = __shfl_sync(0xffffffffu, meta, 3) - m.A0;
  m.A1 = __shfl_sync(0xffffffffu, meta, 4);
  const int32_t cE = __shfl_sync(0xffffffffu, meta, 5), c2E = __shfl_sync(0xffffffffu, meta, 6);
  m.hbase = edges ? (int64_t)m.A0 : (int64_t)cE + (m.A0 - c2E);
  m.x0 = x0;
  m.cb0 = cb0;
  m.nx = nx;
  return true;
}

// Reference COO layout (any COO data of this field's slot layout), a warp per
// entity: its two columns are summed in shared memory, item by item in the
// plan's order, so that each entry adds its contributions in the order of the
// other layouts; the plan holds no lists for it. The 20 rows of an item's tet are
// 20 different rows of the column, one lane each, and the values of COO_ITEMS
// items are in flight.
constexpr int COO_ITEMS = 4;

template <typename R, bool TWO>
__global__ void k_gather_coo(const int32_t *ent_ptr, const int32_t *order, const Item *items, const uint32_t *ent_cnt,
                             int64_t E, int64_t F, const int32_t *indptr, const void *v1, const void *v2, double ar,
                             double ai, double br, double bi, int max_col, double2 *A) {
  extern __shared__ __align__(16) double2 coo_cols[];
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  const int64_t g = (int64_t)blockIdx.x * (blockDim.x >> 5) + w;
  const int64_t nec = n_edge_chunks(E), nch = n_chunks(E, F);
  if (g >= nch * CHUNK) return;
  const int64_t chunk = __ldg(order + g / CHUNK);
  if (chunk < 0 || chunk >= nch) return;  // only a corrupted plan can hold this
  const bool edges = chunk < nec;
  const int64_t x = (edges ? chunk * CHUNK : E + (chunk - nec) * CHUNK) + g % CHUNK;
  if (x >= (edges ? E : E + F)) return;
  const int64_t c0 = edges ? x : E + x, c1 = edges ? x + E : E + F + x;
  const int64_t A0 = indptr[c0], A1 = indptr[c1];
  const int rows = (int)(indptr[c0 + 1] - A0);
  if (rows > max_col) return;  // as above
  const uint32_t cnt = ent_cnt[x];
  const int ne = (int)(cnt & 0xffffu), nf = (int)(cnt >> 16);
  double2 *s0 = coo_cols + (int64_t)w * 2 * max_col, *s1 = s0 + max_col;
  for (int i = lane; i < rows; i += 32) s0[i] = s1[i] = make_double2(0.0, 0.0);
  __syncwarp();
  const int r = lane;  // row slot of the tet
  const int slot = r < 6 ? r : (r < 12 ? r - 6 : (r < 16 ? r - 6 : r - 10));
  const int off = r < 6 ? 0 : (r < 12 ? ne : (r < 16 ? 2 * ne : 2 * ne + nf));
  const int b = ent_ptr[x], e = ent_ptr[x + 1];
  for (int k0 = b; k0 < e; k0 += COO_ITEMS) {
    C64 u[COO_ITEMS][2], t[COO_ITEMS][2];
    int at[COO_ITEMS];
#pragma unroll
    for (int k = 0; k < COO_ITEMS; ++k) {
      at[k] = -1;
      if (k0 + k >= e || r >= 20) continue;
      const Item rec = items[k0 + k];
      at[k] = off + rec.pos[slot];
      load_coo_pair<R>(v1, rec.ia, rec.slot, r, u[k][0], u[k][1]);
      if (TWO) load_coo_pair<R>(v2, rec.ia, rec.slot, r, t[k][0], t[k][1]);
    }
#pragma unroll
    for (int k = 0; k < COO_ITEMS; ++k) {
      if (at[k] >= 0 && at[k] < rows)
#pragma unroll
        for (int c = 0; c < 2; ++c) {
          double2 s = (c ? s1 : s0)[at[k]];
          s.x += ar * u[k][c].re - ai * u[k][c].im;
          s.y += ar * u[k][c].im + ai * u[k][c].re;
          if (TWO) {
            s.x += br * t[k][c].re - bi * t[k][c].im;
            s.y += br * t[k][c].im + bi * t[k][c].re;
          }
          (c ? s1 : s0)[at[k]] = s;
        }
      __syncwarp();
    }
  }
  for (int i = lane; i < rows; i += 32) {
    A[A0 + i] = s0[i];
    A[A1 + i] = s1[i];
  }
}

// packed layout (the assembly path): per contribution the two value indices
// come from the plan, as an int2 or as one compact uint32 (first index + a
// bit, the second slot from kSecondSlot)
__constant__ SecondSlotTable kSecondSlot = make_second_slot_table();

// Complex128 values (R = double): the list bounds of a lane's next position
// are loaded while the current one is summed, which takes one dependent load
// off each position's chain, with the register count held for six CTAs per
// SM. Complex64 values keep the plain loop (32 registers and eight CTAs per SM
// with 8-byte records), where the prefetch measured slower.
// Warps per CTA and CTAs per SM. A warp's time follows its chunk's list
// lengths, and a CTA's slot frees only when its slowest warp ends, so small
// CTAs keep more warps resident: 4-warp CTAs, 12 per SM at 40 registers
// (complex128) or 16 at 32 (complex64). Compact records keep 8-warp CTAs.
template <typename R, bool COMPACT>
struct PackedShape {
  static constexpr bool c128 = std::is_same<R, double>::value;
  static constexpr int warps = !COMPACT ? 4 : PG_WARPS;
  static constexpr int min_blocks = (c128 && !COMPACT) ? 12 : (!COMPACT ? 16 : 6);
};

// One warp's chunk of the packed gather (chunk meta already read).
template <typename R, bool COMPACT>
__device__ __forceinline__ void gather_packed_chunk(const ChunkMeta &m, const void *pidx_v, const uint16_t *posoff,
                                                    int64_t n_values, const void *v, double ar, double ai,
                                                    double2 *A, const uint8_t (*slot2)[210]) {
  const int lane = threadIdx.x & 31;
  const int total = 20 * (m.I1 - m.I0);
  constexpr bool PREFETCH = std::is_same<R, double>::value;
  int n0 = 0, n1 = 0;
  if (PREFETCH && lane < m.Lsum) {
    n0 = posoff[m.hbase + lane];
    n1 = lane + 1 < m.Lsum ? (int)posoff[m.hbase + lane + 1] : total;
  }
  for (int p = lane; p < m.Lsum; p += 32) {
    int o0, o1;
    if constexpr (PREFETCH) {
      o0 = n0;
      o1 = min(n1, total);
      if (p + 32 < m.Lsum) {
        n0 = posoff[m.hbase + p + 32];
        n1 = p + 33 < m.Lsum ? (int)posoff[m.hbase + p + 33] : total;
      }
    } else {
      o0 = posoff[m.hbase + p];
      o1 = min(p + 1 < m.Lsum ? (int)posoff[m.hbase + p + 1] : total, total);
    }
    double s0r = 0.0, s0i = 0.0, s1r = 0.0, s1i = 0.0;
    for (int k = o0; k < o1; ++k) {
      int64_t qx, qy;
      if constexpr (COMPACT) {
        const uint32_t c = __ldg(static_cast<const uint32_t *>(pidx_v) + (int64_t)20 * m.I0 + k);
        const uint32_t x = c & 0x7fffffffu;
        const uint32_t p0 = x % 210u;
        qx = x;
        qy = (int64_t)(x - p0) + slot2[c >> 31][p0];
      } else {
        const int2 q = __ldg(static_cast<const int2 *>(pidx_v) + (int64_t)20 * m.I0 + k);
        qx = (uint32_t)q.x;
        qy = (uint32_t)q.y;
      }
      if (qx >= n_values || qy >= n_values) continue;
      const C64 u0 = load_val<R>(v, qx), u1 = load_val<R>(v, qy);
      s0r += u0.re;
      s0i += u0.im;
      s1r += u1.re;
      s1i += u1.im;
    }
    A[m.A0 + p] = make_double2(ar * s0r - ai * s0i, ar * s0i + ai * s0r);
    A[m.A1 + p] = make_double2(ar * s1r - ai * s1i, ar * s1i + ai * s1r);
  }
}


template <typename R, bool COMPACT>
__global__ void __launch_bounds__(PackedShape<R, COMPACT>::warps * 32, PackedShape<R, COMPACT>::min_blocks)
    k_gather_packed(const int32_t *ent_ptr, const int32_t *order, const void *pidx_v, const uint16_t *posoff,
                    int64_t E, int64_t F, int64_t n_values, const int32_t *indptr, const void *v, double ar,
                    double ai, double2 *A) {
  __shared__ uint8_t slot2[2][210];
  if constexpr (COMPACT) {
    for (int i = threadIdx.x; i < 420; i += blockDim.x) slot2[i / 210][i % 210] = kSecondSlot.v[i / 210][i % 210];
    __syncthreads();
  }
  ChunkMeta m;
  if (!chunk_meta(ent_ptr, order, indptr, E, F,
                  (int64_t)blockIdx.x * PackedShape<R, COMPACT>::warps + (threadIdx.x >> 5), m))
    return;
  gather_packed_chunk<R, COMPACT>(m, pidx_v, posoff, n_values, v, ar, ai, A, slot2);
}

// ---- entity-pair block layout (EMG_LAYOUT_BLOCK). A row pair of a chunk's
// first-DoF run -- the first-DoF row p of an adjacent entity and its partner
// row p' (the entity's second DoF) -- gets four entries of A, the sums over its
// tets, in item order, of the 2x2 blocks of that entity pair.
//
// A CTA gathers one chunk. Two lanes share a row pair, half a block (two values,
// one 32-byte or, complex64, 16-byte load) each. Two different entities of a
// conforming mesh share at most two tets, so a row pair's record is two block
// numbers, loaded without a list start, and every lane has four loads in
// flight; only an entity's pair with itself (5-6 tets around an edge) is
// longer, and its list has a known place. Chain of dependent loads per chunk:
// descriptor, records, values.
//
// A lane per row pair that walked its list ran as long as the warp's longest
// list, 5-6 dependent record -> value loads where the mean list has 1.4: 1,008,000
// tets took 2,380 us complex128 and 1,850 complex64; now 1,600 and 1,402. Bound:
// HBM for complex128 (10.2 GB, 6.4 TB/s), latency for complex64 (5.0 TB/s).
// Two warps per CTA and 18 CTAs per SM (56 registers): 16 CTAs 1,653 / 1,447,
// 20 (spills) 1,793 / 1,445; one warp 1,812 / 1,488, four 1,761 / 1,544. Four
// lanes per row pair: 2,069 / 1,790. The chunk's runs of A staged in shared
// memory and written by bulk copies: 1,849 / 1,608 -- the stage takes the L1 that
// holds the loads in flight -- and with the chunks pipelined through cp.async, up
// to eight per CTA: 2,082 / 1,738.
constexpr int BG_WARPS = 2;
constexpr int BG_CTAS = 18;  // per SM

// value q (0..3) of the stored block of record r, or zero
template <typename R>
__device__ __forceinline__ C64 load_block_value(const void *v, uint32_t r, int q, uint32_t n_blocks, uint64_t pol) {
  const uint32_t b = r & 0x7fffffffu;
  if (b >= n_blocks) return {0.0, 0.0};  // no block (kBlockNone), or a plan whose build was flagged
  // bit 31: stored transposed, the middle two values swap
  return load_val_last<R>(v, 4 * (int64_t)b + (((r >> 31) && (q == 1 || q == 2)) ? 3 - q : q), pol);
}

// half y of block b: its values 2y and 2y + 1 (v_y: the values' start plus y
// halves); WIDE: one load, which needs the values aligned to half a block
template <typename R, bool WIDE>
__device__ __forceinline__ void load_half_block(const char *v_y, uint32_t b, uint32_t n_blocks, uint64_t pol, R u[4]) {
  u[0] = u[1] = u[2] = u[3] = 0;
  if (b >= n_blocks) return;
  const char *p = v_y + (uint64_t)b * (8 * sizeof(R));
  if constexpr (!WIDE) {
    const C64 a = load_val_last<R>(p, 0, pol), c = load_val_last<R>(p, 1, pol);
    u[0] = (R)a.re, u[1] = (R)a.im, u[2] = (R)c.re, u[3] = (R)c.im;
  } else if constexpr (sizeof(R) == 8) {
    asm volatile("ld.global.nc.L2::cache_hint.v4.f64 {%0, %1, %2, %3}, [%4], %5;"
                 : "=d"(u[0]), "=d"(u[1]), "=d"(u[2]), "=d"(u[3])
                 : "l"(p), "l"(pol));
  } else {
    asm volatile("ld.global.nc.L2::cache_hint.v4.f32 {%0, %1, %2, %3}, [%4], %5;"
                 : "=f"(u[0]), "=f"(u[1]), "=f"(u[2]), "=f"(u[3])
                 : "l"(p), "l"(pol));
  }
}

// The chunk's entities' pairs with themselves (lists of more than two), one
// warp: a quad of lanes per entity, one value of the block each, eight blocks
// in flight, added in list order.
template <typename R>
__device__ __forceinline__ void gather_self_pairs(const ChunkDesc &d, const uint32_t *self, uint32_t n_blocks,
                                                  const void *v, double ar, double ai, uint64_t pol, double2 *A) {
  const int lane = threadIdx.x & 31, q = lane & 3, e = lane >> 2, H = d.H;
  const int n = d.cnt[e];
  for (int k = 0; k < e; ++k) self += d.cnt[k];
  double sr = 0.0, si = 0.0;
  for (int k0 = 0; __any_sync(0xffffffffu, n > 2 && k0 < n); k0 += 8) {
    const uint32_t r0 = k0 + q < n ? __ldg(self + k0 + q) : kBlockNone;
    const uint32_t r1 = k0 + q + 4 < n ? __ldg(self + k0 + q + 4) : kBlockNone;
    R u[8][2];
#pragma unroll
    for (int k = 0; k < 8; ++k) {
      const uint32_t r = __shfl_sync(0xffffffffu, k < 4 ? r0 : r1, (lane & 28) | (k & 3));
      const C64 t = load_block_value<R>(v, r, q, n_blocks, pol);
      u[k][0] = (R)t.re, u[k][1] = (R)t.im;
    }
#pragma unroll
    for (int k = 0; k < 8; ++k) {
      sr += (double)u[k][0];
      si += (double)u[k][1];
    }
  }
  if (n > 2) {
    const int ne = d.ne[e], nf = (e + 1 < CHUNK ? d.hs[e + 1] : H) - d.hs[e] - ne;
    const int p = 2 * d.hs[e] + (d.faces ? 2 * ne : 0) + d.self[e] + ((q & 2) ? (d.faces ? nf : ne) : 0);
    if (p < 2 * H) A[((q & 1) ? d.A1 : d.A0) + p] = make_double2(ar * sr - ai * si, ar * si + ai * sr);
  }
}

template <typename R, bool WIDE>
__device__ __forceinline__ void gather_block_chunk(const ChunkDesc *desc, const uint32_t *brec, uint32_t n_blocks,
                                                   const void *v, double ar, double ai, double2 *A) {
  __shared__ ChunkDesc d;
  if (threadIdx.x < sizeof(ChunkDesc) / 4)
    reinterpret_cast<uint32_t *>(&d)[threadIdx.x] = __ldg(reinterpret_cast<const uint32_t *>(desc) + threadIdx.x);
  __syncthreads();
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5, y = lane & 1;
  const int H = d.H, to_A1 = d.A1 - d.A0;
  double2 *A0 = A + d.A0;
  const uint64_t pol = policy_evict_last();
  const char *v_y = static_cast<const char *>(v) + y * 4 * sizeof(R);
  const uint32_t *words = brec + (int64_t)kPairWords * d.I0;
  const uint2 *pairs = reinterpret_cast<const uint2 *>(words);
  const uint2 none = make_uint2(kBlockNone, kBlockNone);
  uint2 nxt = threadIdx.x < H ? __ldg(pairs + threadIdx.x) : none;
  if (w == BG_WARPS - 1) gather_self_pairs<R>(d, words + 2 * H, n_blocks, v, ar, ai, pol, A);

  for (int h0 = 32 * w; h0 < H; h0 += 32 * BG_WARPS) {
    const int h = h0 + lane;
    uint2 pr = nxt;  // the next records are loaded while these are summed
    nxt = h + 32 * BG_WARPS < H ? __ldg(pairs + h + 32 * BG_WARPS) : none;
    // the row pair's first row p in the run, p' - p, transposed
    uint32_t pk = 0;
    if (h < H) {
      int x = h >= d.hs[4] ? 4 : 0;
      x += h >= d.hs[x + 2] ? 2 : 0;
      x += h >= d.hs[x + 1] ? 1 : 0;
      const int hb = d.hs[x], hl = h - hb, ne = d.ne[x], nf = (x + 1 < CHUNK ? d.hs[x + 1] : H) - hb - ne;
      pk = (uint32_t)(hl < ne ? h + hb : h + hb + ne) | ((uint32_t)(hl < ne ? ne : nf) << 16) | (pr.x & 0x80000000u);
    }
    const bool is_long = pr.y == kBlockLong;
    // longer lists of two different entities: only a mesh that is not
    // conforming has any, so they are summed one by one
    unsigned longs = __ballot_sync(0xffffffffu, is_long && pr.x != 0);
    while (longs) {
      const int src = __ffs(longs) - 1;
      longs &= longs - 1;
      const uint32_t x = __shfl_sync(0xffffffffu, pr.x, src), z = __shfl_sync(0xffffffffu, pk, src);
      if (lane < 4) {
        const int off = (int)(x & 0xffffu), end = min(off + (int)(x >> 16), kPairWords * (int)d.nI);
        double sr = 0.0, si = 0.0;
        for (int i = off; i < end; ++i) {
          const C64 u = load_block_value<R>(v, __ldg(words + i), lane, n_blocks, pol);
          sr += u.re;
          si += u.im;
        }
        const int p = (int)(z & 0xffffu) + ((lane & 2) ? (int)((z >> 16) & 0x7fffu) : 0);
        A0[((lane & 1) ? to_A1 : 0) + p] = make_double2(ar * sr - ai * si, ar * si + ai * sr);
      }
    }
    if (h >= H || is_long) pk = 0xffffu;  // nothing to store
    if (is_long) pr = none;
    R u[2][2][4];
    uint32_t at[2];
#pragma unroll
    for (int j = 0; j < 2; ++j) {
      const int src = 16 * j + (lane >> 1);
      load_half_block<R, WIDE>(v_y, __shfl_sync(0xffffffffu, pr.x, src) & 0x7fffffffu, n_blocks, pol, u[j][0]);
      load_half_block<R, WIDE>(v_y, __shfl_sync(0xffffffffu, pr.y, src) & 0x7fffffffu, n_blocks, pol, u[j][1]);
      at[j] = __shfl_sync(0xffffffffu, pk, src);
    }
#pragma unroll
    for (int j = 0; j < 2; ++j) {
      const int p = at[j] & 0xffffu, dp = (at[j] >> 16) & 0x7fffu;
      const bool tr = at[j] >> 31;
      // values 2y, 2y + 1 belong to row y and columns 0, 1, or, transposed, to column y and rows 0, 1
      double2 *o = A0 + p + (y ? (tr ? to_A1 : dp) : 0);
      const int step = tr ? dp : to_A1;
      if (p != 0xffffu)
#pragma unroll
        for (int k = 0; k < 2; ++k) {
          double sr = 0.0, si = 0.0;
          sr += (double)u[j][0][2 * k];
          si += (double)u[j][0][2 * k + 1];
          sr += (double)u[j][1][2 * k];
          si += (double)u[j][1][2 * k + 1];
          o[k * step] = make_double2(ar * sr - ai * si, ar * si + ai * sr);
        }
    }
  }
}

template <typename R, bool WIDE>
__global__ void __launch_bounds__(BG_WARPS * 32, BG_CTAS)
    k_gather_block(const ChunkDesc *desc, const uint32_t *brec, uint32_t n_blocks, const void *v, double ar, double ai,
                   double2 *A) {
  gather_block_chunk<R, WIDE>(desc + blockIdx.x, brec, n_blocks, v, ar, ai, A);
}

// whether the values can be read half a block at a time
static bool half_block_aligned(const void *v, bool f32) {
  return reinterpret_cast<uintptr_t>(v) % (f32 ? 16 : 32) == 0;
}

// Several jobs' packed gathers (8-byte records, alpha = 1) in one launch: job
// j owns the CTAs [cta_start[j], cta_start[j + 1]) and its chunks in CTA
// order, as if launched alone.
template <typename R>
__global__ void __launch_bounds__(PackedShape<R, false>::warps * 32, PackedShape<R, false>::min_blocks)
    k_gather_packed_batch(const GatherJob *jobs, const int64_t *cta_start, int n_jobs) {
  const int64_t b = blockIdx.x;
  int lo = 0, hi = n_jobs - 1;
  while (lo < hi) {
    const int mid = (lo + hi + 1) >> 1;
    if (cta_start[mid] <= b) lo = mid;
    else hi = mid - 1;
  }
  if (n_jobs <= 0 || b >= cta_start[n_jobs]) return;
  const GatherJob &j = jobs[lo];
  ChunkMeta m;
  if (!chunk_meta(j.ent_ptr, j.order, j.indptr, j.E, j.F,
                  (b - cta_start[lo]) * PackedShape<R, false>::warps + (threadIdx.x >> 5), m))
    return;
  gather_packed_chunk<R, false>(m, j.pidx, j.posoff, j.n_values, j.values, 1.0, 0.0, j.A, nullptr);
}

// Several jobs' block gathers (alpha = 1) in one launch, as k_gather_packed_batch.
template <typename R, bool WIDE>
__global__ void __launch_bounds__(BG_WARPS * 32, BG_CTAS)
    k_gather_block_batch(const GatherJob *jobs, const int64_t *cta_start, int n_jobs) {
  const int64_t b = blockIdx.x;
  int lo = 0, hi = n_jobs - 1;
  while (lo < hi) {
    const int mid = (lo + hi + 1) >> 1;
    if (cta_start[mid] <= b) lo = mid;
    else hi = mid - 1;
  }
  if (n_jobs <= 0 || b >= cta_start[n_jobs]) return;
  const GatherJob &j = jobs[lo];
  gather_block_chunk<R, WIDE>(j.desc + (b - cta_start[lo]), static_cast<const uint32_t *>(j.pidx),
                              (uint32_t)j.n_values, j.values, 1.0, 0.0, j.A);
}

// ---------------------------------------------------------------------------
// frequency sweep: A_f = a_f K + b_f M (+ c_f P)
// ---------------------------------------------------------------------------
constexpr int SWEEP_MAX = 32;
// CTAs per SM, oversubscribed: at 28.8M nonzeros and 12 frequencies 64 take 1,003
// us, 8 1,033; one 16-byte access per element and 8 CTAs 1,181. Bound: HBM (6.5 TB/s).
constexpr int SWEEP_CTAS = 64;
struct SweepCoef {
  double c[SWEEP_MAX][6];
};

// Elements of a thread per access: two (32-byte loads and stores) where every
// array is aligned to that and nnz is even, else one.
template <int V>
struct Elems {
  double2 v[V];
};

template <int V>
__device__ __forceinline__ Elems<V> ld_elems(const double2 *p) {
  Elems<V> e;
  if constexpr (V == 2)
    asm volatile("ld.global.nc.v4.f64 {%0, %1, %2, %3}, [%4];"
                 : "=d"(e.v[0].x), "=d"(e.v[0].y), "=d"(e.v[1].x), "=d"(e.v[1].y)
                 : "l"(p));
  else
    e.v[0] = __ldg(p);
  return e;
}

template <int V>
__device__ __forceinline__ void st_elems(double2 *p, const Elems<V> &e) {
  if constexpr (V == 2)
    asm volatile("st.global.v4.f64 [%0], {%1, %2, %3, %4};" ::"l"(p), "d"(e.v[0].x), "d"(e.v[0].y), "d"(e.v[1].x),
                 "d"(e.v[1].y)
                 : "memory");
  else
    *p = e.v[0];
}

// SWEEP_U accesses of K, M (and P) per thread per pass, all in flight before the
// first output; the arithmetic per value is the same for all V.
constexpr int SWEEP_U = 2;
template <bool HASP, int V>
__global__ void __launch_bounds__(256) k_form_sweep(const double2 *__restrict__ K, const double2 *__restrict__ M,
                                                    const double2 *__restrict__ P, int64_t nnz, SweepCoef cf, int nf,
                                                    double2 *__restrict__ out, int64_t stride) {
  constexpr int U = SWEEP_U;
  const int64_t T = (int64_t)gridDim.x * blockDim.x, n = nnz / V;
  for (int64_t i0 = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i0 < n; i0 += U * T) {
    Elems<V> k[U], m[U], p[U];
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const int64_t i = min(i0 + u * T, n - 1) * V;
      k[u] = ld_elems<V>(K + i);
      m[u] = ld_elems<V>(M + i);
      if (HASP) p[u] = ld_elems<V>(P + i);
    }
    for (int f = 0; f < nf; ++f) {
      const double *c = cf.c[f];
#pragma unroll
      for (int u = 0; u < U; ++u) {
        const int64_t i = i0 + u * T;
        if (i >= n) break;
        Elems<V> o;
#pragma unroll
        for (int q = 0; q < V; ++q) {
          o.v[q].x = c[0] * k[u].v[q].x - c[1] * k[u].v[q].y + c[2] * m[u].v[q].x - c[3] * m[u].v[q].y;
          o.v[q].y = c[0] * k[u].v[q].y + c[1] * k[u].v[q].x + c[2] * m[u].v[q].y + c[3] * m[u].v[q].x;
          if (HASP) {
            o.v[q].x += c[4] * p[u].v[q].x - c[5] * p[u].v[q].y;
            o.v[q].y += c[4] * p[u].v[q].y + c[5] * p[u].v[q].x;
          }
        }
        st_elems<V>(out + (int64_t)f * stride + i * V, o);
      }
    }
  }
}

// serving batch: grid-stride over tiles of all items
constexpr int FORM_TILE = 32768;

__global__ void __launch_bounds__(256) k_form_batch(const emg_form_item *items, const int64_t *tile_start,
                                                    const int32_t *n_items_p, int max_items) {
  const int n = min(*n_items_p, max_items);
  if (n <= 0) return;
  const int64_t total = tile_start[n];
  for (int64_t t = blockIdx.x; t < total; t += gridDim.x) {
    int lo = 0, hi = n - 1;  // item with tile_start[i] <= t < tile_start[i+1]
    while (lo < hi) {
      const int mid = (lo + hi + 1) >> 1;
      if (tile_start[mid] <= t) lo = mid; else hi = mid - 1;
    }
    const emg_form_item &it = items[lo];
    const int64_t b = (t - tile_start[lo]) * FORM_TILE;
    const int64_t e = min(b + FORM_TILE, it.nnz);
    const int g = max(1, min(it.group, n - lo));  // the group's items share K, M, P: read them once
    const double2 *K = static_cast<const double2 *>(it.K);
    const double2 *M = static_cast<const double2 *>(it.M);
    const double2 *P = static_cast<const double2 *>(it.P);
    for (int64_t i = b + threadIdx.x; i < e; i += blockDim.x) {
      const double2 k = K[i], m = M[i];
      const double2 p = P ? P[i] : make_double2(0.0, 0.0);
      for (int f = 0; f < g; ++f) {
        const double *c = items[lo + f].coef;
        double2 o;
        o.x = c[0] * k.x - c[1] * k.y + c[2] * m.x - c[3] * m.y;
        o.y = c[0] * k.y + c[1] * k.x + c[2] * m.y + c[3] * m.x;
        if (P) {
          o.x += c[4] * p.x - c[5] * p.y;
          o.y += c[4] * p.y + c[5] * p.x;
        }
        static_cast<double2 *>(items[lo + f].out)[i] = o;
      }
    }
  }
}

}  // namespace

int launch_gather(const emg_plan *p, const void *d_plan, const int32_t *d_indptr, const void *d_v1, const void *d_v2,
                  int precision, int layout, double ar, double ai, double br, double bi, void *d_A, int64_t *d_status,
                  cudaStream_t s) {
  (void)d_status;
  if (p->n_ent == 0) return EMG_OK;
  if (precision < EMG_FP64 || precision > EMG_EXACT) return fail(EMG_EINVAL, "bad precision %d", precision);
  if (layout != EMG_LAYOUT_COO && layout != EMG_LAYOUT_PACKED && layout != EMG_LAYOUT_BLOCK)
    return fail(EMG_EINVAL, "bad layout %d", layout);
  const char *plan = static_cast<const char *>(d_plan);
  const int32_t *ent_ptr = reinterpret_cast<const int32_t *>(plan + p->off_ent_ptr);
  const Item *items = reinterpret_cast<const Item *>(plan + p->off_item);
  const int32_t *order = reinterpret_cast<const int32_t *>(plan + p->off_order);
  const uint16_t *posoff = reinterpret_cast<const uint16_t *>(plan + p->off_posoff);
  double2 *A = static_cast<double2 *>(d_A);
  const bool two = d_v2 != nullptr;
  const bool f32 = values_fp32(precision);
  if (layout == EMG_LAYOUT_BLOCK) {
    if (two) return fail(EMG_EINVAL, "the block layout takes one value array");
    const uint32_t *brec = reinterpret_cast<const uint32_t *>(plan + p->off_pidx);
    const ChunkDesc *desc = reinterpret_cast<const ChunkDesc *>(plan + p->off_hoff);
    const unsigned nch = (unsigned)n_chunks(p->n_edges, p->n_tris);
    const uint32_t nb = (uint32_t)(p->n_assy * 55);  // below 2^31: block_record_fits
#define EMG_BG(R, W) k_gather_block<R, W><<<nch, BG_WARPS * 32, 0, s>>>(desc, brec, nb, d_v1, ar, ai, A)
    const bool wide = half_block_aligned(d_v1, f32);
    if (f32) {
      if (wide) EMG_BG(float, true); else EMG_BG(float, false);
    } else {
      if (wide) EMG_BG(double, true); else EMG_BG(double, false);
    }
#undef EMG_BG
    return launch_check("k_gather_block");
  }
  if (layout == EMG_LAYOUT_PACKED) {
    if (two) return fail(EMG_EINVAL, "the packed layout takes one value array");
    const void *pidx = plan + p->off_pidx;
    const int64_t nv = p->n_assy * 210;
    const bool compact = p->record_bytes == 4;
#define EMG_PK(R, C)                                                                                    \
  k_gather_packed<R, C><<<grid_for(n_chunks(p->n_edges, p->n_tris), PackedShape<R, C>::warps),           \
                          PackedShape<R, C>::warps * 32, 0, s>>>(ent_ptr, order, pidx, posoff, p->n_edges,  \
                                                                 p->n_tris, nv, d_indptr, d_v1, ar, ai, A)
    if (f32) {
      if (compact) EMG_PK(float, true); else EMG_PK(float, false);
    } else {
      if (compact) EMG_PK(double, true); else EMG_PK(double, false);
    }
#undef EMG_PK
    return launch_check("k_gather_packed");
  }
  // two columns per warp, at most four warps and 48 KB per CTA
  const uint32_t *ent_cnt = reinterpret_cast<const uint32_t *>(plan + p->off_ent_cnt);
  const int max_col = p->max_col > 0 && p->max_col < 1536 ? (int)p->max_col : 1536;
  const int warps = std::max(1, std::min(4, (48 << 10) / (32 * max_col)));
  const int g = grid_for(n_chunks(p->n_edges, p->n_tris) * CHUNK, warps);
#define EMG_COO(R, TWO)                                                                                             \
  k_gather_coo<R, TWO><<<g, warps * 32, 32 * max_col * warps, s>>>(ent_ptr, order, items, ent_cnt, p->n_edges,       \
                                                                   p->n_tris, d_indptr, d_v1, d_v2, ar, ai, br, bi, \
                                                                   max_col, A)
  if (f32) {
    if (two) EMG_COO(float, true); else EMG_COO(float, false);
  } else {
    if (two) EMG_COO(double, true); else EMG_COO(double, false);
  }
#undef EMG_COO
  return launch_check("k_gather_coo");
}

int gather_job_fill(const emg_plan *p, const void *d_plan, const int32_t *d_indptr, const void *d_values, void *d_A,
                    int precision, GatherJob *out) {
  const bool block = p->value_layout == EMG_LAYOUT_BLOCK;
  if (!block && p->record_bytes != 8)
    return fail(EMG_EINVAL, "batched gathers take block-layout plans or packed ones with 8-byte records");
  const char *plan = static_cast<const char *>(d_plan);
  out->ent_ptr = reinterpret_cast<const int32_t *>(plan + p->off_ent_ptr);
  out->order = reinterpret_cast<const int32_t *>(plan + p->off_order);
  out->pidx = plan + p->off_pidx;
  out->posoff = reinterpret_cast<const uint16_t *>(plan + p->off_posoff);
  out->indptr = d_indptr;
  out->desc = reinterpret_cast<const ChunkDesc *>(plan + p->off_hoff);
  out->values = d_values;
  out->A = static_cast<double2 *>(d_A);
  out->E = p->n_edges;
  out->F = p->n_tris;
  out->n_values = p->n_assy * (block ? 55 : 210);
  const int per_cta = block ? 1 : PackedShape<double, false>::warps;  // chunks
  out->n_ctas = (n_chunks(p->n_edges, p->n_tris) + per_cta - 1) / per_cta;
  out->wide = block && half_block_aligned(d_values, values_fp32(precision));
  return EMG_OK;
}

int launch_gather_batch(const GatherJob *d_jobs, const int64_t *d_cta_start, int n_jobs, int64_t total_ctas,
                        bool wide, int precision, int layout, cudaStream_t s) {
  if (n_jobs == 0 || total_ctas == 0) return EMG_OK;
  if (total_ctas > INT32_MAX) return fail(EMG_ERANGE, "too many CTAs (%lld)", (long long)total_ctas);
  if (layout == EMG_LAYOUT_BLOCK) {
#define EMG_BGB(R, W) \
  k_gather_block_batch<R, W><<<(unsigned)total_ctas, BG_WARPS * 32, 0, s>>>(d_jobs, d_cta_start, n_jobs)
    if (values_fp32(precision)) {
      if (wide) EMG_BGB(float, true); else EMG_BGB(float, false);
    } else {
      if (wide) EMG_BGB(double, true); else EMG_BGB(double, false);
    }
#undef EMG_BGB
    return launch_check("k_gather_block_batch");
  }
  static_assert(PackedShape<double, false>::warps == PackedShape<float, false>::warps, "same chunks per CTA");
  if (values_fp32(precision))
    k_gather_packed_batch<float><<<(unsigned)total_ctas, PackedShape<float, false>::warps * 32, 0, s>>>(
        d_jobs, d_cta_start, n_jobs);
  else
    k_gather_packed_batch<double><<<(unsigned)total_ctas, PackedShape<double, false>::warps * 32, 0, s>>>(
        d_jobs, d_cta_start, n_jobs);
  return launch_check("k_gather_packed_batch");
}

int launch_form_batch(const emg_form_item *items, const int64_t *tile_start, const int32_t *n_items, int max_items,
                      cudaStream_t s) {
  // many short-lived CTAs (a few tiles each) rather than a persistent grid,
  // so that kernels of higher-priority streams are scheduled between them
  k_form_batch<<<persistent_ctas(16), 256, 0, s>>>(items, tile_start, n_items, max_items);
  return launch_check("k_form_batch");
}

int launch_form_sweep(const void *d_K, const void *d_M, const void *d_P, int64_t nnz, const double *h_coef, int nf,
                      void *d_out, int64_t out_stride, cudaStream_t s) {
  for (int f0 = 0; f0 < nf; f0 += SWEEP_MAX) {
    int n = nf - f0 < SWEEP_MAX ? nf - f0 : SWEEP_MAX;
    SweepCoef c;
    memcpy(c.c, h_coef + (size_t)f0 * 6, (size_t)n * 6 * sizeof(double));
    double2 *o = static_cast<double2 *>(d_out) + (int64_t)f0 * out_stride;
    const int g = std::min(persistent_ctas(SWEEP_CTAS), grid_for(nnz, 256));
    auto aligned = [](const void *p) { return reinterpret_cast<uintptr_t>(p) % 32 == 0; };
    const bool two = nnz % 2 == 0 && out_stride % 2 == 0 && aligned(d_K) && aligned(d_M) && aligned(d_P) && aligned(o);
#define EMG_FS(HASP, V) \
  k_form_sweep<HASP, V><<<g, 256, 0, s>>>((const double2 *)d_K, (const double2 *)d_M, (const double2 *)d_P, nnz, c, n, o, out_stride)
    if (d_P) {
      if (two) EMG_FS(true, 2); else EMG_FS(true, 1);
    } else {
      if (two) EMG_FS(false, 2); else EMG_FS(false, 1);
    }
#undef EMG_FS
    int rc = launch_check("k_form_sweep");
    if (rc) return rc;
  }
  return EMG_OK;
}

}  // namespace emg
