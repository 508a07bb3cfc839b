// element.cuh -- per-tet Nedelec-2 element kernel.
//
// Replaces _matrix_builder + ned2_tet_stiff_mass + tet_coefficients +
// local_mapping + matinv (physics/microwave/assembly/curlcurl.py:127-214,
// 285-456; mth/optimized.py:262-357). Thread per assembled tet, three forms:
//
//  FORM_REF64 (EMG_FP64, plain) reproduces the reference's arithmetic: its
//    barycentric coefficients from absolute-coordinate cofactors, its KEAST4
//    points and its values L~ of the four barycentric functions at them, all
//    in FP64 without fused multiply-adds in the reference's operation order.
//    The 11-point sums are then evaluated exactly as the per-tet quadrature
//    moments mu[alpha] = sum_q w_q L~_q^alpha (degree <= 4) contracted with
//    the tensors G = V (eps grad L~_m).grad L~_n and H = V (mu^-1 X_P).X_Q
//    through generated tables (nedelec_moment_tables.cuh).
//  FORM_REF32 (EMG_MIXED): FP64 geometry from edge vectors (Jacobian,
//    determinant, gradients, orientation sign), the tensors G and H formed in
//    FP64 and rounded to FP32, then contracted in FP32 with FP32 accumulation
//    against the closed-form tables (nedelec_tables.cuh). KEAST4 integrates
//    every product of two basis values or curls of this element exactly, so
//    its 11-point sums are fixed rational combinations of the tensors; the
//    tables hold them, evaluated once when the tables are generated. Element
//    values complex64.
//  FORM_EXACT (EMG_EXACT): exact closed-form integrals (nedelec_tables.cuh)
//    on accurate edge-vector geometry, free of the reference's cancellation.
//
// Every form writes one of three layouts (element_cta): the reference's COO
// block value[ia*400 + 20*a + b], the packed canonical upper triangle
// [ia][210], or the entity-pair blocks [ia][220] of the assembly path. Of the
// first two, one row at a time is staged in shared memory and the warp writes its
// tets' rows as contiguous runs; the blocks are stored straight from registers
// where a lane holds whole values.
#pragma once
#include "common.cuh"

namespace emg {
namespace {

enum { FORM_REF64 = 0, FORM_REF32 = 1, FORM_EXACT = 2 };

// Complex tensors in FP64 (diagonal and full materials, both FP64 forms): two
// lanes share a tet, the even one computes the real parts of its values, the
// odd one the imaginary parts. With alpha and beta multiplied into the tensors
// first, each part is a real contraction, half the tensor registers of a complex
// one, and the lanes share the quadrature points (REF64). A lane per tet spilled
// 1.1 KB (diagonal) and 6.9 KB (full). Measured: diagonal at 1,008,000 tets 2,447
// -> 1,110 us (EXACT 726 -> 660), full at 414,720 1,856 -> 555 (1,276 -> 361).
// Bound: FP64 latency at eight warps per SM (254 registers).
// Tets with symmetric tensors (all of a reciprocal material) need only those halves; a
// warp that has any others goes through these in a pass of their own, with the
// antisymmetric halves beside the symmetric ones (KIND_PAIR_BOTH). 103,680 tets, none
// symmetric, packed / block values: FP64 442 / 525 us, exact 270 / 279, against 506 / 485
// and 336 / 326 for a lane per tet and 895 / 770 and 645 / 479 for a second pass over the
// whole warp that added the antisymmetric part to the values in memory. Its 14,000
// instructions do not fit the instruction cache (no-instruction stalls 6.5 of 11.4 cycles
// per instruction; a symmetric tet's pass 0.6 of 5.6).
enum { KIND_PAIR = 3, KIND_PAIR_FULL = 4, KIND_PAIR_BOTH = 5 };
__host__ __device__ constexpr int tensor_kind(int form, int kind) {
  return form == FORM_REF32 || kind == EMG_MAT_ISO ? kind : (kind == EMG_MAT_DIAG ? KIND_PAIR : KIND_PAIR_FULL);
}
__host__ __device__ constexpr int lanes_per_tet(int tensor_kind) { return tensor_kind >= KIND_PAIR ? 2 : 1; }
template <int FORM>
struct FormReal {
  using T = double;
};
template <>
struct FormReal<FORM_REF32> {
  using T = float;
};

struct C64 {
  double re, im;
};
struct C32 {
  float re, im;
};

__device__ __forceinline__ C64 cmul(C64 a, C64 b) { return {a.re * b.re - a.im * b.im, a.re * b.im + a.im * b.re}; }
__device__ __forceinline__ C64 cadd(C64 a, C64 b) { return {a.re + b.re, a.im + b.im}; }
__device__ __forceinline__ C64 csub(C64 a, C64 b) { return {a.re - b.re, a.im - b.im}; }
__device__ __forceinline__ C64 crecip(C64 a) {
  double d = a.re * a.re + a.im * a.im;
  return {a.re / d, -a.im / d};
}
__device__ __forceinline__ C64 cdiv(C64 a, C64 b) {
  double d = b.re * b.re + b.im * b.im;
  return {(a.re * b.re + a.im * b.im) / d, (a.im * b.re - a.re * b.im) / d};
}
__device__ __forceinline__ bool cis0(C64 a) { return a.re == 0.0 && a.im == 0.0; }

__device__ __forceinline__ C64 ld_c64(const void *p, int64_t idx) {
  const double2 v = reinterpret_cast<const double2 *>(p)[idx];
  return {v.x, v.y};
}

// matinv of the reference (optimized.py:315-357): 3x3 complex inverse with the
// diagonal fast path.
__device__ void matinv3(const C64 M[9], C64 out[9]) {
  if (cis0(M[1]) && cis0(M[2]) && cis0(M[3]) && cis0(M[5]) && cis0(M[6]) && cis0(M[7])) {
#pragma unroll
    for (int i = 0; i < 9; ++i) out[i] = {0.0, 0.0};
    out[0] = crecip(M[0]);
    out[4] = crecip(M[4]);
    out[8] = crecip(M[8]);
    return;
  }
  C64 det = csub(csub(cmul(cmul(M[0], M[4]), M[8]), cmul(cmul(M[0], M[5]), M[7])), cmul(cmul(M[1], M[3]), M[8]));
  det = cadd(det, cmul(cmul(M[1], M[5]), M[6]));
  det = cadd(det, cmul(cmul(M[2], M[3]), M[7]));
  det = csub(det, cmul(cmul(M[2], M[4]), M[6]));
  C64 a[9];
  a[0] = csub(cmul(M[4], M[8]), cmul(M[5], M[7]));
  a[1] = csub(cmul(M[2], M[7]), cmul(M[1], M[8]));
  a[2] = csub(cmul(M[1], M[5]), cmul(M[2], M[4]));
  a[3] = csub(cmul(M[5], M[6]), cmul(M[3], M[8]));
  a[4] = csub(cmul(M[0], M[8]), cmul(M[2], M[6]));
  a[5] = csub(cmul(M[2], M[3]), cmul(M[0], M[5]));
  a[6] = csub(cmul(M[3], M[7]), cmul(M[4], M[6]));
  a[7] = csub(cmul(M[1], M[6]), cmul(M[0], M[7]));
  a[8] = csub(cmul(M[0], M[4]), cmul(M[1], M[3]));
#pragma unroll
  for (int i = 0; i < 9; ++i) out[i] = cdiv(a[i], det);
}


// KEAST4 11-point rule exactly as the reference prints it (curlcurl.py:277-283):
// row 0 weights, rows 1-4 barycentric coordinates of the points.
__constant__ double kDP[5][11] = {
    {-0.07893333333333329982, 0.04573333333333329948, 0.04573333333333329948, 0.04573333333333329948,
     0.04573333333333329948, 0.14933333333333329018, 0.14933333333333329018, 0.14933333333333329018,
     0.14933333333333329018, 0.14933333333333329018, 0.14933333333333329018},
    {0.25000000000000000000, 0.78571428571428569843, 0.07142857142857139685, 0.07142857142857139685,
     0.07142857142857139685, 0.10059642383320080428, 0.39940357616679922348, 0.39940357616679922348,
     0.39940357616679922348, 0.10059642383320080428, 0.10059642383320080428},
    {0.25000000000000000000, 0.07142857142857139685, 0.07142857142857139685, 0.07142857142857139685,
     0.78571428571428569843, 0.39940357616679922348, 0.10059642383320080428, 0.39940357616679922348,
     0.10059642383320080428, 0.39940357616679922348, 0.10059642383320080428},
    {0.25000000000000000000, 0.07142857142857139685, 0.07142857142857139685, 0.78571428571428569843,
     0.07142857142857139685, 0.39940357616679922348, 0.39940357616679922348, 0.10059642383320080428,
     0.10059642383320080428, 0.10059642383320080428, 0.39940357616679922348},
    {0.25000000000000000000, 0.07142857142857150787, 0.78571428571428580945, 0.07142857142857150787,
     0.07142857142857150787, 0.10059642383320077652, 0.10059642383320077652, 0.10059642383320074877,
     0.39940357616679922348, 0.39940357616679922348, 0.39940357616679922348},
};

// Per-tet geometry in the canonical (vertex-rank) frame.
struct Geo {
  double g[4][3];  // gradients by vertex rank: reference forms grad L~, exact form grad lambda
  double V;        // |det| / 6 (reference determinant in the reference forms)
  double sig;      // sign(det) in the tet's own vertex order (exact form only)
  uint64_t inv;    // nibble c (0..9 canonical entity) -> reference entity slot (0..9)
};


// Barycentric coefficients exactly as the reference forms them
// (tet_coefficients, curlcurl.py:127-214): 24-term determinant and signed
// cofactors in ABSOLUTE coordinates, evaluated left to right without fused
// multiply-adds, V = |det| / 6, coefficient = cofactor / (6 V). These
// expressions cancel heavily (terms ~|x|^3 against det ~h^3), so the
// reference's element matrices carry that rounding; reproducing the same
// operation order keeps the GPU values within ulps of the reference's
// instead of differing by the cancellation error.
#define EMG_M2(a, b) __dmul_rn((a), (b))
#define EMG_M3(a, b, c) __dmul_rn(__dmul_rn((a), (b)), (c))
#define EMG_A(a, b) __dadd_rn((a), (b))
#define EMG_S(a, b) __dsub_rn((a), (b))

__device__ __forceinline__ void ref_coefficients(const double X[3][4], double ca[4], double cb[4], double cc[4],
                                                 double cd[4], double &det) {
  const double x1 = X[0][0], x2 = X[0][1], x3 = X[0][2], x4 = X[0][3];
  const double y1 = X[1][0], y2 = X[1][1], y3 = X[1][2], y4 = X[1][3];
  const double z1 = X[2][0], z2 = X[2][1], z3 = X[2][2], z4 = X[2][3];
  double d = EMG_M3(-x1, y2, z3);
  d = EMG_A(d, EMG_M3(x1, y2, z4));
  d = EMG_A(d, EMG_M3(x1, y3, z2));
  d = EMG_S(d, EMG_M3(x1, y3, z4));
  d = EMG_S(d, EMG_M3(x1, y4, z2));
  d = EMG_A(d, EMG_M3(x1, y4, z3));
  d = EMG_A(d, EMG_M3(x2, y1, z3));
  d = EMG_S(d, EMG_M3(x2, y1, z4));
  d = EMG_S(d, EMG_M3(x2, y3, z1));
  d = EMG_A(d, EMG_M3(x2, y3, z4));
  d = EMG_A(d, EMG_M3(x2, y4, z1));
  d = EMG_S(d, EMG_M3(x2, y4, z3));
  d = EMG_S(d, EMG_M3(x3, y1, z2));
  d = EMG_A(d, EMG_M3(x3, y1, z4));
  d = EMG_A(d, EMG_M3(x3, y2, z1));
  d = EMG_S(d, EMG_M3(x3, y2, z4));
  d = EMG_S(d, EMG_M3(x3, y4, z1));
  d = EMG_A(d, EMG_M3(x3, y4, z2));
  d = EMG_A(d, EMG_M3(x4, y1, z2));
  d = EMG_S(d, EMG_M3(x4, y1, z3));
  d = EMG_S(d, EMG_M3(x4, y2, z1));
  d = EMG_A(d, EMG_M3(x4, y2, z3));
  d = EMG_A(d, EMG_M3(x4, y3, z1));
  d = EMG_S(d, EMG_M3(x4, y3, z2));
  det = d;
  // six-term cofactor sums (the reference's bbs, ccs, dds)
#define EMG_C6(s1, a1, b1, s2, a2, b2, s3, a3, b3, s4, a4, b4, s5, a5, b5, s6, a6, b6)                   \
  EMG_##s6(EMG_##s5(EMG_##s4(EMG_##s3(EMG_##s2(EMG_M2(s1 a1, b1), EMG_M2(a2, b2)), EMG_M2(a3, b3)),       \
                             EMG_M2(a4, b4)),                                                             \
                    EMG_M2(a5, b5)),                                                                      \
           EMG_M2(a6, b6))
  cb[0] = EMG_C6(-, y2, z3, A, y2, z4, A, y3, z2, S, y3, z4, S, y4, z2, A, y4, z3);
  cb[1] = EMG_C6(+, y1, z3, S, y1, z4, S, y3, z1, A, y3, z4, A, y4, z1, S, y4, z3);
  cb[2] = EMG_C6(-, y1, z2, A, y1, z4, A, y2, z1, S, y2, z4, S, y4, z1, A, y4, z2);
  cb[3] = EMG_C6(+, y1, z2, S, y1, z3, S, y2, z1, A, y2, z3, A, y3, z1, S, y3, z2);
  cc[0] = EMG_C6(+, x2, z3, S, x2, z4, S, x3, z2, A, x3, z4, A, x4, z2, S, x4, z3);
  cc[1] = EMG_C6(-, x1, z3, A, x1, z4, A, x3, z1, S, x3, z4, S, x4, z1, A, x4, z3);
  cc[2] = EMG_C6(+, x1, z2, S, x1, z4, S, x2, z1, A, x2, z4, A, x4, z1, S, x4, z2);
  cc[3] = EMG_C6(-, x1, z2, A, x1, z3, A, x2, z1, S, x2, z3, S, x3, z1, A, x3, z2);
  cd[0] = EMG_C6(-, x2, y3, A, x2, y4, A, x3, y2, S, x3, y4, S, x4, y2, A, x4, y3);
  cd[1] = EMG_C6(+, x1, y3, S, x1, y4, S, x3, y1, A, x3, y4, A, x4, y1, S, x4, y3);
  cd[2] = EMG_C6(-, x1, y2, A, x1, y4, A, x2, y1, S, x2, y4, S, x4, y1, A, x4, y2);
  cd[3] = EMG_C6(+, x1, y2, S, x1, y3, S, x2, y1, A, x2, y3, A, x3, y1, S, x3, y2);
#undef EMG_C6
  // six-term triple-product sums (the reference's aas)
#define EMG_T6(s1, a1, b1, c1, s2, a2, b2, c2, s3, a3, b3, c3, s4, a4, b4, c4, s5, a5, b5, c5, s6, a6, b6, c6)   \
  EMG_##s6(EMG_##s5(EMG_##s4(EMG_##s3(EMG_##s2(EMG_M3(s1 a1, b1, c1), EMG_M3(a2, b2, c2)), EMG_M3(a3, b3, c3)),     \
                             EMG_M3(a4, b4, c4)),                                                                \
                    EMG_M3(a5, b5, c5)),                                                                         \
           EMG_M3(a6, b6, c6))
  ca[0] = EMG_T6(+, x2, y3, z4, S, x2, y4, z3, S, x3, y2, z4, A, x3, y4, z2, A, x4, y2, z3, S, x4, y3, z2);
  ca[1] = EMG_T6(-, x1, y3, z4, A, x1, y4, z3, A, x3, y1, z4, S, x3, y4, z1, S, x4, y1, z3, A, x4, y3, z1);
  ca[2] = EMG_T6(+, x1, y2, z4, S, x1, y4, z2, S, x2, y1, z4, A, x2, y4, z1, A, x4, y1, z2, S, x4, y2, z1);
  ca[3] = EMG_T6(-, x1, y2, z3, A, x1, y3, z2, A, x2, y1, z3, S, x2, y3, z1, S, x3, y1, z2, A, x3, y2, z1);
#undef EMG_T6
}


// vertex ranks by global id, and the canonical -> reference entity map
__device__ __forceinline__ bool ranks_and_map(const int64_t v[4], int rank[4], uint64_t &inv) {
#pragma unroll
  for (int q = 0; q < 4; ++q) {
    int r = 0;
#pragma unroll
    for (int p = 0; p < 4; ++p) r += (v[p] < v[q]) ? 1 : 0;
    rank[q] = r;
  }
  const bool distinct = (v[0] != v[1]) && (v[0] != v[2]) && (v[0] != v[3]) && (v[1] != v[2]) && (v[1] != v[3]) &&
                        (v[2] != v[3]);
  // reference edge slots (local vertex pairs) and the vertex missing from each face slot
  const int eu[6] = {0, 0, 0, 1, 3, 2}, ev[6] = {1, 2, 3, 2, 1, 3};
  const int fmiss[4] = {3, 1, 2, 0};
  uint64_t m = 0;
  if (distinct) {
#pragma unroll
    for (int s = 0; s < 6; ++s) m |= (uint64_t)s << (4 * canon_edge(rank[eu[s]], rank[ev[s]]));
#pragma unroll
    for (int f = 0; f < 4; ++f) m |= (uint64_t)(6 + f) << (4 * (6 + 3 - rank[fmiss[f]]));
  }
  inv = m;
  return distinct;
}

template <typename T>
__device__ __forceinline__ void scatter_rank(const T in[4], const int rank[4], T out[4]) {
#pragma unroll
  for (int q = 0; q < 4; ++q)
#pragma unroll
    for (int r = 0; r < 4; ++r)
      if (rank[q] == r) out[r] = in[q];
}

}  // namespace

// the generated tables call emg_mac unqualified: include them inside emg
template <typename R>
struct CR {
  R re, im;
};
// Every multiply-add of the generated tables goes through rounding
// intrinsics, which the compiler neither re-associates nor re-contracts: the
// (x, y) and (y, x) entries, computed in different rows, are then bitwise
// equal, so the element blocks and A stay exactly symmetric.
__device__ __forceinline__ void emg_mac(double &acc, double a, double b) { acc = __fma_rn(a, b, acc); }
__device__ __forceinline__ void emg_mac(float &acc, double c, float v) { acc = __fmaf_rn((float)c, v, acc); }
__device__ __forceinline__ void emg_mac(float &acc, float a, float b) { acc = __fmaf_rn(a, b, acc); }
__device__ __forceinline__ void emg_mac(CR<double> &acc, double c, const CR<double> &v) {
  acc.re = __fma_rn(c, v.re, acc.re);
  acc.im = __fma_rn(c, v.im, acc.im);
}
__device__ __forceinline__ void emg_mac(CR<float> &acc, double c, const CR<float> &v) {
  acc.re = __fmaf_rn((float)c, v.re, acc.re);
  acc.im = __fmaf_rn((float)c, v.im, acc.im);
}
__device__ __forceinline__ void emg_mac(CR<double> &acc, const CR<double> &t, double w) {
  acc.re = __fma_rn(t.re, w, acc.re);
  acc.im = __fma_rn(t.im, w, acc.im);
}
__device__ __forceinline__ void emg_mac(CR<float> &acc, const CR<float> &t, float w) {
  acc.re = __fmaf_rn(t.re, w, acc.re);
  acc.im = __fmaf_rn(t.im, w, acc.im);
}
// inner moment sums of the generated tables: c0*mu0, then fma(c, mu, t)
__device__ __forceinline__ double emg_mul(double c, double m) { return __dmul_rn(c, m); }
__device__ __forceinline__ float emg_mul(double c, float m) { return __fmul_rn((float)c, m); }
__device__ __forceinline__ double emg_fma(double t, double c, double m) { return __fma_rn(c, m, t); }
__device__ __forceinline__ float emg_fma(float t, double c, float m) { return __fmaf_rn((float)c, m, t); }
#include "nedelec_moment_tables.cuh"
#include "nedelec_tables.cuh"

namespace {

constexpr int NMOM = emg_mtables::kNumMoments;

// Reference forms: coefficients, quadrature points and L~ exactly as the
// reference computes them, then the quadrature moments: of all 11 points, or
// (PAIR) of this lane's half of them, the even lane's the first six. Returns
// false for a degenerate tet.
template <bool PAIR, typename R>
__device__ __forceinline__ bool ref_geometry(const double X[3][4], const int64_t v[4], Geo &G, R mu[NMOM]) {
  int rank[4];
  uint64_t inv;
  const bool distinct = ranks_and_map(v, rank, inv);
  double ca[4], cb[4], cc[4], cd[4], det;
  ref_coefficients(X, ca, cb, cc, cd, det);
  if (!distinct || !(det != 0.0) || !isfinite(det)) return false;
  const double V = fabs(det) / 6.0;
  const double six_v = __dmul_rn(6.0, V);
  double a[4], b[4], c[4], d[4];
#pragma unroll
  for (int q = 0; q < 4; ++q) {
    a[q] = ca[q] / six_v;
    b[q] = cb[q] / six_v;
    c[q] = cc[q] / six_v;
    d[q] = cd[q] / six_v;
  }
  double Ar[4], br[4], cr[4], dr[4];
  scatter_rank(a, rank, Ar);
  scatter_rank(b, rank, br);
  scatter_rank(c, rank, cr);
  scatter_rank(d, rank, dr);
#pragma unroll
  for (int r = 0; r < 4; ++r) {
    G.g[r][0] = br[r];
    G.g[r][1] = cr[r];
    G.g[r][2] = dr[r];
  }
  G.V = V;
  G.sig = 1.0;
  G.inv = inv;
  // rolled on purpose: the kernel is instruction-fetch bound, and the point
  // loop body is the same for all 11 points
#pragma unroll 1
  for (int i = 0; i < (PAIR ? 6 : 11); ++i) {
    const int q = PAIR ? min(((threadIdx.x & 1) ? 6 : 0) + i, 10) : i;
    const double w = PAIR && (threadIdx.x & 1) && i == 5 ? 0.0 : kDP[0][q];  // the odd lane has five points
    const double p1 = kDP[1][q], p2 = kDP[2][q], p3 = kDP[3][q], p4 = kDP[4][q];
    double xq[3];
#pragma unroll
    for (int k = 0; k < 3; ++k)
      xq[k] = EMG_A(EMG_A(EMG_A(EMG_M2(X[k][0], p1), EMG_M2(X[k][1], p2)), EMG_M2(X[k][2], p3)), EMG_M2(X[k][3], p4));
    R Lq[4];
#pragma unroll
    for (int r = 0; r < 4; ++r)
      Lq[r] = (R)EMG_A(EMG_A(EMG_A(Ar[r], EMG_M2(br[r], xq[0])), EMG_M2(cr[r], xq[1])), EMG_M2(dr[r], xq[2]));
    emg_mtables::emg_moments<R>(Lq, (R)w, mu);
  }
  return true;
}

// Exact form: accurate gradients from edge vectors (relative to vertex 0).
__device__ __forceinline__ bool exact_geometry(const double X[3][4], const int64_t v[4], Geo &G) {
  int rank[4];
  uint64_t inv;
  const bool distinct = ranks_and_map(v, rank, inv);
  double e1[3], e2[3], e3[3];
#pragma unroll
  for (int d = 0; d < 3; ++d) {
    e1[d] = X[d][1] - X[d][0];
    e2[d] = X[d][2] - X[d][0];
    e3[d] = X[d][3] - X[d][0];
  }
  double c23[3] = {e2[1] * e3[2] - e2[2] * e3[1], e2[2] * e3[0] - e2[0] * e3[2], e2[0] * e3[1] - e2[1] * e3[0]};
  double c31[3] = {e3[1] * e1[2] - e3[2] * e1[1], e3[2] * e1[0] - e3[0] * e1[2], e3[0] * e1[1] - e3[1] * e1[0]};
  double c12[3] = {e1[1] * e2[2] - e1[2] * e2[1], e1[2] * e2[0] - e1[0] * e2[2], e1[0] * e2[1] - e1[1] * e2[0]};
  double det = e1[0] * c23[0] + e1[1] * c23[1] + e1[2] * c23[2];
  if (!distinct || !(det != 0.0) || !isfinite(det)) return false;
  const double id = 1.0 / det;
  double gx[4], gy[4], gz[4];
  gx[1] = c23[0] * id, gy[1] = c23[1] * id, gz[1] = c23[2] * id;
  gx[2] = c31[0] * id, gy[2] = c31[1] * id, gz[2] = c31[2] * id;
  gx[3] = c12[0] * id, gy[3] = c12[1] * id, gz[3] = c12[2] * id;
  gx[0] = -(gx[1] + gx[2] + gx[3]);
  gy[0] = -(gy[1] + gy[2] + gy[3]);
  gz[0] = -(gz[1] + gz[2] + gz[3]);
  double rx[4], ry[4], rz[4];
  scatter_rank(gx, rank, rx);
  scatter_rank(gy, rank, ry);
  scatter_rank(gz, rank, rz);
#pragma unroll
  for (int r = 0; r < 4; ++r) {
    G.g[r][0] = rx[r];
    G.g[r][1] = ry[r];
    G.g[r][2] = rz[r];
  }
  G.V = fabs(det) / 6.0;
  G.sig = det > 0.0 ? 1.0 : -1.0;
  G.inv = inv;
  return true;
}

// reference DoF index (0..19) of canonical DoF y
__device__ __forceinline__ int ref_dof(uint64_t inv, int y) {
  int c = y < 6 ? y : (y < 12 ? y - 6 : (y < 16 ? y - 6 : y - 10));  // canonical entity 0..9
  int s = (int)((inv >> (4 * c)) & 15ull);                             // reference entity slot 0..9
  return y < 6 ? s : (y < 12 ? 6 + s : (y < 16 ? 12 + (s - 6) : 16 + (s - 6)));
}

// Per-tet tensors, V folded in: G[m][n] = V (eps g_m).g_n, H[P][Q] = V (mu^-1 X_P).X_Q.
// ISO: real (material scalars applied per entry); DIAG symmetric / FULL general: complex.
template <int KIND, typename R>
struct Tensors {
  CR<R> G[4][4], H[6][6];
};
template <typename R>
struct Tensors<EMG_MAT_ISO, R> {
  R G[4][4], H[6][6];
};
// the lane's part (real or imaginary) of beta G and alpha H
template <typename R>
struct Tensors<KIND_PAIR, R> {
  R G[4][4], H[6][6];
};
template <typename R>
struct Tensors<KIND_PAIR_FULL, R> {
  R G[4][4], H[6][6];
};
// G, H of the symmetric halves; the antisymmetric halves' 6 and 15 values above the
// diagonals lie in shared memory, value i at anti[32 i]: in registers they spilled
// 4.9 KB beside the moments
constexpr int ANTI_VALUES = 21;
template <typename R>
struct Tensors<KIND_PAIR_BOTH, R> {
  R G[4][4], H[6][6];
  R *anti;
};

// row-major N x N antisymmetric matrix over its values above the diagonal
template <int N, typename R>
struct Anti {
  const R *v;
  struct Row {
    const R *v;
    int m;
    __device__ __forceinline__ R operator[](int n) const {
      if (m == n) return (R)0;
      const int lo = m < n ? m : n, hi = m < n ? n : m;
      const R x = v[32 * (lo * (2 * N - 1 - lo) / 2 + hi - lo - 1)];
      return m < n ? x : -x;
    }
  };
  __device__ __forceinline__ Row operator[](int m) const { return {v, m}; }
};

__device__ __forceinline__ void cross3(const double a[3], const double b[3], double o[3]) {
  o[0] = a[1] * b[2] - a[2] * b[1];
  o[1] = a[2] * b[0] - a[0] * b[2];
  o[2] = a[0] * b[1] - a[1] * b[0];
}

template <typename R>
__device__ __forceinline__ void build_iso(const Geo &Gm, Tensors<EMG_MAT_ISO, R> &T) {
  double X[6][3];
  const int pa[6] = {0, 0, 0, 1, 1, 2}, pb[6] = {1, 2, 3, 2, 3, 3};
#pragma unroll
  for (int p = 0; p < 6; ++p) cross3(Gm.g[pa[p]], Gm.g[pb[p]], X[p]);
#pragma unroll
  for (int m = 0; m < 4; ++m)
#pragma unroll
    for (int n = m; n < 4; ++n) {
      double s = (Gm.g[m][0] * Gm.g[n][0] + Gm.g[m][1] * Gm.g[n][1] + Gm.g[m][2] * Gm.g[n][2]) * Gm.V;
      T.G[m][n] = T.G[n][m] = (R)s;
    }
#pragma unroll
  for (int p = 0; p < 6; ++p)
#pragma unroll
    for (int q = p; q < 6; ++q) {
      double s = (X[p][0] * X[q][0] + X[p][1] * X[q][1] + X[p][2] * X[q][2]) * Gm.V;
      T.H[p][q] = T.H[q][p] = (R)s;
    }
}

// complex tensors: eps, minv are 3x3 row-major complex; (A u).w = sum_r w_r sum_c A[r][c] u_c
template <int KIND, typename R>
__device__ __forceinline__ void build_cplx(const Geo &Gm, const C64 eps[9], const C64 minv[9], Tensors<KIND, R> &T) {
  double X[6][3];
  const int pa[6] = {0, 0, 0, 1, 1, 2}, pb[6] = {1, 2, 3, 2, 3, 3};
#pragma unroll
  for (int p = 0; p < 6; ++p) cross3(Gm.g[pa[p]], Gm.g[pb[p]], X[p]);
#pragma unroll
  for (int m = 0; m < 4; ++m)
#pragma unroll
    for (int n = 0; n < 4; ++n) {
      if (KIND == EMG_MAT_DIAG && n < m) {
        T.G[m][n] = T.G[n][m];
        continue;
      }
      double sr = 0, si = 0;
#pragma unroll
      for (int r = 0; r < 3; ++r)
#pragma unroll
        for (int c = 0; c < 3; ++c) {
          if (KIND == EMG_MAT_DIAG && r != c) continue;
          double w = Gm.g[n][r] * Gm.g[m][c];
          sr += eps[3 * r + c].re * w;
          si += eps[3 * r + c].im * w;
        }
      T.G[m][n] = {(R)(sr * Gm.V), (R)(si * Gm.V)};
    }
#pragma unroll
  for (int p = 0; p < 6; ++p)
#pragma unroll
    for (int q = 0; q < 6; ++q) {
      if (KIND == EMG_MAT_DIAG && q < p) {
        T.H[p][q] = T.H[q][p];
        continue;
      }
      double sr = 0, si = 0;
#pragma unroll
      for (int r = 0; r < 3; ++r)
#pragma unroll
        for (int c = 0; c < 3; ++c) {
          if (KIND == EMG_MAT_DIAG && r != c) continue;
          double w = X[q][r] * X[p][c];
          sr += minv[3 * r + c].re * w;
          si += minv[3 * r + c].im * w;
        }
      T.H[p][q] = {(R)(sr * Gm.V), (R)(si * Gm.V)};
    }
}

// The lane's part of the forms V b . t a of a 3x3 tensor t (row-major): (e g_m).g_n
// into G and (u X_P).X_Q into H, of the tensors' symmetric halves and, KIND_PAIR_BOTH,
// of their antisymmetric ones.
template <int KIND, typename R>
__device__ __forceinline__ void build_pair(const Geo &Gm, const double e[9], const double u[9], Tensors<KIND, R> &T) {
  double X[6][3];
  const int pa[6] = {0, 0, 0, 1, 1, 2}, pb[6] = {1, 2, 3, 2, 3, 3};
#pragma unroll
  for (int p = 0; p < 6; ++p) cross3(Gm.g[pa[p]], Gm.g[pb[p]], X[p]);
  auto form = [&](const double t[9], const double a[3], const double b[3]) {
    double s = 0.0;
#pragma unroll
    for (int r = 0; r < 3; ++r)
#pragma unroll
      for (int c = 0; c < 3; ++c) {
        if (KIND == KIND_PAIR && r != c) continue;
        const double v = r == c ? t[4 * r] : 0.5 * (t[3 * r + c] + t[3 * c + r]);
        s += v * (b[r] * a[c]);
      }
    return s * Gm.V;
  };
  // b . t a = w . (a x b), w = (t21, t02, t10)
  auto anti = [&](const double t[9], const double a[3], const double b[3]) {
    double c[3];
    cross3(a, b, c);
    return 0.5 * ((t[7] - t[5]) * c[0] + (t[2] - t[6]) * c[1] + (t[3] - t[1]) * c[2]) * Gm.V;
  };
  int i = 0;
#pragma unroll
  for (int m = 0; m < 4; ++m)
#pragma unroll
    for (int n = m; n < 4; ++n) {
      T.G[m][n] = T.G[n][m] = (R)form(e, Gm.g[m], Gm.g[n]);
      if constexpr (KIND == KIND_PAIR_BOTH)
        if (n > m) T.anti[32 * i++] = (R)anti(e, Gm.g[m], Gm.g[n]);
    }
#pragma unroll
  for (int p = 0; p < 6; ++p)
#pragma unroll
    for (int q = p; q < 6; ++q) {
      T.H[p][q] = T.H[q][p] = (R)form(u, X[p], X[q]);
      if constexpr (KIND == KIND_PAIR_BOTH)
        if (q > p) T.anti[32 * i++] = (R)anti(u, X[p], X[q]);
    }
}

template <int KIND, typename R>
struct EntryT {
  using T = CR<R>;
};
template <typename R>
struct EntryT<KIND_PAIR, R> {
  using T = R;
};
template <typename R>
struct EntryT<KIND_PAIR_FULL, R> {
  using T = R;
};
template <typename R>
struct EntryT<KIND_PAIR_BOTH, R> {
  using T = R;
};
template <typename R>
struct EntryT<EMG_MAT_ISO, R> {
  using T = R;
};

template <typename A>
__device__ __forceinline__ void scale_sign(A &x, double s);
template <>
__device__ __forceinline__ void scale_sign(double &x, double s) { x *= s; }
template <>
__device__ __forceinline__ void scale_sign(float &x, double s) { x *= (float)s; }
template <>
__device__ __forceinline__ void scale_sign(CR<double> &x, double s) { x.re *= s, x.im *= s; }
template <>
__device__ __forceinline__ void scale_sign(CR<float> &x, double s) { x.re *= (float)s, x.im *= (float)s; }

// entry (first=f, second=s) of K and M in the canonical frame, of the tensors G and H
template <int f, int s, int FORM, typename E, typename TG, typename TH, typename R>
__device__ __forceinline__ void contract(const TG &G, const TH &H, const R *mu, double sig, E &k, E &m) {
  E ak{}, am{};
  if constexpr (FORM != FORM_REF64) {
    emg_tables::Pair<f, s>::stiff(ak, H);
    emg_tables::Pair<f, s>::mass(am, G);
    if (emg_tables::odd(f) != emg_tables::odd(s)) {
      scale_sign(ak, sig);
      scale_sign(am, sig);
    }
  } else {
    emg_mtables::MPair<f, s>::stiff(ak, H, mu);
    emg_mtables::MPair<f, s>::mass(am, G, mu);
  }
  k = ak;
  m = am;
}

template <int f, int s, int FORM, int KIND, typename R>
__device__ __forceinline__ void entry(const Tensors<KIND, R> &T, const R *mu, double sig,
                                      typename EntryT<KIND, R>::T &k, typename EntryT<KIND, R>::T &m) {
  contract<f, s, FORM>(T.G, T.H, mu, sig, k, m);
}

// The lane's part of entry (lo, hi). Antisymmetric half: the first function is
// the DoF with the lower reference index (curlcurl.py:358-376).
template <int lo, int hi, int FORM, int KIND, typename R>
__device__ __forceinline__ R pair_value(const Tensors<KIND, R> &T, const R *mu, double sig, uint64_t inv) {
  R k, m;
  entry<lo, hi, FORM, KIND, R>(T, mu, sig, k, m);
  if constexpr (KIND == KIND_PAIR_BOTH && lo != hi) {
    R ka, ma;
    contract<lo, hi, FORM>(Anti<4, R>{T.anti}, Anti<6, R>{T.anti + 32 * 6}, mu, sig, ka, ma);
    return (k + m) + (ref_dof(inv, lo) > ref_dof(inv, hi) ? -(ka + ma) : ka + ma);
  }
  return k + m;
}

template <typename R>
struct StoreT;
template <>
struct StoreT<double> {
  using T = double2;
};
template <>
struct StoreT<float> {
  using T = float2;
};

constexpr int ELEM_THREADS = 128;

__device__ __forceinline__ double cfma(double a, double b, double c) { return __fma_rn(a, b, c); }
__device__ __forceinline__ float cfma(float a, float b, float c) { return __fmaf_rn(a, b, c); }
__device__ __forceinline__ double cmul_rn(double a, double b) { return __dmul_rn(a, b); }
__device__ __forceinline__ float cmul_rn(float a, float b) { return __fmul_rn(a, b); }

template <int x, int y, int FORM, int KIND, typename R>
__device__ __forceinline__ void compute_store(const Tensors<KIND, R> &T, const R *mu, double sig, const CR<R> &cK,
                                              const CR<R> &cM, uint64_t inv, int rx, typename StoreT<R>::T *row) {
  using ST = typename StoreT<R>::T;
  constexpr int lo = x < y ? x : y, hi = x < y ? y : x;
  const int b = ref_dof(inv, y);
  ST v;
  if constexpr (KIND >= KIND_PAIR) {
    reinterpret_cast<R *>(row + b)[threadIdx.x & 1] = pair_value<lo, hi, FORM, KIND, R>(T, mu, sig, inv);
    return;
  } else if constexpr (KIND == EMG_MAT_ISO) {
    R k0, m0;
    entry<lo, hi, FORM, KIND, R>(T, mu, sig, k0, m0);
    v.x = cfma(cK.re, k0, cmul_rn(cM.re, m0));
    v.y = cfma(cK.im, k0, cmul_rn(cM.im, m0));
  } else {
    CR<R> k, m;
    if constexpr (KIND == EMG_MAT_DIAG) {
      entry<lo, hi, FORM, KIND, R>(T, mu, sig, k, m);
    } else {
      // first = the DoF with the lower reference index (curlcurl.py:358-376)
      if (rx <= b) {
        entry<x, y, FORM, KIND, R>(T, mu, sig, k, m);
      } else {
        entry<y, x, FORM, KIND, R>(T, mu, sig, k, m);
      }
    }
    v.x = cfma(cK.re, k.re, cfma(-cK.im, k.im, cfma(cM.re, m.re, cmul_rn(-cM.im, m.im))));
    v.y = cfma(cK.re, k.im, cfma(cK.im, k.re, cfma(cM.re, m.im, cmul_rn(cM.im, m.re))));
  }
  row[b] = v;
}

// A row of KIND_PAIR_BOTH into the stage: entries (x, row_dof<LAYOUT, b>(s)), s < W, at
// row + s; of the COO block in the reference's order. A group of values is formed before
// the first is stored, as a store makes the compiler load the antisymmetric halves again.
template <int FORM>
__host__ __device__ constexpr int both_group() {
  return FORM == FORM_REF64 ? 2 : 20;
}

template <int LAYOUT, int b>
__host__ __device__ constexpr int row_dof(int s) {
  return LAYOUT == 0 ? s : (LAYOUT == 1 ? b + s : (s & 1 ? ent_dof2(b + s / 2) : ent_dof1(b + s / 2)));
}

template <int LAYOUT, int x, int b, int W, int FORM, int s, typename R>
__device__ __forceinline__ R both_value(const Tensors<KIND_PAIR_BOTH, R> &T, const R *mu, double sig, uint64_t inv) {
  if constexpr (s < W) {
    constexpr int y = row_dof<LAYOUT, b>(s);
    return pair_value<(x < y ? x : y), (x < y ? y : x), FORM, KIND_PAIR_BOTH, R>(T, mu, sig, inv);
  } else {
    return (R)0;
  }
}

template <int LAYOUT, int x, int b, int W, int FORM, int s0, typename R, int... Ss>
__device__ __forceinline__ void stage_both_group(const Tensors<KIND_PAIR_BOTH, R> &T, const R *mu, double sig,
                                                 uint64_t inv, double2 *row, std::integer_sequence<int, Ss...>) {
  const R v[] = {both_value<LAYOUT, x, b, W, FORM, s0 + Ss, R>(T, mu, sig, inv)...};
#pragma unroll
  for (int k = 0; k < both_group<FORM>(); ++k)
    if (s0 + k < W)
      reinterpret_cast<R *>(row + (LAYOUT == 0 ? ref_dof(inv, s0 + k) : s0 + k))[threadIdx.x & 1] = v[k];
}

template <int LAYOUT, int x, int b, int W, int FORM, typename R, int... Gs>
__device__ __forceinline__ void stage_both_row(const Tensors<KIND_PAIR_BOTH, R> &T, const R *mu, double sig,
                                               uint64_t inv, double2 *row, std::integer_sequence<int, Gs...>) {
  (stage_both_group<LAYOUT, x, b, W, FORM, both_group<FORM>() * Gs, R>(
       T, mu, sig, inv, row, std::make_integer_sequence<int, both_group<FORM>()>{}),
   ...);
}

template <int W, int FORM>
using both_groups = std::make_integer_sequence<int, (W + both_group<FORM>() - 1) / both_group<FORM>()>;

template <int x, int FORM, int KIND, typename R, int... Ys>
__device__ __forceinline__ void compute_row(const Tensors<KIND, R> &T, const R *mu, double sig, const CR<R> &cK,
                                            const CR<R> &cM, uint64_t inv, int rx, typename StoreT<R>::T *row,
                                            std::integer_sequence<int, Ys...>) {
  (compute_store<x, Ys, FORM, KIND, R>(T, mu, sig, cK, cM, inv, rx, row), ...);
}

template <int FORM, int KIND, typename R, int X>
__device__ __forceinline__ void do_row(const Tensors<KIND, R> &T, const R *mu, double sig, const CR<R> &cK,
                                       const CR<R> &cM, uint64_t inv, bool active, int ia,
                                       typename StoreT<R>::T *stage, typename StoreT<R>::T *out) {
  constexpr int LPT = lanes_per_tet(KIND);
  const int lane = threadIdx.x & 31;
  const int rx = ref_dof(inv, X);
  if (active) {
    if constexpr (KIND == KIND_PAIR_BOTH)
      stage_both_row<0, X, 0, 20, FORM, R>(T, mu, sig, inv, stage + lane / LPT * 21, both_groups<20, FORM>{});
    else
      compute_row<X, FORM, KIND, R>(T, mu, sig, cK, cM, inv, rx, stage + lane / LPT * 21,
                                    std::make_integer_sequence<int, 20>{});
  }
  __syncwarp();
  // cooperative, coalesced write of the warp's rows (one of 20 contiguous values per tet)
#pragma unroll 1
  for (int it = 0; it < 20 / LPT; ++it) {
    int e = it * 32 + lane;
    int r = e / 20, c = e - r * 20;
    int ia_r = __shfl_sync(0xffffffffu, ia, r * LPT);
    int a_r = __shfl_sync(0xffffffffu, rx, r * LPT);
    bool act_r = __shfl_sync(0xffffffffu, (int)active, r * LPT);
    if (act_r) out[(int64_t)ia_r * 400 + a_r * 20 + c] = stage[r * 21 + c];
  }
  __syncwarp();
}

template <int FORM, int KIND, typename R, int... Xs>
__device__ __forceinline__ void all_rows(const Tensors<KIND, R> &T, const R *mu, double sig, const CR<R> &cK,
                                         const CR<R> &cM, uint64_t inv, bool active, int ia,
                                         typename StoreT<R>::T *stage, typename StoreT<R>::T *out,
                                         std::integer_sequence<int, Xs...>) {
  (do_row<FORM, KIND, R, Xs>(T, mu, sig, cK, cM, inv, active, ia, stage, out), ...);
}

// ---- packed canonical layout: value[ia*210 + packed_index(x, y)], x <= y,
// canonical DoFs. Each unique pair is computed once; canonical row X (its
// 20 - X upper-triangle entries) is staged in shared memory and the warp
// writes its 32 row segments as contiguous runs.
template <int x, int y, int FORM, int KIND, typename R>
__device__ __forceinline__ typename StoreT<R>::T packed_value(const Tensors<KIND, R> &T, const R *mu, double sig,
                                                              const CR<R> &cK, const CR<R> &cM, uint64_t inv) {
  static_assert(KIND < KIND_PAIR, "a pair's lanes hold half a value each");
  typename StoreT<R>::T v;
  if constexpr (KIND == EMG_MAT_ISO) {
    R k0, m0;
    entry<x, y, FORM, KIND, R>(T, mu, sig, k0, m0);
    v.x = cfma(cK.re, k0, cmul_rn(cM.re, m0));
    v.y = cfma(cK.im, k0, cmul_rn(cM.im, m0));
  } else {
    CR<R> k, m;
    if constexpr (KIND == EMG_MAT_DIAG) {
      entry<x, y, FORM, KIND, R>(T, mu, sig, k, m);
    } else {
      // first = the DoF with the lower reference index (curlcurl.py:358-376)
      if (ref_dof(inv, x) <= ref_dof(inv, y)) {
        entry<x, y, FORM, KIND, R>(T, mu, sig, k, m);
      } else {
        entry<y, x, FORM, KIND, R>(T, mu, sig, k, m);
      }
    }
    v.x = cfma(cK.re, k.re, cfma(-cK.im, k.im, cfma(cM.re, m.re, cmul_rn(-cM.im, m.im))));
    v.y = cfma(cK.re, k.im, cfma(cK.im, k.re, cfma(cM.re, m.im, cmul_rn(cM.im, m.re))));
  }
  return v;
}

template <int x, int y, int FORM, int KIND, typename R>
__device__ __forceinline__ void compute_store_packed(const Tensors<KIND, R> &T, const R *mu, double sig,
                                                     const CR<R> &cK, const CR<R> &cM, uint64_t inv,
                                                     typename StoreT<R>::T *row) {
  if constexpr (KIND >= KIND_PAIR)
    reinterpret_cast<R *>(row + (y - x))[threadIdx.x & 1] = pair_value<x, y, FORM, KIND, R>(T, mu, sig, inv);
  else
    row[y - x] = packed_value<x, y, FORM, KIND, R>(T, mu, sig, cK, cM, inv);
}

template <int x, int FORM, int KIND, typename R, int... Ds>
__device__ __forceinline__ void compute_row_packed(const Tensors<KIND, R> &T, const R *mu, double sig,
                                                   const CR<R> &cK, const CR<R> &cM, uint64_t inv,
                                                   typename StoreT<R>::T *row, std::integer_sequence<int, Ds...>) {
  (compute_store_packed<x, x + Ds, FORM, KIND, R>(T, mu, sig, cK, cM, inv, row), ...);
}

template <int FORM, int KIND, typename R, int X>
__device__ __forceinline__ void do_row_packed(const Tensors<KIND, R> &T, const R *mu, double sig, const CR<R> &cK,
                                              const CR<R> &cM, uint64_t inv, bool active, int ia,
                                              typename StoreT<R>::T *stage, typename StoreT<R>::T *out) {
  constexpr int W = 20 - X, LPT = lanes_per_tet(KIND);
  const int lane = threadIdx.x & 31;
  if (active) {
    if constexpr (KIND == KIND_PAIR_BOTH)
      stage_both_row<1, X, X, W, FORM, R>(T, mu, sig, inv, stage + lane / LPT * (W | 1), both_groups<W, FORM>{});
    else
      compute_row_packed<X, FORM, KIND, R>(T, mu, sig, cK, cM, inv, stage + lane / LPT * (W | 1),
                                           std::make_integer_sequence<int, W>{});
  }
  // the warp's tets are consecutive assembled indices: the r-th one's is ia - lane / LPT + r
  const unsigned act = __ballot_sync(0xffffffffu, active);
  const int64_t ia_w = (int64_t)ia - lane / LPT;
  __syncwarp();
#pragma unroll 2
  for (int e = lane; e < 32 / LPT * W; e += 32) {
    const int r = e / W, c = e - r * W;
    if ((act >> (r * LPT)) & 1u) out[(ia_w + r) * 210 + packed_index(X, X) + c] = stage[r * (W | 1) + c];
  }
  __syncwarp();
}

template <int FORM, int KIND, typename R, int... Xs>
__device__ __forceinline__ void all_rows_packed(const Tensors<KIND, R> &T, const R *mu, double sig, const CR<R> &cK,
                                                const CR<R> &cM, uint64_t inv, bool active, int ia,
                                                typename StoreT<R>::T *stage, typename StoreT<R>::T *out,
                                                std::integer_sequence<int, Xs...>) {
  (do_row_packed<FORM, KIND, R, Xs>(T, mu, sig, cK, cM, inv, active, ia, stage, out), ...);
}

// ---- entity-pair block layout: value[ia*220 + 4*block_index(i, j) + k] for
// canonical entities i <= j. Each value is the packed layout's (min, max) entry.
// wide: values aligned to 32 bytes, written a whole sector at a time; others are
// written one by one.
//
// A lane that owns its tet stores the values straight from registers, a sector per
// instruction: half a complex128 block or a complex64 block. The stores need no
// answer and drain beside the arithmetic. Staged in shared memory and written by
// the warp as runs of up to 640 bytes, rows and write-back took turns in the eight
// warps that the registers leave an SM. 1.008M tets: isotropic FP64 779 -> 640 us
// (3.55 GB; 447 without its stores), exact isotropic 619. The mixed form, 367 ->
// 362, is bound by these writes: 82 without them, and tets 1,760 bytes apart take
// them at 4.9 TB/s where a fill reaches 7.3. Tiles of 4 to 32 tets per block
// would be written faster (mixed 314 to 332) but scatter what the gather reads:
// 1,426 -> 2,326 us with the tets in random order.
__device__ __forceinline__ void store_half(double2 *o, double2 v0, double2 v1, bool wide) {
  if (wide) {
    asm volatile("st.global.v4.f64 [%0], {%1, %2, %3, %4};" ::"l"(o), "d"(v0.x), "d"(v0.y), "d"(v1.x), "d"(v1.y)
                 : "memory");
  } else {
    o[0] = v0;
    o[1] = v1;
  }
}

__device__ __forceinline__ void store_block(float2 *o, float2 v0, float2 v1, float2 v2, float2 v3, bool wide) {
  if (wide) {
    asm volatile("st.global.v8.f32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8};" ::"l"(o), "f"(v0.x), "f"(v0.y),
                 "f"(v1.x), "f"(v1.y), "f"(v2.x), "f"(v2.y), "f"(v3.x), "f"(v3.y)
                 : "memory");
  } else {
    o[0] = v0;
    o[1] = v1;
    o[2] = v2;
    o[3] = v3;
  }
}

// A block row's values as one lane forms them, in the order that it stores them:
// FP64 the first DoF's entries of all blocks, then the second's (the packed
// triangle's row order); FP32 block by block.
template <int FORM, int KIND, typename R>
struct BlockRow {
  using ST = typename StoreT<R>::T;
  const Tensors<KIND, R> &T;
  const R *mu;
  const double sig;
  const CR<R> &cK, &cM;
  const uint64_t inv;
  const bool wide;

  template <int x, int y>
  __device__ __forceinline__ ST value() const {
    return packed_value<(x < y ? x : y), (x < y ? y : x), FORM, KIND, R>(T, mu, sig, cK, cM, inv);
  }
  // entries (x, first DoF of entity j) and (x, second DoF of j)
  template <int x, int j>
  __device__ __forceinline__ void half(ST *o) const {
    const ST v0 = value<x, ent_dof1(j)>(), v1 = value<x, ent_dof2(j)>();
    store_half(o, v0, v1, wide);
  }
  template <int i, int j>
  __device__ __forceinline__ void block(ST *o) const {
    const ST v0 = value<ent_dof1(i), ent_dof1(j)>(), v1 = value<ent_dof1(i), ent_dof2(j)>();
    const ST v2 = value<ent_dof2(i), ent_dof1(j)>(), v3 = value<ent_dof2(i), ent_dof2(j)>();
    store_block(o, v0, v1, v2, v3, wide);
  }
  template <int i, int... Js>
  __device__ __forceinline__ void store(ST *row, std::integer_sequence<int, Js...>) const {
    if constexpr (sizeof(R) == 4) {
      (block<i, i + Js>(row + 4 * Js), ...);
    } else {
      (half<ent_dof1(i), i + Js>(row + 4 * Js), ...);
      (half<ent_dof2(i), i + Js>(row + 4 * Js + 2), ...);
    }
  }
};

// A pair's lanes hold half a value each, so their row is staged, one tet's values
// an odd number apart, and the warp writes its 16 tets' rows, for diagonal tensors
// two values at a time: 1.008M tets, one 1,120 us, two 1,060, exchanged by a shuffle
// and stored by the lanes 1,100. Full tensors leave no registers for it (504k tets,
// one 690 us, two 799, by the lanes 904).
template <int x, int y, int FORM, int KIND, typename R>
__device__ __forceinline__ void stage_half_value(const Tensors<KIND, R> &T, const R *mu, double sig, uint64_t inv,
                                                 double2 *dst) {
  reinterpret_cast<R *>(dst)[threadIdx.x & 1] =
      pair_value<(x < y ? x : y), (x < y ? y : x), FORM, KIND, R>(T, mu, sig, inv);
}

template <int i, int FORM, int KIND, typename R, int... Js>
__device__ __forceinline__ void stage_block_row(const Tensors<KIND, R> &T, const R *mu, double sig, uint64_t inv,
                                                double2 *row, std::integer_sequence<int, Js...>) {
  ((stage_half_value<ent_dof1(i), ent_dof1(i + Js), FORM, KIND, R>(T, mu, sig, inv, row + 4 * Js + 0),
    stage_half_value<ent_dof1(i), ent_dof2(i + Js), FORM, KIND, R>(T, mu, sig, inv, row + 4 * Js + 1)),
   ...);
  ((stage_half_value<ent_dof2(i), ent_dof1(i + Js), FORM, KIND, R>(T, mu, sig, inv, row + 4 * Js + 2),
    stage_half_value<ent_dof2(i), ent_dof2(i + Js), FORM, KIND, R>(T, mu, sig, inv, row + 4 * Js + 3)),
   ...);
}

// HALF 0, 1: the first, the second DoF's entries of block row I (KIND_PAIR_BOTH); 2: both
template <int FORM, int KIND, typename R, int I, int HALF>
__device__ __forceinline__ void store_pair_row(const Tensors<KIND, R> &T, const R *mu, double sig, uint64_t inv,
                                               bool active, int ia, bool wide, double2 *stage, double2 *out) {
  // V values at a time
  constexpr int W = (HALF == 2 ? 4 : 2) * (10 - I), LPT = lanes_per_tet(KIND), V = KIND == KIND_PAIR ? 2 : 1;
  constexpr int ROUNDS = W / LPT / V;
  static_assert(W % (LPT * V) == 0, "whole rounds of the warp");
  const int lane = threadIdx.x & 31;
  if (active) {
    if constexpr (HALF == 2)
      stage_block_row<I, FORM, KIND, R>(T, mu, sig, inv, stage + lane / LPT * (W | 1),
                                        std::make_integer_sequence<int, 10 - I>{});
    else
      stage_both_row<2, HALF ? ent_dof2(I) : ent_dof1(I), I, W, FORM, R>(T, mu, sig, inv, stage + lane / LPT * (W | 1),
                                                                         both_groups<W, FORM>{});
  }
  // the warp's tets are consecutive assembled indices: the r-th one's is ia - lane / LPT + r
  const unsigned act = __ballot_sync(0xffffffffu, active);
  const int64_t ia_w = (int64_t)ia - lane / LPT;
  __syncwarp();
#pragma unroll 2
  for (int it = 0; it < ROUNDS; ++it) {
    const int e = it * 32 + lane;
    const int r = e / (W / V), c = V * (e - r * (W / V));
    if ((act >> (r * LPT)) & 1u) {
      const int at = HALF == 2 ? c : 2 * HALF + 4 * (c / 2) + (c & 1);
      double2 *o = out + (ia_w + r) * kBlockValues + 4 * block_index(I, I) + at;
      const double2 *v = stage + r * (W | 1) + c;
      if constexpr (V == 2)
        store_half(o, v[0], v[1], wide);
      else
        *o = v[0];
    }
  }
  __syncwarp();
}

template <int FORM, int KIND, typename R, int I>
__device__ __forceinline__ void do_row_block(const Tensors<KIND, R> &T, const R *mu, double sig, const CR<R> &cK,
                                             const CR<R> &cM, uint64_t inv, bool active, int ia, bool wide,
                                             typename StoreT<R>::T *stage, typename StoreT<R>::T *out) {
  if constexpr (KIND < KIND_PAIR) {
    if (active)
      BlockRow<FORM, KIND, R>{T, mu, sig, cK, cM, inv, wide}.template store<I>(
          out + (int64_t)ia * kBlockValues + 4 * block_index(I, I), std::make_integer_sequence<int, 10 - I>{});
    __syncwarp();  // the compiler would otherwise form products of later rows ahead, and spill them
  } else if constexpr (KIND == KIND_PAIR_BOTH) {
    store_pair_row<FORM, KIND, R, I, 0>(T, mu, sig, inv, active, ia, wide, stage, out);
    store_pair_row<FORM, KIND, R, I, 1>(T, mu, sig, inv, active, ia, wide, stage, out);
  } else {
    store_pair_row<FORM, KIND, R, I, 2>(T, mu, sig, inv, active, ia, wide, stage, out);
  }
}

template <int FORM, int KIND, typename R, int... Is>
__device__ __forceinline__ void all_rows_block(const Tensors<KIND, R> &T, const R *mu, double sig, const CR<R> &cK,
                                               const CR<R> &cM, uint64_t inv, bool active, int ia, unsigned rows,
                                               typename StoreT<R>::T *stage, typename StoreT<R>::T *out,
                                               std::integer_sequence<int, Is...>) {
  const bool wide = (reinterpret_cast<uintptr_t>(out) & 31) == 0;
  ((rows >> Is & 1u ? do_row_block<FORM, KIND, R, Is>(T, mu, sig, cK, cM, inv, active, ia, wide, stage, out)
                    : (void)0),
   ...);
}

// staged values per tet: the longest row, its stride odd, so that the lanes' stores
// of one value position fall in distinct shared-memory bank groups
template <int LAYOUT, int TK>
__host__ __device__ constexpr int stage_values() {
  return LAYOUT != 2 ? 21 : (TK == KIND_PAIR_BOTH ? 21 : (TK >= KIND_PAIR ? 41 : 0));
}

// shared memory of a warp: its tets' staged rows; for full tensors in pairs at least the
// rows and the antisymmetric halves of KIND_PAIR_BOTH (which stages half block rows)
template <int LAYOUT, int TK, typename ST>
__host__ __device__ constexpr size_t stage_bytes() {
  const size_t rows = (size_t)32 / lanes_per_tet(TK) * stage_values<LAYOUT, TK>() * sizeof(ST);
  const size_t both = (size_t)16 * stage_values<LAYOUT, KIND_PAIR_BOTH>() * sizeof(ST) + 32 * ANTI_VALUES * sizeof(double);
  return TK == KIND_PAIR_FULL && both > rows ? both : rows;
}

// LAYOUT 0: the reference's COO block [ia][a][b] (400 values, each entry
//           computed in both of its rows);
// LAYOUT 1: the packed canonical upper triangle [ia][210] (each unique
//           entry computed once);
// LAYOUT 2: the entity-pair blocks [ia][220] (the assembly path)
// One CTA's tets (elem_tets_per_cta), from assembled index ia0 of the job a on
// (every thread of the CTA calls it with the same ia0).
// TK: the tensors' form; mine: whether this lane's tet takes part.
template <int FORM, int KIND, int LAYOUT, int TK>
__device__ __forceinline__ void element_pass(const ElemArgs &a, int64_t ia0, bool mine, unsigned rows,
                                             unsigned char *stage_raw) {
  using R = typename FormReal<FORM>::T;
  using ST = typename StoreT<R>::T;
  constexpr int LPT = lanes_per_tet(TK);
  unsigned char *const shared = stage_raw + (threadIdx.x >> 5) * stage_bytes<LAYOUT, tensor_kind(FORM, KIND), ST>();
  ST *stage = reinterpret_cast<ST *>(shared);
  ST *out = reinterpret_cast<ST *>(a.out);
  const int64_t ia64 = ia0 + threadIdx.x / LPT;
  bool active = mine && ia64 < a.nA;
  const int ia = (int)ia64;
  Geo G;
  Tensors<TK, R> T;
  R mu[FORM == FORM_REF64 ? NMOM : 1];
  if constexpr (FORM == FORM_REF64) {
#pragma unroll
    for (int i = 0; i < NMOM; ++i) mu[i] = (R)0;
  }
  CR<R> cK{0, 0}, cM{0, 0};
  double sig = 1.0;
  uint64_t inv = 0;
  if constexpr (TK == KIND_PAIR_BOTH)
    T.anti = reinterpret_cast<R *>(shared + 32 / LPT * stage_values<LAYOUT, TK>() * sizeof(ST)) + (threadIdx.x & 31);
  if (active) {
    int64_t it = a.tetids ? (int64_t)a.tetids[ia] : ia64;
    int64_t v[4];
    bool ok = (it >= 0 && it < a.nT);
    if (ok) {
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        v[q] = a.tets[(int64_t)q * a.nT + it];
        ok &= (v[q] >= 0 && v[q] < a.nN);
      }
    }
    if (!ok) {
      flag(a.st, EMG_ST_INDEX, ia64);
      active = false;
    } else {
      double X[3][4];
#pragma unroll
      for (int q = 0; q < 4; ++q)
#pragma unroll
        for (int d = 0; d < 3; ++d) X[d][q] = a.nodes[(int64_t)d * a.nN + v[q]];
      bool good;
      if constexpr (FORM != FORM_REF64) {
        good = exact_geometry(X, v, G);
      } else {
        good = ref_geometry<LPT == 2, R>(X, v, G, mu);
      }
      if (!good) {
        flag(a.st, EMG_ST_DEGENERATE, ia64);
        active = false;
      } else {
        sig = G.sig;
        inv = G.inv;
        const C64 alpha{a.ar, a.ai}, beta{a.br, a.bi};
        if constexpr (KIND == EMG_MAT_ISO) {
          C64 eps = ld_c64(a.er, it);
          C64 minv = a.ur ? crecip(ld_c64(a.ur, it)) : C64{1.0, 0.0};
          C64 k = cmul(alpha, minv), m = cmul(beta, eps);
          cK = {(R)k.re, (R)k.im};
          cM = {(R)m.re, (R)m.im};
          build_iso<R>(G, T);
        } else {
          C64 eps[9], mu3[9], minv[9];
#pragma unroll
          for (int r = 0; r < 3; ++r)
#pragma unroll
            for (int c = 0; c < 3; ++c) {
              // DIAG: compact diagonals [3][nT]; FULL: the reference's [3][3][nT]
              const bool need = (KIND == EMG_MAT_FULL) || r == c;
              const int64_t o = (KIND == EMG_MAT_FULL) ? (int64_t)(3 * r + c) * a.nT + it : (int64_t)r * a.nT + it;
              eps[3 * r + c] = need ? ld_c64(a.er, o) : C64{0.0, 0.0};
              mu3[3 * r + c] = (need && a.ur) ? ld_c64(a.ur, o) : C64{(r == c) ? 1.0 : 0.0, 0.0};
            }
          matinv3(mu3, minv);
          if constexpr (LPT == 2) {
            double e[9], u[9];
#pragma unroll
            for (int i = 0; i < 9; ++i) {
              const C64 ce = cmul(beta, eps[i]), cu = cmul(alpha, minv[i]);
              e[i] = (threadIdx.x & 1) ? ce.im : ce.re;
              u[i] = (threadIdx.x & 1) ? cu.im : cu.re;
            }
            build_pair<TK, R>(G, e, u, T);
          } else {
            cK = {(R)alpha.re, (R)alpha.im};
            cM = {(R)beta.re, (R)beta.im};
            build_cplx<KIND, R>(G, eps, minv, T);
          }
        }
      }
    }
  }
  if constexpr (LPT == 2 && FORM == FORM_REF64) {  // both halves of the points
#pragma unroll
    for (int i = 0; i < NMOM; ++i) mu[i] += __shfl_xor_sync(0xffffffffu, mu[i], 1);
  }
  if constexpr (LAYOUT == 0) {
    all_rows<FORM, TK, R>(T, mu, sig, cK, cM, inv, active, ia, stage, out, std::make_integer_sequence<int, 20>{});
  } else if constexpr (LAYOUT == 2) {
    all_rows_block<FORM, TK, R>(T, mu, sig, cK, cM, inv, active, ia, rows, stage, out,
                                std::make_integer_sequence<int, 10>{});
  } else {
    all_rows_packed<FORM, TK, R>(T, mu, sig, cK, cM, inv, active, ia, stage, out,
                                   std::make_integer_sequence<int, 20>{});
  }
}

// Whether a tensor of the lane's tet is not symmetric; the even lane of a pair looks at
// its eps, the odd one at its mu.
__device__ __forceinline__ bool not_reciprocal(const ElemArgs &a, int64_t ia) {
  bool other = false;
  const double2 *t = static_cast<const double2 *>((threadIdx.x & 1) ? a.ur : a.er);
  const int64_t it = ia < a.nA ? (a.tetids ? (int64_t)a.tetids[ia] : ia) : -1;
  if (t && it >= 0 && it < a.nT) {
#pragma unroll
    for (int i = 0; i < 3; ++i) {
      const int rc[3] = {1, 2, 5}, cr[3] = {3, 6, 7};
      const double2 x = __ldg(t + rc[i] * a.nT + it), y = __ldg(t + cr[i] * a.nT + it);
      other = other || x.x != y.x || x.y != y.y;
    }
  }
  return __shfl_xor_sync(0xffffffffu, (int)other, 1) || other;
}

// rows: bit i set to write block row i (block layout; the others write all rows).
// Full tensors in pairs: a tet's pass depends on its own tensors alone, so its values
// are the same whatever its neighbours are.
template <int FORM, int KIND, int LAYOUT>
__device__ __forceinline__ void element_cta(const ElemArgs &a, int64_t ia0, unsigned rows, unsigned char *stage_raw) {
  constexpr int TK = tensor_kind(FORM, KIND);
  if constexpr (TK == KIND_PAIR_FULL) {
    const int64_t ia = ia0 + threadIdx.x / 2;
    const bool other = not_reciprocal(a, ia);
    if (__any_sync(0xffffffffu, !other && ia < a.nA))
      element_pass<FORM, KIND, LAYOUT, TK>(a, ia0, !other, rows, stage_raw);
    if (__any_sync(0xffffffffu, other)) element_pass<FORM, KIND, LAYOUT, KIND_PAIR_BOTH>(a, ia0, other, rows, stage_raw);
  } else {
    element_pass<FORM, KIND, LAYOUT, TK>(a, ia0, true, rows, stage_raw);
  }
}

// A mesh that leaves SMs idle: its tets are gone through by several CTAs,
// blockIdx.y of n_parts, each of which forms the geometry and moments again but only
// some of the block rows (row i has 10 - i blocks). The time of such a launch is that
// of one tet. As many parts as give each CTA an SM of its own. One assembly (element
// and gather, graph replays) on one stream, and per assembly with eight streams at
// once, whole -> in parts: 576 tets FP64 (five parts) 23.0 -> 16.7 us and 3.6 -> 2.9;
// 4,950 (three) FP64 27.1 -> 21.6 and 11.6 -> 13.3, mixed 16.7 -> 14.4 and 8.9 -> 8.4;
// 8,640 (two) FP64 33.2 -> 29.1 and 19.2 -> 20.7, mixed 21.2 -> 19.7 and 14.5 -> 14.2.
// As many parts as fit two CTAs per SM (five, three, two at 12,960 tets): FP64 22.9, 30.5
// and 42.1 us, no faster, but 15.4, 22.5 and 31.0 with eight streams, as the repeated
// part takes the other launches' SMs.
constexpr unsigned ALL_ROWS = 0x3ffu;
__device__ __forceinline__ unsigned part_rows(int part, int n_parts) {
  if (n_parts == 2) return part ? 0x3f8u : 0x007u;                                  // 27 and 28 blocks
  if (n_parts == 3) return part == 0 ? 0x003u : (part == 1 ? 0x10cu : 0x2f0u);      // 19, 17, 19
  if (n_parts == 5) return (1u << part) | (1u << (9 - part));                       // 11 each
  return ALL_ROWS;
}

// CTAs per SM the compiler must fit. The isotropic FP64 forms at their natural
// 232-255 registers (two CTAs) beat every cap (three CTAs, 2.01M tets: 1.84 ->
// 3.68 ms, 1.9 KB of spills); the mixed form takes 88-254 (five CTAs per SM for the
// isotropic instance; held to six or seven, 1.008M tets: 362 -> 375 / 385 us).
template <int FORM, int KIND>
constexpr int elem_min_blocks() {
  return 1;
}

// tets of a CTA; elem_tets_per_cta for the host
template <int FORM, int KIND>
__host__ __device__ constexpr int elem_tets() {
  return ELEM_THREADS / lanes_per_tet(tensor_kind(FORM, KIND));
}

template <int FORM, int KIND, int LAYOUT>
__global__ void __launch_bounds__(ELEM_THREADS, elem_min_blocks<FORM, KIND>()) k_element(ElemArgs a) {
  extern __shared__ __align__(16) unsigned char stage_raw[];
  element_cta<FORM, KIND, LAYOUT>(a, (int64_t)blockIdx.x * elem_tets<FORM, KIND>(), part_rows(blockIdx.y, gridDim.y),
                                  stage_raw);
}

// Several jobs (meshes, materials, coefficients, outputs) in one launch of
// the packed form: job j owns the CTAs [cta_start[j], cta_start[j + 1]) and
// its tets in CTA order, as if launched alone.
template <int FORM, int KIND, int LAYOUT>
__global__ void __launch_bounds__(ELEM_THREADS, elem_min_blocks<FORM, KIND>())
    k_element_batch(const ElemArgs *jobs, const int64_t *cta_start, int n_jobs) {
  extern __shared__ __align__(16) unsigned char stage_raw[];
  const int64_t b = blockIdx.x;
  int lo = 0, hi = n_jobs - 1;  // the job with cta_start[j] <= b < cta_start[j + 1]
  while (lo < hi) {
    const int mid = (lo + hi + 1) >> 1;
    if (cta_start[mid] <= b) lo = mid;
    else hi = mid - 1;
  }
  if (n_jobs <= 0 || b >= cta_start[n_jobs]) return;
  element_cta<FORM, KIND, LAYOUT>(jobs[lo], (b - cta_start[lo]) * elem_tets<FORM, KIND>(), ALL_ROWS, stage_raw);
}

template <int FORM, int KIND, int LAYOUT>
int launch_element_t(const ElemArgs &a, cudaStream_t s) {
  using ST = typename StoreT<typename FormReal<FORM>::T>::T;
  constexpr size_t smem = ELEM_THREADS / 32 * stage_bytes<LAYOUT, tensor_kind(FORM, KIND), ST>();
  static_assert(elem_tets<FORM, KIND>() == elem_tets_per_cta(FORM, KIND), "the host's table of CTAs");
  // the attribute belongs to the current device: set once per device (benign
  // race: every thread that gets here sets the same value)
  static bool configured[64] = {false};
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0) dev = 0;
  if (dev >= 64 || !configured[dev]) {
    cudaError_t e = cudaFuncSetAttribute(k_element<FORM, KIND, LAYOUT>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                         (int)smem);
    if (e != cudaSuccess) return fail(EMG_ECUDA, "cudaFuncSetAttribute(k_element): %s", cudaGetErrorString(e));
    if (dev < 64) configured[dev] = true;
  }
  if (a.nA == 0) return EMG_OK;
  const int ctas = grid_for(a.nA, elem_tets<FORM, KIND>());
  int parts = 1;
  if (LAYOUT == 2)  // the most parts that still have an SM each
    for (int p : {2, 3, 5})
      if ((int64_t)ctas * p <= persistent_ctas(1)) parts = p;
  k_element<FORM, KIND, LAYOUT><<<dim3(ctas, parts), ELEM_THREADS, smem, s>>>(a);
  return launch_check("k_element");
}

template <int FORM, int KIND, int LAYOUT>
int launch_element_batch_t(const ElemArgs *d_jobs, const int64_t *d_cta_start, int n_jobs, int64_t total_ctas,
                           cudaStream_t s) {
  using ST = typename StoreT<typename FormReal<FORM>::T>::T;
  constexpr size_t smem = ELEM_THREADS / 32 * stage_bytes<LAYOUT, tensor_kind(FORM, KIND), ST>();
  static bool configured[64] = {false};
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0) dev = 0;
  if (dev >= 64 || !configured[dev]) {
    cudaError_t e =
        cudaFuncSetAttribute(k_element_batch<FORM, KIND, LAYOUT>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                             (int)smem);
    if (e != cudaSuccess) return fail(EMG_ECUDA, "cudaFuncSetAttribute(k_element_batch): %s", cudaGetErrorString(e));
    if (dev < 64) configured[dev] = true;
  }
  if (n_jobs == 0 || total_ctas == 0) return EMG_OK;
  if (total_ctas > INT32_MAX) return fail(EMG_ERANGE, "too many CTAs (%lld)", (long long)total_ctas);
  k_element_batch<FORM, KIND, LAYOUT><<<(unsigned)total_ctas, ELEM_THREADS, smem, s>>>(d_jobs, d_cta_start,
                                                                                       n_jobs);
  return launch_check("k_element_batch");
}

template <int FORM, int KIND>
int launch_element_k(const ElemArgs &a, int layout, cudaStream_t s) {
  if (layout == EMG_LAYOUT_COO) return launch_element_t<FORM, KIND, 0>(a, s);
  if (layout == EMG_LAYOUT_PACKED) return launch_element_t<FORM, KIND, 1>(a, s);
  if (layout == EMG_LAYOUT_BLOCK) return launch_element_t<FORM, KIND, 2>(a, s);
  return fail(EMG_EINVAL, "bad layout %d", layout);
}

}  // namespace
}  // namespace emg
