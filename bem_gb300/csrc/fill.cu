// PMCHWT RWG impedance fill on the GPU: Zts (src/Impedance.cpp:276-413).
//
// Work decomposition
//   * far pairs (no shared vertex): the reference contracts the inner integrals
//     per half-RWG (Gphi[j], DGxphi[j], src/Impedance.cpp:126-167); here a pair
//     is reduced to the 3 x 3 moments over {1, eta1, eta2} x {1, xi1, xi2} (the
//     two triangles' barycentric coordinates) of g and of q (g, q of
//     GreensFunction::scalar_gradient, gradient = q (r_t - r_s)), from which all
//     nine (i, j) products L_ij, K_ij follow in closed form (far_contract()).
//     One thread per pair with the 6-point rule, one warp per pair with a larger
//     one.  Both triangles of a far pair take the same rule, so L and K are
//     symmetric in the pair: a fill of a tree against itself integrates each
//     unordered pair once and writes both its places.
//   * near pairs (same triangle or a shared vertex): one warp per pair, which
//     reduces the smooth inner rule and the closed-form singular terms to real
//     moments (powers of R: no frequency in them) and serves the exterior and
//     the interior Green's function of a body in one pass; see near_pairs_kernel.
//   * every pair writes its nine (c L_ij, c K_ij) half-pair products into a
//     half-pair block array H (one 128-byte block per RWG pair (i, j), four
//     slots for (pos/neg test half) x (pos/neg source half)); each slot has
//     exactly one writer, so no atomics are needed.  A gather kernel then
//     reduces each block into the 2x2 (J, M) entries of Z in RWG-pair order with
//     coalesced stores (src/Impedance.cpp:365-384).
#include "bemgpu_internal.h"
#include "quadrature_tables.h"
#include "even_rules.h"
#include "fill_num.cuh"

#include <algorithm>
#include <cmath>
#include <cstring>
#include <type_traits>
#include <vector>

namespace {

struct GreenDev {
  double ikr, iki;      // ik
  double k2r, k2i;      // k2 = -ksquared/2
  double ksqr, ksqi;    // ksquared
  // the same as double-float pairs (hi, lo), split on the host
  float ikr_f[2], iki_f[2], k2r_f[2], k2i_f[2], ksqr_f[2], ksqi_f[2];
};

struct FarOpts {
  double th6, th10, th15, th21;
};

// Fill arithmetic: FP64 (parity path), FP32 far pairs beyond 3 edge lengths,
// or double-float for every quadrature node pair.
enum { FILL_FP64 = 0, FILL_FP32_FAR = 1, FILL_DF = 2 };

// A node of a triangle rule: barycentric coordinates, weight, weight times each.
template <typename T>
struct RuleNode {
  T x1, x2, w, w1, w2;
};
// The far rules' nodes one after the other, in both number types.
enum { NODES6 = 0, NODES10 = 6, NODES15 = 16, NODES21 = 31, NODES36 = 52, NODES_FAR = 88 };
__constant__ RuleNode<double> c_far_d[NODES_FAR];
__constant__ RuleNode<df> c_far_f[NODES_FAR];
// Sums of {w, w x1, w x2} per rule, and the square of the weights' sum less one.
enum { SUM6, SUM10, SUM15, SUM21, SUM36, SUM91, SUM105, NSUMS };
struct RuleSum {
  double w[3], ww1;
};
__constant__ RuleSum c_sums[NSUMS];
template <typename T>
__device__ __forceinline__ RuleNode<T> far_node(int k);
template <>
__device__ __forceinline__ RuleNode<double> far_node<double>(int k) { return c_far_d[k]; }
template <>
__device__ __forceinline__ RuleNode<df> far_node<df>(int k) { return c_far_f[k]; }
__constant__ double c_rule6[6][3];
__constant__ double c_rule10[10][3];
__constant__ double c_rule15[15][3];
__constant__ double c_rule21[21][3];
__constant__ double c_rule36[36][3];
__constant__ double c_line15[15][2];

// ---------------- small FP64 vector / complex helpers ----------------
struct d3 {
  double x, y, z;
};
struct z1 {
  double r, i;
};

__device__ __forceinline__ d3 ld3(const double *p) { return {p[0], p[1], p[2]}; }
__device__ __forceinline__ d3 operator-(d3 a, d3 b) { return {a.x - b.x, a.y - b.y, a.z - b.z}; }
__device__ __forceinline__ double dot(d3 a, d3 b) { return a.x * b.x + a.y * b.y + a.z * b.z; }
__device__ __forceinline__ z1 zmul(z1 a, z1 b) { return {a.r * b.r - a.i * b.i, a.r * b.i + a.i * b.r}; }
__device__ __forceinline__ z1 zadd(z1 a, z1 b) { return {a.r + b.r, a.i + b.i}; }

__device__ __forceinline__ int shares_vertex(const int *a, const int *b) {
  int c = 0;
#pragma unroll
  for (int i = 0; i < 3; i++) c += (a[i] == b[0]) | (a[i] == b[1]) | (a[i] == b[2]);
  return c;
}

// IEEE-exact squared distance without contraction (the far-rule test compares
// it with emax^2, src/Impedance.cpp:329-336).
__device__ __forceinline__ double dist2_rn(const double *a, const double *b) {
  double x = __dsub_rn(a[0], b[0]), y = __dsub_rn(a[1], b[1]), z = __dsub_rn(a[2], b[2]);
  return __dadd_rn(__dadd_rn(__dmul_rn(x, x), __dmul_rn(y, y)), __dmul_rn(z, z));
}

__device__ __forceinline__ void store_block(HalfPairBlock *H, int ntr, int i, int a, int j, int b, z1 cL, z1 cK) {
  double2 *p = reinterpret_cast<double2 *>(&H[(size_t)j * ntr + i].v[(a * 2 + b) * 4]);
  p[0] = make_double2(cL.r, cL.i);
  p[1] = make_double2(cK.r, cK.i);
}

// Double-float fill: the block holds each value as a float pair (hi, lo) in
// its 8-byte slot; the gather widens hi + lo (exact in FP64).
__device__ __forceinline__ void store_block_df(HalfPairBlock *H, int ntr, int i, int a, int j, int b, df Lr, df Li,
                                               df Kr, df Ki) {
  float4 *p = reinterpret_cast<float4 *>(&H[(size_t)j * ntr + i].v[(a * 2 + b) * 4]);
  p[0] = make_float4(Lr.hi, Lr.lo, Li.hi, Li.lo);
  p[1] = make_float4(Kr.hi, Kr.lo, Ki.hi, Ki.lo);
}

// Scatter coefficient of src/Impedance.cpp:372-375.
__device__ __forceinline__ double scatter_coef(const TriRec &T, int i, const TriRec &S, int j) {
  double c = BEM_ONEOVER4PI * T.helen[i] * S.helen[j];
  return (T.hneg[i] != S.hneg[j]) ? -c : c;
}

// What a far pair reads of a triangle in double-float, built once per fill.
struct TriDF {
  float p0[3][2];              // df frame origin (first half-RWG's free vertex)
  float v01[3][2], v02[3][2];  // df edge vectors of the first half-RWG's frame
  float hs[3][2];              // df helen[i] / sqrt(4 pi)
};

// The records of every tree of a group of fills in one launch: task i's test
// triangles at TD, its source triangles at SD (the same records when both
// trees are one).
struct TriDFJob {
  const TriRec *R;
  TriDF *D;
  int n;
};

__global__ void tri_df_kernel(const TriDFJob *__restrict__ jobs) {
  const TriDFJob jb = jobs[blockIdx.y];
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < jb.n; i += gridDim.x * blockDim.x) {
    const TriRec &T = jb.R[i];
    TriDF o;
    const double sc = sqrt(BEM_ONEOVER4PI);
    for (int c = 0; c < 3; c++) {
      const df a = df_make(T.v01[c]), b = df_make(T.v02[c]), p = df_make(T.p0[c]);
      o.p0[c][0] = p.hi; o.p0[c][1] = p.lo;
      o.v01[c][0] = a.hi; o.v01[c][1] = a.lo;
      o.v02[c][0] = b.hi; o.v02[c][1] = b.lo;
    }
    for (int h = 0; h < 3; h++) {
      const df l = df_make(h < T.nh ? T.helen[h] * sc : 0.0);
      o.hs[h][0] = l.hi; o.hs[h][1] = l.lo;
    }
    jb.D[i] = o;
  }
}

// Green's function constants in the fill's number type.
template <typename T>
struct GreenT {
  T ikr, iki, k2r, k2i, ksqr, ksqi;
};
template <typename T>
__device__ __forceinline__ GreenT<T> green_of(const GreenDev &g);
template <>
__device__ __forceinline__ GreenT<double> green_of<double>(const GreenDev &g) {
  return {g.ikr, g.iki, g.k2r, g.k2i, g.ksqr, g.ksqi};
}
template <>
__device__ __forceinline__ GreenT<df> green_of<df>(const GreenDev &g) {
  return {{g.ikr_f[0], g.ikr_f[1]}, {g.iki_f[0], g.iki_f[1]}, {g.k2r_f[0], g.k2r_f[1]},
          {g.k2i_f[0], g.k2i_f[1]}, {g.ksqr_f[0], g.ksqr_f[1]}, {g.ksqi_f[0], g.ksqi_f[1]}};
}

// (er, ei) = e^{ikR} and (ur, ui) = e^{ikR} (1 - ikR).  REALK: a lossless
// medium (ik imaginary), whose e^{ikR} has modulus one.  em: Im e^{ikR}, in
// double-float less Im(ik) R.
//
// The double-float fill keeps Im g = Im e^{ikR}/R less its constant Im(ik).  An
// RWG pair is the signed sum of four half-pair terms in which that constant's
// share of -U0 cancels exactly, while what is left is only ~(kR)^2/6 of it: the
// sum keeps as many more digits.  These decide the (small) dissipation that an
// ill-conditioned solve rests on.  What each rule's weights leave of the
// constant (their sum is 1 to ~1e-13) stays.
template <typename T, bool REALK>
__device__ __forceinline__ void wave_at(const GreenT<T> &g, T R, T &er, T &ei, T &em, T &ur, T &ui) {
  typedef Num<T> N;
  const T th = g.iki * R;
  N::sincos_(th, ei, er, em);
  if (REALK) {
    ur = N::muladd(ei, th, er);
    ui = N::muladd(-er, th, ei);
    return;
  }
  const T a = g.ikr * R;
  if (N::LESS && N::head(a) < -85) {  // double-float, below FP32's range: e^-85 of the neighbouring nodes' size
    er = ei = ur = ui = N::of(0.0);
    em = -th;
    return;
  }
  T m1;
  const T m = N::exp_(a, m1);
  er = m * er;
  ei = m * ei;
  em = N::LESS ? N::dot2(m, em, th, m1) : ei;
  const T om = N::of(1.0) - a;
  ur = N::dot2(er, om, ei, th);
  ui = N::dot2(ei, om, -er, th);
}

// scalar_gradient, src/GreensFunction.cpp:41-52, at the (unnormalized)
// difference x: f = {Re g, Im g (less Im(ik), see wave_at), Re q, Im q}.
template <typename T, bool REALK>
__device__ __forceinline__ void far_values(const GreenT<T> &g, V3<T> x, T (&f)[4]) {
  typedef Num<T> N;
  T R, Ri, er, ei, em, ur, ui;
  N::sqrt_rcp(N::sumsq(x.x, x.y, x.z), R, Ri);
  wave_at<T, REALK>(g, R, er, ei, em, ur, ui);
  f[0] = er * Ri;
  f[1] = em * Ri;
  const T Ri3 = Ri * (Ri * Ri);
  f[2] = ur * Ri3;
  f[3] = ui * Ri3;
}

// A far pair's triangles: origins' difference and edge vectors.
template <typename T>
struct FarGeom {
  V3<T> D0;      // P_t - P_s
  V3<T> a1, a2;  // test edges v01, v02
  V3<T> c1, c2;  // source edges v01, v02
};
template <typename T>
__device__ __forceinline__ FarGeom<T> far_geom(const TriRec &T_, const TriRec &S, const TriDF *TD, const TriDF *SD);
template <>
__device__ __forceinline__ FarGeom<double> far_geom<double>(const TriRec &T_, const TriRec &S, const TriDF *,
                                                            const TriDF *) {
  auto v = [](const double *p) { return V3<double>{p[0], p[1], p[2]}; };
  return {v(T_.p0) - v(S.p0), v(T_.v01), v(T_.v02), v(S.v01), v(S.v02)};
}
template <>
__device__ __forceinline__ FarGeom<df> far_geom<df>(const TriRec &, const TriRec &, const TriDF *TD, const TriDF *SD) {
  auto v = [](const float (*p)[2]) { return V3<df>{{p[0][0], p[0][1]}, {p[1][0], p[1][1]}, {p[2][0], p[2][1]}}; };
  return {v(TD->p0) - v(SD->p0), v(TD->v01), v(TD->v02), v(SD->v01), v(SD->v02)};
}

// Moments of a far pair with the 6-point rule, by one thread:
// M[(c * 3 + a) * 3 + b] = sum_qu w_q w_u eta^a xi^b f_c.  rho: the outer
// nodes relative to P_t (shared memory: the warp has one test triangle).
template <typename T, bool REALK>
__device__ __forceinline__ void far_moments6(const FarGeom<T> &ge, const GreenT<T> &g, const V3<T> *rho, T (&M)[36]) {
  typedef Num<T> N;
#pragma unroll
  for (int k = 0; k < 36; k++) M[k] = N::of(0.0);
#pragma unroll 1
  for (int u = 0; u < 6; u++) {
    const RuleNode<T> nu = far_node<T>(NODES6 + u);
    const V3<T> base = ge.D0 - (nu.x1 * ge.c1 + nu.x2 * ge.c2);
    T S[12];
#pragma unroll
    for (int k = 0; k < 12; k++) S[k] = N::of(0.0);
#pragma unroll 1
    for (int q = 0; q < 6; q++) {
      const V3<T> r = rho[q];
      const V3<T> x = {N::diff(base.x, -r.x), N::diff(base.y, -r.y), N::diff(base.z, -r.z)};
      T f[4];
      far_values<T, REALK>(g, x, f);
      const RuleNode<T> nq = far_node<T>(NODES6 + q);
#pragma unroll
      for (int c = 0; c < 4; c++) {
        N::mac(S[c * 3 + 0], f[c], nq.w);
        N::mac(S[c * 3 + 1], f[c], nq.w1);
        N::mac(S[c * 3 + 2], f[c], nq.w2);
      }
    }
#pragma unroll
    for (int k = 0; k < 12; k++) {
      const T v = N::fin(S[k]);
      N::mac(M[k * 3 + 0], v, nu.w);
      N::mac(M[k * 3 + 1], v, nu.w1);
      N::mac(M[k * 3 + 2], v, nu.w2);
    }
  }
#pragma unroll
  for (int k = 0; k < 36; k++) M[k] = N::fin(M[k]);
}

// The same with an nr-point rule (first node off), by one warp: the lanes take
// (outer node, run of inner nodes) pieces.  rt, rs: the warp's staging of the
// pair's outer nodes (relative to P_s) and inner nodes.  The sums land in out[36].
template <typename T>
struct FarStage {
  V3<T> p[36];
  T w[36][3];
};
template <typename T, bool REALK>
__device__ __forceinline__ void far_moments_warp(const FarGeom<T> &ge, const GreenT<T> &g, int off, int nr,
                                                 FarStage<T> *st, FarStage<T> *ss, T *out, int lane) {
  typedef Num<T> N;
  for (int k = lane; k < nr; k += 32) {
    const RuleNode<T> n = far_node<T>(off + k);
    st->p[k] = ge.D0 + (n.x1 * ge.a1 + n.x2 * ge.a2);
    ss->p[k] = n.x1 * ge.c1 + n.x2 * ge.c2;
    st->w[k][0] = ss->w[k][0] = n.w;
    st->w[k][1] = ss->w[k][1] = n.w1;
    st->w[k][2] = ss->w[k][2] = n.w2;
  }
  __syncwarp();
  T M[40];
#pragma unroll
  for (int k = 0; k < 40; k++) M[k] = N::of(0.0);
  const int pieces = (nr + 8) / 9, run = (nr + pieces - 1) / pieces;
#pragma unroll 1
  for (int it = lane; it < nr * pieces; it += 32) {
    const int q = it / pieces, u0 = (it - q * pieces) * run, u1 = min(nr, u0 + run);
    const V3<T> r = st->p[q];
    T S[12];
#pragma unroll
    for (int k = 0; k < 12; k++) S[k] = N::of(0.0);
#pragma unroll 1
    for (int u = u0; u < u1; u++) {
      const V3<T> l = ss->p[u];
      const V3<T> x = {N::diff(r.x, l.x), N::diff(r.y, l.y), N::diff(r.z, l.z)};
      T f[4];
      far_values<T, REALK>(g, x, f);
#pragma unroll
      for (int c = 0; c < 4; c++)
#pragma unroll
        for (int b = 0; b < 3; b++) N::mac(S[c * 3 + b], f[c], ss->w[u][b]);
    }
#pragma unroll
    for (int c = 0; c < 4; c++)
#pragma unroll
      for (int b = 0; b < 3; b++) {
        const T v = N::fin(S[c * 3 + b]);
#pragma unroll
        for (int a = 0; a < 3; a++) N::mac(M[(c * 3 + a) * 3 + b], v, st->w[q][a]);
      }
  }
  const int at = reduce8_index(lane);
#pragma unroll
  for (int k = 0; k < 5; k++) {
    T v[8];
#pragma unroll
    for (int j = 0; j < 8; j++) v[j] = N::fin(M[k * 8 + j]);
    const T r = reduce8<T>(v, lane);
    if ((lane & 3) == 0 && k * 8 + at < 36) out[k * 8 + at] = r;
  }
  __syncwarp();
}

// Scatter coefficient of src/Impedance.cpp:372-375 in the fill's number type.
template <typename T>
__device__ __forceinline__ T scatter_coef_t(const TriRec &T_, const TriDF *TD, int i, const TriRec &S, const TriDF *SD,
                                            int j);
template <>
__device__ __forceinline__ double scatter_coef_t<double>(const TriRec &T_, const TriDF *, int i, const TriRec &S,
                                                         const TriDF *, int j) {
  return scatter_coef(T_, i, S, j);
}
template <>
__device__ __forceinline__ df scatter_coef_t<df>(const TriRec &T_, const TriDF *TD, int i, const TriRec &S,
                                                 const TriDF *SD, int j) {
  const df c = df_mul({TD->hs[i][0], TD->hs[i][1]}, {SD->hs[j][0], SD->hs[j][1]});
  return T_.hneg[i] != S.hneg[j] ? df_neg(c) : c;
}
__device__ __forceinline__ void store_pair(HalfPairBlock *H, int ntr, int i, int a, int j, int b, C1<double> L,
                                           C1<double> K) {
  store_block(H, ntr, i, a, j, b, {L.r, L.i}, {K.r, K.i});
}
__device__ __forceinline__ void store_pair(HalfPairBlock *H, int ntr, int i, int a, int j, int b, C1<df> L, C1<df> K) {
  store_block_df(H, ntr, i, a, j, b, L.r, L.i, K.r, K.i);
}

// The nine (c L_ij, c K_ij) of a far pair from its moments.
//
// The half-RWGs' free vertices are the triangles' vertices P_v, S_w, so with
// the edges a_1, a_2 of the test and c_1, c_2 of the source triangle from P_0
// and S_0, phi_i = (rho - e_i)/2 and e_i in {0, a_1, a_2}:
//   L_vw = k^2/4 sum_{ab} (a_a . c_b) [G_ab - [b=w] G_a0 - [a=v] G_0b + [a=v][b=w] G_00] - G_00
// (a, b = 1, 2), G the moments of g.  In barycentric moments B of q,
// phi_i . ((r_t - r_s) x phi_j) expands to the six-fold volumes of the
// tetrahedra on an edge of each triangle:
//   K_vw = -1/4 sum_{v' != v, w' != w} B_v'w' (P_v - S_w) . ((S_w' - S_w) x (P_v' - P_v)),
// nine volumes for the nine edge pairs (src/Impedance.cpp:154-168 summed over
// the outer rule).  sum: the rule's, for the constant of Im g (wave_at).
// mirror: the pair's transposed place too.
template <typename T, bool REALK>
__device__ __noinline__ void far_contract(const TriRec &T_, const TriRec &S, const TriDF *TD, const TriDF *SD,
                                          const GreenT<T> &g, const T *M, int sum, HalfPairBlock *H, int ntr, bool mirror) {
  typedef Num<T> N;
  const FarGeom<T> ge = far_geom<T>(T_, S, TD, SD);
  const V3<T> a[2] = {ge.a1, ge.a2}, cs[2] = {ge.c1, ge.c2};
  // L's brackets
  C1<T> G[3][3];
#pragma unroll
  for (int x = 0; x < 3; x++)
#pragma unroll
    for (int y = 0; y < 3; y++) G[x][y] = {M[x * 3 + y], M[9 + x * 3 + y]};
  C1<T> U0 = G[0][0];
  if (N::LESS) {
    U0.i = U0.i + g.iki * N::of(c_sums[sum].ww1);
#pragma unroll
    for (int x = 0; x < 3; x++) {
      const T kw = g.iki * N::of(c_sums[sum].w[x]);
#pragma unroll
      for (int y = 0; y < 3; y++) G[x][y].i = N::muladd(kw, N::of(c_sums[sum].w[y]), G[x][y].i);
    }
  }
  C1<T> br[3][3];
  {
    C1<T> U1 = {N::of(0.0), N::of(0.0)}, dU2[2] = {U1, U1}, eU3[2] = {U1, U1}, ed[2][2];
#pragma unroll
    for (int x = 0; x < 2; x++)
#pragma unroll
      for (int y = 0; y < 2; y++) {
        const T d = vdot(a[x], cs[y]);
        U1 = U1 + d * G[x + 1][y + 1];
        dU2[y] = dU2[y] + d * G[x + 1][0];
        eU3[x] = eU3[x] + d * G[0][y + 1];
        ed[x][y] = d * G[0][0];
      }
    br[0][0] = U1;
#pragma unroll
    for (int x = 0; x < 2; x++) {
      br[0][x + 1] = U1 - dU2[x];
      br[x + 1][0] = U1 - eU3[x];
    }
#pragma unroll
    for (int x = 0; x < 2; x++)
#pragma unroll
      for (int y = 0; y < 2; y++) br[x + 1][y + 1] = (br[0][y + 1] - eU3[x]) + ed[x][y];
  }
  // barycentric moments of q
  C1<T> B[3][3];
#pragma unroll
  for (int x = 0; x < 3; x++)
#pragma unroll
    for (int y = 0; y < 3; y++) B[x][y] = {M[18 + x * 3 + y], M[27 + x * 3 + y]};
#pragma unroll
  for (int y = 0; y < 3; y++) B[0][y] = (B[0][y] - B[1][y]) - B[2][y];
#pragma unroll
  for (int x = 0; x < 3; x++) B[x][0] = (B[x][0] - B[x][1]) - B[x][2];
  // volumes of the edge pairs (edges 01, 02, 12 of each triangle)
  T V[3][3];
  {
    const V3<T> C00 = vcross(cs[0], a[0]), C01 = vcross(cs[0], a[1]), C10 = vcross(cs[1], a[0]),
                C11 = vcross(cs[1], a[1]);  // C_xy = c_x x a_y
    V[0][0] = vdot(ge.D0, C00);
    V[0][1] = vdot(ge.D0, C10);
    V[1][0] = vdot(ge.D0, C01);
    V[1][1] = vdot(ge.D0, C11);
    const T a01 = vdot(a[0], C01), a11 = vdot(a[0], C11);    // a_1 . (c_x x a_2)
    const T c10 = vdot(cs[0], C10), c11 = vdot(cs[0], C11);  // c_1 . (c_2 x a_y)
    V[2][0] = (V[1][0] - V[0][0]) + a01;
    V[2][1] = (V[1][1] - V[0][1]) + a11;
    V[0][2] = (V[0][1] - V[0][0]) - c10;
    V[1][2] = (V[1][1] - V[1][0]) - c11;
    V[2][2] = ((V[1][1] - V[0][1]) - (V[1][0] - V[0][0])) + ((a11 - a01) - (c11 - c10));
  }
  const T ksr = N::pow2(g.ksqr, 0.25f), ksi = N::pow2(g.ksqi, 0.25f);
  int at[3], as[3];  // the halves (bits) whose free vertex is v
#pragma unroll
  for (int v = 0; v < 3; v++) {
    at[v] = as[v] = 0;
#pragma unroll
    for (int h = 0; h < 3; h++) {
      at[v] |= (h < T_.nh && ((T_.hvert >> (2 * h)) & 3) == v) ? 1 << h : 0;
      as[v] |= (h < S.nh && ((S.hvert >> (2 * h)) & 3) == v) ? 1 << h : 0;
    }
  }
#pragma unroll
  for (int v = 0; v < 3; v++)
#pragma unroll
    for (int w = 0; w < 3; w++) {
      C1<T> K = {N::of(0.0), N::of(0.0)};
#pragma unroll
      for (int x = 0; x < 3; x++)
#pragma unroll
        for (int y = 0; y < 3; y++) {
          if (x == v || y == w) continue;
          const T vol = V[v + x - 1][w + y - 1];  // edge {v, x} -> 01: 0, 02: 1, 12: 2
          const bool minus = (v > x) != (w > y);
          N::mac(K.r, B[x][y].r, minus ? vol : -vol);
          N::mac(K.i, B[x][y].i, minus ? vol : -vol);
        }
      K = {N::pow2(N::fin(K.r), 0.25f), N::pow2(N::fin(K.i), 0.25f)};
      C1<T> L;
      if (REALK)
        L = {N::muladd(ksr, br[v][w].r, -U0.r), N::muladd(ksr, br[v][w].i, -U0.i)};
      else
        L = cmul(C1<T>{ksr, ksi}, br[v][w]) - U0;
      for (int hi = at[v]; hi; hi &= hi - 1)
        for (int hj = as[w]; hj; hj &= hj - 1) {
          const int i = __ffs(hi) - 1, j = __ffs(hj) - 1;
          const T c = scatter_coef_t<T>(T_, TD, i, S, SD, j);
          const C1<T> cL = c * L, cK = c * K;
          store_pair(H, ntr, T_.hrwg[i], T_.hneg[i], S.hrwg[j], S.hneg[j], cL, cK);
          if (mirror) store_pair(H, ntr, S.hrwg[j], S.hneg[j], T_.hrwg[i], T_.hneg[i], cL, cK);
        }
    }
}

// ---------------- far pairs in FP32 (mixed precision) ----------------
//
// Closed form of the nine products from outer moments.  With P_t, P_s the frame
// origins (p0 of t[0], s[0]), rho = r_t - P_t, l = r_s - P_s, e_i = p0_i - P_t,
// d_j = p0_j - P_s, D_ij = p0_i - p0_j, the inner moments I0 = sum w g,
// A = sum w g l, Q0 = sum w q, Q1 = sum w q l and the outer ones U0 = sum w I0,
// U1 = sum w rho.A, U2 = sum w I0 rho, U3 = sum w A, V0 = sum w Q0,
// V1 = sum w Q1 x rho, V2 = sum w Q1, V3 = sum w Q0 rho:
//   L_ij = k^2/4 [U1 - d_j.U2 - e_i.U3 + (e_i.d_j) U0] - U0
//   K_ij = -1/4 D_ij . [V1 - V2 x e_i - d_j x V3 + V0 (d_j x e_i)]
// which is LKFarOuterIntegrand (src/Impedance.cpp:154-168) summed over the
// outer rule, here in FP32 with a pair-centred
// distance: r_t - r_s = D0 + u, D0 = P_t - P_s (FP64 once per pair), u = rho - l
// (small, FP32).  R = R0 + dR with R0 = |D0| in FP64 and
// dR = (2 D0.u + u.u) / (R0 + R) in FP32, so the phase k R is k R0 reduced
// modulo 2 pi in FP64 once per pair plus k dR in FP32; the relative error of
// every node's e^{ikR}/R stays near FP32 rounding at any distance.
struct f3 {
  float x, y, z;
};
struct c1 {
  float r, i;
};
struct c3 {
  c1 x, y, z;
};
__device__ __forceinline__ f3 f3of(d3 a) { return {(float)a.x, (float)a.y, (float)a.z}; }
__device__ __forceinline__ f3 operator+(f3 a, f3 b) { return {a.x + b.x, a.y + b.y, a.z + b.z}; }
__device__ __forceinline__ f3 operator-(f3 a, f3 b) { return {a.x - b.x, a.y - b.y, a.z - b.z}; }
__device__ __forceinline__ f3 operator*(float c, f3 a) { return {c * a.x, c * a.y, c * a.z}; }
__device__ __forceinline__ float fdot(f3 a, f3 b) { return a.x * b.x + a.y * b.y + a.z * b.z; }
__device__ __forceinline__ f3 fcross(f3 a, f3 b) {
  return {a.y * b.z - a.z * b.y, a.z * b.x - a.x * b.z, a.x * b.y - a.y * b.x};
}
__device__ __forceinline__ c1 cmulf(c1 a, c1 b) { return {a.r * b.r - a.i * b.i, a.r * b.i + a.i * b.r}; }
__device__ __forceinline__ c1 csubf(c1 a, c1 b) { return {a.r - b.r, a.i - b.i}; }
__device__ __forceinline__ c1 cscalef(float c, c1 a) { return {c * a.r, c * a.i}; }
__device__ __forceinline__ void caccf(c1 &a, c1 b) { a.r += b.r; a.i += b.i; }
__device__ __forceinline__ c3 c3zerof() { return {{0, 0}, {0, 0}, {0, 0}}; }
__device__ __forceinline__ c3 cs_vf(c1 c, f3 v) { return {{c.r * v.x, c.i * v.x}, {c.r * v.y, c.i * v.y}, {c.r * v.z, c.i * v.z}}; }
__device__ __forceinline__ void c3accf(c3 &a, c3 b) {
  caccf(a.x, b.x); caccf(a.y, b.y); caccf(a.z, b.z);
}
__device__ __forceinline__ c3 c3scalef(float c, c3 a) { return {cscalef(c, a.x), cscalef(c, a.y), cscalef(c, a.z)}; }
__device__ __forceinline__ c3 c3subf(c3 a, c3 b) { return {csubf(a.x, b.x), csubf(a.y, b.y), csubf(a.z, b.z)}; }
__device__ __forceinline__ c1 rdotf(f3 a, c3 b) {
  return {a.x * b.x.r + a.y * b.y.r + a.z * b.z.r, a.x * b.x.i + a.y * b.y.i + a.z * b.z.i};
}
__device__ __forceinline__ c3 zcrossf(c3 a, f3 b) {
  return {{a.y.r * b.z - a.z.r * b.y, a.y.i * b.z - a.z.i * b.y},
          {a.z.r * b.x - a.x.r * b.z, a.z.i * b.x - a.x.i * b.z},
          {a.x.r * b.y - a.y.r * b.x, a.x.i * b.y - a.y.i * b.x}};
}
__device__ __forceinline__ c3 rcrossf(f3 a, c3 b) {
  return {{a.y * b.z.r - a.z * b.y.r, a.y * b.z.i - a.z * b.y.i},
          {a.z * b.x.r - a.x * b.z.r, a.z * b.x.i - a.x * b.z.i},
          {a.x * b.y.r - a.y * b.x.r, a.x * b.y.i - a.y * b.x.i}};
}

__device__ __noinline__ void far_pair_fp32(const TriRec &T, const TriRec &S, const GreenDev &g,
                                           const double (*rule)[3], int nr, HalfPairBlock *H, int ntr) {
  const d3 Pt = ld3(T.p0), Ps = ld3(S.p0);
  const d3 D0d = Pt - Ps;
  const double R0d = sqrt(dot(D0d, D0d));
  // per-pair FP64: magnitude and phase of e^{ik R0}
  const double ph0d = g.iki * R0d;
  const double ph0r = ph0d - 6.283185307179586476925286766559 * rint(ph0d * 0.15915494309189533576888376337251);
  const float ph0 = (float)ph0r;
  const float m0 = (float)exp(g.ikr * R0d);
  const float R0 = (float)R0d, R0sq = (float)(R0d * R0d);
  const f3 D0 = f3of(D0d);
  const float ikr = (float)g.ikr, iki = (float)g.iki;
  const f3 v01t = f3of(ld3(T.v01)), v02t = f3of(ld3(T.v02)), v01s = f3of(ld3(S.v01)), v02s = f3of(ld3(S.v02));
  c1 U0 = {0, 0}, U1 = {0, 0}, V0 = {0, 0};
  c3 U2 = c3zerof(), U3 = c3zerof(), V1 = c3zerof(), V2 = c3zerof(), V3 = c3zerof();
  for (int q = 0; q < nr; q++) {
    const float a = (float)rule[q][0], b = (float)rule[q][1], w = (float)rule[q][2];
    const f3 rho = a * v01t + b * v02t;
    c1 I0 = {0, 0}, Q0 = {0, 0};
    c3 A = c3zerof(), Q1 = c3zerof();
    for (int uix = 0; uix < nr; uix++) {
      const float as = (float)rule[uix][0], bs = (float)rule[uix][1], ws = (float)rule[uix][2];
      const f3 l = as * v01s + bs * v02s;
      const f3 u = rho - l;
      const float sdel = 2.0f * fdot(D0, u) + fdot(u, u);
      const float Rf = sqrtf(R0sq + sdel);
      const float dR = sdel / (R0 + Rf);
      const float R = R0 + dR;
      float sn, cs;
      sincosf(ph0 + iki * dR, &sn, &cs);
      const float mag = m0 * expf(ikr * dR);
      const float Ri = 1.0f / R;
      const c1 gs = {mag * cs * Ri, mag * sn * Ri};
      const c1 one_m_ikR = {1.0f - ikr * R, -iki * R};
      const c1 qq = cscalef(Ri * Ri, cmulf(gs, one_m_ikR));
      const c1 gw = cscalef(ws, gs), qw = cscalef(ws, qq);
      caccf(I0, gw);
      c3accf(A, cs_vf(gw, l));
      caccf(Q0, qw);
      c3accf(Q1, cs_vf(qw, l));
    }
    caccf(U0, cscalef(w, I0));
    caccf(U1, cscalef(w, rdotf(rho, A)));
    c3accf(U2, cs_vf(cscalef(w, I0), rho));
    c3accf(U3, c3scalef(w, A));
    caccf(V0, cscalef(w, Q0));
    c3accf(V1, c3scalef(w, zcrossf(Q1, rho)));
    c3accf(V2, c3scalef(w, Q1));
    c3accf(V3, cs_vf(cscalef(w, Q0), rho));
  }
  const c1 ksq = {(float)g.ksqr, (float)g.ksqi};
  for (int i = 0; i < T.nh; i++) {
    const f3 ei = f3of(ld3(T.hp0[i]) - Pt);
    for (int j = 0; j < S.nh; j++) {
      const f3 dj = f3of(ld3(S.hp0[j]) - Ps);
      const f3 D = (D0 + ei) - dj;
      c1 bracket = csubf(csubf(U1, rdotf(dj, U2)), rdotf(ei, U3));
      caccf(bracket, cscalef(fdot(ei, dj), U0));
      const c1 L = csubf(cscalef(0.25f, cmulf(ksq, bracket)), U0);
      c3 X = c3subf(c3subf(V1, zcrossf(V2, ei)), rcrossf(dj, V3));
      c3accf(X, cs_vf(V0, fcross(dj, ei)));
      const c1 K = cscalef(-0.25f, rdotf(D, X));
      const double c = scatter_coef(T, i, S, j);
      store_block(H, ntr, T.hrwg[i], T.hneg[i], S.hrwg[j], S.hneg[j], z1{c * L.r, c * L.i}, z1{c * K.r, c * K.i});
    }
  }
}

// The far pairs of one fill of a group launch: Zts(t, s, g) into the half-pair
// blocks H, with its share of the group's far tiles (prefix offset).
struct FillTask {
  const TriRec *T, *S;       // test and source trees' records
  const TriDF *TD, *SD;      // their double-float records (double-float mode), else null
  HalfPairBlock *H;          // this fill's half-pair blocks
  int64_t far0;              // first far tile of the group that is this task's
  int ntT, ntS, ntr, far_tx; // triangles of t and s, RWGs of t, far tiles along s
  int sym;                   // t is s: each unordered far pair is integrated once
  GreenDev g;
};

__device__ __forceinline__ int task_of_far(const FillTask *tk, int n, int64_t u) {
  int i = n - 1;
  while (i > 0 && u < tk[i].far0) i--;
  return i;
}

// Far tiles of one fill: 32 source x rows test triangles each; a symmetric
// fill has those of the lower-triangular 32 x 32 blocks only.
int64_t far_tiles_of(bool sym, int ntT, int ntS, int rows) {
  if (!sym) return (int64_t)((ntS + 31) / 32) * ((ntT + rows - 1) / rows);
  const int64_t nb = (ntT + 31) / 32;
  return nb * (nb + 1) / 2 * (32 / rows);
}

// The first test triangle and the first source triangle of a far tile.
__device__ __forceinline__ void far_tile_at(const FillTask &tk, int64_t local, int rows, int &ta0, int &sb0) {
  if (!tk.sym) {
    sb0 = (int)(local % tk.far_tx) * 32;
    ta0 = (int)(local / tk.far_tx) * rows;
    return;
  }
  const int sub = 32 / rows;
  const int64_t m = local / sub;  // block number: row r holds blocks r (r + 1) / 2 ...
  int64_t r = (int64_t)((sqrt(8.0 * (double)m + 1.0) - 1.0) * 0.5);
  while (r * (r + 1) / 2 > m) r--;
  while ((r + 1) * (r + 2) / 2 <= m) r++;
  ta0 = (int)r * 32 + (int)(local - m * sub) * rows;
  sb0 = (int)(m - r * (r + 1) / 2) * 32;
}

// A group of fills in one launch (the three Zts of a solve, or of several
// requests): CTA b takes far tile b of the task whose range holds it, lane =
// source triangle, warp = test triangle.  MODE FILL_FP32_FAR: pairs whose
// centroid distance exceeds 3 edge lengths (the longer of the two triangles'
// longest edges) in FP32, every ordered pair by itself; the others, and every
// pair of the other modes, in FP64 (FILL_FP64, FILL_FP32_FAR) or double-float.
//
// A pair with the 6-point rule is one thread's; the others (triangles that
// face each other across a gap narrower than their edges: 1296 node pairs
// against 36) are listed in shared memory and taken by whole warps, so that
// one such pair does not hold its warp's other 31 lanes.
//
// Bound by FP32 issue (double-float) or by the FP64 pipe.  The chains of one
// node pair are long, so resident warps count: 168 registers (12 warps an SM)
// against the 206 the compiler takes by itself (8) gave 6.1 -> 4.6 ms; two or
// three nodes in flight per thread, or 128 registers with spills, were slower.
// The three fills of a solve, before (every ordered pair, Cartesian moments,
// normalized sums, one thread for every rule) and now: icospheres at N = 7680
// 16.9 -> 4.6 ms, slabs 50 nm apart at N = 11520 43.7 -> 10.9 ms, cubes at
// N = 288 1.08 -> 0.11 ms; in FP64 cubes at N = 1152 6.3 -> 0.87 ms.
constexpr int FAR_BATCH = 32;  // listed pairs whose moments are held at once

template <int MODE>
__global__ void __maxnreg__(168) far_pairs_group_kernel(const FillTask *__restrict__ tasks, int ntask,
                                                              FarOpts o) {
  typedef typename std::conditional<MODE == FILL_DF, df, double>::type T;
  __shared__ GreenDev s_g;
  __shared__ V3<T> s_rho[8][6];
  __shared__ FarStage<T> s_st[8], s_ss[8];
  __shared__ T s_mom[FAR_BATCH][36];
  __shared__ int2 s_list[256];
  __shared__ int s_rule[256], s_n;
  const int lane = threadIdx.x, wid = threadIdx.y, rows = blockDim.y;
  const int ti = task_of_far(tasks, ntask, blockIdx.x);
  const FillTask &tk = tasks[ti];
  if (lane == 0 && wid == 0) {
    s_g = tk.g;
    s_n = 0;
  }
  int ta0, sb0;
  far_tile_at(tk, (int64_t)blockIdx.x - tk.far0, rows, ta0, sb0);
  const int ta = ta0 + wid, sb = sb0 + lane;
  const bool sym = MODE != FILL_FP32_FAR && tk.sym;
  if (lane < 6 && ta < tk.ntT) {
    const TriDF *TD = tk.TD ? tk.TD + ta : nullptr;
    const FarGeom<T> ge = far_geom<T>(tk.T[ta], tk.T[ta], TD, TD);
    const RuleNode<T> n = far_node<T>(NODES6 + lane);
    s_rho[wid][lane] = n.x1 * ge.a1 + n.x2 * ge.a2;
  }
  __syncthreads();
  const GreenT<T> g = green_of<T>(s_g);
  const bool realk = s_g.ikr == 0.0 && s_g.ksqi == 0.0;
  if (ta < tk.ntT && sb < tk.ntS && (!sym || ta > sb)) {
    const TriRec &Tr = tk.T[ta];
    const TriRec &Sr = tk.S[sb];
    if (Tr.gid != Sr.gid && !shares_vertex(Tr.vid, Sr.vid)) {  // else the near kernel's
      // far-rule choice, src/Impedance.cpp:329-360
      const double d = dist2_rn(Tr.c, Sr.c);
      const double e = fmax(Tr.emax, Sr.emax);
      const double emax2 = __dmul_rn(e, e);
      const int rule = __dmul_rn(d, o.th6) > emax2    ? 6
                       : __dmul_rn(d, o.th10) > emax2 ? 10
                       : __dmul_rn(d, o.th15) > emax2 ? 15
                       : __dmul_rn(d, o.th21) > emax2 ? 21
                                                      : 36;
      if (MODE == FILL_FP32_FAR && d > 9.0 * emax2) {
        // beyond 3 edge lengths every default threshold selects the 6-point
        // rule; the others serve non-default Options
        const double(*nodes)[3] = rule == 6 ? c_rule6 : rule == 10 ? c_rule10 : rule == 15 ? c_rule15
                                  : rule == 21 ? c_rule21 : c_rule36;
        far_pair_fp32(Tr, Sr, s_g, nodes, rule, tk.H, tk.ntr);
      } else if (rule == 6) {
        const TriDF *TD = tk.TD ? tk.TD + ta : nullptr, *SD = tk.SD ? tk.SD + sb : nullptr;
        T M[36];
        const FarGeom<T> ge = far_geom<T>(Tr, Sr, TD, SD);
        if (realk) {
          far_moments6<T, true>(ge, g, s_rho[wid], M);
          T Mc[36];
#pragma unroll
          for (int k = 0; k < 36; k++) Mc[k] = M[k];
          far_contract<T, true>(Tr, Sr, TD, SD, g, Mc, SUM6, tk.H, tk.ntr, sym);
        } else {
          far_moments6<T, false>(ge, g, s_rho[wid], M);
          T Mc[36];
#pragma unroll
          for (int k = 0; k < 36; k++) Mc[k] = M[k];
          far_contract<T, false>(Tr, Sr, TD, SD, g, Mc, SUM6, tk.H, tk.ntr, sym);
        }
      } else {
        const int at = atomicAdd(&s_n, 1);
        s_list[at] = make_int2(ta, sb);
        s_rule[at] = rule;
      }
    }
  }
  __syncthreads();
  const int n = s_n;
  for (int b = 0; b < n; b += FAR_BATCH) {
    const int m = min(FAR_BATCH, n - b);
    for (int k = wid; k < m; k += rows) {
      const int2 pr = s_list[b + k];
      const int nr = s_rule[b + k];
      const int off = nr == 10 ? NODES10 : nr == 15 ? NODES15 : nr == 21 ? NODES21 : NODES36;
      const FarGeom<T> ge = far_geom<T>(tk.T[pr.x], tk.S[pr.y], tk.TD ? tk.TD + pr.x : nullptr,
                                        tk.SD ? tk.SD + pr.y : nullptr);
      if (realk)
        far_moments_warp<T, true>(ge, g, off, nr, &s_st[wid], &s_ss[wid], s_mom[k], lane);
      else
        far_moments_warp<T, false>(ge, g, off, nr, &s_st[wid], &s_ss[wid], s_mom[k], lane);
    }
    __syncthreads();
    if (wid == 0 && lane < m) {
      const int2 pr = s_list[b + lane];
      const TriDF *TD = tk.TD ? tk.TD + pr.x : nullptr, *SD = tk.SD ? tk.SD + pr.y : nullptr;
      const int nr = s_rule[b + lane];
      const int sum = nr == 10 ? SUM10 : nr == 15 ? SUM15 : nr == 21 ? SUM21 : SUM36;
      if (realk)
        far_contract<T, true>(tk.T[pr.x], tk.S[pr.y], TD, SD, g, s_mom[lane], sum, tk.H, tk.ntr, sym);
      else
        far_contract<T, false>(tk.T[pr.x], tk.S[pr.y], TD, SD, g, s_mom[lane], sum, tk.H, tk.ntr, sym);
    }
    __syncthreads();
  }
}

void launch_far(int mode, unsigned tiles, int rows, cudaStream_t st, const FillTask *tasks, int ntask, FarOpts fo) {
  const dim3 blk(32, rows);
  if (mode == FILL_DF)
    far_pairs_group_kernel<FILL_DF><<<tiles, blk, 0, st>>>(tasks, ntask, fo);
  else if (mode == FILL_FP32_FAR)
    far_pairs_group_kernel<FILL_FP32_FAR><<<tiles, blk, 0, st>>>(tasks, ntask, fo);
  else
    far_pairs_group_kernel<FILL_FP64><<<tiles, blk, 0, st>>>(tasks, ntask, fo);
}

// ---------------- near pairs ----------------
//
// A near pair (same triangle, or a shared vertex) is the smooth inner rule (91
// source nodes at each of the 105 test nodes, LKSmoothInnerIntegrand,
// src/Impedance.cpp:93-105, with scalar_gradient_smooth,
// src/GreensFunction.cpp:54-69), the closed-form singular terms
// (EHNonSmoothIntegral, src/Source.cpp:16-86) at the test nodes, the close-pair
// contraction (src/Impedance.cpp:194-250) and, for neighbours, the edge
// correction of K (src/Impedance.cpp:301-324).  One warp takes one pair and
// reduces it to moments; the nine (i, j) products follow in closed form.
//
// Smooth part.  g~ = (e^{ikR} - 1)/R - k2 R and q~ = (e^{ikR}(1 - ikR) + k2 R^2
// - 1)/R^3 are power series in R without the terms that the singular part
// takes:
//   g~ = sum_{n>=1, n!=2} (ik)^n R^{n-1}/n!,   q~ = sum_{n>=3} (1-n)(ik)^n R^{n-3}/n!.
// Their moments over {1, eta1, eta2} x {1, xi1, xi2} (as a far pair's) are
// therefore sums over the moments of the powers of R alone, which are real and
// know no frequency and no medium:
//   odd powers R^{2j+1}: 91 x 105 node pairs;
//   even powers (R^2)^j: polynomials, which the rules integrate exactly up to
//   their degree, so that 36 x 36 nodes give the same sums (even_rules.h: their
//   weights carry the large rules' own moments).  The 36-point rule's degree is 13:
//   (R^2)^7 to (R^2)^9 of the FP64 series are off by up to 6e-7 of terms below 3e-12.
// So there is no sincos, exp or division per node pair, the cancellation in the
// closed forms of g~ and q~ is gone, and one pass over a pair serves the
// exterior and its body's interior Green's function at once.  The terms fall
// like x^n/n!, x = |k| R: the first powers are carried in full, those below
// 2^-24 of the singular part in FP32 (double-float fill).  Coordinates are
// scaled by a power of two so that R <= 1.
// Above x = 1.1 (coarse meshes at an interior resonance) g~ and q~ are evaluated
// directly per node pair (NEAR_DIRECT).
//
// Singular part: with X = IL1 + ISn1 rho' (rho' the test node's foot on the
// source plane) and its k2 counterpart, 23 real moments over the test nodes.
enum { NEAR_DIRECT = 0, NEAR_SERIES1 = 1, NEAR_SERIES2 = 2, NEAR_KINDS = 3 };
constexpr double NEAR_X1 = 0.47, NEAR_X2 = 1.1;  // largest |k| R of the two series kinds

// Powers carried: JF in full, JT in all (even powers 1..JT beside the constant).
// Double-float: at x = 0.47 the first FP32 term is x^8/8! = 6e-8 and the first
// dropped x^14/14! = 3e-16 of the singular part; at x = 1.1 6e-9 and 9e-16.
template <typename T, int KIND>
struct NearCfg;
template <>
struct NearCfg<df, NEAR_SERIES1> { static constexpr int JF = 3, JT = 6; };
template <>
struct NearCfg<df, NEAR_SERIES2> { static constexpr int JF = 5, JT = 8; };
template <>
struct NearCfg<double, NEAR_SERIES1> { static constexpr int JF = 7, JT = 7; };
template <>
struct NearCfg<double, NEAR_SERIES2> { static constexpr int JF = 9, JT = 9; };
template <typename T>
struct NearCfg<T, NEAR_DIRECT> { static constexpr int JF = 4, JT = 4; };  // the four values of g~ and q~
constexpr int NEAR_NJ = 10;  // coefficients kept per series

// One Green's function of a near task: where its products go, the source and
// test triangles it covers (all of the task's, or one body's of a two-body
// tree), and its series coefficients (complex, in the fill's number type).
struct NearGreen {
  HalfPairBlock *H;
  int ntr, rwg0;    // RWGs of its test tree; index of its first RWG in the task's tree
  int tri0, tri1;   // its triangles of the task's tree
  int realk;
  GreenDev g;
  // read 16 bytes at a time
  alignas(16) double ge[NEAR_NJ][2];
  alignas(16) double go[NEAR_NJ][2];
  alignas(16) double qe[NEAR_NJ][2];
  alignas(16) double qo[NEAR_NJ][2];
};
struct alignas(16) NearTask {
  const TriRec *T, *S;
  const NearPair *near;
  int64_t nnear, unit0;  // pairs; the task's first unit of the launch
  double scale;          // power of two: R scale <= 1
  int ngreen;            // the first covers every pair, the others one body's
  NearGreen g[3];
};
static_assert(sizeof(NearTask) % 16 == 0 && sizeof(NearGreen) % 16 == 0, "an array of tasks keeps their alignment");

// The rules of the near kernels, in both number types: 105 test nodes, 91
// source nodes, 36 + 36 even-power nodes.
enum { NN105 = 0, NN91 = 105, NNE105 = 196, NNE91 = 232, NN_ALL = 268 };
__constant__ RuleNode<double> c_near_d[NN_ALL];
__constant__ RuleNode<df> c_near_f[NN_ALL];
__constant__ double c_near_ww1;  // product of the 105- and 91-point weights' sums, less one
template <typename T>
__device__ __forceinline__ const RuleNode<T> *near_nodes();
template <>
__device__ __forceinline__ const RuleNode<double> *near_nodes<double>() { return c_near_d; }
template <>
__device__ __forceinline__ const RuleNode<df> *near_nodes<df>() { return c_near_f; }

// A triangle relative to the test triangle's p0: vertices, normal, edges 01,
// 12, 20, their outward in-plane normals, and inverse edge lengths.
template <typename T>
struct NearFrame {
  V3<T> p[3], n, e[3], m[3];
  T ei[3];
};

// The closed-form potential integrals of a triangle F seen from the point r:
// the analytic part of EHNonSmoothIntegral (src/Source.cpp:16-86) and, with
// full false, of LKEdgeIntegral (src/Impedance.cpp:13-73: ISn1, IL1, h only).
// h = (r - p0) . n.  tol is the edge-line cut-off of the logarithms.
template <typename T>
struct NearPot {
  T ISn3h, ISn1, IS1, h;
  V3<T> IL1, IL3;
};
template <typename T>
__device__ __noinline__ void near_potentials(const NearFrame<T> &F, V3<T> r, typename Num<T>::Tail tol, bool full,
                                             NearPot<T> &o) {
  typedef Num<T> N;
  const T zero = N::of(0.0);
  V3<T> p[3], a[3];
  T R2[3], R[3];
#pragma unroll
  for (int k = 0; k < 3; k++) {
    p[k] = r - F.p[k];
    R2[k] = vdot(p[k], p[k]);
    R[k] = N::sqrt_(R2[k]);
    a[k] = N::rcp(R[k]) * p[k];
  }
  const T x = (vdot(a[0], a[1] + a[2]) + vdot(a[1], a[2])) + N::of(1.0);
  const T y = N::abs_(vdot(a[0], vcross(a[1], a[2])));
  o.h = vdot(p[0], F.n);
  o.ISn3h = N::pow2(N::atan2_(y, x), N::head(o.h) < 0 ? -2.f : 2.f);
  T tl = zero, tI = zero;
  o.IL1 = vzero<T>();
  o.IL3 = vzero<T>();
#pragma unroll
  for (int k = 0; k < 3; k++) {
    const int k1 = (k + 1) % 3;
    const T s0 = F.ei[k] * vdot(F.e[k], p[k]), s1 = F.ei[k] * vdot(F.e[k], p[k1]);
    const T num = R[k1] - s1, den = R[k] - s0;
    T ln = zero;
    if (!(fabs(N::head(num)) < tol || fabs(N::head(den)) < tol)) ln = N::log_(num * N::rcp(den));
    const T t = vdot(F.m[k], p[k]);
    tl = N::muladd(t, ln, tl);
    const T d2 = R2[k] - s0 * s0;
    const T Rs0 = R[k] * s0, Rs1 = R[k1] * s1;
    const T l1 = N::pow2(N::muladd(d2, ln, Rs0 - Rs1), 0.5f);
    o.IL1 = o.IL1 + l1 * F.m[k];
    if (full) {
      const T l3 = N::muladd(N::of(0.75) * d2, l1, N::pow2(N::dot2(R2[k], Rs0, -R2[k1], Rs1), 0.25f));
      tI = N::muladd(t, l1, tI);
      o.IL3 = o.IL3 + l3 * F.m[k];
    }
  }
  o.ISn1 = -N::muladd(o.h, o.ISn3h, tl);
  if (full) o.IS1 = N::of(BEM_ONETHIRD) * N::muladd(o.h * o.h, o.ISn1, -tI);
}

// scalar_gradient_smooth, src/GreensFunction.cpp:54-69, directly.
template <typename T, bool REALK>
__device__ __forceinline__ void near_values(const GreenT<T> &g, V3<T> x, T (&f)[4]) {
  typedef Num<T> N;
  const T R2 = N::sumsq(x.x, x.y, x.z);
  T R, Ri, er, ei, em, ur, ui;
  N::sqrt_rcp(R2, R, Ri);
  wave_at<T, REALK>(g, R, er, ei, em, ur, ui);
  const T one = N::of(1.0), Ri3 = Ri * (Ri * Ri);
  f[0] = N::dot2(er - one, Ri, -g.k2r, R);
  f[2] = (N::muladd(R2, g.k2r, ur) - one) * Ri3;
  if (REALK) {
    f[1] = em * Ri;
    f[3] = ui * Ri3;
  } else {
    f[1] = N::dot2(em, Ri, -g.k2i, R);
    f[3] = N::muladd(R2, g.k2i, ui) * Ri3;
  }
}

constexpr int NEAR_WARPS = 4;

// A test node as the loops over source nodes read it: position relative to the
// source triangle's p0, weight, weight times each barycentric coordinate.
template <typename T>
struct __align__(16) NearNode {
  V3<T> p;
  T w, w1, w2;
};

// A warp's staging of its pair.
template <typename T>
struct NearStage {
  NearNode<T> q[105];
  // odd and even moments [j][a][b], or the four values' moments (NEAR_DIRECT)
  T odd[9 * 9], even[9 * 10];
  T sing[24];
  T edge_sum[3][4];
  // per Green's function: Re and Im of the moments of g~, Re and Im of the
  // barycentric moments of q~, and Im of -U0 (its first entry)
  T mom[2][5][9];
  T qraw[2][2][9];
  NearFrame<T> Sf, Tf;
  // the 45 edge nodes' terms take the test nodes' place
  __device__ __forceinline__ T *edge(int k) { return reinterpret_cast<T *>(q) + 4 * k; }
};

// Adds the warp's sums of NV values per lane, eight at a time, to out[0..NV).
template <typename T, int NV, typename F>
__device__ __forceinline__ void near_reduce(T *out, int lane, F value) {
  const int at = reduce8_index(lane);
#pragma unroll
  for (int c = 0; c < (NV + 7) / 8; c++) {
    T v[8];
#pragma unroll
    for (int k = 0; k < 8; k++) v[k] = c * 8 + k < NV ? value(c * 8 + k) : Num<T>::of(0.0);
    const T r = reduce8<T>(v, lane);
    if ((lane & 3) == 0 && c * 8 + at < NV) out[c * 8 + at] = out[c * 8 + at] + r;
  }
}

// Sums over the staged test nodes q0, q0 + step, ... < nq, seen from the lane's
// source node (l relative to P_s): ODD the powers R^{2j+1}, else (R^2)^{j+1},
// j < JT, times {w, w eta1, w eta2}.
template <typename T, int JF, int JT, bool ODD>
__device__ __forceinline__ void near_power_sums(const NearNode<T> *qn, int q0, int nq, int step, V3<T> l,
                                                T (&S)[JF][3], typename Num<T>::Tail (&St)[JT - JF + 1][3]) {
  typedef Num<T> N;
#pragma unroll
  for (int j = 0; j < JF; j++) S[j][0] = S[j][1] = S[j][2] = N::of(0.0);
#pragma unroll
  for (int j = 0; j < JT - JF; j++) St[j][0] = St[j][1] = St[j][2] = 0;
#pragma unroll 1
  for (int q = q0; q < nq; q += step) {
    const NearNode<T> nd = qn[q];
    const T s = N::sumsq(N::diff(nd.p.x, l.x), N::diff(nd.p.y, l.y), N::diff(nd.p.z, l.z));
    T p = ODD ? N::sqrt_(s) : s;
#pragma unroll
    for (int j = 0; j < JF; j++) {
      N::mac(S[j][0], p, nd.w);
      N::mac(S[j][1], p, nd.w1);
      N::mac(S[j][2], p, nd.w2);
      if (j + 1 < JF) p = p * s;
    }
    typename N::Tail pt = N::head(p);
#pragma unroll
    for (int j = 0; j < JT - JF; j++) {
      pt *= N::head(s);
      St[j][0] += pt * N::head(nd.w);
      St[j][1] += pt * N::head(nd.w1);
      St[j][2] += pt * N::head(nd.w2);
    }
  }
#pragma unroll
  for (int j = 0; j < JF; j++)
#pragma unroll
    for (int a = 0; a < 3; a++) S[j][a] = N::fin(S[j][a]);
}

// Green's function coefficients are stored as pairs of the number type.
template <typename T>
__device__ __forceinline__ C1<T> near_coef(const double (*c)[2], int j);
template <>
__device__ __forceinline__ C1<double> near_coef<double>(const double (*c)[2], int j) { return {c[j][0], c[j][1]}; }
template <>
__device__ __forceinline__ C1<df> near_coef<df>(const double (*c)[2], int j) {
  const float4 v = *reinterpret_cast<const float4 *>(c[j]);
  return {{v.x, v.y}, {v.z, v.w}};
}

// The pair's product (i, j) from its moments, by one lane.
//   L_ij = k^2/4 sum_{ab} (a_a . c_b) [...] - G_00   (as far_contract's)
//          + k^2 (A0_ij + k2 A1_ij) - 2 (B0 + k2 B1)
//   A_ij = Ai/4 [s - e_i . S_X - p_j . S_1rho + (e_i . p_j) S_1],  B = Ai/2 S_1
//   K_ij = -1/4 sum B_vw (volumes) - Ai/4 [(p_j - p_i) x n . T + k2 (p_i - p_j) . (Z - e_i x S_Y)] + edges
// (positions relative to P_t; S_.., T, Z, S_Y the singular moments).
template <typename T>
__device__ __noinline__ void near_product(const NearStage<T> &st, const T (*mom)[9], const GreenDev &gd,
                                             const TriRec &Tr, const TriRec &Sr, int vi, int vj, bool same,
                                             C1<T> &L, C1<T> &K) {
  typedef Num<T> N;
  const GreenT<T> g = green_of<T>(gd);
  const V3<T> pi = st.Tf.p[vi], pj = st.Sf.p[vj], P0 = st.Sf.p[0];
  const V3<T> D = pi - pj;
  // smooth L
  C1<T> br = {N::of(0.0), N::of(0.0)};
  auto G = [&](int a, int b) {
    C1<T> v = {mom[0][a * 3 + b], mom[1][a * 3 + b]};
    return v;
  };
#pragma unroll
  for (int a = 1; a < 3; a++)
#pragma unroll
    for (int b = 1; b < 3; b++) {
      const T d = vdot(st.Tf.p[a], st.Sf.p[b] - P0);
      C1<T> m = G(a, b);
      if (b == vj) m = m - G(a, 0);
      if (a == vi) m = m - G(0, b);
      if (a == vi && b == vj) m = m + G(0, 0);
      br = br + d * m;
    }
  const C1<T> ksq = {g.ksqr, g.ksqi}, k2 = {g.k2r, g.k2i};
  // singular L
  const T Ai2 = N::of(0.5 * Sr.Ai);
  const T *s0 = st.sing, *s1 = st.sing + 7;
  const V3<T> a1 = st.Tf.p[1], a2 = st.Tf.p[2];
  auto A_of = [&](const T *s) {
    const V3<T> SX = {s[1], s[2], s[3]};
    const V3<T> Sr1 = s[5] * a1 + s[6] * a2;
    const T v = ((s[0] - vdot(pi, SX)) - vdot(pj, Sr1)) + vdot(pi, pj) * s[4];
    return N::pow2(Ai2 * v, 0.5f);
  };
  const T A0 = A_of(s0), A1 = A_of(s1);
  const T B0 = Ai2 * s0[4], B1 = Ai2 * s1[4];
  const C1<T> inner = {N::muladd(g.k2r, A1, N::muladd(N::of(0.25), br.r, A0)), N::muladd(g.k2i, A1, N::pow2(br.i, 0.25f))};
  C1<T> g00 = G(0, 0);
  if (N::LESS) {
    // Im g~'s constant Im(ik) is left out of -G_00 but for what the rules'
    // weights leave of it (wave_at); the moments above hold it in full
    g00.i = mom[4][0];
  }
  L = cmul(ksq, inner) - g00;
  L.r = L.r - N::pow2(N::muladd(k2.r, B1, B0), 2.f);
  L.i = L.i - N::pow2(k2.i * B1, 2.f);
  // smooth K
  K = {N::of(0.0), N::of(0.0)};
#pragma unroll
  for (int v = 1; v < 3; v++)
#pragma unroll
    for (int w = 1; w < 3; w++) {
      const int x = (vi + v) % 3, y = (vj + w) % 3;
      const T vol = vdot(D, vcross(st.Sf.p[y] - pj, st.Tf.p[x] - pi));
      N::mac(K.r, mom[2][x * 3 + y], vol);
      N::mac(K.i, mom[3][x * 3 + y], vol);
    }
  const T q = N::of(-0.25);
  K = {q * N::fin(K.r), q * N::fin(K.i)};
  // singular K
  const T *t = st.sing + 14;
  const V3<T> n = st.Sf.n;
  const V3<T> Tv = (t[1] * a1 + t[2] * a2) - t[0] * pi;
  const T kt = vdot(vcross(-N::of(1.0) * D, n), Tv);
  const V3<T> SY = {t[3], t[4], t[5]}, Z = {t[6], t[7], t[8]};
  const T kz = vdot(D, Z - vcross(pi, SY));
  const T h = N::pow2(Ai2, 0.5f);
  K.r = K.r - h * N::muladd(k2.r, kz, kt);
  K.i = K.i - h * (k2.i * kz);
  if (!same) {
    T ke = N::of(0.0);
#pragma unroll
    for (int e = 0; e < 3; e++) {
      const T *x = st.edge_sum[e];
      const V3<T> Ke = V3<T>{x[0], x[1], x[2]} - x[3] * pi;
      ke = N::muladd(vdot(vcross(D, st.Sf.m[e]), Ke), N::rcp(st.Sf.ei[e]), ke);
    }
    K.r = N::muladd(N::of(0.125 * Tr.Ai * Sr.Ai), ke, K.r);
  }
}

// Scatter coefficient of src/Impedance.cpp:372-375.
template <typename T>
__device__ __forceinline__ T near_scatter(const TriRec &T_, int i, const TriRec &S, int j) {
  return Num<T>::of(scatter_coef(T_, i, S, j));
}

// A launch's near pairs: warp w of CTA b takes units b * NEAR_WARPS + w + k *
// (grid warps).  MINB: CTAs per SM that the register allocation must allow (the
// context's tuning).  sync: the CTA's warps meet at a barrier after each pair,
// which keeps them in the same code region.
//
// Bound by FP32 issue (double-float) or the FP64 pipe.  A warp's lanes take the
// 91 source nodes (three rounds of 32, 95 % busy) and each loops over the 105
// test nodes, which are the same for the whole warp (shared-memory broadcasts);
// lanes over test nodes would need four rounds of 82 %.  Double-float, both
// Green's functions of a body's pair at once: about 200 FP32 instructions a
// node pair at |k| R <= 0.47, against about 900 for each of the two with sincos,
// 1/R and Cartesian moments.  The near pairs of a solve's three fills, before
// (two pairs per warp over the test nodes) and now: icospheres N = 7680 31.8 ->
// 4.2 ms, slabs N = 11520 (interiors direct) 47.1 -> 21.0 ms, cubes N = 1152
// 4.9 -> 2.1 ms; in FP64 cubes N = 1152 (interiors direct) 23.7 -> 14.6 ms, the
// exterior fill of icospheres N = 1920 18.1 -> 8.1 ms.  168 registers (12 warps
// an SM) against 226 (8): 4.7 -> 4.2 ms; 128 with spills the same; without the
// barrier 4.4 ms.
template <typename T, int KIND, int MINB>
__global__ void __launch_bounds__(32 * NEAR_WARPS, MINB) near_pairs_kernel(const NearTask *__restrict__ tasks, int ntask,
                                                                           int64_t units, int sync) {
  typedef Num<T> N;
  typedef NearCfg<T, KIND> Cfg;
  constexpr int JF = Cfg::JF, JT = Cfg::JT;
  __shared__ RuleNode<T> rule[NN_ALL];
  __shared__ NearStage<T> stages[NEAR_WARPS];
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  NearStage<T> &st = stages[wid];
  for (int k = threadIdx.x; k < NN_ALL; k += blockDim.x) rule[k] = near_nodes<T>()[k];
  __syncthreads();
  const int64_t nw = (int64_t)gridDim.x * NEAR_WARPS;
  for (int64_t base = (int64_t)blockIdx.x * NEAR_WARPS; base < units; base += nw) {
    const int64_t u = base + wid;
    if (u < units) {
      int ti = ntask - 1;
      while (ti > 0 && u < tasks[ti].unit0) ti--;
      const NearTask &tk = tasks[ti];
      const NearPair np = tk.near[u - tk.unit0];
      const TriRec &Tr = tk.T[np.t];
      const TriRec &Sr = tk.S[np.s];
      const bool same = np.same != 0;
      // the Green's functions of this pair
      int second = 0;
      for (int k = 1; k < tk.ngreen; k++)
        if (np.t >= tk.g[k].tri0 && np.t < tk.g[k].tri1 && np.s >= tk.g[k].tri0 && np.s < tk.g[k].tri1) second = k;
      // both triangles relative to P_t, the test nodes relative to P_s (scaled)
      {
        const double *O = Tr.p0;
        T *Fs = reinterpret_cast<T *>(&st.Sf), *Ft = reinterpret_cast<T *>(&st.Tf);
        for (int k = lane; k < 66; k += 32) {
          const int f = k < 33 ? k : k - 33;
          // NearFrame's order within a TriRec: p0 p1 p2 | n | v01 v12 v20 | m01 m12 m20 | 1/|v|
          const int src = f < 9 ? f : f < 12 ? f + 12 : f < 21 ? f - 3 : f + 3;
          const double *rec = reinterpret_cast<const double *>(k < 33 ? &Sr : &Tr);
          const T v = N::of(f < 9 ? rec[src] - O[f % 3] : rec[src]);
          if (k < 33) Fs[f] = v;
          else Ft[f] = v;
        }
      }
      const float sc = (float)tk.scale;
      V3<T> d0, a1, a2, c1, c2;
      {
        auto v = [](const double *p) { return V3<T>{N::of(p[0]), N::of(p[1]), N::of(p[2])}; };
        d0 = vscale2(V3<T>{N::of(Tr.p0[0] - Sr.p0[0]), N::of(Tr.p0[1] - Sr.p0[1]), N::of(Tr.p0[2] - Sr.p0[2])}, sc);
        a1 = vscale2(v(Tr.v01), sc);
        a2 = vscale2(v(Tr.v02), sc);
        c1 = vscale2(v(Sr.v01), sc);
        c2 = vscale2(v(Sr.v02), sc);
      }
      for (int k = lane; k < 105; k += 32) {
        const RuleNode<T> n = rule[NN105 + k];
        st.q[k] = {d0 + (n.x1 * a1 + n.x2 * a2), n.w, n.w1, n.w2};
      }
      for (int k = lane; k < 81; k += 32) st.odd[k] = N::of(0.0);
      for (int k = lane; k < 90; k += 32) st.even[k] = N::of(0.0);
      if (lane < 24) st.sing[lane] = N::of(0.0);
      __syncwarp();
      // ---- smooth part: moments of the powers of R, or of g~ and q~
#pragma unroll 1
      for (int r = 0; r < 3; r++) {
        const int k = lane + 32 * r;
        RuleNode<T> n = rule[NN91 + (k < 91 ? k : 0)];
        if (k >= 91) n.w = n.w1 = n.w2 = N::of(0.0);
        const V3<T> l = n.x1 * c1 + n.x2 * c2;
        if constexpr (KIND == NEAR_DIRECT) {
          const GreenT<T> g = green_of<T>(tk.g[0].g);
          // unscaled coordinates: scale is 1 in this kind
          T S[4][3];
#pragma unroll
          for (int c = 0; c < 4; c++) S[c][0] = S[c][1] = S[c][2] = N::of(0.0);
          auto loop = [&](auto real) {
#pragma unroll 1
            for (int q = 0; q < 105; q++) {
              const NearNode<T> nd = st.q[q];
              T f[4];
              near_values<T, decltype(real)::value>(
                  g, {N::diff(nd.p.x, l.x), N::diff(nd.p.y, l.y), N::diff(nd.p.z, l.z)}, f);
#pragma unroll
              for (int c = 0; c < 4; c++) {
                N::mac(S[c][0], f[c], nd.w);
                N::mac(S[c][1], f[c], nd.w1);
                N::mac(S[c][2], f[c], nd.w2);
              }
            }
          };
          if (tk.g[0].realk) loop(std::true_type{});
          else loop(std::false_type{});
#pragma unroll
          for (int c = 0; c < 4; c++)
#pragma unroll
            for (int a = 0; a < 3; a++) S[c][a] = N::fin(S[c][a]);
          near_reduce<T, 36>(st.odd, lane, [&](int v) {
            const int b = v % 3;
            return (b == 0 ? n.w : b == 1 ? n.w1 : n.w2) * S[v / 9][v / 3 % 3];
          });
        } else {
          T S[JF][3];
          typename N::Tail St[JT - JF + 1][3];
          near_power_sums<T, JF, JT, true>(st.q, 0, 105, 1, l, S, St);
          near_reduce<T, JF * 9>(st.odd, lane, [&](int v) {
            const int b = v % 3;
            return (b == 0 ? n.w : b == 1 ? n.w1 : n.w2) * S[v / 9][v / 3 % 3];
          });
          if constexpr (JT > JF)
            near_reduce<T, (JT - JF) * 9>(st.odd + JF * 9, lane, [&](int v) {
              const int b = v % 3;
              return N::tail(N::head(b == 0 ? n.w : b == 1 ? n.w1 : n.w2) * St[v / 9][v / 3 % 3]);
            });
        }
      }
      if constexpr (KIND != NEAR_DIRECT) {
        // even powers over 36 x 36 nodes: 32 source nodes by the lanes, then the
        // last four by eight lanes each
        __syncwarp();
        for (int k = lane; k < 36; k += 32) {
          const RuleNode<T> n = rule[NNE105 + k];
          st.q[k] = {d0 + (n.x1 * a1 + n.x2 * a2), n.w, n.w1, n.w2};
        }
        __syncwarp();
#pragma unroll 1
        for (int r = 0; r < 2; r++) {
          const RuleNode<T> n = rule[NNE91 + (r == 0 ? lane : 32 + (lane & 3))];
          const V3<T> l = n.x1 * c1 + n.x2 * c2;
          T S[JF][3];
          typename N::Tail St[JT - JF + 1][3];
          near_power_sums<T, JF, JT, false>(st.q, r == 0 ? 0 : lane >> 2, 36, r == 0 ? 1 : 8, l, S, St);
          near_reduce<T, JF * 9>(st.even + 9, lane, [&](int v) {
            const int b = v % 3;
            return (b == 0 ? n.w : b == 1 ? n.w1 : n.w2) * S[v / 9][v / 3 % 3];
          });
          if constexpr (JT > JF)
            near_reduce<T, (JT - JF) * 9>(st.even + 9 + JF * 9, lane, [&](int v) {
              const int b = v % 3;
              return N::tail(N::head(b == 0 ? n.w : b == 1 ? n.w1 : n.w2) * St[v / 9][v / 3 % 3]);
            });
        }
        // the constant's moments: products of the rules' sums
        if (lane < 9) st.even[lane] = N::of(c_sums[SUM105].w[lane / 3]) * N::of(c_sums[SUM91].w[lane % 3]);
      }
      // ---- singular part: the 105 test nodes, then the neighbours' 45 edge nodes
      {
        T s[23];
#pragma unroll
        for (int k = 0; k < 23; k++) s[k] = N::of(0.0);
        const V3<T> e1 = st.Tf.p[1], e2 = st.Tf.p[2];
        const typename N::Tail tol = (typename N::Tail)(1e-6 * Sr.elen0),
                               tol_plane = (typename N::Tail)(1e-8 * Sr.elen0),
                               tol_edge = (typename N::Tail)(1e-8 * Tr.elen0);
#pragma unroll 1
        for (int it = lane; it < (same ? 105 : 150); it += 32) {
          const bool node = it < 105;
          RuleNode<T> n = rule[NN105 + (node ? it : 0)];
          V3<T> r;
          T wl = N::of(0.0);
          if (node) {
            r = n.x1 * e1 + n.x2 * e2;
          } else {
            const int e = (it - 105) / 15, k = (it - 105) - e * 15;
            r = st.Sf.p[e] + N::of(c_line15[k][0]) * st.Sf.e[e];
            wl = N::of(c_line15[k][1]);
          }
          NearPot<T> o;
          near_potentials<T>(node ? st.Sf : st.Tf, r, node ? tol : tol_edge, node, o);
          if (node) {
            const bool flat = fabs(N::head(o.h)) < tol_plane;
            const V3<T> rp = flat ? r : r - o.h * st.Sf.n;
            const V3<T> X0 = o.IL1 + o.ISn1 * rp, X1 = N::of(BEM_ONETHIRD) * o.IL3 + o.IS1 * rp;
            N::mac(s[0], n.w, vdot(r, X0));
            N::mac(s[1], n.w, X0.x); N::mac(s[2], n.w, X0.y); N::mac(s[3], n.w, X0.z);
            N::mac(s[4], n.w, o.ISn1); N::mac(s[5], n.w1, o.ISn1); N::mac(s[6], n.w2, o.ISn1);
            N::mac(s[7], n.w, vdot(r, X1));
            N::mac(s[8], n.w, X1.x); N::mac(s[9], n.w, X1.y); N::mac(s[10], n.w, X1.z);
            N::mac(s[11], n.w, o.IS1); N::mac(s[12], n.w1, o.IS1); N::mac(s[13], n.w2, o.IS1);
            if (!flat) {
              N::mac(s[14], n.w, o.ISn3h); N::mac(s[15], n.w1, o.ISn3h); N::mac(s[16], n.w2, o.ISn3h);
              const V3<T> Y = o.IL1 - (o.h * o.ISn1) * st.Sf.n;
              const V3<T> rY = vcross(r, Y);
              N::mac(s[17], n.w, Y.x); N::mac(s[18], n.w, Y.y); N::mac(s[19], n.w, Y.z);
              N::mac(s[20], n.w, rY.x); N::mac(s[21], n.w, rY.y); N::mac(s[22], n.w, rY.z);
            }
          } else {
            const V3<T> X = wl * (o.IL1 + o.ISn1 * (r - o.h * st.Tf.n));
            T *e = st.edge(it - 105);
            e[0] = X.x; e[1] = X.y; e[2] = X.z;
            e[3] = wl * o.ISn1;
          }
        }
        __syncwarp();
        near_reduce<T, 23>(st.sing, lane, [&](int v) { return N::fin(s[v]); });
        if (!same && lane < 12) {
          T a = N::of(0.0);
          for (int k = 0; k < 15; k++) a = a + st.edge((lane >> 2) * 15 + k)[lane & 3];
          st.edge_sum[lane >> 2][lane & 3] = a;
        }
      }
      __syncwarp();
      // ---- moments of g~ and q~ of the pair's Green's functions
      const int ng = second ? 2 : 1;
      for (int k = lane; k < 18 * ng; k += 32) {
        const int gi = k / 18, c = (k - gi * 18) / 9, ab = k % 9;
        const NearGreen &G = tk.g[gi ? second : 0];
        C1<T> v;
        if constexpr (KIND == NEAR_DIRECT) {
          v = {st.odd[c * 18 + ab], st.odd[c * 18 + 9 + ab]};
          // the constant that near_values leaves out of Im g~ (wave_at)
          if (N::LESS && c == 0) {
            const T kk = green_of<T>(G.g).iki;
            if (ab == 0) st.mom[gi][4][0] = v.i + kk * N::of(c_near_ww1);
            v.i = N::muladd(kk * N::of(c_sums[SUM105].w[ab / 3]), N::of(c_sums[SUM91].w[ab % 3]), v.i);
          }
        } else {
          const double(*ce)[2] = c ? G.qe : G.ge, (*co)[2] = c ? G.qo : G.go;
          T vr = N::of(0.0), vi = vr;
#pragma unroll 1
          for (int j = JT; j >= 1; j--) {
            const C1<T> e = near_coef<T>(ce, j), o = near_coef<T>(co, j - 1);
            N::mac(vr, e.r, st.even[j * 9 + ab]);
            N::mac(vi, e.i, st.even[j * 9 + ab]);
            N::mac(vr, o.r, st.odd[(j - 1) * 9 + ab]);
            N::mac(vi, o.i, st.odd[(j - 1) * 9 + ab]);
          }
          const C1<T> e = near_coef<T>(ce, 0);
          vr = N::fin(vr);
          vi = N::fin(vi);
          // -G_00 without the constant Im(ik) (wave_at)
          if (N::LESS && c == 0 && ab == 0) st.mom[gi][4][0] = vi + e.i * N::of(c_near_ww1);
          v = {N::muladd(e.r, st.even[ab], vr), N::muladd(e.i, st.even[ab], vi)};
        }
        if (c == 0) {
          st.mom[gi][0][ab] = v.r;
          st.mom[gi][1][ab] = v.i;
        } else {
          st.qraw[gi][0][ab] = v.r;
          st.qraw[gi][1][ab] = v.i;
        }
      }
      __syncwarp();
      for (int k = lane; k < 18 * ng; k += 32) {  // barycentric: B_v = sum over {1, x1, x2} with 1 - x1 - x2 for v = 0
        const int gi = k / 18, ri = (k - gi * 18) / 9, ab = k % 9, x = ab / 3, y = ab % 3;
        const T *Q = st.qraw[gi][ri];
        auto along = [&](int row) { return y ? Q[row * 3 + y] : (Q[row * 3] - Q[row * 3 + 1]) - Q[row * 3 + 2]; };
        st.mom[gi][2 + ri][ab] = x ? along(x) : (along(0) - along(1)) - along(2);
      }
      __syncwarp();
      // ---- the nine products: lanes 0..8 the first Green's function, 16..24 the second
      {
        const int gi = lane >> 4, ij = lane & 15;
        if (gi < ng && ij < 9 && ij / 3 < Tr.nh && ij % 3 < Sr.nh) {
          const int i = ij / 3, j = ij % 3;
          const NearGreen &G = tk.g[gi ? second : 0];
          C1<T> L, K;
          near_product<T>(st, st.mom[gi], G.g, Tr, Sr, (Tr.hvert >> (2 * i)) & 3,
                          (Sr.hvert >> (2 * j)) & 3, same, L, K);
          const T c = near_scatter<T>(Tr, i, Sr, j);
          store_pair(G.H, G.ntr, Tr.hrwg[i] - G.rwg0, Tr.hneg[i], Sr.hrwg[j] - G.rwg0, Sr.hneg[j], c * L, c * K);
        }
      }
      __syncwarp();
    }
    // base is the same for the whole CTA: every warp meets the barrier
    if (sync) __syncthreads();
  }
}

template <typename T, int MINB>
void launch_near_kind(int kind, int nb, cudaStream_t st, const NearTask *tasks, int ntask, int64_t units, int sync) {
  if (kind == NEAR_SERIES1)
    near_pairs_kernel<T, NEAR_SERIES1, MINB><<<nb, 32 * NEAR_WARPS, 0, st>>>(tasks, ntask, units, sync);
  else if (kind == NEAR_SERIES2)
    near_pairs_kernel<T, NEAR_SERIES2, MINB><<<nb, 32 * NEAR_WARPS, 0, st>>>(tasks, ntask, units, sync);
  else
    near_pairs_kernel<T, NEAR_DIRECT, MINB><<<nb, 32 * NEAR_WARPS, 0, st>>>(tasks, ntask, units, sync);
}

// The near pairs of `ntask` tasks of one kind.
void launch_near(bool dfl, int minb, int kind, int nb, cudaStream_t st, const NearTask *tasks, int ntask, int64_t units,
                 int sync) {
  if (!dfl)
    launch_near_kind<double, 2>(kind, nb, st, tasks, ntask, units, sync);
  else if (minb == 3)
    launch_near_kind<df, 3>(kind, nb, st, tasks, ntask, units, sync);
  else if (minb == 4)
    launch_near_kind<df, 4>(kind, nb, st, tasks, ntask, units, sync);
  else
    launch_near_kind<df, 2>(kind, nb, st, tasks, ntask, units, sync);
}

// ---------------- gather: half-pair blocks -> Z ----------------
struct ZDev {
  double zer, zei, zmr, zmi;  // Zeps, Zmu
};

template <bool DFH>
__device__ __forceinline__ void block_sum(const HalfPairBlock &b, z1 &sL, z1 &sK) {
  sL = {0, 0};
  sK = {0, 0};
  if (DFH) {
    // the four half-pair terms summed in double-float, widened once
    const float4 *p = reinterpret_cast<const float4 *>(b.v);
    df Lr = {0.f, 0.f}, Li = Lr, Kr = Lr, Ki = Lr;
#pragma unroll
    for (int k = 0; k < 4; k++) {
      const float4 l = p[2 * k], kk = p[2 * k + 1];
      Lr = df_add(Lr, {l.x, l.y});
      Li = df_add(Li, {l.z, l.w});
      Kr = df_add(Kr, {kk.x, kk.y});
      Ki = df_add(Ki, {kk.z, kk.w});
    }
    sL = {df_to_double(Lr), df_to_double(Li)};
    sK = {df_to_double(Kr), df_to_double(Ki)};
    return;
  }
  const double2 *p = reinterpret_cast<const double2 *>(b.v);
#pragma unroll
  for (int k = 0; k < 4; k++) {
    const double2 l = p[2 * k], kk = p[2 * k + 1];
    sL.r += l.x; sL.i += l.y;
    sK.r += kk.x; sK.i += kk.y;
  }
}

__device__ __forceinline__ void write_2x2(double *Z, int64_t ld, int i, int j, z1 Ze, z1 Zm, z1 sL, z1 sK) {
  // src/Impedance.cpp:378-381
  const z1 a = zmul(Ze, sL), d = zmul(Zm, sL);
  double2 *c0 = reinterpret_cast<double2 *>(Z + 2 * ((int64_t)2 * i + ld * (2 * (int64_t)j)));
  double2 *c1 = reinterpret_cast<double2 *>(Z + 2 * ((int64_t)2 * i + ld * (2 * (int64_t)j + 1)));
  c0[0] = make_double2(a.r, a.i);
  c0[1] = make_double2(-sK.r, -sK.i);
  c1[0] = make_double2(sK.r, sK.i);
  c1[1] = make_double2(d.r, d.i);
}

template <bool DFH>
__global__ void gather_z_kernel(const HalfPairBlock *__restrict__ H, int ntr, int nsr, ZDev z, double *Z, int64_t ld) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  const int j = blockIdx.y;
  if (i >= ntr) return;
  z1 sL, sK;
  block_sum<DFH>(H[(size_t)j * ntr + i], sL, sK);
  write_2x2(Z, ld, i, j, {z.zer, z.zei}, {z.zmr, z.zmi}, sL, sK);
}

// W = Z_ext + blockdiag(G1, G2) and the G blocks themselves (src/HeatTransfer.cpp:26-35).
template <bool DFH>
__global__ void gather_w_kernel(const HalfPairBlock *__restrict__ He, const HalfPairBlock *__restrict__ H1,
                                const HalfPairBlock *__restrict__ H2, int ns, int nt, ZDev ze, ZDev z1d, ZDev z2d,
                                double *W, int64_t ldw, double *G1, int64_t ld1, double *G2, int64_t ld2) {
  const int n = ns + nt;
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  const int j = blockIdx.y;
  if (i >= n) return;
  z1 sL, sK;
  block_sum<DFH>(He[(size_t)j * n + i], sL, sK);
  z1 a = zmul({ze.zer, ze.zei}, sL), d = zmul({ze.zmr, ze.zmi}, sL), k = sK;
  const bool in1 = i < ns && j < ns, in2 = i >= ns && j >= ns;
  if (in1 || in2) {
    z1 gL, gK;
    const ZDev &zz = in1 ? z1d : z2d;
    const int li = in1 ? i : i - ns, lj = in1 ? j : j - ns, nn = in1 ? ns : nt;
    block_sum<DFH>((in1 ? H1 : H2)[(size_t)lj * nn + li], gL, gK);
    write_2x2(in1 ? G1 : G2, in1 ? ld1 : ld2, li, lj, {zz.zer, zz.zei}, {zz.zmr, zz.zmi}, gL, gK);
    const z1 ga = zmul({zz.zer, zz.zei}, gL), gd = zmul({zz.zmr, zz.zmi}, gL);
    a = zadd(a, ga);
    d = zadd(d, gd);
    k = zadd(k, gK);
  }
  double2 *c0 = reinterpret_cast<double2 *>(W + 2 * ((int64_t)2 * i + ldw * (2 * (int64_t)j)));
  double2 *c1 = reinterpret_cast<double2 *>(W + 2 * ((int64_t)2 * i + ldw * (2 * (int64_t)j + 1)));
  c0[0] = make_double2(a.r, a.i);
  c0[1] = make_double2(-k.r, -k.i);
  c1[0] = make_double2(k.r, k.i);
  c1[1] = make_double2(d.r, d.i);
}

void split_df(double x, float out[2]) {
  out[0] = (float)x;
  out[1] = (float)(x - (double)out[0]);
}

df host_df(double x) {
  const float h = (float)x;
  return {h, (float)(x - (double)h)};
}

GreenDev to_dev(const bemgpu_green_t *g) {
  GreenDev d;
  d.ikr = g->ik[0]; d.iki = g->ik[1];
  d.k2r = g->k2[0]; d.k2i = g->k2[1];
  d.ksqr = g->ksquared[0]; d.ksqi = g->ksquared[1];
  split_df(d.ikr, d.ikr_f); split_df(d.iki, d.iki_f);
  split_df(d.k2r, d.k2r_f); split_df(d.k2i, d.k2i_f);
  split_df(d.ksqr, d.ksqr_f); split_df(d.ksqi, d.ksqi_f);
  return d;
}

ZDev to_zdev(const bemgpu_green_t *g) { return {g->Zeps[0], g->Zeps[1], g->Zmu[0], g->Zmu[1]}; }

// The kind of a near task whose Green's functions have wavenumbers of at most
// kabs and whose triangles' edges are at most emax long: two triangles that
// share a vertex have no points farther apart than two edges.
int near_kind(double kabs, double emax) {
  const double x = kabs * 2.0 * emax;
  return x <= NEAR_X1 ? NEAR_SERIES1 : x <= NEAR_X2 ? NEAR_SERIES2 : NEAR_DIRECT;
}

double green_kabs(const bemgpu_green_t *g) { return std::hypot(g->ik[0], g->ik[1]); }

// The power of two that brings distances of up to 2 emax below one.
double near_scale(double emax) {
  int e = 0;
  std::frexp(2.0 * emax, &e);
  return std::ldexp(1.0, -e);
}

// One Green's function of a near task: (ik)^n / n! (times 1 - n for q~) in
// powers of the scaled distance.
NearGreen near_green(const bemgpu_green_t *g, double scale, bool dfl, HalfPairBlock *H, int ntr, int rwg0, int tri0,
                     int tri1) {
  NearGreen G;
  memset(&G, 0, sizeof G);
  G.H = H;
  G.ntr = ntr;
  G.rwg0 = rwg0;
  G.tri0 = tri0;
  G.tri1 = tri1;
  G.realk = g->ik[0] == 0.0 && g->ksquared[1] == 0.0;
  G.g = to_dev(g);
  const long double kr = (long double)g->ik[0] / scale, ki = (long double)g->ik[1] / scale;
  long double pr = 1.0L, pi = 0.0L;  // (ik / scale)^n / n!
  auto put = [&](double (*c)[2], int j, long double f) {
    if (j < 0 || j >= NEAR_NJ) return;
    const double re = (double)(f * pr), im = (double)(f * pi);
    if (dfl) {
      const df a = host_df(re), b = host_df(im);
      const float v[4] = {a.hi, a.lo, b.hi, b.lo};
      memcpy(c[j], v, sizeof v);
    } else {
      c[j][0] = re;
      c[j][1] = im;
    }
  };
  const long double s1 = scale, s3 = (long double)scale * scale * scale;
  for (int n = 1; n <= 2 * NEAR_NJ + 2; n++) {
    const long double r = (pr * kr - pi * ki) / n, i = (pr * ki + pi * kr) / n;
    pr = r;
    pi = i;
    if (n % 2) {
      put(G.ge, (n - 1) / 2, s1);
      if (n >= 3) put(G.qe, (n - 3) / 2, s3 * (1 - n));
    } else if (n >= 4) {
      put(G.go, (n - 2) / 2, s1);
      put(G.qo, (n - 4) / 2, s3 * (1 - n));
    }
  }
  return G;
}

// Whether top is the tree of a's RWGs followed by b's, on separate triangles:
// its triangles are then a's followed by b's, with the same frames.
bool is_two_body(const bemgpu_tree_s *top, const bemgpu_tree_s *a, const bemgpu_tree_s *b) {
  return top->geom == a->geom && top->geom == b->geom && top->nrwg == a->nrwg + b->nrwg &&
         top->ntri == a->ntri + b->ntri && top->rwg.size() == a->rwg.size() + b->rwg.size() &&
         std::equal(a->rwg.begin(), a->rwg.end(), top->rwg.begin()) &&
         std::equal(b->rwg.begin(), b->rwg.end(), top->rwg.begin() + (std::ptrdiff_t)a->rwg.size());
}

bool g_tables_loaded[BEM_MAX_DEVICES] = {false};

std::mutex g_tables_mu;

int load_tables(bemgpu_ctx_s *ctx) {
  // once per device; contexts on several host threads (farm lanes) may race here
  if (ctx->device < 0 || ctx->device >= BEM_MAX_DEVICES)
    return bem_fail(ctx, BEMGPU_ERR_ARG, "device %d outside 0..%d", ctx->device, BEM_MAX_DEVICES - 1);
  std::lock_guard<std::mutex> lk(g_tables_mu);
  if (g_tables_loaded[ctx->device]) return BEMGPU_OK;
  BEM_CUDA_TRY(ctx, cudaMemcpyToSymbol(c_rule6, bemgpu_tri_rule6, sizeof(bemgpu_tri_rule6)));
  BEM_CUDA_TRY(ctx, cudaMemcpyToSymbol(c_rule10, bemgpu_tri_rule10, sizeof(bemgpu_tri_rule10)));
  BEM_CUDA_TRY(ctx, cudaMemcpyToSymbol(c_rule15, bemgpu_tri_rule15, sizeof(bemgpu_tri_rule15)));
  BEM_CUDA_TRY(ctx, cudaMemcpyToSymbol(c_rule21, bemgpu_tri_rule21, sizeof(bemgpu_tri_rule21)));
  BEM_CUDA_TRY(ctx, cudaMemcpyToSymbol(c_rule36, bemgpu_tri_rule36, sizeof(bemgpu_tri_rule36)));
  BEM_CUDA_TRY(ctx, cudaMemcpyToSymbol(c_line15, bemgpu_line_rule15, sizeof(bemgpu_line_rule15)));
  {
    const struct {
      const double (*rule)[3];
      int off, n;
    } far[5] = {{bemgpu_tri_rule6, NODES6, 6}, {bemgpu_tri_rule10, NODES10, 10}, {bemgpu_tri_rule15, NODES15, 15},
                {bemgpu_tri_rule21, NODES21, 21}, {bemgpu_tri_rule36, NODES36, 36}};
    std::vector<RuleNode<double>> nd(NODES_FAR);
    std::vector<RuleNode<df>> nf(NODES_FAR);
    for (const auto &r : far)
      for (int k = 0; k < r.n; k++) {
        const double x1 = r.rule[k][0], x2 = r.rule[k][1], w = r.rule[k][2];
        nd[r.off + k] = {x1, x2, w, w * x1, w * x2};
        nf[r.off + k] = {host_df(x1), host_df(x2), host_df(w), host_df(w * x1), host_df(w * x2)};
      }
    const struct {
      const double (*rule)[3];
      int n;
    } all[NSUMS] = {{bemgpu_tri_rule6, 6},   {bemgpu_tri_rule10, 10}, {bemgpu_tri_rule15, 15},  {bemgpu_tri_rule21, 21},
                    {bemgpu_tri_rule36, 36}, {bemgpu_tri_rule91, 91}, {bemgpu_tri_rule105, 105}};
    RuleSum sums[NSUMS];
    double less[NSUMS];
    for (int i = 0; i < NSUMS; i++) {
      long double a[3] = {-1.0L, 0.0L, 0.0L};  // the weights' sum less one
      for (int k = 0; k < all[i].n; k++) {
        const long double w = all[i].rule[k][2];
        a[0] += w;
        a[1] += w * all[i].rule[k][0];
        a[2] += w * all[i].rule[k][1];
      }
      less[i] = (double)a[0];
      sums[i] = {{(double)(1.0L + a[0]), (double)a[1], (double)a[2]}, (double)(2.0L * a[0] + a[0] * a[0])};
    }
    BEM_CUDA_TRY(ctx, cudaMemcpyToSymbol(c_sums, sums, sizeof sums));
    {
      std::vector<RuleNode<double>> qd(NN_ALL);
      std::vector<RuleNode<df>> qf(NN_ALL);
      auto put = [&](int at, const double *node, double w) {
        const double x1 = node[0], x2 = node[1];
        qd[at] = {x1, x2, w, w * x1, w * x2};
        qf[at] = {host_df(x1), host_df(x2), host_df(w), host_df(w * x1), host_df(w * x2)};
      };
      for (int k = 0; k < 105; k++) put(NN105 + k, bemgpu_tri_rule105[k], bemgpu_tri_rule105[k][2]);
      for (int k = 0; k < 91; k++) put(NN91 + k, bemgpu_tri_rule91[k], bemgpu_tri_rule91[k][2]);
      for (int k = 0; k < 36; k++) {
        put(NNE105 + k, bemgpu_tri_rule36[k], bemgpu_even_w105[k]);
        put(NNE91 + k, bemgpu_tri_rule36[k], bemgpu_even_w91[k]);
      }
      BEM_CUDA_TRY(ctx, cudaMemcpyToSymbol(c_near_d, qd.data(), sizeof(RuleNode<double>) * NN_ALL));
      BEM_CUDA_TRY(ctx, cudaMemcpyToSymbol(c_near_f, qf.data(), sizeof(RuleNode<df>) * NN_ALL));
      const double ww1 = less[SUM105] + less[SUM91] + less[SUM105] * less[SUM91];
      BEM_CUDA_TRY(ctx, cudaMemcpyToSymbol(c_near_ww1, &ww1, sizeof ww1));
    }
    BEM_CUDA_TRY(ctx, cudaMemcpyToSymbol(c_far_d, nd.data(), sizeof(RuleNode<double>) * nd.size()));
    BEM_CUDA_TRY(ctx, cudaMemcpyToSymbol(c_far_f, nf.data(), sizeof(RuleNode<df>) * nf.size()));
  }
  // the copies from host memory may return before they land: every stream
  // of the device reads the tables from now on
  BEM_CUDA_TRY(ctx, cudaDeviceSynchronize());
  g_tables_loaded[ctx->device] = true;
  return BEMGPU_OK;
}

}  // namespace

int bem_fill_group(bemgpu_ctx_s *ctx, FillJob *jobs, int njobs, const bemgpu_options_t *opt, int precision,
                   cudaStream_t stream) {
  if (njobs < 1) return BEMGPU_OK;
  int rc = load_tables(ctx);
  if (rc) return rc;
  const int mode = precision == BEMGPU_PREC_MIXED ? FILL_FP32_FAR : precision == BEMGPU_PREC_MIXED_LA ? FILL_DF : FILL_FP64;
  const FarOpts fo = {opt->farThresh6, opt->farThresh10, opt->farThresh15, opt->farThresh21};
  const int fr = ctx->tune.far_rows;
  std::vector<FillTask> tasks(njobs);
  std::vector<const NearList *> lists(njobs);
  // double-float records: one set per tree of the group
  std::vector<const bemgpu_tree_s *> trees;
  std::vector<size_t> tree_off;
  size_t ndf = 0;
  auto records_of = [&](const bemgpu_tree_s *x) {
    for (size_t k = 0; k < trees.size(); k++)
      if (trees[k] == x) return tree_off[k];
    trees.push_back(x);
    tree_off.push_back(ndf);
    ndf += x->ntri;
    return tree_off.back();
  };
  for (int i = 0; i < njobs; i++) {
    lists[i] = bem_near_list(ctx, jobs[i].t, jobs[i].s);
    if (!lists[i]) return bem_fail(ctx, BEMGPU_ERR_OOM, "near list allocation failed");
    records_of(jobs[i].t);
    records_of(jobs[i].s);
  }
  TriDF *df_rec = nullptr;
  if (mode == FILL_DF) {
    df_rec = (TriDF *)bem_workspace(ctx, "fill_tdf", sizeof(TriDF) * ndf);
    if (!df_rec) return bem_fail(ctx, BEMGPU_ERR_OOM, "fill: double-float records");
  }
  // the near pairs' tasks, by kind: a fill of a two-body tree takes the two
  // bodies' own fills that follow it along (their near pairs are its own, with
  // other Green's functions), unless one of them needs the direct kind
  std::vector<NearTask> near[NEAR_KINDS];
  int64_t near_units[NEAR_KINDS] = {};
  {
    std::vector<char> taken(njobs, 0);
    const bool dfl = mode == FILL_DF;
    for (int i = 0; i < njobs; i++) {
      if (taken[i] || lists[i]->n == 0) continue;
      const bemgpu_tree_s *t = jobs[i].t, *s = jobs[i].s;
      const double emax = std::max(t->emax, s->emax);
      int kind = near_kind(green_kabs(&jobs[i].g), emax);
      const double scale = kind == NEAR_DIRECT ? 1.0 : near_scale(emax);
      NearTask nt;
      memset(&nt, 0, sizeof nt);
      nt.T = t->d_rec;
      nt.S = s->d_rec;
      nt.near = lists[i]->d;
      nt.nnear = lists[i]->n;
      nt.scale = scale;
      nt.ngreen = 1;
      nt.g[0] = near_green(&jobs[i].g, scale, dfl, jobs[i].H, t->nrwg, 0, 0, t->ntri);
      if (kind != NEAR_DIRECT && t == s && i + 2 < njobs && jobs[i + 1].t == jobs[i + 1].s &&
          jobs[i + 2].t == jobs[i + 2].s && is_two_body(t, jobs[i + 1].t, jobs[i + 2].t)) {
        for (int k = 1; k <= 2; k++) {
          const bemgpu_tree_s *b = jobs[i + k].t;
          const int kb = near_kind(green_kabs(&jobs[i + k].g), emax);
          if (taken[i + k] || kb == NEAR_DIRECT) continue;
          const int rwg0 = k == 1 ? 0 : jobs[i + 1].t->nrwg, tri0 = k == 1 ? 0 : jobs[i + 1].t->ntri;
          nt.g[nt.ngreen++] = near_green(&jobs[i + k].g, scale, dfl, jobs[i + k].H, b->nrwg, rwg0, tri0, tri0 + b->ntri);
          kind = std::max(kind, kb);  // SERIES2 carries more powers than SERIES1
          taken[i + k] = 1;
        }
      }
      nt.unit0 = near_units[kind];
      near_units[kind] += nt.nnear;
      near[kind].push_back(nt);
    }
  }
  const size_t nnear = near[0].size() + near[1].size() + near[2].size();
  // one upload: the far tasks, the near tasks, the records' jobs
  const size_t tasks_bytes = (sizeof(FillTask) * (size_t)njobs + 15) / 16 * 16, near_bytes_ = sizeof(NearTask) * nnear,
               tdf_bytes = sizeof(TriDFJob) * trees.size();
  unsigned char *dtable = (unsigned char *)bem_workspace(ctx, "fill_tasks", tasks_bytes + near_bytes_ + tdf_bytes);
  if (!dtable) return bem_fail(ctx, BEMGPU_ERR_OOM, "fill: task table");
  FillTask *dtasks = (FillTask *)dtable;
  const NearTask *dnear = (const NearTask *)(dtable + tasks_bytes);
  double far_flops = 0, far_bytes = 0, near_flops = 0, near_bytes = 0;
  int64_t far_tiles = 0;
  for (int i = 0; i < njobs; i++) {
    const bemgpu_tree_s *t = jobs[i].t, *s = jobs[i].s;
    FillTask &tk = tasks[i];
    tk.T = t->d_rec;
    tk.S = s->d_rec;
    tk.TD = tk.SD = nullptr;
    if (df_rec) {
      tk.TD = df_rec + records_of(t);
      tk.SD = df_rec + records_of(s);
    }
    tk.H = jobs[i].H;
    tk.ntT = t->ntri;
    tk.ntS = s->ntri;
    tk.ntr = t->nrwg;
    tk.far_tx = (s->ntri + 31) / 32;
    tk.far0 = far_tiles;
    tk.sym = t == s && mode != FILL_FP32_FAR;
    far_tiles += far_tiles_of(tk.sym, t->ntri, s->ntri, fr);
    tk.g = to_dev(&jobs[i].g);
    jobs[i].near = lists[i]->n;
    jobs[i].far = (int64_t)t->ntri * s->ntri - lists[i]->n;
    if (ctx->prof) {
      const int64_t *fc = bem_far_rule_counts(ctx, t, s, opt);
      const int P[5] = {6, 10, 15, 21, 36};
      int64_t nfar = 0;
      for (int k = 0; k < 5; k++) { far_flops += fc[k] * bem_far_pair_flops(P[k]); nfar += fc[k]; }
      // half-pair products written: 9 per pair on average (nh_t * nh_s)
      far_bytes += (double)nfar * 9.0 * BEM_HALFPAIR_BYTES_FP64;
      near_flops += (double)lists[i]->n * bem_near_pair_flops(true);
      near_bytes += (double)lists[i]->n * 9.0 * BEM_HALFPAIR_BYTES_FP64;
    }
  }
  // the tables are copied from this call's host vector before the call returns
  std::vector<unsigned char> table(tasks_bytes + near_bytes_ + tdf_bytes);
  memcpy(table.data(), tasks.data(), sizeof(FillTask) * (size_t)njobs);
  {
    size_t at = tasks_bytes;
    for (int k = 0; k < NEAR_KINDS; k++) {
      if (!near[k].empty()) memcpy(table.data() + at, near[k].data(), sizeof(NearTask) * near[k].size());
      at += sizeof(NearTask) * near[k].size();
    }
  }
  int most = 0;
  for (size_t k = 0; k < trees.size(); k++) {
    const TriDFJob jb = {trees[k]->d_rec, df_rec ? df_rec + tree_off[k] : nullptr, trees[k]->ntri};
    memcpy(table.data() + tasks_bytes + near_bytes_ + k * sizeof(TriDFJob), &jb, sizeof jb);
    most = std::max(most, jb.n);
  }
  BEM_CUDA_TRY(ctx, cudaMemcpyAsync(dtable, table.data(), table.size(), cudaMemcpyHostToDevice, stream));
  if (df_rec) {
    tri_df_kernel<<<dim3((most + 127) / 128, (unsigned)trees.size()), 128, 0, stream>>>(
        (const TriDFJob *)(dtable + tasks_bytes + near_bytes_));
    ctx->launches++;
  }
  if (far_tiles > 0) {
    if (far_tiles > 0x7fffffffll) return bem_fail(ctx, BEMGPU_ERR_ARG, "fill: %lld far tiles", (long long)far_tiles);
    ProfScope ps(ctx, BEMGPU_K_FILL_FAR, stream, far_flops, far_bytes);
    launch_far(mode, (unsigned)far_tiles, fr, stream, dtasks, njobs, fo);
    ctx->launches++;
  }
  BEM_CUDA_TRY(ctx, cudaGetLastError());
  if (nnear > 0) {
    ProfScope ps(ctx, BEMGPU_K_FILL_NEAR, stream, near_flops, near_bytes);
    size_t at = 0;
    for (int k = 0; k < NEAR_KINDS; k++) {
      if (near[k].empty()) continue;
      const int nb = (int)std::min<int64_t>((near_units[k] + NEAR_WARPS - 1) / NEAR_WARPS,
                                            (int64_t)ctx->num_sms * ctx->tune.near_grid);
      launch_near(mode == FILL_DF, ctx->tune.near_minb, k, nb, stream, dnear + at, (int)near[k].size(), near_units[k],
                  ctx->tune.near_sync);
      ctx->launches++;
      at += near[k].size();
    }
  }
  BEM_CUDA_TRY(ctx, cudaGetLastError());
  return BEMGPU_OK;
}

int bem_fill_pairs(bemgpu_ctx_s *ctx, const bemgpu_tree_s *t, const bemgpu_tree_s *s, const bemgpu_green_t *g,
                   const bemgpu_options_t *opt, int precision, HalfPairBlock *H, cudaStream_t stream,
                   int64_t *n_near, int64_t *n_far) {
  FillJob job = {t, s, *g, H, 0, 0};
  const int rc = bem_fill_group(ctx, &job, 1, opt, precision, stream);
  if (n_near) *n_near = job.near;
  if (n_far) *n_far = job.far;
  return rc;
}

int bem_gather_z(bemgpu_ctx_s *ctx, const HalfPairBlock *H, int ntr, int nsr, const bemgpu_green_t *g, double *Z,
                 int64_t ld, cudaStream_t stream, bool df) {
  dim3 blk(128);
  dim3 grd((ntr + 127) / 128, nsr);
  ProfScope ps(ctx, BEMGPU_K_GATHER, stream, (double)ntr * nsr * (6 * 8 + 2 * 6), (double)ntr * nsr * (128 + 64));
  if (df)
    gather_z_kernel<true><<<grd, blk, 0, stream>>>(H, ntr, nsr, to_zdev(g), Z, ld);
  else
    gather_z_kernel<false><<<grd, blk, 0, stream>>>(H, ntr, nsr, to_zdev(g), Z, ld);
  ctx->launches++;
  BEM_CUDA_TRY(ctx, cudaGetLastError());
  return BEMGPU_OK;
}

int bem_gather_w(bemgpu_ctx_s *ctx, const HalfPairBlock *Hext, const HalfPairBlock *H1, const HalfPairBlock *H2,
                 int ns, int nt, const bemgpu_green_t *gext, const bemgpu_green_t *g1, const bemgpu_green_t *g2,
                 double *W, int64_t ldw, double *G1, int64_t ld1, double *G2, int64_t ld2, cudaStream_t stream,
                 bool df) {
  dim3 blk(128);
  dim3 grd((ns + nt + 127) / 128, ns + nt);
  const double nn = (double)(ns + nt) * (ns + nt), nd = (double)ns * ns + (double)nt * nt;
  ProfScope ps(ctx, BEMGPU_K_GATHER, stream, nn * 60 + nd * 80, nn * 192 + nd * 192);
  if (df)
    gather_w_kernel<true><<<grd, blk, 0, stream>>>(Hext, H1, H2, ns, nt, to_zdev(gext), to_zdev(g1), to_zdev(g2), W,
                                                   ldw, G1, ld1, G2, ld2);
  else
    gather_w_kernel<false><<<grd, blk, 0, stream>>>(Hext, H1, H2, ns, nt, to_zdev(gext), to_zdev(g1), to_zdev(g2), W,
                                                    ldw, G1, ld1, G2, ld2);
  ctx->launches++;
  BEM_CUDA_TRY(ctx, cudaGetLastError());
  return BEMGPU_OK;
}

// ---------------- public Zts ----------------
extern "C" int bemgpu_zts(bemgpu_ctx_t ctx, bemgpu_tree_t t, bemgpu_tree_t s, const bemgpu_green_t *g,
                          const bemgpu_options_t *opt, int precision, void *dZ, int64_t ldz, void *stream) {
  if (!ctx || !t || !s || !g || !dZ) return bem_fail(ctx, BEMGPU_ERR_ARG, "zts: null argument");
  if (t->geom != s->geom) return bem_fail(ctx, BEMGPU_ERR_ARG, "zts: t and s must share one geometry");
  if (ldz < 2 * (int64_t)t->nrwg) return bem_fail(ctx, BEMGPU_ERR_ARG, "zts: ldz < 2*size(t)");
  if (precision != BEMGPU_PREC_FP64 && precision != BEMGPU_PREC_MIXED && precision != BEMGPU_PREC_MIXED_LA)
    return bem_fail(ctx, BEMGPU_ERR_ARG, "zts: unknown precision %d", precision);
  bemgpu_options_t o;
  if (opt) o = *opt; else bemgpu_options_default(&o);
  std::lock_guard<std::mutex> lk(ctx->mu);
  cudaSetDevice(ctx->device);
  cudaStream_t st = stream ? (cudaStream_t)stream : ctx->stream;
  HalfPairBlock *H = (HalfPairBlock *)bem_workspace(ctx, "H0", sizeof(HalfPairBlock) * (size_t)t->nrwg * s->nrwg);
  if (!H) return bem_fail(ctx, BEMGPU_ERR_OOM, "zts: workspace allocation failed");
  int rc = bem_fill_pairs(ctx, t, s, g, &o, precision, H, st, nullptr, nullptr);
  if (rc) return rc;
  return bem_gather_z(ctx, H, t->nrwg, s->nrwg, g, (double *)dZ, ldz, st, precision == BEMGPU_PREC_MIXED_LA);
}

extern "C" int bemgpu_zts_host(bemgpu_ctx_t ctx, bemgpu_tree_t t, bemgpu_tree_t s, const bemgpu_green_t *g,
                               const bemgpu_options_t *opt, int precision, double *Z, int64_t ldz) {
  if (!ctx || !t || !s || !Z) return bem_fail(ctx, BEMGPU_ERR_ARG, "zts_host: null argument");
  const int64_t m = 2 * (int64_t)t->nrwg, n = 2 * (int64_t)s->nrwg;
  if (ldz < m) return bem_fail(ctx, BEMGPU_ERR_ARG, "zts_host: ldz < 2*size(t)");
  double *dZ = nullptr;
  {
    std::lock_guard<std::mutex> lk(ctx->mu);
    cudaSetDevice(ctx->device);
    dZ = (double *)bem_workspace(ctx, "Zhost", sizeof(double) * 2 * m * n);
    if (!dZ) return bem_fail(ctx, BEMGPU_ERR_OOM, "zts_host: workspace allocation failed");
  }
  int rc = bemgpu_zts(ctx, t, s, g, opt, precision, dZ, m, nullptr);
  if (rc) return rc;
  std::lock_guard<std::mutex> lk(ctx->mu);
  BEM_CUDA_TRY(ctx, cudaMemcpy2DAsync(Z, sizeof(double) * 2 * ldz, dZ, sizeof(double) * 2 * m, sizeof(double) * 2 * m,
                                      n, cudaMemcpyDeviceToHost, ctx->stream));
  BEM_CUDA_TRY(ctx, cudaStreamSynchronize(ctx->stream));
  return BEMGPU_OK;
}

// ---------------- Zts without device allocation ----------------
//
// For callers that must not allocate device memory while they run: a solver
// loop with a latency budget that cannot stall in cudaMalloc (which may
// synchronise the device), or a host application whose own memory pool has
// claimed the device memory, so that a library allocation would fail or
// break its accounting.  bemgpu_zts_noalloc does the same FP64 fill as
// bemgpu_zts into the caller's buffer, but keeps its scratch (the half-pair
// blocks and the near-pair list) in one file-scope device array of fixed
// size, created when the library's module is loaded on a GPU and held until
// the process exits.
//
// What each call still does on the host: it builds the near-pair list of
// (t, s) in host memory (a std::vector), copies it into the scratch with
// cudaMemcpyAsync on the caller's stream and synchronises that stream before
// returning, since the host copy belongs to the call.  The first call on a
// device also does that device's set-up: cudaGetSymbolAddress of the scratch
// and, if no other fill ran there yet, the upload of the quadrature tables
// (cudaMemcpyToSymbol); make that first call before any stream capture.
namespace {

constexpr size_t NOALLOC_SCRATCH_BYTES = 32u << 20;   // 32 MiB
constexpr size_t NOALLOC_NEAR_BYTES = 2u << 20;       // first 2 MiB: the near-pair list
static __device__ __align__(256) unsigned char g_noalloc_scratch[NOALLOC_SCRATCH_BYTES];
// its task table: the far pairs' and the near pairs'
struct NoallocTasks {
  FillTask far;
  NearTask near;
};
static __device__ __align__(256) unsigned char g_noalloc_task[sizeof(NoallocTasks)];

std::mutex g_noalloc_mu;
std::mutex g_noalloc_run_mu;  // one call at a time uses the shared scratch
void *g_noalloc_addr[BEM_MAX_DEVICES] = {nullptr};
void *g_noalloc_task_addr[BEM_MAX_DEVICES] = {nullptr};

}  // namespace

extern "C" int bemgpu_zts_noalloc(bemgpu_ctx_t ctx, bemgpu_tree_t t, bemgpu_tree_t s, const bemgpu_green_t *g,
                                  const bemgpu_options_t *opt, void *dZ, int64_t ldz, void *stream) {
  if (!ctx || !t || !s || !g || !dZ) return bem_fail(ctx, BEMGPU_ERR_ARG, "zts_noalloc: null argument");
  if (t->geom != s->geom) return bem_fail(ctx, BEMGPU_ERR_ARG, "zts_noalloc: t and s must share one geometry");
  if (ldz < 2 * (int64_t)t->nrwg) return bem_fail(ctx, BEMGPU_ERR_ARG, "zts_noalloc: ldz < 2*size(t)");
  if (ctx->device < 0 || ctx->device >= BEM_MAX_DEVICES)
    return bem_fail(ctx, BEMGPU_ERR_ARG, "zts_noalloc: device %d outside 0..%d", ctx->device, BEM_MAX_DEVICES - 1);
  const size_t hbytes = sizeof(HalfPairBlock) * (size_t)t->nrwg * (size_t)s->nrwg;
  if (hbytes > NOALLOC_SCRATCH_BYTES - NOALLOC_NEAR_BYTES)
    return bem_fail(ctx, BEMGPU_ERR_ARG,
                    "zts_noalloc: %d x %d RWGs need %zu bytes of scratch, the fixed scratch holds %zu "
                    "(at most size(t) * size(s) = %zu)",
                    t->nrwg, s->nrwg, hbytes, NOALLOC_SCRATCH_BYTES - NOALLOC_NEAR_BYTES,
                    (NOALLOC_SCRATCH_BYTES - NOALLOC_NEAR_BYTES) / sizeof(HalfPairBlock));
  std::vector<NearPair> pairs;
  bem_build_near_pairs(t, s, pairs);
  if (pairs.size() * sizeof(NearPair) > NOALLOC_NEAR_BYTES)
    return bem_fail(ctx, BEMGPU_ERR_ARG, "zts_noalloc: %zu near pairs exceed the fixed scratch (%zu)", pairs.size(),
                    NOALLOC_NEAR_BYTES / sizeof(NearPair));
  bemgpu_options_t o;
  if (opt) o = *opt; else bemgpu_options_default(&o);
  std::lock_guard<std::mutex> lk(ctx->mu);
  // the scratch is one array per process: calls from several contexts take
  // turns (each call ends with its stream synchronised)
  std::lock_guard<std::mutex> lkrun(g_noalloc_run_mu);
  cudaSetDevice(ctx->device);
  // Set-up, once per device with that device current: the host-side name of
  // the array is not a device address; ask the runtime for the address.
  unsigned char *base = nullptr;
  NoallocTasks *dtask = nullptr;
  {
    std::lock_guard<std::mutex> lk2(g_noalloc_mu);
    if (!g_noalloc_addr[ctx->device]) {
      void *p = nullptr;
      cudaError_t e = cudaGetSymbolAddress(&p, g_noalloc_scratch);
      if (e != cudaSuccess || !p)
        return bem_fail(ctx, BEMGPU_ERR_CUDA, "zts_noalloc: cudaGetSymbolAddress failed: %s", cudaGetErrorString(e));
      void *q = nullptr;
      e = cudaGetSymbolAddress(&q, g_noalloc_task);
      if (e != cudaSuccess || !q)
        return bem_fail(ctx, BEMGPU_ERR_CUDA, "zts_noalloc: cudaGetSymbolAddress failed: %s", cudaGetErrorString(e));
      g_noalloc_addr[ctx->device] = p;
      g_noalloc_task_addr[ctx->device] = q;
    }
    base = (unsigned char *)g_noalloc_addr[ctx->device];
    dtask = (NoallocTasks *)g_noalloc_task_addr[ctx->device];
  }
  int rc = load_tables(ctx);
  if (rc) return rc;
  cudaStream_t st = stream ? (cudaStream_t)stream : ctx->stream;
  NearPair *dnear = reinterpret_cast<NearPair *>(base);
  HalfPairBlock *H = reinterpret_cast<HalfPairBlock *>(base + NOALLOC_NEAR_BYTES);
  if (!pairs.empty())
    BEM_CUDA_TRY(ctx, cudaMemcpyAsync(dnear, pairs.data(), pairs.size() * sizeof(NearPair), cudaMemcpyHostToDevice, st));
  // Every half-pair slot of H has exactly one writer (the pair kernels below),
  // so nothing left by an earlier call needs clearing.
  const FarOpts fo = {o.farThresh6, o.farThresh10, o.farThresh15, o.farThresh21};
  NoallocTasks tasks;
  memset(&tasks, 0, sizeof tasks);
  FillTask &task = tasks.far;
  task.T = t->d_rec;
  task.S = s->d_rec;
  task.H = H;
  task.ntT = t->ntri;
  task.ntS = s->ntri;
  task.ntr = t->nrwg;
  task.far_tx = (s->ntri + 31) / 32;
  task.sym = t == s;
  task.g = to_dev(g);
  const double emax = std::max(t->emax, s->emax);
  const int kind = near_kind(green_kabs(g), emax);
  const int64_t np = (int64_t)pairs.size();
  NearTask &nt = tasks.near;
  nt.T = t->d_rec;
  nt.S = s->d_rec;
  nt.near = dnear;
  nt.nnear = np;
  nt.scale = kind == NEAR_DIRECT ? 1.0 : near_scale(emax);
  nt.ngreen = 1;
  nt.g[0] = near_green(g, nt.scale, false, H, t->nrwg, 0, 0, t->ntri);
  BEM_CUDA_TRY(ctx, cudaMemcpyAsync(dtask, &tasks, sizeof tasks, cudaMemcpyHostToDevice, st));
  launch_far(FILL_FP64, (unsigned)far_tiles_of(task.sym, t->ntri, s->ntri, 4), 4, st, &dtask->far, 1, fo);
  ctx->launches++;
  if (np > 0) {
    const int nb = (int)std::min<int64_t>((np + NEAR_WARPS - 1) / NEAR_WARPS, (int64_t)ctx->num_sms * 16);
    launch_near(false, 2, kind, nb, st, &dtask->near, 1, np, 0);
    ctx->launches++;
  }
  dim3 gblk(128);
  dim3 ggrd((t->nrwg + 127) / 128, s->nrwg);
  gather_z_kernel<false><<<ggrd, gblk, 0, st>>>(H, t->nrwg, s->nrwg, to_zdev(g), (double *)dZ, ldz);
  ctx->launches++;
  BEM_CUDA_TRY(ctx, cudaGetLastError());
  // The near-pair list was copied from host memory owned by this call.
  BEM_CUDA_TRY(ctx, cudaStreamSynchronize(st));
  return BEMGPU_OK;
}
