// Device layout of a built triangle soup (the state behind gwn_soup).
#pragma once

#include <cuda_runtime.h>

#include <cstdint>
#include <cstring>

#include "gwn_common.cuh"

namespace gwn {

// 96-byte FP32 node record, read by the mixed-precision walk.
//   a: P (average point) xyz, maxPDist2
//   b: N xyz, A_xx     c: A_yy, A_zz, A_xy, A_xz     d: A_yz, K_xxx, K_yyy, K_zzz
//   e: K_xxy, K_xxz, K_xyy, K_yyz     f: K_xzz, K_yzz, K_xyz, link (int bits)
// A and K are the coefficients of the far field's order-1 quadratic and
// order-2 cubic forms in the unit direction (pack_far32 below).
// link >= 0: internal node, index one past its subtree (pre-order);
// link < 0: leaf, triangle slot ~link.
struct __align__(32) SoupNodeF {
  float4 a, b, c, d, e, f;
};
static_assert(sizeof(SoupNodeF) == 96, "96-byte records: a..b, c..d, e..f are 32-byte aligned");

// The far field of FWNFS.h:7195-7251 with q = (x - P)/|x - P|,
// m1 = 1/|x - P|, m2 = m1^2:
//   omega = -m2 q.N
//         + m2 m1 (S - 3 (sum_i q_i^2 Nii + q_x q_y Nxy_yx + ...))          (order 1)
//         + m2 m1^2 (1.5 q.L - 7.5 (sum_i q_i^3 Niii + q_x q_y q_z perm + ...)) (order 2)
// with S = Nxx + Nyy + Nzz and L_i = 3 Niii + the two c2 sums of FWNFS.h:
// 7228-7233.  Since |q| = 1, S = S |q|^2 and q.L = (q.L)|q|^2, so the order-1
// bracket is a quadratic form A(q) and the order-2 bracket a cubic form K(q):
//   omega = m2 (m1 (A(q) + m1 K(q)) - q.N),
// 6 + 10 coefficients in place of the 9 + 10 moments, and about half the
// operations per evaluation.  The coefficients are formed here in FP64 from
// the node's moments and rounded once.
__host__ __device__ inline void pack_far32(SoupNodeF& R, const double N[3], const double Nii[3],
                                           double Nxy_yx, double Nyz_zy, double Nzx_xz,
                                           const double Niii[3], double perm, const double c2[6],
                                           int link) {
  const double S = Nii[0] + Nii[1] + Nii[2];
  const double Lx = 3 * Niii[0] + (c2[3] + c2[4]);
  const double Ly = 3 * Niii[1] + (c2[5] + c2[0]);
  const double Lz = 3 * Niii[2] + (c2[1] + c2[2]);
  R.b = make_float4((float)N[0], (float)N[1], (float)N[2], (float)(S - 3 * Nii[0]));
  R.c = make_float4((float)(S - 3 * Nii[1]), (float)(S - 3 * Nii[2]), (float)(-3 * Nxy_yx),
                    (float)(-3 * Nzx_xz));
  R.d = make_float4((float)(-3 * Nyz_zy), (float)(1.5 * Lx - 7.5 * Niii[0]),
                    (float)(1.5 * Ly - 7.5 * Niii[1]), (float)(1.5 * Lz - 7.5 * Niii[2]));
  R.e = make_float4((float)(1.5 * Ly - 7.5 * c2[0]), (float)(1.5 * Lz - 7.5 * c2[1]),
                    (float)(1.5 * Lx - 7.5 * c2[3]), (float)(1.5 * Lz - 7.5 * c2[2]));
  float lf;
  memcpy(&lf, &link, sizeof(float));
  R.f = make_float4((float)(1.5 * Lx - 7.5 * c2[4]), (float)(1.5 * Ly - 7.5 * c2[5]),
                    (float)(-7.5 * perm), lf);
}

// 192-byte FP64 node record (plain FP64 walk, FP64 re-checks): the same forms
// in FP64.  The quadratic form has no trace and the cubic form no Laplacian
// (both brackets are harmonic), so A_zz = -(A_xx + A_yy), K_xzz = -(3 K_xxx +
// K_xyy), K_yzz = -(3 K_yyy + K_xxy) and K_zzz = -(K_xxz + K_yyz) / 3 are not
// stored; S and L, the parts of the moments that the forms do not hold, are
// kept for gwn_soup_export.
struct __align__(16) SoupNodeD {
  double P[3], maxP2;
  double N[3];
  double A[5];  // xx yy xy xz yz
  double K[7];  // xxx yyy xxy xxz xyy yyz xyz
  double S, L[3];
  long long link;
};
static_assert(sizeof(SoupNodeD) == 24 * sizeof(double), "node record layout");

__host__ __device__ inline void pack_far64(SoupNodeD& D, const double N[3], const double Nii[3],
                                           double Nxy_yx, double Nyz_zy, double Nzx_xz,
                                           const double Niii[3], double perm, const double c2[6]) {
  D.S = Nii[0] + Nii[1] + Nii[2];
  D.L[0] = 3 * Niii[0] + (c2[3] + c2[4]);
  D.L[1] = 3 * Niii[1] + (c2[5] + c2[0]);
  D.L[2] = 3 * Niii[2] + (c2[1] + c2[2]);
  for (int d = 0; d < 3; ++d) D.N[d] = N[d];
  D.A[0] = D.S - 3 * Nii[0];
  D.A[1] = D.S - 3 * Nii[1];
  D.A[2] = -3 * Nxy_yx;
  D.A[3] = -3 * Nzx_xz;
  D.A[4] = -3 * Nyz_zy;
  D.K[0] = 1.5 * D.L[0] - 7.5 * Niii[0];
  D.K[1] = 1.5 * D.L[1] - 7.5 * Niii[1];
  D.K[2] = 1.5 * D.L[1] - 7.5 * c2[0];
  D.K[3] = 1.5 * D.L[2] - 7.5 * c2[1];
  D.K[4] = 1.5 * D.L[0] - 7.5 * c2[3];
  D.K[5] = 1.5 * D.L[2] - 7.5 * c2[2];
  D.K[6] = -7.5 * perm;
}

// The moments of a record, m = {N, Nii, Nxy_yx, Nyz_zy, Nzx_xz, Niii, perm,
// c2}: 19 values.
inline void unpack_far64(const SoupNodeD& D, double m[19]) {
  for (int d = 0; d < 3; ++d) m[d] = D.N[d];
  m[3] = (D.S - D.A[0]) / 3;
  m[4] = (D.S - D.A[1]) / 3;
  m[5] = (D.S + (D.A[0] + D.A[1])) / 3;
  m[6] = -D.A[2] / 3;
  m[7] = -D.A[4] / 3;
  m[8] = -D.A[3] / 3;
  const double Kzzz = -(D.K[3] + D.K[5]) / 3, Kxzz = -(3 * D.K[0] + D.K[4]),
               Kyzz = -(3 * D.K[1] + D.K[2]);
  auto u = [](double L, double K) { return (1.5 * L - K) / 7.5; };
  m[9] = u(D.L[0], D.K[0]);
  m[10] = u(D.L[1], D.K[1]);
  m[11] = u(D.L[2], Kzzz);
  m[12] = -D.K[6] / 7.5;
  m[13] = u(D.L[1], D.K[2]);
  m[14] = u(D.L[2], D.K[3]);
  m[15] = u(D.L[2], D.K[5]);
  m[16] = u(D.L[0], D.K[4]);
  m[17] = u(D.L[0], Kxzz);
  m[18] = u(D.L[1], Kyzz);
}

#ifdef __CUDACC__
// Error slack of the FP32 closest-point screen for one triangle (v: three
// FP64 corners; distance.cu): 32 u (|e1|^2 |e2|^2 / |e1 x e2|^2) L + 8 u
// max|v|, u = 2^-24, L the longest edge; infinite for a (near) degenerate one.
__device__ inline float tri_screen_slack(const double* v) {
  double e1[3], e2[3], e3[3], cr[3];
  double l1 = 0, l2 = 0, l3 = 0, vm = 0;
  for (int d = 0; d < 3; ++d) {
    e1[d] = v[3 + d] - v[d];
    e2[d] = v[6 + d] - v[d];
    e3[d] = v[6 + d] - v[3 + d];
    l1 += e1[d] * e1[d];
    l2 += e2[d] * e2[d];
    l3 += e3[d] * e3[d];
    vm = fmax(vm, fmax(fabs(v[d]), fmax(fabs(v[3 + d]), fabs(v[6 + d]))));
  }
  cr[0] = e1[1] * e2[2] - e1[2] * e2[1];
  cr[1] = e1[2] * e2[0] - e1[0] * e2[2];
  cr[2] = e1[0] * e2[1] - e1[1] * e2[0];
  const double den = cr[0] * cr[0] + cr[1] * cr[1] + cr[2] * cr[2];
  const double cond = den > 0 ? l1 * l2 / den : INFINITY;
  const double u = 5.9604644775390625e-08;
  if (cond < 1e6) return (float)(32 * u * cond * sqrt(fmax(l1, fmax(l2, l3))) + 8 * u * vm);
  return INFINITY;
}
#endif

#ifdef __CUDACC__
// Frame of a search node's box.  With n the unit vector of stereographic
// coordinates (p, r), p^2 + r^2 <= 1, and k = 2 / (1 + p^2 + r^2):
//   n = (k p, k r, k - 1), u = (1 - k p^2, -k p r, -k p), w = (-k p r, 1 - k r^2, -k r),
// so that with g = k (p x + r y + z) the coordinates of (x, y, z) are
// (x - p g, y - r g, g - z).  p = r = 0 is the frame of the axes.  p and r are
// held as 16-bit multiples of 2^-15 (exact in FP32).  k is the same FP32 number
// wherever a frame is read; its relative error e leaves the map's norm at most
// 1 + 2 e, 5e-7 with the approximate reciprocal.
struct SearchFrame {
  float p, r, k;
  __device__ __forceinline__ explicit SearchFrame(float bits) {
    const uint32_t b = __float_as_uint(bits);
    p = fmaf(__uint_as_float(0x4b000000u | (b & 0xffffu)), 0x1p-15f, -257.f);
    r = fmaf(__uint_as_float(0x4b000000u | (b >> 16)), 0x1p-15f, -257.f);
    float s = fmaf(p, p, fmaf(r, r, 1.f));
    asm("rcp.approx.f32 %0, %1;" : "=f"(k) : "f"(s));
    k *= 2.f;
  }
  // Coordinates of a point within 13 u max(|x|, |y|, |z|) each, u = 2^-24.
  __device__ __forceinline__ float3 operator()(float x, float y, float z) const {
    const float g = k * fmaf(p, x, fmaf(r, y, z));
    return make_float3(fmaf(-p, g, x), fmaf(-r, g, y), g - z);
  }
  // The bits of the frame whose third axis is nearest to +-n; any n will do.
  __device__ static float bits_of(float3 n) {
    const float l = sqrtf(n.x * n.x + n.y * n.y + n.z * n.z);
    float p = 0.f, r = 0.f;
    if (l > 0.f && isfinite(l)) {
      const float q = copysignf(1.f, n.z) / (l + fabsf(n.z));
      p = n.x * q;
      r = n.y * q;
    }
    auto enc = [](float v) {
      return (uint32_t)min(max(__float2int_rz(v * 32768.f), -32767), 32767) + 32768u;
    };
    return __uint_as_float(enc(p) | (enc(r) << 16));
  }
};
#endif

struct gwn_soup_impl {
  int device = 0;
  int order = 2;
  // GWN_TREE_REFERENCE: the reference's 4-wide tree (soup_ref.cu), whose
  // open test is the reference's FP32 one; GWN_TREE_BINNED: the binary
  // tree of soup_tree.cu.
  int tree = GWN_TREE_BINNED;
  int64_t ref_nodes = 0;       // nodes of the 4-wide tree (reference numbering)
  DevMem<uint32_t> ref_child;  // 4 lanes per node, the reference's encoding
  int64_t n_input = 0;   // triangles passed in
  int64_t n = 0;         // triangles kept (finite, valid)
  int64_t nnodes = 0;    // 2n-1
  int max_depth = 0;
  double lo[3] = {0, 0, 0}, hi[3] = {0, 0, 0};  // bbox of kept vertices
  double eps = 0;        // near-field distance: 1e-3 * bbox diagonal
  double cmax = 0;       // max |coordinate| inside the bbox
  DevMem<SoupNodeF> nf;
  DevMem<SoupNodeD> nd;
  DevMem<float4> tf;     // 3 float4 per slot: a.xyz b.x | b.yz c.xy | c.z
  DevMem<double> td;     // 9 doubles per slot
  DevMem<int32_t> tri_index;  // input triangle id per slot
  // Closest-point search nodes, one per internal node of the binary tree in
  // build order (root 0): for each of the two children 2 float4, its box in
  // the frame of SearchFrame and the child (internal index, or ~slot for a
  // leaf): {lo.xyz, child}, {hi.xyz, frame}.
  DevMem<float4> snode;
  // every FP64 moment finite and within 1e100 in magnitude: then no far
  // field at |q - P|^2 >= 1e-100 can overflow, and the plain FP64 walk may
  // queue its far fields (soup_walk.cuh)
  bool moments_bounded = false;
  size_t bytes = 0;
};

// Binary tree over the n triangles vals[0..n) (soup_tree.cu): on return
// vals holds the leaf (slot) order; internal nodes are 0..n-2 (root 0) and
// leaf j is node n-1+j; clo/chi bound the triangles' centroids.  Vertex
// indices outside [0, nV) read vertex 0 (callers report them).
void soup_tree_build(const double* V, int64_t nV, const int32_t* F, int32_t* vals, int n,
                     const double* clo, const double* chi, int32_t* left, int32_t* right,
                     int32_t* parent, cudaStream_t st);

// search_only: what soup_squared_distance reads alone (no moments, no walk
// records), where the tree's depth allows it.
void soup_build(gwn_soup_impl& s, const double* V, int64_t nV, const int32_t* F, int64_t nF,
                int order, bool host_mode, cudaStream_t st, bool search_only = false);
// Whether the depth-first search's stack holds a tree of this depth.
bool soup_search_fits(int max_depth);
// The reference's own 4-wide tree and FP32 moments (soup_ref.cu); fills the
// same walk records (slot 0 the root, then every child lane depth-first),
// without the closest-point search nodes.
void soup_build_ref(gwn_soup_impl& s, const double* V, int64_t nV, const int32_t* F, int64_t nF,
                    int order, bool host_mode, cudaStream_t st);
// The binned tree over the triangles of a GWN_TREE_REFERENCE soup (its
// slot-ordered FP64 corners), for the closest-point search; the search
// tree's triangle ids are the reference soup's leaf slots.
void soup_build_search(const gwn_soup_impl& ref, gwn_soup_impl& search, cudaStream_t st);
// Sets s.moments_bounded from the FP64 records (one reduction, one host read).
void soup_check_moments(gwn_soup_impl& s, cudaStream_t st);
// I[q] <- map[I[q]] where I[q] >= 0.
void soup_remap_index(const int32_t* map, int32_t* I, int64_t n, cudaStream_t st);
// Instrumented mixed walk over FP64 device queries: out7 = {warp steps,
// lane visits, far-field evaluations, FP32 exact triangles, FP64 near-field
// triangles, FP64 decision re-checks, threshold re-evaluations}.
void soup_walk_stats(const gwn_soup_impl& s, float beta, const double* Q, int64_t nQ,
                     unsigned long long* out7, cudaStream_t st);
// Lanes that share a query in a call of nQ queries on a tree of `slots` slots
// (1: 32 queries per warp).  With more than one, the query's FP32 sum is kept
// with its rounding error (soup_walk.cuh, PairSum), because the lanes' terms are
// added in another order, and a served request of that size takes the same sum.
int soup_team_size(int64_t nQ, int64_t slots, int precision);
void soup_eval(const gwn_soup_impl& s, float beta, const void* Q, int q_dtype, int64_t nQ,
               void* W, int w_dtype, int precision, cudaStream_t st);
// Closest triangle of each query (distance.cu): squared distance below
// up_sqr_d (else up_sqr_d and I = -1), input triangle index, closest point.
void soup_squared_distance(const gwn_soup_impl& s, const void* Q, int q_dtype, int64_t nQ,
                           double up_sqr_d, double* sqrD, int32_t* I, double* C,
                           cudaStream_t st);

}  // namespace gwn
