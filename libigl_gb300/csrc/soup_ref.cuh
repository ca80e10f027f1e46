// Moments of the reference-tree soup build (soup_ref.cu): the per-triangle and
// per-node data in T = float, bit for bit the reference's (compiled in
// soup_ref.cu without fused multiply-adds), or T = double (soup_ref64.cu, with
// them), and the kernels that compute them.
#pragma once

#include <cuda_runtime.h>

#include <cstdint>

#include "gwn_common.cuh"
#include "soup.cuh"

namespace gwn {
namespace refsoup {

constexpr uint32_t kEmpty = 0xffffffffu;     // empty child lane
constexpr uint32_t kInternal = 0x80000000u;  // child lane that is a node

struct Box {
  float lo[3], hi[3];
};

// Counters of the build; the fields before ntop are zeroed for every depth, those
// before max_n each time a depth's rounds run.
struct BuildCounts {
  uint32_t lists[3][3];  // per round: parts for a warp, a CTA, the whole GPU
  uint32_t nwaiting;     // nodes that wait for nthElement
  uint32_t max_n;        // the largest node of the next depth
  uint32_t ntop, nsub, nodes, max_depth, unbounded;
};

// A subtree of at most kSub boxes: the boxes idx[start .. start + n).
struct SubRoot {
  uint32_t start, n, depth;
  Box all;
};
// What the subtree kernel leaves per subtree node, at [start + local id]
// (local ids breadth-first; a subtree of n boxes has at most n - 1 nodes):
// the children (kSubNode | local id, local box index, kSubNone) and the
// node's depth-first number, slot and first leaf slot relative to the
// subtree's root, and the slots and items below it.
struct SubNode {
  uint16_t child[4];
  uint16_t pre, slot, item, nslots, nitems, pad;
};
constexpr uint16_t kSubNode = 0x8000u, kSubNone = 0xffffu;
struct SubTotals {
  uint32_t nodes, slots, levels;
};
struct Place {
  uint32_t pre, slot, item;
};

inline unsigned blocks_for(uint64_t n, unsigned t = 256) { return (unsigned)((n + t - 1) / t); }

// A triangle's box as UT_SolidAngle::init makes it: initBounds(v0), then
// enlargeBounds(v1), enlargeBounds(v2) with SYSmin / SYSmax
// (FWNFS.h:255-256, 4023-4028).  (a > b) ? b : a keeps a NaN of the first
// vertex and drops one of a later vertex.
template <typename T>
__device__ __forceinline__ void tri_box(const T* a, const T* b, const T* c, T* lo, T* hi) {
  for (int d = 0; d < 3; ++d) {
    lo[d] = a[d];
    hi[d] = a[d];
    lo[d] = lo[d] > b[d] ? b[d] : lo[d];
    hi[d] = hi[d] < b[d] ? b[d] : hi[d];
    lo[d] = lo[d] > c[d] ? c[d] : lo[d];
    hi[d] = hi[d] < c[d] ? c[d] : hi[d];
  }
}

// ------------------------------------------------------------- moments --
// Per-node data as the reference's post() returns it to the parent (about
// the node's own average point P), in T = float (the reference's values) or
// double.
// Aligned so that it moves in words of two values: threads read their
// children's data at unrelated places, and L1 does not hold the lines between
// one scalar load and the next (FP64 subtree merges of 1.3M triangles: 1089 ->
// 990 us).
template <typename T>
struct alignas(2 * sizeof(T)) Loc {
  T lo[3], hi[3];
  T P[3], areaP[3], N[3], area;
  T Nii[3], Nxy, Nyx, Nyz, Nzy, Nzx, Nxz;
  T Niii[3], perm, c2[6];
};
constexpr int kLocWords = 18;
static_assert(sizeof(Loc<double>) == kLocWords * 16 && sizeof(Loc<float>) == kLocWords * 8, "");

__device__ __forceinline__ Loc<double> load_loc(const Loc<double>* p) {
  Loc<double> r;
  const double2* a = reinterpret_cast<const double2*>(p);
  double2* b = reinterpret_cast<double2*>(&r);
#pragma unroll
  for (int i = 0; i < kLocWords; ++i) b[i] = a[i];
  return r;
}
__device__ __forceinline__ Loc<float> load_loc(const Loc<float>* p) {
  Loc<float> r;
  const float2* a = reinterpret_cast<const float2*>(p);
  float2* b = reinterpret_cast<float2*>(&r);
#pragma unroll
  for (int i = 0; i < kLocWords; ++i) b[i] = a[i];
  return r;
}

template <typename T>
__device__ void zero_loc(Loc<T>& L) {
  T* p = reinterpret_cast<T*>(&L);
  for (size_t i = 0; i < sizeof(Loc<T>) / sizeof(T); ++i) p[i] = T(0);
}

// Second-moment integrals of one triangle (FWNFS.h:6727-6884), corners
// A <= B <= C along axis i.
template <typename T>
__device__ void tri_integrals(const T* A, const T* B, const T* C, const T* P, T area, T* ii, T* ij,
                              T* ik, int i) {
  T oab[3], oac[3], ocb[3];
  for (int d = 0; d < 3; ++d) {
    oab[d] = B[d] - A[d];
    oac[d] = C[d] - A[d];
    ocb[d] = B[d] - C[d];
  }
  const int j = (i == 2) ? 0 : i + 1, k = (j == 2) ? 0 : j + 1;
  T t, jd, kd, sa, sc;
  if constexpr (sizeof(T) == 4) {
    t = oab[i] / oac[i];
    jd = t * oac[j] - oab[j];
    kd = t * oac[k] - oab[k];
    const T xa0 = jd * oab[k] - kd * oab[j], xa1 = kd * oab[i], xa2 = jd * oab[i];
    const T xc0 = jd * ocb[k] - kd * ocb[j], xc1 = kd * ocb[i], xc2 = jd * ocb[i];
    sa = sqrt(xa0 * xa0 + xa1 * xa1 + xa2 * xa2);
    sc = sqrt(xc0 * xc0 + xc1 * xc1 + xc2 * xc2);
  } else {
    // sa and sc are twice the areas of the parts that the plane through B cuts
    // off at A and C: t and 1 - t of the triangle (two square roots and 20
    // operations less on the FP64 pipe that bounds the items: 920 -> 701 us for
    // 1.3M triangles)
    const T inv = T(1) / oac[i];
    T rest = -ocb[i] * inv;
    t = oab[i] * inv;
    if (isinf(inv)) {  // an extent below 5.6e-309
      t = oab[i] / oac[i];
      rest = -ocb[i] / oac[i];
    }
    jd = t * oac[j] - oab[j];
    kd = t * oac[k] - oab[k];
    sa = 2 * area * t;
    sc = 2 * area * rest;
  }
  const T Pai = A[i] - P[i], Pci = C[i] - P[i];
  const T two3 = T(2.0 / 3.0), one3 = T(1.0 / 3.0), half = T(0.5), qtr = T(0.25);
  const T ia = sa * (half * Pai * Pai + two3 * Pai * oab[i] + qtr * oab[i] * oab[i]);
  const T ic = sc * (half * Pci * Pci + two3 * Pci * ocb[i] + qtr * ocb[i] * ocb[i]);
  *ii = ia + ic;
  for (int s = 0; s < 2; ++s) {
    T* out = s == 0 ? ij : ik;
    if (!out) continue;
    const int jk = s == 0 ? j : k;
    const T df = s == 0 ? jd : kd;
    const T mid = B[jk] + half * df;
    const T am = mid - A[jk], cm = mid - C[jk];
    const T Paj = A[jk] - P[jk], Pcj = C[jk] - P[jk];
    const T ija = sa * (half * Pai * Paj + one3 * Pai * am + one3 * Paj * oab[i] + qtr * oab[i] * am);
    const T ijc = sc * (half * Pci * Pcj + one3 * Pci * cm + one3 * Pcj * ocb[i] + qtr * ocb[i] * cm);
    *out = ija + ijc;
  }
}

// Per-triangle data (the reference's item(), FWNFS.h:6668-6890).
template <typename T>
__device__ void item_loc(const T* a, const T* b, const T* c, int order, Loc<T>& L) {
  zero_loc(L);
  tri_box(a, b, c, L.lo, L.hi);
  T ab[3], ac[3];
  for (int d = 0; d < 3; ++d) {
    ab[d] = b[d] - a[d];
    ac[d] = c[d] - a[d];
  }
  L.N[0] = T(0.5) * (ab[1] * ac[2] - ab[2] * ac[1]);
  L.N[1] = T(0.5) * (ab[2] * ac[0] - ab[0] * ac[2]);
  L.N[2] = T(0.5) * (ab[0] * ac[1] - ab[1] * ac[0]);
  const T area = sqrt(L.N[0] * L.N[0] + L.N[1] * L.N[1] + L.N[2] * L.N[2]);
  const T third = T(1) / T(3);
  for (int d = 0; d < 3; ++d) {
    L.P[d] = ((a[d] + b[d]) + c[d]) * third;
    L.areaP[d] = L.P[d] * area;
  }
  L.area = area;
  if (order < 2 || area == T(0)) return;
  const T inv = T(1) / area;
  const T n[3] = {L.N[0] * inv, L.N[1] * inv, L.N[2] * inv};
  const T* v[3] = {a, b, c};
  int o[3][3];
  for (int ax = 0; ax < 3; ++ax) {
    int* q = o[ax];
    q[0] = 0;
    q[1] = 1;
    q[2] = 2;
    int t;
    if (a[ax] > b[ax]) { t = q[0]; q[0] = q[1]; q[1] = t; }
    if (v[q[0]][ax] > c[ax]) { t = q[0]; q[0] = q[2]; q[2] = t; }
    if (v[q[1]][ax] > v[q[2]][ax]) { t = q[1]; q[1] = q[2]; q[2] = t; }
  }
  const T dx = v[o[0][2]][0] - v[o[0][0]][0];
  const T dy = v[o[1][2]][1] - v[o[1][0]][1];
  const T dz = v[o[2][2]][2] - v[o[2][0]][2];
  T xx = 0, xy = 0, yy = 0, yz = 0, zz = 0, zx = 0;
  if (dx > T(0))
    tri_integrals(v[o[0][0]], v[o[0][1]], v[o[0][2]], L.P, area, &xx,
                  (dx >= dy && dy > T(0)) ? &xy : (T*)nullptr,
                  (dx >= dz && dz > T(0)) ? &zx : (T*)nullptr, 0);
  if (dy > T(0))
    tri_integrals(v[o[1][0]], v[o[1][1]], v[o[1][2]], L.P, area, &yy,
                  (dy >= dz && dz > T(0)) ? &yz : (T*)nullptr,
                  (dx < dy && dx > T(0)) ? &xy : (T*)nullptr, 1);
  if (dz > T(0))
    tri_integrals(v[o[2][0]], v[o[2][1]], v[o[2][2]], L.P, area, &zz,
                  (dx < dz && dx > T(0)) ? &zx : (T*)nullptr,
                  (dy < dz && dy > T(0)) ? &yz : (T*)nullptr, 2);
  L.Niii[0] = xx * n[0];
  L.Niii[1] = yy * n[1];
  L.Niii[2] = zz * n[2];
  L.perm = T(2) * (n[0] * yz + n[1] * zx + n[2] * xy);
  const T Nxxy = n[0] * xy, Nxxz = n[0] * zx, Nyyz = n[1] * yz, Nyyx = n[1] * xy, Nzzx = n[2] * zx,
          Nzzy = n[2] * yz;
  L.c2[0] = T(2) * Nxxy + n[1] * xx;
  L.c2[1] = T(2) * Nxxz + n[2] * xx;
  L.c2[2] = T(2) * Nyyz + n[2] * yy;
  L.c2[3] = T(2) * Nyyx + n[0] * yy;
  L.c2[4] = T(2) * Nzzx + n[0] * zz;
  L.c2[5] = T(2) * Nzzy + n[1] * zz;
}

// A lane's maxP^2: the farthest box corner coordinate from P, squared and
// summed (FWNFS.h:6940-6955).
template <typename T>
__device__ __forceinline__ T lane_maxP2(const Loc<T>& C) {
  T m2 = T(0);
  for (int d = 0; d < 3; ++d) {
    const T a = C.P[d] - C.lo[d], b = C.hi[d] - C.P[d];
    const T mx = a > b ? a : b;
    m2 = d == 0 ? mx * mx : m2 + mx * mx;
  }
  return m2;
}

// A node's own data from its children's (the reference's post(),
// FWNFS.h:6892-7118), in the reference's order of operations.
template <typename T>
__device__ __forceinline__ void merge_loc(const Loc<T>* const* ch, int nch, int order, Loc<T>& out) {
  // the sums over the children, each in lane order
  zero_loc(out);
#pragma unroll 1
  for (int i = 0; i < nch; ++i) {
    const Loc<T> C = load_loc(ch[i]);
    if (i == 0) {
      for (int d = 0; d < 3; ++d) {
        out.N[d] = C.N[d];
        out.areaP[d] = C.areaP[d];
        out.lo[d] = C.lo[d];
        out.hi[d] = C.hi[d];
      }
      out.area = C.area;
      if (order < 1) continue;
      for (int d = 0; d < 3; ++d) {
        out.Nii[d] = C.Nii[d];
        out.Niii[d] = C.Niii[d];
      }
      out.perm = C.perm;
      for (int k = 0; k < 6; ++k) out.c2[k] = C.c2[k];
      continue;
    }
    for (int d = 0; d < 3; ++d) {
      out.N[d] += C.N[d];
      out.areaP[d] += C.areaP[d];
      out.lo[d] = out.lo[d] < C.lo[d] ? out.lo[d] : C.lo[d];
      out.hi[d] = out.hi[d] > C.hi[d] ? out.hi[d] : C.hi[d];
    }
    out.area += C.area;
    if (order < 1) continue;
    for (int d = 0; d < 3; ++d) {
      out.Nii[d] += C.Nii[d];
      out.Niii[d] += C.Niii[d];
    }
    out.perm += C.perm;
    for (int k = 0; k < 6; ++k) out.c2[k] += C.c2[k];
  }
  if (out.area > T(0)) {
    const T inv = T(1) / out.area;
    for (int d = 0; d < 3; ++d) out.P[d] = out.areaP[d] * inv;
  } else {
    for (int d = 0; d < 3; ++d) out.P[d] = T(0.5) * (out.lo[d] + out.hi[d]);
  }
  if (order < 1) return;
  // then the children's shifts to the common point
#pragma unroll 1
  for (int i = 0; i < nch; ++i) {
    const Loc<T> C = load_loc(ch[i]);
    const T dx = C.P[0] - out.P[0], dy = C.P[1] - out.P[1], dz = C.P[2] - out.P[2];
    const T* n = C.N;
    out.Nii[0] += n[0] * dx;
    out.Nii[1] += n[1] * dy;
    out.Nii[2] += n[2] * dz;
    const T Nxy = C.Nxy + n[0] * dy, Nyx = C.Nyx + n[1] * dx, Nyz = C.Nyz + n[1] * dz,
            Nzy = C.Nzy + n[2] * dy, Nzx = C.Nzx + n[2] * dx, Nxz = C.Nxz + n[0] * dz;
    out.Nxy += Nxy;
    out.Nyx += Nyx;
    out.Nyz += Nyz;
    out.Nzy += Nzy;
    out.Nzx += Nzx;
    out.Nxz += Nxz;
    if (order >= 2) {
      const T dd[3] = {dx, dy, dz};
      for (int d = 0; d < 3; ++d) out.Niii[d] += T(2) * dd[d] * C.Nii[d] + dd[d] * dd[d] * n[d];
      out.perm += (dx * (Nyz + Nzy) + dy * (Nzx + Nxz) + dz * (Nxy + Nyx));
      out.c2[0] += T(2) * (dy * C.Nii[0] + dx * C.Nxy + n[0] * dx * dy) + T(2) * C.Nyx * dx + n[1] * dx * dx;
      out.c2[1] += T(2) * (dz * C.Nii[0] + dx * C.Nxz + n[0] * dx * dz) + T(2) * C.Nzx * dx + n[2] * dx * dx;
      out.c2[2] += T(2) * (dz * C.Nii[1] + dy * C.Nyz + n[1] * dy * dz) + T(2) * C.Nzy * dy + n[2] * dy * dy;
      out.c2[3] += T(2) * (dx * C.Nii[1] + dy * C.Nyx + n[1] * dy * dx) + T(2) * C.Nxy * dy + n[0] * dy * dy;
      out.c2[4] += T(2) * (dx * C.Nii[2] + dz * C.Nzx + n[2] * dz * dx) + T(2) * C.Nxz * dz + n[0] * dz * dz;
      out.c2[5] += T(2) * (dy * C.Nii[2] + dz * C.Nzy + n[2] * dz * dy) + T(2) * C.Nyz * dz + n[1] * dz * dz;
    }
  }
}

__device__ __forceinline__ void load_tri(const double* __restrict__ V, int64_t nV, const int32_t* __restrict__ F,
                         uint32_t f, double* v) {
  for (int c = 0; c < 3; ++c) {
    int32_t i = F[(int64_t)f * 3 + c];
    if (i < 0 || i >= nV) i = 0;  // reported at the box pass; excluded there
    for (int d = 0; d < 3; ++d) v[c * 3 + d] = V[(int64_t)i * 3 + d];
  }
}

// What the kernels below read and write, in T's precision.
struct MomentArgs {
  // items: by leaf slot
  int64_t m;
  const int32_t* tri_index;
  const uint32_t* item_slot;
  const double* V;
  int64_t nV;
  const int32_t* F;
  int order;
  // nodes: by depth-first number; kid: an item's leaf slot or kInternal | node
  const uint4* kid;
  const uint2* slots;
  // subtrees and the nodes above them
  uint32_t nsub;
  const SubRoot* subs;
  const SubTotals* totals;
  const Place* sub_place;
  const SubNode* sn;
  const uint16_t* lev;
  const Place* place;
  const uint32_t* level;  // host: depth d of the top is [level[d], level[d + 1])
  int top_depths;
  // results
  Loc<float>* L32;  // items at [0, m), nodes at [m, m + nodes)
  Loc<double>* L64;
  SoupNodeF* nf;
  SoupNodeD* nd;
  float4* tf;
  double* td;
  BuildCounts* bc;
};

// Writes the walk's record of a slot.
__device__ __forceinline__ void write_record(const MomentArgs& A, const Loc<float>& C,
                                             uint32_t slot, int link, bool root) {
  SoupNodeF R;
  R.a = make_float4(C.P[0], C.P[1], C.P[2], root ? INFINITY : lane_maxP2(C));
  // the reference's FP32 moments (with its FP32 sums of the mixed terms),
  // packed into the walk's far-field forms
  double N[3], Nii[3], Niii[3], c2[6];
  for (int d = 0; d < 3; ++d) {
    N[d] = C.N[d];
    Nii[d] = C.Nii[d];
    Niii[d] = C.Niii[d];
  }
  for (int k = 0; k < 6; ++k) c2[k] = C.c2[k];
  pack_far32(R, N, Nii, (double)(C.Nxy + C.Nyx), (double)(C.Nyz + C.Nzy),
             (double)(C.Nzx + C.Nxz), Niii, (double)C.perm, c2, link);
  A.nf[slot] = R;
}

// Sets bc->unbounded where a value is not finite or beyond 1e100 in magnitude
// (gwn_soup_impl::moments_bounded); the bit patterns of non-negative doubles
// compare as the values do, NaN above all.
__device__ __forceinline__ bool beyond(double x) {
  return (__double_as_longlong(x) & 0x7fffffffffffffffll) > __double_as_longlong(1e100);
}
__device__ __forceinline__ void write_record(const MomentArgs& A, const Loc<double>& C,
                                             uint32_t slot, int link, bool root) {
  SoupNodeD D;
  for (int d = 0; d < 3; ++d) D.P[d] = C.P[d];
  D.maxP2 = root ? (double)INFINITY : lane_maxP2(C);
  pack_far64(D, C.N, C.Nii, C.Nxy + C.Nyx, C.Nyz + C.Nzy, C.Nzx + C.Nxz, C.Niii, C.perm, C.c2);
  bool bad = beyond(D.S);
  for (int d = 0; d < 3; ++d) bad |= beyond(D.N[d]) || beyond(D.L[d]);
  for (int k = 0; k < 5; ++k) bad |= beyond(D.A[k]);
  for (int k = 0; k < 7; ++k) bad |= beyond(D.K[k]);
  D.link = link;
  A.nd[slot] = D;
  if (bad) A.bc->unbounded = 1;
}


template <typename T>
__device__ __forceinline__ Loc<T>* locs(const MomentArgs& A) {
  if constexpr (sizeof(T) == 4) return A.L32;
  else return A.L64;
}

// Items: one thread per leaf slot computes the triangle's data and records and
// leaves the data for the merges.  (One thread per node did all this for its
// items, in both precisions, and kept up to four children's data in local
// memory: 4.16 ms for 1.3M triangles.)
template <typename T>
__global__ void __launch_bounds__(128) items_kernel(MomentArgs A) {
  const int64_t ib = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (ib >= A.m) return;
  double v[9];
  load_tri(A.V, A.nV, A.F, (uint32_t)A.tri_index[ib], v);
  T w[9];
  for (int k = 0; k < 9; ++k) w[k] = (T)v[k];
  Loc<T> C;
  item_loc<T>(w, w + 3, w + 6, A.order, C);
  write_record(A, C, A.item_slot[ib], (int)~ib, false);
  locs<T>(A)[ib] = C;
  if constexpr (sizeof(T) == 4) {
    A.tf[ib * 3 + 0] = make_float4(w[0], w[1], w[2], w[3]);
    A.tf[ib * 3 + 1] = make_float4(w[4], w[5], w[6], w[7]);
    A.tf[ib * 3 + 2] = make_float4(w[8], tri_screen_slack(v), 0.f, 0.f);
  } else {
    for (int k = 0; k < 9; ++k) A.td[ib * 9 + k] = v[k];
  }
}

// One node p (depth-first number): merges its children's data and writes its
// slot's record.
template <typename T>
__device__ __forceinline__ void merge_at(const MomentArgs& A, uint32_t p) {
  const uint4 kid = A.kid[p];
  const uint2 sl = A.slots[p];
  const uint32_t k[4] = {kid.x, kid.y, kid.z, kid.w};
  Loc<T>* L = locs<T>(A);
  const Loc<T>* ch[4];
  int nch = 0;
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    ch[i] = L;
    if (k[i] == kEmpty) continue;
    ch[i] = L + ((k[i] & kInternal) ? (uint32_t)A.m + (k[i] & ~kInternal) : k[i]);
    nch = i + 1;
  }
  Loc<T> C;
  merge_loc<T>(ch, nch, A.order, C);
  L[A.m + p] = C;
  write_record(A, C, sl.x, (int)sl.y, p == 0);
}

// All nodes of a subtree, deepest depth first; one CTA per subtree.
template <typename T>
__global__ void __launch_bounds__(128) sub_merge_kernel(MomentArgs A) {
  const uint32_t start = A.subs[blockIdx.x].start, pre = A.sub_place[blockIdx.x].pre;
  for (uint32_t d = A.totals[blockIdx.x].levels; d-- > 0;) {
    for (uint32_t x = A.lev[start + d] + threadIdx.x; x < A.lev[start + d + 1]; x += blockDim.x)
      merge_at<T>(A, pre + A.sn[start + x].pre);
    __syncthreads();
  }
}

// One depth of the nodes above the subtrees.
template <typename T>
__global__ void __launch_bounds__(128) top_merge_kernel(MomentArgs A, uint32_t lb, uint32_t le) {
  const uint32_t x = lb + blockIdx.x * blockDim.x + threadIdx.x;
  if (x < le) merge_at<T>(A, A.place[x].pre);
}

template <typename T>
void launch_moments(const MomentArgs& A, cudaStream_t st) {
  launch_kernel(items_kernel<T>, blocks_for(A.m, 128), 128, 0, st, A);
  launch_kernel(sub_merge_kernel<T>, A.nsub, 128, 0, st, A);
  for (int d = A.top_depths - 1; d >= 0; --d)
    launch_kernel(top_merge_kernel<T>, blocks_for(A.level[d + 1] - A.level[d], 128), 128, 0, st, A,
                  A.level[d], A.level[d + 1]);
}

// The FP64 moments (soup_ref64.cu).
void launch_moments64(const MomentArgs& A, cudaStream_t st);

}  // namespace refsoup
}  // namespace gwn
