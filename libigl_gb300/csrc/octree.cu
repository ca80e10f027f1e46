// GPU octree build, bit-exact with igl::octree (include/igl/octree.cpp:5-170).
//
// Reference semantics restated: the root cube is the points' AABB (centre =
// (min+max)/2, width = largest extent, :142-153); a cell with more than one
// point and depth < 30000 (:16, :98) gets 8 children whose centres are
// parent + (+-h/2 per axis), h = width/2 (:59-81, :104-113, octant bits x=1,
// y=2, z=4 from `>=` against the parent centre, :32-53); every cell's point
// list is the parent's list filtered in order (:117-122), so lists are
// ascending; child ids are m..m+7 handed out when a cell is visited in
// depth-first pre-order (:100-131).
//
// Device algorithm: points sorted by their octant paths (below, "build from
// sorted paths").  Where points share more octants than that build follows:
//  * level by level, the points of the cells being split form one array of
//    (segment, point) entries in segment order; the octant of each point is
//    found with the same FP64 `>=` tests, and a stable radix sort on
//    segment*8+octant performs every cell's stable partition at once; child
//    cells are emitted with the same FP64 centre recurrence;
//  * a cell whose points can never separate again (all identical, or a
//    centre that no longer moves in FP64 with all points in one octant)
//    would recurse to depth 30000 one octant at a time: such chains are
//    emitted by one thread each instead of one level per launch;
//  * ids: the i-th internal cell in depth-first pre-order owns ids
//    1+8i..8+8i.  Internal cells of different depths nest and cells of one
//    depth have disjoint point ranges, so pre-order is the order of
//    (first point position, depth); one sort of that key gives every rank.
#include <cuda_runtime.h>

#include <algorithm>
#include <vector>

#include "gwn_common.cuh"
#include "octree.cuh"
#include "sort.cuh"

namespace gwn {
namespace {

constexpr int kMaxDepth = 30000;

// Creation-order cell records (SoA).
struct Cells {
  DevBuf<double> c;       // 3 per cell
  DevBuf<double> w;
  DevBuf<int64_t> start;
  DevBuf<int32_t> count;
  DevBuf<int32_t> depth;
  DevBuf<int32_t> parent;
  DevBuf<int32_t> oct;
  int64_t size = 0, cap = 0;

  template <typename T>
  static void grow(DevBuf<T>& b, size_t old_n, size_t new_n, cudaStream_t st) {
    DevBuf<T> nb(new_n, st);
    if (old_n)
      GWN_CUDA(cudaMemcpyAsync(nb.get(), b.get(), old_n * sizeof(T), cudaMemcpyDeviceToDevice, st));
    b = std::move(nb);
  }
  void reserve(int64_t need, cudaStream_t st) {
    if (need <= cap) return;
    int64_t nc = std::max<int64_t>(need, cap * 2 + 64);
    grow(c, (size_t)size * 3, (size_t)nc * 3, st);
    grow(w, (size_t)size, (size_t)nc, st);
    grow(start, (size_t)size, (size_t)nc, st);
    grow(count, (size_t)size, (size_t)nc, st);
    grow(depth, (size_t)size, (size_t)nc, st);
    grow(parent, (size_t)size, (size_t)nc, st);
    grow(oct, (size_t)size, (size_t)nc, st);
    cap = nc;
  }
};

__global__ void root_kernel(const unsigned long long* __restrict__ mm, int64_t n, double* c,
                            double* w, int64_t* start, int32_t* count, int32_t* depth,
                            int32_t* parent, int32_t* oct) {
  double lo[3], hi[3];
  for (int d = 0; d < 3; ++d) {
    lo[d] = n > 0 ? from_ordered_bits(mm[d]) : 0.0;
    hi[d] = n > 0 ? from_ordered_bits(mm[3 + d]) : 0.0;
  }
  for (int d = 0; d < 3; ++d) c[d] = (lo[d] + hi[d]) / 2.0;
  double width = hi[0] - lo[0];
  for (int d = 1; d < 3; ++d) {
    const double e = hi[d] - lo[d];
    if (e > width) width = e;
  }
  *w = width;
  *start = 0;
  *count = (int32_t)n;
  *depth = 0;
  *parent = -1;
  *oct = 0;
}

// min/max over all points (NaN coordinates take part as in a plain compare
// loop: they never win a min/max).
__global__ void point_bbox_kernel(const double* __restrict__ P, int64_t n,
                                  unsigned long long* __restrict__ mm) {
  double lo[3] = {INFINITY, INFINITY, INFINITY}, hi[3] = {-INFINITY, -INFINITY, -INFINITY};
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n;
       i += (int64_t)gridDim.x * blockDim.x)
    for (int d = 0; d < 3; ++d) {
      const double v = P[i * 3 + d];
      lo[d] = fmin(lo[d], v);
      hi[d] = fmax(hi[d], v);
    }
  for (int d = 0; d < 3; ++d) {
    for (int o = 16; o > 0; o >>= 1) {
      lo[d] = fmin(lo[d], __shfl_xor_sync(0xffffffffu, lo[d], o));
      hi[d] = fmax(hi[d], __shfl_xor_sync(0xffffffffu, hi[d], o));
    }
    if ((threadIdx.x & 31) == 0) {
      atomicMin(&mm[d], ordered_bits(lo[d]));
      atomicMax(&mm[3 + d], ordered_bits(hi[d]));
    }
  }
}

__global__ void iota_kernel(int32_t* a, int64_t n) {
  const int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (i < n) a[i] = (int32_t)i;
}

__global__ void fill_i32_kernel(int32_t* a, int64_t n, int32_t v) {
  const int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (i < n) a[i] = v;
}

// Octant of every active entry against its segment's centre; flags whether a
// segment's points occupy one octant only and whether they are all equal.
__global__ void octant_kernel(const double* __restrict__ P, const int32_t* __restrict__ act_pt,
                              const int32_t* __restrict__ act_seg, int64_t M,
                              const int32_t* __restrict__ seg_cell,
                              const int32_t* __restrict__ seg_first,
                              const double* __restrict__ cc, unsigned* __restrict__ key,
                              unsigned* __restrict__ seg_mask, unsigned* __restrict__ seg_diff) {
  const int64_t m = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (m >= M) return;
  const int k = act_seg[m];
  const int cell = seg_cell[k];
  const int32_t p = act_pt[m];
  const double px = P[(int64_t)p * 3], py = P[(int64_t)p * 3 + 1], pz = P[(int64_t)p * 3 + 2];
  int o = 0;
  if (px >= cc[(int64_t)cell * 3 + 0]) o += 1;
  if (py >= cc[(int64_t)cell * 3 + 1]) o += 2;
  if (pz >= cc[(int64_t)cell * 3 + 2]) o += 4;
  key[m] = (unsigned)k * 8u + (unsigned)o;
  // All points of a segment hit the same two words: read first and skip the
  // atomic once the bit is set (at the top levels millions of points share
  // one segment, and same-address atomics serialize).
  const unsigned bit = 1u << o;
  if ((*(volatile unsigned*)&seg_mask[k] & bit) == 0u) atomicOr(&seg_mask[k], bit);
  const int32_t f = act_pt[seg_first[k]];
  if ((px != P[(int64_t)f * 3] || py != P[(int64_t)f * 3 + 1] || pz != P[(int64_t)f * 3 + 2]) &&
      *(volatile unsigned*)&seg_diff[k] == 0u)
    atomicOr(&seg_diff[k], 1u);
}

// Points per child from the sorted keys: each run of equal keys adds its end
// and subtracts its start (two uncontended atomics per run; child_count is
// zero on entry).
__global__ void child_count_kernel(const unsigned* __restrict__ key, int64_t M,
                                   unsigned* __restrict__ child_count) {
  const int64_t m = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (m >= M) return;
  const unsigned k = key[m];
  if (m == 0 || key[m - 1] != k) atomicSub(&child_count[k], (unsigned)m);
  if (m == M - 1 || key[m + 1] != k) atomicAdd(&child_count[k], (unsigned)(m + 1));
}

// Whether the FP64 centre recurrence can no longer move `c` on any axis:
// c + w/4 and c - w/4 both round back to c.
__device__ __forceinline__ bool centre_stuck(const double* c, double w) {
  const double q = __dmul_rn(__dmul_rn(w, 0.5), 0.5);
  for (int d = 0; d < 3; ++d)
    if (__dadd_rn(c[d], q) != c[d] || __dadd_rn(c[d], -q) != c[d]) return false;
  return true;
}

// Emit the 8 children of every segment (thread per (segment, octant)).
// child_state: 0 = leaf, 1 = active next level, 2 = chain.
__global__ void emit_children_kernel(int K, const int32_t* __restrict__ seg_cell,
                                     const int64_t* __restrict__ seg_pstart,
                                     const unsigned* __restrict__ seg_mask,
                                     const unsigned* __restrict__ seg_diff,
                                     const unsigned* __restrict__ child_count, int64_t base,
                                     double* cc, double* cw, int64_t* cstart, int32_t* ccount,
                                     int32_t* cdepth, int32_t* cparent, int32_t* coct,
                                     unsigned* __restrict__ child_state) {
  const int64_t t = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (t >= (int64_t)K * 8) return;
  const int k = (int)(t >> 3), o = (int)(t & 7);
  const int cell = seg_cell[k];
  const double pc[3] = {cc[(int64_t)cell * 3], cc[(int64_t)cell * 3 + 1], cc[(int64_t)cell * 3 + 2]};
  const double h = __dmul_rn(cw[cell], 0.5);
  const double hh = __dmul_rn(h, 0.5);
  int64_t s = seg_pstart[k];
  for (int j = 0; j < o; ++j) s += child_count[(int64_t)k * 8 + j];
  const unsigned cnt = child_count[t];
  const int64_t x = base + t;
  cc[x * 3 + 0] = __dadd_rn(pc[0], (o & 1) ? hh : -hh);
  cc[x * 3 + 1] = __dadd_rn(pc[1], (o == 2 || o == 3 || o == 6 || o == 7) ? hh : -hh);
  cc[x * 3 + 2] = __dadd_rn(pc[2], (o > 3) ? hh : -hh);
  cw[x] = h;
  cstart[x] = s;
  ccount[x] = (int32_t)cnt;
  const int d = cdepth[cell] + 1;
  cdepth[x] = d;
  cparent[x] = cell;
  coct[x] = o;
  unsigned state = 0;
  if (cnt > 1 && d < kMaxDepth) {
    const bool one_octant = __popc(seg_mask[k]) == 1;
    const bool chain = one_octant && (seg_diff[k] == 0 || centre_stuck(pc, cw[cell]));
    state = chain ? 2u : 1u;
  }
  child_state[t] = state;
}

// Scatter the sorted entries of this level into perm and compact the entries
// of children that stay active into the next level's arrays.
__global__ void advance_kernel(const int32_t* __restrict__ pt_sorted,
                               const unsigned* __restrict__ key_sorted, int64_t M,
                               const int32_t* __restrict__ seg_first,
                               const int64_t* __restrict__ seg_pstart,
                               const unsigned* __restrict__ child_state,
                               const unsigned* __restrict__ child_newseg,
                               const unsigned* __restrict__ entry_pos, int32_t* __restrict__ perm,
                               int32_t* __restrict__ next_pt, int32_t* __restrict__ next_seg) {
  const int64_t m = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (m >= M) return;
  const unsigned key = key_sorted[m];
  const int k = (int)(key >> 3);
  const int32_t p = pt_sorted[m];
  perm[seg_pstart[k] + (m - seg_first[k])] = p;
  if (child_state[key] == 1u) {
    const unsigned pos = entry_pos[m];
    next_pt[pos] = p;
    next_seg[pos] = (int32_t)child_newseg[key];
  }
}

__global__ void entry_flag_kernel(const unsigned* __restrict__ key_sorted, int64_t M,
                                  const unsigned* __restrict__ child_state,
                                  unsigned* __restrict__ flag) {
  const int64_t m = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (m < M) flag[m] = child_state[key_sorted[m]] == 1u ? 1u : 0u;
}

__global__ void state_flag_kernel(const unsigned* __restrict__ child_state, int64_t n, unsigned v,
                                  unsigned* __restrict__ flag) {
  const int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (i < n) flag[i] = child_state[i] == v ? 1u : 0u;
}

// The level's totals in one word array, read by the host with one copy:
// {last child state, new segments before the last child, chains before it,
//  last entry's flag, entries before it}.
__global__ void level_totals_kernel(const unsigned* __restrict__ child_state,
                                    const unsigned* __restrict__ child_newseg,
                                    const unsigned* __restrict__ child_chainslot, int64_t K8,
                                    const unsigned* __restrict__ eflag,
                                    const unsigned* __restrict__ epos, int64_t M,
                                    unsigned* __restrict__ out) {
  out[0] = child_state[K8 - 1];
  out[1] = child_newseg[K8 - 1];
  out[2] = child_chainslot[K8 - 1];
  out[3] = eflag[M - 1];
  out[4] = epos[M - 1];
}

// Next level's segment table and the chain list.
__global__ void next_segments_kernel(int64_t K8, const unsigned* __restrict__ child_state,
                                     const unsigned* __restrict__ child_newseg,
                                     const unsigned* __restrict__ child_chainslot,
                                     const unsigned* __restrict__ entry_pos_of_child,
                                     int64_t base, const int64_t* __restrict__ cstart,
                                     const int32_t* __restrict__ ccount,
                                     int32_t* __restrict__ nseg_cell,
                                     int32_t* __restrict__ nseg_first,
                                     int64_t* __restrict__ nseg_pstart,
                                     int32_t* __restrict__ chain_cell) {
  const int64_t t = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (t >= K8) return;
  const unsigned s = child_state[t];
  if (s == 1u) {
    const unsigned j = child_newseg[t];
    nseg_cell[j] = (int32_t)(base + t);
    nseg_first[j] = (int32_t)entry_pos_of_child[t];
    nseg_pstart[j] = cstart[base + t];
  } else if (s == 2u) {
    chain_cell[child_chainslot[t]] = (int32_t)(base + t);
  }
}

// First entry position (in the next level's compacted array) of each active
// child: the number of active entries before it = exclusive scan of the
// active children's counts.
__global__ void active_count_kernel(const unsigned* __restrict__ child_state,
                                    const unsigned* __restrict__ child_count, int64_t K8,
                                    unsigned* __restrict__ out) {
  const int64_t t = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (t < K8) out[t] = child_state[t] == 1u ? child_count[t] : 0u;
}

// One thread per chain: the cell's points share one octant at every deeper
// level; emit 8 children per level down to depth 30000.
__global__ void chain_kernel(const double* __restrict__ P, const int32_t* __restrict__ perm,
                             const int32_t* __restrict__ chain_cell, int nchains,
                             const int64_t* __restrict__ chain_base, double* cc, double* cw,
                             int64_t* cstart, int32_t* ccount, int32_t* cdepth, int32_t* cparent,
                             int32_t* coct) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= nchains) return;
  int64_t cur = chain_cell[i];
  const int64_t s = cstart[cur];
  const int32_t cnt = ccount[cur];
  const int32_t rep = perm[s];
  const double px = P[(int64_t)rep * 3], py = P[(int64_t)rep * 3 + 1], pz = P[(int64_t)rep * 3 + 2];
  double c[3] = {cc[cur * 3], cc[cur * 3 + 1], cc[cur * 3 + 2]};
  double w = cw[cur];
  int d = cdepth[cur];
  int64_t x = chain_base[i];
  while (d < kMaxDepth) {
    int o = 0;
    if (px >= c[0]) o += 1;
    if (py >= c[1]) o += 2;
    if (pz >= c[2]) o += 4;
    const double h = __dmul_rn(w, 0.5);
    const double hh = __dmul_rn(h, 0.5);
    int64_t next = -1;
    for (int j = 0; j < 8; ++j, ++x) {
      cc[x * 3 + 0] = __dadd_rn(c[0], (j & 1) ? hh : -hh);
      cc[x * 3 + 1] = __dadd_rn(c[1], (j == 2 || j == 3 || j == 6 || j == 7) ? hh : -hh);
      cc[x * 3 + 2] = __dadd_rn(c[2], (j > 3) ? hh : -hh);
      cw[x] = h;
      cstart[x] = s;
      ccount[x] = j == o ? cnt : 0;
      cdepth[x] = d + 1;
      cparent[x] = (int32_t)cur;
      coct[x] = j;
      if (j == o) next = x;
    }
    cur = next;
    c[0] = cc[cur * 3];
    c[1] = cc[cur * 3 + 1];
    c[2] = cc[cur * 3 + 2];
    w = h;
    ++d;
  }
}

__global__ void internal_keys_kernel(const int64_t* __restrict__ cstart,
                                     const int32_t* __restrict__ ccount,
                                     const int32_t* __restrict__ cdepth, int64_t ncells,
                                     unsigned long long* __restrict__ key, int32_t* __restrict__ val,
                                     unsigned* __restrict__ is_internal) {
  const int64_t x = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (x >= ncells) return;
  const bool internal = ccount[x] > 1 && cdepth[x] < kMaxDepth;
  is_internal[x] = internal ? 1u : 0u;
  // non-internal cells sort after every internal one
  key[x] = internal ? (((unsigned long long)cstart[x] << 15) | (unsigned long long)cdepth[x])
                    : ((1ull << 48) - 1);
  val[x] = (int32_t)x;
}

__global__ void rank_kernel(const int32_t* __restrict__ sorted_cell, int64_t ninternal,
                            int32_t* __restrict__ rank) {
  const int64_t r = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (r < ninternal) rank[sorted_cell[r]] = (int32_t)r;
}

__global__ void final_layout_kernel(int64_t ncells, const double* __restrict__ cc,
                                    const double* __restrict__ cw,
                                    const int64_t* __restrict__ cstart,
                                    const int32_t* __restrict__ ccount,
                                    const int32_t* __restrict__ cdepth,
                                    const int32_t* __restrict__ cparent,
                                    const int32_t* __restrict__ coct,
                                    const int32_t* __restrict__ rank, double* __restrict__ cn,
                                    double* __restrict__ w, int32_t* __restrict__ ch,
                                    int64_t* __restrict__ start, int32_t* __restrict__ count,
                                    int32_t* __restrict__ depth) {
  const int64_t x = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (x >= ncells) return;
  const int32_t par = cparent[x];
  const int64_t id = par < 0 ? 0 : 1 + 8 * (int64_t)rank[par] + coct[x];
  for (int d = 0; d < 3; ++d) cn[id * 3 + d] = cc[x * 3 + d];
  w[id] = cw[x];
  start[id] = cstart[x];
  count[id] = ccount[x];
  depth[id] = cdepth[x];
  const bool internal = ccount[x] > 1 && cdepth[x] < kMaxDepth;
  for (int j = 0; j < 8; ++j) ch[id * 8 + j] = internal ? (int32_t)(1 + 8 * (int64_t)rank[x] + j) : -1;
}

// ------------------------------------------------ build from sorted paths --
// The usual build, without a level loop.  A cell's centre follows from its
// octant path alone, so every point can walk its own path from the root; the
// points sorted by path (stably: equal paths keep the input order) are the
// final permutation, and with cpl[p] = the octants that the sorted points
// p - 1 and p share (-1 at both ends), the internal cells whose first point is
// p are those of the depths cpl[p] + 1 .. cpl[p + 1]: listed p by p, that is
// depth-first pre-order, the order of the ids.  A cell's end and its children
// are found by searching the sorted keys.
// The key is one word of 10, 16 or 21 octants (4, 6 or 8 sort passes, by the
// point count) or, where many points share those (a far outlier, points at all
// scales), three words of 21, sorted last word first.  Runs of equal keys are
// ordered by their deeper octants, one thread per run of up to kTieRun points.
// Where points share kTieDepth octants (identical ones above all), or more than
// kTieRun of them all three words, the whole build is left to the level loop
// below, which follows them to depth 30000.
// In place of about 20 launches, 6 scans and a host read per level, over every
// point: 2M points 7.5 -> 1.6 ms.
constexpr int kKeyDepth = 21;
constexpr int kKeyWords = 3;
constexpr int kTieDepth = 64;
constexpr int kTieRun = 32;
// A run this long is not expected to be split by the 5 octants that the longest
// one-word key has more than the shorter one.
constexpr int kLongRun = 4096;

// A point's key: W words of kd octants.
template <int W>
struct PathKeys {
  unsigned long long* w[W];
  int kd;

  __device__ __forceinline__ bool equal(int64_t a, int64_t b) const {
    bool eq = true;
#pragma unroll
    for (int i = 0; i < W; ++i) eq = eq && w[i][a] == w[i][b];
    return eq;
  }
};
// Octant l of a key; whether the first d octants of two keys agree.
template <int W>
struct PathKey {
  unsigned long long w[W];
  __device__ __forceinline__ PathKey(const PathKeys<W>& k, int64_t p) {
#pragma unroll
    for (int i = 0; i < W; ++i) w[i] = k.w[i][p];
  }
  __device__ __forceinline__ int octant(int kd, int l) const {
    unsigned long long v = w[0];
    if (W > 1) {
#pragma unroll
      for (int i = 1; i < W; ++i)
        if (l >= i * kd) v = w[i];
      l %= kd;
    }
    return (int)((v >> (3 * (kd - 1 - l))) & 7ull);
  }
  __device__ __forceinline__ bool agrees(const PathKey& o, int kd, int d) const {
    bool eq = true;
#pragma unroll
    for (int i = 0; i < W; ++i) {
      const int left = min(max(d - i * kd, 0), kd);  // octants of this word
      eq = eq && (left == 0 || ((w[i] ^ o.w[i]) >> (3 * (kd - left))) == 0);
    }
    return eq;
  }
};

// By depth: the cell width and the step from a centre to its children's, as
// the reference halves them.
struct Widths {
  double w[kTieDepth + 2], step[kTieDepth + 2];
};
__global__ void widths_kernel(const double* __restrict__ rw, Widths* __restrict__ t) {
  double w = *rw;
  for (int d = 0; d < kTieDepth + 2; ++d) {
    const double h = __dmul_rn(w, 0.5);
    t->w[d] = w;
    t->step[d] = __dmul_rn(h, 0.5);
    w = h;
  }
}

struct PathTotals {
  unsigned long long nindices;
  uint32_t ninternal, max_cpl;
  uint32_t deep;              // points share kTieDepth octants
  uint32_t long_run, longer;  // a run of more than kTieRun / kLongRun equal keys
};

// The octant walk of one point: the centre of its cell.
struct Walk {
  double c[3];
  __device__ __forceinline__ int octant(const double* p) const {
    return (p[0] >= c[0] ? 1 : 0) + (p[1] >= c[1] ? 2 : 0) + (p[2] >= c[2] ? 4 : 0);
  }
  __device__ __forceinline__ void descend(int o, double step) {
    c[0] = __dadd_rn(c[0], (o & 1) ? step : -step);
    c[1] = __dadd_rn(c[1], (o & 2) ? step : -step);
    c[2] = __dadd_rn(c[2], (o & 4) ? step : -step);
  }
};

template <int W>
__global__ void path_keys_kernel(const double* __restrict__ P, int64_t n,
                                 const double* __restrict__ rc, const Widths* __restrict__ t,
                                 PathKeys<W> keys, int32_t* __restrict__ val) {
  const int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (i >= n) return;
  const double p[3] = {P[i * 3], P[i * 3 + 1], P[i * 3 + 2]};
  Walk w{{rc[0], rc[1], rc[2]}};
#pragma unroll
  for (int j = 0; j < W; ++j) {
    unsigned long long k = 0;
    for (int d = 0; d < keys.kd; ++d) {
      const int o = w.octant(p);
      k = k << 3 | (unsigned)o;
      w.descend(o, t->step[j * keys.kd + d]);
    }
    keys.w[j][i] = k;
  }
  val[i] = (int32_t)i;
}

__global__ void gather_keys_kernel(const unsigned long long* __restrict__ key,
                                   const int32_t* __restrict__ val, int64_t n,
                                   unsigned long long* __restrict__ out) {
  const int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (i < n) out[i] = key[val[i]];
}

// Octants that points a and b share, up to kTieDepth; less: a's path is the
// smaller one.
__device__ int shared_octants(const double* P, int32_t a, int32_t b, const double* rc,
                              const Widths* t, bool& less) {
  const double pa[3] = {P[(int64_t)a * 3], P[(int64_t)a * 3 + 1], P[(int64_t)a * 3 + 2]};
  const double pb[3] = {P[(int64_t)b * 3], P[(int64_t)b * 3 + 1], P[(int64_t)b * 3 + 2]};
  Walk w{{rc[0], rc[1], rc[2]}};
  less = false;
  for (int d = 0; d < kTieDepth; ++d) {
    const int oa = w.octant(pa), ob = w.octant(pb);
    if (oa != ob) {
      less = oa < ob;
      return d;
    }
    w.descend(oa, t->step[d]);
  }
  return kTieDepth;
}

// Runs of equal keys, ordered by the octants past the key: one thread per run.
// Once a run is too long the key will not do, and what has not begun ends here.
template <int W>
__global__ void tie_runs_kernel(const double* __restrict__ P, int64_t n,
                                const double* __restrict__ rc, const Widths* __restrict__ t,
                                PathKeys<W> keys, int32_t* val, PathTotals* tot) {
  const int64_t p = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (p + 1 >= n || !keys.equal(p, p + 1) || (p > 0 && keys.equal(p - 1, p))) return;
  if (p + kTieRun < n && keys.equal(p, p + kTieRun)) {
    tot->long_run = 1;
    if (p + kLongRun < n && keys.equal(p, p + kLongRun)) tot->longer = 1;
    return;
  }
  if (__ldcg(&tot->long_run)) return;
  int64_t e = p + 2;
  while (e < n && keys.equal(p, e)) ++e;
  for (int64_t i = p + 1; i < e; ++i) {  // stable insertion sort
    const int32_t v = val[i];
    int64_t j = i;
    while (j > p) {
      bool less;
      if (shared_octants(P, v, val[j - 1], rc, t, less) == kTieDepth) tot->deep = 1;
      if (!less) break;
      val[j] = val[j - 1];
      --j;
    }
    val[j] = v;
  }
}

// cpl[p] and, per point, how many internal cells start at it.
template <int W>
__global__ void __launch_bounds__(256) cpl_kernel(const double* __restrict__ P, int64_t n,
                                                  const double* __restrict__ rc,
                                                  const Widths* __restrict__ t,
                                                  PathKeys<W> keys,
                                                  const int32_t* __restrict__ val,
                                                  int8_t* __restrict__ cpl,
                                                  uint32_t* __restrict__ starts,
                                                  PathTotals* __restrict__ tot) {
  if (tot->long_run || tot->deep) return;
  const int64_t p = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  auto shared = [&](int64_t q) {  // octants shared by the sorted points q - 1 and q
    if (q <= 0 || q >= n) return -1;
#pragma unroll
    for (int i = 0; i < W; ++i) {
      const unsigned long long x = keys.w[i][q - 1] ^ keys.w[i][q];
      if (x) return i * keys.kd + (__clzll((long long)x) - (64 - 3 * keys.kd)) / 3;
    }
    bool less;
    const int d = shared_octants(P, val[q - 1], val[q], rc, t, less);
    if (d == kTieDepth) tot->deep = 1;
    return d;
  };
  uint32_t depth = 0, mx = 0;
  if (p < n) {
    const int a = shared(p), b = shared(p + 1);
    cpl[p] = (int8_t)a;
    starts[p] = b > a ? (uint32_t)(b - a) : 0u;
    mx = (uint32_t)max(a, 0);
    depth = (uint32_t)(max(a, b) + 2);  // cells that hold the point
  }
  depth = __reduce_add_sync(0xffffffffu, depth);
  mx = __reduce_max_sync(0xffffffffu, mx);
  __shared__ uint32_t s[8], m[8];
  if ((threadIdx.x & 31) == 0) {
    s[threadIdx.x >> 5] = depth;
    m[threadIdx.x >> 5] = mx;
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    unsigned long long sum = 0;
    for (int w = 0; w < 8; ++w) {
      sum += s[w];
      mx = max(mx, m[w]);
    }
    atomicAdd(&tot->nindices, sum);
    if (mx > tot->max_cpl) atomicMax(&tot->max_cpl, mx);
  }
}

__global__ void path_totals_kernel(const uint32_t* __restrict__ base,
                                   const uint32_t* __restrict__ last, int64_t n,
                                   PathTotals* __restrict__ tot) {
  tot->ninternal = base[n - 1] + *last;
}

// (first point, depth) of every internal cell, in pre-order.
__global__ void list_cells_kernel(const int8_t* __restrict__ cpl, const uint32_t* __restrict__ base,
                                  int64_t n, uint32_t ninternal, int32_t* __restrict__ cell_first,
                                  int8_t* __restrict__ cell_depth) {
  const int64_t p = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (p >= n) return;
  const uint32_t b = base[p], e = p + 1 < n ? base[p + 1] : ninternal;
  for (uint32_t r = b; r < e; ++r) {
    cell_first[r] = (int32_t)p;
    cell_depth[r] = (int8_t)(cpl[p] + 1 + (int)(r - b));
  }
}

// Eight lanes per internal cell, one per child: the cell's points are
// [p, e), child o's those whose octant at this depth is o.
template <int W>
__global__ void __launch_bounds__(256) cells_kernel(
    const double* __restrict__ P, int64_t n, const double* __restrict__ rc,
    const Widths* __restrict__ t, PathKeys<W> keys, const int32_t* __restrict__ val, const int8_t* __restrict__ cpl,
    const uint32_t* __restrict__ base, uint32_t ninternal, const int32_t* __restrict__ cell_first,
    const int8_t* __restrict__ cell_depth, double* __restrict__ cn, double* __restrict__ cw,
    int32_t* __restrict__ ch, int64_t* __restrict__ start, int32_t* __restrict__ count,
    int32_t* __restrict__ depth) {
  const unsigned full = 0xffffffffu;
  const int lane = threadIdx.x & 31, o = lane & 7, g0 = lane & ~7;
  const int64_t r = (blockIdx.x * (int64_t)blockDim.x + threadIdx.x) >> 3;
  const bool live = r < ninternal;
  const int64_t p = live ? cell_first[r] : 0;
  const int d = live ? cell_depth[r] : 0;
  const int kw = keys.kd, kd = W * kw;  // octants per word, of the key
  const PathKey<W> kp(keys, p);
  const int32_t pt = live ? val[p] : 0;
  // centre: lane o follows axis o mod 3 down the path of the cell's first point
  const int axis = o % 3;
  double c = rc[axis];
  const double x = P[(int64_t)pt * 3 + axis];
  const int dmax = __reduce_max_sync(full, d);
  for (int l = 0; l < dmax; ++l) {
    if (l < d) {
      const bool up = l < kd ? (kp.octant(kw, l) >> axis) & 1 : x >= c;
      const double step = t->step[l];
      c = __dadd_rn(c, up ? step : -step);
    }
  }
  double cc[3];
  for (int a = 0; a < 3; ++a) cc[a] = __shfl_sync(full, c, g0 + a);
  // end of the cell: the first position past p that leaves its path
  int64_t e = n, lb = p;
  if (live) {
    if (d > kd) {
      e = p + 1;
      while (e < n && cpl[e] >= d) ++e;
    } else if (d > 0) {
      auto inside = [&](int64_t m) { return kp.agrees(PathKey<W>(keys, m), kw, d); };
      int64_t step = 1, a = p, b = p + 1;  // a inside, b the first known outside
      while (b < n && inside(b)) {
        a = b;
        step *= 2;
        b = p + step;
      }
      b = min(b, n);
      while (b - a > 1) {
        const int64_t m = (a + b) >> 1;
        if (inside(m)) a = m;
        else b = m;
      }
      e = b;
    }
    // first point of the cell with octant >= o
    if (d >= kd) {
      while (lb < e) {
        const int32_t q = val[lb];
        const int oq = (P[(int64_t)q * 3] >= cc[0] ? 1 : 0) +
                       (P[(int64_t)q * 3 + 1] >= cc[1] ? 2 : 0) +
                       (P[(int64_t)q * 3 + 2] >= cc[2] ? 4 : 0);
        if (oq >= o) break;
        ++lb;
      }
    } else if (o > 0) {
      int64_t a = p - 1, b = e;  // octant(a) < o <= octant(b)
      while (b - a > 1) {
        const int64_t m = (a + b) >> 1;
        if (PathKey<W>(keys, m).octant(kw, d) >= o) b = m;
        else a = m;
      }
      lb = b;
    }
  }
  const int64_t up = __shfl_down_sync(full, lb, 1);
  if (!live) return;
  const int64_t cnt = (o == 7 ? e : up) - lb;
  const int64_t id = 1 + 8 * r + o;
  const double hh = t->step[d];
  cn[id * 3 + 0] = __dadd_rn(cc[0], (o & 1) ? hh : -hh);
  cn[id * 3 + 1] = __dadd_rn(cc[1], (o & 2) ? hh : -hh);
  cn[id * 3 + 2] = __dadd_rn(cc[2], (o & 4) ? hh : -hh);
  cw[id] = t->w[d + 1];
  start[id] = lb;
  count[id] = (int32_t)cnt;
  depth[id] = d + 1;
  int4 lo = make_int4(-1, -1, -1, -1), hi = lo;
  if (cnt > 1) {  // internal: the cell of depth d + 1 that starts at lb
    const int32_t f = 1 + 8 * (int32_t)(base[lb] + (uint32_t)(d - (int)cpl[lb]));
    lo = make_int4(f, f + 1, f + 2, f + 3);
    hi = make_int4(f + 4, f + 5, f + 6, f + 7);
  }
  int4* row = reinterpret_cast<int4*>(ch + id * 8);
  row[0] = lo;
  row[1] = hi;
  if (r == 0 && o == 0) {  // the root
    cn[0] = rc[0];
    cn[1] = rc[1];
    cn[2] = rc[2];
    cw[0] = t->w[0];
    start[0] = 0;
    count[0] = (int32_t)n;
    depth[0] = 0;
    row = reinterpret_cast<int4*>(ch);
    row[0] = make_int4(1, 2, 3, 4);
    row[1] = make_int4(5, 6, 7, 8);
  }
}

// Gather each cell's point range into the CSR index array (warp per cell),
// with a (cell id, point id) sort key: a cell's range in perm is ordered by
// octant path, the reference's lists are ascending (octree.cpp:117-122).
__global__ void csr_gather_kernel(const int64_t* __restrict__ off, const int64_t* __restrict__ start,
                                  const int32_t* __restrict__ count, const int32_t* __restrict__ perm,
                                  int64_t ncells, int32_t* __restrict__ idx,
                                  unsigned long long* __restrict__ key) {
  const int64_t warp = (blockIdx.x * (int64_t)blockDim.x + threadIdx.x) >> 5;
  const int lane = threadIdx.x & 31;
  if (warp >= ncells) return;
  const int64_t o = off[warp], s = start[warp];
  const int32_t c = count[warp];
  for (int32_t j = lane; j < c; j += 32) {
    const int32_t p = perm[s + j];
    idx[o + j] = p;
    key[o + j] = ((unsigned long long)warp << 30) | (unsigned long long)p;
  }
}

// 64-bit exclusive scan of per-cell counts (block-partials, recursive).
__global__ void scan64_partials(const int32_t* __restrict__ cnt, int64_t n,
                                int64_t* __restrict__ part) {
  __shared__ int64_t s[1024];
  const int64_t base = blockIdx.x * 4096LL;
  int64_t v = 0;
  for (int k = 0; k < 4; ++k) {
    const int64_t i = base + threadIdx.x * 4 + k;
    if (i < n) v += cnt[i];
  }
  s[threadIdx.x] = v;
  __syncthreads();
  for (int o = 512; o > 0; o >>= 1) {
    if (threadIdx.x < o) s[threadIdx.x] += s[threadIdx.x + o];
    __syncthreads();
  }
  if (threadIdx.x == 0) part[blockIdx.x] = s[0];
}

__global__ void scan64_tiles(const int32_t* __restrict__ cnt, int64_t n,
                             const int64_t* __restrict__ part_off, int64_t* __restrict__ off) {
  __shared__ int64_t s[1024];
  const int64_t base = blockIdx.x * 4096LL;
  int64_t v[4], t = 0;
  for (int k = 0; k < 4; ++k) {
    const int64_t i = base + threadIdx.x * 4 + k;
    v[k] = i < n ? cnt[i] : 0;
    t += v[k];
  }
  s[threadIdx.x] = t;
  __syncthreads();
  for (int o = 1; o < 1024; o <<= 1) {
    const int64_t a = threadIdx.x >= o ? s[threadIdx.x - o] : 0;
    __syncthreads();
    s[threadIdx.x] += a;
    __syncthreads();
  }
  int64_t run = s[threadIdx.x] - t + (part_off ? part_off[blockIdx.x] : 0);
  for (int k = 0; k < 4; ++k) {
    const int64_t i = base + threadIdx.x * 4 + k;
    if (i < n) off[i] = run;
    run += v[k];
  }
  if (base + 4096 >= n && threadIdx.x == 1023) off[n] = run;
}

void exclusive_scan_counts64(const int32_t* cnt, int64_t n, int64_t* off, cudaStream_t st) {
  const int64_t nb = (n + 4095) / 4096;
  if (nb <= 1) {
    launch_kernel(scan64_tiles, 1, 1024, 0, st, cnt, n, nullptr, off);
    GWN_CUDA(cudaGetLastError());
    return;
  }
  DevBuf<int64_t> part((size_t)nb, st), part_off((size_t)nb + 1, st);
  launch_kernel(scan64_partials, (unsigned)nb, 1024, 0, st, cnt, n, part.get());
  // partials are few (<= 2^20 for 2^32 cells); scan them on the host
  std::vector<int64_t> h((size_t)nb), ho((size_t)nb + 1);
  GWN_CUDA(cudaMemcpyAsync(h.data(), part.get(), (size_t)nb * sizeof(int64_t),
                           cudaMemcpyDeviceToHost, st));
  GWN_CUDA(cudaStreamSynchronize(st));
  ho[0] = 0;
  for (int64_t i = 0; i < nb; ++i) ho[(size_t)i + 1] = ho[(size_t)i] + h[(size_t)i];
  GWN_CUDA(cudaMemcpyAsync(part_off.get(), ho.data(), ((size_t)nb + 1) * sizeof(int64_t),
                           cudaMemcpyHostToDevice, st));
  launch_kernel(scan64_tiles, (unsigned)nb, 1024, 0, st, cnt, n, part_off.get(), off);
  GWN_CUDA(cudaGetLastError());
  GWN_CUDA(cudaStreamSynchronize(st));  // ho must outlive the copy
}

inline unsigned blocks(int64_t n, int t = 256) { return (unsigned)std::max<int64_t>(1, (n + t - 1) / t); }

int bits_for(uint64_t maxval) {
  int b = 1;
  while (b < 64 && (maxval >> b)) ++b;
  return b;
}

}  // namespace

// One attempt of the build from sorted paths with keys of W words of kd octants:
// sorts, and fills the tree unless the totals say that the key will not do.
template <int W>
static PathTotals octree_try_paths(gwn_octree_impl& t, const double* dP, int64_t n,
                                   const double* rc, const Widths* wt, int kd, cudaStream_t st) {
  using Key = unsigned long long;
  const size_t N = (size_t)n;
  DevBuf<Key> sorted(N, st), tmp(N, st), word[W];
  DevBuf<int32_t> val(N, st), val_tmp(N, st);
  DevBuf<int8_t> cpl(N, st);
  DevBuf<uint32_t> starts(N, st), base(N, st);
  DevBuf<PathTotals> tot(1, st);
  PathTotals* h = reinterpret_cast<PathTotals*>(pinned_words());
  tot.zero(st);
  PathKeys<W> keys;
  keys.kd = kd;
  for (int i = 0; i < W; ++i) {  // by point
    if (W > 1) word[i].alloc(N, st);
    keys.w[i] = W > 1 ? word[i].get() : sorted.get();
  }
  launch_kernel(path_keys_kernel<W>, blocks(n), 256, 0, st, dP, n, rc, wt, keys, val.get());
  for (int i = W - 1; i >= 0; --i) {  // stable: the last word first
    if (W > 1)
      launch_kernel(gather_keys_kernel, blocks(n), 256, 0, st, (const Key*)word[i].get(),
                    (const int32_t*)val.get(), n, sorted.get());
    radix_sort_pairs<Key>(sorted.get(), val.get(), tmp.get(), val_tmp.get(), n, 0, 3 * kd, st);
  }
  keys.w[0] = sorted.get();
  for (int i = 1; i < W; ++i) {  // the other words in the sorted order
    Key* out = i == 1 ? tmp.get() : word[i - 2].get();
    launch_kernel(gather_keys_kernel, blocks(n), 256, 0, st, (const Key*)word[i].get(),
                  (const int32_t*)val.get(), n, out);
    keys.w[i] = out;
  }
  launch_kernel(tie_runs_kernel<W>, blocks(n), 256, 0, st, dP, n, rc, wt, keys, val.get(),
                tot.get());
  launch_kernel(cpl_kernel<W>, blocks(n), 256, 0, st, dP, n, rc, wt, keys,
                (const int32_t*)val.get(), cpl.get(), starts.get(), tot.get());
  exclusive_scan_u32(starts.get(), base.get(), n, st);
  launch_kernel(path_totals_kernel, 1, 1, 0, st, (const uint32_t*)base.get(),
                (const uint32_t*)(starts.get() + (n - 1)), n, tot.get());
  GWN_CUDA(cudaMemcpyAsync(h, tot.get(), sizeof(PathTotals), cudaMemcpyDeviceToHost, st));
  GWN_CUDA(cudaStreamSynchronize(st));
  const PathTotals r = *h;
  if (r.deep || r.long_run) return r;
  const uint32_t ni = r.ninternal;
  t.ncells = 1 + 8 * (int64_t)ni;
  GWN_REQUIRE(t.ncells < (int64_t(1) << 31), "octree has more than 2^31 cells");
  t.nindices = (int64_t)r.nindices;
  t.max_depth = (int32_t)r.max_cpl + 1;
  t.cn.alloc((size_t)t.ncells * 3);
  t.w.alloc((size_t)t.ncells);
  t.ch.alloc((size_t)t.ncells * 8);
  t.start.alloc((size_t)t.ncells);
  t.count.alloc((size_t)t.ncells);
  t.depth.alloc((size_t)t.ncells);
  t.perm.alloc(N);
  DevBuf<int32_t> cell_first(ni, st);
  DevBuf<int8_t> cell_depth(ni, st);
  launch_kernel(list_cells_kernel, blocks(n), 256, 0, st, (const int8_t*)cpl.get(),
                (const uint32_t*)base.get(), n, ni, cell_first.get(), cell_depth.get());
  launch_kernel(cells_kernel<W>, blocks((int64_t)ni * 8), 256, 0, st, dP, n, rc, wt, keys,
                (const int32_t*)val.get(), (const int8_t*)cpl.get(), (const uint32_t*)base.get(),
                ni, (const int32_t*)cell_first.get(), (const int8_t*)cell_depth.get(), t.cn.get(),
                t.w.get(), t.ch.get(), t.start.get(), t.count.get(), t.depth.get());
  GWN_CUDA(cudaMemcpyAsync(t.perm.get(), val.get(), N * 4, cudaMemcpyDeviceToDevice, st));
  GWN_CUDA(cudaStreamSynchronize(st));
  return r;
}

// The build from sorted paths; false when the level loop has to do it.
static bool octree_build_paths(gwn_octree_impl& t, const double* dP, int64_t n, const double* rc,
                               const double* rw, cudaStream_t st) {
  DevBuf<Widths> widths(1, st);
  launch_kernel(widths_kernel, 1, 1, 0, st, rw, widths.get());
  // Octants per key: points spread over a surface share about log2(n) / 2, so
  // 10 (four passes) and 16 (six) leave few equal keys to 4096 and 16M points.
  int kd = n <= 4096 ? 10 : (n <= (int64_t(16) << 20) ? 16 : kKeyDepth);
  for (;;) {
    const PathTotals r = octree_try_paths<1>(t, dP, n, rc, widths.get(), kd, st);
    if (r.deep) return false;
    if (!r.long_run) return true;
    if (kd == kKeyDepth || r.longer) break;
    kd = kKeyDepth;
  }
  const PathTotals r = octree_try_paths<kKeyWords>(t, dP, n, rc, widths.get(), kKeyDepth, st);
  return !r.deep && !r.long_run;
}

void octree_build(gwn_octree_impl& t, const double* P, int64_t n, bool host_mode, cudaStream_t st) {
  (void)host_mode;
  GWN_REQUIRE(n <= (int64_t(1) << 29), "at most 2^29 points");
  t.n = n;
  t.P.alloc((size_t)std::max<int64_t>(n, 1) * 3);
  if (n)
    GWN_CUDA(cudaMemcpyAsync(t.P.get(), P, (size_t)n * 3 * sizeof(double), cudaMemcpyDeviceToDevice, st));
  const double* dP = t.P.get();
  Cells cells;
  cells.reserve(64, st);
  DevBuf<unsigned long long> mm(6, st);
  init_minmax(mm.get(), 3, st);
  if (n > 0) {
    launch_kernel(point_bbox_kernel, std::min<unsigned>(blocks(n), 1024u), 256, 0, st, dP, n, mm.get());
    GWN_CUDA(cudaGetLastError());
  }
  launch_kernel(root_kernel, 1, 1, 0, st, mm.get(), n, cells.c.get(), cells.w.get(), cells.start.get(),
                               cells.count.get(), cells.depth.get(), cells.parent.get(),
                               cells.oct.get());
  GWN_CUDA(cudaGetLastError());
  cells.size = 1;
  if (n >= 2 && octree_build_paths(t, dP, n, cells.c.get(), cells.w.get(), st)) return;
  cells.reserve(std::max<int64_t>(64, 9 + n / 2), st);
  DevBuf<int32_t> perm((size_t)std::max<int64_t>(n, 1), st);
  launch_kernel(iota_kernel, blocks(n), 256, 0, st, perm.get(), n);

  // level state
  int64_t M = n >= 2 ? n : 0;  // active entries
  int K = n >= 2 ? 1 : 0;      // active segments
  DevBuf<int32_t> act_pt((size_t)std::max<int64_t>(M, 1), st), act_seg((size_t)std::max<int64_t>(M, 1), st);
  DevBuf<int32_t> seg_cell(1, st), seg_first(1, st);
  DevBuf<int64_t> seg_pstart(1, st);
  if (K) {
    launch_kernel(iota_kernel, blocks(M), 256, 0, st, act_pt.get(), M);
    launch_kernel(fill_i32_kernel, blocks(M), 256, 0, st, act_seg.get(), M, 0);
    launch_kernel(fill_i32_kernel, 1, 32, 0, st, seg_cell.get(), 1, 0);
    launch_kernel(fill_i32_kernel, 1, 32, 0, st, seg_first.get(), 1, 0);
    GWN_CUDA(cudaMemsetAsync(seg_pstart.get(), 0, sizeof(int64_t), st));
  }
  bool had_chain = false;
  int levels = 0;
  DevBuf<unsigned> totals_d(8, st);
  unsigned* totals_h = pinned_words();
  while (K > 0) {
    ++levels;
    const int64_t K8 = (int64_t)K * 8;
    DevBuf<unsigned> key((size_t)M, st), key_tmp((size_t)M, st);
    DevBuf<int32_t> pt_tmp((size_t)M, st);
    DevBuf<unsigned> seg_mask((size_t)K, st), seg_diff((size_t)K, st), child_count((size_t)K8, st);
    seg_mask.zero(st);
    seg_diff.zero(st);
    child_count.zero(st);
    launch_kernel(octant_kernel, blocks(M), 256, 0, st, dP, act_pt.get(), act_seg.get(), M, seg_cell.get(),
                                             seg_first.get(), cells.c.get(), key.get(),
                                             seg_mask.get(), seg_diff.get());
    GWN_CUDA(cudaGetLastError());
    radix_sort_pairs<uint32_t>(key.get(), act_pt.get(), key_tmp.get(), pt_tmp.get(), M, 0,
                               bits_for((uint64_t)K8 - 1), st);
    launch_kernel(child_count_kernel, blocks(M), 256, 0, st, key.get(), M, child_count.get());
    cells.reserve(cells.size + K8, st);
    const int64_t base = cells.size;
    DevBuf<unsigned> child_state((size_t)K8, st);
    launch_kernel(emit_children_kernel, blocks(K8), 256, 0, st, 
        K, seg_cell.get(), seg_pstart.get(), seg_mask.get(), seg_diff.get(), child_count.get(), base,
        cells.c.get(), cells.w.get(), cells.start.get(), cells.count.get(), cells.depth.get(),
        cells.parent.get(), cells.oct.get(), child_state.get());
    GWN_CUDA(cudaGetLastError());
    cells.size += K8;
    // scans: new segment ids, chain slots, first entry of each active child,
    // compacted entry positions
    DevBuf<unsigned> child_newseg((size_t)K8, st), child_chainslot((size_t)K8, st),
        child_firstpos((size_t)K8, st), tmp((size_t)K8, st);
    launch_kernel(state_flag_kernel, blocks(K8), 256, 0, st, child_state.get(), K8, 1u, tmp.get());
    exclusive_scan_u32(tmp.get(), child_newseg.get(), K8, st);
    launch_kernel(state_flag_kernel, blocks(K8), 256, 0, st, child_state.get(), K8, 2u, tmp.get());
    exclusive_scan_u32(tmp.get(), child_chainslot.get(), K8, st);
    launch_kernel(active_count_kernel, blocks(K8), 256, 0, st, child_state.get(), child_count.get(), K8,
                                                    tmp.get());
    exclusive_scan_u32(tmp.get(), child_firstpos.get(), K8, st);
    DevBuf<unsigned> eflag((size_t)M, st), epos((size_t)M, st);
    launch_kernel(entry_flag_kernel, blocks(M), 256, 0, st, key.get(), M, child_state.get(), eflag.get());
    exclusive_scan_u32(eflag.get(), epos.get(), M, st);
    // totals: one small kernel and one copy into pinned memory per level
    launch_kernel(level_totals_kernel, 1, 1, 0, st, (const unsigned*)child_state.get(),
                  (const unsigned*)child_newseg.get(), (const unsigned*)child_chainslot.get(), K8,
                  (const unsigned*)eflag.get(), (const unsigned*)epos.get(), M, totals_d.get());
    GWN_CUDA(cudaMemcpyAsync(totals_h, totals_d.get(), 5 * sizeof(unsigned),
                             cudaMemcpyDeviceToHost, st));
    GWN_CUDA(cudaStreamSynchronize(st));
    const unsigned last_state = totals_h[0], last_newseg = totals_h[1],
                   last_chain = totals_h[2], last_eflag = totals_h[3],
                   last_epos = totals_h[4];
    const int nK = (int)(last_newseg + (last_state == 1u ? 1u : 0u));
    const int nChains = (int)(last_chain + (last_state == 2u ? 1u : 0u));
    const int64_t nM = (int64_t)last_epos + last_eflag;
    DevBuf<int32_t> next_pt((size_t)std::max<int64_t>(nM, 1), st),
        next_seg((size_t)std::max<int64_t>(nM, 1), st);
    launch_kernel(advance_kernel, blocks(M), 256, 0, st, act_pt.get(), key.get(), M, seg_first.get(),
                                              seg_pstart.get(), child_state.get(),
                                              child_newseg.get(), epos.get(), perm.get(),
                                              next_pt.get(), next_seg.get());
    GWN_CUDA(cudaGetLastError());
    DevBuf<int32_t> nseg_cell((size_t)std::max(nK, 1), st), nseg_first((size_t)std::max(nK, 1), st);
    DevBuf<int64_t> nseg_pstart((size_t)std::max(nK, 1), st);
    DevBuf<int32_t> chain_cell((size_t)std::max(nChains, 1), st);
    launch_kernel(next_segments_kernel, blocks(K8), 256, 0, st, 
        K8, child_state.get(), child_newseg.get(), child_chainslot.get(), child_firstpos.get(), base,
        cells.start.get(), cells.count.get(), nseg_cell.get(), nseg_first.get(), nseg_pstart.get(),
        chain_cell.get());
    GWN_CUDA(cudaGetLastError());
    if (nChains > 0) {
      had_chain = true;
      std::vector<int32_t> cc_h((size_t)nChains), cd_h((size_t)nChains);
      GWN_CUDA(cudaMemcpyAsync(cc_h.data(), chain_cell.get(), (size_t)nChains * 4,
                               cudaMemcpyDeviceToHost, st));
      GWN_CUDA(cudaStreamSynchronize(st));
      // depth of each chain head: all chains created at this level have the same depth
      int32_t dh = 0;
      GWN_CUDA(cudaMemcpy(&dh, cells.depth.get() + cc_h[0], 4, cudaMemcpyDeviceToHost));
      const int64_t per = 8LL * (kMaxDepth - dh);
      std::vector<int64_t> cb((size_t)nChains);
      for (int i = 0; i < nChains; ++i) cb[(size_t)i] = cells.size + per * i;
      cells.reserve(cells.size + per * nChains, st);
      DevBuf<int64_t> chain_base((size_t)nChains, st);
      chain_base.upload(cb.data(), (size_t)nChains, st);
      launch_kernel(chain_kernel, blocks(nChains, 64), 64, 0, st, 
          dP, perm.get(), chain_cell.get(), nChains, chain_base.get(), cells.c.get(), cells.w.get(),
          cells.start.get(), cells.count.get(), cells.depth.get(), cells.parent.get(),
          cells.oct.get());
      GWN_CUDA(cudaGetLastError());
      GWN_CUDA(cudaStreamSynchronize(st));  // cb outlives its copy
      cells.size += per * nChains;
    }
    act_pt = std::move(next_pt);
    act_seg = std::move(next_seg);
    seg_cell = std::move(nseg_cell);
    seg_first = std::move(nseg_first);
    seg_pstart = std::move(nseg_pstart);
    M = nM;
    K = nK;
  }
  // ids
  const int64_t ncells = cells.size;
  GWN_REQUIRE(ncells < (int64_t(1) << 31), "octree has more than 2^31 cells");
  DevBuf<unsigned long long> ikey((size_t)ncells, st), ikey_tmp((size_t)ncells, st);
  DevBuf<int32_t> ival((size_t)ncells, st), ival_tmp((size_t)ncells, st);
  DevBuf<unsigned> is_internal((size_t)ncells, st);
  launch_kernel(internal_keys_kernel, blocks(ncells), 256, 0, st, cells.start.get(), cells.count.get(),
                                                       cells.depth.get(), ncells, ikey.get(),
                                                       ival.get(), is_internal.get());
  GWN_CUDA(cudaGetLastError());
  radix_sort_pairs<unsigned long long>(ikey.get(), ival.get(), ikey_tmp.get(), ival_tmp.get(),
                                       ncells, 0, 48, st);
  const int64_t ninternal = (ncells - 1) / 8;
  DevBuf<int32_t> rank((size_t)ncells, st);
  if (ninternal > 0)
    launch_kernel(rank_kernel, blocks(ninternal), 256, 0, st, ival.get(), ninternal, rank.get());
  t.ncells = ncells;
  t.cn.alloc((size_t)ncells * 3);
  t.w.alloc((size_t)ncells);
  t.ch.alloc((size_t)ncells * 8);
  t.start.alloc((size_t)ncells);
  t.count.alloc((size_t)ncells);
  t.depth.alloc((size_t)ncells);
  launch_kernel(final_layout_kernel, blocks(ncells), 256, 0, st, 
      ncells, cells.c.get(), cells.w.get(), cells.start.get(), cells.count.get(), cells.depth.get(),
      cells.parent.get(), cells.oct.get(), rank.get(), t.cn.get(), t.w.get(), t.ch.get(),
      t.start.get(), t.count.get(), t.depth.get());
  GWN_CUDA(cudaGetLastError());
  t.perm.alloc((size_t)std::max<int64_t>(n, 1));
  if (n)
    GWN_CUDA(cudaMemcpyAsync(t.perm.get(), perm.get(), (size_t)n * 4, cudaMemcpyDeviceToDevice, st));
  // total index count
  DevBuf<int64_t> off((size_t)ncells + 1, st);
  exclusive_scan_counts64(t.count.get(), ncells, off.get(), st);
  GWN_CUDA(cudaMemcpyAsync(&t.nindices, off.get() + ncells, sizeof(int64_t), cudaMemcpyDeviceToHost, st));
  GWN_CUDA(cudaStreamSynchronize(st));
  // deepest cell: a chain reaches 30000, otherwise one level per iteration
  t.max_depth = had_chain ? kMaxDepth : levels;
}

void octree_export_csr(const gwn_octree_impl& t, int64_t* pi_offsets, int32_t* pi_indices,
                       cudaStream_t st) {
  exclusive_scan_counts64(t.count.get(), t.ncells, pi_offsets, st);
  if (pi_indices && t.nindices > 0) {
    GWN_REQUIRE(t.nindices < (int64_t(1) << 32), "point lists exceed 2^32 entries");
    const int64_t threads = t.ncells * 32;
    DevBuf<unsigned long long> key((size_t)t.nindices, st), key_tmp((size_t)t.nindices, st);
    DevBuf<int32_t> tmp((size_t)t.nindices, st);
    launch_kernel(csr_gather_kernel, blocks(threads), 256, 0, st, pi_offsets, t.start.get(), t.count.get(),
                                                       t.perm.get(), t.ncells, pi_indices,
                                                       key.get());
    GWN_CUDA(cudaGetLastError());
    // entries are already grouped by cell; sort by the full key to order
    // every cell's points ascending
    radix_sort_pairs<unsigned long long>(key.get(), pi_indices, key_tmp.get(), tmp.get(),
                                         t.nindices, 0, 30 + bits_for((uint64_t)t.ncells), st);
  }
}

}  // namespace gwn
