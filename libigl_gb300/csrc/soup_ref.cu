// The reference's own triangle-soup tree, built on the GPU node for node,
// with the reference's per-child moments.
//
// igl::fast_winding_number(V,F,order,bvh) (include/igl/fast_winding_number.cpp:
// 380-416) calls UT_SolidAngle<float,float>::init, which builds a 4-wide
// BVH (UT_BVH<4>::init with the BOX_AREA heuristic,
// include/igl/FastWindingNumberForSoups.h:4581-4634) over float copies of the
// vertices and stores, per node, one moment record per child lane
// (FWNFS.h:6543-7133).  This file rebuilds exactly that tree and those FP32
// moments on the device, plus the same moments in FP64, and lays them out as
// the pre-order child-slot records the soup walks read (soup.cuh): slot 0 is
// the root (always opened), then every child lane of every node in
// depth-first order, a lane that is a triangle being a leaf slot.
//
// It is compiled with --fmad=false: every FP32 expression rounds after each
// operation, as the reference's SSE code (no fused multiply-add) does, so
// centres, split heuristics, boxes and moments are bit for bit the
// reference's.
//
// Tree build (UT_BVH<4>::initNode, FWNFS.h:4918-5047).  A node of at most 4
// boxes holds them as items; a larger node makes the reference's three binary
// splits (multiSplit, FWNFS.h:5249-5346: split all, then twice the part with
// the largest area x count).
//   Nodes of more than 1024 boxes (kSub): one depth at a time, split by split
//     across the depth; by size a split runs in one warp, in one CTA, or by
//     chunks across the GPU, each with the reference's in-place partition
//     reproduced exactly (below).  A large node without a balanced span waits
//     until the others' splits are made (nthElement across the GPU).
//   Smaller subtrees: one CTA each, whole, in shared memory, a warp per node.
// Span counts and boxes are order-independent (counts, min, max), so every
// decision equals the serial code's.
//
// The in-place three-way partition (partitionByCentre, FWNFS.h:5903-5944)
// keeps the boxes below the pivot in order at the front; the boxes equal to
// the pivot and those above it form two queues, and each arrival of a box
// below the pivot (or, for the upper queue, below or equal) moves the front
// of a non-empty queue to its back.  The final order of a queue is read off
// a tape of its operations: an append writes the box, the r-th rotation
// writes a copy of tape entry r, and the queue is the tape's last k entries.
// Every box finds its tape positions from prefix counts; a copy is followed to
// the earlier entries it refers to.  nthElement (FWNFS.h:5847-5900), the
// fallback when no span is balanced enough, repeats such partitions.
//
// Moments (UT_SolidAngle::init's per-item data and its post() merge,
// FWNFS.h:6668-7118): triangles first, then bottom-up by depth, inside each
// subtree in one CTA and above them one launch a depth; a node's lanes are its
// children's data, and its own data is what its parent's lane holds.
#include <cuda_runtime.h>

#include <algorithm>
#include <cfloat>
#include <climits>
#include <cmath>
#include <vector>

#include "gwn_common.cuh"
#include "soup.cuh"
#include "soup_ref.cuh"
#include "sort.cuh"

namespace gwn {
namespace {

using namespace refsoup;

constexpr int kSpans = 16;
constexpr int kSplits = kSpans - 1;
constexpr uint32_t kMinFraction = 16;
constexpr uint32_t kSmallMax = 2 * kSpans;  // exhaustive / sorted splits
constexpr uint32_t kSub = 1024;              // subtrees built by one CTA, splits by one warp
constexpr uint32_t kCtaMax = 32768;          // splits by one CTA
constexpr uint32_t kChunk = 1024;            // positions per CTA in GPU-wide passes
constexpr uint32_t kSubRef = 0xc0000000u;    // child that is a subtree (above 30-bit items)
constexpr uint32_t kTerm = 0x80000000u;      // tape entry holding a box index
constexpr uint32_t kNone = 0xffffffffu;
constexpr double kNearFrac = 1e-3;

__host__ __device__ inline void box_empty(Box& b) {
  for (int a = 0; a < 3; ++a) {
    b.lo[a] = FLT_MAX;
    b.hi[a] = -FLT_MAX;
  }
}
__device__ __forceinline__ void box_add(Box& b, const Box& o) {
  for (int a = 0; a < 3; ++a) {
    b.lo[a] = b.lo[a] < o.lo[a] ? b.lo[a] : o.lo[a];
    b.hi[a] = b.hi[a] > o.hi[a] ? b.hi[a] : o.hi[a];
  }
}
// BOX_AREA heuristic: half the surface area (FWNFS.h:4064-4080).
__device__ __forceinline__ float half_area(const Box& b) {
  const float d0 = b.hi[0] - b.lo[0], d1 = b.hi[1] - b.lo[1], d2 = b.hi[2] - b.lo[2];
  return d0 * d1 + d1 * d2 + d2 * d0;
}
// Twice the box centre along an axis (utBoxCenter).
__device__ __forceinline__ float centre2(const Box& b, int a) { return b.lo[a] + b.hi[a]; }

// The longest axis of a box, the first on ties.
__device__ __forceinline__ int longest_axis(const Box& b, float& len) {
  int axis = 0;
  len = b.hi[0] - b.lo[0];
  for (int a = 1; a < 3; ++a) {
    const float l = b.hi[a] - b.lo[a];
    if (l > len) {
      axis = a;
      len = l;
    }
  }
  return axis;
}

// float -> int as the reference's x86 build converts (cvttss2si): out of
// range or NaN gives INT_MIN.
__device__ __forceinline__ int cvt_x86(float v) {
  return (v >= -2147483648.0f && v < 2147483648.0f) ? (int)v : INT_MIN;
}
__device__ __forceinline__ int span_of(float c2, float min2, float scale) {
  const int s = cvt_x86((c2 - min2) * scale);
  return s < 0 ? 0 : (s > kSpans - 1 ? kSpans - 1 : s);
}

// Order-preserving float keys for atomic min / max (-0 taken as +0, which
// no decision distinguishes).
__device__ __forceinline__ uint32_t fkey(float x) {
  if (x == 0.0f) x = 0.0f;
  const uint32_t u = __float_as_uint(x);
  return (u & 0x80000000u) ? ~u : (u | 0x80000000u);
}
__device__ __forceinline__ float fkey_inv(uint32_t k) {
  const uint32_t u = (k & 0x80000000u) ? (k & 0x7fffffffu) : ~k;
  return __uint_as_float(u);
}
struct BoxKeys {
  uint32_t lo[3], hi[3];
};
__device__ __forceinline__ void keys_init(uint32_t* k) {
  for (int a = 0; a < 3; ++a) {
    k[a] = 0xffffffffu;
    k[3 + a] = 0u;
  }
}
__device__ __forceinline__ void keys_add(uint32_t* k, const Box& b) {
  for (int a = 0; a < 3; ++a) {
    atomicMin(&k[a], fkey(b.lo[a]));
    atomicMax(&k[3 + a], fkey(b.hi[a]));
  }
}
__device__ __forceinline__ Box keys_box(const uint32_t* k) {
  Box b;
  for (int a = 0; a < 3; ++a) {
    b.lo[a] = fkey_inv(k[a]);
    b.hi[a] = fkey_inv(k[3 + a]);
  }
  return b;
}

// One node above the subtrees (numbered depth by depth).
struct RNode {
  uint32_t start, n;  // its boxes: idx[start .. start + n)
  Box all;            // the box its parent's split handed down
  uint32_t cut[5];    // sub-ranges after the splits made so far
  Box sub[4];
  float area[4];
  int32_t choice;
  uint32_t done;      // splits made; 4: its children are made too
  uint32_t waiting;   // its split needs nthElement across the GPU
  uint32_t child[4];  // item (triangle id), kInternal | node, kSubRef | subtree
  // the split of the current round
  uint32_t t_start, t_n, t_mid;
  Box t_box, t_out[2];
};

// --------------------------------------------------------------- boxes --
// Triangle boxes over float copies of the vertices (UT_SolidAngle::init,
// FWNFS.h:6560-6590); a box with a non-finite bound is excluded
// (FWNFS.h:4606-4615).  Triangles with an index outside V are reported and
// excluded.
__global__ void tri_box_kernel(const double* __restrict__ V, int64_t nV,
                               const int32_t* __restrict__ F, int64_t nF, Box* __restrict__ box,
                               uint32_t* __restrict__ keep, unsigned* __restrict__ status) {
  const int64_t f = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (f >= nF) return;
  bool ok = true;
  float p[3][3];
  for (int c = 0; c < 3; ++c) {
    const int32_t i = F[f * 3 + c];
    if (i < 0 || i >= nV) {
      atomicOr(status, kStatusBadInput);
      ok = false;
      for (int d = 0; d < 3; ++d) p[c][d] = 0.f;
      continue;
    }
    for (int d = 0; d < 3; ++d) p[c][d] = (float)V[(int64_t)i * 3 + d];
  }
  Box b;
  tri_box(p[0], p[1], p[2], b.lo, b.hi);
  for (int a = 0; a < 3; ++a)
    if (!isfinite(b.lo[a]) || !isfinite(b.hi[a])) ok = false;
  box[f] = b;
  keep[f] = ok ? 1u : 0u;
}

// Kept triangles in input order, and the root box: a fixed grid strides the
// triangles and each CTA adds its box once (with an atomic set per warp of
// triangles, 240,000 atomics on six words: 158 us for 1.3M triangles).
__global__ void __launch_bounds__(256) compact_kernel(const uint32_t* __restrict__ keep,
                                                      const uint32_t* __restrict__ pos, int64_t nF,
                                                      const Box* __restrict__ box,
                                                      uint32_t* __restrict__ idx,
                                                      uint32_t* __restrict__ root_keys) {
  __shared__ uint32_t s_keys[6];
  if (threadIdx.x == 0) keys_init(s_keys);
  __syncthreads();
  uint32_t kk[6];
  keys_init(kk);
  for (int64_t f = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; f < nF;
       f += (int64_t)gridDim.x * blockDim.x) {
    if (!keep[f]) continue;
    idx[pos[f]] = (uint32_t)f;
    const Box b = box[f];
    for (int a = 0; a < 3; ++a) {
      kk[a] = min(kk[a], fkey(b.lo[a]));
      kk[3 + a] = max(kk[3 + a], fkey(b.hi[a]));
    }
  }
  const unsigned full = 0xffffffffu;
  for (int a = 0; a < 3; ++a) {
    kk[a] = __reduce_min_sync(full, kk[a]);
    kk[3 + a] = __reduce_max_sync(full, kk[3 + a]);
  }
  if ((threadIdx.x & 31) == 0)
    for (int a = 0; a < 3; ++a) {
      atomicMin(&s_keys[a], kk[a]);
      atomicMax(&s_keys[3 + a], kk[3 + a]);
    }
  __syncthreads();
  if (threadIdx.x < 3) atomicMin(&root_keys[threadIdx.x], s_keys[threadIdx.x]);
  else if (threadIdx.x < 6) atomicMax(&root_keys[threadIdx.x], s_keys[threadIdx.x]);
}

__global__ void keys_init_kernel(uint32_t* keys) { keys_init(keys); }

// ------------------------------------------------ one split by one warp --
// Splits of at most kSub boxes run in one warp on shared memory: boxes by
// local index (bx: lo xyz, hi xyz), their current order in perm.  A serial
// thread per split (insertion sort, three-way partition) was bound by its
// dependent shared- and local-memory accesses: 4.8 ms of split kernels for
// 1.3M triangles, most of it one thread per CTA partitioning.
struct SplitMem {
  const float* bx;  // [6][stride]
  int stride;
  uint16_t *perm, *tmp, *tape_e, *tape_g;  // by position
};
struct SplitScratch {  // one per warp
  uint32_t cnt[kSpans];
  uint32_t keys[kSpans][6];
  Box sub[4];
  float area[4];
  uint32_t cut[5];
};
constexpr unsigned kFull = 0xffffffffu;
constexpr uint16_t kTerm16 = 0x8000u;

__device__ __forceinline__ Box mem_box(const SplitMem& m, uint32_t e) {
  Box b;
  for (int a = 0; a < 3; ++a) {
    b.lo[a] = m.bx[a * m.stride + e];
    b.hi[a] = m.bx[(3 + a) * m.stride + e];
  }
  return b;
}
__device__ __forceinline__ float mem_centre2(const SplitMem& m, uint32_t e, int axis) {
  return m.bx[axis * m.stride + e] + m.bx[(3 + axis) * m.stride + e];
}
__device__ __forceinline__ Box shfl_box(const Box& b, int src) {
  Box r;
  for (int a = 0; a < 3; ++a) {
    r.lo[a] = __shfl_sync(kFull, b.lo[a], src);
    r.hi[a] = __shfl_sync(kFull, b.hi[a], src);
  }
  return r;
}
// Inclusive scans of boxes over the lanes (from lane 0 up / from lane 31 down).
__device__ __forceinline__ Box scan_box_up(Box b) {
  const int lane = threadIdx.x & 31;
  for (int o = 1; o < 32; o <<= 1) {
    Box t;
    for (int a = 0; a < 3; ++a) {
      t.lo[a] = __shfl_up_sync(kFull, b.lo[a], o);
      t.hi[a] = __shfl_up_sync(kFull, b.hi[a], o);
    }
    if (lane >= o) box_add(b, t);
  }
  return b;
}
__device__ __forceinline__ Box scan_box_down(Box b) {
  const int lane = threadIdx.x & 31;
  for (int o = 1; o < 32; o <<= 1) {
    Box t;
    for (int a = 0; a < 3; ++a) {
      t.lo[a] = __shfl_down_sync(kFull, b.lo[a], o);
      t.hi[a] = __shfl_down_sync(kFull, b.hi[a], o);
    }
    if (lane + o < 32) box_add(b, t);
  }
  return b;
}
// Lane of the serial rule "start from lane 0, take a later one when strictly
// smaller": the first smallest value, or lane 0 if its value is NaN.
__device__ __forceinline__ int first_smallest(float h, bool valid) {
  const int lane = threadIdx.x & 31;
  uint32_t k = (valid && h == h) ? fkey(h) : 0xffffffffu;
  if (lane == 0 && !(h == h)) k = 0u;
  const uint32_t best = __reduce_min_sync(kFull, k);
  return __ffs(__ballot_sync(kFull, k == best)) - 1;
}

// Span statistics (16 spans of counts and box keys) -> the chosen span, or -1
// when none keeps 1/16 of the boxes on each side (FWNFS.h:5684-5706), with
// the left / right boxes of that span.  Lane i holds span i.
__device__ int choose_span(const uint32_t* cnt, const uint32_t (*keys)[6], uint32_t n, Box& Lb,
                           Box& Rb, uint32_t& left_count, uint32_t& lc0, uint32_t& lc14) {
  const int lane = threadIdx.x & 31;
  Box b;
  box_empty(b);
  uint32_t lc = 0;
  if (lane < kSpans && cnt[lane]) {
    lc = cnt[lane];
    b = keys_box(keys[lane]);
  }
  const Box L = scan_box_up(b);
  Box R = scan_box_down(b);
  for (int a = 0; a < 3; ++a) {  // the spans after this lane's
    R.lo[a] = __shfl_down_sync(kFull, R.lo[a], 1);
    R.hi[a] = __shfl_down_sync(kFull, R.hi[a], 1);
  }
  for (int o = 1; o < 32; o <<= 1) {
    const uint32_t t = __shfl_up_sync(kFull, lc, o);
    if (lane >= o) lc += t;
  }
  const uint32_t min_count = n / kMinFraction;
  const uint32_t max_count = (uint32_t)(((uint64_t)(kMinFraction - 1) * n) / kMinFraction);
  const float h = (float)lc * half_area(L) + (float)(n - lc) * half_area(R);
  const bool ok = lane < kSplits && lc >= min_count && lc <= max_count && h < INFINITY;
  const uint32_t k = ok ? fkey(h) : 0xffffffffu;
  const uint32_t best = __reduce_min_sync(kFull, k);
  lc0 = __shfl_sync(kFull, lc, 0);
  lc14 = __shfl_sync(kFull, lc, kSplits - 1);
  if (best == 0xffffffffu) return -1;
  const int si = __ffs(__ballot_sync(kFull, k == best)) - 1;
  Lb = shfl_box(L, si);
  Rb = shfl_box(R, si);
  left_count = __shfl_sync(kFull, lc, si);
  return si;
}

// The fallback's target order statistic (FWNFS.h:5718-5740).
__device__ __forceinline__ uint32_t nth_target(uint32_t n, uint32_t lc0, uint32_t lc14) {
  const uint32_t min_count = n / kMinFraction;
  const uint32_t max_count = (uint32_t)(((uint64_t)(kMinFraction - 1) * n) / kMinFraction);
  if (lc0 > max_count) return max_count;
  if (lc14 < min_count) return min_count;
  return n / 2;
}

// Median of three centres as nthElement picks its pivot (FWNFS.h:5852-5870).
__device__ __forceinline__ float median3(float a, float b, float c) {
  float p0 = a, p1 = b, p2 = c, t;
  if (p0 < p1) { t = p0; p0 = p1; p1 = t; }
  if (p0 < p2) { t = p0; p0 = p2; p2 = t; }
  if (p1 < p2) { t = p1; p1 = p2; p2 = t; }
  return p1;
}

// Prefix state of the partition's tapes: boxes below / equal to the pivot so
// far, and the counts at the first equal / first upper box.
struct TapeState {
  uint32_t nL = 0, nE = 0, firstE = kNone, firstG = kNone, L_atE = 0, LE_atG = 0;
};
// One lane's box (class k: 0 below, 1 equal, 2 above, 3 none) of 32 at job
// position rel: advances the state and returns what the box writes: its
// place below the pivot (L), its tape entries.
struct TapeOps {
  uint32_t L, te, tg, rotE, rotG;
  bool afterE, afterG;
};
__device__ __forceinline__ TapeOps tape_step(TapeState& s, int k, uint32_t rel0) {
  const int lane = threadIdx.x & 31;
  const unsigned lt = (1u << lane) - 1u;
  const unsigned mL = __ballot_sync(kFull, k == 0), mE = __ballot_sync(kFull, k == 1),
                 mG = __ballot_sync(kFull, k == 2);
  if (s.firstE == kNone && mE) {
    const int f = __ffs(mE) - 1;
    s.firstE = rel0 + f;
    s.L_atE = s.nL + __popc(mL & ((1u << f) - 1u));
  }
  if (s.firstG == kNone && mG) {
    const int f = __ffs(mG) - 1;
    s.firstG = rel0 + f;
    s.LE_atG = s.nL + s.nE + __popc((mL | mE) & ((1u << f) - 1u));
  }
  TapeOps o;
  const uint32_t rel = rel0 + lane;
  o.L = s.nL + __popc(mL & lt);
  const uint32_t E = s.nE + __popc(mE & lt), G = rel - o.L - E;
  o.afterE = s.firstE != kNone && rel > s.firstE;
  o.afterG = s.firstG != kNone && rel > s.firstG;
  o.rotE = o.afterE ? o.L - s.L_atE : 0u;
  o.rotG = o.afterG ? (o.L + E) - s.LE_atG : 0u;
  o.te = E + o.rotE;
  o.tg = G + o.rotG;
  s.nL += __popc(mL);
  s.nE += __popc(mE);
  return o;
}

// partitionByCentre of positions [lo, hi) about the pivot (see the file
// comment: the queues' tapes), by one warp in shared memory.
__device__ void warp_partition(const SplitMem& m, int axis, uint32_t lo, uint32_t hi, float pivot,
                               uint32_t& ps, uint32_t& pe) {
  const int lane = threadIdx.x & 31;
  TapeState s;
  for (uint32_t base = lo; base < hi; base += 32) {
    const uint32_t p = base + lane;
    uint16_t e = 0;
    int k = 3;
    if (p < hi) {
      e = m.perm[p];
      const float c = mem_centre2(m, e, axis);
      k = c < pivot ? 0 : (c == pivot ? 1 : 2);
    }
    const TapeOps o = tape_step(s, k, base - lo);
    if (k == 0) {
      m.tmp[lo + o.L] = e;
      if (o.afterE) m.tape_e[lo + o.te] = (uint16_t)o.rotE;
      if (o.afterG) m.tape_g[lo + o.tg] = (uint16_t)o.rotG;
    } else if (k == 1) {
      m.tape_e[lo + o.te] = kTerm16 | e;
      if (o.afterG) m.tape_g[lo + o.tg] = (uint16_t)o.rotG;
    } else if (k == 2) {
      m.tape_g[lo + o.tg] = kTerm16 | e;
    }
  }
  __syncwarp();
  const uint32_t RE = s.firstE != kNone ? s.nL - s.L_atE : 0u;
  const uint32_t RG = s.firstG != kNone ? s.nL + s.nE - s.LE_atG : 0u;
  for (uint32_t rel = lane; rel < hi - lo; rel += 32) {
    uint16_t v;
    if (rel < s.nL) {
      v = m.tmp[lo + rel];
    } else {
      const bool eq = rel < s.nL + s.nE;
      const uint16_t* tape = (eq ? m.tape_e : m.tape_g) + lo;
      v = tape[eq ? RE + (rel - s.nL) : RG + (rel - s.nL - s.nE)];
      while (!(v & kTerm16)) v = tape[v];  // each copy refers to an earlier entry
    }
    m.perm[lo + rel] = v & (kTerm16 - 1);
  }
  __syncwarp();
  ps = lo + s.nL;
  pe = ps + s.nE;
}

// One split of the boxes at positions [s, s + n) (FWNFS.h:5350-5800); box
// `all` is the range's; the cut is [s, mid), [mid, s + n).  Every lane gets
// the results.
__device__ void warp_split(const SplitMem& m, SplitScratch& sc, uint32_t s, uint32_t n,
                           const Box& all, uint32_t& mid, Box& o0, Box& o1, unsigned* status) {
  const int lane = threadIdx.x & 31;
  if (n == 2) {
    o0 = mem_box(m, m.perm[s]);
    o1 = mem_box(m, m.perm[s + 1]);
    mid = s + 1;
    return;
  }
  if (n <= 6) {  // every 2-partition with box 0 on side 0, one per lane
    const uint32_t bits = lane + 1;
    const bool valid = bits < (1u << (n - 1));
    Box s0 = mem_box(m, m.perm[s]), s1;
    box_empty(s1);
    uint32_t c0 = 1, c1 = 0;
    for (uint32_t b = 0; b + 1 < n; ++b) {
      const Box x = mem_box(m, m.perm[s + b + 1]);
      if ((bits >> b) & 1u) {
        box_add(s1, x);
        ++c1;
      } else {
        box_add(s0, x);
        ++c0;
      }
    }
    const float h = half_area(s0) * (float)c0 + half_area(s1) * (float)c1;
    const int w = first_smallest(h, valid);
    o0 = shfl_box(s0, w);
    o1 = shfl_box(s1, w);
    const uint32_t best = (uint32_t)w + 1, zeros = (n - 1) - __popc(best);
    mid = s + 1 + zeros;
    uint16_t e = 0;
    uint32_t to = 0;
    const bool move = lane >= 1 && (uint32_t)lane < n;
    if (move) {
      e = m.perm[s + lane];
      const uint32_t below = (1u << (lane - 1)) - 1u;
      to = ((best >> (lane - 1)) & 1u) ? 1 + zeros + __popc(best & below)
                                       : 1 + __popc(~best & below);
    }
    __syncwarp();
    if (move) m.perm[s + to] = e;
    __syncwarp();
    return;
  }
  float len;
  const int axis = longest_axis(all, len);
  if (!(len > 0.f)) {  // a single point or NaN: an arbitrary split
    mid = s + n / 2;
    o0 = all;
    o1 = all;
    return;
  }
  if (n <= kSmallMax) {
    // stable sort by centre (the reference's chunked insertion sort + merges
    // is a stable sort), one box per lane, then the sweep by scans
    const bool in = (uint32_t)lane < n;
    const uint16_t e = in ? m.perm[s + lane] : 0;
    const float c = in ? mem_centre2(m, e, axis) : 0.f;
    uint32_t rank = 0;
    for (uint32_t j = 0; j < n; ++j) {
      const float cj = __shfl_sync(kFull, c, j);
      if (cj < c || (cj == c && j < (uint32_t)lane)) ++rank;
    }
    __syncwarp();
    if (in) m.perm[s + rank] = e;
    __syncwarp();
    const uint32_t ns = n - 1;
    Box b, r;
    box_empty(b);
    box_empty(r);
    if (in) b = mem_box(m, m.perm[s + lane]);
    const Box L = scan_box_up(b);
    // right boxes as the reference accumulates them: starting from box ns-1,
    // so the last box never enters (FWNFS.h:5560-5565)
    if ((uint32_t)lane < ns) r = b;
    Box R = scan_box_down(r);
    Box R1;
    for (int a = 0; a < 3; ++a) {
      R1.lo[a] = __shfl_down_sync(kFull, R.lo[a], 1);
      R1.hi[a] = __shfl_down_sync(kFull, R.hi[a], 1);
    }
    if ((uint32_t)lane + 1 < ns) R = R1;  // lane ns-1 keeps box ns-1
    const float h = half_area(L) * (float)(lane + 1) + half_area(R) * (float)(n - (lane + 1));
    const int w = first_smallest(h, (uint32_t)lane < ns);
    mid = s + w + 1;
    o0 = shfl_box(L, w);
    o1 = shfl_box(R, w);
    return;
  }
  // spans
  for (int i = lane; i < kSpans; i += 32) {
    sc.cnt[i] = 0;
    keys_init(sc.keys[i]);
  }
  __syncwarp();
  const float min2 = 2.0f * all.lo[axis];
  const float scale = (0.5f * (float)kSpans) / len;
  for (uint32_t p = s + lane; p < s + n; p += 32) {
    const Box b = mem_box(m, m.perm[p]);
    const int si = span_of(centre2(b, axis), min2, scale);
    atomicAdd(&sc.cnt[si], 1u);
    keys_add(sc.keys[si], b);
  }
  __syncwarp();
  uint32_t lcs = 0, lc0, lc14, ps, pe;
  const int si = choose_span(sc.cnt, sc.keys, n, o0, o1, lcs, lc0, lc14);
  if (si >= 0) {
    const float pivot = min2 + (float)(si + 1) * len / (float)(kSpans / 2);
    warp_partition(m, axis, s, s + n, pivot, ps, pe);
    mid = s + lcs;
    if (mid >= ps && mid <= pe) return;
    mid = mid < ps ? ps : pe;
    if (mid == s) ++mid;
    else if (mid == s + n) --mid;
  } else {
    // nthElement: each step narrows [lo, hi) by at least the pivot's own
    // box; the bound only guards against a hang
    mid = s + nth_target(n, lc0, lc14);
    uint32_t lo = s, hi = s + n;
    bool done = false;
    for (uint32_t step = 0; step <= n && !done; ++step) {
      const float pv = median3(mem_centre2(m, m.perm[lo], axis),
                               mem_centre2(m, m.perm[lo + (hi - lo) / 2], axis),
                               mem_centre2(m, m.perm[hi - 1], axis));
      __syncwarp();
      warp_partition(m, axis, lo, hi, pv, ps, pe);
      if (mid < ps) hi = ps;
      else if (mid < pe) done = true;
      else lo = pe;
      if (hi <= lo + 1) done = true;
    }
    if (!done && lane == 0) atomicOr(status, kStatusInternal);
  }
  // the cut moved off the span's, or came from nthElement: the sides' boxes
  uint32_t k0[6], k1[6];
  keys_init(k0);
  keys_init(k1);
  for (uint32_t p = s + lane; p < s + n; p += 32) {
    const Box b = mem_box(m, m.perm[p]);
    uint32_t* k = p < mid ? k0 : k1;
    for (int a = 0; a < 3; ++a) {
      k[a] = min(k[a], fkey(b.lo[a]));
      k[3 + a] = max(k[3 + a], fkey(b.hi[a]));
    }
  }
  for (int a = 0; a < 3; ++a) {
    k0[a] = __reduce_min_sync(kFull, k0[a]);
    k1[a] = __reduce_min_sync(kFull, k1[a]);
    k0[3 + a] = __reduce_max_sync(kFull, k0[3 + a]);
    k1[3 + a] = __reduce_max_sync(kFull, k1[3 + a]);
  }
  o0 = keys_box(k0);
  o1 = keys_box(k1);
}

// The part a node splits in rounds 1 and 2: the largest area x count, the
// first on ties.
__device__ __forceinline__ int choose_part(const uint32_t* cut, const float* area, int nsub) {
  int choice = -1;
  float best = 0.f;
  for (int i = 0; i < nsub; ++i) {
    const uint32_t c = cut[i + 1] - cut[i];
    if (c > 1) {
      const float h = area[i] * (float)c;
      if (choice < 0 || h > best) {
        choice = i;
        best = h;
      }
    }
  }
  return choice;
}
// Part c of nsub becomes two, cut at mid with boxes o0, o1.
__device__ __forceinline__ void insert_cut(uint32_t* cut, Box* sub, float* area, int nsub, int c,
                                           uint32_t mid, const Box& o0, const Box& o1) {
  for (int i = nsub; i > c; --i) cut[i + 1] = cut[i];
  for (int i = nsub - 1; i > c; --i) {
    sub[i + 1] = sub[i];
    area[i + 1] = area[i];
  }
  cut[c + 1] = mid;
  sub[c] = o0;
  sub[c + 1] = o1;
  area[c] = half_area(o0);
  area[c + 1] = half_area(o1);
}

// ------------------------------------------------------------- subtrees --
struct SubList {  // a node of the current depth with more than 4 boxes
  uint16_t s, n, id, pad;
  Box all;
};
constexpr int kSubWarps = 8;
constexpr int kSubListCap = kSub / 5 + 1;
struct SubShared {
  union {
    float bx[6][kSub];
    struct {
      uint16_t nodes[kSub], slots[kSub], items[kSub], pre[kSub], slot[kSub], item[kSub];
    } z;
  };
  uint16_t perm[kSub], tmp[kSub], tape_e[kSub], tape_g[kSub];
  uint16_t child[kSub][4];
  uint16_t lev[kSub + 2];  // depth d: local ids [lev[d], lev[d + 1])
  SplitScratch sc[kSubWarps];
  SubList list[2][kSubListCap];
  uint32_t nodes, take, next;
};

// Builds the whole subtree below each root in shared memory, one CTA per
// subtree: depth by depth, a warp per node, the node's three splits one after
// the other (multiSplit).  In place of one launch per depth, round and size
// class with host reads between them (82k triangles: 400 launches and 80
// blocking reads, 5.7 ms).
__global__ void __launch_bounds__(kSubWarps * 32) subtree_kernel(
    const SubRoot* __restrict__ roots, uint32_t nroots, const uint32_t* __restrict__ idx,
    const Box* __restrict__ tb, SubNode* __restrict__ out,
    uint16_t* __restrict__ lev_out, SubTotals* __restrict__ totals, unsigned* __restrict__ status) {
  extern __shared__ __align__(16) unsigned char s_raw[];
  SubShared& S = *reinterpret_cast<SubShared*>(s_raw);
  if (blockIdx.x >= nroots) return;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const SubRoot root = roots[blockIdx.x];
  for (uint32_t i = tid; i < root.n; i += blockDim.x) {
    const Box b = tb[idx[root.start + i]];
    for (int a = 0; a < 3; ++a) {
      S.bx[a][i] = b.lo[a];
      S.bx[3 + a][i] = b.hi[a];
    }
    S.perm[i] = (uint16_t)i;
  }
  if (tid == 0) {
    S.nodes = 1;
    S.lev[0] = 0;
    S.lev[1] = 1;
    if (root.n <= 4) {
      for (uint32_t i = 0; i < 4; ++i) S.child[0][i] = i < root.n ? (uint16_t)i : kSubNone;
    } else {
      S.list[0][0] = SubList{0, (uint16_t)root.n, 0, 0, root.all};
    }
  }
  const SplitMem mem{&S.bx[0][0], (int)kSub, S.perm, S.tmp, S.tape_e, S.tape_g};
  SplitScratch& sc = S.sc[warp];
  uint32_t ncur = root.n <= 4 ? 0 : 1;
  uint32_t depths = 1;
  int cur = 0;
  while (ncur > 0) {
    if (tid == 0) S.take = S.next = 0;
    __syncthreads();
    for (;;) {
      uint32_t k = 0;
      if (lane == 0) k = atomicAdd(&S.take, 1u);
      k = __shfl_sync(kFull, k, 0);
      if (k >= ncur) break;
      const SubList N = S.list[cur][k];
      if (lane == 0) {
        sc.cut[0] = N.s;
        sc.cut[1] = (uint32_t)N.s + N.n;
      }
      __syncwarp();
      for (int round = 0; round < 3; ++round) {
        const int c = round == 0 ? 0 : choose_part(sc.cut, sc.area, round + 1);
        const uint32_t s = sc.cut[c], n = sc.cut[c + 1] - s;
        const Box all = round == 0 ? N.all : sc.sub[c];
        uint32_t mid;
        Box o0, o1;
        warp_split(mem, sc, s, n, all, mid, o0, o1, status);
        __syncwarp();
        if (lane == 0) insert_cut(sc.cut, sc.sub, sc.area, round + 1, c, mid, o0, o1);
        __syncwarp();
      }
      // children: lane i takes part i
      const uint32_t s = lane < 4 ? sc.cut[lane] : 0, n = lane < 4 ? sc.cut[lane + 1] - s : 1;
      const unsigned inner = __ballot_sync(kFull, n > 1);
      uint32_t id = 0;
      if (lane == 0) id = atomicAdd(&S.nodes, (uint32_t)__popc(inner));
      id = __shfl_sync(kFull, id, 0) + __popc(inner & ((1u << lane) - 1u));
      if (lane < 4) {
        S.child[N.id][lane] = n > 1 ? (uint16_t)(kSubNode | id) : S.perm[s];
        if (n > 4) {
          S.list[cur ^ 1][atomicAdd(&S.next, 1u)] =
              SubList{(uint16_t)s, (uint16_t)n, (uint16_t)id, 0, sc.sub[lane]};
        } else if (n > 1) {
          for (uint32_t i = 0; i < 4; ++i) S.child[id][i] = i < n ? S.perm[s + i] : kSubNone;
        }
      }
      __syncwarp();
    }
    __syncthreads();
    ncur = S.next;
    cur ^= 1;
    const uint32_t made = S.nodes;
    if (made > S.lev[depths]) ++depths;
    __syncthreads();
    if (tid == 0) S.lev[depths] = (uint16_t)made;
    __syncthreads();
  }
  __syncthreads();  // the boxes' memory is reused from here
  for (uint32_t d = depths; d-- > 0;) {
    for (uint32_t x = S.lev[d] + tid; x < S.lev[d + 1]; x += blockDim.x) {
      uint32_t nodes = 1, slots = 1, items = 0;
      for (int i = 0; i < 4; ++i) {
        const uint16_t c = S.child[x][i];
        if (c == kSubNone) continue;
        if (c & kSubNode) {
          nodes += S.z.nodes[c & ~kSubNode];
          slots += S.z.slots[c & ~kSubNode];
          items += S.z.items[c & ~kSubNode];
        } else {
          ++slots;
          ++items;
        }
      }
      S.z.nodes[x] = (uint16_t)nodes;
      S.z.slots[x] = (uint16_t)slots;
      S.z.items[x] = (uint16_t)items;
    }
    __syncthreads();
  }
  if (tid == 0) {
    S.z.pre[0] = S.z.slot[0] = S.z.item[0] = 0;
    totals[blockIdx.x] = SubTotals{S.nodes, S.z.slots[0], depths};
  }
  __syncthreads();
  for (uint32_t d = 0; d < depths; ++d) {
    for (uint32_t x = S.lev[d] + tid; x < S.lev[d + 1]; x += blockDim.x) {
      uint32_t pre = S.z.pre[x] + 1, slot = S.z.slot[x] + 1, item = S.z.item[x];
      SubNode o;
      o.pre = S.z.pre[x];
      o.slot = S.z.slot[x];
      o.item = S.z.item[x];
      o.nslots = S.z.slots[x];
      o.nitems = S.z.items[x];
      o.pad = 0;
      for (int i = 0; i < 4; ++i) {
        const uint16_t c = S.child[x][i];
        o.child[i] = c;
        if (c == kSubNone) continue;
        if (c & kSubNode) {
          const uint32_t y = c & ~kSubNode;
          S.z.pre[y] = (uint16_t)pre;
          S.z.slot[y] = (uint16_t)slot;
          S.z.item[y] = (uint16_t)item;
          pre += S.z.nodes[y];
          slot += S.z.slots[y];
          item += S.z.items[y];
        } else {
          ++slot;
          ++item;
        }
      }
      out[root.start + x] = o;
    }
    __syncthreads();
  }
  for (uint32_t d = tid; d <= depths; d += blockDim.x) lev_out[root.start + d] = S.lev[d];
}
// ------------------------------------------------------- the top of the tree --
// Nodes of more than kSub boxes, one depth at a time.  Their splits run by
// size: up to kSub boxes in a warp, up to kCtaMax in a CTA, more across the
// GPU; every kernel reads its task count on the device, so a depth ends with
// one host read.
__global__ void __launch_bounds__(32) part_warp_kernel(RNode* __restrict__ nodes,
                                                       const uint32_t* __restrict__ list,
                                                       const uint32_t* __restrict__ count,
                                                       uint32_t* __restrict__ idx,
                                                       const Box* __restrict__ tb,
                                                       unsigned* __restrict__ status) {
  __shared__ float bx[6][kSub];
  __shared__ uint32_t id[kSub];
  __shared__ uint16_t perm[kSub], tmp[kSub], tape_e[kSub], tape_g[kSub];
  __shared__ SplitScratch sc;
  if (blockIdx.x >= *count) return;
  const int lane = threadIdx.x;
  RNode& N = nodes[list[blockIdx.x]];
  const uint32_t s = N.t_start, n = N.t_n;
  for (uint32_t i = lane; i < n; i += 32) {
    id[i] = idx[s + i];
    const Box b = tb[id[i]];
    for (int a = 0; a < 3; ++a) {
      bx[a][i] = b.lo[a];
      bx[3 + a][i] = b.hi[a];
    }
    perm[i] = (uint16_t)i;
  }
  __syncwarp();
  const SplitMem mem{&bx[0][0], (int)kSub, perm, tmp, tape_e, tape_g};
  const Box all = N.t_box;
  uint32_t mid;
  Box o0, o1;
  warp_split(mem, sc, 0, n, all, mid, o0, o1, status);
  __syncwarp();
  for (uint32_t i = lane; i < n; i += 32) idx[s + i] = id[perm[i]];
  if (lane == 0) {
    N.t_mid = s + mid;
    N.t_out[0] = o0;
    N.t_out[1] = o1;
  }
}

// Entries first, first + stride, .. below n of a tape follow their copies back to
// a box.  All entries walk at once and keep their progress in the tape, so a walk
// meets entries that are already (partly) resolved: pointer doubling without
// rounds.  Each step goes to an earlier entry, so a walk ends whatever the others
// do.
__device__ __forceinline__ void resolve_tape(uint32_t* tape, uint32_t n, uint32_t first,
                                             uint32_t stride) {
  for (uint32_t rel = first; rel < n; rel += stride) {
    uint32_t at = rel, v = __ldcg(tape + rel);
    while (!(v & kTerm) && v < at) {
      at = v;
      v = __ldcg(tape + v);
      __stcg(tape + rel, v);
    }
  }
}

// partitionByCentre of positions [lo, hi) by one CTA of 32 warps, centres in
// cen: each warp counts its segment, the segments' prefixes give every warp
// its tape state, then the tapes are written and resolved.
struct CtaPart {
  uint32_t nL[32], nE[32], fE[32], fG[32], L_atE[32], LE_atG[32];
};
__device__ void cta_partition(CtaPart& S, uint32_t* idx, float* cen, uint32_t* tmp,
                              uint32_t* tape_e, uint32_t* tape_g, uint32_t lo, uint32_t hi,
                              float pivot, uint32_t& ps, uint32_t& pe) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const uint32_t jn = hi - lo, seg = (jn + 1023) / 1024 * 32;
  const uint32_t wlo = min(hi, lo + warp * seg), whi = min(hi, wlo + seg);
  auto cls = [&](uint32_t p) {
    if (p >= whi) return 3;
    const float c = cen[p];
    return c < pivot ? 0 : (c == pivot ? 1 : 2);
  };
  TapeState w;
  for (uint32_t base = wlo; base < whi; base += 32) tape_step(w, cls(base + lane), base - lo);
  if (lane == 0) {
    S.nL[warp] = w.nL;
    S.nE[warp] = w.nE;
    S.fE[warp] = w.firstE;
    S.fG[warp] = w.firstG;
    S.L_atE[warp] = w.L_atE;
    S.LE_atG[warp] = w.LE_atG;
  }
  __syncthreads();
  // lane i holds warp i's counts; exclusive prefixes
  uint32_t aL = S.nL[lane], aE = S.nE[lane];
  for (int o = 1; o < 32; o <<= 1) {
    const uint32_t tL = __shfl_up_sync(kFull, aL, o), tE = __shfl_up_sync(kFull, aE, o);
    if (lane >= o) {
      aL += tL;
      aE += tE;
    }
  }
  const uint32_t nL = __shfl_sync(kFull, aL, 31), nE = __shfl_sync(kFull, aE, 31);
  aL -= S.nL[lane];
  aE -= S.nE[lane];
  const unsigned hasE = __ballot_sync(kFull, S.fE[lane] != kNone),
                 hasG = __ballot_sync(kFull, S.fG[lane] != kNone);
  TapeState t;
  t.nL = __shfl_sync(kFull, aL, warp);
  t.nE = __shfl_sync(kFull, aE, warp);
  if (hasE) {
    const int f = __ffs(hasE) - 1;
    t.firstE = S.fE[f];
    t.L_atE = S.L_atE[f] + __shfl_sync(kFull, aL, f);
  }
  if (hasG) {
    const int f = __ffs(hasG) - 1;
    t.firstG = S.fG[f];
    t.LE_atG = S.LE_atG[f] + __shfl_sync(kFull, aL + aE, f);
  }
  for (uint32_t base = wlo; base < whi; base += 32) {
    const uint32_t p = base + lane;
    const int k = cls(p);
    const uint32_t e = p < whi ? idx[p] : 0;
    const TapeOps o = tape_step(t, k, base - lo);
    if (k == 0) {
      tmp[lo + o.L] = e;
      if (o.afterE) tape_e[lo + o.te] = o.rotE;
      if (o.afterG) tape_g[lo + o.tg] = o.rotG;
    } else if (k == 1) {
      tape_e[lo + o.te] = kTerm | e;
      if (o.afterG) tape_g[lo + o.tg] = o.rotG;
    } else if (k == 2) {
      tape_g[lo + o.tg] = kTerm | e;
    }
  }
  __syncthreads();
  const uint32_t RE = t.firstE != kNone ? nL - t.L_atE : 0u;
  const uint32_t RG = t.firstG != kNone ? nL + nE - t.LE_atG : 0u;
  resolve_tape(tape_e + lo, nE + RE, threadIdx.x, blockDim.x);
  resolve_tape(tape_g + lo, jn - nL - nE + RG, threadIdx.x, blockDim.x);
  __syncthreads();
  for (uint32_t rel = threadIdx.x; rel < jn; rel += blockDim.x) {
    uint32_t v;
    if (rel < nL) v = tmp[lo + rel];
    else if (rel < nL + nE) v = __ldcg(tape_e + lo + RE + (rel - nL));
    else v = __ldcg(tape_g + lo + RG + (rel - nL - nE));
    idx[lo + rel] = v & ~kTerm;
  }
  __syncthreads();
  ps = lo + nL;
  pe = ps + nE;
}

// nthElement (FWNFS.h:5847-5900) of positions [lo, hi) about position mid by one
// CTA; false if it did not end, which cannot happen: each step narrows [lo, hi)
// by at least the pivot's own box, the bound only guards against a hang.
__device__ bool cta_nth(CtaPart& S, uint32_t* idx, float* cen, uint32_t* tmp, uint32_t* tape_e,
                        uint32_t* tape_g, const Box* __restrict__ tb, int axis, uint32_t lo,
                        uint32_t hi, uint32_t mid) {
  bool done = false;
  for (uint32_t step = 0, n = hi - lo; step <= n && !done; ++step) {
    const float pv = median3(cen[lo], cen[lo + (hi - lo) / 2], cen[hi - 1]);
    __syncthreads();
    uint32_t ps, pe;
    cta_partition(S, idx, cen, tmp, tape_e, tape_g, lo, hi, pv, ps, pe);
    for (uint32_t p = lo + threadIdx.x; p < hi; p += blockDim.x) cen[p] = centre2(tb[idx[p]], axis);
    if (mid < ps) hi = ps;
    else if (mid < pe) done = true;
    else lo = pe;
    if (hi <= lo + 1) done = true;
    __syncthreads();
  }
  return done;
}

__global__ void __launch_bounds__(1024) part_cta_kernel(
    RNode* nodes, const uint32_t* list, const uint32_t* count, uint32_t* idx, float* cen,
    uint32_t* tmp, uint32_t* tape_e, uint32_t* tape_g, const Box* __restrict__ tb,
    unsigned* status) {
  __shared__ uint32_t s_cnt[32][kSpans];
  __shared__ uint32_t s_keys[32][kSpans][6];
  __shared__ CtaPart s_part;
  __shared__ Box s_L, s_R;
  __shared__ int s_si;
  __shared__ uint32_t s_lcs, s_target, s_bk[2][6];
  if (blockIdx.x >= *count) return;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  RNode& N = nodes[list[blockIdx.x]];
  const uint32_t s = N.t_start, n = N.t_n;
  const Box B = N.t_box;
  float len;
  const int axis = longest_axis(B, len);
  if (!(len > 0.f)) {
    __syncthreads();
    if (tid == 0) {
      N.t_mid = s + n / 2;
      N.t_out[0] = B;
      N.t_out[1] = B;
    }
    return;
  }
  for (int i = lane; i < kSpans; i += 32) {
    s_cnt[warp][i] = 0;
    keys_init(s_keys[warp][i]);
  }
  if (tid < 2) keys_init(s_bk[tid]);
  __syncwarp();
  const float min2 = 2.0f * B.lo[axis];
  const float scale = (0.5f * (float)kSpans) / len;
  for (uint32_t p = s + tid; p < s + n; p += blockDim.x) {
    const Box b = tb[idx[p]];
    const float c = centre2(b, axis);
    cen[p] = c;
    const int si = span_of(c, min2, scale);
    atomicAdd(&s_cnt[warp][si], 1u);
    keys_add(s_keys[warp][si], b);
  }
  __syncthreads();
  if (tid < kSpans * 7) {  // the warps' tables into the first
    const int i = tid / 7, f = tid % 7;
    if (f == 6) {
      uint32_t v = 0;
      for (int w = 0; w < 32; ++w) v += s_cnt[w][i];
      s_cnt[0][i] = v;
    } else {
      uint32_t v = s_keys[0][i][f];
      for (int w = 1; w < 32; ++w) v = f < 3 ? min(v, s_keys[w][i][f]) : max(v, s_keys[w][i][f]);
      s_keys[0][i][f] = v;
    }
  }
  __syncthreads();
  if (warp == 0) {
    uint32_t lcs = 0, lc0, lc14;
    Box Lb = B, Rb = B;
    const int si = choose_span(s_cnt[0], s_keys[0], n, Lb, Rb, lcs, lc0, lc14);
    if (lane == 0) {
      s_si = si;
      s_lcs = lcs;
      s_target = nth_target(n, lc0, lc14);
      s_L = Lb;
      s_R = Rb;
    }
  }
  __syncthreads();
  uint32_t mid, ps, pe;
  if (s_si >= 0) {
    const float pivot = min2 + (float)(s_si + 1) * len / (float)(kSpans / 2);
    cta_partition(s_part, idx, cen, tmp, tape_e, tape_g, s, s + n, pivot, ps, pe);
    mid = s + s_lcs;
    if (mid >= ps && mid <= pe) {
      if (tid == 0) {
        N.t_mid = mid;
        N.t_out[0] = s_L;
        N.t_out[1] = s_R;
      }
      return;
    }
    mid = mid < ps ? ps : pe;
    if (mid == s) ++mid;
    else if (mid == s + n) --mid;
  } else {
    mid = s + s_target;
    if (!cta_nth(s_part, idx, cen, tmp, tape_e, tape_g, tb, axis, s, s + n, mid) && tid == 0)
      atomicOr(status, kStatusInternal);
  }
  // the cut moved off the span's, or came from nthElement: the sides' boxes
  for (uint32_t p0 = s; p0 < s + n; p0 += blockDim.x) {
    const uint32_t p = p0 + tid;
    const bool in = p < s + n;
    const Box b = in ? tb[idx[p]] : B;
    for (int side = 0; side < 2; ++side) {
      const bool mine = in && (p < mid) == (side == 0);
      for (int a = 0; a < 3; ++a) {
        const uint32_t l = __reduce_min_sync(kFull, mine ? fkey(b.lo[a]) : 0xffffffffu);
        const uint32_t h = __reduce_max_sync(kFull, mine ? fkey(b.hi[a]) : 0u);
        if (lane == 0) {
          atomicMin(&s_bk[side][a], l);
          atomicMax(&s_bk[side][3 + a], h);
        }
      }
    }
  }
  __syncthreads();
  if (tid == 0) {
    N.t_mid = mid;
    N.t_out[0] = keys_box(s_bk[0]);
    N.t_out[1] = keys_box(s_bk[1]);
  }
}

// ---------------------------------------------- splits across the GPU --
struct LTask {
  uint32_t node, start, n;
  int32_t axis;
  float len, min2, scale, pivot;
  uint32_t cnt[kSpans];
  uint32_t keys[kSpans][6];
  Box Lb, Rb;
  uint32_t lcs;
  int32_t live;                        // takes part in the partition
  int32_t more;                        // nthElement has not ended
  uint32_t chunk0;                     // its first chunk
  uint32_t firstE, firstG, nL, nE;     // of the partition, relative to start
  uint32_t L_atE, LE_atG;              // prefix counts at firstE / firstG
  uint32_t mid;
  int32_t need;                        // the sides' boxes must be recomputed
  uint32_t bk[2][6];
};

// Tasks of the list and their chunks of kChunk positions; one CTA.  A task
// with no longest axis goes to the CTA kernel's list.
__global__ void wide_init_kernel(const RNode* __restrict__ nodes,
                                 const uint32_t* __restrict__ list,
                                 const uint32_t* __restrict__ count, LTask* __restrict__ T,
                                 int4* __restrict__ chunks, uint32_t* __restrict__ nchunks) {
  __shared__ uint32_t s_total;
  const uint32_t n = *count;
  if (threadIdx.x == 0) s_total = 0;
  for (uint32_t k0 = 0; k0 < n; k0 += 32) {  // warp 0: tasks and chunk offsets
    __syncthreads();
    if (threadIdx.x < 32) {
      const uint32_t k = k0 + threadIdx.x;
      uint32_t c = 0;
      if (k < n) {
        LTask& t = T[k];
        const RNode& N = nodes[list[k]];
        t.node = list[k];
        t.start = N.t_start;
        t.n = N.t_n;
        t.axis = longest_axis(N.t_box, t.len);
        t.min2 = 2.0f * N.t_box.lo[t.axis];
        t.scale = (0.5f * (float)kSpans) / t.len;
        for (int i = 0; i < kSpans; ++i) {
          t.cnt[i] = 0;
          keys_init(t.keys[i]);
        }
        keys_init(t.bk[0]);
        keys_init(t.bk[1]);
        t.live = t.len > 0.f;
        t.firstE = t.firstG = kNone;
        t.nL = t.nE = t.L_atE = t.LE_atG = 0;
        t.need = 0;
        c = (t.n + kChunk - 1) / kChunk;
      }
      uint32_t incl = c;
      for (int o = 1; o < 32; o <<= 1) {
        const uint32_t v = __shfl_up_sync(kFull, incl, o);
        if ((int)threadIdx.x >= o) incl += v;
      }
      if (k < n) T[k].chunk0 = s_total + incl - c;
      __syncwarp();
      if (threadIdx.x == 31) s_total += incl;
    }
  }
  __syncthreads();
  if (threadIdx.x == 0) *nchunks = s_total;
  for (uint32_t k = 0; k < n; ++k) {
    const uint32_t s = T[k].start, len = T[k].n, c0 = T[k].chunk0;
    for (uint32_t c = threadIdx.x; c * kChunk < len; c += blockDim.x)
      chunks[c0 + c] = make_int4((int)k, (int)(s + c * kChunk),
                                 (int)(s + min(len, (c + 1) * kChunk)), 0);
  }
}

__global__ void __launch_bounds__(256) wide_span_kernel(const int4* __restrict__ chunks,
                                                        const uint32_t* __restrict__ nchunks,
                                                        LTask* __restrict__ T,
                                                        const uint32_t* __restrict__ idx,
                                                        const Box* __restrict__ tb,
                                                        float* __restrict__ cen) {
  __shared__ uint32_t s_cnt[8][kSpans];
  __shared__ uint32_t s_keys[8][kSpans][6];
  if (blockIdx.x >= *nchunks) return;
  const int4 ch = chunks[blockIdx.x];
  LTask& t = T[ch.x];
  if (!t.live) return;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  for (int i = lane; i < kSpans; i += 32) {
    s_cnt[warp][i] = 0;
    keys_init(s_keys[warp][i]);
  }
  __syncwarp();
  const int axis = t.axis;
  const float min2 = t.min2, scale = t.scale;
  for (int p = ch.y + tid; p < ch.z; p += blockDim.x) {
    const Box b = tb[idx[p]];
    const float c = centre2(b, axis);
    cen[p] = c;
    const int si = span_of(c, min2, scale);
    atomicAdd(&s_cnt[warp][si], 1u);
    keys_add(s_keys[warp][si], b);
  }
  __syncthreads();
  if (tid < kSpans * 7) {
    const int i = tid / 7, f = tid % 7;
    uint32_t total = 0;
    for (int w = 0; w < 8; ++w) total += s_cnt[w][i];
    if (total) {
      if (f == 6) {
        atomicAdd(&t.cnt[i], total);
      } else {
        uint32_t v = s_keys[0][i][f];
        for (int w = 1; w < 8; ++w) v = f < 3 ? min(v, s_keys[w][i][f]) : max(v, s_keys[w][i][f]);
        if (f < 3) atomicMin(&t.keys[i][f], v);
        else atomicMax(&t.keys[i][f], v);
      }
    }
  }
}

// One warp per task: the span and pivot.  Without a longest axis the CTA kernel
// cuts it anywhere; without a balanced span the node waits for nthElement.
__global__ void wide_choose_kernel(LTask* __restrict__ T, const uint32_t* __restrict__ count,
                                   uint32_t* __restrict__ cta_list,
                                   uint32_t* __restrict__ cta_count, RNode* __restrict__ nodes,
                                   uint32_t* __restrict__ waiting, uint32_t* __restrict__ nwaiting) {
  if (blockIdx.x >= *count) return;
  LTask& t = T[blockIdx.x];
  const int lane = threadIdx.x;
  int si = -1;
  uint32_t lcs = 0, lc0 = 0, lc14 = 0;
  Box Lb, Rb;
  if (t.live) si = choose_span(t.cnt, t.keys, t.n, Lb, Rb, lcs, lc0, lc14);
  __syncwarp();
  if (lane != 0) return;
  if (si < 0) {
    if (t.live) {
      RNode& N = nodes[t.node];
      N.waiting = 1;
      N.t_mid = t.start + nth_target(t.n, lc0, lc14);
      waiting[atomicAdd(nwaiting, 1u)] = t.node;
    } else {
      cta_list[atomicAdd(cta_count, 1u)] = t.node;
    }
    t.live = 0;
    return;
  }
  t.Lb = Lb;
  t.Rb = Rb;
  t.lcs = lcs;
  t.pivot = t.min2 + (float)(si + 1) * t.len / (float)(kSpans / 2);
}

// Pass 1: counts of the classes (below, equal, above) per chunk, first equal
// and first upper box per task.
__global__ void __launch_bounds__(256) wide_classify_kernel(const int4* __restrict__ chunks,
                                                            const uint32_t* __restrict__ nchunks,
                                                            LTask* __restrict__ T,
                                                            const float* __restrict__ cen,
                                                            uint2* __restrict__ chunk_cnt) {
  __shared__ uint32_t s_n[2], s_f[2];
  if (blockIdx.x >= *nchunks) return;
  const int4 ch = chunks[blockIdx.x];
  LTask& t = T[ch.x];
  if (!t.live) return;
  const int tid = threadIdx.x, lane = tid & 31;
  if (tid < 2) {
    s_n[tid] = 0;
    s_f[tid] = kNone;
  }
  __syncthreads();
  const float pivot = t.pivot;
  uint32_t n0 = 0, n1 = 0, fE = kNone, fG = kNone;
  for (int p = ch.y + tid; p < ch.z; p += blockDim.x) {
    const float c = cen[p];
    const uint32_t rel = (uint32_t)p - t.start;
    if (c < pivot) {
      ++n0;
    } else if (c == pivot) {
      ++n1;
      fE = min(fE, rel);
    } else {
      fG = min(fG, rel);
    }
  }
  n0 = __reduce_add_sync(kFull, n0);
  n1 = __reduce_add_sync(kFull, n1);
  fE = __reduce_min_sync(kFull, fE);
  fG = __reduce_min_sync(kFull, fG);
  if (lane == 0) {
    atomicAdd(&s_n[0], n0);
    atomicAdd(&s_n[1], n1);
    atomicMin(&s_f[0], fE);
    atomicMin(&s_f[1], fG);
  }
  __syncthreads();
  if (tid == 0) {
    chunk_cnt[blockIdx.x] = make_uint2(s_n[0], s_n[1]);
    if (s_f[0] != kNone) atomicMin(&t.firstE, s_f[0]);
    if (s_f[1] != kNone) atomicMin(&t.firstG, s_f[1]);
  }
}

// Pass 2: one warp per task turns its chunks' counts into the counts before
// each chunk.
__global__ void wide_scan_kernel(LTask* __restrict__ T, const uint32_t* __restrict__ count,
                                 uint2* __restrict__ chunk_cnt) {
  if (blockIdx.x >= *count) return;
  LTask& t = T[blockIdx.x];
  if (!t.live) return;
  const int lane = threadIdx.x;
  const uint32_t nc = (t.n + kChunk - 1) / kChunk;
  uint32_t baseL = 0, baseE = 0;
  for (uint32_t c0 = 0; c0 < nc; c0 += 32) {
    const bool in = c0 + lane < nc;
    const uint2 v = in ? chunk_cnt[t.chunk0 + c0 + lane] : make_uint2(0, 0);
    uint32_t a = v.x, b = v.y;
    for (int o = 1; o < 32; o <<= 1) {
      const uint32_t ta = __shfl_up_sync(kFull, a, o), tb = __shfl_up_sync(kFull, b, o);
      if (lane >= o) {
        a += ta;
        b += tb;
      }
    }
    if (in) chunk_cnt[t.chunk0 + c0 + lane] = make_uint2(baseL + a - v.x, baseE + b - v.y);
    baseL += __shfl_sync(kFull, a, 31);
    baseE += __shfl_sync(kFull, b, 31);
  }
  if (lane == 0) {
    t.nL = baseL;
    t.nE = baseE;
  }
}

// The chunk's prefix counts of "below" and "equal" at the thread's first
// position (thread t of the CTA owns positions 4t .. 4t+3) and the classes of
// its positions.
__device__ __forceinline__ void chunk_prefix(const int4& ch, const float* cen, float pivot,
                                             uint2 base, uint8_t* k, uint32_t& L, uint32_t& E) {
  __shared__ uint32_t s_warp[8];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int p0 = ch.y + 4 * tid;
  uint32_t own = 0;  // below in the low 16 bits, equal in the high 16
  for (int j = 0; j < 4; ++j) {
    const int p = p0 + j;
    k[j] = 2;
    if (p < ch.z) {
      const float c = cen[p];
      k[j] = c < pivot ? 0 : (c == pivot ? 1 : 2);
    }
    own += k[j] == 0 ? 1u : (k[j] == 1 ? 0x10000u : 0u);
  }
  uint32_t incl = own;
  for (int o = 1; o < 32; o <<= 1) {
    const uint32_t v = __shfl_up_sync(kFull, incl, o);
    if (lane >= o) incl += v;
  }
  if (lane == 31) s_warp[warp] = incl;
  __syncthreads();
  uint32_t run = incl - own;
  for (int w = 0; w < warp; ++w) run += s_warp[w];
  L = base.x + (run & 0xffffu);
  E = base.y + (run >> 16);
}

// Pass 3: the prefix counts at each task's first equal / first upper box.
__global__ void __launch_bounds__(256) wide_first_kernel(const int4* __restrict__ chunks,
                                                         const uint32_t* __restrict__ nchunks,
                                                         LTask* __restrict__ T,
                                                         const float* __restrict__ cen,
                                                         const uint2* __restrict__ chunk_base) {
  if (blockIdx.x >= *nchunks) return;
  const int4 ch = chunks[blockIdx.x];
  LTask& t = T[ch.x];
  if (!t.live) return;
  const uint32_t r0 = (uint32_t)ch.y - t.start, r1 = (uint32_t)ch.z - t.start;
  const uint32_t fE = t.firstE, fG = t.firstG;
  if (!((fE >= r0 && fE < r1) || (fG >= r0 && fG < r1))) return;
  uint8_t k[4];
  uint32_t L, E;
  chunk_prefix(ch, cen, t.pivot, chunk_base[blockIdx.x], k, L, E);
  for (int j = 0; j < 4; ++j) {
    const uint32_t rel = r0 + 4 * threadIdx.x + j;
    if (rel >= r1) break;
    if (rel == fE) t.L_atE = L;
    if (rel == fG) t.LE_atG = L + E;
    if (k[j] == 0) ++L;
    else if (k[j] == 1) ++E;
  }
}

// Pass 4: boxes below the pivot go to their place (in tmp); the equal and
// upper queues' operations are written to their tapes.
__global__ void __launch_bounds__(256) wide_tape_kernel(
    const int4* __restrict__ chunks, const uint32_t* __restrict__ nchunks,
    const LTask* __restrict__ T, const uint32_t* __restrict__ idx, const float* __restrict__ cen,
    const uint2* __restrict__ chunk_base, uint32_t* __restrict__ tmp,
    uint32_t* __restrict__ tape_e, uint32_t* __restrict__ tape_g) {
  if (blockIdx.x >= *nchunks) return;
  const int4 ch = chunks[blockIdx.x];
  const LTask& t = T[ch.x];
  if (!t.live) return;
  const uint32_t s = t.start, fE = t.firstE, fG = t.firstG, n = t.n;
  uint8_t k[4];
  uint32_t L, E;
  chunk_prefix(ch, cen, t.pivot, chunk_base[blockIdx.x], k, L, E);
  for (int j = 0; j < 4; ++j) {
    const uint32_t p = (uint32_t)ch.y + 4 * threadIdx.x + j;
    if (p >= (uint32_t)ch.z) break;
    const uint32_t rel = p - s, e = idx[p], G = rel - L - E;
    const bool afterE = fE != kNone && rel > fE, afterG = fG != kNone && rel > fG;
    const uint32_t rotE = afterE ? L - t.L_atE : 0u;
    const uint32_t rotG = afterG ? (L + E) - t.LE_atG : 0u;
    // every tape position is below the task's size (a tape holds at most
    // one entry per box of the task); the checks only guard the memory
    const uint32_t te = E + rotE, tg = G + rotG;
    if (k[j] == 0) {
      if (L < n) tmp[s + L] = e;
      if (afterE && te < n) tape_e[s + te] = rotE;
      if (afterG && tg < n) tape_g[s + tg] = rotG;
      ++L;
    } else if (k[j] == 1) {
      if (te < n) tape_e[s + te] = kTerm | e;
      if (afterG && tg < n) tape_g[s + tg] = rotG;
      ++E;
    } else if (tg < n) {
      tape_g[s + tg] = kTerm | e;
    }
  }
}

// Pass 5: the tapes' copies.
__global__ void __launch_bounds__(256) wide_resolve_kernel(const int4* __restrict__ chunks,
                                                           const uint32_t* __restrict__ nchunks,
                                                           const LTask* __restrict__ T,
                                                           uint32_t* tape_e, uint32_t* tape_g) {
  if (blockIdx.x >= *nchunks) return;
  const int4 ch = chunks[blockIdx.x];
  const LTask& t = T[ch.x];
  if (!t.live) return;
  const uint32_t s = t.start, first = (uint32_t)ch.y - s + threadIdx.x, end = (uint32_t)ch.z - s;
  const uint32_t nG = t.n - t.nL - t.nE;
  const uint32_t lenE = t.nE + (t.firstE != kNone ? t.nL - t.L_atE : 0u);
  const uint32_t lenG = nG + (t.firstG != kNone ? (t.nL + t.nE) - t.LE_atG : 0u);
  resolve_tape(tape_e + s, min(lenE, end), first, blockDim.x);
  resolve_tape(tape_g + s, min(lenG, end), first, blockDim.x);
}

// Pass 6: the partitioned order back into idx: below | equal queue | upper
// queue (each queue = the last k entries of its tape).
__global__ void __launch_bounds__(256) wide_scatter_kernel(const int4* __restrict__ chunks,
                                                           const uint32_t* __restrict__ nchunks,
                                                           const LTask* __restrict__ T,
                                                           const uint32_t* __restrict__ tmp,
                                                           const uint32_t* __restrict__ tape_e,
                                                           const uint32_t* __restrict__ tape_g,
                                                           uint32_t* __restrict__ idx,
                                                           unsigned* __restrict__ status) {
  if (blockIdx.x >= *nchunks) return;
  const int4 ch = chunks[blockIdx.x];
  const LTask& t = T[ch.x];
  if (!t.live) return;
  const uint32_t s = t.start;
  const uint32_t RE = t.firstE != kNone ? t.nL - t.L_atE : 0u;
  const uint32_t RG = t.firstG != kNone ? (t.nL + t.nE) - t.LE_atG : 0u;
  for (int p = ch.y + threadIdx.x; p < ch.z; p += blockDim.x) {
    const uint32_t rel = (uint32_t)p - s;
    uint32_t v = 0;
    if (rel < t.nL) {
      v = tmp[p] | kTerm;
    } else if (rel < t.nL + t.nE) {
      const uint32_t q = RE + (rel - t.nL);
      if (q < t.n) v = tape_e[s + q];
    } else {
      const uint32_t q = RG + (rel - t.nL - t.nE);
      if (q < t.n) v = tape_g[s + q];
    }
    if (!(v & kTerm)) {  // an unresolved queue entry: an internal error, never expected
      atomicOr(status, kStatusInternal);
      v = idx[p] | kTerm;
    }
    idx[p] = v & ~kTerm;
  }
}

// After the partition: the cut, and whether it moved off the span's.
__global__ void wide_cut_kernel(LTask* __restrict__ T, const uint32_t* __restrict__ count) {
  const uint32_t k = blockIdx.x * blockDim.x + threadIdx.x;
  if (k >= *count || !T[k].live) return;
  LTask& t = T[k];
  const uint32_t ps = t.start + t.nL, pe = ps + t.nE;
  uint32_t mid = t.start + t.lcs;
  if (mid < ps || mid > pe) {
    mid = mid < ps ? ps : pe;
    if (mid == t.start) ++mid;
    else if (mid == t.start + t.n) --mid;
    t.need = 1;
  }
  t.mid = mid;
}

__global__ void __launch_bounds__(256) wide_boxes_kernel(const int4* __restrict__ chunks,
                                                         const uint32_t* __restrict__ nchunks,
                                                         LTask* __restrict__ T,
                                                         const uint32_t* __restrict__ idx,
                                                         const Box* __restrict__ tb) {
  __shared__ uint32_t s_bk[2][6];
  if (blockIdx.x >= *nchunks) return;
  const int4 ch = chunks[blockIdx.x];
  LTask& t = T[ch.x];
  if (!t.live || !t.need) return;
  const int tid = threadIdx.x;
  if (tid < 2) keys_init(s_bk[tid]);
  __syncthreads();
  for (int p = ch.y + tid; p < ch.z; p += blockDim.x)
    keys_add(s_bk[(uint32_t)p < t.mid ? 0 : 1], tb[idx[p]]);
  __syncthreads();
  if (tid < 12) {
    const int side = tid / 6, j = tid % 6;
    if (j < 3) atomicMin(&t.bk[side][j], s_bk[side][j]);
    else atomicMax(&t.bk[side][j], s_bk[side][j]);
  }
}

__global__ void wide_finish_kernel(RNode* __restrict__ nodes, const LTask* __restrict__ T,
                                   const uint32_t* __restrict__ count) {
  const uint32_t k = blockIdx.x * blockDim.x + threadIdx.x;
  if (k >= *count || !T[k].live) return;
  const LTask& t = T[k];
  RNode& N = nodes[t.node];
  N.t_mid = t.mid;
  if (t.need) {
    N.t_out[0] = keys_box(t.bk[0]);
    N.t_out[1] = keys_box(t.bk[1]);
  } else {
    N.t_out[0] = t.Lb;
    N.t_out[1] = t.Rb;
  }
}

// ---------------------------------------- nthElement across the GPU --
// A large node without a balanced span waits for these: its partitions about
// medians of three run through the passes above until the range that holds the
// cut is small enough for a CTA (kCtaMax), all waiting nodes together.  The usual
// depth has none, and the host learns of them with the depth's counts.  Builds of
// 1.3M and 12M triangles with one far away 20.3 and 233 ms in one CTA from the
// start, 8.5 and 46.9 ms so (5.4 and 36.4 without the far one); 12M at sizes and
// places over five decades 677 and 116 ms.
__global__ void nth_begin_kernel(const RNode* __restrict__ nodes,
                                 const uint32_t* __restrict__ waiting, uint32_t n,
                                 LTask* __restrict__ T) {
  const uint32_t k = blockIdx.x * blockDim.x + threadIdx.x;
  if (k >= n) return;
  LTask& t = T[k];
  const RNode& N = nodes[waiting[k]];
  t.node = waiting[k];
  t.start = N.t_start;
  t.n = N.t_n;
  t.mid = N.t_mid;
  t.axis = longest_axis(N.t_box, t.len);
  t.more = 1;
}

// Chunks of the next partitions and their pivots, or of the whole parts (whole:
// for the sides' boxes); one CTA.
__global__ void nth_chunks_kernel(const RNode* __restrict__ nodes, uint32_t n, bool whole,
                                  const float* __restrict__ cen, LTask* __restrict__ T,
                                  int4* __restrict__ chunks, uint32_t* __restrict__ nchunks) {
  __shared__ uint32_t s_total;
  if (threadIdx.x == 0) s_total = 0;
  for (uint32_t k0 = 0; k0 < n; k0 += 32) {  // warp 0: tasks and chunk offsets
    __syncthreads();
    if (threadIdx.x < 32) {
      const uint32_t k = k0 + threadIdx.x;
      uint32_t c = 0;
      if (k < n) {
        LTask& t = T[k];
        if (whole) {
          t.start = nodes[t.node].t_start;
          t.n = nodes[t.node].t_n;
          t.live = t.need = 1;
          keys_init(t.bk[0]);
          keys_init(t.bk[1]);
        } else {
          t.live = t.more && t.n > kCtaMax;
          t.firstE = t.firstG = kNone;
          t.nL = t.nE = t.L_atE = t.LE_atG = 0;
          if (t.live)
            t.pivot = median3(cen[t.start], cen[t.start + t.n / 2], cen[t.start + t.n - 1]);
        }
        if (t.live) c = (t.n + kChunk - 1) / kChunk;
      }
      uint32_t incl = c;
      for (int o = 1; o < 32; o <<= 1) {
        const uint32_t v = __shfl_up_sync(kFull, incl, o);
        if ((int)threadIdx.x >= o) incl += v;
      }
      if (k < n) T[k].chunk0 = s_total + incl - c;
      __syncwarp();
      if (threadIdx.x == 31) s_total += incl;
    }
  }
  __syncthreads();
  if (threadIdx.x == 0) *nchunks = s_total;
  for (uint32_t k = 0; k < n; ++k) {
    if (!T[k].live) continue;
    const uint32_t s = T[k].start, len = T[k].n, c0 = T[k].chunk0;
    for (uint32_t c = threadIdx.x; c * kChunk < len; c += blockDim.x)
      chunks[c0 + c] = make_int4((int)k, (int)(s + c * kChunk),
                                 (int)(s + min(len, (c + 1) * kChunk)), 0);
  }
}

// The centres in their new order.
__global__ void __launch_bounds__(256) nth_centres_kernel(const int4* __restrict__ chunks,
                                                          const uint32_t* __restrict__ nchunks,
                                                          const LTask* __restrict__ T,
                                                          const uint32_t* __restrict__ idx,
                                                          const Box* __restrict__ tb,
                                                          float* __restrict__ cen) {
  if (blockIdx.x >= *nchunks) return;
  const int4 ch = chunks[blockIdx.x];
  const int axis = T[ch.x].axis;
  for (int p = ch.y + threadIdx.x; p < ch.z; p += blockDim.x) cen[p] = centre2(tb[idx[p]], axis);
}

// The range that holds the cut, as in cta_nth.
__global__ void nth_narrow_kernel(LTask* __restrict__ T, uint32_t n) {
  const uint32_t k = blockIdx.x * blockDim.x + threadIdx.x;
  if (k >= n || !T[k].live) return;
  LTask& t = T[k];
  uint32_t lo = t.start, hi = t.start + t.n;
  const uint32_t ps = lo + t.nL, pe = ps + t.nE;
  if (t.mid < ps) hi = ps;
  else if (t.mid < pe) t.more = 0;
  else lo = pe;
  if (hi <= lo + 1) t.more = 0;
  t.start = lo;
  t.n = hi - lo;
}

// What is left of each, in a CTA.
__global__ void __launch_bounds__(1024) nth_cta_kernel(const LTask* __restrict__ T, uint32_t* idx,
                                                       float* cen, uint32_t* tmp, uint32_t* tape_e,
                                                       uint32_t* tape_g,
                                                       const Box* __restrict__ tb,
                                                       unsigned* status) {
  __shared__ CtaPart s_part;
  const LTask& t = T[blockIdx.x];
  if (!t.more) return;
  if (!cta_nth(s_part, idx, cen, tmp, tape_e, tape_g, tb, t.axis, t.start, t.start + t.n, t.mid) &&
      threadIdx.x == 0)
    atomicOr(status, kStatusInternal);
}

__global__ void nth_end_kernel(RNode* __restrict__ nodes, const uint32_t* __restrict__ waiting,
                               uint32_t n) {
  const uint32_t k = blockIdx.x * blockDim.x + threadIdx.x;
  if (k >= n) return;
  RNode& N = nodes[waiting[k]];
  insert_cut(N.cut, N.sub, N.area, N.done + 1, N.choice, N.t_mid, N.t_out[0], N.t_out[1]);
  ++N.done;
  N.waiting = 0;
}

// The root: a node, or the only subtree when it is small enough.
__global__ void tree_init_kernel(RNode* nodes, SubRoot* subs, uint32_t m,
                                 const uint32_t* __restrict__ root_keys, BuildCounts* bc) {
  BuildCounts c = {};
  if (m > kSub) {
    nodes[0].start = 0;
    nodes[0].n = m;
    nodes[0].all = keys_box(root_keys);
    nodes[0].done = nodes[0].waiting = 0;
    c.ntop = 1;
  } else {
    subs[0] = SubRoot{0, m, 0, keys_box(root_keys)};
    c.nsub = 1;
  }
  *bc = c;
}

// --------------------------------------------------- rounds and depths --
// The split each node makes this round (multiSplit: round 0 splits the
// whole range; rounds 1 and 2 the part with the largest area x count,
// the first on ties), sorted into the three size classes.  A node that waits for
// nthElement sits out the rest of the rounds and goes on from there when they
// run again.
__global__ void prepare_round_kernel(RNode* __restrict__ nodes, uint32_t lb, uint32_t le,
                                     int round, uint32_t* __restrict__ lists, uint32_t cap,
                                     uint32_t* __restrict__ counts) {
  const uint32_t x = lb + blockIdx.x * blockDim.x + threadIdx.x;
  if (x >= le) return;
  RNode& N = nodes[x];
  if (N.done != (uint32_t)round || N.waiting) return;
  const int c = round == 0 ? 0 : choose_part(N.cut, N.area, round + 1);
  if (round == 0) {
    N.cut[0] = N.start;
    N.cut[1] = N.start + N.n;
  }
  N.choice = c;
  N.t_start = N.cut[c];
  N.t_n = N.cut[c + 1] - N.cut[c];
  N.t_box = round == 0 ? N.all : N.sub[c];
  const int cat = N.t_n <= kSub ? 0 : (N.t_n <= kCtaMax ? 1 : 2);
  const uint32_t pos = atomicAdd(&counts[cat], 1u);
  lists[(size_t)cat * cap + pos] = x;
}

__global__ void finish_round_kernel(RNode* __restrict__ nodes, uint32_t lb, uint32_t le,
                                    int round) {
  const uint32_t x = lb + blockIdx.x * blockDim.x + threadIdx.x;
  if (x >= le) return;
  RNode& N = nodes[x];
  if (N.done != (uint32_t)round || N.waiting) return;
  insert_cut(N.cut, N.sub, N.area, round + 1, N.choice, N.t_mid, N.t_out[0], N.t_out[1]);
  N.done = round + 1;
}

// Children of a depth's nodes whose splits are made: single boxes are items; parts of at most kSub boxes
// become subtrees, larger ones the nodes of the next depth (numbered from le).
__global__ void make_children_kernel(RNode* __restrict__ nodes, uint32_t lb, uint32_t le,
                                     uint32_t depth, const uint32_t* __restrict__ idx,
                                     SubRoot* __restrict__ subs, BuildCounts* __restrict__ bc) {
  const uint32_t x = lb + blockIdx.x * blockDim.x + threadIdx.x;
  if (x >= le) return;
  RNode& N = nodes[x];
  if (N.done != 3) return;
  N.done = 4;
  for (int i = 0; i < 4; ++i) {
    const uint32_t s = N.cut[i], c = N.cut[i + 1] - s;
    if (c == 1) {
      N.child[i] = idx[s];
    } else if (c <= kSub) {
      const uint32_t k = atomicAdd(&bc->nsub, 1u);
      subs[k] = SubRoot{s, c, depth + 1, N.sub[i]};
      N.child[i] = kSubRef | k;
    } else {
      const uint32_t o = atomicAdd(&bc->ntop, 1u);
      atomicMax(&bc->max_n, c);
      N.child[i] = kInternal | o;
      RNode& C = nodes[o];
      C.start = s;
      C.n = c;
      C.all = N.sub[i];
      C.done = C.waiting = 0;
    }
  }
}

// Subtree sizes bottom-up and depth-first positions top-down over the nodes
// above the subtrees (a few thousand at most): one CTA, depth by depth.
__global__ void __launch_bounds__(1024) top_positions_kernel(
    const RNode* __restrict__ nodes, const uint32_t* __restrict__ lev, int depths,
    const SubRoot* __restrict__ subs, const SubTotals* __restrict__ totals, uint32_t nsub,
    Place* size, Place* place, Place* __restrict__ sub_place, BuildCounts* __restrict__ bc) {
  const int tid = threadIdx.x;
  uint32_t deepest = (uint32_t)depths;
  for (uint32_t k = tid; k < nsub; k += blockDim.x)
    deepest = max(deepest, subs[k].depth + totals[k].levels);
  atomicMax(&bc->max_depth, deepest);
  if (depths == 0) {
    if (tid == 0) {
      sub_place[0] = Place{0, 0, 0};
      bc->nodes = totals[0].nodes;
    }
    return;
  }
  auto size_of = [&](uint32_t c) {
    if ((c & kSubRef) == kSubRef) {
      const uint32_t k = c & ~kSubRef;
      return Place{totals[k].nodes, totals[k].slots, subs[k].n};
    }
    return (c & kInternal) ? size[c & ~kInternal] : Place{0, 1, 1};
  };
  for (int d = depths - 1; d >= 0; --d) {
    for (uint32_t x = lev[d] + tid; x < lev[d + 1]; x += blockDim.x) {
      Place z{1, 1, 0};
      for (int i = 0; i < 4; ++i) {
        const Place c = size_of(nodes[x].child[i]);
        z.pre += c.pre;
        z.slot += c.slot;
        z.item += c.item;
      }
      size[x] = z;
    }
    __syncthreads();
  }
  if (tid == 0) {
    place[0] = Place{0, 0, 0};
    bc->nodes = size[0].pre;
  }
  __syncthreads();
  for (int d = 0; d < depths; ++d) {
    for (uint32_t x = lev[d] + tid; x < lev[d + 1]; x += blockDim.x) {
      Place p = place[x];
      ++p.pre;
      ++p.slot;
      for (int i = 0; i < 4; ++i) {
        const uint32_t c = nodes[x].child[i];
        if ((c & kSubRef) == kSubRef) sub_place[c & ~kSubRef] = p;
        else if (c & kInternal) place[c & ~kInternal] = p;
        const Place z = size_of(c);
        p.pre += z.pre;
        p.slot += z.slot;
        p.item += z.item;
      }
    }
    __syncthreads();
  }
}

// Per node in depth-first numbering: the reference's child array, what its
// merge reads (kid: an item's leaf slot or kInternal | node) and its slot and
// the slot past its subtree; per item its triangle and slot.
__global__ void __launch_bounds__(128) sub_emit_kernel(
    const SubRoot* __restrict__ subs, const SubTotals* __restrict__ totals,
    const Place* __restrict__ sub_place, const SubNode* __restrict__ sn,
    const uint32_t* __restrict__ idx, uint4* __restrict__ child, uint4* __restrict__ kid,
    uint2* __restrict__ slots, int32_t* __restrict__ tri_index, uint32_t* __restrict__ item_slot) {
  const uint32_t start = subs[blockIdx.x].start;
  const Place r = sub_place[blockIdx.x];
  for (uint32_t x = threadIdx.x; x < totals[blockIdx.x].nodes; x += blockDim.x) {
    const SubNode N = sn[start + x];
    uint32_t slot = r.slot + N.slot + 1, item = r.item + N.item;
    uint32_t c[4], q[4];
    for (int i = 0; i < 4; ++i) {
      c[i] = q[i] = kEmpty;
      if (N.child[i] == kSubNone) continue;
      if (N.child[i] & kSubNode) {
        const SubNode Y = sn[start + (N.child[i] & ~kSubNode)];
        c[i] = q[i] = kInternal | (r.pre + Y.pre);
        slot = r.slot + Y.slot + Y.nslots;
        item = r.item + Y.item + Y.nitems;
      } else {
        c[i] = idx[start + N.child[i]];
        q[i] = item;
        tri_index[item] = (int32_t)c[i];
        item_slot[item] = slot;
        ++slot;
        ++item;
      }
    }
    const uint32_t p = r.pre + N.pre;
    child[p] = make_uint4(c[0], c[1], c[2], c[3]);
    kid[p] = make_uint4(q[0], q[1], q[2], q[3]);
    slots[p] = make_uint2(r.slot + N.slot, r.slot + N.slot + N.nslots);
  }
}

__global__ void top_emit_kernel(const RNode* __restrict__ nodes, uint32_t n,
                                const Place* __restrict__ size, const Place* __restrict__ place,
                                const SubRoot* __restrict__ subs,
                                const SubTotals* __restrict__ totals,
                                const Place* __restrict__ sub_place, uint4* __restrict__ child,
                                uint4* __restrict__ kid, uint2* __restrict__ slots,
                                int32_t* __restrict__ tri_index,
                                uint32_t* __restrict__ item_slot) {
  const uint32_t x = blockIdx.x * blockDim.x + threadIdx.x;
  if (x >= n) return;
  const Place me = place[x];
  uint32_t slot = me.slot + 1, item = me.item;
  uint32_t c[4], q[4];
  for (int i = 0; i < 4; ++i) {
    const uint32_t y = nodes[x].child[i];
    if ((y & kSubRef) == kSubRef) {
      const uint32_t k = y & ~kSubRef;
      c[i] = q[i] = kInternal | sub_place[k].pre;
      slot += totals[k].slots;
      item += subs[k].n;
    } else if (y & kInternal) {
      const uint32_t k = y & ~kInternal;
      c[i] = q[i] = kInternal | place[k].pre;
      slot += size[k].slot;
      item += size[k].item;
    } else {
      c[i] = y;
      q[i] = item;
      tri_index[item] = (int32_t)y;
      item_slot[item] = slot;
      ++slot;
      ++item;
    }
  }
  child[me.pre] = make_uint4(c[0], c[1], c[2], c[3]);
  kid[me.pre] = make_uint4(q[0], q[1], q[2], q[3]);
  slots[me.pre] = make_uint2(me.slot, me.slot + size[x].slot);
}

__global__ void iota3_kernel(int32_t* F, int64_t m) {
  const int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (i < m * 3) F[i] = (int32_t)i;
}

__global__ void remap_kernel(const int32_t* __restrict__ map, int32_t* __restrict__ I, int64_t n) {
  const int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (i < n && I[i] >= 0) I[i] = map[I[i]];
}

}  // namespace

void soup_build_search(const gwn_soup_impl& ref, gwn_soup_impl& search, cudaStream_t st) {
  const int64_t m = ref.n;
  DevBuf<int32_t> F((size_t)std::max<int64_t>(m * 3, 1), st);
  if (m) launch_kernel(iota3_kernel, blocks_for((uint64_t)m * 3), 256, 0, st, F.get(), m);
  soup_build(search, ref.td.get(), m * 3, F.get(), m, ref.order, false, st, true);
  GWN_CUDA(cudaStreamSynchronize(st));
}

void soup_remap_index(const int32_t* map, int32_t* I, int64_t n, cudaStream_t st) {
  if (n) launch_kernel(remap_kernel, blocks_for((uint64_t)n), 256, 0, st, map, I, n);
}

void soup_build_ref(gwn_soup_impl& s, const double* V, int64_t nV, const int32_t* F, int64_t nF,
                    int order, bool host_mode, cudaStream_t st) {
  GWN_REQUIRE(order >= 0 && order <= 2, "order must be 0, 1 or 2");
  GWN_REQUIRE(nF < (int64_t(1) << 30), "at most 2^30 triangles");
  s.order = order;
  s.n_input = nF;
  s.tree = GWN_TREE_REFERENCE;
  DeviceStatus status(st, host_mode);
  const size_t nF1 = (size_t)std::max<int64_t>(nF, 1);
  DevBuf<Box> tb(nF1, st);
  DevBuf<uint32_t> keep(nF1, st), pos(nF1, st), idx(nF1, st), root_keys(6, st);
  uint32_t m = 0;
  if (nF > 0) {
    launch_kernel(tri_box_kernel, blocks_for((uint64_t)nF), 256, 0, st, V, nV, F, nF, tb.get(),
                  keep.get(), status.ptr());
    exclusive_scan_u32(keep.get(), pos.get(), nF, st);
    launch_kernel(keys_init_kernel, 1, 1, 0, st, root_keys.get());
    launch_kernel(compact_kernel, std::min(blocks_for((uint64_t)nF), 4u * num_sms()), 256, 0, st,
                  (const uint32_t*)keep.get(),
                  (const uint32_t*)pos.get(), nF, (const Box*)tb.get(), idx.get(), root_keys.get());
    unsigned* last = pinned_words();
    GWN_CUDA(cudaMemcpyAsync(&last[0], pos.get() + (nF - 1), 4, cudaMemcpyDeviceToHost, st));
    GWN_CUDA(cudaMemcpyAsync(&last[1], keep.get() + (nF - 1), 4, cudaMemcpyDeviceToHost, st));
    GWN_CUDA(cudaStreamSynchronize(st));
    m = last[0] + last[1];
  }
  if (host_mode) status.check(st, "soup_build");
  s.n = m;
  if (m == 0) {
    s.nnodes = 0;
    s.ref_nodes = 0;
    for (int d = 0; d < 3; ++d) s.lo[d] = s.hi[d] = 0;
    return;
  }
  // ---- tree: depth by depth down to kSub boxes, then whole subtrees
  const uint32_t split_max = m / (kSub + 1) + 1;  // parts of more than kSub boxes in a depth
  const uint32_t wide_max = m / (kCtaMax + 1) + 1;
  const uint32_t chunk_max = m / kChunk + wide_max;
  uint32_t node_cap = m > kSub ? 8 * split_max + 64 : 1;
  DevBuf<RNode> nodes(node_cap, st);
  DevBuf<uint32_t> lists((size_t)split_max * 3, st);
  DevBuf<SubRoot> subs((size_t)m / 2 + 1, st);
  DevBuf<BuildCounts> bc(1, st);
  BuildCounts* hbc = reinterpret_cast<BuildCounts*>(pinned_words());
  static_assert(sizeof(BuildCounts) <= 64 * sizeof(unsigned), "pinned words");
  auto read_counts = [&]() {
    GWN_CUDA(cudaMemcpyAsync(hbc, bc.get(), sizeof(BuildCounts), cudaMemcpyDeviceToHost, st));
    GWN_CUDA(cudaStreamSynchronize(st));
  };
  launch_kernel(tree_init_kernel, 1, 1, 0, st, nodes.get(), subs.get(), m,
                (const uint32_t*)root_keys.get(), bc.get());
  std::vector<uint32_t> level = {0};  // depth d of the top holds nodes [level[d], level[d + 1])
  uint32_t nsub = 1;
  if (m > kSub) {
    DevBuf<uint32_t> tmp(m, st), tapeE(m, st), tapeG(m, st), nchunks(1, st), waiting;
    DevBuf<float> cen(m, st);
    DevBuf<LTask> tasks;
    DevBuf<int4> chunks;
    DevBuf<uint2> chunk_cnt;
    if (m > kCtaMax) {
      tasks.alloc(wide_max, st);
      chunks.alloc(chunk_max, st);
      chunk_cnt.alloc(chunk_max, st);
      waiting.alloc(wide_max, st);
    }
    const int4* ch = chunks.get();
    const uint32_t* nch = nchunks.get();
    LTask* T = tasks.get();
    // the passes of one partition of all live tasks (of nt; count on the device)
    auto partition = [&](uint32_t nt, const uint32_t* count) {
      launch_kernel(wide_classify_kernel, chunk_max, 256, 0, st, ch, nch, T,
                    (const float*)cen.get(), chunk_cnt.get());
      launch_kernel(wide_scan_kernel, nt, 32, 0, st, T, count, chunk_cnt.get());
      launch_kernel(wide_first_kernel, chunk_max, 256, 0, st, ch, nch, T, (const float*)cen.get(),
                    (const uint2*)chunk_cnt.get());
      launch_kernel(wide_tape_kernel, chunk_max, 256, 0, st, ch, nch, (const LTask*)T,
                    (const uint32_t*)idx.get(), (const float*)cen.get(),
                    (const uint2*)chunk_cnt.get(), tmp.get(), tapeE.get(), tapeG.get());
      launch_kernel(wide_resolve_kernel, chunk_max, 256, 0, st, ch, nch, (const LTask*)T,
                    tapeE.get(), tapeG.get());
      launch_kernel(wide_scatter_kernel, chunk_max, 256, 0, st, ch, nch, (const LTask*)T,
                    (const uint32_t*)tmp.get(), (const uint32_t*)tapeE.get(),
                    (const uint32_t*)tapeG.get(), idx.get(), status.ptr());
    };
    // the waiting nodes' splits, the host reading every kNthBatch partitions
    // whether any is still large; after kNthMax they are left to a CTA whatever
    // their size
    constexpr int kNthBatch = 4, kNthMax = 64;
    auto run_waiting = [&](uint32_t n) {
      const uint32_t* count = &bc.get()->nwaiting;
      unsigned* left = pinned_words() + 24;
      const unsigned grid = blocks_for(n, 64);
      auto make_chunks = [&](bool whole) {
        launch_kernel(nth_chunks_kernel, 1, 512, 0, st, (const RNode*)nodes.get(), n, whole,
                      (const float*)cen.get(), T, chunks.get(), nchunks.get());
      };
      launch_kernel(nth_begin_kernel, grid, 64, 0, st, (const RNode*)nodes.get(),
                    (const uint32_t*)waiting.get(), n, T);
      for (int it = 1; it <= kNthMax; ++it) {
        make_chunks(false);
        partition(n, count);
        launch_kernel(nth_centres_kernel, chunk_max, 256, 0, st, ch, nch, (const LTask*)T,
                      (const uint32_t*)idx.get(), (const Box*)tb.get(), cen.get());
        launch_kernel(nth_narrow_kernel, grid, 64, 0, st, T, n);
        if (it % kNthBatch) continue;
        GWN_CUDA(cudaMemcpyAsync(left, nchunks.get(), 4, cudaMemcpyDeviceToHost, st));
        GWN_CUDA(cudaStreamSynchronize(st));
        if (*left == 0) break;
      }
      launch_kernel(nth_cta_kernel, n, 1024, 0, st, (const LTask*)T, idx.get(), cen.get(),
                    tmp.get(), tapeE.get(), tapeG.get(), (const Box*)tb.get(), status.ptr());
      make_chunks(true);
      launch_kernel(wide_boxes_kernel, chunk_max, 256, 0, st, ch, nch, T,
                    (const uint32_t*)idx.get(), (const Box*)tb.get());
      launch_kernel(wide_finish_kernel, grid, 64, 0, st, nodes.get(), (const LTask*)T, count);
      launch_kernel(nth_end_kernel, grid, 64, 0, st, nodes.get(), (const uint32_t*)waiting.get(), n);
    };
    uint32_t lb = 0, le = 1, max_n = m;
    level.push_back(1);
    while (le > lb) {
      const uint32_t nl = le - lb, parts = std::min(nl, split_max);
      if (le + split_max > node_cap) {
        const uint32_t cap2 = 2 * node_cap + split_max;
        DevBuf<RNode> more(cap2, st);
        GWN_CUDA(cudaMemcpyAsync(more.get(), nodes.get(), (size_t)le * sizeof(RNode),
                                 cudaMemcpyDeviceToDevice, st));
        nodes = std::move(more);
        node_cap = cap2;
      }
      GWN_CUDA(cudaMemsetAsync(bc.get(), 0, offsetof(BuildCounts, ntop), st));
      for (;;) {
        for (int round = 0; round < 3; ++round) {
          uint32_t* cnt = bc.get()->lists[round];
          uint32_t *lw = lists.get(), *lc = lw + split_max, *lg = lc + split_max;
          launch_kernel(prepare_round_kernel, blocks_for(nl), 256, 0, st, nodes.get(), lb, le,
                        round, lists.get(), split_max, cnt);
          if (max_n > kCtaMax) {
            const uint32_t* c2 = cnt + 2;
            const uint32_t nt = std::min(nl, wide_max);
            launch_kernel(wide_init_kernel, 1, 512, 0, st, (const RNode*)nodes.get(),
                          (const uint32_t*)lg, c2, T, chunks.get(), nchunks.get());
            launch_kernel(wide_span_kernel, chunk_max, 256, 0, st, ch, nch, T,
                          (const uint32_t*)idx.get(), (const Box*)tb.get(), cen.get());
            launch_kernel(wide_choose_kernel, nt, 32, 0, st, T, c2, lc, cnt + 1, nodes.get(),
                          waiting.get(), &bc.get()->nwaiting);
            partition(nt, c2);
            launch_kernel(wide_cut_kernel, blocks_for(nt, 64), 64, 0, st, T, c2);
            launch_kernel(wide_boxes_kernel, chunk_max, 256, 0, st, ch, nch, T,
                          (const uint32_t*)idx.get(), (const Box*)tb.get());
            launch_kernel(wide_finish_kernel, blocks_for(nt, 64), 64, 0, st, nodes.get(),
                          (const LTask*)T, c2);
          }
          launch_kernel(part_cta_kernel, parts, 1024, 0, st, nodes.get(), (const uint32_t*)lc,
                        (const uint32_t*)(cnt + 1), idx.get(), cen.get(), tmp.get(), tapeE.get(),
                        tapeG.get(), (const Box*)tb.get(), status.ptr());
          if (round > 0)  // a whole node has more than kSub boxes
            launch_kernel(part_warp_kernel, nl, 32, 0, st, nodes.get(), (const uint32_t*)lw,
                          (const uint32_t*)cnt, idx.get(), (const Box*)tb.get(), status.ptr());
          launch_kernel(finish_round_kernel, blocks_for(nl), 256, 0, st, nodes.get(), lb, le,
                        round);
        }
        launch_kernel(make_children_kernel, blocks_for(nl), 256, 0, st, nodes.get(), lb, le,
                      (uint32_t)level.size() - 2, (const uint32_t*)idx.get(), subs.get(),
                      bc.get());
        read_counts();
        if (host_mode) status.check(st, "soup_build");
        if (hbc->nwaiting == 0) break;
        // at most three times a depth: every waiting node makes a split here
        run_waiting(hbc->nwaiting);
        GWN_CUDA(cudaMemsetAsync(bc.get(), 0, offsetof(BuildCounts, max_n), st));
      }
      lb = le;
      le = hbc->ntop;
      nsub = hbc->nsub;
      max_n = hbc->max_n;
      GWN_REQUIRE(le <= node_cap, "soup_build: tree larger than its bound");
      if (le > lb) level.push_back(le);
    }
  }
  const int top_depths = (int)level.size() - 1;
  const uint32_t ntop = level.back();
  DevBuf<SubNode> sn(m, st);
  DevBuf<uint16_t> lev((size_t)m + 1, st);  // a subtree of n > 1 boxes is at most n - 1 deep
  DevBuf<SubTotals> totals(nsub, st);
  DevBuf<Place> size(std::max<uint32_t>(ntop, 1), st), place(std::max<uint32_t>(ntop, 1), st),
      sub_place(nsub, st);
  DevBuf<uint32_t> dlevel(level.size(), st);
  dlevel.upload(level.data(), level.size(), st);
  {
    static_assert(sizeof(SubShared) <= 100 * 1024, "two CTAs per SM");
    GWN_CUDA(cudaFuncSetAttribute(subtree_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                  (int)sizeof(SubShared)));
    launch_kernel(subtree_kernel, nsub, kSubWarps * 32, sizeof(SubShared), st,
                  (const SubRoot*)subs.get(), nsub, (const uint32_t*)idx.get(),
                  (const Box*)tb.get(), sn.get(), lev.get(), totals.get(), status.ptr());
  }
  launch_kernel(top_positions_kernel, 1, 1024, 0, st, (const RNode*)nodes.get(),
                (const uint32_t*)dlevel.get(), top_depths, (const SubRoot*)subs.get(),
                (const SubTotals*)totals.get(), nsub, size.get(), place.get(), sub_place.get(),
                bc.get());
  read_counts();
  if (host_mode) status.check(st, "soup_build");
  const uint32_t nn = hbc->nodes;
  // ---- moments and the walk's slot records: a slot per node and per item
  const uint32_t total_slots = nn + m;
  s.nnodes = total_slots;
  s.ref_nodes = nn;
  s.max_depth = (int)hbc->max_depth;
  s.tri_index.alloc(m);
  s.nf.alloc(total_slots);
  // the walk reads records with 256-bit loads
  if (reinterpret_cast<uintptr_t>(s.nf.get()) % 32)
    throw Error(GWN_ERR_INTERNAL, "node records are not 32-byte aligned");
  s.nd.alloc(total_slots);
  s.tf.alloc((size_t)m * 3);
  s.td.alloc((size_t)m * 9);
  s.ref_child.alloc((size_t)nn * 4);
  {
    DevBuf<uint4> kid(nn, st);
    DevBuf<uint2> slots(nn, st);
    DevBuf<uint32_t> item_slot(m, st);
    uint4* child = reinterpret_cast<uint4*>(s.ref_child.get());
    launch_kernel(sub_emit_kernel, nsub, 128, 0, st, (const SubRoot*)subs.get(),
                  (const SubTotals*)totals.get(), (const Place*)sub_place.get(),
                  (const SubNode*)sn.get(), (const uint32_t*)idx.get(), child, kid.get(),
                  slots.get(), s.tri_index.get(), item_slot.get());
    if (ntop)
      launch_kernel(top_emit_kernel, blocks_for(ntop, 128), 128, 0, st, (const RNode*)nodes.get(),
                    ntop, (const Place*)size.get(), (const Place*)place.get(),
                    (const SubRoot*)subs.get(), (const SubTotals*)totals.get(),
                    (const Place*)sub_place.get(), child, kid.get(), slots.get(),
                    s.tri_index.get(), item_slot.get());
    DevBuf<Loc<float>> L32((size_t)total_slots, st);
    DevBuf<Loc<double>> L64((size_t)total_slots, st);
    MomentArgs ma = {};
    ma.m = m;
    ma.tri_index = s.tri_index.get();
    ma.item_slot = item_slot.get();
    ma.V = V;
    ma.nV = nV;
    ma.F = F;
    ma.order = order;
    ma.kid = kid.get();
    ma.slots = slots.get();
    ma.nsub = nsub;
    ma.subs = subs.get();
    ma.totals = totals.get();
    ma.sub_place = sub_place.get();
    ma.sn = sn.get();
    ma.lev = lev.get();
    ma.place = place.get();
    ma.level = level.data();
    ma.top_depths = top_depths;
    ma.L32 = L32.get();
    ma.L64 = L64.get();
    ma.nf = s.nf.get();
    ma.nd = s.nd.get();
    ma.tf = s.tf.get();
    ma.td = s.td.get();
    ma.bc = bc.get();
    launch_moments<float>(ma, st);
    launch_moments64(ma, st);
    double* root = reinterpret_cast<double*>(pinned_words() + 32);
    GWN_CUDA(cudaMemcpyAsync(root, L64.get() + m, 6 * sizeof(double), cudaMemcpyDeviceToHost, st));
    read_counts();
    s.moments_bounded = hbc->unbounded == 0;
    double diag2 = 0, cmax = 0;
    for (int d = 0; d < 3; ++d) {  // Loc starts with the box
      s.lo[d] = root[d];
      s.hi[d] = root[3 + d];
      const double e = s.hi[d] - s.lo[d];
      diag2 += e * e;
      cmax = fmax(cmax, fmax(fabs(s.lo[d]), fabs(s.hi[d])));
    }
    s.eps = kNearFrac * sqrt(diag2);
    s.cmax = cmax;
  }
  if (host_mode) status.check(st, "soup_build");
  s.bytes = s.nf.bytes() + s.nd.bytes() + s.tf.bytes() + s.td.bytes() + s.tri_index.bytes() +
            s.ref_child.bytes();
}

}  // namespace gwn
