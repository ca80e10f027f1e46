// Pieces shared by the Barnes-Hut paths (triangle soup and point cloud):
// Morton keys, query ordering, and the FP64 decision / guard-band rule that
// keeps the mixed-precision traversal's open/approximate decisions identical
// to the plain FP64 traversal's.
#pragma once

#include <cuda_runtime.h>

#include <cstdint>

#include "gwn_common.cuh"

namespace gwn {

// Spread the low 10 / 21 bits of x so that two zero bits separate each bit.
__host__ __device__ inline uint32_t spread10(uint32_t x) {
  x &= 0x3ffu;
  x = (x | (x << 16)) & 0x030000ffu;
  x = (x | (x << 8)) & 0x0300f00fu;
  x = (x | (x << 4)) & 0x030c30c3u;
  x = (x | (x << 2)) & 0x09249249u;
  return x;
}
__host__ __device__ inline unsigned long long spread21(unsigned long long x) {
  x &= 0x1fffffull;
  x = (x | (x << 32)) & 0x1f00000000ffffull;
  x = (x | (x << 16)) & 0x1f0000ff0000ffull;
  x = (x | (x << 8)) & 0x100f00f00f00f00full;
  x = (x | (x << 4)) & 0x10c30c30c30c30c3ull;
  x = (x | (x << 2)) & 0x1249249249249249ull;
  return x;
}

// Position of cell (x, y, z) of a grid of 2^b cells per axis along the Hilbert
// curve, as 3 b bits: Skilling's transposition of the coordinates ("Programming
// the Hilbert curve", 2004), interleaved.  Its leading bits are the position on
// the coarser grids' curves.
template <int b>
__host__ __device__ inline uint32_t hilbert3(uint32_t x, uint32_t y, uint32_t z) {
  for (uint32_t q = 1u << (b - 1); q > 1; q >>= 1) {
    const uint32_t p = q - 1;
    if (x & q) x ^= p;
    uint32_t t = (x ^ y) & p;
    if (y & q) {
      x ^= p;
    } else {
      x ^= t;
      y ^= t;
    }
    t = (x ^ z) & p;
    if (z & q) {
      x ^= p;
    } else {
      x ^= t;
      z ^= t;
    }
  }
  y ^= x;
  z ^= y;
  uint32_t t = 0;
  for (uint32_t q = 1u << (b - 1); q > 1; q >>= 1)
    if (z & q) t ^= q - 1;
  x ^= t;
  y ^= t;
  z ^= t;
  return (spread10(x) << 2) | (spread10(y) << 1) | spread10(z);
}

// Query ordering for warp coherence: position of each query's cell along a
// Hilbert curve through a box (lo, inv_extent), sorted; the traversal then
// reads queries through the returned permutation.
struct QueryOrder {
  DevBuf<int32_t> perm;
  bool active = false;
};

// Builds `out.perm` (or leaves it inactive for tiny batches).  Q is nQ x 3 of
// QT (float or double), device memory.
void order_queries(const void* Q, int q_dtype, int64_t nQ, const double lo[3],
                   const double hi[3], QueryOrder& out, cudaStream_t st);

#ifdef __CUDACC__
// Precision-exact math for the templated walks: the float versions must not
// promote to double (FP64 is a slow pipe on this GPU).
__device__ __forceinline__ float g_sqrt(float x) { return sqrtf(x); }
__device__ __forceinline__ double g_sqrt(double x) { return sqrt(x); }
__device__ __forceinline__ float g_rsqrt(float x) { return rsqrtf(x); }
__device__ __forceinline__ double g_rsqrt(double x) { return 1.0 / sqrt(x); }
__device__ __forceinline__ float g_atan2(float y, float x) { return atan2f(y, x); }
__device__ __forceinline__ double g_atan2(double y, double x) { return atan2(y, x); }
// 256-bit read-only global load (ld.global.nc.v8, sm_100 and later) of the
// 32 bytes at p, which must be 32-byte aligned.
__device__ __forceinline__ void ldg256(const void* p, float4& lo, float4& hi) {
  asm("ld.global.nc.v8.f32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
      : "=f"(lo.x), "=f"(lo.y), "=f"(lo.z), "=f"(lo.w), "=f"(hi.x), "=f"(hi.y), "=f"(hi.z),
        "=f"(hi.w)
      : "l"(p));
}
__device__ __forceinline__ float g_rcp(float x) { return __frcp_rn(x); }
__device__ __forceinline__ double g_rcp(double x) { return 1.0 / x; }

// The FP64 open test shared by both precisions: open (do not approximate)
// iff |q - c|^2 <= r2max * beta2.  Operations are pinned (no contraction) so
// that every kernel evaluates the identical expression.
__device__ __forceinline__ bool open_test64(double qx, double qy, double qz, double cx,
                                            double cy, double cz, double r2max, double beta2) {
  const double dx = __dsub_rn(qx, cx), dy = __dsub_rn(qy, cy), dz = __dsub_rn(qz, cz);
  const double r2 = __fma_rn(dz, dz, __fma_rn(dy, dy, __dmul_rn(dx, dx)));
  return r2 <= __dmul_rn(r2max, beta2);
}

// Whether an FP32 comparison of r2 against thr may disagree with the FP64
// one.  With u = 2^-24 and S = max|q| + max|c|, the FP32 error of r2 - thr
// is at most (eps + 3u) r2 + 3u thr + 3 delta^2 (1 + 1/eps), delta = 3 u S,
// eps = 1e-5; the band below doubles that bound.
__device__ __forceinline__ bool in_guard_band(float r2, float thr, float sigma) {
  return fabsf(r2 - thr) <= fmaf(2e-5f, r2 + thr, sigma);
}
__host__ __device__ inline float guard_sigma(float S) { return 2e-8f * S * S; }

// ------------------------------------------------------------ team walks --
// Small batches.  The warp-coherent walk needs about 150 dependent steps (a
// node record's latency each) per warp however few queries there are, and
// more when 32 neighbouring queries are far apart, so a batch that does not
// fill the GPU is bound by that chain.  Here T lanes share one query: an item
// is a range of pre-order slots [c, e) that its lane walks without a stack
// (an opened node moves to c + 1, any other to its link); a lane that opens
// a node with siblings after it leaves them as a new item on the team's
// stack in shared memory, from which idle lanes take the newest.  A full
// stack only means that the lane keeps the siblings itself.  Items go to
// lanes in lane order, so the terms each lane adds, and the butterfly sum of
// the lanes at the end, depend on the query alone.
// The slots visited and the terms are the warp-coherent walk's; their order
// of summation is not.
constexpr int kTeamStack = 128;  // items per warp, shared by its 32 / T teams

struct Team {
  int2* stk;          // this team's items
  unsigned mask, lt;  // lanes of the team; lanes below this one
  int cap;            // of stk
  int c = 0, e = 0, sp = 0;

  __device__ __forceinline__ Team(int T, int2* warp_stack, bool valid, int nnodes) {
    const int lane = threadIdx.x & 31;
    cap = kTeamStack * T / 32;
    stk = warp_stack + (lane / T) * cap;
    mask = (0xffffffffu >> (32 - T)) << (lane & ~(T - 1));
    lt = (1u << lane) - 1u;
    if (valid && (lane & (T - 1)) == 0) {
      c = nnodes > 1 ? 1 : 0;  // an internal root is always opened
      e = nnodes;
    }
  }
  // Idle lanes take items; false once no lane of the warp has work.
  __device__ __forceinline__ bool take() {
    __syncwarp();
    const unsigned idle = __ballot_sync(0xffffffffu, c >= e) & mask;
    const int rank = __popc(idle & lt);
    if (c >= e && rank < sp) {
      const int2 it = stk[sp - 1 - rank];
      c = it.x;
      e = it.y;
    }
    sp -= min(sp, __popc(idle));
    __syncwarp();
    return __any_sync(0xffffffffu, c < e);
  }
  // Moves past the current slot: into it (open) or to `next`, the slot after
  // its subtree.
  __device__ __forceinline__ void advance(bool act, bool open, int next) {
    const bool push = act && open && next < e;
    const unsigned m = __ballot_sync(0xffffffffu, push) & mask;
    const bool room = sp + __popc(m) <= cap;
    if (act) {
      if (push && room) {
        stk[sp + __popc(m & lt)] = make_int2(next, e);
        e = next;
      }
      c = open ? c + 1 : next;
    }
    if (room) sp += __popc(m);
  }
};

template <typename V>
__device__ __forceinline__ V team_sum(V v, int T) {
  for (int o = T >> 1; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}

#endif

}  // namespace gwn
