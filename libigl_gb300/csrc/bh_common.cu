// Query ordering for the Barnes-Hut walks: queries grouped by their cell of a
// Hilbert-curve grid over the tree's bounding box (one counting pass), the
// permutation handed to the walk.
#include <cuda_runtime.h>

#include "bh_common.cuh"
#include "sort.cuh"

namespace gwn {
namespace {

constexpr int64_t kMinOrdered = 8192;  // smaller batches are walked in input order

template <typename QT>
__global__ void query_keys_kernel(const QT* __restrict__ Q, int64_t n, float3 lo, float3 inv,
                                  int shift, uint32_t* __restrict__ keys,
                                  uint32_t* __restrict__ cnt, uint32_t* __restrict__ rank) {
  const int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (i >= n) return;
  const float x = (float)Q[i * 3 + 0], y = (float)Q[i * 3 + 1], z = (float)Q[i * 3 + 2];
  auto q = [](float v, float l, float s) -> uint32_t {
    float t = (v - l) * s;
    t = fminf(fmaxf(t, 0.f), 255.f);  // NaN -> 0 via fmaxf
    return (uint32_t)t;
  };
  const uint32_t k =
      hilbert3<8>(q(x, lo.x, inv.x), q(y, lo.y, inv.y), q(z, lo.z, inv.z)) >> shift;
  keys[i] = k;
  rank[i] = atomicAdd(&cnt[k], 1u);  // the order in a cell does not matter
}

}  // namespace

void order_queries(const void* Q, int q_dtype, int64_t nQ, const double lo[3], const double hi[3],
                   QueryOrder& out, cudaStream_t st) {
  out.active = false;
  if (nQ < kMinOrdered) return;
  GWN_REQUIRE(nQ < (int64_t(1) << 31), "at most 2^31-1 queries per call");
  // grow the box a little so queries just outside still spread over keys
  float3 l, inv;
  double c[3], h[3];
  for (int d = 0; d < 3; ++d) {
    c[d] = 0.5 * (lo[d] + hi[d]);
    h[d] = 0.5 * (hi[d] - lo[d]) * 1.25 + 1e-12;
  }
  l = make_float3((float)(c[0] - h[0]), (float)(c[1] - h[1]), (float)(c[2] - h[2]));
  inv = make_float3((float)(256.0 / (2 * h[0])), (float)(256.0 / (2 * h[1])),
                    (float)(256.0 / (2 * h[2])));
  // The 24-bit position among 256^3 cells from 4M queries, its leading bits with
  // four to eight cells per query below, because clearing and scanning the
  // cells' counters costs more than the queries' own passes there (100,000
  // queries with 2^24 cells: 77 us of the 95 us that the ordering took).
  int bits = 12;
  while (bits < 24 && (int64_t(4) << 20 >> (24 - bits)) < nQ) ++bits;
  DevBuf<uint32_t> keys((size_t)nQ, st), rank((size_t)nQ, st), cnt((size_t)1 << bits, st);
  cnt.zero(st);
  out.perm.alloc((size_t)nQ, st);
  const unsigned grid = (unsigned)((nQ + 255) / 256);
  if (q_dtype == GWN_F64)
    launch_kernel(query_keys_kernel<double>, grid, 256, 0, st, static_cast<const double*>(Q), nQ,
                  l, inv, 24 - bits, keys.get(), cnt.get(), rank.get());
  else
    launch_kernel(query_keys_kernel<float>, grid, 256, 0, st, static_cast<const float*>(Q), nQ,
                  l, inv, 24 - bits, keys.get(), cnt.get(), rank.get());
  bucket_place(keys.get(), rank.get(), nQ, cnt.get(), 1u << bits, out.perm.get(), st);
  out.active = true;
}

}  // namespace gwn
