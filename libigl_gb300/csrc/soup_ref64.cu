// FP64 moments of the reference-tree soup build (soup_ref.cuh).  Apart from
// soup_ref.cu because that file is compiled without fused multiply-adds: its
// FP32 data are bit for bit the reference's, while the FP64 data have no
// counterpart there and are bound by the FP64 pipe, where a fused operation
// halves the work.
#include "soup_ref.cuh"

namespace gwn {
namespace refsoup {

void launch_moments64(const MomentArgs& A, cudaStream_t st) { launch_moments<double>(A, st); }

}  // namespace refsoup
}  // namespace gwn
