// The mixed form's SNAP kernels (snap_kernel.cuh): pair scalars and U_tot
// in FP64, Z, Y and the pair forces in FP32.  Compiled apart from snap.cu so
// that the pair scalars may use fused multiply-adds; the FP64 drop-in keeps
// -fmad=false.
#include "snap_kernel.cuh"

namespace emd {

using namespace snapk;

void snap_mixed_pairs(const SnapArgs& A, cudaStream_t s) { launch_pairs<float>(A, s); }

void snap_mixed_u(const SnapArgs& A, cudaStream_t s) { launch_u<float>(A, s); }

void snap_mixed_y(const SnapArgs& A, cudaStream_t s) {
  if (A.S.twojmax <= 9) launch_y<float, 5>(A, s);
  else launch_y<float, 8>(A, s);
}

void snap_mixed_force(const SnapArgs& A, int threads, cudaStream_t s) {
  if (A.S.twojmax <= 8) launch_force<float, 9>(A, threads, s);
  else launch_force<float, 15>(A, threads, s);
}

}  // namespace emd
