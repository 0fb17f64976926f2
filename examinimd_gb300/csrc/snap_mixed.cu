// The mixed form's SNAP kernels (snap_kernel.cuh, snap_split.cuh): pair scalars and
// U_tot in FP32 pairs of 48 bits, Z, Y and the pair forces in FP32.  Compiled apart from
// snap.cu so that plain FP32 expressions may use fused multiply-adds; the FP64 drop-in
// keeps -fmad=false.
#include "snap_kernel.cuh"
#include "snap_split.cuh"

namespace emd {

using namespace snapk;

void snap_mixed_pairs(const SnapArgs& A, cudaStream_t s) { launch_pairs<float>(A, s); }

void snap_mixed_u(const SnapArgs& A, cudaStream_t s) { launch_u32(A, s); }

void snap_mixed_y(const SnapArgs& A, cudaStream_t s) {
  if (A.S.twojmax > 9) {
    if (A.ta == 32) launch_y32<8, 1, true>(A, s);
    else launch_y32<8, 1, false>(A, s);
  } else if (A.ta == 64) {
    launch_y32<5, 2, true>(A, s);
  } else if (A.ta == 32) {
    launch_y32<5, 1, true>(A, s);
  } else {
    launch_y32<5, 1, false>(A, s);
  }
}

void snap_mixed_force(const SnapArgs& A, int threads, cudaStream_t s) { launch_force<float>(A, threads, s); }

}  // namespace emd
