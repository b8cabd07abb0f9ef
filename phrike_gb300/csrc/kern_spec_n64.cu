// Truncated-spectra passes for pencils of 64 points: strided passes and the
// Euler x pass (the MHD x pass is in kern_specm_n64.cu).
#include "spec_launch.cuh"

namespace ps {
PS_DEFINE_SPEC_LAUNCHERS(64)
PS_DEFINE_SPEC_X(64, 0)
}  // namespace ps
