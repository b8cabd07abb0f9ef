// Truncated-spectra passes for pencils of 32 points: strided passes and the
// Euler x pass (the MHD x pass is in kern_specm_n32.cu).
#include "spec_launch.cuh"

namespace ps {
PS_DEFINE_SPEC_LAUNCHERS(32)
PS_DEFINE_SPEC_X(32, 0)
}  // namespace ps
