// Truncated-spectra passes for pencils of 128 points: strided passes and the
// Euler x pass (the MHD x pass is in kern_specm_n128.cu).
#include "spec_launch.cuh"

namespace ps {
PS_DEFINE_SPEC_LAUNCHERS(128)
PS_DEFINE_SPEC_X(128, 0)
}  // namespace ps
