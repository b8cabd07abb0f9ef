// Truncated-spectra passes for pencils of 8 points: strided passes and the
// Euler x pass (the MHD x pass is in kern_specm_n8.cu).
#include "spec_launch.cuh"

namespace ps {
PS_DEFINE_SPEC_LAUNCHERS(8)
PS_DEFINE_SPEC_X(8, 0)
}  // namespace ps
