// Truncated-spectra passes for pencils of 512 points: strided passes and the
// Euler x pass (the MHD x pass is in kern_specm_n512.cu).
#include "spec_launch.cuh"

namespace ps {
PS_DEFINE_SPEC_LAUNCHERS(512)
PS_DEFINE_SPEC_X(512, 0)
}  // namespace ps
