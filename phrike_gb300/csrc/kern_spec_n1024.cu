// Truncated-spectra passes for pencils of 1024 points: strided passes and the
// Euler x pass (the MHD x pass is in kern_specm_n1024.cu).
#include "spec_launch.cuh"

namespace ps {
PS_DEFINE_SPEC_LAUNCHERS(1024)
PS_DEFINE_SPEC_X(1024, 0)
}  // namespace ps
