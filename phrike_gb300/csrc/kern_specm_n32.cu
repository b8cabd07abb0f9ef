// MHD x pass over truncated spectra for pencils of 32 points.
#include "spec_launch.cuh"

namespace ps {
PS_DEFINE_SPEC_X(32, 1)
}  // namespace ps
