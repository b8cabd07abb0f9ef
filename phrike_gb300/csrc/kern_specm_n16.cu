// MHD x pass over truncated spectra for pencils of 16 points.
#include "spec_launch.cuh"

namespace ps {
PS_DEFINE_SPEC_X(16, 1)
}  // namespace ps
