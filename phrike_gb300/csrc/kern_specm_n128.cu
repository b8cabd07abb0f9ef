// MHD x pass over truncated spectra for pencils of 128 points.
#include "spec_launch.cuh"

namespace ps {
PS_DEFINE_SPEC_X(128, 1)
}  // namespace ps
