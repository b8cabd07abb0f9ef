// MHD x pass over truncated spectra for pencils of 8 points.
#include "spec_launch.cuh"

namespace ps {
PS_DEFINE_SPEC_X(8, 1)
}  // namespace ps
