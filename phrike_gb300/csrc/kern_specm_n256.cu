// MHD x pass over truncated spectra for pencils of 256 points.
#include "spec_launch.cuh"

namespace ps {
PS_DEFINE_SPEC_X(256, 1)
}  // namespace ps
