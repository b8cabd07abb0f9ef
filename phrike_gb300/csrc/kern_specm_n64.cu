// MHD x pass over truncated spectra for pencils of 64 points.
#include "spec_launch.cuh"

namespace ps {
PS_DEFINE_SPEC_X(64, 1)
}  // namespace ps
