// MHD x pass over truncated spectra for pencils of 1024 points.
#include "spec_launch.cuh"

namespace ps {
PS_DEFINE_SPEC_X(1024, 1)
}  // namespace ps
