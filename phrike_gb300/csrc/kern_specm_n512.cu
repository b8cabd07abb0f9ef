// MHD x pass over truncated spectra for pencils of 512 points.
#include "spec_launch.cuh"

namespace ps {
PS_DEFINE_SPEC_X(512, 1)
}  // namespace ps
