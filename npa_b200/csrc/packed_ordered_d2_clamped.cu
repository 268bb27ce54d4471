// Instantiates the packed perception sweep of recorded steps for dim 2, clamped boundary.
#include "packed_ordered.cuh"

namespace npa {
template int launch_packed_ordered_geom<2, false>(const Geom &, const FeatureFwdArgs &, cudaStream_t);
}  // namespace npa
