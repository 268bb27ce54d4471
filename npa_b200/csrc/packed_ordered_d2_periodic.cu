// Instantiates the packed perception sweep of recorded steps for dim 2, periodic boundary.
#include "packed_ordered.cuh"

namespace npa {
template int launch_packed_ordered_geom<2, true>(const Geom &, const FeatureFwdArgs &, cudaStream_t);
}  // namespace npa
