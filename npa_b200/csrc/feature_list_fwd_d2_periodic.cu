// Instantiates the forward feature kernels over neighbour lists for dim 2, periodic boundary.
#include "feature_list.cuh"

namespace npa {
template int launch_feature_list_forward_geom<2, true>(const Geom &, int, const FeatureFwdArgs &, cudaStream_t);
}  // namespace npa
