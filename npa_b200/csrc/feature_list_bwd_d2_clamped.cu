// Instantiates the backward feature kernels over neighbour lists for dim 2, clamped boundary.
#include "feature_list.cuh"

namespace npa {
template int launch_feature_list_backward_geom<2, false, true>(const Geom &, int, const FeatureListBwdArgs &, cudaStream_t);
template int launch_feature_list_backward_geom<2, false, false>(const Geom &, int, const FeatureListBwdArgs &, cudaStream_t);
}  // namespace npa
