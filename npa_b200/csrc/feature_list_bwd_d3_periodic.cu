// Instantiates the backward feature kernels over neighbour lists for dim 3, periodic boundary.
#include "feature_list.cuh"

namespace npa {
template int launch_feature_list_backward_geom<3, true, true>(const Geom &, int, const FeatureListBwdArgs &, cudaStream_t);
template int launch_feature_list_backward_geom<3, true, false>(const Geom &, int, const FeatureListBwdArgs &, cudaStream_t);
}  // namespace npa
