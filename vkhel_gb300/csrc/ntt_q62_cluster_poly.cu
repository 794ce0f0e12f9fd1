// Fused polynomial multiply on a thread-block cluster: other q < 2^62.
#include "ntt_cluster.cuh"

namespace vk {

template int poly_cluster<Mod62>(cudaStream_t, const vkcu_poly_job*, int, const vkcu_poly_job&, int, int, const vkcu_lift*);

}  // namespace vk
