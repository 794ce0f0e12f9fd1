// Sub-blocks of transforms and products past one cluster: odd q < 2^60.
#include "ntt_cluster.cuh"

namespace vk {

template int fwd_cluster_sub<Mod60>(cudaStream_t, const vkcu_ntt_job*, int, const vkcu_ntt_job&, int, int);
template int inv_cluster_sub<Mod60>(cudaStream_t, const vkcu_ntt_job*, int, const vkcu_ntt_job&, int, int);
template int poly_cluster_sub<Mod60>(cudaStream_t, const vkcu_poly_job*, int, const vkcu_poly_job&, int, int);

}  // namespace vk
