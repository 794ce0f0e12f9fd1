// Fused polynomial multiply on a thread-block cluster: odd q < 2^60.
#include "ntt_cluster.cuh"

namespace vk {

template int poly_cluster<Mod60>(cudaStream_t, const vkcu_poly_job*, int, const vkcu_poly_job&, int, int, const vkcu_lift*);

}  // namespace vk
