// Fused polynomial multiply on a thread-block cluster with a fused lift epilogue: odd q < 2^60.
#include "ntt_cluster_lift.cuh"

namespace vk {

template int poly_cluster_lifted<Mod60>(cudaStream_t, const vkcu_poly_job*, int, const vkcu_poly_job&, int, int, const vkcu_lift&);

}  // namespace vk
