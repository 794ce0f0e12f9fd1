// Inverse transform on a thread-block cluster with a fused lift epilogue: other q < 2^62.
#include "ntt_cluster_lift.cuh"

namespace vk {

template int inv_cluster_lifted<Mod62>(cudaStream_t, const vkcu_ntt_job*, int, const vkcu_ntt_job&, int, int, const vkcu_lift&);

}  // namespace vk
