// Forward transform on a thread-block cluster: other q < 2^62.
#include "ntt_cluster.cuh"

namespace vk {

template int fwd_cluster<Mod62>(cudaStream_t, const vkcu_ntt_job*, int, const vkcu_ntt_job&, int, int);

}  // namespace vk
