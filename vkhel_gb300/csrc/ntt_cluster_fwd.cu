// Forward transform on a thread-block cluster: odd q < 2^60.
#include "ntt_cluster.cuh"

namespace vk {

template int fwd_cluster<Mod60>(cudaStream_t, const vkcu_ntt_job*, int, const vkcu_ntt_job&, int, int);

}  // namespace vk
