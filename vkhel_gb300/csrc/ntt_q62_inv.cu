// CTA-resident inverse transforms for 2^8 <= n <= 2^14: other q < 2^62.
#include "ntt_launch.cuh"

namespace vk {

template int inv_cta<Mod62>(cudaStream_t, const vkcu_ntt_job*, int, const vkcu_ntt_job&, int, int, int);
template int inv_cta_sub<Mod62>(cudaStream_t, const vkcu_ntt_job*, int, const vkcu_ntt_job&, int, int);

}  // namespace vk
