// The single-launch ragged kernel for other q < 2^62.
#include "ntt_ragged.cuh"

namespace vk {

template int ragged<Mod62>(cudaStream_t, const vkcu_ragged_item*, int, int, const vkcu_poly_job*, unsigned*);

}  // namespace vk
