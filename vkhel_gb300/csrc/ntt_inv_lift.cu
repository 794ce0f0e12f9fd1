// CTA-resident inverse transforms with a fused epilogue (the
// reference's centred-lift element-wise ops after the last stage): odd q < 2^60.
#include "ntt_launch.cuh"

namespace vk {

template int inv_cta_lift<Mod60>(cudaStream_t, const vkcu_ntt_job*, int, const vkcu_ntt_job&, int, int, const vkcu_lift&);

}  // namespace vk
