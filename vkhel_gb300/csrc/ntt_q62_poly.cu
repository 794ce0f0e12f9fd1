// CTA-resident fused polynomial multiplies for 2^8 <= n <= 2^14: other q < 2^62.
#include "ntt_launch.cuh"

namespace vk {

template int poly_cta<Mod62>(cudaStream_t, const vkcu_poly_job*, int, const vkcu_poly_job&, int, int, int);

}  // namespace vk
