// CTA-resident fused polynomial multiplies with a fused
// epilogue, every shape variant of each degree: odd q < 2^60.
#include "ntt_launch.cuh"

namespace vk {

template int poly_cta_lift<Mod60>(cudaStream_t, const vkcu_poly_job*, int, const vkcu_poly_job&, int, int, int, const vkcu_lift&);

}  // namespace vk
