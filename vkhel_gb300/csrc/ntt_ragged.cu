// The single-launch ragged kernel for odd q < 2^60, and its dispatch.
#include "ntt_ragged.cuh"

namespace vk {

extern template int ragged<Mod62>(cudaStream_t, const vkcu_ragged_item*, int, int, const vkcu_poly_job*, unsigned*);

}  // namespace vk

using namespace vk;

extern "C" int vkcu_polymul_ragged(void* stream, const vkcu_ragged_item* items, int n_cluster_items, int n_items,
                                   const vkcu_poly_job* jobs, unsigned* counters, int qclass) {
  cudaStream_t st = (cudaStream_t)stream;
  if (n_items < 1 || !items || !jobs || !counters) return (int)cudaErrorInvalidValue;
  if (qclass == VKCU_Q60) return ragged<Mod60>(st, items, n_cluster_items, n_items, jobs, counters);
  if (qclass == VKCU_Q62) return ragged<Mod62>(st, items, n_cluster_items, n_items, jobs, counters);
  return (int)cudaErrorInvalidValue;
}
