#pragma once
// Launchers of the cluster kernels with a fused lift epilogue.
#include "ntt_cluster.cuh"

namespace vk {

template <class M>
int inv_cluster_lifted(cudaStream_t st, const vkcu_ntt_job* jobs, int njobs, const vkcu_ntt_job& one, int logc,
                       int logs, const vkcu_lift& l) {
#define X(L, S) launch_cluster<L, S, k_ntt_inv_cluster<L, S, true>>(st, njobs, jobs, njobs, one, 0, l)
  VK_CLUSTER_SHAPES(X)
#undef X
}

template <class M>
int poly_cluster_lifted(cudaStream_t st, const vkcu_poly_job* jobs, int njobs, const vkcu_poly_job& one, int logc,
                        int logs, const vkcu_lift& l) {
#define X(L, S) launch_cluster<L, S, k_polymul_cluster<L, S, true>>(st, njobs, jobs, njobs, one, 0, l)
  if (logc == 4 && logs == 13) return X(4, Small13<M>);
  VK_CLUSTER_SHAPES(X)
#undef X
}

}  // namespace vk
