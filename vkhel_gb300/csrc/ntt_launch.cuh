#pragma once
// Launchers of the CTA-resident kernels (ntt_core.cuh), templates over the
// modulus class; each translation unit instantiates one of them for one class
// so that they compile in parallel.
#include "ntt_core.cuh"

namespace vk {

template <class M>
int fwd_cta(cudaStream_t st, const vkcu_ntt_job* jobs, int njobs, const vkcu_ntt_job& one, int log_n, int sms,
            int variant) {
retry:
#define X(L, E, U) launch_cta<Shape<L, E, U, M>, k_ntt_fwd<L, E, U, M>>(st, (long)njobs, sms, jobs, njobs, one, 0)
  VK_FOR_LOGN(X)
#undef X
}

template <class M>
int inv_cta(cudaStream_t st, const vkcu_ntt_job* jobs, int njobs, const vkcu_ntt_job& one, int log_n, int sms,
            int variant) {
  const vkcu_lift none{};
retry:
#define X(L, E, U) \
  launch_cta<Shape<L, E, U, M>, k_ntt_inv<L, E, U, false, M>>(st, (long)njobs, sms, jobs, njobs, one, 0, none)
  VK_FOR_LOGN(X)
#undef X
}

template <class M>
int inv_cta_lift(cudaStream_t st, const vkcu_ntt_job* jobs, int njobs, const vkcu_ntt_job& one, int log_n, int sms,
                 const vkcu_lift& lift) {
#define X(L, E, U) \
  launch_cta<Shape<L, E, U, M>, k_ntt_inv<L, E, U, true, M>>(st, (long)njobs, sms, jobs, njobs, one, 0, lift)
  VK_FOR_LOGN_DEFAULT(X)
#undef X
}

template <class M>
int fwd_cta_sub(cudaStream_t st, const vkcu_ntt_job* jobs, int njobs, const vkcu_ntt_job& one, int sub_log, int sms) {
  return launch_cta<Shape<14, 32, 1, M>, k_ntt_fwd<14, 32, 1, M, true>>(st, (long)njobs << sub_log, sms, jobs, njobs,
                                                                        one, sub_log);
}

template <class M>
int inv_cta_sub(cudaStream_t st, const vkcu_ntt_job* jobs, int njobs, const vkcu_ntt_job& one, int sub_log, int sms) {
  const vkcu_lift none{};
  return launch_cta<Shape<14, 32, 1, M>, k_ntt_inv<14, 32, 1, false, M, true>>(st, (long)njobs << sub_log, sms, jobs,
                                                                               njobs, one, sub_log, none);
}

template <class M>
int poly_cta(cudaStream_t st, const vkcu_poly_job* jobs, int njobs, const vkcu_poly_job& one, int log_n, int sms,
             int variant) {
  const vkcu_lift none{};
retry:
#define X(L, E, U) \
  launch_cta<Shape<L, E, U, M>, k_polymul<L, E, U, false, M>>(st, (long)njobs, sms, jobs, njobs, one, none)
  VK_FOR_LOGN(X)
#undef X
}

template <class M>
int poly_cta_lift(cudaStream_t st, const vkcu_poly_job* jobs, int njobs, const vkcu_poly_job& one, int log_n, int sms,
                  int variant, const vkcu_lift& lift) {
retry:
#define X(L, E, U) \
  launch_cta<Shape<L, E, U, M>, k_polymul<L, E, U, true, M>>(st, (long)njobs, sms, jobs, njobs, one, lift)
  VK_FOR_LOGN(X)
#undef X
}

}  // namespace vk
