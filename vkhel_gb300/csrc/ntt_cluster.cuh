#pragma once
// Transforms and fused polynomial multiply for n = 2^15 .. 2^17 on a thread-
// block cluster of C = n / 2^14 CTAs with distributed shared memory (the
// four-step decomposition):
//
//   forward:  column pass  -- the first log2 C stages act on columns
//                             (words i, i + 2^14, ..., i + (C-1) 2^14); CTA r
//                             reads its 2^14 / C columns from global memory,
//                             runs the radix-C network in registers and writes
//                             output j of every column into CTA j's shared
//                             memory (DSMEM);
//                             (and the sub-block's first pass with them where
//                             both fit one radix-16 group: Cols below);
//             row passes   -- each CTA then runs the remaining stages on its
//                             own 2^14-word sub-block, which is the contiguous
//                             words [r 2^14, (r+1) 2^14) of the bit-reversed
//                             output; the twiddle of local stage m' and local
//                             block b is table[(C + r) m' + b];
//   inverse:  row passes on each sub-block, then the column pass gathers every
//             column from the C CTAs over DSMEM and runs the last log2 C
//             stages with n^-1 folded in, writing global memory coalesced.
//
// The sub-block is 2^14 words (n = 2^15 .. 2^17, one CTA per SM), or 2^9 ..
// 2^13 words for n = 2^12 .. 2^17 split over 2 .. 16 CTAs when there are too
// few jobs to fill the GPU otherwise (single calls, small batches, server
// micro-batches, the jobs past a batch's whole rounds: split_log and Tail in
// ntt.cu).  Past one cluster (n >= 2^18, and few jobs of 2^17) the same kernels
// run the sub-blocks that the global passes leave (SUB: 2^16 words on 4 CTAs,
// or 2^14 on 8).
//
// Cluster barriers separate the phases: before a forward column pass writes
// another CTA's shared memory (its owner has finished reading it; in the
// polymul this one is split: each CTA arrives, loads and transforms its first
// columns, and waits just before its first remote store), after it (the
// sub-blocks are complete), and before the inverse gather.  Every CTA of a
// cluster walks the same job sequence, and a final barrier keeps each CTA's
// shared memory alive until the last remote read.
#include <cooperative_groups.h>

#include "ntt_core.cuh"

namespace cg = cooperative_groups;

namespace vk {

template <class M>
using SubShape = Shape<14, 32, 1, M>;  // the large-n sub-block

// The column pass: the first LOGC stages, which mix the sub-blocks, and with
// them the sub-block's own first pass (FIRSTK stages) where both fit one
// radix-16 group -- 2^15 and 2^16 on 2^14-word sub-blocks, 2^16 on 8 CTAs --
// which saves that pass over shared memory and its barrier (64 products of 2^16
// words 161.9 -> 153.7 us, 150 inverse transforms of 2^15 with a lift
// 75.9 -> 71.8 us, the ragged batch of 512 instances 3.22 -> 3.06 ms).
// A group is W = 2^KK words TM apart; word j belongs to CTA j >> LJ.
template <int LOGC, class S>
struct Cols {
  static constexpr int C = 1 << LOGC, SUB = S::N;
  static constexpr bool MERGED = S::R == 4 && LOGC + S::FIRSTK <= 4;
  static constexpr int LJ = MERGED ? S::FIRSTK : 0;
  static constexpr int KK = LOGC + LJ, W = 1 << KK;
  static constexpr int TM = SUB >> LJ;
  static constexpr int COLS = TM >> LOGC;   // groups per CTA
  static constexpr int PER = COLS >= S::T ? COLS / S::T : 1;  // groups per thread
  static constexpr int H = PER >= 2 ? PER / 2 : 1;            // of them in flight at once
  static constexpr int N16 = C * SUB / 16;  // groups of the last four stages
  static_assert(COLS >= S::T ? PER * W == S::E : COLS % 32 == 0, "whole warps move the columns");
  static_assert(W <= S::T, "a thread per slice prefetches");
  // with fewer columns than threads (radix-4 shapes) the first warps have one each
  __device__ __forceinline__ static bool active() { return COLS >= S::T || (int)threadIdx.x < COLS; }
  __device__ __forceinline__ static int col(int rank, int k) { return rank * COLS + (int)threadIdx.x + k * S::T; }
  // word j of column c: its CTA (static) and its place there
  static constexpr int cta(int j) { return j >> LJ; }
  __device__ __forceinline__ static int local(int c, int j) { return pad(c + (j & ((1 << LJ) - 1)) * TM); }
};

// The cluster barrier split in two: arrive (release: this thread's accesses
// to shared memory so far, its own CTA's and remote, are ordered before what
// other CTAs do after their wait) and wait (acquire).  Every thread of the
// cluster executes each exactly once per barrier phase.
__device__ __forceinline__ void cluster_arrive() { asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory"); }
__device__ __forceinline__ void cluster_wait() { asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory"); }

// Forward column pass: global stages 0 .. KK-1 (exact first-stage rule),
// outputs scattered to the owning CTAs' shared memory, forward-lazy.  A
// thread's PER columns go in two rounds of H = PER / 2 (16 words in flight:
// all 32 at once would spill).  SPLIT: the caller has arrived on the cluster
// barrier that frees the other CTAs' shared memory, and the first round's
// loads and butterflies run before the wait, which comes just before the
// first remote store (the fused polymul: 1-2.4 % faster; the forward
// transform alone was 0.8 % slower this way and synchronizes before).
// rbase: the cluster rank of this transform's CTA 0 (a larger cluster can
// hold several transforms of C CTAs each).  SUB: a sub-block of a larger
// transform after its global passes, twiddle multiplier `base`; its words are
// forward-lazy already.
template <int LOGC, class S, bool SPLIT, bool SUB = false>
__device__ __forceinline__ void col_fwd(const u64* __restrict__ in, u64* sm, const cg::cluster_group& cl, int rank,
                                        const Tw& t, int rbase = 0, u32 base = 1u) {
  using K = Cols<LOGC, S>;
  auto load = [&](u64(&v)[K::H * K::W], int k0) {
#pragma unroll
    for (int k = 0; k < K::H; k++)
#pragma unroll
      for (int j = 0; j < K::W; j++) v[k * K::W + j] = ld_stream(in + K::col(rank, k0 + k) + (size_t)j * K::TM);
    static_for<0, K::H>([&](auto kc) {
      constexpr int k = decltype(kc)::value;
      ct_first_group<typename S::M, K::KK, k * K::W, !SUB>(v, RowTw{t.fwd, base}, t);
    });
  };
  auto scatter = [&](const u64(&v)[K::H * K::W], int k0) {
#pragma unroll
    for (int j = 0; j < K::W; j++) {
      u64* rem = cl.map_shared_rank(sm, rbase + K::cta(j));
#pragma unroll
      for (int k = 0; k < K::H; k++) rem[K::local(K::col(rank, k0 + k), j)] = v[k * K::W + j];
    }
  };
  if constexpr (K::COLS >= S::T) {
#pragma unroll 1
    for (int k0 = 0; k0 < K::PER; k0 += K::H) {
      u64 v[K::H * K::W];
      load(v, k0);
      if (SPLIT && k0 == 0) cluster_wait();
      scatter(v, k0);
    }
  } else {
    u64 v[K::H * K::W];
    if (K::active()) load(v, 0);
    if (SPLIT) cluster_wait();  // every thread's
    if (K::active()) scatter(v, 0);
  }
}

// Inverse column pass: gather, global stages KK-1 .. 0 with n^-1 folded in,
// canonical words to global memory; two rounds of H columns as above.  SUB:
// no fold, words below one unit.
template <int LOGC, class S, bool SUB, class Epi>
__device__ __forceinline__ void col_inv(u64* __restrict__ out, u64* sm, const cg::cluster_group& cl, int rank,
                                        const Tw& t, const Epi& epi, int rbase = 0, u32 base = 1u) {
  using K = Cols<LOGC, S>;
  if (!K::active()) return;
#pragma unroll 1
  for (int k0 = 0; k0 < K::PER; k0 += K::H) {
    u64 v[K::H * K::W];
#pragma unroll
    for (int j = 0; j < K::W; j++) {
      const u64* rem = cl.map_shared_rank(sm, rbase + K::cta(j));
#pragma unroll
      for (int k = 0; k < K::H; k++) v[k * K::W + j] = rem[K::local(K::col(rank, k0 + k), j)];
    }
    static_for<0, K::H>([&](auto kc) {
      constexpr int k = decltype(kc)::value;
      gs_group<typename S::M, K::KK, k * K::W, false, !SUB>(v, RowTw{t.inv, base}, t);
    });
    epi.apply(v);
#pragma unroll
    for (int k = 0; k < K::H; k++)
#pragma unroll
      for (int j = 0; j < K::W; j++) out[K::col(rank, k0 + k) + (size_t)j * K::TM] = v[k * K::W + j];
  }
}

// The passes of a sub-block between the column pass and the last radix-16
// pass, with the cluster barriers: forward after col_fwd, inverse before
// col_inv.
template <int LOGC, class S>
__device__ __forceinline__ void sub_fwd(u64* sm, const cg::cluster_group& cl, const Tw& t, u32 tw_mult) {
  cl.sync();
  if constexpr (!Cols<LOGC, S>::MERGED) fwd_first_smem<S>(sm, t, tw_mult);
}

template <int LOGC, class S, class L>
__device__ __forceinline__ void sub_inv(u64* sm, const cg::cluster_group& cl, const Tw& t, u32 tw_mult,
                                        const L& last_inv) {
  inv_passes<S>(sm, t, tw_mult, last_inv);
  if constexpr (!Cols<LOGC, S>::MERGED) {
    __syncthreads();
    inv_last_smem<S>(sm, t, tw_mult);
  }
  cl.sync();
}

template <int LOGC, class S, bool LIFT, bool SUB = false>
__device__ __forceinline__ void col_inv_out(u64* __restrict__ out, u64* sm, const cg::cluster_group& cl, int rank,
                                            const Tw& t, const vkcu_lift* lift, int rbase = 0, u32 base = 1u) {
  if constexpr (LIFT)
    col_inv<LOGC, S, SUB>(out, sm, cl, rank, t, LiftFold(lift, t.q), rbase, base);
  else
    col_inv<LOGC, S, SUB>(out, sm, cl, rank, t, NoLift{}, rbase, base);
}

// Which cluster job (and, with SUB, which of its 2^sub_log sub-blocks) a
// work item is: twiddle multiplier base, first word off, and the roots of the
// last four stages for this CTA.
template <int LOGC, class S, bool SUB>
struct ClusterItem {
  using K = Cols<LOGC, S>;
  int job, sub, sub_log;
  u32 base;
  size_t off;
  __device__ __forceinline__ ClusterItem(int w, int sub_log_)
      : job(SUB ? w >> sub_log_ : w),
        sub(SUB ? w & ((1 << sub_log_) - 1) : 0),
        sub_log(SUB ? sub_log_ : 0),
        base(SUB ? (1u << sub_log_) + (u32)sub : 1u),
        off(SUB ? (size_t)sub * (K::C * K::SUB) : 0) {}
  __device__ __forceinline__ u32 tw_mult(int rank) const { return base * K::C + (u32)rank; }
  using Last = LastTable<SUB ? 0 : K::N16>;
  __device__ __forceinline__ Last last(const ulonglong2* table, int rank) const {
    return Last(table, sub * K::N16 + rank * (S::N / 16), (u32)K::N16 << sub_log);
  }
};

// CTAs per SM the register budget is sized for: two of 256 threads (128
// registers), so that an SM holds a CTA of each of two clusters (19 products
// of 2^15 words on 8 CTAs each 54 -> 42 us, 19 of 2^16 100 -> 78 us); the
// smaller shapes are single calls first of all, and 128 registers cost those
// 4-10 % (one product of 2^13 19.7 -> 20.5 us).
template <class S>
constexpr int cluster_blocks() {
  return S::T == 256 ? 2 : 1;
}

template <int LOGC, class S, bool SUB = false>
__global__ void __launch_bounds__(S::T, cluster_blocks<S>())
    k_ntt_fwd_cluster(const vkcu_ntt_job* __restrict__ jobs, int njobs, vkcu_ntt_job one, int sub_log) {
  using K = Cols<LOGC, S>;
  extern __shared__ u64 sm[];
  cg::cluster_group cl = cg::this_cluster();
  const int rank = (int)cl.block_rank();
  const int ncl = (int)gridDim.x / K::C, cid = (int)blockIdx.x / K::C;
  const int items = SUB ? njobs << sub_log : njobs;
#pragma unroll 1
  for (int w = cid; w < items; w += ncl) {
    const ClusterItem<LOGC, S, SUB> it(w, sub_log);
    const vkcu_ntt_job job = fetch_job(jobs, one, it.job);
    const Tw t = load_tw(job.tw);
    const u32 tw_mult = it.tw_mult(rank);
    const auto last = it.last(t.fwd, rank);
    u64* out = reinterpret_cast<u64*>(job.out) + it.off;
    const u64* in = SUB ? out : reinterpret_cast<const u64*>(job.in);
    cl.sync();
    col_fwd<LOGC, S, false, SUB>(in, sm, cl, rank, t, 0, it.base);
    sub_fwd<LOGC, S>(sm, cl, t, tw_mult);
    out += (size_t)rank * K::SUB;
    fwd_passes<S>(sm, t, tw_mult, last, [&](int g, u64(&v)[S::W]) {
      const typename S::M::Out to(t);
#pragma unroll
      for (int j = 0; j < S::W; j++) v[j] = to.canon(v[j]);
      if constexpr (staged_stores<S>())
        store_group_staged(v, out, sm, g);
      else
        store_group(v, out + S::W * g);
    });
  }
  cl.sync();
}

template <int LOGC, class S, bool LIFT, bool SUB = false>
__global__ void __launch_bounds__(S::T, cluster_blocks<S>())
    k_ntt_inv_cluster(const vkcu_ntt_job* __restrict__ jobs, int njobs, vkcu_ntt_job one, int sub_log,
                      const __grid_constant__ vkcu_lift lift) {
  using K = Cols<LOGC, S>;
  extern __shared__ u64 sm[];
  cg::cluster_group cl = cg::this_cluster();
  const int rank = (int)cl.block_rank();
  const int ncl = (int)gridDim.x / K::C, cid = (int)blockIdx.x / K::C;
  const int items = SUB ? njobs << sub_log : njobs;
#pragma unroll 1
  for (int w = cid; w < items; w += ncl) {
    const ClusterItem<LOGC, S, SUB> it(w, sub_log);
    const vkcu_ntt_job job = fetch_job(jobs, one, it.job);
    const Tw t = load_tw(job.tw);
    const auto last = it.last(t.inv, rank);
    const u64* in = reinterpret_cast<const u64*>(job.in) + it.off + (size_t)rank * K::SUB;
    cl.sync();
#pragma unroll 1
    for (int i = 0; i < S::GROUPS; i++) {
      const int g = S::group(i);
      u64 v[S::W];
      if constexpr (staged_loads<S>())
        load_group_staged<S>(v, in, sm, g, [] {});
      else
        load_group(v, in + S::W * g);
      gs_group<typename S::M, S::R, 0, true, false>(v, last.template at<4 - S::R>(g), t);
#pragma unroll
      for (int j = 0; j < S::W; j++) sm[pad(S::W * g) + j] = v[j];
    }
    sub_inv<LOGC, S>(sm, cl, t, it.tw_mult(rank), last);
    col_inv_out<LOGC, S, LIFT, SUB>(reinterpret_cast<u64*>(job.out) + it.off, sm, cl, rank, t, &lift, 0, it.base);
  }
  cl.sync();
}

// SUB: the sub-block products of a larger polymul: the global passes have left
// their words of a in c and of b in scratch (b_ntt: NTT(b) whole in b).
template <int LOGC, class S, bool LIFT, bool SUB = false>
__global__ void __launch_bounds__(S::T, cluster_blocks<S>())
    k_polymul_cluster(const vkcu_poly_job* __restrict__ jobs, int njobs, vkcu_poly_job one, int sub_log,
                      const __grid_constant__ vkcu_lift lift) {
  using K = Cols<LOGC, S>;
  extern __shared__ u64 sm[];
  cg::cluster_group cl = cg::this_cluster();
  const int rank = (int)cl.block_rank();
  const int ncl = (int)gridDim.x / K::C, cid = (int)blockIdx.x / K::C;
  const int items = SUB ? njobs << sub_log : njobs;
  constexpr unsigned kSlice = (unsigned)(K::COLS * 8);
  constexpr bool FLAGS = LIFT || SUB;  // the instantiations that read the job's flags
#pragma unroll 1
  for (int w = cid; w < items; w += ncl) {
    const ClusterItem<LOGC, S, SUB> it(w, sub_log);
    const vkcu_poly_job job = fetch_job(jobs, one, it.job);
    const Tw t = load_tw_product<typename S::M>(job.tw);
    // b holds NTT(b): phase 0 is skipped
    const bool b_ntt = FLAGS && (job.flags & VKCU_JOB_B_NTT);
    const u32 tw_mult = it.tw_mult(rank);
    const u64* a = (SUB ? reinterpret_cast<const u64*>(job.c) : reinterpret_cast<const u64*>(job.a)) + it.off;
    const u64* b = (SUB && !b_ntt ? reinterpret_cast<const u64*>(job.scratch) : reinterpret_cast<const u64*>(job.b)) +
                   it.off;
    u64* scratch = reinterpret_cast<u64*>(job.scratch) + it.off + (size_t)rank * K::SUB;
    const auto last = it.last(t.fwd, rank), last_inv = it.last(t.inv, rank);
    if ((int)threadIdx.x < K::W)  // this CTA's column slices of a, for phase 1
      prefetch_l2(a + (size_t)threadIdx.x * K::TM + rank * K::COLS, kSlice);
#pragma unroll 1
    for (int ph = b_ntt ? 1 : 0; ph < 2; ph++) {
      cluster_arrive();  // done with every shared memory the column pass writes (col_fwd waits)
      col_fwd<LOGC, S, true, SUB>(ph ? a : b, sm, cl, rank, t, 0, it.base);
      sub_fwd<LOGC, S>(sm, cl, t, tw_mult);
      fwd_passes<S>(sm, t, tw_mult, last, [&](int g, u64(&v)[S::W]) {
        using M = typename S::M;
        if (ph == 0) {
          const typename M::Out to(t);
#pragma unroll
          for (int j = 0; j < S::W; j++) v[j] = to.park(v[j]);
          park_group(v, scratch, g, S::N / S::W);
        } else {
          u64 bh[S::W];
          if (b_ntt) {
            load_group(bh, b + (size_t)rank * K::SUB + S::W * g);
            reduce_operands(bh, t);
          } else {
            unpark_group(bh, scratch, g, S::N / S::W);
          }
          const typename M::Product product(t);
#pragma unroll
          for (int j = 0; j < S::W; j++) v[j] = product(v[j], bh[j]);
          // the sub-block's first inverse pass (stages HEAD + 3 .. HEAD) on the same words
          gs_group<M, S::R, 0, M::EXACT_AFTER_PRODUCT, false>(v, last_inv.template at<4 - S::R>(g), t);
#pragma unroll
          for (int j = 0; j < S::W; j++) sm[pad(S::W * g) + j] = v[j];
        }
      });
    }
    if (!SUB && w + ncl < items && (int)threadIdx.x < K::W) {
      // the next job's b: its column slices, or (NTT(b) given) this CTA's sub-block
      const vkcu_poly_job nx = fetch_job(jobs, one, w + ncl);
      const size_t off = (LIFT && (nx.flags & VKCU_JOB_B_NTT)) ? (size_t)rank * K::SUB + (size_t)threadIdx.x * K::COLS
                                                     : (size_t)threadIdx.x * K::TM + rank * K::COLS;
      prefetch_l2(reinterpret_cast<const u64*>(nx.b) + off, kSlice);
    }
    sub_inv<LOGC, S>(sm, cl, t, tw_mult, last_inv);
    col_inv_out<LOGC, S, LIFT, SUB>(reinterpret_cast<u64*>(job.c) + it.off, sm, cl, rank, t, &lift, 0, it.base);
  }
  cl.sync();
}

// The kernel is a template argument so that each kernel gets its own
// one-time attribute set-up (forward and inverse kernels share a signature).
// The clusters are spread over SMs: a cluster of small CTAs would otherwise
// be packed onto few SMs.
template <int LOGC, class S, auto kern, class... Args>
static int launch_cluster(cudaStream_t st, int njobs, Args... args) {
  constexpr int C = 1 << LOGC;
  static KernelSetup setup;  // resident clusters per device
  cudaLaunchConfig_t cfg = {};
  cudaLaunchAttribute attr[2];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = C;
  attr[0].val.clusterDim.y = 1;
  attr[0].val.clusterDim.z = 1;
  attr[1].id = cudaLaunchAttributeClusterSchedulingPolicyPreference;
  attr[1].val.clusterSchedulingPolicyPreference = cudaClusterSchedulingPolicySpread;
  cfg.blockDim = dim3(S::T);
  cfg.dynamicSmemBytes = S::SMEM_BYTES;
  cfg.stream = st;
  cfg.attrs = attr;
  cfg.numAttrs = 2;
  cfg.gridDim = dim3(C);
  const int dev = current_device();
  const bool cached = dev >= 0 && dev < 32;
  int max_clusters = cached ? setup.per_dev[dev].load(std::memory_order_acquire) : 0;
  if (max_clusters < 0) return (int)cudaErrorInvalidConfiguration;  // no such cluster fits this GPU
  cudaError_t e = cudaSuccess;
  if (max_clusters < 1) {
    e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, S::SMEM_BYTES);
    if (e == cudaSuccess && C > 8) e = cudaFuncSetAttribute(kern, cudaFuncAttributeNonPortableClusterSizeAllowed, 1);
    if (e == cudaSuccess) e = cudaOccupancyMaxActiveClusters(&max_clusters, kern, &cfg);
    if (e != cudaSuccess) return (int)e;
    if (max_clusters < 1) {
      if (cached) setup.per_dev[dev].store(-1, std::memory_order_release);
      return (int)cudaErrorInvalidConfiguration;
    }
    if (cached) setup.per_dev[dev].store(max_clusters, std::memory_order_release);
  }
  const int nclusters = njobs < max_clusters ? njobs : max_clusters;
  cfg.gridDim = dim3(nclusters * C);
  e = cudaLaunchKernelEx(&cfg, kern, args...);
  vkcu_count_launches(1);
  return (int)e;
}

// Sub-blocks of 2^9 .. 2^13 words for n = 2^12 .. 2^16 on 8 CTAs: 4 words per
// thread and radix-4 passes to 2^10, 16 words per thread above (32 at 2^13, so
// that 256 threads fit the register file).
template <class M>
using Small9 = Shape<9, 4, 1, M, false, 2>;
template <class M>
using Small10 = Shape<10, 4, 1, M, false, 2>;
template <class M>
using Small11 = Shape<11, 16, 1, M>;
template <class M>
using Small12 = Shape<12, 16, 1, M>;
template <class M>
using Small13 = Shape<13, 32, 1, M>;

// logc: cluster size 2^logc; logs: sub-block size 2^logs: 14, or, for fewer
// jobs than SMs, 9 .. 13 with logc = 3, 12 / 13 with logc = 1 or 2 (n = 2^13,
// 2^14), 10 .. 12 with logc = 4 (n = 2^14 .. 2^16 on 16 CTAs, a cluster size
// the GPU allows on request).  Products have 13 with logc = 4 too, for one of
// 2^17 without the scratch that the global passes want.
#define VK_CLUSTER_SHAPES(X)                                 \
  switch (logc * 32 + logs) {                                \
    case 1 * 32 + 14: return X(1, SubShape<M>);              \
    case 2 * 32 + 14: return X(2, SubShape<M>);              \
    case 3 * 32 + 14: return X(3, SubShape<M>);              \
    case 3 * 32 + 9: return X(3, Small9<M>);                 \
    case 1 * 32 + 12: return X(1, Small12<M>);               \
    case 1 * 32 + 13: return X(1, Small13<M>);               \
    case 2 * 32 + 12: return X(2, Small12<M>);               \
    case 3 * 32 + 10: return X(3, Small10<M>);               \
    case 3 * 32 + 11: return X(3, Small11<M>);               \
    case 3 * 32 + 12: return X(3, Small12<M>);               \
    case 3 * 32 + 13: return X(3, Small13<M>);               \
    case 4 * 32 + 10: return X(4, Small10<M>);               \
    case 4 * 32 + 11: return X(4, Small11<M>);               \
    case 4 * 32 + 12: return X(4, Small12<M>);               \
    default: return (int)cudaErrorInvalidValue;              \
  }

// The launchers (ntt_core.cuh declares them) are instantiated per modulus
// class, the lifted inverse and polymul kernels in their own translation
// units, so that the cluster kernels compile in parallel.
template <class M>
int inv_cluster_lifted(cudaStream_t st, const vkcu_ntt_job* jobs, int njobs, const vkcu_ntt_job& one, int logc,
                       int logs, const vkcu_lift& lift);
template <class M>
int poly_cluster_lifted(cudaStream_t st, const vkcu_poly_job* jobs, int njobs, const vkcu_poly_job& one, int logc,
                        int logs, const vkcu_lift& lift);

template <class M>
int fwd_cluster(cudaStream_t st, const vkcu_ntt_job* jobs, int njobs, const vkcu_ntt_job& one, int logc, int logs) {
#define X(L, S) launch_cluster<L, S, k_ntt_fwd_cluster<L, S>>(st, njobs, jobs, njobs, one, 0)
  VK_CLUSTER_SHAPES(X)
#undef X
}

template <class M>
int inv_cluster(cudaStream_t st, const vkcu_ntt_job* jobs, int njobs, const vkcu_ntt_job& one, int logc, int logs,
                const vkcu_lift* lift) {
  if (lift) return inv_cluster_lifted<M>(st, jobs, njobs, one, logc, logs, *lift);
  const vkcu_lift l{};
#define X(L, S) launch_cluster<L, S, k_ntt_inv_cluster<L, S, false>>(st, njobs, jobs, njobs, one, 0, l)
  VK_CLUSTER_SHAPES(X)
#undef X
}

template <class M>
int poly_cluster(cudaStream_t st, const vkcu_poly_job* jobs, int njobs, const vkcu_poly_job& one, int logc, int logs,
                 const vkcu_lift* lift) {
  if (lift) return poly_cluster_lifted<M>(st, jobs, njobs, one, logc, logs, *lift);
  const vkcu_lift l{};
#define X(L, S) launch_cluster<L, S, k_polymul_cluster<L, S, false>>(st, njobs, jobs, njobs, one, 0, l)
  if (logc == 4 && logs == 13) return X(4, Small13<M>);
  VK_CLUSTER_SHAPES(X)
#undef X
}

// (log_n - sub_log is 16 or 14.)
template <class M>
int fwd_cluster_sub(cudaStream_t st, const vkcu_ntt_job* jobs, int njobs, const vkcu_ntt_job& one, int log_n,
                    int sub_log) {
#define X(L, S) launch_cluster<L, S, k_ntt_fwd_cluster<L, S, true>>(st, njobs << sub_log, jobs, njobs, one, sub_log)
  return log_n - sub_log == 16 ? X(2, SubShape<M>) : X(3, Small11<M>);
#undef X
}

template <class M>
int inv_cluster_sub(cudaStream_t st, const vkcu_ntt_job* jobs, int njobs, const vkcu_ntt_job& one, int log_n,
                    int sub_log) {
  const vkcu_lift l{};
#define X(L, S) \
  launch_cluster<L, S, k_ntt_inv_cluster<L, S, false, true>>(st, njobs << sub_log, jobs, njobs, one, sub_log, l)
  return log_n - sub_log == 16 ? X(2, SubShape<M>) : X(3, Small11<M>);
#undef X
}

template <class M>
int poly_cluster_sub(cudaStream_t st, const vkcu_poly_job* jobs, int njobs, const vkcu_poly_job& one, int log_n,
                     int sub_log) {
  const vkcu_lift l{};
#define X(L, S) \
  launch_cluster<L, S, k_polymul_cluster<L, S, false, true>>(st, njobs << sub_log, jobs, njobs, one, sub_log, l)
  return log_n - sub_log == 16 ? X(2, SubShape<M>) : X(3, Small11<M>);
#undef X
}

}  // namespace vk
