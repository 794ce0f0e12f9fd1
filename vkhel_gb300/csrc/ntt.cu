// Transform dispatch and the kernels outside the CTA-resident families:
// simple one-stage-per-barrier kernels (n < 256, unaligned operands), the
// global-memory passes of n >= 2^18, and the pointwise step of a composed
// polynomial multiply.  Every launcher takes the modulus class of its jobs
// (`qclass`, VKCU_Q60 .. VKCU_Q63).  The CTA-resident kernels are in
// ntt_core.cuh with one launcher per family (ntt_fwd.cu, ntt_inv.cu,
// ntt_poly.cu).
#include "elem_ops.cuh"
#include "ntt_core.cuh"

namespace vk {

// ---------------------------------------------------------------------------
// Simple kernels: one CTA per job, whole vector in shared memory, one
// radix-2 stage per __syncthreads.  Used for n < 256, for n <= 2^14 when a
// pointer is not 32-byte aligned, and as an independent cross-check.  Latency
// bounds them: a few loads and log2 n dependent butterflies.  So the products
// are plain C, whose four multiplies run side by side where the throughput
// kernels' chain of fused multiply-adds waits on itself; Mod62 serves q < 2^60
// too, as its outputs need no constants beyond q; and below 2^8 a root's place
// is its index.  With the throughput kernels' forms 8000 forward transforms of
// 2^7 took 16.4 us and 100 products 16.4, now 14.4 and 14.4.
__device__ __forceinline__ u64 shoup_lazy_short(u64 x, u64 w, u64 wp, u64 q) { return x * w - mulhi(x, wp) * q; }

struct Simple62 : Mod62 {
  template <bool REDUCE>
  __device__ __forceinline__ static void ct(u64& x, u64& y, u64 w, u64 wp, const Tw& t) {
    const u64 xr = csub(x, t.q2), wy = shoup_lazy_short(y, w, wp, t.q);
    x = xr + wy;
    y = xr - wy + t.q2;
  }
  __device__ __forceinline__ static u64 mul(u64 d, u64 w, u64 wp, const Tw& t) {
    return shoup_lazy_short(d, w, wp, t.q);
  }
};

struct Simple63 : Mod63 {
  template <bool REDUCE>
  __device__ __forceinline__ static void ct(u64& x, u64& y, u64 w, u64 wp, const Tw& t) {
    const u64 xr = csub(x, t.q), wy = csub(shoup_lazy_short(y, w, wp, t.q), t.q);
    x = xr + wy;
    y = xr - wy + t.q;
  }
  __device__ __forceinline__ static u64 mul(u64 d, u64 w, u64 wp, const Tw& t) {
    return shoup_lazy_short(d, w, wp, t.q);
  }
};

// ROWS: n >= 2^8, whose last roots stand in rows (vkcu_tw_slot).
template <class M, bool ROWS>
__global__ void k_ntt_fwd_simple(const vkcu_ntt_job* __restrict__ jobs, int njobs, vkcu_ntt_job one,
                                 int log_n) {
  extern __shared__ u64 sm[];
  const int n = 1 << log_n;
  for (int w = blockIdx.x; w < njobs; w += gridDim.x) {
    const vkcu_ntt_job job = fetch_job(jobs, one, w);
    const Tw t = load_tw(job.tw);
    const typename M::Out to(t);
    const u64* in = reinterpret_cast<const u64*>(job.in);
    for (int i = threadIdx.x; i < n; i += blockDim.x) sm[i] = in[i];
    __syncthreads();
    for (int s = 0; s < log_n; s++) {
      const int half = n >> (s + 1);
      for (int p = threadIdx.x; p < n / 2; p += blockDim.x) {
        const int blk = p >> (log_n - 1 - s);
        const int x = blk * 2 * half + (p & (half - 1));
        const ulonglong2 wt =
            ld_tw(ROWS ? t.fwd + vkcu_tw_slot(log_n, (1u << s) + blk) : t.fwd + (1 << s) + blk);
        if (s == 0)
          ct_first<M>(sm[x], sm[x + half], wt.x, wt.y, t);
        else
          M::template ct<true>(sm[x], sm[x + half], wt.x, wt.y, t);
      }
      __syncthreads();
    }
    u64* out = reinterpret_cast<u64*>(job.out);
    for (int i = threadIdx.x; i < n; i += blockDim.x) out[i] = to.canon(sm[i]);
    __syncthreads();
  }
}

template <class M, bool ROWS>
__global__ void k_ntt_inv_simple(const vkcu_ntt_job* __restrict__ jobs, int njobs, vkcu_ntt_job one,
                                 int log_n) {
  extern __shared__ u64 sm[];
  const int n = 1 << log_n;
  for (int w = blockIdx.x; w < njobs; w += gridDim.x) {
    const vkcu_ntt_job job = fetch_job(jobs, one, w);
    const Tw t = load_tw(job.tw);
    const ulonglong2 f0 = ld_late2(t.fold), f1 = ld_late2(t.fold + 1);
    const u64* in = reinterpret_cast<const u64*>(job.in);
    for (int i = threadIdx.x; i < n; i += blockDim.x) sm[i] = in[i];
    __syncthreads();
    for (int s = log_n - 1; s >= 0; s--) {
      const int half = n >> (s + 1);
      for (int p = threadIdx.x; p < n / 2; p += blockDim.x) {
        const int blk = p >> (log_n - 1 - s);
        const int x = blk * 2 * half + (p & (half - 1));
        u64 sum, dif;
        if (s == log_n - 1)
          gs_first_sd<M>(sm[x], sm[x + half], t, sum, dif);
        else
          M::template sd<1>(sm[x], sm[x + half], t, sum, dif);
        if (s == 0) {
          sm[x] = csub(shoup_lazy_short(sum, f0.x, f0.y, t.q), t.q);
          sm[x + half] = csub(shoup_lazy_short(dif, f1.x, f1.y, t.q), t.q);
        } else {
          const ulonglong2 wt =
            ld_tw(ROWS ? t.inv + vkcu_tw_slot(log_n, (1u << s) + blk) : t.inv + (1 << s) + blk);
          sm[x] = M::template settle<M::sum_bound(1)>(M::sum(sum, t), t);
          sm[x + half] = M::mul(dif, wt.x, wt.y, t);
        }
      }
      __syncthreads();
    }
    u64* out = reinterpret_cast<u64*>(job.out);
    for (int i = threadIdx.x; i < n; i += blockDim.x) out[i] = sm[i];
    __syncthreads();
  }
}

// ---------------------------------------------------------------------------
// Global-memory passes for n >= 2^18: the first (forward) or last (inverse)
// stages run over HBM in passes of KK <= 4 stages each, and the CTA or cluster
// kernels run the others on every sub-block (sub-block r uses twiddle
// multiplier n / its size + r).  A pass starting at stage s0 gives each thread
// one radix-2^KK group: the 2^KK words at stride t = n >> (s0 + KK) inside one
// block of stage s0 (blocks of n >> s0 words), twiddle base 2^s0 + block (root
// index m + block of the reference's stage loop, src/vector.c:536-566).
// Consecutive threads take consecutive offsets, so every load and store is
// coalesced.

// Forward: stages s0 .. s0 + KK - 1, in -> out, forward-lazy; stage 0 takes
// the reference's exact first-stage rule.
template <int KK, class M>
__global__ void __launch_bounds__(256)
    k_fwd_global(const vkcu_ntt_job* __restrict__ jobs, int njobs, vkcu_ntt_job one, int log_n, int s0) {
  const int lt = log_n - s0 - KK;  // log2 of the stride
  const long groups = 1L << (log_n - KK);
  const long total = (long)njobs * groups;
  for (long w = blockIdx.x * (long)blockDim.x + threadIdx.x; w < total; w += (long)gridDim.x * blockDim.x) {
    const vkcu_ntt_job job = fetch_job(jobs, one, (int)(w >> (log_n - KK)));
    const long g = w & (groups - 1);
    const long blk = g >> lt;
    const size_t first = ((size_t)blk << (log_n - s0)) | (size_t)(g & ((1L << lt) - 1));
    const size_t st = (size_t)1 << lt;
    const Tw t = load_tw(job.tw);
    const u64* in = reinterpret_cast<const u64*>(s0 ? job.out : job.in);
    u64 v[1 << KK];
#pragma unroll
    for (int j = 0; j < (1 << KK); j++) v[j] = ld_stream(in + first + j * st);
    const RowTw tw{t.fwd, (1u << s0) + (u32)blk};
    if (s0 == 0)
      ct_first_group<M, KK, 0, true>(v, tw, t);
    else
      ct_first_group<M, KK, 0, false>(v, tw, t);
    u64* out = reinterpret_cast<u64*>(job.out);
#pragma unroll
    for (int j = 0; j < (1 << KK); j++) out[first + j * st] = v[j];
  }
}

// Inverse: stages s0 + KK - 1 .. s0 on `out` in place (after the sub-block
// kernels, which leave words below one unit); the pass with s0 = 0 folds n^-1
// into stage 0, writes canonical words and applies the epilogue (LIFT).
// product: the sub-blocks' products were Product's (fold constants to match).
template <int KK, class M, bool LIFT>
__global__ void __launch_bounds__(256)
    k_inv_global(const vkcu_ntt_job* __restrict__ jobs, int njobs, vkcu_ntt_job one, int log_n, int s0, int product,
                 const __grid_constant__ vkcu_lift lift) {
  const int lt = log_n - s0 - KK;
  const long groups = 1L << (log_n - KK);
  const long total = (long)njobs * groups;
  for (long w = blockIdx.x * (long)blockDim.x + threadIdx.x; w < total; w += (long)gridDim.x * blockDim.x) {
    const vkcu_ntt_job job = fetch_job(jobs, one, (int)(w >> (log_n - KK)));
    const long g = w & (groups - 1);
    const long blk = g >> lt;
    const size_t first = ((size_t)blk << (log_n - s0)) | (size_t)(g & ((1L << lt) - 1));
    const size_t st = (size_t)1 << lt;
    const Tw t = product ? load_tw_product<M>(job.tw) : load_tw(job.tw);
    u64* out = reinterpret_cast<u64*>(job.out);
    u64 v[1 << KK];
#pragma unroll
    for (int j = 0; j < (1 << KK); j++) v[j] = out[first + j * st];
    const RowTw tw{t.inv, (1u << s0) + (u32)blk};
    if (s0 == 0) {
      gs_group<M, KK, 0, false, true>(v, tw, t);
      if constexpr (LIFT) LiftFold(&lift, t.q).apply(v);
    } else {
      gs_group<M, KK, 0, false, false>(v, tw, t);
    }
#pragma unroll
    for (int j = 0; j < (1 << KK); j++) out[first + j * st] = v[j];
  }
}

static constexpr int kMaxCta = 14;      // one CTA per transform
static constexpr int kMaxCluster = 17;  // one cluster of up to 8 CTAs
static constexpr int kMaxLogN = 26;     // global passes + sub-blocks of 2^14 or 2^16 words

static bool aligned32(const void* p) { return (reinterpret_cast<uintptr_t>(p) & 31) == 0; }

template <class S, bool ROWS>
static int simple_launch(cudaStream_t st, bool inverse, const vkcu_ntt_job* jobs, int njobs, const vkcu_ntt_job& one,
                         int log_n, int sms) {
  const int n = 1 << log_n;
  const int threads = n / 2 < 32 ? 32 : (n / 2 > 512 ? 512 : n / 2);
  const int smem = n * 8;
  auto kern = inverse ? k_ntt_inv_simple<S, ROWS> : k_ntt_fwd_simple<S, ROWS>;
  // threads and shared memory depend on n: one occupancy per direction and
  // degree; the kernel's shared-memory limit is the largest n (2^14) always
  static KernelSetup setups[2][kMaxCta + 1];
  int per_sm = 1;
  if (int e = setup_cta(kern, threads, smem, setups[inverse ? 1 : 0][log_n], &per_sm, (1 << kMaxCta) * 8)) return e;
  const int grid = grid_from(per_sm, njobs, sms);
  kern<<<grid, threads, smem, st>>>(jobs, njobs, one, log_n);
  vkcu_count_launches(1);
  return (int)cudaGetLastError();
}

template <class M>
static int simple(cudaStream_t st, bool inverse, const vkcu_ntt_job* jobs, int njobs, const vkcu_ntt_job& one,
                  int log_n, int sms) {
  using S = std::conditional_t<std::is_same<M, Mod63>::value, Simple63, Simple62>;
  return log_n < VKCU_TW_ROWS_LOG_N ? simple_launch<S, false>(st, inverse, jobs, njobs, one, log_n, sms)
                                    : simple_launch<S, true>(st, inverse, jobs, njobs, one, log_n, sms);
}

// The stages above the sub-blocks: `g` of them in as few passes of <= 4 as
// possible, sizes as equal as possible (5: 3 + 2).
struct GlobalPlan {
  int g;
  int passes() const { return (g + 3) / 4; }
  void pass(int p, int* s0, int* kk) const {  // 0-based, in forward order
    const int np = passes(), small = g / np, big = g % np;
    *s0 = p * small + (p < big ? p : big);
    *kk = small + (p < big ? 1 : 0);
  }
};

// Blocks of 256 threads, of 64 where those would leave SMs without one.
static int pass_threads(long work, int sms) { return work < (long)sms * 512 ? 64 : 256; }

template <class M>
static int forward_passes(cudaStream_t st, const vkcu_ntt_job* jobs, int njobs, const vkcu_ntt_job& one, int log_n,
                          GlobalPlan plan, int sms) {
  for (int p = 0; p < plan.passes(); p++) {
    int s0, kk;
    plan.pass(p, &s0, &kk);
    const long work = (long)njobs << (log_n - kk);
    const int threads = pass_threads(work, sms);
    const long blocks = (work + threads - 1) / threads, cap = (long)sms * 8;
    const unsigned grid = (unsigned)(blocks < cap ? blocks : cap);
    switch (kk) {
#define G(K)                                                                       \
  case K:                                                                          \
    k_fwd_global<K, M><<<grid, threads, 0, st>>>(jobs, njobs, one, log_n, s0);      \
    break;
      G(1)
      G(2)
      G(3)
      G(4)
#undef G
      default:
        return (int)cudaErrorInvalidValue;
    }
    vkcu_count_launches(1);
    if (const int e = (int)cudaGetLastError()) return e;
  }
  return 0;
}

template <class M>
static int inverse_passes(cudaStream_t st, const vkcu_ntt_job* jobs, int njobs, const vkcu_ntt_job& one, int log_n,
                          GlobalPlan plan, int sms, int product, const vkcu_lift* lift) {
  const vkcu_lift none{};
  for (int p = plan.passes() - 1; p >= 0; p--) {
    int s0, kk;
    plan.pass(p, &s0, &kk);
    const long work = (long)njobs << (log_n - kk);
    const int threads = pass_threads(work, sms);
    const long blocks = (work + threads - 1) / threads, cap = (long)sms * 8;
    const unsigned grid = (unsigned)(blocks < cap ? blocks : cap);
    switch (kk * 2 + (lift && s0 == 0 ? 1 : 0)) {
#define G(K)                                                                                                     \
  case 2 * K:                                                                                                    \
    k_inv_global<K, M, false><<<grid, threads, 0, st>>>(jobs, njobs, one, log_n, s0, product, none);             \
    break;                                                                                                       \
  case 2 * K + 1:                                                                                                \
    k_inv_global<K, M, true><<<grid, threads, 0, st>>>(jobs, njobs, one, log_n, s0, product, *lift);             \
    break;
      G(1)
      G(2)
      G(3)
      G(4)
#undef G
      default:
        return (int)cudaErrorInvalidValue;
    }
    vkcu_count_launches(1);
    if (const int e = (int)cudaGetLastError()) return e;
  }
  return 0;
}

// log2 of the sub-blocks per transform of 2^log_n >= 2^17 words, and whether each
// is one CTA's:
//   * few: 2^14 words on clusters of 8 small CTAs, where 2^16-word sub-blocks
//     would leave half of the SMs idle.  Products, 4-CTA / 8-CTA: 1 of 2^18 (4
//     sub-blocks of 2^16) 86 / 37 us, 4 of 2^18 (16) 94 / 66 us, 9 of 2^18 (36)
//     108 / 128 us, 15 of 2^20 (240) 722 / 907 us;
//   * 2^16 words on clusters of 4 CTAs: two stages less above them, one pass over
//     HBM less for it at most degrees, and a product's sub-blocks in one launch;
//   * 2^14 words on one CTA (products: both transforms, the pointwise kernel and
//     the inverse): no room lost between clusters -- 36 of 4 CTAs fit 152 SMs --
//     and rounds of 38 in their place.
// Transforms take the last where it adds no pass over HBM or saves one round in
// eight, products where it saves one in five, which outweighs three more
// launches over HBM.  4-CTA clusters / CTAs, us,
// q < 2^60: 19 x 2^18 (3 rounds / 2) forward 95 / 66, inverse 96 / 68, product
// 272 / 212; 18 x 2^18 (2 / 2) 70 / 64, 70 / 66, 196 / 209; 7 x 2^20 (4 / 3) 135
// / 105, 141 / 118, 394 / 345; 13 x 2^20 (6 / 6) 215 / 208, 225 / 227, 615 /
// 685; 14 x 2^20 (7 / 6) 244 / 214, 253 / 234, 696 / 710; 4 x 2^21 (4 / 4) 156
// / 144, 164 / 165, 442 / 473; 2 x 2^24 (15 / 14) 632 / 618, 684 / 711, 1800 /
// 2062; q in [2^60, 2^62): 19 x 2^18 105 / 72, 109 / 76,
// 310 / 232; 7 x 2^20 150 / 117, 161 / 129, 454 / 380.
struct Subs {
  int log = 0;
  bool cta = false;
  Subs(int njobs, int log_n, int sms, bool product) {
    const long subs = log_n < 18 ? 0 : (long)njobs << (log_n - 16);  // of 2^16 words
    if (subs * 8 <= sms) {
      log = log_n - 14;
      return;
    }
    const long clusters = sms * 9L / 38, ctas = sms / 4;
    const long rounds = (subs + clusters - 1) / clusters, cta_rounds = (subs + ctas - 1) / ctas;
    const bool no_more_passes = log_n == 18 || log_n == 21;  // 2 or 5 stages above 2^16 words, 4 or 7 above 2^14
    const long saved = rounds - cta_rounds;
    cta = product ? saved * 5 >= rounds : saved * 8 >= rounds || no_more_passes;
    log = log_n - (cta ? 14 : 16);
  }
};

}  // namespace vk

using namespace vk;

extern "C" uint32_t vkcu_max_fused_log_n(void) { return kMaxCluster; }
extern "C" uint32_t vkcu_max_log_n(void) { return kMaxLogN; }

static bool jobs_aligned(const vkcu_ntt_job* jobs, const vkcu_ntt_job* one) {
  // Device job arrays are built by the library with aligned vectors; a single
  // job is checked here.
  return jobs != nullptr || (aligned32(one->in) && aligned32(one->out));
}

// log2 of the CTAs that share a job where a launch has fewer jobs than the SMs
// it may count on (`avail`: all, or its share of a batch's concurrent classes),
// 0 for the degree's own kernel (one CTA to 2^14, 2 / 4 CTAs at 2^15 / 2^16).
// A single call (one job passed by value) of 2^14 .. 2^16 takes 16 CTAs, and so
// does a product of 2^17 without scratch (few_of_17 below has the others);
// batches and server micro-batches keep to 8, since their classes run beside other
// kernels and a 16-CTA cluster can only start once 16 SMs of one GPC are free
// at the same time.  Tuning entry (3, 1) = 1 turns the split off, (3, 3) = 1
// keeps single calls on 8.  The lines, from products timed per job count and
// split on 152 SMs (us; the kernel without a split / on 2 / 4 / 8 CTAs a job):
//   2^13: 30 jobs 33 / 25 / 21 / 18, 38: 33 / 25 / 25 / 29, 76: 33 / 25 / 41 / 41,
//         100: 33 / 37 / 43 / 43
//   2^14: 30 jobs 64 / 45 / 27 / 27, 50: 66 / 45 / 40 / 45, 76: 66 / 47 / 57 / 67,
//         100: 66 / 70 / 57 / 72
//   2^15: (2 / 4 / 8) 19 jobs 70 / 47 / 41, 50: 72 / 75 / 62, 60: 72 / 76 / 88
//   2^16: (4 / 8) 19 jobs 78 / 78, 24: 78 / 86
// (2^14 stops at half the SMs although 100 products would still gain on 4 CTAs:
// transforms and products with NTT(b) given lose there, see Tail, which tells
// them apart.)
static int split_log(long njobs, uint32_t log_n, long avail, bool single) {
  if (log_n < 12 || log_n > 17 || vkh_variant(3, 1) != 0) return 0;
  if (single && log_n >= 14 && njobs * 16 <= avail && vkh_variant(3, 3) == 0) return 4;
  if (log_n == 17) return 0;
  switch (log_n) {
    case 13: return njobs * 5 <= avail ? 3 : njobs * 2 <= avail ? 1 : 0;
    case 14: return njobs * 5 <= avail ? 3 : njobs * 5 <= 2 * avail ? 2 : njobs * 2 <= avail ? 1 : 0;
    case 15: return njobs * 3 <= avail ? 3 : 0;
    default: return njobs * 8 <= avail ? 3 : 0;
  }
}

// Few transforms and products of 2^17 take the path of larger degrees: a global
// pass and 2^14-word sub-blocks on 8 small CTAs, 64 SMs a job instead of 8 or
// 16 (forward transforms, 8-CTA clusters / so: 1 33 / 12 us, 4 33 / 16, 9 35 /
// 27; products 1 83 / 29 us, 4 83 / 37, 9 85 / 63; 12 jobs are even).
static bool few_of_17(long njobs, uint32_t log_n, long avail) {
  return log_n == 17 && njobs * 16 <= avail && vkh_variant(3, 1) == 0;
}

// The last jobs of a launch whose kernel runs `round` jobs at a time, one per
// SM or SM pair: those past the whole rounds, where a split finishes them
// sooner than a round of their own.  Only where the launch may count on the
// whole GPU -- concurrent classes of a batch fill a partial round anyway (the
// server's chunks, whose classes run one after another on a stream each, count
// on it too).  Products of 2^14
// in us, without / with the split tail: 160 (8 past the round) 129 / 91, 200
// (48) 131 / 108, 344 (40) 193 / 172; of 2^15, 80 (4) 139 / 103, 160 (8) 207 /
// 172, 120 (44) 142 / 135.  A tail of 77 .. 106 products of 2^14 on 4 CTAs each
// still gains (256 products 131.6 -> 128.2), the shorter transforms and
// products with NTT(b) given lose 2-4 % there, as do 48 products of 2^15 with
// NTT(b) given.
struct Tail {
  int jobs = 0, lc = 0;
  // `long_job`: a product with both forward transforms
  Tail(bool batch, int njobs, uint32_t log_n, int round, int sms, int avail, bool long_job) {
    if (!batch || avail < sms || round < 1 || njobs <= round || vkh_variant(3, 1) != 0) return;
    const int r = njobs % round;
    if (r == 0 || (log_n == 15 && r * 10 > 3 * sms)) return;
    lc = split_log(r, log_n, sms, false);
    if (!lc && log_n == 14 && long_job && r * 10 <= 7 * sms) lc = 2;
    if (lc) jobs = r;
  }
};
// Jobs of one round: 2^14 words take an SM each (139 KB of shared memory),
// 2^13 ones in the 512-thread shape (variant 2) too, 2^15 ones two SMs; 0
// for the others, whose rounds overlap.
static int round_jobs(uint32_t log_n, int variant, int sms) {
  return log_n == 14 || (log_n == 13 && variant == 2) ? sms : log_n == 15 ? sms / 2 : 0;
}

// f(M{}) for the modulus class's M; the wide class has launchers of its own.
template <class M>
static constexpr bool kWide = std::is_same<M, Mod63>::value;

template <class F>
static int by_class(int qclass, F&& f) {
  return qclass == VKCU_Q60 ? f(Mod60{}) : qclass == VKCU_Q62 ? f(Mod62{}) : f(Mod63{});
}

template <class M>
static int forward(void* stream, const vkcu_ntt_job* jobs, int njobs, const vkcu_ntt_job* one, uint32_t log_n,
                   int sms, int avail) {
  cudaStream_t st = (cudaStream_t)stream;
  const vkcu_ntt_job o = one ? *one : vkcu_ntt_job{};
  if (log_n < 1 || log_n > (uint32_t)kMaxLogN || njobs < 1) return (int)cudaErrorInvalidValue;
  const bool aligned = jobs_aligned(jobs, one);
  if (log_n < 8 || (log_n <= (uint32_t)kMaxCta && !aligned))
    return simple<M>(st, false, jobs, njobs, o, (int)log_n, sms);
  if (!aligned) return (int)cudaErrorMisalignedAddress;
  if constexpr (kWide<M>) {
    if (log_n <= (uint32_t)kMaxCta) return fwd_cta_wide(st, jobs, njobs, o, (int)log_n, 0, sms);
    if (log_n <= (uint32_t)kMaxCluster) return fwd_cluster_wide(st, jobs, njobs, o, (int)log_n - kMaxCta);
  } else {
    if (const int lc = log_n < (uint32_t)kMaxCluster ? split_log(njobs, log_n, avail, jobs == nullptr) : 0) {
      const int e = fwd_cluster<M>(st, jobs, njobs, o, lc, (int)log_n - lc);
      // a GPU that cannot host 16-CTA clusters: the set-up refuses before any launch
      return e == (int)cudaErrorInvalidConfiguration && lc == 4
                 ? fwd_cluster<M>(st, jobs, njobs, o, 3, (int)log_n - 3)
                 : e;
    }
    if (log_n <= (uint32_t)kMaxCluster && !few_of_17(njobs, log_n, avail)) {
      const int variant = log_n <= (uint32_t)kMaxCta ? vkh_variant_jobs(1, (int)log_n, njobs, sms) : 0;
      const Tail tail(jobs != nullptr, njobs, log_n, round_jobs(log_n, variant, sms), sms, avail, false);
      const int main = njobs - tail.jobs;
      const int e = log_n <= (uint32_t)kMaxCta ? fwd_cta<M>(st, jobs, main, o, (int)log_n, sms, variant)
                                               : fwd_cluster<M>(st, jobs, main, o, (int)log_n - kMaxCta, kMaxCta);
      return e || !tail.jobs ? e : fwd_cluster<M>(st, jobs + main, tail.jobs, o, tail.lc, (int)log_n - tail.lc);
    }
  }
  if constexpr (kWide<M>) {
    const int sub_log = (int)log_n - kMaxCta;
    const int e = forward_passes<M>(st, jobs, njobs, o, (int)log_n, GlobalPlan{sub_log}, sms);
    return e ? e : fwd_cta_wide(st, jobs, njobs, o, kMaxCta, sub_log, sms);
  } else {
    const Subs subs(njobs, (int)log_n, sms, false);
    if (const int e = forward_passes<M>(st, jobs, njobs, o, (int)log_n, GlobalPlan{subs.log}, sms)) return e;
    return subs.cta ? fwd_cta_sub<M>(st, jobs, njobs, o, subs.log, sms)
                    : fwd_cluster_sub<M>(st, jobs, njobs, o, (int)log_n, subs.log);
  }
}

extern "C" int vkcu_ntt_forward(void* stream, const vkcu_ntt_job* jobs, int njobs, const vkcu_ntt_job* one,
                                uint32_t log_n, int qclass, int sms, int avail) {
  return by_class(qclass, [&](auto m) { return forward<decltype(m)>(stream, jobs, njobs, one, log_n, sms, avail); });
}

static bool has_lift(const vkcu_lift* lift) { return lift && lift->count > 0; }

template <class M>
static int inverse(void* stream, const vkcu_ntt_job* jobs, int njobs, const vkcu_ntt_job* one, uint32_t log_n, int sms,
                   int avail, const vkcu_lift* lift) {
  cudaStream_t st = (cudaStream_t)stream;
  const vkcu_ntt_job o = one ? *one : vkcu_ntt_job{};
  if (log_n < 1 || log_n > (uint32_t)kMaxLogN || njobs < 1) return (int)cudaErrorInvalidValue;
  if (has_lift(lift) && lift->count > VKCU_MAX_LIFT) return (int)cudaErrorInvalidValue;
  const bool aligned = jobs_aligned(jobs, one);
  const bool lifted = has_lift(lift);
  const vkcu_lift* lp = lifted ? lift : nullptr;
  int e;
  if (log_n < 8 || (log_n <= (uint32_t)kMaxCta && !aligned)) {
    e = simple<M>(st, true, jobs, njobs, o, (int)log_n, sms);
  } else if (!aligned) {
    return (int)cudaErrorMisalignedAddress;
  } else {
    if constexpr (kWide<M>) {
      if (log_n <= (uint32_t)kMaxCta) return inv_cta_wide(st, jobs, njobs, o, (int)log_n, 0, sms, lp);
      if (log_n <= (uint32_t)kMaxCluster) return inv_cluster_wide(st, jobs, njobs, o, (int)log_n - kMaxCta, lp);
    } else {
      if (const int lc = log_n < (uint32_t)kMaxCluster ? split_log(njobs, log_n, avail, jobs == nullptr) : 0) {
        const int r = inv_cluster<M>(st, jobs, njobs, o, lc, (int)log_n - lc, lp);
        return r == (int)cudaErrorInvalidConfiguration && lc == 4
                   ? inv_cluster<M>(st, jobs, njobs, o, 3, (int)log_n - 3, lp)
                   : r;
      }
      if (log_n <= (uint32_t)kMaxCluster && !few_of_17(njobs, log_n, avail)) {
        // the lifted CTA kernels run in the default shape
        const int variant = log_n <= (uint32_t)kMaxCta && !lifted ? vkh_variant_jobs(2, (int)log_n, njobs, sms) : 0;
        const Tail tail(jobs != nullptr, njobs, log_n, round_jobs(log_n, variant, sms), sms, avail, false);
        const int main = njobs - tail.jobs;
        const int r = log_n > (uint32_t)kMaxCta ? inv_cluster<M>(st, jobs, main, o, (int)log_n - kMaxCta, kMaxCta, lp)
                      : lifted                  ? inv_cta_lift<M>(st, jobs, main, o, (int)log_n, sms, *lift)
                                                : inv_cta<M>(st, jobs, main, o, (int)log_n, sms, variant);
        return r || !tail.jobs ? r : inv_cluster<M>(st, jobs + main, tail.jobs, o, tail.lc, (int)log_n - tail.lc, lp);
      }
    }
    int sub_log;
    if constexpr (kWide<M>) {
      sub_log = (int)log_n - kMaxCta;
      e = inv_cta_wide(st, jobs, njobs, o, kMaxCta, sub_log, sms, nullptr);
    } else {
      const Subs subs(njobs, (int)log_n, sms, false);
      sub_log = subs.log;
      e = subs.cta ? inv_cta_sub<M>(st, jobs, njobs, o, sub_log, sms)
                   : inv_cluster_sub<M>(st, jobs, njobs, o, (int)log_n, sub_log);
    }
    return e ? e : inverse_passes<M>(st, jobs, njobs, o, (int)log_n, GlobalPlan{sub_log}, sms, 0, lp);
  }
  // the simple kernels take the epilogue as one more element-wise launch
  if (!e && lifted) e = vkcu_lift_jobs(stream, jobs, njobs, one, log_n, sms, lift);
  return e;
}

extern "C" int vkcu_ntt_inverse_lift(void* stream, const vkcu_ntt_job* jobs, int njobs, const vkcu_ntt_job* one,
                                     uint32_t log_n, int qclass, int sms, int avail, const vkcu_lift* lift) {
  return by_class(qclass,
                  [&](auto m) { return inverse<decltype(m)>(stream, jobs, njobs, one, log_n, sms, avail, lift); });
}

// A product of 2^17 .. 2^26 in clusters, q < 2^62: the global passes of b
// (into scratch) and of a (into c), one launch for every sub-block's forward,
// product and inverse, the inverse global passes of c.  b, a and c give these
// the jobs of the passes.
template <class M>
static int polymul_large(cudaStream_t st, const vkcu_poly_job* jobs, const vkcu_ntt_job* b, const vkcu_ntt_job* a,
                         const vkcu_ntt_job* c, int njobs, const vkcu_poly_job& one, int log_n, int sms,
                         const vkcu_lift* lift, int b_ntt) {
  const vkcu_ntt_job ob{one.b, one.scratch, one.tw}, oa{one.a, one.c, one.tw}, oc{one.c, one.c, one.tw};
  const int sub_log = Subs(njobs, log_n, sms, true).log;
  const GlobalPlan plan{sub_log};
  int e = b_ntt ? 0 : forward_passes<M>(st, b, njobs, ob, log_n, plan, sms);
  if (!e) e = forward_passes<M>(st, a, njobs, oa, log_n, plan, sms);
  if (!e) e = poly_cluster_sub<M>(st, jobs, njobs, one, log_n, sub_log);
  if (!e) e = inverse_passes<M>(st, c, njobs, oc, log_n, plan, sms, 1, lift);
  return e;
}

template <class M>
static int polymul(void* stream, const vkcu_poly_job* jobs, int njobs, const vkcu_poly_job* one, uint32_t log_n,
                   int sms, int avail, const vkcu_lift* lift, int b_ntt) {
  cudaStream_t st = (cudaStream_t)stream;
  const vkcu_poly_job o = one ? *one : vkcu_poly_job{};
  if (log_n < 8 || log_n > (uint32_t)kMaxCluster || njobs < 1) return (int)cudaErrorInvalidValue;
  if (has_lift(lift) && lift->count > VKCU_MAX_LIFT) return (int)cudaErrorInvalidValue;
  static const vkcu_lift kNoSteps{};  // the epilogue instantiations with nothing to apply
  const vkcu_lift* lp = has_lift(lift) ? lift : b_ntt ? &kNoSteps : nullptr;
  if constexpr (kWide<M>) {
    if (log_n <= (uint32_t)kMaxCta) return poly_cta_wide(st, jobs, njobs, o, (int)log_n, sms, lp);
    return poly_cluster_wide(st, jobs, njobs, o, (int)log_n - kMaxCta, lp);
  } else {
    if (const int lc = split_log(njobs, log_n, avail, jobs == nullptr)) {
      const int e = poly_cluster<M>(st, jobs, njobs, o, lc, (int)log_n - lc, lp);
      return e == (int)cudaErrorInvalidConfiguration && lc == 4
                 ? poly_cluster<M>(st, jobs, njobs, o, 3, (int)log_n - 3, lp)
                 : e;
    }
    const int variant = log_n <= (uint32_t)kMaxCta ? vkh_variant_jobs(0, (int)log_n, njobs, sms) : 0;
    const Tail tail(jobs != nullptr, njobs, log_n, round_jobs(log_n, variant, sms), sms, avail, !b_ntt);
    const int main = njobs - tail.jobs;
    const int e = log_n > (uint32_t)kMaxCta ? poly_cluster<M>(st, jobs, main, o, (int)log_n - kMaxCta, kMaxCta, lp)
                  : lp                      ? poly_cta_lift<M>(st, jobs, main, o, (int)log_n, sms, variant, *lp)
                                            : poly_cta<M>(st, jobs, main, o, (int)log_n, sms, variant);
    return e || !tail.jobs ? e : poly_cluster<M>(st, jobs + main, tail.jobs, o, tail.lc, (int)log_n - tail.lc, lp);
  }
}

extern "C" int vkcu_polymul_lift(void* stream, const vkcu_poly_job* jobs, int njobs, const vkcu_poly_job* one,
                                 uint32_t log_n, int qclass, int sms, int avail, const vkcu_lift* lift, int b_ntt) {
  return by_class(
      qclass, [&](auto m) { return polymul<decltype(m)>(stream, jobs, njobs, one, log_n, sms, avail, lift, b_ntt); });
}

extern "C" int vkcu_polymul(void* stream, const vkcu_poly_job* jobs, int njobs, const vkcu_poly_job* one,
                            uint32_t log_n, int qclass, int sms) {
  return vkcu_polymul_lift(stream, jobs, njobs, one, log_n, qclass, sms, sms, nullptr, 0);
}

// A product outside the single-launch degrees (or few of 2^17): as above; for
// n < 2^8, and past one cluster where each sub-block is one CTA's (Subs above,
// q >= 2^62), forward(b), forward(a), pointwise, inverse.
extern "C" int vkcu_few_composed(long njobs, uint32_t log_n, int qclass, int avail) {
  return qclass != VKCU_Q63 && few_of_17(njobs, log_n, avail);
}

extern "C" int vkcu_polymul_composed(void* stream, const vkcu_poly_job* jobs, const vkcu_ntt_job* b,
                                     const vkcu_ntt_job* a, const vkcu_ntt_job* c, int njobs,
                                     const vkcu_poly_job* one, uint32_t log_n, int qclass, int sms,
                                     const vkcu_lift* lift, int b_ntt) {
  cudaStream_t st = (cudaStream_t)stream;
  const vkcu_poly_job o = one ? *one : vkcu_poly_job{};
  if (log_n < 1 || log_n > (uint32_t)kMaxLogN || njobs < 1) return (int)cudaErrorInvalidValue;
  if (has_lift(lift) && lift->count > VKCU_MAX_LIFT) return (int)cudaErrorInvalidValue;
  const vkcu_lift* lp = has_lift(lift) ? lift : nullptr;
  const bool aligned =
      jobs != nullptr || (aligned32(o.a) && aligned32(o.b) && aligned32(o.c) && aligned32(o.scratch));
  if (log_n >= (uint32_t)kMaxCluster && !aligned) return (int)cudaErrorMisalignedAddress;
  const bool clusters = log_n >= (uint32_t)kMaxCluster && !(jobs && Subs(njobs, (int)log_n, sms, true).cta);
  if (clusters && qclass == VKCU_Q60)
    return polymul_large<Mod60>(st, jobs, b, a, c, njobs, o, (int)log_n, sms, lp, b_ntt);
  if (clusters && qclass == VKCU_Q62)
    return polymul_large<Mod62>(st, jobs, b, a, c, njobs, o, (int)log_n, sms, lp, b_ntt);
  if (!jobs) return (int)cudaErrorInvalidValue;  // single calls issue these four themselves
  int e = b_ntt ? 0 : vkcu_ntt_forward(stream, b, njobs, nullptr, log_n, qclass, sms, sms);
  if (!e) e = vkcu_ntt_forward(stream, a, njobs, nullptr, log_n, qclass, sms, sms);
  if (!e) e = vkcu_pointwise(stream, jobs, njobs, log_n, qclass, sms);
  if (!e) e = vkcu_ntt_inverse_lift(stream, c, njobs, nullptr, log_n, qclass, sms, sms, lift);
  return e;
}

// The epilogue as its own element-wise pass: over `len` words at p, or over
// the n output words of each job (q from the job's twiddle set).  Words move
// as 16-byte pairs, two pairs per thread per round, software pipelined (the
// next round's loads are issued before this round's four words walk the
// step list together and are stored); a word before the first 16-byte
// boundary and an odd last word are done alone, and a job whose output is
// not 16-byte aligned word by word.  The grid is one wave of resident blocks.
__device__ __forceinline__ void lift_pairs(u64* __restrict__ a, long lo, long hi, long stride, const LiftRun& lr) {
  ulonglong2 x0 = make_ulonglong2(0, 0), x1 = x0;
  if (lo < hi) x0 = ld2(a + 2 * lo);
  if (lo + stride < hi) x1 = ld2(a + 2 * (lo + stride));
  for (long p = lo; p < hi; p += 2 * stride) {
    const long n0 = p + 2 * stride, n1 = n0 + stride;
    ulonglong2 y0 = x0, y1 = x1;
    if (n0 < hi) y0 = ld2(a + 2 * n0);
    if (n1 < hi) y1 = ld2(a + 2 * n1);
    u64 v[4] = {x0.x, x0.y, x1.x, x1.y};
    lr.apply(v);
    st2(a + 2 * p, v[0], v[1]);
    if (p + stride < hi) st2(a + 2 * (p + stride), v[2], v[3]);
    x0 = y0;
    x1 = y1;
  }
}

__global__ void __launch_bounds__(256) k_lift_range(u64* __restrict__ p, u64 len, u64 q,
                                                    const __grid_constant__ vkcu_lift lift) {
  const LiftRun lr(&lift, q);
  const u64 head = (reinterpret_cast<uintptr_t>(p) & 15) ? 1 : 0;
  const bool first = blockIdx.x == 0 && threadIdx.x == 0;
  if (head && len && first) p[0] = lr(p[0]);
  u64* a = p + head;
  const u64 rest = len > head ? len - head : 0;
  lift_pairs(a, (long)(blockIdx.x * blockDim.x + threadIdx.x), (long)(rest >> 1), (long)gridDim.x * blockDim.x, lr);
  if ((rest & 1) && first) a[rest - 1] = lr(a[rest - 1]);
}

// The epilogue of the simple kernels' jobs (n < 2^8, and to 2^14 when a pointer
// is off the 32-byte grid): one block per job (grid-stride over the jobs),
// blockDim sized to the job.  Every other path lifts in its last pass.
template <class L>
__device__ __forceinline__ void lift_segment(u64* __restrict__ out, long words, const L& lr) {
  if ((reinterpret_cast<uintptr_t>(out) & 15) == 0) {
    lift_pairs(out, threadIdx.x, words >> 1, blockDim.x, lr);
    if ((words & 1) && threadIdx.x == 0) out[words - 1] = lr(out[words - 1]);
  } else {
    for (long i = threadIdx.x; i < words; i += blockDim.x) out[i] = lr(out[i]);
  }
}

__global__ void __launch_bounds__(256) k_lift_jobs(const vkcu_ntt_job* __restrict__ jobs, int njobs, vkcu_ntt_job one,
                                                   int log_n, const __grid_constant__ vkcu_lift lift) {
  for (int w = blockIdx.x; w < njobs; w += gridDim.x) {
    const vkcu_ntt_job job = fetch_job(jobs, one, w);
    const LiftRun lr(&lift, load_tw(job.tw).q);
    lift_segment(reinterpret_cast<u64*>(job.out), 1L << log_n, lr);
  }
}

template <auto kernel>
static long resident_blocks(int sms) {
  static const int per_sm = [] {
    int b = 0;
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&b, kernel, 256, 0) != cudaSuccess || b < 1) b = 1;
    return b;
  }();
  return (long)(sms > 0 ? sms : 1) * per_sm;
}

extern "C" int vkcu_lift_range(void* stream, uint64_t* p, uint64_t len, uint64_t q, int sms, const vkcu_lift* lift) {
  if (!has_lift(lift) || len == 0) return 0;
  if (lift->count > VKCU_MAX_LIFT) return (int)cudaErrorInvalidValue;
  long blocks = (long)((len + 1023) / 1024);  // four words per thread per round
  const long cap = resident_blocks<k_lift_range>(sms);
  if (blocks > cap) blocks = cap;
  k_lift_range<<<(unsigned)blocks, 256, 0, (cudaStream_t)stream>>>(reinterpret_cast<u64*>(p), len, q, *lift);
  vkcu_count_launches(1);
  return (int)cudaGetLastError();
}

extern "C" int vkcu_lift_jobs(void* stream, const vkcu_ntt_job* jobs, int njobs, const vkcu_ntt_job* one,
                              uint32_t log_n, int sms, const vkcu_lift* lift) {
  if (!has_lift(lift)) return 0;
  if (njobs < 1 || log_n > (uint32_t)kMaxLogN || lift->count > VKCU_MAX_LIFT) return (int)cudaErrorInvalidValue;
  const vkcu_ntt_job o = one ? *one : vkcu_ntt_job{};
  const long pairs = (1L << log_n) / 2;  // a thread per pair up to 256
  const int threads = pairs <= 32 ? 32 : pairs >= 256 ? 256 : (int)pairs;
  const long cap = (long)(sms > 0 ? sms : 1) * 16;
  const long blocks = njobs < cap ? njobs : cap;
  k_lift_jobs<<<(unsigned)blocks, threads, 0, (cudaStream_t)stream>>>(jobs, njobs, o, (int)log_n, *lift);
  vkcu_count_launches(1);
  return (int)cudaGetLastError();
}

// Pointwise step of a composed polymul: c = c * scratch mod q over njobs
// jobs of n words each, the word the reference's elemmul stores: c is a
// canonical NTT output, scratch one too or the caller's NTT(b), reduced as
// elemmul reduces its operands.  A block takes chunks of up to 2048 words of
// one job (the job's constants loaded once per chunk, not per word), each
// thread two 16-byte pairs of c and of scratch per round, loads first.
template <class M>
__global__ void __launch_bounds__(256)
    k_pointwise(const vkcu_poly_job* __restrict__ jobs, int njobs, int log_n) {
  const int lw = log_n < 11 ? log_n : 11;  // log2 of the words of a chunk
  const long cpj = 1L << (log_n - lw);    // chunks per job
  const long total = (long)njobs * cpj;
  const int pairs = 1 << (lw - 1);         // n >= 2
  for (long ch = blockIdx.x; ch < total; ch += gridDim.x) {
    const vkcu_poly_job job = jobs[ch >> (log_n - lw)];
    const Tw t = load_tw(job.tw);
    const long base = (ch & (cpj - 1)) << lw;
    u64* c = reinterpret_cast<u64*>(job.c) + base;
    const u64* y = reinterpret_cast<const u64*>(job.scratch) + base;
    const u64 mu = t.mu();
    const u32 qbits = t.qbits();
    auto prod = [&](u64 x, u64 b) { return M::product_out(x, ref_reduce64_maybe(b, t.q, mu, qbits), t, mu, qbits); };
    for (int p = (int)threadIdx.x; p < pairs; p += 2 * (int)blockDim.x) {
      const int p1 = p + (int)blockDim.x;
      const bool two = p1 < pairs;
      const ulonglong2 x0 = ld2(c + 2 * p), y0 = ld2(y + 2 * p);
      ulonglong2 x1 = x0, y1 = y0;
      if (two) {
        x1 = ld2(c + 2 * p1);
        y1 = ld2(y + 2 * p1);
      }
      st2(c + 2 * p, prod(x0.x, y0.x), prod(x0.y, y0.y));
      if (two) st2(c + 2 * p1, prod(x1.x, y1.x), prod(x1.y, y1.y));
    }
  }
}

extern "C" int vkcu_pointwise(void* stream, const vkcu_poly_job* jobs, int njobs, uint32_t log_n, int qclass, int sms) {
  if (njobs < 1 || !jobs || log_n < 1) return (int)cudaErrorInvalidValue;
  const long chunks = (long)njobs << (log_n > 11 ? log_n - 11 : 0);
  long blocks = chunks;
  if (blocks > (long)sms * 8) blocks = (long)sms * 8;
  return by_class(qclass, [&](auto m) {
    k_pointwise<decltype(m)><<<(int)blocks, 256, 0, (cudaStream_t)stream>>>(jobs, njobs, (int)log_n);
    vkcu_count_launches(1);
    return (int)cudaGetLastError();
  });
}
