// Shared device code of the negacyclic NTT / INTT / fused polymul kernels.
//
// Transform convention (identical to the reference):
//   forward  = the Cooley-Tukey stage loop of src/vector.c:536-566 with the
//              butterfly of src/kernels/shaders/nttfwdbutterfly.comp:41-57,
//              natural order in, bit-reversed order out;
//   inverse  = the Gentleman-Sande loop of src/vector.c:599-630 with the
//              butterfly of nttrevbutterfly.comp:41-57, bit-reversed in,
//              natural out, then x n^-1 (src/vector.c:632-638);
//   twiddles = powers of w in bit-reversed order, root index m + block
//              (src/ntt_tables.c:25-43, src/kernels/nttfwdbutterfly.c:154-159).
//
// GB300 design.  One CTA owns one polynomial of n = 2^LOGN <= 2^14 words
// held in shared memory (padded by one word per 16: index a -> a + a/16,
// which makes every access pattern below free of bank conflicts).  The
// log2(n) butterfly stages run as passes of up to 4 stages: in a pass every
// thread loads radix-2^k groups of words into registers, one group at a time,
// runs the k stages on them and writes them back, so at most 16 words (plus
// their twiddles) are live per thread.  Exceptions:
//   * the first forward pass reads all of the thread's words from global
//     memory up front (the loads are coalesced and all in flight at once);
//   * the last forward pass works on groups of 16 consecutive words, whose
//     results leave through shared memory in whole lines (from 2^9 words; by
//     32-byte vector stores below), or -- in the fused polymul -- are
//     multiplied pointwise by NTT(b) and run through the first inverse pass in
//     the same registers;
//   * the last inverse pass folds n^-1 into its final stage and writes global
//     memory coalesced.
// Butterflies are lazy (Harvey): values stay in [0, kq) and are made canonical
// once at the end, k as large as 64 bits allow: 12 for q < 2^60, 4 for q <
// 2^62, 2 for q < 2^63 (the top of the reference's range: its inverse-mod
// works below 2^63, src/numbers.c:71-99).  The kernels are templates over
// these modulus classes (Mod60, Mod62, Mod63 below).
//
// Bit-exactness for unreduced inputs.  The reference's first stage computes
// (X + WY) mod 2^64 mod q and (X - WY) mod q (forward), or (X + Y) mod 2^64
// mod q and W (X - Y mod q) (inverse).  All later stages see canonical values,
// so only the first stage needs the reference's wrap-around behaviour; it is
// taken on a rarely-used branch whenever an input is past the bound up to which
// the class's lazy butterfly is congruent to it: forward, x >= 3q (Mod60), 2q
// (Mod62) or q (Mod63); inverse, a word of the group >= 2^bits(q), or either
// word >= q (Mod63).
#pragma once

#include <cuda_runtime.h>

#include <atomic>
#include <type_traits>

#include "arith.cuh"
#include "kernels.h"

namespace vk {

template <int I, int N, typename F>
__device__ __forceinline__ void static_for(F&& f) {
  if constexpr (I < N) {
    f(std::integral_constant<int, I>{});
    static_for<I + 1, N>(f);
  }
}

__device__ __forceinline__ int pad(int a) { return a + (a >> 4); }

__device__ __forceinline__ ulonglong2 ld_tw(const ulonglong2* p) {
  ulonglong2 r;
  asm("ld.global.nc.v2.u64 {%0,%1}, [%2];" : "=l"(r.x), "=l"(r.y) : "l"(p));
  return r;
}

__device__ __forceinline__ u64 ld_stream(const u64* p) {
  u64 r;
  asm volatile("ld.global.L1::no_allocate.u64 %0, [%1];" : "=l"(r) : "l"(p));
  return r;
}

__device__ __forceinline__ void ld4(const u64* p, u64& a, u64& b, u64& c, u64& d) {
  asm volatile("ld.global.v4.u64 {%0,%1,%2,%3}, [%4];" : "=l"(a), "=l"(b), "=l"(c), "=l"(d) : "l"(p));
}

__device__ __forceinline__ void st4(u64* p, u64 a, u64 b, u64 c, u64 d) {
  asm volatile("st.global.v4.u64 [%0], {%1,%2,%3,%4};" ::"l"(p), "l"(a), "l"(b), "l"(c), "l"(d) : "memory");
}

// Bring `bytes` at p into L2 ahead of use (no registers, no completion wait).
__device__ __forceinline__ void prefetch_l2(const void* p, unsigned bytes) {
  asm volatile("cp.async.bulk.prefetch.L2.global [%0], %1;" ::"l"(p), "r"(bytes) : "memory");
}

// A constant that is needed late in a kernel, loaded where it is used (an L1
// or L2 hit) instead of holding registers from the start: volatile, so that
// the compiler does not hoist it.
__device__ __forceinline__ u64 ld_late(const u64* p) {
  u64 r;
  asm volatile("ld.global.nc.u64 %0, [%1];" : "=l"(r) : "l"(p));
  return r;
}
__device__ __forceinline__ u32 ld_late32(const u32* p) {
  u32 r;
  asm volatile("ld.global.nc.u32 %0, [%1];" : "=r"(r) : "l"(p));
  return r;
}
__device__ __forceinline__ ulonglong2 ld_late2(const ulonglong2* p) {
  ulonglong2 r;
  asm volatile("ld.global.nc.v2.u64 {%0,%1}, [%2];" : "=l"(r.x), "=l"(r.y) : "l"(p));
  return r;
}

// Per-transform constants: the modulus and the tables in registers, the rest
// of the set loaded where it is used.
struct Tw {
  u64 q, q2;
  const ulonglong2* fwd;
  const ulonglong2* inv;
  const ulonglong2* fold;  // (n^-1, shoup), (w1 n^-1, shoup) of the last inverse stage
  const vkcu_twset* set;
  __device__ __forceinline__ u64 mu() const { return ld_late(reinterpret_cast<const u64*>(&set->mu)); }
  __device__ __forceinline__ u64 qinv() const { return ld_late(reinterpret_cast<const u64*>(&set->qinv)); }
  __device__ __forceinline__ u32 qbits() const { return ld_late32(&set->qbits); }
};

__device__ __forceinline__ Tw load_tw(const vkcu_twset* p) {
  Tw t;
  t.q = __ldg(reinterpret_cast<const u64*>(&p->q));
  t.q2 = __ldg(reinterpret_cast<const u64*>(&p->q2));
  t.fwd = reinterpret_cast<const ulonglong2*>(__ldg(reinterpret_cast<const u64*>(&p->fwd)));
  t.inv = reinterpret_cast<const ulonglong2*>(__ldg(reinterpret_cast<const u64*>(&p->inv)));
  t.fold = reinterpret_cast<const ulonglong2*>(&p->ninv);
  t.set = p;
  return t;
}

// The same for a fused product, whose last stage takes what M::Product left
// (divided by 2^64 by a Montgomery product).
template <class M>
__device__ __forceinline__ Tw load_tw_product(const vkcu_twset* p) {
  Tw t = load_tw(p);
  if (M::MONTGOMERY) t.fold = reinterpret_cast<const ulonglong2*>(&p->ninv_m);
  return t;
}

// A caller-supplied NTT(b) operand reduced as the reference's elemmul reduces
// its operands (reduce64, elemmul.comp:36-47): canonical words pass through.
template <int K>
__device__ __forceinline__ void reduce_operands(u64 (&v)[K], const Tw& t) {
  const u64 mu = t.mu();
  const u32 qbits = t.qbits();
#pragma unroll
  for (int j = 0; j < K; j++) v[j] = ref_reduce64_maybe(v[j], t.q, mu, qbits);
}

// ---------------------------------------------------------------------------
// First-stage butterflies with the reference's exact semantics.

struct U2 {
  u64 x, y;
};

// The reference's stage-0 butterfly for x past the fast path's bound, exactly: X' = (X + WY) mod
// 2^64 mod q, Y' = (X - WY) mod q.  Kept out of line: it is rarely taken.
// reduce64 is an exact remainder for q < 2^62.
static __device__ __noinline__ U2 ct_first_slow(u64 x, u64 y, u64 w, u64 wp, u64 q, const vkcu_twset* set) {
  const u64 mu = set->mu;
  const u32 qbits = set->qbits;
  const u64 wy = shoup(y, w, wp, q);
  const u64 xr = ref_reduce64(x, q, mu, qbits);
  return U2{ref_reduce64(x + wy, q, mu, qbits), xr >= wy ? xr - wy : xr + q - wy};
}

// Inverse, stage m = n/2: the sum s and difference d before the twiddle
// product, exactly as the reference's (X + Y) mod 2^64 mod q and the
// residue of its `while (t < Y) t += q; t -= Y` loop.
static __device__ __noinline__ U2 gs_first_slow(u64 x, u64 y, u64 q, const vkcu_twset* set) {
  const u64 mu = set->mu;
  const u32 qbits = set->qbits;
  const u64 xr = ref_reduce64(x, q, mu, qbits);
  const u64 yr = ref_reduce64(y, q, mu, qbits);
  return U2{ref_reduce64(x + y, q, mu, qbits), xr >= yr ? xr - yr : xr + q - yr};
}

// The same two for 2^62 <= q < 2^63, with the exact 64-bit remainder.
static __device__ __noinline__ U2 ct_first_slow63(u64 x, u64 y, u64 w, u64 wp, u64 q) {
  const u64 wy = shoup(y, w, wp, q);
  const u64 xr = x % q;
  return U2{(x + wy) % q, xr >= wy ? xr - wy : xr + q - wy};
}

static __device__ __noinline__ U2 gs_first_slow63(u64 x, u64 y, u64 q) {
  const u64 xr = x % q, yr = y % q;
  return U2{(x + y) % q, xr >= yr ? xr - yr : xr + q - yr};
}

// ---------------------------------------------------------------------------
// Modulus classes: the butterfly arithmetic every kernel is instantiated with.
// A class M gives
//   ct<REDUCE>   a forward butterfly; REDUCE brings x down first, which the
//                passes ask for in the sub-stages where reduce_at(u)
//   sd<B>        sum and difference of two inverse words below B units before
//                the twiddle product (a unit is the inverse passes' resting
//                bound); the sum, after sum(), is below sum_bound(B) units
//   mul          the twiddle product of a difference, below one unit
//   settle<B>    a word below B units brought below one unit
//   Out          forward words -> canonical, or parked (NTT(b) held for the
//                pointwise product)
//   Product      the pointwise product of a forward word and a parked or
//                canonical one, below one unit (MONTGOMERY: times 2^-64)
//   product_out  of two canonical words, the word the reference's elemmul stores
//
// Mod60 (odd q < 2^60): sixteen q fit in 64 bits.  The Shoup quotient leaves
// out one of four 32-bit products and may be two short, so a twiddle product
// is below 3q; forward words stay below 12q, x being brought below 6q in every
// second stage only (12q -> 6q, then 9q, then 12q); inverse words rest below
// 3q between passes and grow by sums inside a pass, at most to 12q, which the
// compiler follows word by word (gs_bound below): 20 conditional subtractions
// for the 32 butterflies of a radix-16 group instead of 32.  The pointwise
// step is a Montgomery product, its 2^64 folded into the last stage's n^-1.
// Against Mod62 on the same primes: 256 products of 2^14 words 168.0 -> 149.7
// us, 3003 of 2^10 87.4 -> 75.1 us, 64 of 2^16 202.7 -> 182.5 us, 1000 forward
// transforms of 2^14 208 -> 192 us, 150 inverse ones of 2^15 88.1 -> 82.0 us.
//
// Mod62 (q < 2^62): forward values in [0, 4q), inverse values in [0, 2q), one
// conditional subtraction per butterfly (Harvey).  The pointwise product is
// a Barrett product whose result is congruent to the reference's elemmul
// (exact for these moduli).
//
// Mod63 (2^62 <= q < 2^63, where 4q overflows): forward and inverse values in
// [0, 2q), two conditional subtractions per butterfly.  The pointwise
// product restates the reference's elemmul formula word for word
// (elemmul.comp:49-73): with a 63-bit modulus its Barrett estimate
// (hi << 3) + (lo >> 61) wraps past 2^64 for large products, so its results
// are not the true residues, and the polymul must reproduce them; the
// inverse stage that follows then takes the exact first-stage rule, since
// such a word need not be below q.
struct Mod60 {
  static constexpr bool EXACT_AFTER_PRODUCT = false, MONTGOMERY = true;
  static constexpr bool reduce_at(int u) { return (u & 1) == 0; }
  template <bool REDUCE>
  __device__ __forceinline__ static void ct(u64& x, u64& y, u64 w, u64 wp, const Tw& t) {
    const u64 q3 = t.q + t.q2;
    const u64 xr = REDUCE ? csub_sign(x, 2 * q3) : x;
    const u64 wy = shoup_lazy3(y, w, wp, 0 - t.q);
    x = xr + wy;
    y = xr - wy + q3;
  }
  // words below B units of 3q; 4 units come down to 2 first
  template <int B>
  __device__ __forceinline__ static void sd(u64 x, u64 y, const Tw& t, u64& s, u64& d) {
    const u64 q3 = t.q + t.q2;
    if (B == 4) {
      x = csub_sign(x, 2 * q3);
      y = csub_sign(y, 2 * q3);
    }
    s = x + y;
    d = x - y + (B == 1 ? q3 : 2 * q3);
  }
  static constexpr int sum_bound(int b) { return b == 1 ? 2 : 4; }
  __device__ __forceinline__ static u64 sum(u64 s, const Tw&) { return s; }
  __device__ __forceinline__ static u64 mul(u64 d, u64 w, u64 wp, const Tw& t) {
    return shoup_lazy3(d, w, wp, 0 - t.q);
  }
  template <int B>
  __device__ __forceinline__ static u64 settle(u64 x, const Tw& t) {
    const u64 q3 = t.q + t.q2;
    if (B == 4) x = csub_sign(x, 2 * q3);
    if (B >= 2) x = csub_sign(x, q3);
    return x;
  }
  // A forward word (below 12q) below 2q: the quotient from its top 27 bits and
  // floor(2^(qbits + 4) / q), at most 32, is short by less than 1 (its floor)
  // + 0.75 (the 32's) + 2^-22 (the bits left out); all products fit 32 bits.
  struct Out {
    u64 q;
    u32 m, sh, sh2;
    __device__ __forceinline__ explicit Out(const Tw& t) : q(t.q) {
      const u32 bits = t.qbits();
      m = (u32)(t.mu() >> 58);
      sh = bits > 23 ? bits - 23 : 0;
      sh2 = bits + 4 - sh;
    }
    __device__ __forceinline__ u64 park(u64 x) const {
      const u32 k = ((u32)(x >> sh) * m) >> sh2;
      const u64 nq = 0 - q;
      const u64 r = mad_wide(k, lo32(nq), x);
      return pack(lo32(r), hi32(r) + k * hi32(nq));
    }
    __device__ __forceinline__ u64 canon(u64 x) const { return csub_sign(park(x), q); }
  };
  // x < 12q and y < 2q: (x y - ((x y) q^-1 mod 2^64) q) / 2^64 + q, below
  // 24 q q / 2^64 + q < 2.5q
  struct Product {
    u64 q, qinv;
    __device__ __forceinline__ explicit Product(const Tw& t) : q(t.q), qinv(t.qinv()) {}
    __device__ __forceinline__ u64 operator()(u64 x, u64 y) const {
      return mulhi_chain(x, y) - mulhi_chain(x * y * qinv, q) + q;
    }
  };
  __device__ __forceinline__ static u64 product_out(u64 x, u64 y, const Tw& t, u64 mu, u32 qbits) {
    return csub(barrett_mul_lazy(x, y, t.q, t.q2, mu, qbits), t.q);
  }
  // first-stage fast paths: the lazy butterfly is congruent to the reference's
  __device__ __forceinline__ static bool fwd_fast(u64 x, const Tw& t) { return x < t.q + t.q2; }
  __device__ __forceinline__ static bool inv_fast(u64 x, u64 y, const Tw& t) {
    return x < t.q + t.q2 && y < t.q + t.q2;
  }
  __device__ __forceinline__ static U2 ct_slow(u64 x, u64 y, u64 w, u64 wp, const Tw& t) {
    return ct_first_slow(x, y, w, wp, t.q, t.set);
  }
  __device__ __forceinline__ static U2 gs_slow(u64 x, u64 y, const Tw& t) { return gs_first_slow(x, y, t.q, t.set); }
};

struct Mod62 {
  static constexpr bool EXACT_AFTER_PRODUCT = false, MONTGOMERY = false;
  static constexpr bool reduce_at(int) { return true; }
  template <bool REDUCE>
  __device__ __forceinline__ static void ct(u64& x, u64& y, u64 w, u64 wp, const Tw& t) {
    ct_bfly(x, y, w, wp, t.q, t.q2);
  }
  template <int B>
  __device__ __forceinline__ static void sd(u64 x, u64 y, const Tw& t, u64& s, u64& d) {
    s = x + y;
    d = x - y + t.q2;
  }
  static constexpr int sum_bound(int) { return 1; }
  __device__ __forceinline__ static u64 sum(u64 s, const Tw& t) { return csub(s, t.q2); }
  __device__ __forceinline__ static u64 mul(u64 d, u64 w, u64 wp, const Tw& t) { return shoup_lazy(d, w, wp, t.q); }
  template <int B>
  __device__ __forceinline__ static u64 settle(u64 x, const Tw&) {
    return x;
  }
  struct Out {
    u64 q, q2;
    __device__ __forceinline__ explicit Out(const Tw& t) : q(t.q), q2(t.q2) {}
    __device__ __forceinline__ u64 canon(u64 x) const { return canon4(x, q, q2); }
    __device__ __forceinline__ u64 park(u64 x) const { return canon(x); }
  };
  struct Product {
    u64 q, q2, mu;
    u32 qbits;
    __device__ __forceinline__ explicit Product(const Tw& t) : q(t.q), q2(t.q2), mu(t.mu()), qbits(t.qbits()) {}
    __device__ __forceinline__ u64 operator()(u64 x, u64 y) const {
      return barrett_mul_lazy(canon4(x, q, q2), y, q, q2, mu, qbits);
    }
  };
  __device__ __forceinline__ static u64 product_out(u64 x, u64 y, const Tw& t, u64 mu, u32 qbits) {
    return csub(barrett_mul_lazy(x, y, t.q, t.q2, mu, qbits), t.q);
  }
  __device__ __forceinline__ static bool fwd_fast(u64 x, const Tw& t) { return x < t.q2; }
  __device__ __forceinline__ static bool inv_fast(u64 x, u64 y, const Tw& t) { return x < t.q2 && y < t.q2; }
  __device__ __forceinline__ static U2 ct_slow(u64 x, u64 y, u64 w, u64 wp, const Tw& t) {
    return ct_first_slow(x, y, w, wp, t.q, t.set);
  }
  __device__ __forceinline__ static U2 gs_slow(u64 x, u64 y, const Tw& t) { return gs_first_slow(x, y, t.q, t.set); }
};

struct Mod63 {
  static constexpr bool EXACT_AFTER_PRODUCT = true, MONTGOMERY = false;
  static constexpr bool reduce_at(int) { return true; }
  template <bool REDUCE>
  __device__ __forceinline__ static void ct(u64& x, u64& y, u64 w, u64 wp, const Tw& t) {
    const u64 xr = csub(x, t.q);
    const u64 wy = csub(shoup_lazy(y, w, wp, t.q), t.q);
    x = xr + wy;
    y = xr - wy + t.q;
  }
  template <int B>
  __device__ __forceinline__ static void sd(u64 x, u64 y, const Tw& t, u64& s, u64& d) {
    const u64 xr = csub(x, t.q), yr = csub(y, t.q);
    s = xr + yr;
    d = xr - yr + t.q;
  }
  static constexpr int sum_bound(int) { return 1; }
  __device__ __forceinline__ static u64 sum(u64 s, const Tw&) { return s; }
  __device__ __forceinline__ static u64 mul(u64 d, u64 w, u64 wp, const Tw& t) { return shoup_lazy(d, w, wp, t.q); }
  template <int B>
  __device__ __forceinline__ static u64 settle(u64 x, const Tw&) {
    return x;
  }
  struct Out {
    u64 q;
    __device__ __forceinline__ explicit Out(const Tw& t) : q(t.q) {}
    __device__ __forceinline__ u64 canon(u64 x) const { return csub(x, q); }
    __device__ __forceinline__ u64 park(u64 x) const { return csub(x, q); }
  };
  // the reference's elemmul on canonical operands (its reduce64 returns them
  // unchanged): the full 128-bit product through reduce128
  struct Product {
    u64 q, mu;
    u32 qbits;
    __device__ __forceinline__ explicit Product(const Tw& t) : q(t.q), mu(t.mu()), qbits(t.qbits()) {}
    __device__ __forceinline__ u64 operator()(u64 x, u64 y) const {
      const u64 xc = csub(x, q);
      return ref_reduce128(mulhi(xc, y), xc * y, q, mu, qbits);
    }
  };
  __device__ __forceinline__ static u64 product_out(u64 x, u64 y, const Tw& t, u64 mu, u32 qbits) {
    return ref_reduce128(mulhi(x, y), x * y, t.q, mu, qbits);
  }
  __device__ __forceinline__ static bool fwd_fast(u64 x, const Tw& t) { return x < t.q; }
  __device__ __forceinline__ static bool inv_fast(u64 x, u64 y, const Tw& t) { return x < t.q && y < t.q; }
  __device__ __forceinline__ static U2 ct_slow(u64 x, u64 y, u64 w, u64 wp, const Tw& t) {
    return ct_first_slow63(x, y, w, wp, t.q);
  }
  __device__ __forceinline__ static U2 gs_slow(u64 x, u64 y, const Tw& t) { return gs_first_slow63(x, y, t.q); }
};

// Forward, stage m = 1, with the reference's exact rule for inputs outside
// the fast path (x + WY could wrap past 2^64 there).
template <class M>
__device__ __forceinline__ void ct_first(u64& x, u64& y, u64 w, u64 wp, const Tw& t) {
  if (M::fwd_fast(x, t)) {
    M::template ct<false>(x, y, w, wp, t);
  } else {
    const U2 r = M::ct_slow(x, y, w, wp, t);
    x = r.x;
    y = r.y;
  }
}

// Inverse, stage m = n/2: s and d with the exact rule outside the fast path.
template <class M>
__device__ __forceinline__ void gs_first_sd(u64 x, u64 y, const Tw& t, u64& s, u64& d) {
  if (M::inv_fast(x, y, t)) {
    M::template sd<1>(x, y, t, s, d);
  } else {
    const U2 r = M::gs_slow(x, y, t);
    s = r.x;
    d = r.y;
  }
}

// ---------------------------------------------------------------------------
// Register-resident radix-2^KK groups.  A group holds 2^KK words v[G0 + j]
// at stride t_min of the transform, all inside one block of the first stage
// of the pass; tw(u, r) is the root (and Shoup factor) of sub-stage u and
// sub-block r.

// The roots of a pass before the last four stages: base = (tw_mult * m0 +
// block), root (base << u) + r.
struct RowTw {
  const ulonglong2* p;
  u32 base;
  __device__ __forceinline__ ulonglong2 operator()(int u, int r) const { return ld_tw(p + ((base << u) + r)); }
};

// The roots of the last four stages, from the table's rows (vkcu_tw_slot): a
// warp's 32 groups read 32 neighbouring entries, 4 wavefronts a load instead
// of up to 32.  N16 = n/16 for the whole transform, 0 where it is known at run
// time only.  A pass from the V-th of these stages on: p its group's column,
// x its block within the 16 words.
template <int N16, int V>
struct LastTw {
  const ulonglong2* p;
  u32 n16, x;
  __device__ __forceinline__ ulonglong2 operator()(int u, int r) const {
    return ld_tw(p + ((1u << (V + u)) + (V ? x << u : 0u) + (u32)r) * (N16 ? (u32)N16 : n16));
  }
};
// Those of a sub-block: at<V>(b) for block b (within it) of the V-th stage.
template <int N16>
struct LastTable {
  const ulonglong2* p;  // the sub-block's first column
  u32 n16;
  __device__ __forceinline__ LastTable(const ulonglong2* table, int first_group, u32 n16_)
      : p(table + first_group), n16(n16_) {}
  template <int V>
  __device__ __forceinline__ LastTw<N16, V> at(int b) const {
    return LastTw<N16, V>{p + (b >> V), n16, (u32)b & ((1u << V) - 1)};
  }
};
template <class M, int KK, int U0, int G0, int NV, class R>
__device__ __forceinline__ void ct_group(u64 (&v)[NV], const R& tw, const Tw& t) {
  static_for<U0, KK>([&](auto uc) {
    constexpr int u = decltype(uc)::value;
    constexpr int half = 1 << (KK - 1 - u);
    static_for<0, (1 << u)>([&](auto rc) {
      constexpr int r = decltype(rc)::value;
      const ulonglong2 w = tw(u, r);
#pragma unroll
      for (int jj = 0; jj < half; jj++)
        M::template ct<M::reduce_at(u)>(v[G0 + r * 2 * half + jj], v[G0 + r * 2 * half + jj + half], w.x, w.y, t);
    });
  });
}

// The same from sub-stage 0, with the exact rule there where EXACT.
template <class M, int KK, int G0, bool EXACT, int NV, class R>
__device__ __forceinline__ void ct_first_group(u64 (&v)[NV], const R& tw, const Tw& t) {
  if constexpr (EXACT) {
    const ulonglong2 w0 = tw(0, 0);
#pragma unroll
    for (int jj = 0; jj < (1 << (KK - 1)); jj++)
      ct_first<M>(v[G0 + jj], v[G0 + jj + (1 << (KK - 1))], w0.x, w0.y, t);
    ct_group<M, KK, 1, G0>(v, tw, t);
  } else {
    ct_group<M, KK, 0, G0>(v, tw, t);
  }
}

// Bound, in units, of word j of an inverse group of 2^KK words when sub-stage
// u begins: bit KK-1-s of j tells whether sub-stage s left it a sum or a
// twiddle product (below one unit); all words begin below one unit.
template <class M>
constexpr int gs_bound(int KK, int u, int j) {
  int b = 1;
  for (int s = KK - 1; s > u; s--) b = ((j >> (KK - 1 - s)) & 1) ? 1 : M::sum_bound(b);
  return b;
}

// Inverse group: sub-stages KK-1 .. 0, words below one unit before and after.
// EXACT_TOP applies the exact rule to sub-stage KK-1 (global stage m = n/2);
// FOLD folds n^-1 into sub-stage 0 (global stage m = 1, root index 1) and
// leaves canonical outputs.
//
// The exact rule looks at the group's words together: none reaches 2^qbits (at
// most 2q, below the fast path's bound) almost always, and then the first
// sub-stage runs like the others; a group with such a word takes it whole
// through the exact functions.  One test and branch a group instead of two
// compares and a branch a butterfly: 1024 inverse transforms of 2^14 160.0 ->
// 153.4 us, 150 of 2^15 with a lift 69.6 -> 66.0, 16 of 2^20 338 -> 315.  (The
// forward rule, one compare a butterfly, stays as it is: tested so, products
// of 2^16 lost 5 % and transforms gained or lost a few.)
template <class M, int KK, int G0, bool EXACT_TOP, bool FOLD, int NV, class R>
__device__ __forceinline__ void gs_group(u64 (&v)[NV], const R& tw, const Tw& t) {
  constexpr bool BY_GROUP = EXACT_TOP && !M::EXACT_AFTER_PRODUCT;  // (2^62 <= q: the bound is q itself)
  bool fast = true;
  if constexpr (BY_GROUP) {
    u64 any = 0;
#pragma unroll
    for (int j = 0; j < (1 << KK); j++) any |= v[G0 + j];
    fast = (any >> (64 - __clzll((long long)t.q))) == 0;
    if (!fast) {
#pragma unroll
      for (int j = 0; j < (1 << KK); j += 2) {
        const U2 r = M::gs_slow(v[G0 + j], v[G0 + j + 1], t);
        v[G0 + j] = r.x;
        v[G0 + j + 1] = r.y;
      }
    }
  }
  static_for<0, KK>([&](auto uc) {
    constexpr int u = KK - 1 - decltype(uc)::value;
    constexpr int half = 1 << (KK - 1 - u);
    // (both words of a butterfly have the same bound: they differ in a later bit)
    auto sums = [&](auto jc, u64& s, u64& d) {
      constexpr int j = decltype(jc)::value;
      if constexpr (BY_GROUP && u == KK - 1) {
        s = v[G0 + j];  // the exact sum and difference already, or
        d = v[G0 + j + half];
        if (fast) M::template sd<1>(s, d, t, s, d);
      } else if constexpr (EXACT_TOP && u == KK - 1) {
        gs_first_sd<M>(v[G0 + j], v[G0 + j + half], t, s, d);
      } else {
        M::template sd<gs_bound<M>(KK, u, j)>(v[G0 + j], v[G0 + j + half], t, s, d);
      }
    };
    if constexpr (FOLD && u == 0) {
      const ulonglong2 f0 = ld_late2(t.fold), f1 = ld_late2(t.fold + 1);
      static_for<0, half>([&](auto jc) {
        constexpr int j = decltype(jc)::value;
        u64 s, d;
        sums(jc, s, d);
        v[G0 + j] = shoup(s, f0.x, f0.y, t.q);
        v[G0 + j + half] = shoup(d, f1.x, f1.y, t.q);
      });
    } else {
      static_for<0, (1 << u)>([&](auto rc) {
        constexpr int r = decltype(rc)::value;
        const ulonglong2 w = tw(u, r);
        static_for<r * 2 * half, r * 2 * half + half>([&](auto jc) {
          constexpr int j = decltype(jc)::value;
          u64 s, d;
          sums(jc, s, d);
          s = M::sum(s, t);
          if constexpr (u == 0) s = M::template settle<M::sum_bound(gs_bound<M>(KK, 0, j))>(s, t);
          v[G0 + j] = s;
          v[G0 + j + half] = M::mul(d, w.x, w.y, t);
        });
      });
    }
  });
}

// ---------------------------------------------------------------------------
// Pass schedule for n = 2^LOGN held by T = n/E threads.  The first pass has
// FIRSTK <= 4 stages and reads global memory; every later pass has exactly 4
// stages (radix 16) and runs on shared memory; the last one starts at stage
// HEAD = LOGN - 4 and sees groups of 16 consecutive words.  Every pass but the
// first has t_min >= 16 or is the last pass.
//
// Code size matters as much as instruction count here: all radix-16 passes of
// a direction share one loop body (the stage offset is a runtime value), and
// the fused polymul runs its two forward transforms through the same code.

// R: stages of a pass (radix 2^R groups of W words).  4 everywhere but in the
// small sub-blocks of single calls, which run radix-4 passes with 4 words per
// thread: a radix-16 group is 32 butterflies one after another in one thread
// (about 1200 cycles of its SM sub-partition's multiplier), and with 16 words
// per thread a 2^9- or 2^10-word sub-block is one or two warps, so that half or
// more of the SM's four sub-partitions had nothing to do: one product of 2^12
// words 24.5 -> 19.5 us a call, of 2^13 26 -> 21.4, of 2^14 27.5 -> 24.4 (10 us
// of a call are its launch and wait).  With 16 warps the radix-16 passes win:
// 2^11-word sub-blocks, 25 products of 2^14 27 us against 37.
template <int LOGN_, int E_, int U_ = 1, class M_ = Mod60, bool DUAL_ = false, int R_ = 4>
struct Shape {
  using M = M_;  // modulus class
  static constexpr int R = R_, W = 1 << R_;
  // DUAL: the CTA holds 2 T threads running two transforms of this shape in
  // step, thread t on the one of half t / T (shared barriers, separate words)
  static constexpr bool DUAL = DUAL_;
  static constexpr int LOGN = LOGN_, E = E_;
  static constexpr int U = U_;  // groups of a thread in flight at once (1 or 2)
  static constexpr int N = 1 << LOGN, T = N / E;
  static constexpr int HEAD = LOGN - R;  // first stage of the last pass
  static constexpr int FIRSTK = HEAD % R == 0 ? R : HEAD % R;
  static constexpr int GROUPS = E >> R;  // of a thread in a pass
  static constexpr int SMEM_BYTES = (N + N / 16) * 8;
  static_assert((R == 4 || R == 2) && GROUPS >= 1 && (E % W) == 0 && HEAD >= FIRSTK + (R == 2 ? 2 : 0) && T >= 1,
                "unsupported shape");
  // this thread's index within its transform
  __device__ __forceinline__ static int tid() { return DUAL ? (int)(threadIdx.x & (T - 1)) : (int)threadIdx.x; }
  // its i-th group in the radix-16 passes: a warp's groups are consecutive, so
  // that a block of 2^k consecutive words belongs to 2^k / E consecutive
  // threads in every such pass
  __device__ __forceinline__ static int group(int i) {
    const int t = tid();
    return (t >> 5) * (32 * GROUPS) + (t & 31) + 32 * i;
  }
  // Barrier of the threads that share this thread's block of 2^lb words.  A
  // pass mixes words inside its blocks only, so a CTA-wide barrier is needed
  // around the first pass alone; from the 2^8-word blocks of the pass before
  // the last on it is one warp's, and for 2^13 and 2^14 words the pass between
  // synchronizes 2 or 4 parts of the CTA on their own.  Besides the barriers
  // saved, the warps of an SM drift apart, so that one's loads fall into
  // another's arithmetic (256 products of 2^14 words 137.3 -> 132.3 us, 1000
  // forward transforms 175.8 -> 165.9 us).
  __device__ __forceinline__ static void sync_block(int lb) {
    if ((1 << lb) <= 32 * E) {
      __syncwarp(T < 32 ? (1u << (T & 31)) - 1u : 0xffffffffu);
    } else {
      // parts of the CTA: barriers k .. 2k - 1 for k parts, so that no barrier
      // serves blocks of two sizes (15 is the last there is)
      static_assert(!DUAL || N <= 32 * E * 16, "a part of half a CTA");
      const int threads = (1 << lb) / E, parts = T / threads;
      if (parts == 1 || parts > 8)
        __syncthreads();
      else
        asm volatile("bar.sync %0, %1;" ::"r"(parts + tid() / threads), "r"(threads) : "memory");
    }
  }
};

// A radix-2^R pass starting at stage s0 of an n = 2^LOGN transform: group g
// has block g >> lt (lt = log2 t_min), first word (g >> lt) << lb | (g & mask)
// with lb = log2(n >> s0), words at stride t_min, twiddle base tw0 + block.
template <class S>
struct Pass {
  int lt, lb;
  u32 tw0;
  __device__ __forceinline__ Pass(int s0, u32 tw_mult)
      : lt(S::LOGN - s0 - S::R), lb(S::LOGN - s0), tw0(tw_mult << s0) {}
  __device__ __forceinline__ int first(int g) const { return ((g >> lt) << lb) | (g & ((1 << lt) - 1)); }
  __device__ __forceinline__ u32 base(int g) const { return tw0 + (u32)(g >> lt); }
};

// Groups of 2^KK words a thread handles at once in the passes that walk G
// such groups: 16 words per round (fewer leave too little independent work
// between the loads and the stores of a round; more spill).
template <int KK, int G>
constexpr int round_groups() {
  return (16 >> KK) < 1 ? 1 : (G < (16 >> KK) ? G : (16 >> KK));
}

// First forward pass: this thread's words come from global memory (coalesced)
// in rounds of 16 (all of a round's loads in flight at once; 32 words at once
// would spill), then FIRSTK stages per group, results to shared memory.
// EXACT: the first sub-stage uses the exact first-stage rule (not after the
// global passes of a large transform, whose words are forward-lazy already).
// The barrier that frees the shared words comes after the first round's loads
// and butterflies.
template <class S, bool EXACT = true>
__device__ __forceinline__ void fwd_first(u64* sm, const u64* __restrict__ in, const Tw& t, u32 tw_mult) {
  constexpr int KK = S::FIRSTK, G = S::E >> KK, TMIN = S::N >> KK;
  constexpr int GR = round_groups<KK, G>();
#pragma unroll 1
  for (int i0 = 0; i0 < G; i0 += GR) {
    u64 v[GR << KK];
#pragma unroll
    for (int i = 0; i < GR; i++)
#pragma unroll
      for (int j = 0; j < (1 << KK); j++)
        v[i * (1 << KK) + j] = ld_stream(in + S::tid() + (i0 + i) * S::T + j * TMIN);
    static_for<0, GR>([&](auto ic) {
      constexpr int i = decltype(ic)::value;
      ct_first_group<typename S::M, KK, i * (1 << KK), EXACT>(v, RowTw{t.fwd, tw_mult}, t);
    });
    if (i0 == 0) __syncthreads();  // everyone is done with what the shared words held
#pragma unroll
    for (int i = 0; i < GR; i++)
#pragma unroll
      for (int j = 0; j < (1 << KK); j++) sm[pad(S::tid() + (i0 + i) * S::T + j * TMIN)] = v[i * (1 << KK) + j];
  }
  __syncthreads();
}

// First forward pass on data already in shared memory (the sub-blocks of a
// cluster transform): groups of 2^FIRSTK words, twiddle base tw_mult.
template <class S>
__device__ __forceinline__ void fwd_first_smem(u64* sm, const Tw& t, u32 tw_mult) {
  constexpr int KK = S::FIRSTK, G = S::E >> KK, TMIN = S::N >> KK, GR = round_groups<KK, G>();
#pragma unroll 1
  for (int i0 = 0; i0 < G; i0 += GR) {
    const int g0 = S::tid() + i0 * S::T;
    u64 v[GR << KK];
#pragma unroll
    for (int i = 0; i < GR; i++)
#pragma unroll
      for (int j = 0; j < (1 << KK); j++) v[i * (1 << KK) + j] = sm[pad(g0 + i * S::T + j * TMIN)];
    static_for<0, GR>(
        [&](auto ic) { ct_group<typename S::M, KK, 0, decltype(ic)::value * (1 << KK)>(v, RowTw{t.fwd, tw_mult}, t); });
#pragma unroll
    for (int i = 0; i < GR; i++)
#pragma unroll
      for (int j = 0; j < (1 << KK); j++) sm[pad(g0 + i * S::T + j * TMIN)] = v[i * (1 << KK) + j];
  }
  __syncthreads();
}

// Forward passes s0 = FIRSTK, FIRSTK + R, ..., HEAD on shared memory.  The
// last pass hands each group (words W g .. W g + W - 1) to epi(g, v) instead
// of storing it back.  No barrier at the end.
template <class S, class Tws>
__device__ __forceinline__ void fwd_pass(u64* sm, const Tw& t, const Pass<S>& ps, const Tws& tws) {
  const int st = 1 << ps.lt;
#pragma unroll(S::U)
  for (int i = 0; i < S::GROUPS; i++) {
    const int g = S::group(i);
    const int a0 = ps.first(g);
    u64 v[S::W];
#pragma unroll
    for (int j = 0; j < S::W; j++) v[j] = sm[pad(a0 + j * st)];
    ct_group<typename S::M, S::R, 0, 0>(v, tws(g), t);
#pragma unroll
    for (int j = 0; j < S::W; j++) sm[pad(a0 + j * st)] = v[j];
  }
  S::sync_block(ps.lb);
}

template <class S, class L, class Epi>
__device__ __forceinline__ void fwd_passes(u64* sm, const Tw& t, u32 tw_mult, const L& last, Epi&& epi) {
  // radix 4: the pass before the last is one of the last four stages too
  constexpr int ROWS = S::R == 4 ? S::HEAD : S::HEAD - 2;
#pragma unroll 1
  for (int s0 = S::FIRSTK; s0 < ROWS; s0 += S::R) {
    const Pass<S> ps(s0, tw_mult);
    fwd_pass<S>(sm, t, ps, [&](int g) { return RowTw{t.fwd, ps.base(g)}; });
  }
  if constexpr (S::R == 2)
    fwd_pass<S>(sm, t, Pass<S>(ROWS, tw_mult), [&](int g) { return last.template at<0>(g >> 2); });
#pragma unroll(S::U)
  for (int i = 0; i < S::GROUPS; i++) {
    const int g = S::group(i);
    u64 v[S::W];
#pragma unroll
    for (int j = 0; j < S::W; j++) v[j] = sm[pad(S::W * g) + j];
    ct_group<typename S::M, S::R, 0, 0>(v, last.template at<4 - S::R>(g), t);
    epi(g, v);
  }
}

// Inverse passes s0 = HEAD - R, ..., FIRSTK on shared memory (the one at HEAD
// is the caller's), each preceded by a barrier of its blocks; no barrier at
// the end.
template <class S, class Tws>
__device__ __forceinline__ void inv_pass(u64* sm, const Tw& t, const Pass<S>& ps, const Tws& tws) {
  const int st = 1 << ps.lt;
  S::sync_block(ps.lb);
#pragma unroll(S::U)
  for (int i = 0; i < S::GROUPS; i++) {
    const int g = S::group(i);
    const int a0 = ps.first(g);
    u64 v[S::W];
#pragma unroll
    for (int j = 0; j < S::W; j++) v[j] = sm[pad(a0 + j * st)];
    gs_group<typename S::M, S::R, 0, false, false>(v, tws(g), t);
#pragma unroll
    for (int j = 0; j < S::W; j++) sm[pad(a0 + j * st)] = v[j];
  }
}

template <class S, class L>
__device__ __forceinline__ void inv_passes(u64* sm, const Tw& t, u32 tw_mult, const L& last_inv) {
  constexpr int ROWS = S::R == 4 ? S::HEAD : S::HEAD - 2;
  if constexpr (S::R == 2)
    inv_pass<S>(sm, t, Pass<S>(ROWS, tw_mult), [&](int g) { return last_inv.template at<0>(g >> 2); });
#pragma unroll 1
  for (int s0 = ROWS - S::R; s0 >= S::FIRSTK; s0 -= S::R) {
    const Pass<S> ps(s0, tw_mult);
    inv_pass<S>(sm, t, ps, [&](int g) { return RowTw{t.inv, ps.base(g)}; });
  }
}

// Last inverse pass of a cluster sub-block: stages FIRSTK-1 .. 0 in place in
// shared memory, words below one unit; a CTA barrier before it, none after.
template <class S>
__device__ __forceinline__ void inv_last_smem(u64* sm, const Tw& t, u32 tw_mult) {
  constexpr int KK = S::FIRSTK, G = S::E >> KK, TMIN = S::N >> KK, GR = round_groups<KK, G>();
#pragma unroll 1
  for (int i0 = 0; i0 < G; i0 += GR) {
    const int g0 = S::tid() + i0 * S::T;
    u64 v[GR << KK];
#pragma unroll
    for (int i = 0; i < GR; i++)
#pragma unroll
      for (int j = 0; j < (1 << KK); j++) v[i * (1 << KK) + j] = sm[pad(g0 + i * S::T + j * TMIN)];
    static_for<0, GR>(
        [&](auto ic) { gs_group<typename S::M, KK, decltype(ic)::value * (1 << KK), false, false>(v, RowTw{t.inv, tw_mult}, t); });
#pragma unroll
    for (int i = 0; i < GR; i++)
#pragma unroll
      for (int j = 0; j < (1 << KK); j++) sm[pad(g0 + i * S::T + j * TMIN)] = v[i * (1 << KK) + j];
  }
}

// Epilogue of the inverse transforms: the reference's centred-lift ops in
// order on each canonical output word (src/vector.c:342-386, 429-511), with
// the job's modulus resolved once per job for VKCU_LIFT_TABLE_Q steps.
struct LiftRun {
  const vkcu_lift* L;
  u64 bound[VKCU_MAX_LIFT], d[VKCU_MAX_LIFT];
  __device__ __forceinline__ LiftRun(const vkcu_lift* l, u64 q) : L(l) {
#pragma unroll
    for (int s = 0; s < VKCU_MAX_LIFT; s++) {
      const vkcu_lift_step& st = L->step[s];
      const bool tq = (st.kind & VKCU_LIFT_TABLE_Q) != 0;
      bound[s] = tq ? q >> 1 : st.bound;
      d[s] = tq && s < (int)L->count && (st.kind & 0xff) == VKCU_LIFT_GTSUB ? ref_reduce64(q, st.mod, st.mu, st.bits)
                                                                              : st.d;
    }
  }
  __device__ __forceinline__ u64 operator()(u64 x) const {
#pragma unroll
    for (int s = 0; s < VKCU_MAX_LIFT; s++) {
      if (s >= (int)L->count) break;
      const vkcu_lift_step& st = L->step[s];
      const u32 kind = st.kind & 0xff;
      if (kind == VKCU_LIFT_MODTWO)
        x = ref_modtwo(x, bound[s]);
      else if (kind == VKCU_LIFT_GTSUB)
        x = ref_gtsub(x, bound[s], d[s], st.mod, st.mu, st.bits);
      else
        x = ref_gtadd(x, bound[s], d[s]);
    }
    return x;
  }
  // K words through the steps together: one walk of the step list, K
  // independent chains.
  template <int K>
  __device__ __forceinline__ void apply(u64 (&v)[K]) const {
#pragma unroll
    for (int s = 0; s < VKCU_MAX_LIFT; s++) {
      if (s >= (int)L->count) break;
      const vkcu_lift_step& st = L->step[s];
      const u32 kind = st.kind & 0xff;
      if (kind == VKCU_LIFT_MODTWO) {
#pragma unroll
        for (int k = 0; k < K; k++) v[k] = ref_modtwo(v[k], bound[s]);
      } else if (kind == VKCU_LIFT_GTSUB) {
#pragma unroll
        for (int k = 0; k < K; k++) v[k] = ref_gtsub(v[k], bound[s], d[s], st.mod, st.mu, st.bits);
      } else {
#pragma unroll
        for (int k = 0; k < K; k++) v[k] = ref_gtadd(v[k], bound[s], d[s]);
      }
    }
  }
};

// The same inside the transforms, on the words a thread holds: one walk of the
// step list for K words (K independent chains, one branch per step), a step's
// constants resolved as it comes (once per K words), so that the code is one
// step's and not four.  With the steps unrolled word by word the inverse
// cluster kernel waited on instruction fetch (0.83 of 10.5 stall cycles per
// issue): 150 inverse transforms of 2^15 words with one step 77.4 -> 75.9 us.
struct LiftFold {
  const vkcu_lift* L;
  u64 q;
  __device__ __forceinline__ LiftFold(const vkcu_lift* l, u64 q_) : L(l), q(q_) {}
  template <int K>
  __device__ __forceinline__ void apply(u64 (&v)[K]) const {
#pragma unroll 1
    for (int s = 0; s < (int)L->count; s++) {
      const vkcu_lift_step& st = L->step[s];
      const bool tq = (st.kind & VKCU_LIFT_TABLE_Q) != 0;
      const u32 kind = st.kind & 0xff, bits = st.bits;
      const u64 bound = tq ? q >> 1 : st.bound, mod = st.mod, mu = st.mu;
      if (kind == VKCU_LIFT_MODTWO) {
#pragma unroll
        for (int k = 0; k < K; k++) v[k] = ref_modtwo(v[k], bound);
      } else if (kind == VKCU_LIFT_GTSUB) {
        const u64 d = tq ? ref_reduce64(q, mod, mu, bits) : st.d;
#pragma unroll
        for (int k = 0; k < K; k++) {  // ref_gtsub, without its branches
          const u64 r = ref_reduce64_chain(v[k], mod, mu, bits);
          const u64 z = r + mod - d, zr = z >= mod ? z - mod : z;
          v[k] = v[k] > bound ? zr : r;
        }
      } else {
        const u64 d = st.d;
#pragma unroll
        for (int k = 0; k < K; k++) v[k] = ref_gtadd(v[k], bound, d);
      }
    }
  }
};

struct NoLift {
  template <int K>
  __device__ __forceinline__ void apply(u64 (&)[K]) const {}
};

// Last inverse pass (stages FIRSTK-1 .. 0) from shared memory to `out`,
// coalesced, one group at a time (rounds of 16 words measured slower here).
// fold: whole transform, n^-1 folded into stage 0, canonical output;
// otherwise lazy [0, 2q).
template <class S, class Epi>
__device__ __forceinline__ void inv_last_epi(u64* sm, const Tw& t, u32 tw_mult, u64* __restrict__ out, bool fold,
                                             const Epi& epi) {
  constexpr int KK = S::FIRSTK, G = S::E >> KK, TMIN = S::N >> KK;
#pragma unroll 1
  for (int i = 0; i < G; i++) {
    const int g = S::tid() + i * S::T;
    u64 v[1 << KK];
#pragma unroll
    for (int j = 0; j < (1 << KK); j++) v[j] = sm[pad(g + j * TMIN)];
    if (fold)
      gs_group<typename S::M, KK, 0, false, true>(v, RowTw{t.inv, tw_mult}, t);
    else
      gs_group<typename S::M, KK, 0, false, false>(v, RowTw{t.inv, tw_mult}, t);
    epi.apply(v);
#pragma unroll
    for (int j = 0; j < (1 << KK); j++) out[g + j * TMIN] = v[j];
  }
}

// Last inverse pass to global memory; LIFT applies the epilogue (only where
// fold, i.e. this pass ends the transform).
template <class S, bool LIFT = false>
__device__ __forceinline__ void inv_last(u64* sm, const Tw& t, u32 tw_mult, u64* __restrict__ out, bool fold,
                                         const vkcu_lift* lift = nullptr) {
  if constexpr (LIFT)
    inv_last_epi<S>(sm, t, tw_mult, out, fold, LiftFold(lift, t.q));
  else
    inv_last_epi<S>(sm, t, tw_mult, out, fold, NoLift{});
}

// Register groups of K consecutive words <-> global memory (32-byte vectors).
template <int K>
__device__ __forceinline__ void load_group(u64 (&v)[K], const u64* p) {
#pragma unroll
  for (int h = 0; h < K / 4; h++) ld4(p + 4 * h, v[4 * h], v[4 * h + 1], v[4 * h + 2], v[4 * h + 3]);
}

template <int K>
__device__ __forceinline__ void store_group(const u64 (&v)[K], u64* p) {
#pragma unroll
  for (int h = 0; h < K / 4; h++) st4(p + 4 * h, v[4 * h], v[4 * h + 1], v[4 * h + 2], v[4 * h + 3]);
}

// The same for a warp's 32 neighbouring radix-16 groups (512 consecutive
// words), through the shared words of those groups, which the warp must be
// done with: a lane's 32-byte pieces of its own group lie 128 bytes from the
// next lane's, so that a load or store of them costs the LSU about 60
// wavefronts; 16-byte pairs over whole lines and a turn through shared memory
// cost 8 + 8.  g is the lane's group; `sync` runs before the words are written.
// Measured: inverse transforms of 2^11 .. 2^14 3-9 % faster with staged loads
// (1024 of 2^14 175.6 -> 160.0 us, 2048 of 2^13 167.5 -> 151.8; 2^10 even);
// forward ones 0.5-2 % to 2^13 and 4 % from 2^14 on with staged stores (1000 of
// 2^14 163.9 -> 157.6 us, 512 of 2^15 187.4 -> 179.8; storing after all groups
// instead of group by group made 2^14 2.4 % slower than unstaged).  A given
// NTT(b) is staged in the CTA products (480 of 2^14 182.6 -> 179.5 us) and not
// in the cluster ones (150 of 2^15 104.5 -> 106.4).
template <class S>
constexpr bool staged_loads() {
  return S::R == 4 && S::LOGN >= 11;
}
template <class S>
constexpr bool staged_stores() {
  return S::R == 4 && S::LOGN >= 9;  // whole warps
}

template <class S, class Sync>
__device__ __forceinline__ void load_group_staged(u64 (&v)[16], const u64* p, u64* sm, int g, Sync&& sync) {
  const int lane = (int)threadIdx.x & 31, w0 = (g - lane) * 16 + 2 * lane;
  ulonglong2 x[8];
#pragma unroll
  for (int k = 0; k < 8; k++)
    asm volatile("ld.global.L1::no_allocate.v2.u64 {%0,%1}, [%2];" : "=l"(x[k].x), "=l"(x[k].y) : "l"(p + w0 + 64 * k));
  sync();
#pragma unroll
  for (int k = 0; k < 8; k++) {
    sm[pad(w0 + 64 * k)] = x[k].x;
    sm[pad(w0 + 64 * k) + 1] = x[k].y;
  }
  __syncwarp();
#pragma unroll
  for (int j = 0; j < 16; j++) v[j] = sm[pad(16 * g) + j];
}

// (The warp is done with these words: every lane has read its own.)
__device__ __forceinline__ void store_group_staged(const u64 (&v)[16], u64* p, u64* sm, int g) {
#pragma unroll
  for (int j = 0; j < 16; j++) sm[pad(16 * g) + j] = v[j];
  __syncwarp();
  const int lane = (int)threadIdx.x & 31, w0 = (g - lane) * 16 + 2 * lane;
#pragma unroll
  for (int k = 0; k < 8; k++) {
    const int i = w0 + 64 * k;
    asm volatile("st.global.v2.u64 [%0], {%1,%2};" ::"l"(p + i), "l"(sm[pad(i)]), "l"(sm[pad(i) + 1]) : "memory");
  }
}

// NTT(b) parked between the phases of a fused product: 16-byte pairs, pair jj
// of group g (of G) at jj G + g, so that a warp moves whole lines (each thread
// reads back what it wrote).
template <int K>
__device__ __forceinline__ void park_group(const u64 (&v)[K], u64* p, int g, int G) {
#pragma unroll
  for (int jj = 0; jj < K / 2; jj++)
    asm volatile("st.global.v2.u64 [%0], {%1,%2};" ::"l"(p + 2 * (jj * G + g)), "l"(v[2 * jj]), "l"(v[2 * jj + 1])
                 : "memory");
}

template <int K>
__device__ __forceinline__ void unpark_group(u64 (&v)[K], const u64* p, int g, int G) {
#pragma unroll
  for (int jj = 0; jj < K / 2; jj++)
    asm volatile("ld.global.v2.u64 {%0,%1}, [%2];"
                 : "=l"(v[2 * jj]), "=l"(v[2 * jj + 1])
                 : "l"(p + 2 * (jj * G + g)));
}

// Resident CTAs per SM the register budget is sized for: 512 threads per SM
// (128 registers per thread, 16 warps) for the 32-words-per-thread shapes, the
// 16-words-per-thread transforms of n >= 2^12 and polymuls of n >= 2^12; 640
// threads (102 registers, 20 warps) for the 16-word transforms of 2^9 .. 2^11;
// 384 threads (about 170 registers) for the other 16-word shapes.  Measured:
// the 2^12 shapes at 384 took 222 registers (one CTA of 256 threads per SM),
// 128 made them 9 % (polymul) and 17 % (transforms) faster; 640 against 512
// makes the transforms of 2^9 .. 2^11 5-6 % faster (16384 forward ones of 2^10
// 114.6 -> 108.8 us, inverse 123.0 -> 116.9) but the polymuls slower wherever
// the jobs are few (2048 of 2^10 47.8 -> 52.9 us, 54.1 at 512), whose rounds
// then wait on one thread's chain; n = 2^8 (16-thread CTAs) spills above 384.
template <int LOGN, int E, bool POLY = false>
constexpr int min_blocks() {
  constexpr int budget = E >= 32                              ? 512
                         : !POLY && LOGN >= 9 && LOGN <= 11    ? 640
                         : LOGN >= 12                          ? 512
                                                               : 384;
  return (budget / ((1 << LOGN) / E)) < 1 ? 1 : (budget / ((1 << LOGN) / E));
}

template <class J>
__device__ __forceinline__ J fetch_job(const J* jobs, const J& one, int jid) {
  return jobs ? jobs[jid] : one;
}

// ---------------------------------------------------------------------------
// Kernels.  Jobs come from a device array (persistent loop over
// blockIdx.x, blockIdx.x + gridDim.x, ...) or, for a single job, by value.
// sub_log > 0: each job is split into 2^sub_log sub-blocks of 2^LOGN words
// (transforms of 2^(LOGN + sub_log) words after / before the global passes),
// sub-block `sub` using twiddle multiplier 2^sub_log + sub.

// SUB: sub_log may be above 0 (a template flag so that the others know their
// table's row length at compile time).
template <int LOGN, int E, int U, class M = Mod60, bool SUB = false>
__global__ void __launch_bounds__((1 << LOGN) / E, min_blocks<LOGN, E>())
    k_ntt_fwd(const vkcu_ntt_job* __restrict__ jobs, int njobs, vkcu_ntt_job one, int sub_log) {
  using S = Shape<LOGN, E, U, M>;
  extern __shared__ u64 sm[];
  if (!SUB) sub_log = 0;
  const int total = njobs << sub_log;
#pragma unroll 1
  for (int w = blockIdx.x; w < total; w += gridDim.x) {
    const vkcu_ntt_job job = fetch_job(jobs, one, w >> sub_log);
    const int sub = w & ((1 << sub_log) - 1);
    const Tw t = load_tw(job.tw);
    const LastTable<SUB ? 0 : S::N / 16> last(t.fwd, sub * (S::N / 16), (S::N / 16) << sub_log);
    u64* out = reinterpret_cast<u64*>(job.out) + ((size_t)sub << LOGN);
    const u64* in = sub_log ? out : reinterpret_cast<const u64*>(job.in);
    const u32 tw_mult = (1u << sub_log) + sub;
    // the next transform's words into L2 (1000 of 2^14 157.9 -> 156.2 us; even
    // at 2^13, and before the outputs left in whole lines 1 % slower)
    if (!SUB && LOGN == 14 && w + (int)gridDim.x < total && threadIdx.x < 4) {
      const vkcu_ntt_job nx = fetch_job(jobs, one, w + (int)gridDim.x);
      prefetch_l2(reinterpret_cast<const char*>(nx.in) + threadIdx.x * (S::N * 2), S::N * 2);
    }
    fwd_first<S, !SUB>(sm, in, t, tw_mult);
    fwd_passes<S>(sm, t, tw_mult, last, [&](int g, u64(&v)[16]) {
      const typename M::Out to(t);
#pragma unroll
      for (int j = 0; j < 16; j++) v[j] = to.canon(v[j]);
      if constexpr (staged_stores<S>())
        store_group_staged(v, out, sm, g);
      else
        store_group(v, out + 16 * g);
    });
  }
}

// LIFT: the epilogue `lift` follows the last stage (sub_log == 0 only).
template <int LOGN, int E, int U, bool LIFT = false, class M = Mod60, bool SUB = false>
__global__ void __launch_bounds__((1 << LOGN) / E, min_blocks<LOGN, E>())
    k_ntt_inv(const vkcu_ntt_job* __restrict__ jobs, int njobs, vkcu_ntt_job one, int sub_log,
              const __grid_constant__ vkcu_lift lift) {
  using S = Shape<LOGN, E, U, M>;
  extern __shared__ u64 sm[];
  if (!SUB) sub_log = 0;
  const int total = njobs << sub_log;
#pragma unroll 1
  for (int w = blockIdx.x; w < total; w += gridDim.x) {
    const vkcu_ntt_job job = fetch_job(jobs, one, w >> sub_log);
    const int sub = w & ((1 << sub_log) - 1);
    const Tw t = load_tw(job.tw);
    const LastTable<SUB ? 0 : S::N / 16> last(t.inv, sub * (S::N / 16), (S::N / 16) << sub_log);
    const u64* in = reinterpret_cast<const u64*>(job.in) + ((size_t)sub << LOGN);
    u64* out = reinterpret_cast<u64*>(job.out) + ((size_t)sub << LOGN);
    // the next work item's words into L2 while this one runs (2.6-3.4 % on
    // batched inverse transforms)
    if (w + (int)gridDim.x < total && threadIdx.x < 4) {
      const int w2 = w + (int)gridDim.x, sub2 = w2 & ((1 << sub_log) - 1);
      const vkcu_ntt_job nx = fetch_job(jobs, one, w2 >> sub_log);
      prefetch_l2(reinterpret_cast<const char*>(reinterpret_cast<const u64*>(nx.in) + ((size_t)sub2 << LOGN)) +
                      threadIdx.x * (S::N * 2),
                  S::N * 2);
    }
    const u32 tw_mult = (1u << sub_log) + sub;
    // first inverse pass (global stage m = n/2 first, exact rule) from global;
    // U groups in flight, as in the other passes
#pragma unroll(S::U)
    for (int i = 0; i < S::E / 16; i++) {
      const int g = S::group(i);
      u64 v[16];
      auto free_words = [&] {
        if (i == 0) __syncthreads();  // the last job's words are read
      };
      if constexpr (staged_loads<S>())
        load_group_staged<S>(v, in, sm, g, free_words);
      else
        load_group(v, in + 16 * g);
      gs_group<M, 4, 0, true, false>(v, last.template at<0>(g), t);
      if constexpr (!staged_loads<S>()) free_words();
#pragma unroll
      for (int j = 0; j < 16; j++) sm[pad(16 * g + j)] = v[j];
    }
    inv_passes<S>(sm, t, tw_mult, last);
    __syncthreads();
    inv_last<S, LIFT>(sm, t, tw_mult, out, sub_log == 0, &lift);
  }
}

// Fused c = INTT(NTT(a) . NTT(b)).  Phase 0 transforms b and parks NTT(b)
// in job.scratch; phase 1 transforms a with the same code, and its
// last pass multiplies by NTT(b) (read back at the words this thread wrote)
// and runs the first inverse pass on the products in the same registers; the
// rest of the inverse transform then writes c.  a is prefetched
// into L2 while b is transformed, the next job's b while a is.
template <int LOGN, int E, int U, bool LIFT = false, class M = Mod60>
__global__ void __launch_bounds__((1 << LOGN) / E, min_blocks<LOGN, E, true>())
    k_polymul(const vkcu_poly_job* __restrict__ jobs, int njobs, vkcu_poly_job one,
              const __grid_constant__ vkcu_lift lift) {
  using S = Shape<LOGN, E, U, M>;
  extern __shared__ u64 sm[];
  constexpr unsigned kChunk = (unsigned)(S::N * 8 / 4);
#pragma unroll 1
  for (int w = blockIdx.x; w < njobs; w += gridDim.x) {
    const vkcu_poly_job job = fetch_job(jobs, one, w);
    const Tw t = load_tw_product<M>(job.tw);
    // b holds NTT(b): phase 0 is skipped (read by the epilogue instantiations only)
    const bool b_ntt = LIFT && (job.flags & VKCU_JOB_B_NTT);
    u64* scratch = reinterpret_cast<u64*>(job.scratch);
    const LastTable<S::N / 16> last(t.fwd, 0, 0), last_inv(t.inv, 0, 0);
    if (threadIdx.x < 4) prefetch_l2(reinterpret_cast<const char*>(job.a) + threadIdx.x * kChunk, kChunk);
#pragma unroll 1
    for (int ph = b_ntt ? 1 : 0; ph < 2; ph++) {
      fwd_first<S>(sm, reinterpret_cast<const u64*>(ph ? job.a : job.b), t, 1u);
      if (ph == 1 && w + (int)gridDim.x < njobs && threadIdx.x < 4) {
        const vkcu_poly_job nx = fetch_job(jobs, one, w + (int)gridDim.x);
        prefetch_l2(reinterpret_cast<const char*>(nx.b) + threadIdx.x * kChunk, kChunk);
      }
      fwd_passes<S>(sm, t, 1u, last, [&](int g, u64(&v)[16]) {
        if (ph == 0) {
          const typename M::Out to(t);
#pragma unroll
          for (int j = 0; j < 16; j++) v[j] = to.park(v[j]);
          park_group(v, scratch, g, S::N / 16);
        } else {
          u64 bh[16];
          if (b_ntt) {
            if constexpr (staged_loads<S>())
              load_group_staged<S>(bh, reinterpret_cast<const u64*>(job.b), sm, g, [] { __syncwarp(); });
            else
              load_group(bh, reinterpret_cast<const u64*>(job.b) + 16 * g);
            reduce_operands(bh, t);
          } else {
            unpark_group(bh, scratch, g, S::N / 16);
          }
          const typename M::Product product(t);
#pragma unroll
          for (int j = 0; j < 16; j++) v[j] = product(v[j], bh[j]);
          // the first inverse pass (stages HEAD + 3 .. HEAD) on the same 16 words
          gs_group<M, 4, 0, M::EXACT_AFTER_PRODUCT, false>(v, last_inv.template at<0>(g), t);
#pragma unroll
          for (int j = 0; j < 16; j++) sm[pad(16 * g + j)] = v[j];
        }
      });
    }
    inv_passes<S>(sm, t, 1u, last_inv);
    __syncthreads();
    inv_last<S, LIFT>(sm, t, 1u, reinterpret_cast<u64*>(job.c), true, &lift);
  }
}

// ---------------------------------------------------------------------------
// Host side: per-family launchers (one translation unit each).

// M: Mod60 or Mod62 (Mod63 has launchers of its own below).
// variant: 0 = default shape, 1 = two radix-16 groups per thread in flight,
// 2 = the other words-per-thread shape (2^10..2^13 only); others -> 0.
template <class M>
int fwd_cta(cudaStream_t st, const vkcu_ntt_job* jobs, int njobs, const vkcu_ntt_job& one, int log_n, int sms,
            int variant);
template <class M>
int inv_cta(cudaStream_t st, const vkcu_ntt_job* jobs, int njobs, const vkcu_ntt_job& one, int log_n, int sms,
            int variant);
template <class M>
int poly_cta(cudaStream_t st, const vkcu_poly_job* jobs, int njobs, const vkcu_poly_job& one, int log_n, int sms,
             int variant);
// With an epilogue, one CTA per transform: the inverse in the default shape
// of each degree, the polymul in the variant given.
template <class M>
int inv_cta_lift(cudaStream_t st, const vkcu_ntt_job* jobs, int njobs, const vkcu_ntt_job& one, int log_n, int sms,
                 const vkcu_lift& lift);
template <class M>
int poly_cta_lift(cudaStream_t st, const vkcu_poly_job* jobs, int njobs, const vkcu_poly_job& one, int log_n, int sms,
                  int variant, const vkcu_lift& lift);
// cluster of 2^logc CTAs with sub-blocks of 2^logs words, n = 2^(logc + logs):
// logs = 14 for n = 2^15 .. 2^17, 9 .. 13 where few jobs are split further
// (VK_CLUSTER_SHAPES in ntt_cluster.cuh)
template <class M>
int fwd_cluster(cudaStream_t st, const vkcu_ntt_job* jobs, int njobs, const vkcu_ntt_job& one, int logc, int logs);
template <class M>
int inv_cluster(cudaStream_t st, const vkcu_ntt_job* jobs, int njobs, const vkcu_ntt_job& one, int logc, int logs,
                const vkcu_lift* lift = nullptr);
template <class M>
int poly_cluster(cudaStream_t st, const vkcu_poly_job* jobs, int njobs, const vkcu_poly_job& one, int logc, int logs,
                 const vkcu_lift* lift = nullptr);

// The 2^sub_log sub-blocks of 2^14 words of transforms past one cluster, each on
// one CTA, between their global passes (in place in out).
template <class M>
int fwd_cta_sub(cudaStream_t st, const vkcu_ntt_job* jobs, int njobs, const vkcu_ntt_job& one, int sub_log, int sms);
template <class M>
int inv_cta_sub(cudaStream_t st, const vkcu_ntt_job* jobs, int njobs, const vkcu_ntt_job& one, int sub_log, int sms);

// The sub-blocks of 2^(log_n - sub_log) words of transforms and products past
// one cluster, between their global passes (in place in out, or from c and
// scratch to c): 2^16 words on 4 CTAs, or 2^14 words on 8.
template <class M>
int fwd_cluster_sub(cudaStream_t st, const vkcu_ntt_job* jobs, int njobs, const vkcu_ntt_job& one, int log_n,
                    int sub_log);
template <class M>
int inv_cluster_sub(cudaStream_t st, const vkcu_ntt_job* jobs, int njobs, const vkcu_ntt_job& one, int log_n,
                    int sub_log);
template <class M>
int poly_cluster_sub(cudaStream_t st, const vkcu_poly_job* jobs, int njobs, const vkcu_poly_job& one, int log_n,
                     int sub_log);

// The same families for 2^62 <= q < 2^63 (Mod63), default shape of each
// degree, sub-blocks of 2^14 words for the cluster kernels (translation units
// ntt_wide_*.cu).
int fwd_cta_wide(cudaStream_t st, const vkcu_ntt_job* jobs, int njobs, const vkcu_ntt_job& one, int log_n,
                 int sub_log, int sms);
int inv_cta_wide(cudaStream_t st, const vkcu_ntt_job* jobs, int njobs, const vkcu_ntt_job& one, int log_n,
                 int sub_log, int sms, const vkcu_lift* lift);
int poly_cta_wide(cudaStream_t st, const vkcu_poly_job* jobs, int njobs, const vkcu_poly_job& one, int log_n, int sms,
                  const vkcu_lift* lift);
int fwd_cluster_wide(cudaStream_t st, const vkcu_ntt_job* jobs, int njobs, const vkcu_ntt_job& one, int logc);
int inv_cluster_wide(cudaStream_t st, const vkcu_ntt_job* jobs, int njobs, const vkcu_ntt_job& one, int logc,
                     const vkcu_lift* lift);
int poly_cluster_wide(cudaStream_t st, const vkcu_poly_job* jobs, int njobs, const vkcu_poly_job& one, int logc,
                      const vkcu_lift* lift);

// Launch set-up of one kernel, per device: the dynamic shared-memory opt-in
// and the occupancy figure its grid is sized from (resident blocks per SM,
// or resident clusters), both fixed for a kernel on a device, so they are
// computed once per device instead of on every launch (devices beyond 31
// recompute every time).
struct KernelSetup {
  std::atomic<int> per_dev[32];
};

__host__ inline int current_device() {
  int dev = 0;
  return cudaGetDevice(&dev) == cudaSuccess ? dev : -1;
}

// Opts `kernel` into `smem_limit` (default: `smem`) bytes of dynamic shared
// memory -- the attribute belongs to the kernel, so a kernel launched with
// several sizes is opted into the largest -- and returns its resident blocks
// per SM for `threads` threads and `smem` bytes (at least 1) in *per_sm.
template <class K>
static int setup_cta(K kernel, int threads, int smem, KernelSetup& ks, int* per_sm, int smem_limit = 0) {
  const int dev = current_device();
  const bool cached = dev >= 0 && dev < 32;
  if (cached) {
    const int v = ks.per_dev[dev].load(std::memory_order_acquire);
    if (v > 0) {
      *per_sm = v;
      return 0;
    }
  }
  const int e = (int)cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                          smem_limit > smem ? smem_limit : smem);
  if (e) return e;
  int b = 0;
  if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&b, kernel, threads, smem) != cudaSuccess || b < 1) b = 1;
  if (cached) ks.per_dev[dev].store(b, std::memory_order_release);
  *per_sm = b;
  return 0;
}

// A persistent grid: one wave of resident blocks, or fewer when there is less work.
__host__ inline int grid_from(int per_sm, long work, int sms) {
  const long cap = (long)per_sm * (sms > 0 ? sms : 1);
  return (int)(work < cap ? work : cap);
}

// One launch of the CTA-resident kernel `kern` of shape S over `work` work
// items (one-time set-up per kernel and device; grid = one wave of resident
// blocks, or fewer when there is less work).
template <class S, auto kern, class... Args>
static int launch_cta(cudaStream_t st, long work, int sms, Args... args) {
  static KernelSetup setup;
  int per_sm = 1;
  if (const int e = setup_cta(kern, S::T, S::SMEM_BYTES, setup, &per_sm)) return e;
  kern<<<grid_from(per_sm, work, sms), S::T, S::SMEM_BYTES, st>>>(args...);
  vkcu_count_launches(1);
  return (int)cudaGetLastError();
}

// Shapes per degree and variant: words per thread E and group unroll U.
#define VK_FOR_LOGN(X)                                                        \
  switch (log_n * 4 + (variant == 1 ? 1 : variant == 2 ? 2 : 0)) {            \
    case 8 * 4: return X(8, 16, 1);                                           \
    case 8 * 4 + 1: return X(8, 16, 2);                                       \
    case 9 * 4: return X(9, 16, 1);                                           \
    case 9 * 4 + 1: return X(9, 16, 2);                                       \
    case 10 * 4: return X(10, 16, 1);                                         \
    case 10 * 4 + 1: return X(10, 16, 2);                                     \
    case 10 * 4 + 2: return X(10, 32, 1);                                     \
    case 11 * 4: return X(11, 16, 1);                                         \
    case 11 * 4 + 1: return X(11, 16, 2);                                     \
    case 11 * 4 + 2: return X(11, 32, 1);                                     \
    case 12 * 4: return X(12, 16, 1);                                         \
    case 12 * 4 + 1: return X(12, 16, 2);                                     \
    case 12 * 4 + 2: return X(12, 32, 1);                                     \
    case 13 * 4: return X(13, 32, 1);                                         \
    case 13 * 4 + 1: return X(13, 32, 2);                                     \
    case 13 * 4 + 2: return X(13, 16, 1);                                     \
    case 14 * 4: return X(14, 32, 1);                                         \
    case 14 * 4 + 1: return X(14, 32, 2);                                     \
    default:                                                                  \
      if (variant != 0) { variant = 0; goto retry; }                          \
      return (int)cudaErrorInvalidValue;                                      \
  }

// Default shape of each degree (variant 0 above).
#define VK_FOR_LOGN_DEFAULT(X)                                                \
  switch (log_n) {                                                            \
    case 8: return X(8, 16, 1);                                               \
    case 9: return X(9, 16, 1);                                               \
    case 10: return X(10, 16, 1);                                             \
    case 11: return X(11, 16, 1);                                             \
    case 12: return X(12, 16, 1);                                             \
    case 13: return X(13, 32, 1);                                             \
    case 14: return X(14, 32, 1);                                             \
    default: return (int)cudaErrorInvalidValue;                               \
  }

}  // namespace vk
