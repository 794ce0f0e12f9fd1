// Device-side 64-bit modular arithmetic for the vkhel GB300 kernels.
//
// Two families live here:
//
//  * Reference-exact element-wise formulas.  The element-wise operations of the
//    reference are defined by their shader arithmetic, including a Barrett
//    reduction with alpha = 62, beta = -2 (include/priv/numbers.h:7-9,
//    src/kernels/shaders/elemmul.comp:36-60) and a Shoup product with a single
//    conditional subtraction (elemmulconst.comp:42-46).  Those are restated
//    here with the same constants so that every output, canonical or not,
//    equals the reference's for every 64-bit input.
//
//  * What lazy (Harvey) butterflies are made of.  Values travel a few multiples
//    of q above it, as far as 64 bits allow for the modulus class (ntt_core.cuh:
//    12q for q < 2^60, 4q for q < 2^62, 2q for q < 2^63), and are made canonical
//    once at the end, so a butterfly costs one Shoup product and no full
//    reduction.  Canonical outputs equal the reference's stage-by-stage canonical
//    arithmetic (nttfwdbutterfly.comp:44-57, nttrevbutterfly.comp:44-57) because
//    both are the same residues mod q.
#pragma once

#include <cstdint>

namespace vk {

typedef unsigned long long u64;
typedef unsigned int u32;

// ---- 64-bit products from 32-bit halves ------------------------------------
// The transforms are bound by the multiplier pipe, so how a 64-bit product is
// put together from 32x32 -> 64 bit products matters more than anything else
// in them.  A mad.lo.cc / madc.hi pair is one wide multiply-add that takes
// its 64-bit addend in the multiplier (4 issue cycles a warp on GB300, 16
// lanes wide), whereas a product written in C and added afterwards costs the
// same multiply and two adds more; and a difference x w - Q q written as
// x w + Q (-q) runs as one chain of such multiply-adds.  Register-only
// butterflies: 796 G/s with products and sums in C, 851 G/s so; the RNS
// batch of 256 products of 2^14 words 180 -> 168 us.
__device__ __forceinline__ u32 lo32(u64 x) { return (u32)x; }
__device__ __forceinline__ u32 hi32(u64 x) { return (u32)(x >> 32); }
__device__ __forceinline__ u64 pack(u32 l, u32 h) { return ((u64)h << 32) | l; }

// a * b + c mod 2^64 for 32-bit a, b.
__device__ __forceinline__ u64 mad_wide(u32 a, u32 b, u64 c) {
  u32 l, h;
  asm("mad.lo.cc.u32 %0, %2, %3, %4;\n\t"
      "madc.hi.u32 %1, %2, %3, %5;"
      : "=r"(l), "=r"(h)
      : "r"(a), "r"(b), "r"(lo32(c)), "r"(hi32(c)));
  return pack(l, h);
}

__device__ __forceinline__ u64 mulhi(u64 a, u64 b) { return __umul64hi(a, b); }

// floor(a b / 2^64) as one chain of wide multiply-adds, for the transforms.
// The element-wise formulas, bound by memory, keep the compiler's own high
// product (elemmul of 2^25 words: 125 us, 130 us with the chain), and so does
// the pointwise Barrett product of the fused kernels.
__device__ __forceinline__ u64 mulhi_chain(u64 a, u64 b) {
  u32 h0, h1;
  asm("{\n\t"
      ".reg .u32 t, m, c;\n\t"
      "mul.hi.u32 t, %2, %4;\n\t"
      "mad.lo.cc.u32 t, %3, %4, t;\n\t"
      "madc.hi.u32 m, %3, %4, 0;\n\t"
      "mad.lo.cc.u32 t, %2, %5, t;\n\t"
      "madc.hi.cc.u32 m, %2, %5, m;\n\t"
      "addc.u32 c, 0, 0;\n\t"
      "mad.lo.cc.u32 %0, %3, %5, m;\n\t"
      "madc.hi.u32 %1, %3, %5, c;\n\t"
      "}"
      : "=r"(h0), "=r"(h1)
      : "r"(lo32(a)), "r"(hi32(a)), "r"(lo32(b)), "r"(hi32(b)));
  return pack(h0, h1);
}

// floor(a b / 2^64) or one less, from three products: the low one, a0 b0, is
// left out.
__device__ __forceinline__ u64 mulhi_low1(u64 a, u64 b) {
  u32 h0, h1;
  asm("{\n\t"
      ".reg .u32 t, m, c;\n\t"
      "mul.lo.u32 t, %3, %4;\n\t"
      "mul.hi.u32 m, %3, %4;\n\t"
      "mad.lo.cc.u32 t, %2, %5, t;\n\t"
      "madc.hi.cc.u32 m, %2, %5, m;\n\t"
      "addc.u32 c, 0, 0;\n\t"
      "mad.lo.cc.u32 %0, %3, %5, m;\n\t"
      "madc.hi.u32 %1, %3, %5, c;\n\t"
      "}"
      : "=r"(h0), "=r"(h1)
      : "r"(lo32(a)), "r"(hi32(a)), "r"(lo32(b)), "r"(hi32(b)));
  return pack(h0, h1);
}

// a * b + c * d mod 2^64.
__device__ __forceinline__ u64 mad2_lo(u64 a, u64 b, u64 c, u64 d) {
  u64 r;
  asm("mul.wide.u32 %0, %1, %2;" : "=l"(r) : "r"(lo32(a)), "r"(lo32(b)));
  r = mad_wide(lo32(c), lo32(d), r);
  u32 h = hi32(r);
  h += lo32(a) * hi32(b);
  h += hi32(a) * lo32(b);
  h += lo32(c) * hi32(d);
  h += hi32(c) * lo32(d);
  return pack(lo32(r), h);
}

// x * w mod q in [0, 2q) for any 64-bit x, given w < q and wp = floor(w 2^64 / q).
__device__ __forceinline__ u64 shoup_lazy(u64 x, u64 w, u64 wp, u64 q) {
  return mad2_lo(x, w, mulhi_chain(x, wp), 0 - q);
}

// x * w mod q in [0, 3q) for any 64-bit x, with nq = -q: the quotient of
// mulhi_low1 is at most two short of x w / q, and x (w 2^64 - wp q) / 2^64 < q.
__device__ __forceinline__ u64 shoup_lazy3(u64 x, u64 w, u64 wp, u64 nq) {
  return mad2_lo(x, w, mulhi_low1(x, wp), nq);
}

// Same, with one conditional subtraction: canonical for any 64-bit x.
__device__ __forceinline__ u64 shoup(u64 x, u64 w, u64 wp, u64 q) {
  u64 r = shoup_lazy(x, w, wp, q);
  return r >= q ? r - q : r;
}

__device__ __forceinline__ u64 csub(u64 x, u64 m) { return x >= m ? x - m : x; }

// The same for x, m with |x - m| < 2^63, by the sign of the difference: two
// adds, a shift and two ands where a 64-bit compare takes the half-rate
// predicate and select path (about 7 issue cycles a warp against 9).
__device__ __forceinline__ u64 csub_sign(u64 x, u64 m) {
  const u64 d = x - m;
  const u32 s = (u32)((int)hi32(d) >> 31);
  return d + pack(lo32(m) & s, hi32(m) & s);
}

// [0, 4q) -> [0, q)
__device__ __forceinline__ u64 canon4(u64 x, u64 q, u64 q2) { return csub(csub(x, q2), q); }

// Cooley-Tukey butterfly on lazy values: X, Y in [0, 4q) -> [0, 4q).
__device__ __forceinline__ void ct_bfly(u64& x, u64& y, u64 w, u64 wp, u64 q, u64 q2) {
  const u64 xr = csub(x, q2);
  const u64 t = shoup_lazy(y, w, wp, q);
  x = xr + t;
  y = xr - t + q2;
}

// ---- reference-exact Barrett (alpha = 62, beta = -2) ----------------------
// n = bit length of mod (>= 2), mu = floor(2^(n+62) / mod).

// reduce64 (elemmul.comp:36-47): exact for every 64-bit x.
__device__ __forceinline__ u64 ref_reduce64(u64 x, u64 mod, u64 mu, u32 n) {
  const u64 qh = mulhi(x >> (n - 2), mu);
  const u64 z = x - qh * mod;
  return z >= mod ? z - mod : z;
}

// The same with the products as chains, for the epilogues inside the
// transforms (480 inverse transforms of 2^14 words with one step 106.4 -> 102.7
// us with these and no branches; the element-wise kernels are bound by memory).
__device__ __forceinline__ u64 ref_reduce64_chain(u64 x, u64 mod, u64 mu, u32 n) {
  const u64 qh = mulhi_chain(x >> (n - 2), mu), nm = 0 - mod;
  const u64 r = mad_wide(lo32(qh), lo32(nm), x);
  const u64 z = pack(lo32(r), hi32(r) + lo32(qh) * hi32(nm) + hi32(qh) * lo32(nm));
  return z >= mod ? z - mod : z;
}

// The same for operands that are usually reduced already.  For x < mod the
// estimate floor(k mu / 2^64), k = x >> (n - 2) <= 3, mu <= 2^63, is 0: it
// needs k mu >= 2^64, i.e. k = 2 with mod = 2^(n-1) (but x < mod gives
// k <= 1 then) or k = 3 with mod <= 3 2^(n-2) (but x < mod gives k <= 2
// then).  So reduce64 returns x there, the shortcut gives the same word for
// every 64-bit x, and canonical operands skip the multiplies (the branch is
// uniform across a warp of them).
__device__ __forceinline__ u64 ref_reduce64_maybe(u64 x, u64 mod, u64 mu, u32 n) {
  if (__builtin_expect(x < mod, 1)) return x;
  return ref_reduce64(x, mod, mu, n);
}

// reduce128 (elemmul.comp:49-60).  A shift by 64 (only for a 2-bit modulus,
// where the high word is zero) yields zero.
__device__ __forceinline__ u64 ref_reduce128(u64 hi, u64 lo, u64 mod, u64 mu, u32 n) {
  const u32 sh = 66u - n;
  const u64 top = sh >= 64u ? 0ull : (hi << sh);
  const u64 qh = mulhi(top + (lo >> (n - 2)), mu);
  const u64 z = lo - qh * mod;
  return z >= mod ? z - mod : z;
}

// Barrett product for the fused pointwise step: x, y in [0, q), q < 2^62,
// result in [0, 2q) (the estimate is at most two short for a 62-bit q, so one
// subtraction of 2q is applied when needed).
__device__ __forceinline__ u64 barrett_mul_lazy(u64 x, u64 y, u64 q, u64 q2, u64 mu, u32 n) {
  const u64 lo = x * y;
  const u64 hi = mulhi(x, y);
  const u64 qh = mulhi((hi << (66u - n)) | (lo >> (n - 2)), mu);
  return csub(lo - qh * q, q2);
}

// The reference's centred-lift element-wise ops on one word, as their
// shaders compute them (64-bit wrap included):
//   elemgtsub    src/kernels/shaders/elemgtsub.comp:49-67 (d = diff reduced mod `mod`)
//   elemgtadd    src/kernels/shaders/elemgtadd.comp:20-30
//   elemmodbytwo src/kernels/shaders/elemmodbytwo.comp:19-27 (sb = q / 2)
__device__ __forceinline__ u64 ref_gtsub(u64 a, u64 bound, u64 d, u64 mod, u64 mu, u32 bits) {
  const u64 r = ref_reduce64_maybe(a, mod, mu, bits);
  if (a > bound) {
    const u64 z = r + mod - d;
    return z >= mod ? z - mod : z;
  }
  return r;
}

__device__ __forceinline__ u64 ref_gtadd(u64 a, u64 bound, u64 diff) { return a > bound ? a + diff : a; }

__device__ __forceinline__ u64 ref_modtwo(u64 a, u64 sb) {
  const u64 bit = a & 1;
  return a > sb ? 1 - bit : bit;
}

}  // namespace vk
