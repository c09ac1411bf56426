// mgcd_device.cuh -- device arithmetic of the modular GCD kernels (sm_103a).
//
// Per-modulus arithmetic is done in Montgomery form with R = 2^32 (REDC), and modular
// inverses by the extended Euclidean algorithm with float-reciprocal quotient estimates.
// Every result is bit-exact: floats hold integers exactly or only choose a quotient, and
// every inverse is checked (x * x^-1 == 1) before it is used.
#pragma once
#include <cstdint>

namespace mgcd {

// Per-modulus constants, one 16-byte record per table entry.
//   q    : the prime modulus (table order = createModuli order, descending)
//   qinv : q^{-1} mod 2^32 (Montgomery)
//   r2   : 2^64 mod q
//   r1   : 2^32 mod q (the Montgomery form of 1)
struct __align__(16) ModConst {
  uint32_t q, qinv, r2, r1;
};

// State of one modulus during the reduction loop: t = u_q / v_q mod q, or a marker.
constexpr uint32_t T_INF = 0xFFFFFFFFu;      // v == 0 (mod q), u != 0
constexpr uint32_t T_DEGEN = 0xFFFFFFFEu;    // u == v == 0 (mod q): q divides both
constexpr uint32_t T_RETIRED = 0xFFFFFFFDu;  // q was used as a pivot
constexpr uint32_t T_MARK = T_RETIRED;       // t >= T_MARK: not a finite ratio
constexpr uint32_t U_RETIRED = 0xFFFFFFFFu;  // recovery: modulus consumed by a digit
constexpr int32_t MOD_INFINITY = INT32_MIN;  // reference MOD_INFINITY (GmpCudaDevice-getGcdKernel.cu:46)
constexpr uint32_t KEY_INF_HI = 0x80000000u; // |MOD_INFINITY| as the key's high word

// T * 2^-32 mod q for T < q * 2^32; result in [0, q).  With qinv = +q^{-1}, m q and T agree
// modulo 2^32, so (T - m q) / 2^32 is the difference of the high words, in (-q, q): no carry
// from the low words and no 33-bit sum.  What bounds it is the multiplier pipe: a product with
// its reduction takes 5.9 issue cycles per warp; the additive form (T + m q) took 10.3.
__device__ __forceinline__ uint32_t redc(uint64_t T, uint32_t q, uint32_t qinv)
{
  const uint32_t hi = (uint32_t)(T >> 32), mh = __umulhi((uint32_t)T * qinv, q);
  return hi - mh + (hi < mh ? q : 0u);
}

// The same without the canonical choice, for moduli below 2^30 (widths up to 30 bits): result
// in (0, 2q), congruent, for T < q * 2^32.  4q < 2^32, so products of two such values qualify.
__device__ __forceinline__ uint32_t redc_lazy(uint64_t T, uint32_t q, uint32_t qinv)
{
  return (uint32_t)(T >> 32) - __umulhi((uint32_t)T * qinv, q) + q;
}

// a * b * 2^-32 mod q, a, b < q.
__device__ __forceinline__ uint32_t mont_mul(uint32_t a, uint32_t b, uint32_t q, uint32_t qinv)
{
  return redc((uint64_t)a * b, q, qinv);
}

__device__ __forceinline__ uint32_t mod_sub(uint32_t a, uint32_t b, uint32_t q)
{
  return a - b + ((a < b) ? q : 0u);
}

// Symmetric residue with the reference's boundary (toSigned, GmpCudaDevice-getGcdKernel.cu:273-281):
// x >= q/2 maps to x - q.
__device__ __forceinline__ int32_t to_signed(uint32_t x, uint32_t q)
{
  return (x >= (q >> 1)) ? (int32_t)(x - q) : (int32_t)x;
}

// fromSigned (GmpCudaDevice-getGcdKernel.cu:264-271) for |x| < q.
__device__ __forceinline__ uint32_t from_signed(int32_t x, uint32_t q)
{
  return (uint32_t)x + ((x < 0) ? q : 0u);
}

__device__ __forceinline__ float rcp_approx(float y)
{
  float r;
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(y));
  return r;
}

// Exact inverse by integer-only extended Euclid; the fallback for the operands whose quotients
// the fast routine cannot hold (its self-check fails).  Cofactors as magnitudes (at most q),
// signs alternating.  Inline: a call here made the kernels keep their state in callee-saved
// registers.
__device__ __forceinline__ uint32_t inv_mod_slow(uint32_t x, uint32_t q)
{
  uint32_t r0 = q, r1 = x, s0 = 0u, s1 = 1u;
  bool neg = true;                                // sign of s0
#pragma unroll 1
  while (r1 != 0u) {
    const uint32_t Q = r0 / r1, r = r0 - Q * r1, s = s0 + Q * s1;
    r0 = r1; r1 = r;
    s0 = s1; s1 = s;
    neg = !neg;
  }
  return neg ? q - s0 : s0;
}

// Quotient estimate of the inverse's Euclid steps (also run by the certification kernel):
// Q = rint(f0 / f1), |Q| < 2^22, read from the mantissa of f0 * rcp(f1) + 1.5 * 2^23 as two's
// complement; inv_quot returns the float whose low mantissa bits hold Q.
constexpr float INV_MAGIC = 12582912.0f;     // 1.5 * 2^23
constexpr uint32_t INV_MAGIC_BITS = 0x4B400000u;
__device__ __forceinline__ float inv_quot(float f0, float f1)
{
  return __fmaf_rn(f0, rcp_approx(f1), INV_MAGIC);
}

// A step on integer remainders (with their floats, rounded) and one on float remainders
// (exact), the cofactors modulo 2^32; only where `on`.  The caller alternates the roles.
__device__ __forceinline__ void inv_step_int(uint32_t& r0, uint32_t r1, float& f0, float f1, uint32_t& s0, uint32_t s1,
                                             bool on)
{
  const uint32_t Q = __float_as_uint(inv_quot(f0, f1)) - INV_MAGIC_BITS;
  if (on) {
    r0 -= Q * r1;
    s0 -= Q * s1;
    f0 = __int2float_rn((int32_t)r0);
  }
}

__device__ __forceinline__ void inv_step(float& f0, float f1, uint32_t& s0, uint32_t s1, bool on)
{
  const float qm = inv_quot(f0, f1);
  if (on) {
    f0 = __fmaf_rn(INV_MAGIC - qm, f1, f0);
    s0 -= (__float_as_uint(qm) - INV_MAGIC_BITS) * s1;
  }
}

// s with s x == +-1 (mod q), as a signed value modulo 2^32, for 0 < x < q, q an odd prime:
// extended Euclid on (q, x) with nearest-integer quotients (remainders of either sign; about
// 13 steps for 32-bit operands, 10.7 for 27, 8.7 for 22), s_k x == r_k (mod q) throughout.
//   1. Until both remainders are below 2^23: integer remainders (the first two are unsigned,
//      every later one fits a signed word), quotients from their floats.  Operands rounded to
//      float and a reciprocal good to 1 ulp leave the quotient within 1/2 + 2^-22 Q of the
//      ratio, so the larger remainder shrinks in every step.
//   2. Below 2^23 remainders are exact in float: the quotient, and the remainder by one FMA.
// Quotients of 2^22 or more (a remainder that small against the other: about one inverse in
// 10^6 at 32 bits) are not held; the caller's check then fails.  Steps are predicated, two to
// a branch (UNROLL pairs in part 2): a lane that is done keeps its values.
// What bounds it: instruction issue (87 % of the issue slots in a full SM).  In a loop of
// dependent inverses, issue slots per warp inverse and latency in cycles: 271 and 1,136 at
// 32 bits, 218 and 890 at 27, 169 and 698 at 22; a version whose first part ran on the
// rounded operands alone (all float, the remainders rebuilt from the cofactors) took 287 and
// 1,407, 245 and 1,151, 163 and 804.
template <int UNROLL>
__device__ __forceinline__ uint32_t inv_euclid(uint32_t x, uint32_t q)
{
  constexpr float TOP = 8388608.0f;               // 2^23
  uint32_t r0 = q, r1 = x, s0 = 0u, s1 = 1u;
  float f0 = __uint2float_rn(q), f1 = __uint2float_rn(x);
  bool on = f0 >= TOP;
#pragma unroll 1
  while (on) {
    inv_step_int(r0, r1, f0, f1, s0, s1, true);
    on = fabsf(f1) >= TOP;
    inv_step_int(r1, r0, f1, f0, s1, s0, on);
    on = on && fabsf(f0) >= TOP;
  }
  on = fabsf(f0) > 1.0f && fabsf(f1) > 1.0f;
#pragma unroll 1
  while (on) {
#pragma unroll
    for (int u = 0; u < UNROLL; ++u) {
      inv_step(f0, f1, s0, s1, on);
      on = on && fabsf(f0) > 1.0f;
      inv_step(f1, f0, s1, s0, on);
      on = on && fabsf(f1) > 1.0f;
    }
  }
  const bool z = fabsf(f0) == 1.0f;
  const uint32_t s = z ? s0 : s1;
  return (z ? f0 : f1) < 0.0f ? 0u - s : s;       // s x == -1
}

// x^{-1} mod q for 0 < x < q, q an odd prime < 2^32 (inv_euclid).  |s| < q, so s is either
// the 32-bit value read as unsigned or that minus 2^32 (possible only for q > 2^31); the
// candidate whose product with x is 1 is taken, and if neither is, the integer-only routine
// recomputes it, so no float error can reach a result.
template <int UNROLL = 1>
__device__ __forceinline__ uint32_t inv_mod(uint32_t x, uint32_t q, uint32_t qinv)
{
  const uint32_t s = inv_euclid<UNROLL>(x, q);
  // inv * x == 1 (mod q)  <=>  redc(inv * x) == redc(1)
  const uint32_t one = redc(1ull, q, qinv);
  if (q < 0x80000000u) {
    const uint32_t inv = (int32_t)s < 0 ? s + q : s;
    if (redc((uint64_t)inv * x, q, qinv) == one) return inv;
  } else {
    // candidates s mod q and (s - 2^32) mod q = that - (2^32 - q); redc of the second's
    // product with x is the first's minus x
    const uint32_t inv = s >= q ? s - q : s;
    const uint32_t c = redc((uint64_t)inv * x, q, qinv);
    if (c == one) return inv;
    if (mod_sub(c, x, q) == one) return mod_sub(inv, 0u - q, q);
  }
  return inv_mod_slow(x, q);
}

// The same for q < 2^31, where s has one reading.
template <int UNROLL = 1>
__device__ __forceinline__ uint32_t inv_mod_narrow(uint32_t x, uint32_t q, uint32_t qinv)
{
  const uint32_t s = inv_euclid<UNROLL>(x, q);
  const uint32_t one = redc(1ull, q, qinv);
  const uint32_t inv = (int32_t)s < 0 ? s + q : s;
  if (redc((uint64_t)inv * x, q, qinv) == one) return inv;
  return inv_mod_slow(x, q);
}

// Register arrays indexed by a runtime slot number, without spilling them to memory.
template <int K, class V>
__device__ __forceinline__ V pick(const V (&a)[K], int s)
{
  V r = a[0];
#pragma unroll
  for (int t = 1; t < K; ++t)
    if (t == s) r = a[t];
  return r;
}

template <int K, class V>
__device__ __forceinline__ void put(V (&a)[K], int s, V v)
{
#pragma unroll
  for (int t = 0; t < K; ++t)
    if (t == s) a[t] = v;
}

// Key of the reduction loop's pivot choice (postMinPair, GmpCudaDevice-getGcdKernel.cu:152-154):
// high word |value| (0x80000000 for MOD_INFINITY), low word modulus - (value >= 0).
__device__ __forceinline__ void t_key(uint32_t t, uint32_t q, uint32_t& hi, uint32_t& lo)
{
  if (t >= T_MARK) { hi = KEY_INF_HI; lo = q; return; }
  const bool neg = t >= (q >> 1);
  hi = neg ? q - t : t;
  lo = neg ? q : q - 1u;
}

__device__ __forceinline__ bool key_less(uint32_t h1, uint32_t l1, uint32_t h2, uint32_t l2)
{
  return h1 < h2 || (h1 == h2 && l1 < l2);
}

// (p, b) from a key (collectMinPair, GmpCudaDevice-getGcdKernel.cu:214-219).
__device__ __forceinline__ void key_pair(uint32_t hi, uint32_t lo, uint32_t& p, int32_t& b)
{
  p = lo | 1u;
  b = (lo & 1u) ? (int32_t)(0u - hi) : (int32_t)hi;
}

// Lexicographic (hi, lo) minimum over the warp, result in every lane.
__device__ __forceinline__ void warp_min_key(uint32_t& hi, uint32_t& lo)
{
  const uint32_t mh = __reduce_min_sync(0xFFFFFFFFu, hi);
  const uint32_t ml = __reduce_min_sync(0xFFFFFFFFu, hi == mh ? lo : 0xFFFFFFFFu);
  hi = mh;
  lo = ml;
}

// One reduction-loop update of a modulus state t for pivot (p, b):
//   t' = p / (t - b)  (mod q)   since t' = u'/v' = v / ((u - b v)/p)
// with t = INF -> 0 (v was 0: u' = 0, v' = u/p), t == b -> INF (v' = 0), degenerate and
// retired states fixed; the pivot's own modulus retires.  The single pairs' update: its
// latency is on the chain of iterations, so p R is formed beside the inverse and the product
// with it beside the inverse's check (inv_mod's, with the same fallback); for q > 2^31 the
// second candidate is 2^32 - q = R mod q less, its product p R less.
// narrow: q < 2^31.  A pivot p < 2^32 enters the product as it is (p R^2 < q 2^32).
__device__ __forceinline__ uint32_t t_update(uint32_t t, const ModConst& c, uint32_t p, int32_t b, bool narrow)
{
  const uint32_t q = c.q, qinv = c.qinv;
  if (t >= T_MARK) return (t == T_INF) ? 0u : t;
  if (q == p) return T_RETIRED;
  const uint32_t d = mod_sub(t, from_signed(b, q), q);
  if (d == 0u) return T_INF;
  const uint32_t pR = mont_mul(p, c.r2, q, qinv), one = redc(1ull, q, qinv);
  const uint32_t s = inv_euclid<2>(d, q);
  if (narrow) {
    const uint32_t inv = (int32_t)s < 0 ? s + q : s;
    const uint32_t r = mont_mul(pR, inv, q, qinv);
    if (redc((uint64_t)inv * d, q, qinv) == one) return r;
  } else {
    const uint32_t inv = s >= q ? s - q : s;
    const uint32_t r = mont_mul(pR, inv, q, qinv), k = redc((uint64_t)inv * d, q, qinv);
    if (k == one) return r;
    if (mod_sub(k, d, q) == one) return mod_sub(r, pR, q);
  }
  return mont_mul(pR, inv_mod_slow(d, q), q, qinv);
}

// Moduli below 2^30 (widths up to 30 bits): products kept lazily in [0, 2q) where no
// comparison, key or inverse reads them.
__device__ __forceinline__ uint32_t mont_mul_lazy(uint32_t a, uint32_t b, uint32_t q, uint32_t qinv)
{
  return redc_lazy((uint64_t)a * b, q, qinv);
}

// Products of the K-slot update.
template <bool NARROW>
__device__ __forceinline__ uint32_t mul_k(uint32_t a, uint32_t b, uint32_t q, uint32_t qinv)
{
  return NARROW ? mont_mul_lazy(a, b, q, qinv) : mont_mul(a, b, q, qinv);
}

// [0, 2q) -> [0, q), 2q < 2^32: x - q wraps to a large value when x < q.
__device__ __forceinline__ uint32_t mod_canon(uint32_t x, uint32_t q)
{
  return min(x, x - q);
}

// (kh, kl) = the smaller of (kh, kl) and t's key (t_key), without a branch.
__device__ __forceinline__ void t_key_min(uint32_t t, uint32_t q, uint32_t& kh, uint32_t& kl)
{
  const bool neg = t >= (q >> 1);
  uint32_t h = neg ? q - t : t;
  if (t >= T_MARK) h = KEY_INF_HI;
  const uint32_t l = neg ? q : q - 1u;
  const bool less = (h < kh) | ((h == kh) & (l < kl));
  kh = less ? h : kh;
  kl = less ? l : kl;
}

// The update of t_update for K pairs (slots) that share the modulus q, slot s with pivot
// (p[s], b[s]).  `m` (uniform in the warp) has the slots with a live state in the warp's
// positions, and only theirs are read; lanes without a position hold T_RETIRED in them.
// Every lane of the warp calls it; out(s, t) takes each slot's new states, last slot first.
// The inverses are all mod q, so Montgomery's trick replaces them by one: with prefix products
// P_s of the slots' x_s = t_s - b_s and Z = R / (their product), walking back Z P_{s-1} / R =
// R / x_s (then t'_s = p_s / x_s) and Z <- Z x_s / R.  A lane whose slot needs no inverse
// contributes R mod q, the Montgomery one.
//
// What bounds it is instruction issue.  About half the (slot, warp) pairs have no live state
// (the positions are sorted by the set of slots live there), so whole warps skip a dead
// slot's loads, products and key; the rare new states (a pivot's own modulus retires, t = b
// gives INF, INF gives 0) are settled behind one vote, and keys are kept without a branch.
// 2,400 positions, four slots, half of them live, 1,024 threads: 12,485 -> 10,800 cycles
// against computing every slot in every warp, with the same inverse.
//   NARROW  moduli of at most NARROW_MAX_L bits.  Every modulus of a width-L table is an L-bit prime, so
//           |b| <= p / 2 < q puts t - b in (-q, 2q): one conditional add of q makes it lazy,
//           0 mod q exactly at 0 and q.  A pivot p < 2^32 enters a product as it is either
//           way (p y < q 2^32 for a canonical y; p < 2q, y < 2q when lazy).
template <int K, bool NARROW, class Out>
__device__ __forceinline__ void t_update_k(uint32_t (&t)[K], uint32_t m, const ModConst& c, const uint32_t (&p)[K],
                                           const int32_t (&b)[K], Out&& out)
{
  const uint32_t q = c.q, qinv = c.qinv;
  uint32_t x[K], P[K], prod = 0u;
  bool ok[K], odd = false;
#pragma unroll
  for (int s = 0; s < K; ++s) {
    if (!((m >> s) & 1u)) continue;
    uint32_t d;
    bool zero;
    if constexpr (NARROW) {
      const uint32_t dr = t[s] - (uint32_t)b[s];
      d = min(dr, dr + q);                        // dr < 0 wraps above 2^31; dr + q < 3q
      zero = (d == 0u) | (d == q);
    } else {
      d = mod_sub(t[s], from_signed(b[s], q), q);
      zero = d == 0u;
    }
    const bool fin = t[s] < T_MARK;
    ok[s] = fin & !zero & (q != p[s]);
    odd |= (fin & !ok[s]) | (t[s] == T_INF);
    x[s] = ok[s] ? d : c.r1;
    P[s] = prod;
    prod = (m & ((1u << s) - 1u)) ? mul_k<NARROW>(prod, x[s], q, qinv) : x[s];
  }
  uint32_t xr;                                    // prod / R, canonical: then 1 / xr = R / prod
  if constexpr (NARROW) xr = redc_lazy((uint64_t)prod, q, qinv);   // below 2^32: q - mh, in (0, q)
  else xr = redc((uint64_t)prod, q, qinv);
  uint32_t Z = NARROW ? inv_mod_narrow(xr, q, qinv) : inv_mod(xr, q, qinv);
  if (__any_sync(0xFFFFFFFFu, odd)) {
#pragma unroll
    for (int s = 0; s < K; ++s)
      if (((m >> s) & 1u) && !ok[s])
        t[s] = t[s] == T_INF ? 0u : t[s] >= T_MARK ? t[s] : q == p[s] ? T_RETIRED : T_INF;
  }
#pragma unroll
  for (int s = K - 1; s >= 0; --s) {
    if (!((m >> s) & 1u)) continue;
    uint32_t y = Z;
    if (m & ((1u << s) - 1u)) {
      y = mul_k<NARROW>(Z, P[s], q, qinv);
      Z = mul_k<NARROW>(Z, x[s], q, qinv);
    }
    uint32_t v = mul_k<NARROW>(p[s], y, q, qinv);
    if constexpr (NARROW) v = mod_canon(v, q);
    out(s, ok[s] ? v : t[s]);
  }
}

// Size bounds of the reduction loop, for certifying its result: lu >= log2|u_i| and
// lv >= log2|v_i| in fixed point (BOUND_ONE = 1 bit), stepped by
// |v_{i+1}| <= (|u_i| + |b| |v_i|) / p.  Integer arithmetic except for the logarithms
// (log2f, exp2f: within a few ulp, at most 2^-18 bits here), each rounded outward by
// BOUND_SLACK = 2^-17 bits, so the bounds stay upper bounds.
constexpr int BOUND_FRAC = 24;
constexpr long long BOUND_ONE = 1ll << BOUND_FRAC;
constexpr long long BOUND_SLACK = 1ll << (BOUND_FRAC - 17);

__device__ __forceinline__ long long bound_log2(float x)
{
  return (long long)(log2f(x) * (float)BOUND_ONE);
}

// Bit length of the operand limbs (an upper bound of log2 |x|) in bound units.
__device__ __forceinline__ long long bound_init(const uint32_t* limbs, uint32_t len)
{
  return (long long)(((int)len - 1) * 32 + (32 - __clz(limbs[len - 1]))) << BOUND_FRAC;
}

__device__ __forceinline__ void bound_step(long long& lu, long long& lv, uint32_t p, int32_t b)
{
  const uint32_t ab = b < 0 ? 0u - (uint32_t)b : (uint32_t)b;
  long long s = lu;                                 // log2(|u| + |b| |v|) <= s
  if (ab != 0u) {
    const long long y = lv + bound_log2((float)ab) + BOUND_SLACK;
    const long long m = y > lu ? y : lu, d = y > lu ? y - lu : lu - y;
    s = m + BOUND_SLACK;                            // log2(1 + 2^-d) < 2^-17 for d >= 40
    if (d < 40 * BOUND_ONE) s += bound_log2(1.0f + exp2f(-(float)d * (1.0f / (float)BOUND_ONE)));
  }
  lu = lv;
  lv = s - bound_log2((float)p) + BOUND_SLACK;
}

// Certified iff the surviving moduli (each > 2^(L-1)) multiply to more than |v| (so v = 0)
// and more than 2|u| (so the symmetric digits are exact).
__device__ __forceinline__ bool bound_certified(int remaining, int L, long long lu, long long lv)
{
  const long long cap = (long long)remaining * (L - 1) * BOUND_ONE;
  return cap > lu + 2 * BOUND_ONE && cap > lv + BOUND_ONE;
}

// Initial state t = u/v mod q from the residues.
__device__ __forceinline__ uint32_t t_init(uint32_t u, uint32_t v, uint32_t q, uint32_t qinv)
{
  if (v == 0u) return (u == 0u) ? T_DEGEN : T_INF;
  return mont_mul(u, inv_mod(redc((uint64_t)v, q, qinv), q, qinv), q, qinv);
}

}  // namespace mgcd
