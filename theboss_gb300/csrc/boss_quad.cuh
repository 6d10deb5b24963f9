// boss_quad.cuh -- four codes per step over pairs of factors.
//
// Two binary digits, the low ones, take all four sign combinations (d0, d1) at
// every step of the walk over the other (outer) digits.  With u = -D / 2 (Glynn:
// u = U, Ryser: u = -U / 2) a factor is s_f = o_f + d0 u_f0 + d1 u_f1, o_f the
// sum over the outer digits, and the product of two factors is
//     s_f s_g = K(d0 d1) + E(d0, d1),
//     K+- = o_f o_g + (u_f0 +- u_f1)(u_g0 +- u_g1)          (+: d0 = d1, -: d0 = -d1)
//     E+- = o_f (u_g0 +- u_g1) + o_g (u_f0 +- u_f1),
// so its four values are K+ + E+, K+ - E+, K- + E-, K- - E-: one product for four
// codes instead of four, and E+-, linear in the outer digits, walks by additions
// like the row sums do.  Per factor and code that leaves 9 instead of 15 holds of
// the FMA pipe (which bounds the sweeps: a 32 x 32 + 64-bit multiply-add holds it
// for 4 cycles a warp).
//
// Four lanes walk together (a walker): each prepares a quarter of the pairs (moves
// their state, forms the four values, hands them over through shared memory) and
// multiplies one code's chain over all pairs.  A lane's share of the state then fits
// in registers; one thread doing all four codes kept it in shared memory, 8 to 16
// warps per SM and 40 % of the issue slots (n = 20: 1.52 ms against 1.41).
//
// Fixed point: factor f in units 2^-fx_f, its largest possible sum (every digit
// included) below 2^62; a pair's K and E in units 2^(64 - fx_f - fx_g), below 2^61
// (a component of s_f s_g is below 2 * 2^62 * 2^62).  E's coefficients and C+- are
// rounded once from exact 128-bit products; o_f o_g is truncated (bf_mul_high).
//
// Layout of a sweep in the pool (longlong2 = one complex), slots = ceil(nf / 2)
// pairs (an odd last factor is paired with the constant 1 = 2^62 in its units),
// W = 4 slots:
//   rows, one per outer digit: per pair u_f u_g e+ e-, packed (pack_row); the walk
//     adds -2 r times a row (r: the digit's value);
//   base, W: o_f o_g E+ E- per pair at r = 0 (unpacked);
//   constants, 2 per pair: C+, C- - C+.
#pragma once
#include "boss_sweep.cuh"

namespace boss {

constexpr int kQuadLanes = 4;                            // lanes of a walker
constexpr int kQuadBlock = 128;                          // threads per block
constexpr int kQuadWalkers = kQuadBlock / kQuadLanes;    // walkers per block
constexpr long long kQuadOne = 1ll << 62;                // the constant factor, 62 fraction bits

__host__ __device__ __forceinline__ int quad_slots(int nf) { return (nf + 1) >> 1; }
__host__ __device__ __forceinline__ int quad_width(int nf) { return 4 * quad_slots(nf); }
// Pool entries of a quad sweep over ndo outer digits.
__host__ __device__ __forceinline__ int64_t quad_pool(int ndo, int nf) {
  return (int64_t)(ndo + 1) * quad_width(nf) + 2 * quad_slots(nf);
}

struct Cx64 {  // complex fixed point
  long long re, im;
};
__host__ __device__ __forceinline__ Cx64 cx(long long re, long long im) { return Cx64{re, im}; }
__host__ __device__ __forceinline__ Cx64 cx_add(Cx64 a, Cx64 b) { return Cx64{a.re + b.re, a.im + b.im}; }
__host__ __device__ __forceinline__ Cx64 cx_sub(Cx64 a, Cx64 b) { return Cx64{a.re - b.re, a.im - b.im}; }

// (a b + c d) 2^-64 rounded to nearest, from exact 128-bit sums.
__host__ __device__ __forceinline__ long long round_hi(I128 v) { return v.hi + (long long)(v.lo >> 63); }
__host__ __device__ __forceinline__ Cx64 quad_coef(Cx64 a, Cx64 b, Cx64 c, Cx64 d) {
  const I128 re = add128(sub128(mul_s64(a.re, b.re), mul_s64(a.im, b.im)),
                         sub128(mul_s64(c.re, d.re), mul_s64(c.im, d.im)));
  const I128 im = add128(add128(mul_s64(a.re, b.im), mul_s64(a.im, b.re)),
                         add128(mul_s64(c.re, d.im), mul_s64(c.im, d.re)));
  return cx(round_hi(re), round_hi(im));
}
// E+ and E- coefficients of one outer digit: uf, ug its entries; f0 f1 g0 g1 the low digits'.
__host__ __device__ __forceinline__ void quad_row(Cx64 uf, Cx64 ug, Cx64 f0, Cx64 f1, Cx64 g0, Cx64 g1, Cx64& ep,
                                                  Cx64& em) {
  ep = quad_coef(uf, cx_add(g0, g1), ug, cx_add(f0, f1));
  em = quad_coef(uf, cx_sub(g0, g1), ug, cx_sub(f0, f1));
}
// C+ and C- - C+.
__host__ __device__ __forceinline__ void quad_const(Cx64 f0, Cx64 f1, Cx64 g0, Cx64 g1, Cx64& cp, Cx64& cm_cp) {
  const Cx64 z = cx(0, 0);
  cp = quad_coef(cx_add(f0, f1), cx_add(g0, g1), z, z);
  cm_cp = cx_sub(quad_coef(cx_sub(f0, f1), cx_sub(g0, g1), z, z), cp);
}

__host__ __device__ __forceinline__ long long shl64(long long x, int s) {  // 0 <= s < 32
  return join32(fshl32(lo32(x), hi32(x), s), lo32(x) << (s & 31));
}

// The four values q, order (+,+), (-,-), (+,-), (-,+), from K+- and E+- (all below
// 2^61), which are normalised together first, so that no bit is left to the gap
// between the largest possible sum and the sums as they are.  Returns the leading
// bit's position, which quad_exponent takes back.
__host__ __device__ __forceinline__ int quad_values(Cx64 kp, Cx64 km, Cx64 ep, Cx64 em, Cx64 (&q)[4]) {
  const int l0 = lead_bit((int)hi32(kp.re)), l1 = lead_bit((int)hi32(kp.im));
  const int l2 = lead_bit((int)hi32(km.re)), l3 = lead_bit((int)hi32(km.im));
  const int l4 = lead_bit((int)hi32(ep.re)), l5 = lead_bit((int)hi32(ep.im));
  const int l6 = lead_bit((int)hi32(em.re)), l7 = lead_bit((int)hi32(em.im));
  auto mx = [](int a, int b) { return a > b ? a : b; };
  const int l = mx(mx(mx(l0, l1), mx(l2, l3)), mx(mx(l4, l5), mx(l6, l7)));
  const int s = 28 - l;  // 0 .. 29: components below 2^61, their sums below 2^62
  kp = cx(shl64(kp.re, s), shl64(kp.im, s));
  km = cx(shl64(km.re, s), shl64(km.im, s));
  ep = cx(shl64(ep.re, s), shl64(ep.im, s));
  em = cx(shl64(em.re, s), shl64(em.im, s));
  q[0] = cx_add(kp, ep);
  q[1] = cx_sub(kp, ep);
  q[2] = cx_add(km, em);
  q[3] = cx_sub(km, em);
  return l;
}
// A pair: of, og the outer sums, ep, em = E+-, cp, cm_cp the constants.
__host__ __device__ __forceinline__ int quad_pair(Cx64 of, Cx64 og, Cx64 ep, Cx64 em, Cx64 cp, Cx64 cm_cp,
                                                  Cx64 (&q)[4]) {
  Cx64 kp;
  bf_mul_high(of.re, of.im, og.re, og.im, kp.re, kp.im);
  kp = cx_add(kp, cp);
  return quad_values(kp, cx_add(kp, cm_cp), ep, em, q);
}
// One code's running product over the slots: a normal
// value (larger component in [2^61, 2^62], or zero); returns what its exponent
// grows by beyond quad_exponent's share.
__host__ __device__ __forceinline__ int quad_chain_first(long long& re, long long& im, long long qr, long long qi) {
  re = qr;
  im = qi;
  return bf_renorm(re, im);
}
__host__ __device__ __forceinline__ int quad_chain(long long& re, long long& im, long long qr, long long qi) {
  bf_mul_high(re, im, qr, qi, re, im);
  return bf_renorm(re, im);
}
// Exponent of a chain beyond its own sum: e0 = minus the factors' fraction bits, 64
// per pair product and per chain product, the shifts (28 - l a slot, 29 - p a
// chain step) taken back; ls: the slots' leading bits.
__host__ __device__ __forceinline__ int quad_exponent(int e0, int ls, int slots) {
  return e0 + ls + (64 - 28 + 64 - 29) * slots - 64;
}

// The walk over a sweep's (outer) digits: the reflected mixed-radix Gray code changes one
// digit by one per step, so the state moves by one row and is decoded only once.
struct QuadWalk {
  uint64_t g;      // the binary digits
  uint32_t parity; // sign parity
  double w;        // binomial weight of the multi-valued digits
  uint8_t r[kMaxDigits];  // their values (entries nb .. nd - 1; local memory)
};

// The walk at code t.
__device__ __forceinline__ void quad_walk_at(const SweepProblem& P, uint64_t t, QuadWalk& k) {
  const int nb = P.nb;
  k.g = (t ^ (t >> 1));
  if (nb < 64) k.g &= (1ull << nb) - 1ull;
  k.parity = (uint32_t)P.parity0 ^ ((uint32_t)__popcll((long long)k.g) & 1u);
  k.w = 1.0;
  uint64_t th = t >> nb;
  for (int i = nb; i < P.nd; ++i) {
    const uint32_t mu = P.mult[i];
    const uint64_t b = (uint64_t)mu + 1ull, q = th / b;
    const uint32_t dgt = (uint32_t)(th - q * b);
    th = q;
    const uint32_t r = (q & 1ull) ? (mu - dgt) : dgt;
    k.r[i] = (uint8_t)r;
    k.parity ^= r & 1u;
    if (r) k.w *= binom_small((int)mu, (int)r);
  }
}

// The step to code t: the digit that moves, and by how much (+-1).
__device__ __forceinline__ int quad_next(const SweepProblem& P, uint64_t t, QuadWalk& k, int& dr) {
  const int nb = P.nb;
  int i = __ffsll((long long)t) - 1;
  k.parity ^= 1u;
  if (i < nb) {
    dr = ((k.g >> i) & 1ull) ? -1 : 1;
    k.g ^= 1ull << i;
    return i;
  }
  uint64_t th = t >> nb, q;
  uint32_t mu, dgt;
  for (i = nb;; ++i) {  // the lowest digit whose plain value is not back at zero
    mu = P.mult[i];
    q = th / (mu + 1ull);
    dgt = (uint32_t)(th - q * (mu + 1ull));
    if (dgt || i + 1 >= P.nd) break;
    th = q;
  }
  const int r = (int)((q & 1ull) ? (mu - dgt) : dgt), before = k.r[i];
  dr = r - before;
  k.r[i] = (uint8_t)r;
  // C(mu, r) from C(mu, before), exact while the weight is below 2^53
  k.w = dr > 0 ? k.w * (double)(mu - (uint32_t)before) / (double)r : k.w * (double)before / (double)(mu - (uint32_t)r);
  return i;
}

// This lane's walker and its range; lanes past the launch's last walker take the
// last one's problem with an empty range, so that whole warps stay together.
struct QuadRange {
  int64_t q;       // the walker within its sweep
  int64_t a, len;  // its outer codes
  int64_t most;    // the longest range in the warp
  bool live;
};
__device__ __forceinline__ QuadRange quad_range(const SweepProblem& P, int64_t walker, bool live) {
  QuadRange r;
  r.live = live;
  r.q = walker - P.thread_begin;
  thread_range_aligned(P, r.q, P.align, r.a, r.len);
  if (!live) r.len = 0;
  r.most = r.len;
#pragma unroll
  for (int o = 16; o >= 4; o >>= 1) {
    const int64_t x = __shfl_xor_sync(0xffffffffu, r.most, o);
    r.most = x > r.most ? x : r.most;
  }
  return r;
}

}  // namespace boss
