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
// like the row sums do.
//
// Four lanes walk together (a walker): each prepares a quarter of the pairs (moves
// their state, forms the four values, hands them over through shared memory) and
// multiplies one code's chain over all pairs.  A lane's share of the state then fits
// in registers; one thread doing all four codes kept it in shared memory, 8 to 16
// warps per SM and 40 % of the issue slots.
//
// Fixed point: factor f in units 2^-fx_f, its largest possible sum (every digit
// included) below 2^62; a pair's K and E in units 2^(64 - fx_f - fx_g), below 2^61
// (a component of s_f s_g is below 2 * 2^62 * 2^62), with 16 bits more below them.  A
// value K +- E that comes out far below its largest possible size (2^-17 of it: a
// network's weakly coupled modes) has lost those bits, and is formed from the two
// factor sums instead (quad_small): every value handed to a chain is
// within 2^-55 of the pair's product.  (With K and E in 62 bits alone, 12 photons whose
// modes couple by 1e-4 and are doubly occupied at the output: 4.7e-9; now
// 3e-14.)  Haar matrices at 28 photons take the second way for a few values in 10^6; 64
// permanents of n = 22 7.0 ms, with two modes coupled by 1e-6 9.7, a Fourier matrix 9.7, 50:50
// splitters on all pairs of modes 8.8 (exact zeros), these coupled by 1e-9, where every value
// is small, 17.9.
//
// Layout of a sweep in the pool (longlong2 = one complex), slots = ceil(nf / 2)
// pairs (an odd last factor is paired with the constant 1 = 2^62 in its units),
// W = kQuadRow slots:
//   rows, one per outer digit: per pair u_f u_g e+ e-, packed (pack_row), and the e's
//     16 low bits (int4: e+ re im, e- re im); the walk adds -2 r times a row (r: the
//     digit's value);
//   base, W: o_f o_g E+ E- and the E's low parts per pair at r = 0 (unpacked);
//   constants, kQuadConst per pair: C+, C- - C+, their low parts (int4, 0 .. 2^16 - 1), and
//     u_f0 + u_f1, u_f0 - u_f1, u_g0 + u_g1, u_g0 - u_g1.
#pragma once
#include "boss_sweep.cuh"

namespace boss {

constexpr int kQuadLanes = 4;                            // lanes of a walker
constexpr int kQuadBlock = 128;                          // threads per block
constexpr int kQuadWalkers = kQuadBlock / kQuadLanes;    // walkers per block
constexpr long long kQuadOne = 1ll << 62;                // the constant factor, 62 fraction bits

constexpr int kQuadRow = 5;    // entries per pair of a row, of the base
constexpr int kQuadConst = 7;  // and of the constants
__host__ __device__ __forceinline__ int quad_slots(int nf) { return (nf + 1) >> 1; }
__host__ __device__ __forceinline__ int quad_width(int nf) { return kQuadRow * quad_slots(nf); }
// Entries of the base and the constants; of a quad sweep over ndo outer digits.
__host__ __device__ __forceinline__ int quad_base(int nf) { return quad_width(nf) + kQuadConst * quad_slots(nf); }
__host__ __device__ __forceinline__ int64_t quad_pool(int ndo, int nf) {
  return (int64_t)ndo * quad_width(nf) + quad_base(nf);
}

struct Cx64 {  // complex fixed point: re + fr 2^-16, im + fi 2^-16 (the low parts: of pairs' E and C only)
  long long re, im;
  int fr = 0, fi = 0;  // sums of at most 2^14 coefficients' 0 .. 2^16
};
__host__ __device__ __forceinline__ Cx64 cx(long long re, long long im) { return Cx64{re, im}; }
__host__ __device__ __forceinline__ Cx64 cx_add(Cx64 a, Cx64 b) {
  return Cx64{a.re + b.re, a.im + b.im, a.fr + b.fr, a.fi + b.fi};
}
__host__ __device__ __forceinline__ Cx64 cx_sub(Cx64 a, Cx64 b) {
  return Cx64{a.re - b.re, a.im - b.im, a.fr - b.fr, a.fi - b.fi};
}
__host__ __device__ __forceinline__ Cx64 cx_times(Cx64 v, int k) {
  return Cx64{v.re * k, v.im * k, v.fr * k, v.fi * k};
}
// Two complex low parts as one pool entry (int4 in memory).
__host__ __device__ __forceinline__ longlong2 quad_low(Cx64 a, Cx64 b) {
  longlong2 v;
  v.x = join32((unsigned)a.fi, (unsigned)a.fr);
  v.y = join32((unsigned)b.fi, (unsigned)b.fr);
  return v;
}

// v 2^-64 in 64 + 16 bits, rounded to nearest.
__host__ __device__ __forceinline__ int low16(I128 v) { return (int)(v.lo >> 48) + (int)((v.lo >> 47) & 1ull); }
__host__ __device__ __forceinline__ Cx64 quad_coef(Cx64 a, Cx64 b, Cx64 c, Cx64 d) {
  const I128 re = add128(sub128(mul_s64(a.re, b.re), mul_s64(a.im, b.im)),
                         sub128(mul_s64(c.re, d.re), mul_s64(c.im, d.im)));
  const I128 im = add128(add128(mul_s64(a.re, b.im), mul_s64(a.im, b.re)),
                         add128(mul_s64(c.re, d.im), mul_s64(c.im, d.re)));
  return Cx64{re.hi, im.hi, low16(re), low16(im)};
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

__host__ __device__ __forceinline__ Cx64 quad_carry(Cx64 v) {
  return Cx64{v.re + (v.fr >> 16), v.im + (v.fi >> 16), v.fr & 0xffff, v.fi & 0xffff};
}
// A pair's constants as they lie in the pool.
__host__ __device__ __forceinline__ void quad_constants(Cx64 f0, Cx64 f1, Cx64 g0, Cx64 g1, longlong2* out) {
  Cx64 v[6];
  quad_const(f0, f1, g0, g1, v[0], v[1]);
  v[0] = quad_carry(v[0]);
  v[1] = quad_carry(v[1]);
  out[2] = quad_low(v[0], v[1]);
  v[2] = cx_add(f0, f1);
  v[3] = cx_sub(f0, f1);
  v[4] = cx_add(g0, g1);
  v[5] = cx_sub(g0, g1);
  for (int c = 0; c < 6; ++c) {
    out[c < 2 ? c : c + 1].x = v[c].re;
    out[c < 2 ? c : c + 1].y = v[c].im;
  }
}

// 96-bit integers: w2 the highest word.
struct Q96 {
  unsigned w0, w1, w2;
};
__host__ __device__ __forceinline__ Q96 q96(long long hi, unsigned lo) { return Q96{lo, lo32(hi), hi32(hi)}; }
__host__ __device__ __forceinline__ Q96 q96_add(Q96 a, Q96 b) {
#ifdef __CUDA_ARCH__
  Q96 r;
  asm("add.cc.u32 %0, %3, %6;\n\taddc.cc.u32 %1, %4, %7;\n\taddc.u32 %2, %5, %8;"
      : "=r"(r.w0), "=r"(r.w1), "=r"(r.w2)
      : "r"(a.w0), "r"(a.w1), "r"(a.w2), "r"(b.w0), "r"(b.w1), "r"(b.w2));
  return r;
#else
  const unsigned lo = a.w0 + b.w0;
  return q96((long long)((unsigned long long)join32(a.w2, a.w1) + (unsigned long long)join32(b.w2, b.w1) + (lo < b.w0 ? 1u : 0u)), lo);
#endif
}
__host__ __device__ __forceinline__ Q96 q96_sub(Q96 a, Q96 b) {
#ifdef __CUDA_ARCH__
  Q96 r;
  asm("sub.cc.u32 %0, %3, %6;\n\tsubc.cc.u32 %1, %4, %7;\n\tsubc.u32 %2, %5, %8;"
      : "=r"(r.w0), "=r"(r.w1), "=r"(r.w2)
      : "r"(a.w0), "r"(a.w1), "r"(a.w2), "r"(b.w0), "r"(b.w1), "r"(b.w2));
  return r;
#else
  return q96((long long)((unsigned long long)join32(a.w2, a.w1) - (unsigned long long)join32(b.w2, b.w1) - (a.w0 < b.w0 ? 1u : 0u)), a.w0 - b.w0);
#endif
}
// hi + f 2^-16 in units 2^-32.
__host__ __device__ __forceinline__ Q96 q96_of(long long hi, int f) { return q96(hi + (f >> 16), (unsigned)f << 16); }
__host__ __device__ __forceinline__ int mulhi_s32(int a, int b) {
#ifdef __CUDA_ARCH__
  return __mulhi(a, b);
#else
  return (int)(((long long)a * (long long)b) >> 32);
#endif
}
// (x y) 2^-64 in units 2^-32, within 2 of them: bf_mul_high with the cross products'
// low words and the low products' high ones.
__host__ __device__ __forceinline__ void quad_product(Cx64 x, Cx64 y, Q96& re, Q96& im) {
  const Limbs a = limbs_of(x.re), b = limbs_of(x.im), c = limbs_of(y.re), d = limbs_of(y.im);
  const long long p = mad_wide(a.l, c.h, mad_wide(a.h, c.l, mulhi_s32(a.l, c.l)));
  const long long q = mad_wide(b.l, d.h, mad_wide(b.h, d.l, mulhi_s32(b.l, d.l)));
  const long long r = mad_wide(b.l, c.h, mad_wide(b.h, c.l, mad_wide(a.l, d.h, mad_wide(a.h, d.l,
                          (long long)mulhi_s32(a.l, d.l) + mulhi_s32(b.l, c.l)))));
  const long long t = p - q;
  re = q96(mad_wide(-b.h, d.h, mul_wide(a.h, c.h)) + (int)hi32(t), lo32(t));
  im = q96(mad_wide(b.h, c.h, mul_wide(a.h, d.h)) + (int)hi32(r), lo32(r));
}

// A value below 2^(32 + kQuadLeast) of its possible 2^61 is formed again (quad_small):
// above, the 16 low bits (off by a few units: the coefficients' roundings) leave it
// within 2^-55 (32 particles).
constexpr int kQuadLeast = 12;
// re, im in units 2^-32 normalised to 62 bits: (qr + i qi) 2^(l - 29), l the leading bit's
// position in the high word (below kQuadLeast: the value is not to be used).
__host__ __device__ __forceinline__ int quad_value(Q96 re, Q96 im, Cx64& q) {
  const int pr = lead_bit((int)re.w2), pi = lead_bit((int)im.w2);
  const int l = pr > pi ? pr : pi;
  const int s = 29 - l;  // 1 .. 30
  q = cx(join32(fshl32(re.w1, re.w2, s), fshl32(re.w0, re.w1, s)), join32(fshl32(im.w1, im.w2, s), fshl32(im.w0, im.w1, s)));
  return l;
}
// A pair's four values q, order (+,+), (-,-), (+,-), (-,+), each q 2^(l - 29), from of,
// og the outer sums, ep, em = E+-, cp, cm_cp the constants (low parts 0 .. 2^16 - 1,
// quad_carry).  Returns the smallest l.
__host__ __device__ __forceinline__ int quad_values(Cx64 of, Cx64 og, Cx64 ep, Cx64 em, Cx64 cp, Cx64 cm_cp, Cx64 (&q)[4],
                                                    int (&l)[4]) {
  Q96 pr, pi;
  quad_product(of, og, pr, pi);
  const Q96 kpr = q96_add(pr, q96(cp.re, (unsigned)cp.fr << 16)), kpi = q96_add(pi, q96(cp.im, (unsigned)cp.fi << 16));
  const Q96 kmr = q96_add(kpr, q96(cm_cp.re, (unsigned)cm_cp.fr << 16));
  const Q96 kmi = q96_add(kpi, q96(cm_cp.im, (unsigned)cm_cp.fi << 16));
  const Q96 epr = q96_of(ep.re, ep.fr), epi = q96_of(ep.im, ep.fi), emr = q96_of(em.re, em.fr), emi = q96_of(em.im, em.fi);
  l[0] = quad_value(q96_add(kpr, epr), q96_add(kpi, epi), q[0]);
  l[1] = quad_value(q96_sub(kpr, epr), q96_sub(kpi, epi), q[1]);
  l[2] = quad_value(q96_add(kmr, emr), q96_add(kmi, emi), q[2]);
  l[3] = quad_value(q96_sub(kmr, emr), q96_sub(kmi, emi), q[3]);
  const int x = l[0] < l[1] ? l[0] : l[1], y = l[2] < l[3] ? l[2] : l[3];
  return x < y ? x : y;
}
// A factor's sum normalised, also where its high word is empty, or the constant factor
// (2^62, one place too high); the exponent.
__host__ __device__ __forceinline__ int quad_normal(Cx64& s) {
  auto lead = [&] {
    const int pr = lead_bit((int)hi32(s.re)), pi = lead_bit((int)hi32(s.im));
    return pr > pi ? pr : pi;
  };
  auto up = [&] { s = cx((long long)((unsigned long long)s.re << 30), (long long)((unsigned long long)s.im << 30)); };
  int e = -29;
  const int p = lead();
  if ((unsigned)p > 29u) {  // rare
    if (p > 29) {
      s = cx(s.re >> 1, s.im >> 1);
      e += 1;
    } else {
      up();
      e -= 30;
      if (lead() < 0) {
        up();
        e -= 30;
      }
    }
  }
  return e + bf_renorm(s.re, s.im);
}
// Values 2 h and 2 h + 1 of a pair from its factors: the low digits' part is +-low_f,
// +-low_g, u_0 + u_1 for h = 0, u_0 - u_1 for h = 1.  Each within 2^-56 of the product.
__host__ __device__ __forceinline__ void quad_small(Cx64 of, Cx64 og, Cx64 low_f, Cx64 low_g, Cx64 (&q)[2], int (&l)[2]) {
  Cx64 f[2] = {cx_add(of, low_f), cx_sub(of, low_f)}, g[2] = {cx_add(og, low_g), cx_sub(og, low_g)};
  auto zero = [](Cx64 s) { return (s.re | s.im) == 0; };
  l[0] = l[1] = 0;
  q[0] = q[1] = cx(0, 0);
  if ((zero(f[0]) || zero(g[0])) && (zero(f[1]) || zero(g[1]))) return;
  for (int k = 0; k < 2; ++k) {
    l[k] = quad_normal(f[k]) + quad_normal(g[k]);
    bf_mul_high(f[k].re, f[k].im, g[k].re, g[k].im, q[k].re, q[k].im);
    l[k] += bf_renorm(q[k].re, q[k].im);  // the product 2^-64 = q 2^(l - 29)
  }
}
// The same four over one exponent, the largest l (returned), for a check of quad_values.
inline int quad_pair(Cx64 of, Cx64 og, Cx64 ep, Cx64 em, Cx64 cp, Cx64 cm_cp, Cx64 (&q)[4]) {
  int l[4], most = -1;
  quad_values(of, og, ep, em, quad_carry(cp), quad_carry(cm_cp), q, l);
  for (int k = 0; k < 4; ++k) most = l[k] > most ? l[k] : most;
  for (int k = 0; k < 4; ++k) q[k] = cx(q[k].re >> (most - l[k]), q[k].im >> (most - l[k]));
  return most;
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
// The same without the shift (which 29 stands for): the value stays above 2^58, and the
// next step, within 2^-54 of its product then, shifts.
__host__ __device__ __forceinline__ int quad_chain_raw(long long& re, long long& im, long long qr, long long qi) {
  bf_mul_high(re, im, qr, qi, re, im);
  return 29;
}
// Exponent of a chain beyond its own sum: e0 = minus the factors' fraction bits, 64
// per pair product and per chain product, the shifts (29 - l a slot, 29 - p a
// chain step) taken back; ls: the values' leading bits l.
__host__ __device__ __forceinline__ int quad_exponent(int e0, int ls, int slots) {
  return e0 + ls + 2 * (64 - 29) * slots - 64;
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
