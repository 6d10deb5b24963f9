// boss_sweep.cuh -- device-side building blocks of the permanent sweeps.
//
// Every permanent in theboss's hot path is a signed, binomially weighted sum over
// the codes r of a reflected mixed-radix Gray ("Guan") code of a product of
// row sums:
//     sum_r  sign(r) * prod_i C(mult_i, r_i) * prod_f s_f(r),
//     s_f(r) = base_f + sum_i r_i * D_if
// where i runs over the iterated side's distinct modes ("digits", multiplicity
// mult_i, r_i in [0, mult_i]) and f over the product side's particles ("factors":
// a mode occupied p times contributes p identical factors, which is theboss's
// pow(sum, p)):
//   * Ryser (ryser_permanent_calculator.py:45-64): base = 0, D = U,
//     sign (-1)^(n + |r|);
//   * Glynn / Chin-Huh (chin_huh_permanent_calculator.py:38-59,
//     glynn_gray_permanent_calculator.py:41-84): base_f = sum_i mult_i U_if,
//     D = -2U, sign (-1)^|r|, scale 2^-n.
// The binomial weight follows bs_permanent_calculator_base.py:151-164.
//
// GB300 mapping.  The FP64 pipe issues 2 lanes/clk/SM, 1/64 of FP32, so only
// sums over codes use it, and the integer pipes take everything else:
//   * the row sums are exact 64-bit fixed-point integers (value = int * 2^-fx_f,
//     every factor in its own scale), so they never drift;
//   * the products are formed in block floating point on the integer pipe (62-bit
//     mantissas, accumulate_product_bf), rounded to FP64 once per code;
//   * sign flips are integer XORs on the sign bit.
//
// Work split: the codes of a sweep are cut into one contiguous range per thread
// (lengths differ by at most one), each thread decodes its start code in closed
// form and walks the Gray code: step t flips binary digit ctz(t); when ctz(t)
// reaches a multi-valued digit the thread re-decodes.  Binary digits are ordered
// first so that happens once per 2^nb codes.
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

namespace boss {

constexpr int kMaxDigits = 64;       // distinct modes on the iterated side
constexpr int kMaxFactors = 32;      // particles on the product side
constexpr int kMaxMinorDigits = 32;  // digits of an all-minors sweep
constexpr int kSegLog = 16;          // all-minors bookkeeping is settled every 2^16 codes

enum SweepKind : int32_t { kRyser = 0, kGlynn = 1 };

// One sweep (a permanent or an all-minors problem).  Plain old data in device
// memory; built by the host planner or by the sampler's device-side planner.
struct SweepProblem {
  int32_t nd;        // digits walked, binary ones first (without the `low` ones)
  int32_t nb;        // leading binary digits
  int32_t nf;        // product factors
  int32_t kind;      // SweepKind
  int32_t parity0;   // sign parity of the r = 0 code
  int32_t fx;        // minus the sum of the factors' fraction bits (every factor has its own scale 2^fx_f)
  int32_t has_base;  // base sums present
  int32_t out_idx;   // result index
  int64_t n_codes;       // codes in the sweep (low = 2: steps of four codes)
  int64_t thread_begin;  // first global thread of this sweep
  int64_t n_threads;     // threads working on it
  int64_t mat_off;   // rows, nd x nf fixed-point complex (longlong2): D, or -D / 2 packed (pack_row) for the FP64
                     // permanent and all-minors sweeps; low = 2: the layout of boss_quad.cuh
  int64_t base_off;  // nf fixed-point complex
  int64_t part_off;  // partials: n_threads complex (perms) or n_threads x (nd + low + fixed_digit) (all-minors)
  int64_t ff_off;    // float-pair all-minors only: nb x nf rows of D as float pairs (float4: re hi, re lo,
                     // im hi, im lo, each factor in its own scale), then nf int32 exponent biases
  double scale;      // final real scale
  int16_t fixed_digit;  // gradients, all-minors: a binary digit held at r = 0 (Glynn halving) adds a weight-1 row
  int16_t group;     // each aligned group of `group` threads (all-minors: 1, 2, 4, .., 128; above 32 only when the
                     // launch's threads fill whole blocks; low = 2: walkers, permanents up to 8, all-minors up
                     // to 32; the templated permanents 1) sums its partials, so there are n_threads / group of
                     // them; n_threads and thread_begin are multiples of it, and every sweep of the launch has
                     // the same
  int16_t align;     // permanents, all-minors: ranges start at multiples of 2^align codes (range_align)
  int16_t low;       // 2: two more binary digits, all four of whose values are taken at every step (boss_quad.cuh)
  uint8_t mult[kMaxDigits];
};
static_assert(sizeof(SweepProblem) == 168, "the allocation-free entry point's scratch holds one a permanent");

// A row entry of the integer-pipe sweeps (permanents, all-minors): u = -D / 2, the
// 64-bit value hi 2^32 + lo with lo taken as a SIGNED word (hi carries its sign
// bit), so that adding sg times it (sg = +-2 for a flip, -2 r for a digit's value)
// is one 32 x 32 + 64-bit multiply-add and one 32-bit one per component, without
// exclusive-ors for the sign.
__host__ __device__ __forceinline__ long long pack_row(long long v) {
  return (long long)((unsigned long long)v + (((unsigned long long)v & 0x80000000ull) << 1));
}
__host__ __device__ __forceinline__ long long unpack_row(long long v) {
  return (long long)((unsigned long long)v - (((unsigned long long)v & 0x80000000ull) << 1));
}

// ---------------------------------------------------------------------------
// Integer-pipe helpers
// ---------------------------------------------------------------------------
__device__ __forceinline__ double xor_sign(double x, uint32_t neg_mask) {
  return __hiloint2double(__double2hiint(x) ^ (int)neg_mask, __double2loint(x));
}

// Compiler-only barrier: keeps the scheduler from hoisting all of a row's loads
// at once (at large NF that alone would exhaust the register file).
__device__ __forceinline__ void load_fence() { asm volatile("" ::: "memory"); }

__device__ __forceinline__ double binom_small(int n, int k) {
  double r = 1.0;
  for (int i = 1; i <= k; ++i) r = r * (double)(n - k + i) / (double)i;
  return r;
}

// Digit value of code t: digit i is the plain mixed-radix digit d_i when the
// number of completed cycles of digits 0..i is even, mult_i - d_i when odd (the
// closed form of the reflected mixed-radix code); binary digits reduce to
// bit_i(t) ^ bit_(i+1)(t).
__device__ __forceinline__ uint32_t digit_value(const SweepProblem& P, uint64_t t, int i) {
  if (i < P.nb) return (uint32_t)(((t >> i) ^ (t >> (i + 1))) & 1ull);
  uint64_t th = t >> P.nb;
  uint32_t r = 0;
  for (int j = P.nb; j <= i; ++j) {
    const uint32_t mu = P.mult[j];
    const uint64_t b = (uint64_t)mu + 1ull;
    const uint64_t q = th / b;
    const uint32_t dgt = (uint32_t)(th - q * b);
    th = q;
    r = (q & 1ull) ? (mu - dgt) : dgt;
  }
  return r;
}

// a b and a b + c, 32 x 32 -> 64 bits signed: one instruction each.  (Written as
// 64-bit C products of sign-extended words the compiler expanded part of them to
// full 64 x 64-bit products: 64 instead of 45 instructions per factor.)
__host__ __device__ __forceinline__ long long mul_wide(int a, int b) {
#ifdef __CUDA_ARCH__
  long long r;
  asm("mul.wide.s32 %0, %1, %2;" : "=l"(r) : "r"(a), "r"(b));
  return r;
#else
  return (long long)a * (long long)b;
#endif
}
__host__ __device__ __forceinline__ long long mad_wide(int a, int b, long long c) {
#ifdef __CUDA_ARCH__
  long long r;
  asm("mad.wide.s32 %0, %1, %2, %3;" : "=l"(r) : "r"(a), "r"(b), "l"(c));
  return r;
#else
  return (long long)((unsigned long long)((long long)a * (long long)b) + (unsigned long long)c);
#endif
}

// acc + sg * d for a packed row component d (pack_row), sg a small integer.
__device__ __forceinline__ long long add_packed(long long acc, long long d, int sg) {
  const int lo = (int)(unsigned)(unsigned long long)d, hi = (int)((unsigned long long)d >> 32);
  const unsigned long long t = (unsigned long long)mad_wide(lo, sg, acc);
  const unsigned th = (unsigned)(t >> 32) + (unsigned)hi * (unsigned)sg;
  return (long long)(((unsigned long long)th << 32) | (unsigned)t);
}

// Full state at code t: fixed-point sums, sign parity, binomial weight of the
// multi-valued digits, and the bits of the binary digits.  kPacked: the rows are
// packed (pack_row), as the integer-pipe sweeps take them.
template <int NF, bool kPacked = false>
__device__ __forceinline__ void decode_code(const SweepProblem& P, const longlong2* __restrict__ D,
                                            const longlong2* __restrict__ base, uint64_t t, long long (&sr)[NF],
                                            long long (&si)[NF], uint64_t& gbits, uint32_t& parity, double& weight) {
#pragma unroll
  for (int f = 0; f < NF; ++f) {
    if (P.has_base) {
      const longlong2 b = base[f];
      sr[f] = b.x;
      si[f] = b.y;
    } else {
      sr[f] = 0;
      si[f] = 0;
    }
  }
  parity = (uint32_t)P.parity0;
  weight = 1.0;
  gbits = (t ^ (t >> 1));
  if (P.nb < 64) gbits &= (1ull << P.nb) - 1ull;
  uint64_t bits = gbits;
  while (bits) {
    const int i = __ffsll((long long)bits) - 1;
    bits &= bits - 1ull;
    parity ^= 1u;
    const longlong2* row = D + (size_t)i * NF;
#pragma unroll
    for (int f = 0; f < NF; ++f) {
      if (f > 0 && (f & 7) == 0) load_fence();
      const longlong2 d = row[f];
      sr[f] = kPacked ? add_packed(sr[f], d.x, -2) : sr[f] + d.x;
      si[f] = kPacked ? add_packed(si[f], d.y, -2) : si[f] + d.y;
    }
  }
  uint64_t th = t >> P.nb;
  for (int i = P.nb; i < P.nd; ++i) {
    const uint32_t mu = P.mult[i];
    const uint64_t b = (uint64_t)mu + 1ull;
    const uint64_t q = th / b;
    const uint32_t dgt = (uint32_t)(th - q * b);
    th = q;
    const uint32_t r = (q & 1ull) ? (mu - dgt) : dgt;
    if (r) {
      parity ^= (r & 1u);
      weight *= binom_small((int)mu, (int)r);
      const longlong2* row = D + (size_t)i * NF;
#pragma unroll
      for (int f = 0; f < NF; ++f) {
        const longlong2 d = row[f];
        sr[f] = kPacked ? add_packed(sr[f], d.x, -2 * (int)r) : sr[f] + (long long)r * d.x;
        si[f] = kPacked ? add_packed(si[f], d.y, -2 * (int)r) : si[f] + (long long)r * d.y;
      }
    }
  }
}

// Binary digit i moves from `bit` to 1 - bit: sums +/-= D_i (packed rows).
template <int NF>
__device__ __forceinline__ void flip_packed(const longlong2* __restrict__ D, int i, uint32_t bit, long long (&sr)[NF],
                                            long long (&si)[NF]) {
  const longlong2* row = D + (size_t)i * NF;
  const int sg = 4 * (int)bit - 2;  // r 0 -> 1 adds D = -2 u
#pragma unroll
  for (int f = 0; f < NF; ++f) {
    if (f > 0 && (f & 7) == 0) load_fence();
    const longlong2 d = row[f];
    sr[f] = add_packed(sr[f], d.x, sg);
    si[f] = add_packed(si[f], d.y, sg);
  }
}

// ---------------------------------------------------------------------------
// 128-bit integer helpers for the exact products of two fixed-point factors.
// ---------------------------------------------------------------------------
struct I128 {
  unsigned long long lo;
  long long hi;
};
// High half of the signed 128-bit product (floor(a b / 2^64)); a host build uses __int128.
__host__ __device__ __forceinline__ long long mulhi_s64(long long a, long long b) {
#ifdef __CUDA_ARCH__
  return __mul64hi(a, b);
#else
  return (long long)(((__int128)a * (__int128)b) >> 64);
#endif
}
__host__ __device__ __forceinline__ int clz_u64(unsigned long long x) {
#ifdef __CUDA_ARCH__
  return __clzll((long long)x);
#else
  return x ? __builtin_clzll(x) : 64;
#endif
}
__host__ __device__ __forceinline__ I128 mul_s64(long long a, long long b) {
  I128 r;
  r.lo = (unsigned long long)a * (unsigned long long)b;
  r.hi = mulhi_s64(a, b);
  return r;
}
__host__ __device__ __forceinline__ I128 add128(I128 x, I128 y) {
  I128 r;
  r.lo = x.lo + y.lo;
  r.hi = x.hi + y.hi + (r.lo < x.lo ? 1 : 0);
  return r;
}
__host__ __device__ __forceinline__ I128 sub128(I128 x, I128 y) {
  I128 r;
  r.lo = x.lo - y.lo;
  r.hi = x.hi - y.hi - (x.lo < y.lo ? 1 : 0);
  return r;
}
// ---------------------------------------------------------------------------
// Block floating point on the integer pipe.  A complex value is (re + i im) 2^e,
// two 64-bit integers sharing one exponent, normalised so that the larger
// component lies in [2^61, 2^62].  GB300 issues the 32 x 32 + 64-bit multiply-add
// on its FMA pipe and shifts and adds on its ALU pipe, both far faster than its
// FP64 pipe (2 lanes/clk/SM), so whole products are formed without it:
//   * bf_mul: the high half of the product from two signed 32-bit limbs per
//     component, 12 multiply-adds (4 high x high, 8 cross; low x low, below half
//     a unit, is dropped), then one normalising shift.  Of two normal values
//     |product| >= 2^122 before the >> 64, off by less than 2 units a component:
//     relative error below 2^-56.5 of the product's magnitude;
//   * so every factor, a fixed-point sum below 2^62 in its own scale, is normalised
//     before it is multiplied: as it is, the error would be relative to its largest
//     possible sum, and a factor far below that (weakly coupled modes) lose its digits;
//   * bf_to_double: one rounding to FP64 (2^-53) at the end.
//   * in a chain only every second product is shifted back to the normal form: the one
//     between stays above 2^58, and the next is within 2^-54 of its magnitude.
// An FP64 complex product errs by up to about 2^-52 of its magnitude.
// Measured, sweeps of 64 permanents (input-side digits, 2^(n-1) codes each) with the
// templated kernel: n = 20 1.94 ms, n = 24 37.0 (the factors as they are, losing digits: 1.71
// and 33.5); whole calls 2.31 and 37.5 ms (with every product shifted 2.39 and 40.0).
// ---------------------------------------------------------------------------
struct BFloat {
  long long re, im;
  int e;
};
__host__ __device__ __forceinline__ double bits_to_double(unsigned long long b) {
#ifdef __CUDA_ARCH__
  return __longlong_as_double((long long)b);
#else
  double d;
  __builtin_memcpy(&d, &b, sizeof d);
  return d;
#endif
}
// (re + i im) 2^e normalised, for |re|, |im| <= 2^62.  The shift comes from the
// leading bit of the one's-complement magnitudes (|x| or |x| - 1), so a negative
// power of two may land on -2^62; zero stays zero (its exponent drops by 62).
__host__ __device__ __forceinline__ BFloat bf_norm(long long re, long long im, int e) {
  const unsigned long long m = (unsigned long long)(re ^ (re >> 63)) | (unsigned long long)(im ^ (im >> 63));
  const int s = clz_u64(m) - 2;  // >= 0
  BFloat r;
  r.re = (long long)((unsigned long long)re << s);
  r.im = (long long)((unsigned long long)im << s);
  r.e = e - s;
  return r;
}
__host__ __device__ __forceinline__ int clz_u32(unsigned x) {
#ifdef __CUDA_ARCH__
  return __clz((int)x);
#else
  return x ? __builtin_clz(x) : 32;
#endif
}
// Bits [s, s + 32) of (hi, lo) for 0 <= s < 32 (and the left-shift form).
__host__ __device__ __forceinline__ unsigned fshr32(unsigned lo, unsigned hi, int s) {
#ifdef __CUDA_ARCH__
  return __funnelshift_r(lo, hi, s);
#else
  return (unsigned)((((unsigned long long)hi << 32) | lo) >> (s & 31));
#endif
}
__host__ __device__ __forceinline__ unsigned fshl32(unsigned lo, unsigned hi, int s) {
#ifdef __CUDA_ARCH__
  return __funnelshift_l(lo, hi, s);
#else
  return (unsigned)(((((unsigned long long)hi << 32) | lo) << (s & 31)) >> 32);
#endif
}
__host__ __device__ __forceinline__ unsigned lo32(long long x) { return (unsigned)(unsigned long long)x; }
__host__ __device__ __forceinline__ unsigned hi32(long long x) { return (unsigned)((unsigned long long)x >> 32); }
__host__ __device__ __forceinline__ long long join32(unsigned hi, unsigned lo) {
  return (long long)(((unsigned long long)hi << 32) | lo);
}
// One's-complement magnitude of a 64-bit value's high word (the leading bit of |x| or |x| - 1).
__host__ __device__ __forceinline__ unsigned mag_hi32(long long x) {
  const unsigned h = hi32(x);
  return h ^ (unsigned)((int)h >> 31);
}
// Two signed 32-bit limbs of a 64-bit value: x = h 2^32 + l.
struct Limbs {
  int h, l;
};
__host__ __device__ __forceinline__ Limbs limbs_of(long long x) {
  Limbs v;
  v.l = (int)lo32(x);
  v.h = (int)(hi32(x) + (lo32(x) >> 31));
  return v;
}
// Position of the leading bit that differs from the sign, -1 if none.
__host__ __device__ __forceinline__ int lead_bit(int x) {
#ifdef __CUDA_ARCH__
  int p;
  asm("bfind.s32 %0, %1;" : "=r"(p) : "r"(x));
  return p;
#else
  return 31 - clz_u32((unsigned)(x ^ (x >> 31)));
#endif
}
// (x y) 2^-64 within 2 units a component, for |x|'s components <= 2^62 and |y|'s
// <= 2^62 (normal values or fixed-point factors).  Every sum of cross products
// stays below 2^63: a limb pair (h, l) with |h| = 2^30 has l of the sign that
// keeps |value| <= 2^62.
__host__ __device__ __forceinline__ void bf_mul_high(long long xr, long long xi, long long yr, long long yi,
                                                     long long& re, long long& im) {
  const Limbs a = limbs_of(xr), b = limbs_of(xi), c = limbs_of(yr), d = limbs_of(yi);
  const long long p = mad_wide(a.l, c.h, mul_wide(a.h, c.l)), q = mad_wide(b.l, d.h, mul_wide(b.h, d.l));
  const long long r = mad_wide(b.l, c.h, mad_wide(b.h, c.l, mad_wide(a.l, d.h, mul_wide(a.h, d.l))));
  re = mad_wide(-b.h, d.h, mul_wide(a.h, c.h)) + (long long)((int)hi32(p) - (int)hi32(q));
  im = mad_wide(b.h, c.h, mul_wide(a.h, d.h)) + (long long)(int)hi32(r);
}
// The normalising shift of a product's high half: the leading bit (in the high
// word, or below it when the product is tiny) moves up to bit 61; zero stays zero.
__host__ __device__ __forceinline__ int bf_renorm(long long& re, long long& im) {
  const int pr = lead_bit((int)hi32(re)), pi = lead_bit((int)hi32(im));
  const int p = pr > pi ? pr : pi;
  const int s = 29 - p;  // 0 .. 30
  re = join32(fshl32(lo32(re), hi32(re), s), lo32(re) << (s & 31));
  im = join32(fshl32(lo32(im), hi32(im), s), lo32(im) << (s & 31));
  return p;  // the exponent grows by 64 - s = p + 35
}
__host__ __device__ __forceinline__ BFloat bf_mul(const BFloat& x, const BFloat& y) {
  BFloat z;
  bf_mul_high(x.re, x.im, y.re, y.im, z.re, z.im);
  z.e = x.e + y.e + 35 + bf_renorm(z.re, z.im);
  return z;
}
// The 128-bit value (hi, lo) shifted right by r (arithmetic; 1 <= r <= 63), low 64 bits.
__host__ __device__ __forceinline__ long long shr128_lo(I128 x, int r) {
  return (long long)((x.lo >> r) | ((unsigned long long)x.hi << (64 - r)));
}
// (a + ib)(c + id) 2^e for fixed-point factors |a|, |b|, |c|, |d| < 2^61: exact
// 128-bit products (|re|, |im| < 2^123), then one truncation to the normal form.
__host__ __device__ __forceinline__ BFloat bf_pair(long long a, long long b, long long c, long long d, int e) {
  const I128 re = sub128(mul_s64(a, c), mul_s64(b, d));
  const I128 im = add128(mul_s64(a, d), mul_s64(b, c));
  BFloat z;
  const unsigned mt = mag_hi32(re.hi) | mag_hi32(im.hi);
  if (mt != 0) {
    // |value| >= 2^96 (the usual case): the leading bit (127 - clz) lies in the top
    // word, below bit 123, so the shift r = 66 - clz is 32 + rp with rp in [3, 29]
    // and the result is two 32-bit funnel shifts per component.
    const int rp = 34 - clz_u32(mt);
    z.re = join32(fshr32(lo32(re.hi), hi32(re.hi), rp), fshr32(hi32((long long)re.lo), lo32(re.hi), rp));
    z.im = join32(fshr32(lo32(im.hi), hi32(im.hi), rp), fshr32(hi32((long long)im.lo), lo32(im.hi), rp));
    z.e = e + 32 + rp;
    return z;
  }
  const long long sr = re.hi >> 63, si = im.hi >> 63;
  const unsigned long long mh = (unsigned long long)(re.hi ^ sr) | (unsigned long long)(im.hi ^ si);
  if (mh != 0) {
    const int r = 66 - clz_u64(mh);  // the leading bit (127 - clz, below bit 96 here) goes to bit 61: r in [3, 34]
    z.re = shr128_lo(re, r);
    z.im = shr128_lo(im, r);
    z.e = e + r;
    return z;
  }
  // Both high halves are sign bits: |re|, |im| < 2^64 (about 2^-58 of the largest products).
  const unsigned long long ml = (re.lo ^ (unsigned long long)sr) | (im.lo ^ (unsigned long long)si);
  const int r = 2 - clz_u64(ml);  // in [-62, 2]
  if (r > 0) {
    z.re = shr128_lo(re, r);
    z.im = shr128_lo(im, r);
  } else {  // |value| < 2^62: the low half is the value
    z.re = (long long)(re.lo << -r);
    z.im = (long long)(im.lo << -r);
  }
  z.e = e + r;
  return z;
}
// x 2^e rounded to the nearest double (ties away from zero); integer instructions
// except outside FP64's normal range (rare), which goes through ldexp.
__host__ __device__ __forceinline__ double bf_to_double(long long x, int e) {
  const unsigned long long sgn = (unsigned long long)(x >> 63);
  const unsigned long long ax = ((unsigned long long)x ^ sgn) - sgn;
  const int lz = clz_u64(ax);
  const unsigned long long y = ax << (lz & 63);
  const unsigned long long yr = y + 0x400ull;
  const unsigned long long carry = (yr < y) ? 1ull : 0ull;
  const unsigned long long mant = (yr >> 11) & 0xFFFFFFFFFFFFFull;
  const int be = e + 1086 - lz + (int)carry;
  if (be >= 1 && be <= 2046 && ax != 0) return bits_to_double((sgn << 63) | ((unsigned long long)be << 52) | mant);
  return ax ? ldexp((double)x, e) : 0.0;
}
// prod_f s_f with a factor below 2^32 (2^-30 of its possible size), whose digits
// bf_renorm's one shift leaves below the product's last place.
__device__ __noinline__ inline BFloat product_of_small(const long long* sr, const long long* si, int nf, int e0) {
  BFloat x = bf_norm(sr[0], si[0], e0);
  for (int f = 1; f < nf; ++f) x = bf_mul(x, bf_norm(sr[f], si[f], 0));
  return x;
}
// acc += sign * prod_f s_f, every product on the integer pipe, two FP64 adds.  The
// factors are split over two chains (two independent chains of dependent
// instructions hide each other's latency), each factor normalised first: a factor far
// below its largest possible sum keeps its digits (as it is, it would lose up to 2^-60 of
// that largest sum).  e0: minus the factors' fraction bits.
template <int NF>
__device__ __forceinline__ void accumulate_product_bf(const long long (&sr)[NF], const long long (&si)[NF], int e0,
                                                      uint32_t neg_mask, double& ar, double& ai) {
  if constexpr (NF == 1) {
    ar += xor_sign(bf_to_double(sr[0], e0), neg_mask);
    ai += xor_sign(bf_to_double(si[0], e0), neg_mask);
  } else {
    constexpr int H = NF < 4 ? NF : (NF + 1) / 2;  // first chain: factors 0 .. H - 1
    long long xr = sr[0], xi = si[0], yr, yi;
    int e = e0, least = 0;  // the sign of the factors' leading bits
    auto normal = [&](long long& re, long long& im) {
      const int p = bf_renorm(re, im);
      least = p < least ? p : least;
      e += p - 29;
    };
    normal(xr, xi);
    if constexpr (H < NF) {
      yr = sr[H];
      yi = si[H];
      normal(yr, yi);
    }
#pragma unroll
    for (int k = 1; k < H; ++k) {
      long long fr = sr[k], fi = si[k];
      normal(fr, fi);
      bf_mul_high(xr, xi, fr, fi, xr, xi);
      if ((H < NF && k == H - 1) || (k < H - 1 && k % 2 == 0))  // every second, and the last of two chains
        e += 35 + bf_renorm(xr, xi);
      else
        e += 64;
      if (H + k < NF) {
        fr = sr[H + k];
        fi = si[H + k];
        normal(fr, fi);
        bf_mul_high(yr, yi, fr, fi, yr, yi);
        e += (H + k == NF - 1 || k % 2 == 0) ? 35 + bf_renorm(yr, yi) : 64;
      }
    }
    if constexpr (H < NF) {
      bf_mul_high(xr, xi, yr, yi, xr, xi);
      e += 64;
    }
    if (least < 0 && (xr | xi) != 0) {  // rare
      long long tr[NF], ti[NF];
#pragma unroll
      for (int f = 0; f < NF; ++f) {
        tr[f] = sr[f];
        ti[f] = si[f];
      }
      const BFloat z = product_of_small(tr, ti, NF, e0);
      xr = z.re;
      xi = z.im;
      e = z.e;
    }
    ar += xor_sign(bf_to_double(xr, e), neg_mask);
    ai += xor_sign(bf_to_double(xi, e), neg_mask);
  }
}

// ---------------------------------------------------------------------------
// Float pairs on the FP32 pipe.  GB300 issues FP32 at 64x the FP64 rate, so the
// float-pair all-minors sweep keeps each value as an unevaluated sum hi + lo of
// two floats (about 47 significant bits) and uses the classical error-free
// transformations: Knuth's two-sum, the FMA two-product and Dekker's fast
// two-sum (T. J. Dekker, "A floating-point technique for extending the available
// precision", Numer. Math. 18, 1971).
// ---------------------------------------------------------------------------

// x * 2^(fbias - 190) as hi + lo: the 24 leading bits of |x| in hi, the next 23
// (truncated) in lo.  With |x| < 2^(p + 1) and fbias = 189 - p the value is below
// 1 in magnitude and every exponent field stays in [41, 126].  Integer work only.
__device__ __forceinline__ void fx_to_ff(long long x, int fbias, float& hi, float& lo) {
  const unsigned long long sgn = (unsigned long long)(x >> 63);
  const unsigned long long ax = ((unsigned long long)x ^ sgn) - sgn;
  const int lz = __clzll((long long)ax);
  const unsigned long long y = ax << (lz & 63);
  const uint32_t yh = (uint32_t)(y >> 32), yl = (uint32_t)y;
  const int ex = fbias - lz;  // exponent field of the leading bit
  const uint32_t s32 = (uint32_t)sgn & 0x80000000u;
  const uint32_t hb = (((uint32_t)(ex - 1)) << 23) + (yh >> 8);  // the leading bit carries into the field
  const uint32_t nxt = __funnelshift_r(yl, yh, 17) & 0x7FFFFFu;  // bits 39..17 of y
  const uint32_t eb = ((uint32_t)(ex - 23)) << 23;
  const float l = __uint_as_float(eb | nxt) - __uint_as_float(eb);  // exact (Sterbenz)
  hi = ax ? __uint_as_float(hb | s32) : 0.0f;
  lo = ax ? __uint_as_float(__float_as_uint(l) ^ s32) : 0.0f;
}

struct ffc {  // complex float pair
  float rh, rl, ih, il;
};

// (h, l) += sg * (bh, bl), sg = +-1: two-sum of the high parts, the low parts
// added to its error, renormalised by a fast two-sum.
__device__ __forceinline__ void ff_acc(float& h, float& l, float sg, float bh, float bl) {
  const float s = fmaf(sg, bh, h);
  const float bb = s - h;
  const float err = (h - (s - bb)) + fmaf(sg, bh, -bb);
  const float lo = err + fmaf(sg, bl, l);
  h = s + lo;
  l = lo - (h - s);
}

// p + e = a * b up to the a_lo * b_lo term (the FMA two-product of the high parts
// plus the cross terms).  __fmul_rn: p must stay a rounded product, never fused
// into a later add.
__device__ __forceinline__ void ff_prod(float ah, float al, float bh, float bl, float& p, float& e) {
  p = __fmul_rn(ah, bh);
  e = fmaf(ah, bh, -p);
  e = fmaf(ah, bl, e);
  e = fmaf(al, bh, e);
}

// (p1 + e1) + sg * (p2 + e2), normalised.
__device__ __forceinline__ void ff_combine(float p1, float e1, float sg, float p2, float e2, float& h, float& l) {
  const float s = fmaf(sg, p2, p1);
  const float bb = s - p1;
  const float err = (p1 - (s - bb)) + fmaf(sg, p2, -bb);
  const float lo = err + fmaf(sg, e2, e1);
  h = s + lo;
  l = lo - (h - s);
}

__device__ __forceinline__ ffc ff_cmul(const ffc& a, const ffc& b) {
  float p1, e1, p2, e2, p3, e3, p4, e4;
  ff_prod(a.rh, a.rl, b.rh, b.rl, p1, e1);
  ff_prod(a.ih, a.il, b.ih, b.il, p2, e2);
  ff_prod(a.rh, a.rl, b.ih, b.il, p3, e3);
  ff_prod(a.ih, a.il, b.rh, b.rl, p4, e4);
  ffc r;
  ff_combine(p1, e1, -1.0f, p2, e2, r.rh, r.rl);
  ff_combine(p3, e3, 1.0f, p4, e4, r.ih, r.il);
  return r;
}

// The sweep's inner loop skips the renormalisations: a running sum's low part
// then collects the two-sums' exact errors (cascaded summation), and a product's
// low part stays within a few 2^-24 of the complex magnitude, so the next
// product's cross terms lose nothing measurable (about 2^-46 per product against
// 2^-48).  Sums are resynchronised or renormalised before they leave the loop.
__device__ __forceinline__ void ff_add_lazy(float& h, float& l, float sg, float bh, float bl) {
  const float s = fmaf(sg, bh, h);
  const float bb = s - h;
  const float err = (h - (s - bb)) + fmaf(sg, bh, -bb);
  h = s;
  l = err + fmaf(sg, bl, l);
}

__device__ __forceinline__ ffc ff_cmul_lazy(const ffc& a, const ffc& b) {
  float p1, e1, p2, e2, p3, e3, p4, e4;
  ff_prod(a.rh, a.rl, b.rh, b.rl, p1, e1);
  ff_prod(a.ih, a.il, b.ih, b.il, p2, e2);
  ff_prod(a.rh, a.rl, b.ih, b.il, p3, e3);
  ff_prod(a.ih, a.il, b.rh, b.rl, p4, e4);
  ffc r;
  r.rh = p1;
  r.rl = e1;
  ff_add_lazy(r.rh, r.rl, -1.0f, p2, e2);
  r.ih = p3;
  r.il = e3;
  ff_add_lazy(r.ih, r.il, 1.0f, p4, e4);
  return r;
}

// (h, l) * (bh, bl), normalised.
__device__ __forceinline__ void ff_mul(float& h, float& l, float bh, float bl) {
  float p, e;
  ff_prod(h, l, bh, bl, p, e);
  h = p + e;
  l = e - (h - p);
}

__device__ __forceinline__ double ff_to_double(float h, float l) { return (double)h + (double)l; }

// x as a float pair (hi = x rounded to float, lo = the rest rounded): 48 bits.
__device__ __forceinline__ void double_to_ff(double x, float& hi, float& lo) {
  hi = __double2float_rn(x);
  lo = __double2float_rn(x - (double)hi);
}

// |re + i im|^2 for float pairs (re = rs + rc, im = is + ic, unnormalised as a
// compensated sum leaves them), as a normalised float pair.
__device__ __forceinline__ float2 ff_abs2(float rs, float rc, float is, float ic) {
  float rh = rs + rc, ih = is + ic;
  float rl = rc - (rh - rs), il = ic - (ih - is);  // fast two-sums: |s| >= |c|, or s = 0
  float p, e, q, f;
  ff_prod(rh, rl, rh, rl, p, e);
  ff_prod(ih, il, ih, il, q, f);
  ff_combine(p, e, 1.0f, q, f, rh, rl);
  return make_float2(rh, rl);
}

// Compensated dot-product step (Ogita, Rump and Oishi, "Accurate sum and dot
// product", SIAM J. Sci. Comput. 26, 2005): s + c accumulates sg * a * b for
// float pairs a, b, the products' errors and the sums' errors collected in c.
__device__ __forceinline__ void ff_dot_acc(float& s, float& c, float sg, float ah, float al, float bh, float bl) {
  float p, e;
  ff_prod(ah, al, bh, bl, p, e);
  const float t = fmaf(sg, p, s);
  const float bb = t - s;
  const float q = (s - (t - bb)) + fmaf(sg, p, -bb);
  c += fmaf(sg, e, q);
  s = t;
}

__device__ __forceinline__ double warp_sum(double v) {
  // Fixed butterfly order: every lane ends with the same, run-to-run identical sum.
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}

// This thread's code range inside its sweep: lengths differ by at most one.
__device__ __forceinline__ void thread_range(const SweepProblem& P, int64_t q, int64_t& a, int64_t& len) {
  const int64_t per = P.n_codes / P.n_threads, rem = P.n_codes % P.n_threads;
  a = q * per + (q < rem ? q : rem);
  len = per + (q < rem ? 1 : 0);
}

// The same split in whole units of 2^c codes (lengths differ by at most one
// unit; the last unit of the sweep may be short).  Every range then starts at a
// multiple of 2^c, so at every step the lanes of a warp flip the same binary
// digit whenever that digit is below c: their per-digit updates touch the same
// row, and rows laid out by lane are read and written in whole lines.
__device__ __forceinline__ void thread_range_aligned(const SweepProblem& P, int64_t q, int c, int64_t& a,
                                                     int64_t& len) {
  const int64_t units = (P.n_codes + (1ll << c) - 1) >> c;
  const int64_t per = units / P.n_threads, rem = units % P.n_threads;
  a = (q * per + (q < rem ? q : rem)) << c;
  const int64_t want = (per + (q < rem ? 1 : 0)) << c;
  len = (a >= P.n_codes) ? 0 : (a + want <= P.n_codes ? want : P.n_codes - a);
}

__device__ __forceinline__ int find_problem(const SweepProblem* __restrict__ probs, int n, int64_t gt) {
  int lo = 0, hi = n - 1;
  while (lo < hi) {
    const int mid = (lo + hi + 1) >> 1;
    if (probs[mid].thread_begin <= gt) lo = mid; else hi = mid - 1;
  }
  return lo;
}

}  // namespace boss
