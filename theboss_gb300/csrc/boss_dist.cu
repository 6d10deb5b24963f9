// boss_dist.cu -- exact output probabilities under particle losses, all outcomes at once.
//
// theboss's BSDistributionCalculatorWithFixedLosses
// (bs_distribution_calculator_with_fixed_losses.py:84-151) computes, for every
// outcome T with l particles, a sum over the distinct l-particle sub-occupations
// S' of the initial state ("lossy inputs", in the order
// generate_lossy_n_particle_input_states gives them,
// boson_sampling_utilities.py:158-203):
//     p(T) = [ sum_S' |perm(U[T, S'])|^2 / prod_i S'_i! * mult(S') ] / l! / C(n, l) * l! / prod_i T_i!
// with mult(S') = prod_i C(S_i, S_i - S'_i); theboss evaluates one outcome at a
// time (the uniform-loss calculator maps outcomes over a process pool,
// bs_exact_distribution_with_uniform_losses.py:62-71).  Here, for every particle
// count l <= kDistMaxL:
//   * lossy_table_kernel: the row sums of every (lossy input, sign vector);
//   * lossy_walk_kernel: the Glynn permanents of every (lossy input, outcome) from
//     them, then |perm|^2, theboss's divisions and the multiplicity;
//   * lossy_outcome_kernel: per outcome, the sum over lossy inputs in theboss's
//     order and the normalisation, with theboss's operation order.
// Larger l goes through the sweep engine (one Glynn sweep per pair, many threads
// each), and the same host arithmetic.
#include <cuda_runtime.h>
#include <stdint.h>
#include <string.h>

#include <algorithm>
#include <cmath>
#include <mutex>
#include <string>
#include <type_traits>
#include <unordered_map>
#include <vector>

#include "../../include/boss.h"
#include "boss_internal.h"

namespace boss {

extern std::mutex g_api_mutex;

constexpr int kDistMaxL = 10;  // per-thread permanents up to 10 x 10 (512 sign vectors)
constexpr int kDistMaxDiv = 8;  // divisors (factorials of occupations >= 2) kept per state

// The permanent of one L x L matrix of doubles, entry (a, b) at A[(b L + a) n]:
// Glynn's formula with the sign of column 0 fixed, columns 1..L-1 walked in
// binary-reflected Gray order.
template <int L>
__device__ __forceinline__ double2 glynn_small(const longlong2* __restrict__ A, int64_t n) {
  auto entry = [&](int a, int b) {
    const longlong2 u = A[(b * L + a) * n];
    return make_double2(__longlong_as_double(u.x), __longlong_as_double(u.y));
  };
  double sr[L], si[L];
#pragma unroll
  for (int a = 0; a < L; ++a) {
    double x = 0.0, y = 0.0;
#pragma unroll
    for (int b = 0; b < L; ++b) {
      const double2 u = entry(a, b);
      x += u.x;
      y += u.y;
    }
    sr[a] = x;
    si[a] = y;
  }
  double accr = 0.0, acci = 0.0;
  uint32_t neg = 0;  // bit b: column b currently has sign -1
  const uint32_t codes = 1u << (L - 1);
  for (uint32_t t = 0;;) {
    double pr = sr[0], pi = si[0];
#pragma unroll
    for (int a = 1; a < L; ++a) {
      const double r = fma(pr, sr[a], -(pi * si[a]));
      const double i = fma(pr, si[a], pi * sr[a]);
      pr = r;
      pi = i;
    }
    if (__popc(neg) & 1) {
      accr -= pr;
      acci -= pi;
    } else {
      accr += pr;
      acci += pi;
    }
    if (++t >= codes) break;
    const int b = __ffs(t);  // column 1 + ctz(t)
    const double c = ((neg >> b) & 1u) ? 2.0 : -2.0;
    neg ^= 1u << b;
#pragma unroll
    for (int a = 0; a < L; ++a) {
      const double2 u = entry(a, b);
      sr[a] = fma(c, u.x, sr[a]);
      si[a] = fma(c, u.y, si[a]);
    }
  }
  const double s = ldexp(1.0, -(L - 1));
  return make_double2(accr * s, acci * s);
}

// A row's fixed-point scale for sums of at most `terms` of its entries: the fraction
// bits that keep them below 2^62, or kNoScale where that cannot be done (a
// non-finite entry, or sizes near the ends of the exponent range): such rows are
// summed in FP64.
constexpr int kNoScale = 1 << 30;
__host__ __device__ inline int row_fraction_bits(double largest, int terms) {
  if (largest == 0.0) return 56;
  if (!(largest < 1e270 && largest > 1e-270)) return kNoScale;
  return 61 - ilogb(largest * terms);  // largest * terms < 2^(ilogb + 1)
}

// The permanents of a batch by particle count: count l has permanents first[l] to
// first[l + 1] - 1, and their matrices begin at entry mat[l].
struct SmallClasses {
  int64_t first[kSmallPermMax + 2], mat[kSmallPermMax + 2];
};

// One warp per permanent: its particles' modes from len occupations (in page-locked
// host memory, every one read once), and its matrix, every row in the scale that its
// own entries allow: entry (a, b) of permanent i of n of a class at (b l + a) n + i,
// packed (pack_row), e0 minus the rows' fraction bits; or as doubles, e0 = kNoScale,
// where a row has no scale.
__global__ void __launch_bounds__(128) small_prepare_kernel(const double2* __restrict__ U, int m,
                                                            const uint8_t* __restrict__ T,
                                                            const uint8_t* __restrict__ S, int len, SmallClasses c,
                                                            longlong2* __restrict__ A, int32_t* __restrict__ e0s) {
  __shared__ uint16_t modes_s[4][2][kSmallPermMax];
  __shared__ unsigned long long mx_s[4][kSmallPermMax];
  const int64_t k = (int64_t)blockIdx.x * 4 + (threadIdx.x >> 5);
  const int lane = threadIdx.x & 31;
  if (k >= c.first[kSmallPermMax + 1]) return;
  int l = 1;
  while (k >= c.first[l + 1]) ++l;
  uint16_t(&modes)[2][kSmallPermMax] = modes_s[threadIdx.x >> 5];
  unsigned long long* mx = mx_s[threadIdx.x >> 5];
  if (lane < kSmallPermMax) mx[lane] = 0ull;
  int done[2] = {0, 0};
  for (int base = 0; base < len && min(done[0], done[1]) < l; base += 32) {
    const bool in = base + lane < len;
    const int v[2] = {in ? T[k * len + base + lane] : 0, in ? S[k * len + base + lane] : 0};
#pragma unroll
    for (int side = 0; side < 2; ++side) {
      int incl = v[side];
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const int y = __shfl_up_sync(0xffffffffu, incl, o);
        if (lane >= o) incl += y;
      }
      for (int q = 0; q < v[side]; ++q) modes[side][done[side] + incl - v[side] + q] = (uint16_t)(base + lane);
      done[side] += __shfl_sync(0xffffffffu, incl, 31);
    }
  }
  __syncwarp();
  constexpr int kPer = (kSmallPermMax * kSmallPermMax + 31) / 32;  // entries per lane
  double2 v[kPer];
#pragma unroll
  for (int i = 0; i < kPer; ++i) {  // independent gathers in flight
    const int e = lane + 32 * i, b = e / l, a = e - b * l;
    if (e >= l * l) break;
    v[i] = U[(size_t)modes[0][a] * m + modes[1][b]];
    // the row's largest: non-negative doubles order as integers, an infinity above every finite one
    const double x = isfinite(v[i].x) && isfinite(v[i].y) ? fmax(fabs(v[i].x), fabs(v[i].y)) : __longlong_as_double(0x7ff0000000000000ll);
    atomicMax(mx + a, (unsigned long long)__double_as_longlong(x));
  }
  __syncwarp();
  int fx = 0;
  if (lane < l) fx = row_fraction_bits(__longlong_as_double((long long)mx[lane]), l);  // infinite: kNoScale
  const bool fine = __all_sync(0xffffffffu, fx != kNoScale);
  const int e0 = fine ? -__reduce_add_sync(0xffffffffu, fx) : kNoScale;
  if (lane == 0) e0s[k] = e0;
  const int64_t n = c.first[l + 1] - c.first[l];
  longlong2* to = A + c.mat[l] + (k - c.first[l]);
#pragma unroll
  for (int i = 0; i < kPer; ++i) {
    const int e = lane + 32 * i, a = e % l;
    if (32 * i >= l * l) break;  // the whole warp
    const int f = __shfl_sync(0xffffffffu, fx, a);
    if (e >= l * l) continue;
    to[(int64_t)e * n] = fine ? make_longlong2(pack_row(__double2ll_rn(ldexp(v[i].x, f))),
                                               pack_row(__double2ll_rn(ldexp(v[i].y, f))))
                              : make_longlong2(__double_as_longlong(v[i].x), __double_as_longlong(v[i].y));
  }
}

// Small permanents, each of the L x L matrix that small_prepare_kernel (or, for a few,
// the host) laid out.  2^lg lanes per permanent, each over 2^(L - 1 - lg) sign vectors:
// the last lg columns' signs are the lane's bits, the others walk in Gray order, column
// 0 stays +.  The products run on the integer pipe (accumulate_product_bf), so a code
// costs ~45 instructions per factor where FP64 ones hold its pipe for 4 * 64 clocks,
// and a single permanent has all lanes of a block instead of one thread's chain of
// dependent FP64 products (n = 8: 248 -> 27 us a call, planning and synchronisation
// included).  Compiled for 5 to 6 blocks per SM although few run: with the 80 to 94
// registers of no bound, one of n = 10 takes 41.7 us a call instead of 36.7, 31 of n = 9
// 44.4 instead of 39.6.  A permanent with a row that has no scale is summed in FP64 by its first lane.
template <int L>
__global__ void __launch_bounds__(128, L <= 9 ? 6 : 5) small_perm_kernel(const longlong2* __restrict__ A,
                                                         const int32_t* __restrict__ e0s, int64_t count, int lg,
                                                         double2* __restrict__ out) {
  __shared__ double2 part[4];
  const int64_t gid = (int64_t)blockIdx.x * 128 + threadIdx.x;
  const int64_t at = gid >> lg;
  const int64_t k = at < count ? at : count - 1;
  const uint32_t mine = (uint32_t)gid & ((1u << lg) - 1u);
  const longlong2* Ak = A + k;
  const int e0 = e0s[k];
  double ar = 0.0, ai = 0.0;
  if (e0 == kNoScale) {
    if (mine == 0) {
      const double2 p = glynn_small<L>(Ak, count);
      ar = p.x;
      ai = p.y;
    }
  } else {
    long long sr[L], si[L];
#pragma unroll
    for (int a = 0; a < L; ++a) sr[a] = si[a] = 0;
    const int low = L - lg;  // columns low .. L - 1 have the lane's signs
    for (int b = 0; b < L; ++b) {
      const int sg = (b >= low && ((mine >> (b - low)) & 1u)) ? -1 : 1;
#pragma unroll
      for (int a = 0; a < L; ++a) {
        const longlong2 u = Ak[(b * L + a) * count];
        sr[a] = add_packed(sr[a], u.x, sg);
        si[a] = add_packed(si[a], u.y, sg);
      }
    }
    uint32_t neg = 0, parity = __popc(mine) & 1;
    const uint32_t codes = 1u << (low - 1);
    for (uint32_t t = 0;;) {
      accumulate_product_bf<L>(sr, si, e0, parity << 31, ar, ai);
      if (++t >= codes) break;
      const int b = __ffs(t);  // column 1 + ctz(t)
      const int sg = ((neg >> b) & 1u) ? 2 : -2;
      neg ^= 1u << b;
      parity ^= 1u;
#pragma unroll
      for (int a = 0; a < L; ++a) {
        const longlong2 u = Ak[(b * L + a) * count];
        sr[a] = add_packed(sr[a], u.x, sg);
        si[a] = add_packed(si[a], u.y, sg);
      }
    }
    const double s = 1.0 / (double)(1u << (L - 1));
    ar *= s;
    ai *= s;
  }
  for (int o = 1; o < (1 << min(lg, 5)); o <<= 1) {  // the permanent's lanes, in a fixed order
    ar += __shfl_xor_sync(0xffffffffu, ar, o);
    ai += __shfl_xor_sync(0xffffffffu, ai, o);
  }
  if (lg > 5) {  // 2 or 4 whole warps per permanent
    if ((threadIdx.x & 31) == 0) part[threadIdx.x >> 5] = make_double2(ar, ai);
    __syncthreads();
    if (mine == 0)
      for (int w = 1; w < (1 << (lg - 5)); ++w) {
        ar += part[(threadIdx.x >> 5) + w].x;
        ai += part[(threadIdx.x >> 5) + w].y;
      }
  }
  if (mine == 0 && at < count) out[k] = make_double2(ar, ai);
}

// ---------------------------------------------------------------------------
// All (lossy input, outcome) permanents of one particle count L.
//
// For a lossy input and a sign vector d (first sign +) the row sums V[o] =
// sum_b d_b U[o][col b] depend on the output mode o only, so they are tabulated, and
// an outcome's product over its particles' modes (in mode order) shares its leading
// factors with the outcome before it: outcomes in lexicographic order need 1 to 2
// products each instead of L - 1 products and L row updates.  A lane takes one
// (input, sign vector), a warp 32 of them (several sign vectors of one input from
// L = 6 on, several inputs below), and walks a chunk of outcomes with the partial
// products in registers: the same control flow in every lane.
// kFixed: the row sums are exact 64-bit fixed point, each (input, row) in the scale of
// its own L entries, and the products run on the integer pipe (block floating point,
// boss_sweep.cuh): about 45 instructions each against four FP64 ones that hold their
// pipe for 64 clocks.  Otherwise (a matrix with entries that have no scale) both are FP64.
// 8 photons in 16 modes, all 735,471 outcomes: 16.5 ms with one thread per (input,
// outcome) walking all sign vectors, 4.4 with this walk in FP64 (pipe 87 % busy), 2.5
// in fixed point (issue and latency: 190 instructions an outcome and 32 sign vectors).
// ---------------------------------------------------------------------------
constexpr int kWalkChunk = 128;  // outcomes per warp at most (a multiple of 8)

// Every outcome's particles in mode order (bytes 0 .. L - 1) and how many leading
// ones it shares with the outcome before it (byte 15).
__global__ void lossy_rows_kernel(const uint8_t* __restrict__ occ, int m, int64_t O, uint4* __restrict__ rows) {
  const int64_t o = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (o >= O) return;
  uint32_t w[4] = {0, 0, 0, 0};
  const uint8_t* t = occ + o * m;
  const uint8_t* before = o > 0 ? t - m : nullptr;
  int a = 0, same = 0;
  bool equal = before != nullptr;
  for (int i = 0; i < m; ++i) {
    const int c = t[i];
    if (equal) {
      same += min(c, (int)before[i]);
      equal = c == before[i];
    }
    for (int k = 0; k < c && a < 15; ++k, ++a) w[a >> 2] |= (uint32_t)i << (8 * (a & 3));
  }
  w[3] |= (uint32_t)same << 24;
  rows[o] = make_uint4(w[0], w[1], w[2], w[3]);
}

// V[(combo / 32 * m + row) * 32 + combo % 32], combo = input * 2^(L-1) + sign vector:
// doubles, or (ve given) 62-bit mantissas with the exponents ve at the same places, of
// exact fixed-point sums, each (input, row) in the scale of its own entries.
__global__ void lossy_table_kernel(const double2* __restrict__ U, int m, int L, const uint8_t* __restrict__ cols,
                                   int K, int64_t combos, int32_t* __restrict__ ve, double2* __restrict__ V) {
  const int64_t e = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (e >= combos * m) return;
  const int64_t combo = e / ((int64_t)32 * m) * 32 + (e & 31);
  const int row = (int)((e >> 5) % m);
  const int64_t k = combo >> (L - 1);
  double x = 0.0, y = 0.0;
  const uint32_t d = (uint32_t)combo & ((1u << (L - 1)) - 1u);
  if (ve) {
    long long fr = 0, fi = 0;
    int exp = 0;
    if (k < K) {
      unsigned long long mx = 0;  // magnitudes order as integers
      for (int b = 0; b < L; ++b) {
        const double2 u = U[(size_t)row * m + cols[k * L + b]];
        mx = max(mx, max((unsigned long long)__double_as_longlong(fabs(u.x)),
                         (unsigned long long)__double_as_longlong(fabs(u.y))));
      }
      const int f = row_fraction_bits(__longlong_as_double((long long)mx), L);
      const double scale = __longlong_as_double((long long)(1023 + f) << 52);  // 2^f, |f| < 1000
      for (int b = 0; b < L; ++b) {
        const double2 u = U[(size_t)row * m + cols[k * L + b]];
        const bool neg = b > 0 && ((d >> (b - 1)) & 1u);
        const long long ur = __double2ll_rn(u.x * scale), ui = __double2ll_rn(u.y * scale);
        fr += neg ? -ur : ur;
        fi += neg ? -ui : ui;
      }
      const BFloat z = bf_norm(fr, fi, -f);
      fr = z.re;
      fi = z.im;
      exp = z.e;
    }
    ve[e] = exp;
    reinterpret_cast<longlong2*>(V)[e] = make_longlong2(fr, fi);
    return;
  }
  if (k < K) {
    for (int b = 0; b < L; ++b) {
      const double2 u = U[(size_t)row * m + cols[k * L + b]];
      const bool neg = b > 0 && ((d >> (b - 1)) & 1u);
      x += neg ? -u.x : u.x;
      y += neg ? -u.y : u.y;
    }
  }
  V[e] = make_double2(x, y);
}

// One warp per (group of 32 combos of equal input or of several inputs, chunk of
// outcomes); from L = 6 on a group is one input and its 2^(L-6) blocks of 32 sign
// vectors are walked one after the other.
template <int L, bool kFixed>
__global__ void __launch_bounds__(128) lossy_walk_kernel(const double2* __restrict__ V, int m,
                                                         const int32_t* __restrict__ ve,  // kFixed: V's exponents
                                                         const uint4* __restrict__ rows, int64_t O, int K, int groups,
                                                         const double* __restrict__ in_div,    // [K][kDistMaxDiv]
                                                         const int* __restrict__ in_ndiv,      // [K]
                                                         const double* __restrict__ in_mult,   // [K]
                                                         int chunk, double* __restrict__ terms) {  // [K][O]
  constexpr int kBlocks = L >= 6 ? 1 << (L - 6) : 1;  // blocks of 32 sign vectors per input
  constexpr int kLanes = L >= 6 ? 32 : 1 << (L - 1);  // lanes of one input
  __shared__ double2 buf_s[4][8 * 33];
  __shared__ double2 acc_s[4][kWalkChunk];
  const int wp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int64_t chunks = (O + chunk - 1) / chunk;
  const int64_t task = (int64_t)blockIdx.x * 4 + wp;
  if (task >= chunks * groups) return;  // whole warps
  const int g = (int)(task / chunks);
  const int64_t o0 = (task - (int64_t)g * chunks) * chunk;
  const int n = (int)min((int64_t)chunk, O - o0);
  double2* buf = buf_s[wp];
  double2* acc = acc_s[wp];
  const double scale = 1.0 / (double)(1u << (L - 1));
  auto term = [&](double2 p, int k) {
    const double re = p.x * scale, im = p.y * scale;
    double v = fma(re, re, im * im);
    // bs_distribution_calculator_with_fixed_losses.py:137-142, same operation order
    const int nd = in_ndiv[k];
    for (int d = 0; d < nd; ++d) v /= in_div[(size_t)k * kDistMaxDiv + d];
    return v * in_mult[k];
  };
  for (int j = 0; j < kBlocks; ++j) {
    const int64_t block = L >= 6 ? (int64_t)g * kBlocks + j : g;
    const double2* Vg = V + block * 32 * m + lane;
    const uint32_t d = L >= 6 ? (uint32_t)(j * 32 + lane) : (uint32_t)(lane & (kLanes - 1));
    const uint32_t neg = (__popc(d) & 1) << 31;
    const int32_t* eg = kFixed ? ve + block * 32 * m + lane : nullptr;
    double2 P[kFixed ? 1 : L];
    long long pr[kFixed ? L : 1], pi[kFixed ? L : 1];  // normalised, in units of 2^pe
    int pe[kFixed ? L : 1];
    double2 x = make_double2(0.0, 0.0);  // the last product
    for (int q = 0; q < n; ++q) {
      const uint4 r = __ldg(rows + o0 + q);
      const uint32_t w[4] = {r.x, r.y, r.z, r.w};
      const int c = q > 0 ? (int)(r.w >> 24) : 0;
      auto step = [&](auto index) {
        constexpr int a = decltype(index)::value;
        if constexpr (a < L && kFixed) {
          const int row = (int)((w[a >> 2] >> (8 * (a & 3))) & 255u);
          const longlong2 v = __ldg(reinterpret_cast<const longlong2*>(Vg) + (size_t)row * 32);
          long long zr = v.x, zi = v.y;
          int e = __ldg(eg + (size_t)row * 32);
          if constexpr (a > 0) {
            bf_mul_high(pr[a - 1], pi[a - 1], v.x, v.y, zr, zi);
            e += pe[a - 1] + 64;
          }
          if constexpr (a < L - 1) {
            if constexpr (a > 0) e += bf_renorm(zr, zi) - 29;
            pr[a] = zr;
            pi[a] = zi;
            pe[a] = e;
          } else {
            x = make_double2(xor_sign(bf_to_double(zr, e), neg), xor_sign(bf_to_double(zi, e), neg));
          }
        } else if constexpr (a < L) {
          const double2 v = __ldg(Vg + (size_t)((w[a >> 2] >> (8 * (a & 3))) & 255u) * 32);
          if constexpr (a == 0) {
            P[0] = make_double2(xor_sign(v.x, neg), xor_sign(v.y, neg));
          } else {
            const double2 p = P[a - 1];
            P[a] = make_double2(fma(p.x, v.x, -(p.y * v.y)), fma(p.x, v.y, p.y * v.x));
          }
          if constexpr (a == L - 1) x = P[a];
        }
      };
      // a jump into the chain, not a condition per step: predicated-off FP64
      // instructions would hold the pipe all the same
      switch (c) {
        case 0: step(std::integral_constant<int, 0>{}); [[fallthrough]];
        case 1: step(std::integral_constant<int, 1>{}); [[fallthrough]];
        case 2: step(std::integral_constant<int, 2>{}); [[fallthrough]];
        case 3: step(std::integral_constant<int, 3>{}); [[fallthrough]];
        case 4: step(std::integral_constant<int, 4>{}); [[fallthrough]];
        case 5: step(std::integral_constant<int, 5>{}); [[fallthrough]];
        case 6: step(std::integral_constant<int, 6>{}); [[fallthrough]];
        case 7: step(std::integral_constant<int, 7>{}); [[fallthrough]];
        case 8: step(std::integral_constant<int, 8>{}); [[fallthrough]];
        case 9: step(std::integral_constant<int, 9>{}); break;
        default: break;
      }
      if constexpr (L < 6) {
        double2 sum = x;
#pragma unroll
        for (int o = 1; o < kLanes; o <<= 1) {
          sum.x += __shfl_xor_sync(0xffffffffu, sum.x, o);
          sum.y += __shfl_xor_sync(0xffffffffu, sum.y, o);
        }
        const int k = g * (32 / kLanes) + lane / kLanes;
        if ((lane & (kLanes - 1)) == 0 && k < K) terms[(size_t)k * O + o0 + q] = term(sum, k);
      } else {
        // eight outcomes at a time: four lanes add up eight combos each of one outcome
        buf[(q & 7) * 33 + lane] = x;
        if ((q & 7) == 7 || q + 1 == n) {
          __syncwarp();
          const int oo = lane >> 2, part = lane & 3, at = (q & ~7) + oo;
          double2 s = make_double2(0.0, 0.0);
          if (at < n) {
#pragma unroll
            for (int i = 0; i < 8; ++i) {
              const double2 v = buf[oo * 33 + part * 8 + i];
              s.x += v.x;
              s.y += v.y;
            }
          }
#pragma unroll
          for (int o = 1; o < 4; o <<= 1) {
            s.x += __shfl_xor_sync(0xffffffffu, s.x, o);
            s.y += __shfl_xor_sync(0xffffffffu, s.y, o);
          }
          if (part == 0 && at < n) {
            if (j > 0) s = make_double2(s.x + acc[at].x, s.y + acc[at].y);
            acc[at] = s;
          }
          __syncwarp();
        }
      }
    }
  }
  if constexpr (L >= 6) {
    __syncwarp();
    for (int q = lane; q < n; q += 32) terms[(size_t)g * O + o0 + q] = term(acc[q], g);
  }
}

__global__ void lossy_outcome_kernel(const double* __restrict__ terms, int K, int64_t O, int m,
                                     const uint8_t* __restrict__ out_occ,  // [O][m]
                                     const double* __restrict__ fact,      // [256] k! as theboss divides by it
                                     double fact_l, double binom_nl, double* __restrict__ prob) {
  const int64_t o = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (o >= O) return;
  double p = 0.0;
  for (int k = 0; k < K; ++k) p += terms[(size_t)k * O + o];
  // bs_distribution_calculator_with_fixed_losses.py:145-149 and 99-104
  p /= fact_l;
  p /= binom_nl;
  p *= fact_l;
  const uint8_t* occ = out_occ + o * m;
  for (int i = 0; i < m; ++i)
    if (occ[i] >= 2) p /= fact[occ[i]];
  prob[o] = p;
}

// ---------------------------------------------------------------------------
// Host side
// ---------------------------------------------------------------------------
static size_t align256(size_t x) { return (x + 255) & ~(size_t)255; }

static double factorial_d(int k) {  // exact up to 20!, then the nearest double of the product
  if (k <= 20) {
    uint64_t f = 1;
    for (int i = 2; i <= k; ++i) f *= (uint64_t)i;
    return (double)f;
  }
  long double f = 1.0L;
  for (int i = 2; i <= k; ++i) f *= (long double)i;
  return (double)f;
}

static double binom_d(int n, int k) {  // exact below 2^64
  if (k < 0 || k > n) return 0.0;
  k = std::min(k, n - k);
  unsigned __int128 c = 1;
  for (int i = 1; i <= k; ++i) c = c * (unsigned)(n - k + i) / (unsigned)i;
  return (double)c;
}

struct LossyInputs {
  std::vector<std::vector<int32_t>> occ;  // distinct sub-occupations, theboss's order
  std::vector<double> mult;               // prod_i C(S_i, S_i - S'_i)
};

// generate_lossy_n_particle_input_states (boson_sampling_utilities.py:175-203):
// combinations of particle indices in lexicographic order, first occurrence kept.
static int lossy_inputs(const int32_t* S, int m, int l, LossyInputs& out) {
  std::vector<int> x0;
  for (int i = 0; i < m; ++i)
    for (int c = 0; c < S[i]; ++c) x0.push_back(i);
  const int n = (int)x0.size();
  out.occ.clear();
  out.mult.clear();
  if (n == 0) {
    out.occ.push_back(std::vector<int32_t>(S, S + m));
    out.mult.push_back(1.0);
    return kOk;
  }
  if (l > n) return kOk;
  if (binom_d(n, l) > 5e7) {
    set_error("too many lossy input combinations (C(n, l) > 5e7)");
    return kErrLimit;
  }
  std::unordered_map<std::string, int> seen;
  std::vector<int> c(l);
  for (int i = 0; i < l; ++i) c[i] = i;
  std::vector<int32_t> occ(m);
  for (;;) {
    std::fill(occ.begin(), occ.end(), 0);
    for (int i = 0; i < l; ++i) occ[x0[c[i]]]++;
    std::string key((const char*)occ.data(), sizeof(int32_t) * m);
    if (seen.emplace(key, (int)out.occ.size()).second) {
      double mu = 1.0;  // bs_distribution_calculator_with_fixed_losses.py:162-169
      for (int i = 0; i < m; ++i) mu *= binom_d(S[i], S[i] - occ[i]);
      out.occ.push_back(occ);
      out.mult.push_back((double)(int64_t)mu);
    }
    int i = l - 1;
    while (i >= 0 && c[i] == n - l + i) --i;
    if (i < 0) break;
    c[i]++;
    for (int j = i + 1; j < l; ++j) c[j] = c[j - 1] + 1;
  }
  return kOk;
}

// Factorials of the occupations >= 2, in mode order (theboss divides by every
// factorial; those of 0 and 1 leave the value unchanged).
static int divisors(const int32_t* occ, int m, double* div) {
  int nd = 0;
  for (int i = 0; i < m; ++i)
    if (occ[i] >= 2) {
      if (nd == kDistMaxDiv) return -1;
      div[nd++] = factorial_d(occ[i]);
    }
  return nd;
}

static void particle_list(const int32_t* occ, int m, uint8_t* out) {
  int p = 0;
  for (int i = 0; i < m; ++i)
    for (int c = 0; c < occ[i]; ++c) out[p++] = (uint8_t)i;
}

template <int L>
static cudaError_t launch_walk(const double2* V, int m, const int32_t* ve, const uint4* rows, int64_t O, int K, int groups,
                               const double* div, const int* ndiv, const double* mult, double* terms,
                               int sm_count, cudaStream_t s) {
  // chunks of outcomes that leave about 16 warps per SM: a walk is serial (a chunk of
  // 128 takes 80 us), so a few outcomes are spread over more warps
  const int64_t want = O * groups / ((int64_t)sm_count * 16);
  const int chunk = (int)std::min<int64_t>(kWalkChunk, std::max<int64_t>(8, want / 8 * 8));
  const int64_t tasks = (O + chunk - 1) / chunk * groups;
  auto* kernel = ve ? lossy_walk_kernel<L, true> : lossy_walk_kernel<L, false>;
  kernel<<<(unsigned)((tasks + 3) / 4), 128, 0, s>>>(V, m, ve, rows, O, K, groups, div, ndiv, mult, chunk, terms);
  return cudaGetLastError();
}

static cudaError_t launch_walk_l(int l, const double2* V, int m, const int32_t* ve, const uint4* rows, int64_t O, int K, int groups,
                                 const double* div, const int* ndiv, const double* mult, double* terms,
                                 int sms, cudaStream_t s) {
  switch (l) {
    case 1: return launch_walk<1>(V, m, ve, rows, O, K, groups, div, ndiv, mult, terms, sms, s);
    case 2: return launch_walk<2>(V, m, ve, rows, O, K, groups, div, ndiv, mult, terms, sms, s);
    case 3: return launch_walk<3>(V, m, ve, rows, O, K, groups, div, ndiv, mult, terms, sms, s);
    case 4: return launch_walk<4>(V, m, ve, rows, O, K, groups, div, ndiv, mult, terms, sms, s);
    case 5: return launch_walk<5>(V, m, ve, rows, O, K, groups, div, ndiv, mult, terms, sms, s);
    case 6: return launch_walk<6>(V, m, ve, rows, O, K, groups, div, ndiv, mult, terms, sms, s);
    case 7: return launch_walk<7>(V, m, ve, rows, O, K, groups, div, ndiv, mult, terms, sms, s);
    case 8: return launch_walk<8>(V, m, ve, rows, O, K, groups, div, ndiv, mult, terms, sms, s);
    case 9: return launch_walk<9>(V, m, ve, rows, O, K, groups, div, ndiv, mult, terms, sms, s);
    case 10: return launch_walk<10>(V, m, ve, rows, O, K, groups, div, ndiv, mult, terms, sms, s);
    default: return cudaErrorInvalidValue;
  }
}

// The outcomes of the particle counts 1 <= l <= kDistMaxL, grouped: count l's rows
// are first[l] .. first[l] + size[l] - 1 of `occ` (uint8, m per row) and its
// probabilities go to the same places of `prob` (both on the device).
struct SmallGroups {
  const uint8_t* occ;
  double* prob;
  int64_t first[kDistMaxL + 1], size[kDistMaxL + 1];
};

constexpr int64_t kTableBytes = (int64_t)64 << 20;  // the row-sum table of one launch

// Tables and kernels of all groups, queued on the library's stream.
static int queue_small_groups(Context* cx, const double* matrix, int m, int n, const int32_t* initial_state,
                              const SmallGroups& G, float* kernel_ms) {
  std::vector<LossyInputs> LI(kDistMaxL + 1);
  size_t off = 0;
  const size_t o_U = off; off = align256(off + sizeof(double2) * (size_t)m * m);
  const size_t o_fact = off; off = align256(off + sizeof(double) * 256);
  // fixed point if every entry is zero or of a size that has a scale
  bool fixed = true;
  for (size_t i = 0; i < (size_t)2 * m * m; ++i) {
    const double x = std::fabs(matrix[i]);
    fixed = fixed && (x == 0.0 || (x < 1e270 && x > 1e-270));
  }
  size_t o_cols[kDistMaxL + 1], o_div[kDistMaxL + 1], o_ndiv[kDistMaxL + 1], o_mult[kDistMaxL + 1];
  int64_t most_terms = 1, most_O = 1, most_V = 1;
  int st;
  for (int l = 1; l <= kDistMaxL; ++l) {
    if (!G.size[l]) continue;
    if ((st = lossy_inputs(initial_state, m, l, LI[l]))) return st;
    const int64_t K = (int64_t)LI[l].occ.size();
    o_cols[l] = off; off = align256(off + (size_t)K * l);
    o_div[l] = off; off = align256(off + sizeof(double) * (size_t)K * kDistMaxDiv);
    o_ndiv[l] = off; off = align256(off + sizeof(int) * (size_t)K);
    o_mult[l] = off; off = align256(off + sizeof(double) * (size_t)K);
    most_terms = std::max(most_terms, K * G.size[l]);
    most_O = std::max(most_O, G.size[l]);
    const int64_t combos = ((K << (l - 1)) + 31) / 32 * 32;
    most_V = std::max(most_V, std::min(combos * m, std::max<int64_t>(kTableBytes / 16, (int64_t)m << l) + 32 * m));
  }
  if ((st = ensure(cx->dist[0], off))) return st;
  if ((st = ensure(cx->dist[1], sizeof(double) * (size_t)most_terms))) return st;
  const size_t o_V = align256(sizeof(uint4) * (size_t)most_O), o_ve = o_V + align256(sizeof(double2) * (size_t)most_V);
  if ((st = ensure(cx->gpart, o_ve + sizeof(int32_t) * (size_t)most_V))) return st;
  if ((st = ensure_pinned(cx, off))) return st;
  char* h = (char*)cx->pinned;
  memcpy(h + o_U, matrix, sizeof(double2) * (size_t)m * m);
  double* hf = (double*)(h + o_fact);
  for (int k = 0; k < 256; ++k) hf[k] = factorial_d(k);
  for (int l = 1; l <= kDistMaxL; ++l) {
    if (!G.size[l]) continue;
    const int K = (int)LI[l].occ.size();
    for (int k = 0; k < K; ++k) {
      particle_list(LI[l].occ[k].data(), m, (uint8_t*)(h + o_cols[l]) + (size_t)k * l);
      const int nd = divisors(LI[l].occ[k].data(), m, (double*)(h + o_div[l]) + (size_t)k * kDistMaxDiv);
      if (nd < 0) {
        set_error("too many multiply occupied modes in a lossy input");
        return kErrLimit;
      }
      ((int*)(h + o_ndiv[l]))[k] = nd;
      ((double*)(h + o_mult[l]))[k] = LI[l].mult[k];
    }
  }
  char* d = (char*)cx->dist[0].ptr;
  double* terms = (double*)cx->dist[1].ptr;
  uint4* rows = (uint4*)cx->gpart.ptr;
  double2* V = (double2*)((char*)cx->gpart.ptr + o_V);
  int32_t* ve = fixed ? (int32_t*)((char*)cx->gpart.ptr + o_ve) : nullptr;
  cudaStream_t s = cx->stream;
  cudaError_t e = cudaMemcpyAsync(d, h, off, cudaMemcpyHostToDevice, s);
  if (e != cudaSuccess) return fail_cuda(e, "H2D distribution tables");
  cudaEvent_t e0 = nullptr, e1 = nullptr;
  if (kernel_ms) {
    cudaEventCreate(&e0);
    cudaEventCreate(&e1);
    cudaEventRecord(e0, s);
  }
  for (int l = 1; l <= kDistMaxL && e == cudaSuccess; ++l) {
    const int64_t O = G.size[l];
    if (!O) continue;
    const int K = (int)LI[l].occ.size();
    const uint8_t* occ = G.occ + G.first[l] * m;
    lossy_rows_kernel<<<(unsigned)((O + 127) / 128), 128, 0, s>>>(occ, m, O, rows);
    // inputs in chunks whose table stays below kTableBytes (whole warps of combos)
    const int per_warp = l >= 6 ? 1 : 32 >> (l - 1);  // inputs per group of combos
    const int64_t each = (int64_t)m * 16 << (l >= 6 ? l - 1 : 5);  // table bytes of a group
    const int64_t step = std::max<int64_t>(1, kTableBytes / each) * per_warp;
    for (int64_t k0 = 0; k0 < K && e == cudaSuccess; k0 += step) {
      const int kn = (int)std::min<int64_t>(step, K - k0);
      const int groups = (kn + per_warp - 1) / per_warp;
      const int64_t combos = l >= 6 ? (int64_t)kn << (l - 1) : (int64_t)groups * 32;
      const uint8_t* cols = (const uint8_t*)(d + o_cols[l]) + k0 * l;
      lossy_table_kernel<<<(unsigned)((combos * m + 127) / 128), 128, 0, s>>>((const double2*)(d + o_U), m, l, cols, kn,
                                                                             combos, ve, V);
      e = launch_walk_l(l, V, m, ve, rows, O, kn, groups, (const double*)(d + o_div[l]) + k0 * kDistMaxDiv,
                        (const int*)(d + o_ndiv[l]) + k0, (const double*)(d + o_mult[l]) + k0, terms + k0 * O, cx->sm_count, s);
    }
    lossy_outcome_kernel<<<(unsigned)((O + 127) / 128), 128, 0, s>>>(terms, K, O, m, occ, (const double*)(d + o_fact),
                                                                     factorial_d(l), binom_d(n, l),
                                                                     G.prob + G.first[l]);
    if (e == cudaSuccess) e = cudaGetLastError();
  }
  if (kernel_ms) {
    cudaEventRecord(e1, s);
    if (e == cudaSuccess) e = cudaEventSynchronize(e1);
    float ms = 0.f;
    cudaEventElapsedTime(&ms, e0, e1);
    *kernel_ms += ms;
    cudaEventDestroy(e0);
    cudaEventDestroy(e1);
  }
  return e == cudaSuccess ? kOk : fail_cuda(e, "distribution kernels");
}

// Larger l: one Glynn sweep per (lossy input, outcome) on the sweep engine, the
// same arithmetic on the host.
static int group_large(Context* cx, const double* matrix, int m, int n, int l, const LossyInputs& LI,
                       const std::vector<const int32_t*>& outs, double* prob_out, const std::vector<int>& where) {
  const int K = (int)LI.occ.size();
  const int O = (int)outs.size();
  std::vector<double> terms((size_t)K * O, 0.0);
  std::vector<HostSweep> by_class[kSweepClasses];
  std::vector<size_t> which[kSweepClasses];
  for (int k = 0; k < K; ++k)
    for (int o = 0; o < O; ++o) {
      HostSweep hs;
      bool need = false;
      double2 v = make_double2(0.0, 0.0);
      const int st = plan_permanent(matrix, m, LI.occ[k].data(), outs[o], m, BOSS_GLYNN, hs, need, v);
      if (st) return st;
      const size_t t = (size_t)k * O + o;
      if (need) {
        const int c = sweep_class(hs);
        which[c].push_back(t);
        by_class[c].push_back(std::move(hs));
      } else {
        terms[t] = v.x * v.x + v.y * v.y;
      }
    }
  for (int c = 0; c < kSweepClasses; ++c) {
    if (by_class[c].empty()) continue;
    std::vector<double2> res(by_class[c].size());
    const int st = run_sweeps(cx, by_class[c], false, 1, res.data());
    if (st) return st;
    for (size_t a = 0; a < res.size(); ++a) terms[which[c][a]] = fma(res[a].x, res[a].x, res[a].y * res[a].y);
  }
  double div[kDistMaxDiv];
  for (int k = 0; k < K; ++k) {
    const int nd = divisors(LI.occ[k].data(), m, div);
    if (nd < 0) {
      set_error("too many multiply occupied modes in a lossy input");
      return kErrLimit;
    }
    for (int o = 0; o < O; ++o) {
      double v = terms[(size_t)k * O + o];
      for (int d = 0; d < nd; ++d) v /= div[d];
      terms[(size_t)k * O + o] = v * LI.mult[k];
    }
  }
  const double fl = factorial_d(l), bn = binom_d(n, l);
  for (int o = 0; o < O; ++o) {
    double p = 0.0;
    for (int k = 0; k < K; ++k) p += terms[(size_t)k * O + o];
    p /= fl;
    p /= bn;
    p *= fl;
    const int nd = divisors(outs[o], m, div);
    if (nd < 0) {
      set_error("too many multiply occupied modes in an outcome");
      return kErrLimit;
    }
    for (int d = 0; d < nd; ++d) p /= div[d];
    prob_out[where[o]] = p;
  }
  return kOk;
}

struct SmallLaunch {
  const longlong2* A;
  const int32_t* e0;
  int64_t count;
  double2* out;
};

template <int L>
static cudaError_t launch_small(const SmallLaunch& s, int sm_count, cudaStream_t st) {
  // lanes per permanent: as many as keep the launch below a few blocks per SM, at
  // most a block and at least one sign vector each
  int lg = 0;
  while (lg < 7 && lg < L - 1 && (s.count << (lg + 1)) <= (int64_t)sm_count * 256) ++lg;
  const int64_t threads = s.count << lg;
  small_perm_kernel<L><<<(unsigned)((threads + 127) / 128), 128, 0, st>>>(s.A, s.e0, s.count, lg, s.out);
  return cudaGetLastError();
}

static cudaError_t launch_small_l(int l, const SmallLaunch& a, int sms, cudaStream_t s) {
  switch (l) {
    case 1: return launch_small<1>(a, sms, s);
    case 2: return launch_small<2>(a, sms, s);
    case 3: return launch_small<3>(a, sms, s);
    case 4: return launch_small<4>(a, sms, s);
    case 5: return launch_small<5>(a, sms, s);
    case 6: return launch_small<6>(a, sms, s);
    case 7: return launch_small<7>(a, sms, s);
    case 8: return launch_small<8>(a, sms, s);
    case 9: return launch_small<9>(a, sms, s);
    case 10: return launch_small<10>(a, sms, s);
    default: return cudaErrorInvalidValue;
  }
}

static void particle_modes(const int32_t* occ, int len, uint16_t* out) {
  int p = 0;
  for (int i = 0; i < len; ++i)
    for (int c = 0; c < occ[i]; ++c) out[p++] = (uint16_t)i;
}

// A few permanents: each one's matrix is gathered and scaled on the host (L^2
// entries), and the kernel reads it from, and writes its result to, page-locked
// host memory: one launch and one synchronisation, no copies.  done = false: a row
// has no fixed-point scale, nothing was launched.
constexpr int64_t kFewPerms = 16;
// .. and so are more of them while that is not more work for the host than the launch it
// saves (about 4 us): this many matrix entries, and occupations of one side to look through.
constexpr int64_t kFewEntries = 600, kFewOccupations = 3072;

static int small_perm_few(Context* cx, const double* matrix, int m, int len, const int32_t* S, const int32_t* T,
                          const std::vector<int>* by_l, int64_t total, double2* results, bool& done) {
  constexpr int L = kSmallPermMax;
  done = false;
  const size_t o_e0 = align256(sizeof(longlong2) * L * L * (size_t)total);
  const size_t o_out = o_e0 + align256(sizeof(int32_t) * (size_t)total);
  int st;
  if ((st = ensure_pinned(cx, o_out + sizeof(double2) * (size_t)total))) return st;
  char* h = (char*)cx->pinned;
  int64_t q = 0;
  for (int l = 1; l <= L; ++l) {
    longlong2* M = (longlong2*)h + q * L * L;  // the class's matrices, interleaved as on the GPU
    const int64_t n = (int64_t)by_l[l].size();
    int64_t at = 0;
    for (int k : by_l[l]) {
      uint16_t r[L], c[L];
      particle_modes(T + (size_t)k * len, len, r);
      particle_modes(S + (size_t)k * len, len, c);
      int e0 = 0;
      for (int a = 0; a < l; ++a) {
        double mx = 0.0;
        bool fine = true;
        const double* row = matrix + 2 * (size_t)r[a] * m;
        for (int b = 0; b < l; ++b) {
          const double x = row[2 * c[b]], y = row[2 * c[b] + 1];
          fine = fine && std::isfinite(x) && std::isfinite(y);
          mx = std::max(mx, std::max(std::fabs(x), std::fabs(y)));
        }
        const int fx = fine ? row_fraction_bits(mx, l) : kNoScale;
        if (fx == kNoScale) return kOk;
        const double scale = std::ldexp(1.0, fx);
        for (int b = 0; b < l; ++b)
          M[(b * l + a) * n + at] = longlong2{pack_row(std::llrint(row[2 * c[b]] * scale)),
                                              pack_row(std::llrint(row[2 * c[b] + 1] * scale))};
        e0 -= fx;
      }
      ((int32_t*)(h + o_e0))[q + at] = e0;
      ++at;
    }
    q += n;
  }
  q = 0;
  for (int l = 1; l <= L; ++l) {
    const int64_t c = (int64_t)by_l[l].size();
    if (!c) continue;
    const SmallLaunch s{(longlong2*)h + q * L * L, (int32_t*)(h + o_e0) + q, c, (double2*)(h + o_out) + q};
    const cudaError_t e = launch_small_l(l, s, cx->sm_count, cx->stream);
    if (e != cudaSuccess) return fail_cuda(e, "small permanents");
    q += c;
  }
  const cudaError_t e = cudaStreamSynchronize(cx->stream);
  if (e != cudaSuccess) return fail_cuda(e, "small permanents");
  const double2* out = (const double2*)(h + o_out);
  q = 0;
  for (int l = 1; l <= L; ++l)
    for (int k : by_l[l]) results[k] = out[q++];
  done = true;
  return kOk;
}

static void bytes_of(const int32_t* x, size_t n, uint8_t* out) {  // occupations: at most 255
  for (size_t i = 0; i < n; ++i) out[i] = (uint8_t)x[i];
}

// Entries of the matrices of one pass at most (64 MiB); larger batches take several.
constexpr int64_t kSmallPassEntries = 1 << 22;

int small_perm_batch(Context* cx, const double* matrix, int m, int len, const int32_t* S, const int32_t* T,
                     const std::vector<int>* by_l, double2* results) {
  int64_t first[kSmallPermMax + 2] = {}, entries = 0;  // by particle count
  for (int l = 1; l <= kSmallPermMax; ++l) {
    first[l + 1] = first[l] + (int64_t)by_l[l].size();
    entries += (int64_t)l * l * (int64_t)by_l[l].size();
  }
  const int64_t total = first[kSmallPermMax + 1];
  if (total == 0) return kOk;
  int st;
  if (total <= kFewPerms || (entries <= kFewEntries && total * len <= kFewOccupations)) {
    bool done = false;
    if ((st = small_perm_few(cx, matrix, m, len, S, T, by_l, total, results, done)) || done) return st;
  }
  // Page-locked: U, the occupations (grouped by particle count) and the results, which
  // the kernels read and write there; on the device: the matrices of a pass, and U
  // where the gathers read its entries often.  Making the modes here took longer than
  // the permanents (4000 of 5 particles in 64 modes: 0.69 ms a call).
  const size_t mm = (size_t)m * m, occ = (size_t)len;  // a byte each
  const size_t o_T = align256(sizeof(double2) * mm), o_S = o_T + align256(occ * total);
  const size_t o_out = o_S + align256(occ * total);
  const bool copy = entries > 4096 && entries > 4 * (int64_t)mm;
  const size_t o_A = copy ? align256(sizeof(double2) * mm) : 0;
  const int64_t pass = std::min(entries, kSmallPassEntries);
  const size_t o_e0 = o_A + align256(sizeof(longlong2) * (size_t)pass);
  if ((st = ensure(cx->dist[3], o_e0 + sizeof(int32_t) * (size_t)std::min(total, pass)))) return st;
  if ((st = ensure_pinned(cx, o_out + sizeof(double2) * (size_t)total))) return st;
  char* h = (char*)cx->pinned;
  memcpy(h, matrix, sizeof(double2) * mm);
  int64_t q = 0;
  for (int l = 1; l <= kSmallPermMax; ++l) {
    const std::vector<int>& ks = by_l[l];
    for (size_t i = 0, e; i < ks.size(); i = e) {  // neighbours in the batch in one go
      for (e = i + 1; e < ks.size() && ks[e] == ks[e - 1] + 1;) ++e;
      bytes_of(T + (size_t)ks[i] * len, occ * (e - i), (uint8_t*)h + o_T + q * occ);
      bytes_of(S + (size_t)ks[i] * len, occ * (e - i), (uint8_t*)h + o_S + q * occ);
      q += e - i;
    }
  }
  char* d = (char*)cx->dist[3].ptr;
  longlong2* A = (longlong2*)(d + o_A);
  int32_t* e0 = (int32_t*)(d + o_e0);
  cudaStream_t s = cx->stream;
  cudaError_t e = copy ? cudaMemcpyAsync(d, h, sizeof(double2) * mm, cudaMemcpyHostToDevice, s) : cudaSuccess;
  for (int64_t a = 0, b; a < total && e == cudaSuccess; a = b) {  // permanents a to b - 1
    SmallClasses c = {};
    int64_t left = pass;
    b = a;
    for (int l = 1; l <= kSmallPermMax; ++l) {
      c.first[l] = b - a;
      c.mat[l] = pass - left;
      if (b == std::max(a, first[l])) {  // no smaller count had to stop
        const int64_t n = std::min(first[l + 1] - b, left / (l * l));
        if (n > 0) {
          b += n;
          left -= n * l * l;
        }
      }
    }
    c.first[kSmallPermMax + 1] = b - a;
    small_prepare_kernel<<<(unsigned)((b - a + 3) / 4), 128, 0, s>>>((const double2*)(copy ? d : h), m,
                                                                     (const uint8_t*)h + o_T + a * occ,
                                                                     (const uint8_t*)h + o_S + a * occ, len, c, A, e0);
    e = cudaGetLastError();
    for (int l = 1; l <= kSmallPermMax && e == cudaSuccess; ++l) {
      const int64_t n = c.first[l + 1] - c.first[l];
      if (n == 0) continue;
      const SmallLaunch sl{A + c.mat[l], e0 + c.first[l], n, (double2*)(h + o_out) + a + c.first[l]};
      e = launch_small_l(l, sl, cx->sm_count, s);
    }
  }
  const cudaError_t w = cudaStreamSynchronize(s);
  if (e != cudaSuccess || w != cudaSuccess) return fail_cuda(e != cudaSuccess ? e : w, "small permanents");
  const double2* out = (const double2*)(h + o_out);
  q = 0;
  for (int l = 1; l <= kSmallPermMax; ++l)
    for (int k : by_l[l]) results[k] = out[q++];
  return kOk;
}

// Page-locked staging of the outcomes and their probabilities, apart from the
// context's buffer, which holds the tables.  Grow-only, like the context's.
static DeviceBuffer g_outcome_staging;
static int ensure_outcome_staging(size_t bytes) {
  DeviceBuffer& b = g_outcome_staging;
  if (bytes <= b.bytes) return kOk;
  if (b.ptr) cudaFreeHost(b.ptr);
  b = DeviceBuffer{};
  const cudaError_t e = cudaMallocHost(&b.ptr, bytes);
  if (e != cudaSuccess) {
    b.ptr = nullptr;
    return fail_cuda(e, "cudaMallocHost");
  }
  b.bytes = bytes;
  return kOk;
}

}  // namespace boss

using namespace boss;

extern "C" {

int boss_lossy_probabilities(const double* matrix, int32_t m, const int32_t* initial_state, const int32_t* outcomes,
                             int32_t count, double* probabilities, float* kernel_ms) {
  if (!matrix || !initial_state || (count > 0 && (!outcomes || !probabilities)) || m <= 0 || count < 0) {
    set_error("null pointer or bad size");
    return kErrArg;
  }
  if (m > 256) {
    set_error("at most 256 modes");
    return kErrLimit;
  }
  int n = 0;
  for (int i = 0; i < m; ++i) {
    if (initial_state[i] < 0 || initial_state[i] > 255) {
      set_error("occupations must be in [0, 255]");
      return kErrArg;
    }
    n += initial_state[i];
  }
  if (n > 255) {
    set_error("at most 255 input particles");
    return kErrLimit;
  }
  if (kernel_ms) *kernel_ms = 0.f;
  std::lock_guard<std::mutex> lk(g_api_mutex);
  // (1) every outcome's particle count, by slices on the host's threads
  const int T = count < 20000 ? 1 : 8;
  std::vector<uint8_t> ls(count);
  std::vector<std::vector<int64_t>> tally(T, std::vector<int64_t>(n + 1, 0));
  std::vector<int> bad(T, 0);  // 1: an occupation out of range, 2: too many particles (the first of the slice)
  host_parallel(T, [&](int t) {
    const int64_t lo = (int64_t)count * t / T, hi = (int64_t)count * (t + 1) / T;
    for (int64_t o = lo; o < hi; ++o) {
      const int32_t* x = outcomes + o * m;
      int32_t l = 0;
      uint32_t out = 0;
      for (int i = 0; i < m; ++i) {
        l += x[i] & 255;
        out |= (uint32_t)x[i] & ~255u;
      }
      if (out || l > n) {
        bad[t] = out ? 1 : 2;
        return;
      }
      ls[o] = (uint8_t)l;
      ++tally[t][l];
    }
  });
  for (int t = 0; t < T; ++t)
    if (bad[t]) {
      set_error(bad[t] == 1 ? "occupations must be in [0, 255]" : "an outcome holds more particles than the initial state");
      return kErrArg;
    }
  std::vector<int64_t> size(n + 1, 0);
  for (int t = 0; t < T; ++t)
    for (int l = 0; l <= n; ++l) size[l] += tally[t][l];
  // (2) the counts up to kDistMaxL: rows grouped by count in page-locked memory, one
  // copy up, all kernels, one copy down
  SmallGroups G{};
  std::vector<int64_t> first(n + 1, 0);
  int64_t total = 0;
  for (int l = 1; l <= std::min(n, kDistMaxL); ++l) {
    first[l] = total;
    G.first[l] = total;
    G.size[l] = size[l];
    total += size[l];
  }
  // where slice t's outcomes of count l start among the grouped rows
  std::vector<std::vector<int64_t>> start(T, std::vector<int64_t>(n + 1, 0));
  for (int l = 1; l <= n; ++l)
    for (int64_t t = 0, at = first[l]; t < T; ++t) {
      start[t][l] = at;
      at += tally[t][l];
    }
  int st = kOk;
  Context* cx = nullptr;
  if (total > 0) {
    if (!(cx = context(&st))) return st;
    const size_t o_prob = align256((size_t)total * m);
    if ((st = ensure(cx->dist[2], o_prob + sizeof(double) * (size_t)total))) return st;
    if ((st = ensure_outcome_staging(o_prob + sizeof(double) * (size_t)total))) return st;
    uint8_t* h = (uint8_t*)g_outcome_staging.ptr;
    host_parallel(T, [&](int t) {
      std::vector<int64_t> at = start[t];
      const int64_t lo = (int64_t)count * t / T, hi = (int64_t)count * (t + 1) / T;
      for (int64_t o = lo; o < hi; ++o) {
        const int l = ls[o];
        if (l == 0 || l > kDistMaxL) continue;
        const int32_t* x = outcomes + o * m;
        uint8_t* y = h + at[l]++ * m;
        for (int i = 0; i < m; ++i) y[i] = (uint8_t)x[i];
      }
    });
    uint8_t* d = (uint8_t*)cx->dist[2].ptr;
    G.occ = d;
    G.prob = (double*)(d + o_prob);
    cudaError_t e = cudaMemcpyAsync(d, h, (size_t)total * m, cudaMemcpyHostToDevice, cx->stream);
    if (e != cudaSuccess) return fail_cuda(e, "H2D outcomes");
    if ((st = queue_small_groups(cx, matrix, m, n, initial_state, G, kernel_ms))) {
      cudaStreamSynchronize(cx->stream);  // nothing queued may outlive the call's staging
      return st;
    }
    e = cudaMemcpyAsync(h + o_prob, G.prob, sizeof(double) * (size_t)total, cudaMemcpyDeviceToHost, cx->stream);
    if (e == cudaSuccess) e = cudaStreamSynchronize(cx->stream);
    if (e != cudaSuccess) return fail_cuda(e, "distribution kernels");
    const double* hp = (const double*)(h + o_prob);
    host_parallel(T, [&](int t) {
      std::vector<int64_t> at = start[t];
      const int64_t lo = (int64_t)count * t / T, hi = (int64_t)count * (t + 1) / T;
      for (int64_t o = lo; o < hi; ++o)
        if (ls[o] && ls[o] <= kDistMaxL) probabilities[o] = hp[at[ls[o]]++];
    });
  }
  // (3) no particle: the empty lossy input, perm = 1, every factor 1; larger counts
  // through the sweep engine
  if (size[0])
    for (int64_t o = 0; o < count; ++o)
      if (!ls[o]) probabilities[o] = 1.0;
  for (int l = kDistMaxL + 1; l <= n; ++l) {
    if (!size[l]) continue;
    if (!cx && !(cx = context(&st))) return st;
    std::vector<const int32_t*> outs;
    std::vector<int> where;
    for (int o = 0; o < count; ++o)
      if (ls[o] == l) {
        outs.push_back(outcomes + (size_t)o * m);
        where.push_back(o);
      }
    LossyInputs LI;
    if ((st = lossy_inputs(initial_state, m, l, LI))) return st;
    if ((st = group_large(cx, matrix, m, n, l, LI, outs, probabilities, where))) return st;
  }
  return kOk;
}

}  // extern "C"
