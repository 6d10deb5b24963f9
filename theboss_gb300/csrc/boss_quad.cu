// boss_quad.cu -- four codes per step over pairs of factors (boss_quad.cuh): the
// sweeps with two binary digits and enough factors (kQuadMinFactors,
// kQuadMinMinorFactors).  The templated kernels of boss_sweep_kernels.cuh take the
// others.
//
// Measured (sweeps of 64 permanents, input-side digits): n = 16 89 us, n = 20 1.67 ms, n = 24
// 28.1; with the pairs in 62 bits, which lost weakly coupled networks' digits, 88, 1.41 and
// 24.4.  The benchmark's output-side batch n = 28 120 ms (104).  Bound by fixed latencies
// of one dependent chain a lane at 12 to 16 warps per SM, which more warps do not lessen.
#include <algorithm>

#include "boss_internal.h"
#include "boss_quad.cuh"

namespace boss {

// Blocks of 128 per SM the kernels are compiled for: the state is 20 registers per
// four slots.  Calls of 64 permanents n = 20: 3 blocks 1.82 ms, 4 blocks (spills) 1.88; n = 24
// 29.1 and 30.3; 8 of n = 28: 3 blocks 73.1 ms, 2 blocks 78.4 (every product shifted then).
constexpr int quad_blocks(int slots) { return slots <= 4 ? 5 : slots <= 8 ? 4 : 3; }

// A lane's slots are 4 i + (lane & 3) of its walker, i = 0 .. ceil(S / 4) - 1, their
// state in registers (lanes past the last slot repeat it, so that no lane
// branches).  Shared memory, two buffers for the slots' four values on their way to
// the chains' lanes, 16-byte entries, value v of thread t at [v * kQuadXStride + t]
// (the odd stride puts a walker's four readers in different banks).  Their exponents
// stay with the slots' lanes, summed, two 16-bit sums a register (low + 2^16 high).
constexpr int kQuadXStride = kQuadBlock + 1;
constexpr int kQuadX = 4 * kQuadXStride;
template <int S>
struct QuadState {
  static constexpr int kRounds = (S + 3) / 4;
  Cx64 v[kRounds][4];  // o_f o_g E+ E-
  __device__ __forceinline__ static int slot(int i) {
    const int s = 4 * i + (int)(threadIdx.x & 3);
    return 4 * i + 4 <= S ? s : min(s, S - 1);
  }
};

// A pair's state moved by sg times its entries of a row.
__device__ __forceinline__ void quad_move(Cx64 (&v)[4], const longlong2* __restrict__ row, int sg) {
  const int4 low = __ldg(reinterpret_cast<const int4*>(row + 4));
#pragma unroll
  for (int c = 0; c < 4; ++c) {
    const longlong2 d = __ldg(row + c);
    v[c].re = add_packed(v[c].re, d.x, sg);
    v[c].im = add_packed(v[c].im, d.y, sg);
  }
  v[2].fr += sg * low.x;
  v[2].fi += sg * low.y;
  v[3].fr += sg * low.z;
  v[3].fi += sg * low.w;
}

// Two of a pair's values, 2 half and 2 half + 1, formed from its factors, in place (con: the
// pair's constants); returns their exponents as one pair.
__device__ __forceinline__ int quad_redo(longlong2* vals, int half, const longlong2* __restrict__ con, Cx64 of, Cx64 og) {
  const longlong2 f = __ldg(con + 3 + half), g = __ldg(con + 5 + half);
  Cx64 q[2];
  int l[2];
  quad_small(of, og, cx(f.x, f.y), cx(g.x, g.y), q, l);
#pragma unroll
  for (int k = 0; k < 2; ++k) vals[(2 * half + k) * kQuadXStride] = make_longlong2(q[k].re, q[k].im);
  return l[0] + l[1] * 65536;
}

// The walk at outer code t, and this lane's state.
template <int S>
__device__ __forceinline__ void quad_decode(const SweepProblem& P, const longlong2* __restrict__ rows,
                                            const longlong2* __restrict__ base, uint64_t t, QuadState<S>& st, QuadWalk& k) {
  constexpr int W = kQuadRow * S;
  const int nb = P.nb;
  quad_walk_at(P, t, k);
#pragma unroll
  for (int i = 0; i < QuadState<S>::kRounds; ++i) {
    const longlong2* b = base + kQuadRow * QuadState<S>::slot(i);
    const int4 low = *reinterpret_cast<const int4*>(b + 4);
    st.v[i][0] = cx(b[0].x, b[0].y);
    st.v[i][1] = cx(b[1].x, b[1].y);
    st.v[i][2] = Cx64{b[2].x, b[2].y, low.x, low.y};
    st.v[i][3] = Cx64{b[3].x, b[3].y, low.z, low.w};
  }
  auto add = [&](int d, int sg) {
#pragma unroll
    for (int i = 0; i < QuadState<S>::kRounds; ++i)
      quad_move(st.v[i], rows + (int64_t)d * W + kQuadRow * QuadState<S>::slot(i), sg);
  };
  for (uint64_t bits = k.g; bits; bits &= bits - 1ull) add(__ffsll((long long)bits) - 1, -2);
  for (int d = nb; d < P.nd; ++d)
    if (k.r[d]) add(d, -2 * (int)k.r[d]);
}

// Moves the state by sg times a row (sg = 0: as it is) and multiplies this lane's
// code over S slots: the product is (re + i im) 2^e.  Every lane of the warp calls
// it.  The next round's slots are prepared beside the chains of the one before.
template <int S>
__device__ __forceinline__ void quad_eval(QuadState<S>& st, longlong2* xbuf, const longlong2* __restrict__ row, int sg,
                                          const longlong2* __restrict__ consts, int e0, long long& re, long long& im,
                                          int& e) {
  constexpr int kRounds = (S + 3) / 4;
  const int kk = threadIdx.x & 3;
  int2 ls = make_int2(0, 0);  // exponents of this lane's values
  const int from = kk * kQuadXStride + (threadIdx.x & ~3);
  int ps = 0;  // and of its chain
  auto prepare = [&](int i) {
    const int s = QuadState<S>::slot(i), at = (i & 1) * kQuadX + (int)threadIdx.x;
    const longlong2* con = consts + kQuadConst * s;
    const longlong2 cp = __ldg(con), cm = __ldg(con + 1);
    const int4 low = __ldg(reinterpret_cast<const int4*>(con + 2));
    Cx64(&v)[4] = st.v[i];
    quad_move(v, row + kQuadRow * s, sg);
    Cx64 q[4];
    int l[4];
    const int least = quad_values(v[0], v[1], v[2], v[3], Cx64{cp.x, cp.y, low.x, low.y}, Cx64{cm.x, cm.y, low.z, low.w}, q, l);
#pragma unroll
    for (int c = 0; c < 4; ++c) xbuf[at + c * kQuadXStride] = make_longlong2(q[c].re, q[c].im);
    int2 lv = make_int2(l[0] + l[1] * 65536, l[2] + l[3] * 65536);
    if (least < kQuadLeast) {  // rare but for weakly coupled modes: the half of the values that has the small one
      const int half = min(l[0], l[1]) < kQuadLeast ? 0 : 1;
      const bool both = half == 0 && min(l[2], l[3]) < kQuadLeast;
#pragma unroll 1
      for (int h = half; h <= (both ? 1 : half); ++h) {
        const int x = quad_redo(xbuf + at, h, con, v[0], v[1]);
        lv = h ? make_int2(lv.x, x) : make_int2(x, lv.y);
      }
    }
    if (4 * i + 4 <= S || 4 * i + kk < S) ls = make_int2(ls.x + lv.x, ls.y + lv.y);
  };
  prepare(0);
  __syncwarp();
#pragma unroll
  for (int i = 0; i < kRounds; ++i) {
    if (i + 1 < kRounds) prepare(i + 1);
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      if (4 * i + j >= S) break;
      const longlong2 q = xbuf[(i & 1) * kQuadX + from + j];
      const int n = 4 * i + j;
      ps += n == 0 ? quad_chain_first(re, im, q.x, q.y)
            : n % 2 ? quad_chain_raw(re, im, q.x, q.y)
                    : quad_chain(re, im, q.x, q.y);
    }
    __syncwarp();
  }
#pragma unroll
  for (int o = 1; o < 4; o <<= 1) {
    ls.x += __shfl_xor_sync(0xffffffffu, ls.x, o);
    ls.y += __shfl_xor_sync(0xffffffffu, ls.y, o);
  }
  const int l = (kk & 2) ? ls.y : ls.x, low = (short)l;  // the sum of this chain's values
  e = quad_exponent(e0, (kk & 1) ? (l - low) >> 16 : low, S) + ps;
}

// A lane's sum is closed every so many steps: a sum of the benchmark's 10^5 codes a lane
// in one piece rounds by its own growth (n = 30 in a batch of 64: 5.7e-13 off; closed
// every 1024, 256, 64 steps 9e-14, 1.8e-13, 1.0e-13).
constexpr int64_t kQuadSettle = 64;

// One permanent per sweep problem; every group of walkers writes one complex partial.
template <int S>
__global__ void __launch_bounds__(kQuadBlock, quad_blocks(S)) perm_quad_kernel(const SweepProblem* __restrict__ probs,
                                                                        int n_probs,
                                                                        const longlong2* __restrict__ pool,
                                                                        int64_t total_walkers,
                                                                        double2* __restrict__ partials) {
  extern __shared__ longlong2 quad_smem[];
  const int64_t at = (int64_t)blockIdx.x * kQuadWalkers + (threadIdx.x >> 2);
  const bool live = at < total_walkers;
  const int64_t walker = live ? at : total_walkers - 1;
  const SweepProblem& P = probs[find_problem(probs, n_probs, walker)];
  const QuadRange R = quad_range(P, walker, live);
  constexpr int W = kQuadRow * S;
  const longlong2* rows = pool + P.mat_off;
  const longlong2* base = pool + P.base_off;
  QuadState<S> st;
  QuadWalk k;
  quad_decode<S>(P, rows, base, (uint64_t)(R.len > 0 ? R.a : 0), st, k);
  // sign of this lane's code: + for (+,+) and (-,-), - for the mixed ones
  const uint32_t mixed = (threadIdx.x >> 1) & 1u;
  double ar = 0.0, ai = 0.0;  // since the last settling; before, in shared memory:
  double2* total = reinterpret_cast<double2*>(quad_smem + (S > 4 ? 2 : 1) * kQuadX) + threadIdx.x;
  *total = make_double2(0.0, 0.0);
  const longlong2* row = base;
  int sg = 0;
  for (int64_t it = 0; it < R.most; ++it) {
    if (it > 0 && it < R.len) {
      int dr;
      row = rows + (int64_t)quad_next(P, (uint64_t)(R.a + it), k, dr) * W;
      sg = -2 * dr;
    }
    if (it >= R.len) sg = 0;
    long long re, im;
    int e;
    quad_eval<S>(st, quad_smem, row, sg, base + W, P.fx, re, im, e);
    const double w = it < R.len ? xor_sign(k.w, (k.parity ^ mixed) << 31) : 0.0;
    ar = fma(w, bf_to_double(re, e), ar);
    ai = fma(w, bf_to_double(im, e), ai);
    if ((it & (kQuadSettle - 1)) == kQuadSettle - 1) {
      const double2 v = *total;
      *total = make_double2(v.x + ar, v.y + ai);
      ar = ai = 0.0;
    }
  }
  ar += total->x;
  ai += total->y;
  const int G = P.group;  // 1, 2, 4 or 8 walkers (one warp at most), the same for the whole launch
  for (int o = 1; o < 4 * G; o <<= 1) {  // the walkers' codes, in a fixed order
    ar += __shfl_xor_sync(0xffffffffu, ar, o);
    ai += __shfl_xor_sync(0xffffffffu, ai, o);
  }
  if (live && (threadIdx.x & (4 * G - 1)) == 0) partials[P.part_off + R.q / G] = make_double2(ar, ai);
}

// All-minors in Glynn form (see minors_walk): half of every minor, row order low
// digits, outer digits, held digit.  A lane's code has fixed low digits, so the low
// digits' minors are +- its total; an outer digit's weight w_j = mult_j - 2 r_j
// changes by -+2 when the digit moves, so its row then takes +-R, R the lane's
// running total of signed and weighted products, and w_j R / 2 when the total is
// closed (every 2^16 steps and at the end).
template <int S>
__global__ void __launch_bounds__(kQuadBlock, quad_blocks(S)) minors_quad_kernel(const SweepProblem* __restrict__ probs,
                                                                          int n_probs,
                                                                          const longlong2* __restrict__ pool,
                                                                          int64_t total_walkers,
                                                                          double2* __restrict__ partials,
                                                                          int64_t uniform_walkers) {
  extern __shared__ longlong2 quad_smem[];
  const int64_t at = (int64_t)blockIdx.x * kQuadWalkers + (threadIdx.x >> 2);
  const bool live = at < total_walkers;
  const int64_t walker = live ? at : total_walkers - 1;
  const SweepProblem& P =
      probs[uniform_walkers > 0 ? (int)(walker / uniform_walkers) : find_problem(probs, n_probs, walker)];
  const QuadRange R = quad_range(P, walker, live);
  constexpr int W = kQuadRow * S;
  const int ndo = P.nd, nb = P.nb;
  const longlong2* rows = pool + P.mat_off;
  const longlong2* base = pool + P.base_off;
  QuadState<S> st;
  double2 M[kMaxMinorDigits];  // outer digits' rows (local memory: row i is touched when digit i moves)
  for (int j = 0; j < ndo; ++j) M[j] = make_double2(0.0, 0.0);
  double hr = 0.0, hi = 0.0;   // half of the lane's total
  QuadWalk k;
  quad_decode<S>(P, rows, base, (uint64_t)(R.len > 0 ? R.a : 0), st, k);
  const uint32_t mixed = (threadIdx.x >> 1) & 1u;
  double Rr = 0.0, Ri = 0.0;  // since the last settle
  auto settle = [&]() {
    const double wr = 0.5 * Rr, wi = 0.5 * Ri;
    for (int j = 0; j < ndo; ++j) {
      const double f = j < nb ? (((k.g >> j) & 1ull) ? -1.0 : 1.0) : (double)P.mult[j] - 2.0 * (double)k.r[j];
      M[j].x = fma(wr, f, M[j].x);
      M[j].y = fma(wi, f, M[j].y);
    }
    hr += wr;
    hi += wi;
    Rr = Ri = 0.0;
  };
  const longlong2* row = base;
  int sg = 0;
  for (int64_t it = 0; it < R.most; ++it) {
    if (it > 0 && it < R.len) {
      if ((it & ((1ll << kSegLog) - 1ll)) == 0) settle();
      int dr;
      const int i = quad_next(P, (uint64_t)(R.a + it), k, dr);
      const uint32_t neg = (uint32_t)dr & 0x80000000u;  // the digit goes down: -R
      double2 m = M[i];
      m.x += xor_sign(Rr, neg);
      m.y += xor_sign(Ri, neg);
      M[i] = m;
      row = rows + (int64_t)i * W;
      sg = -2 * dr;
    }
    if (it >= R.len) sg = 0;
    long long re, im;
    int e;
    quad_eval<S>(st, quad_smem, row, sg, base + W, P.fx, re, im, e);
    const double w = it < R.len ? xor_sign(k.w, (k.parity ^ mixed) << 31) : 0.0;
    Rr = fma(w, bf_to_double(re, e), Rr);
    Ri = fma(w, bf_to_double(im, e), Ri);
  }
  settle();
  // Each aligned group of G walkers (4 G lanes) sums its rows through the block's
  // shared memory (every warp done with its buffers): component c of row j of thread t at
  // smem[(2 j + c) * kQuadBlock + t].  The group's lanes take the components in turn,
  // each in a fixed, staggered order (fewer bank conflicts).
  const int nd = ndo + 2 + P.fixed_digit, G = max(P.group, 1), GL = 4 * G;
  double* ms = reinterpret_cast<double*>(quad_smem);
  __syncthreads();  // the rows lie across other warps' buffers
  {
    const int kk = threadIdx.x & 3;
    const uint32_t n0 = (kk == 1 || kk == 3) ? 0x80000000u : 0u;  // d0 = -1
    const uint32_t n1 = (kk == 1 || kk == 2) ? 0x80000000u : 0u;  // d1 = -1
    double* o = ms + threadIdx.x;
    o[0] = xor_sign(hr, n0);
    o[kQuadBlock] = xor_sign(hi, n0);
    o[2 * kQuadBlock] = xor_sign(hr, n1);
    o[3 * kQuadBlock] = xor_sign(hi, n1);
    for (int j = 0; j < ndo; ++j) {
      const double2 m = M[j];
      o[(4 + 2 * j) * kQuadBlock] = m.x;
      o[(5 + 2 * j) * kQuadBlock] = m.y;
    }
    if (P.fixed_digit) {
      o[(4 + 2 * ndo) * kQuadBlock] = hr;
      o[(5 + 2 * ndo) * kQuadBlock] = hi;
    }
  }
  if (GL > 32) __syncthreads(); else __syncwarp();  // a group's rows are its own columns
  const int gl = threadIdx.x & (GL - 1);
  const double* grp = ms + (threadIdx.x - gl);
  double* out = reinterpret_cast<double*>(partials + P.part_off + (R.q / G) * nd);
  for (int c = gl; c < 2 * nd; c += GL) {
    const double* col = grp + c * kQuadBlock;
    double s = 0.0;
    for (int i = 0; i < GL; ++i) s += col[(i + gl) & (GL - 1)];
    if (live) out[c] = s;
  }
}

// rows: of minors; 0: permanents, whose lanes keep a sum each behind the buffers.
static size_t quad_smem_bytes(int slots, int rows) {
  const int x = (slots > 4 ? 2 : 1) * kQuadX;
  return sizeof(longlong2) * (size_t)(rows > 0 ? std::max(x, rows * kQuadBlock) : x + kQuadBlock);
}

constexpr int kQuadMaxSlots = (kMaxFactors + 1) / 2;
using PermQuad = void (*)(const SweepProblem*, int, const longlong2*, int64_t, double2*);
using MinorsQuad = void (*)(const SweepProblem*, int, const longlong2*, int64_t, double2*, int64_t);
static const PermQuad kPermQuad[kQuadMaxSlots + 1] = {
    nullptr,           perm_quad_kernel<1>,  perm_quad_kernel<2>,  perm_quad_kernel<3>,  perm_quad_kernel<4>,
    perm_quad_kernel<5>,  perm_quad_kernel<6>,  perm_quad_kernel<7>,  perm_quad_kernel<8>,  perm_quad_kernel<9>,
    perm_quad_kernel<10>, perm_quad_kernel<11>, perm_quad_kernel<12>, perm_quad_kernel<13>, perm_quad_kernel<14>,
    perm_quad_kernel<15>, perm_quad_kernel<16>};
static const MinorsQuad kMinorsQuad[kQuadMaxSlots + 1] = {
    nullptr,           minors_quad_kernel<1>,  minors_quad_kernel<2>,  minors_quad_kernel<3>,  minors_quad_kernel<4>,
    minors_quad_kernel<5>,  minors_quad_kernel<6>,  minors_quad_kernel<7>,  minors_quad_kernel<8>,  minors_quad_kernel<9>,
    minors_quad_kernel<10>, minors_quad_kernel<11>, minors_quad_kernel<12>, minors_quad_kernel<13>, minors_quad_kernel<14>,
    minors_quad_kernel<15>, minors_quad_kernel<16>};

static int g_quad_occ[2][kQuadMaxSlots + 1][kMaxMinorDigits + 1];

cudaError_t prepare_quad_kernels() {
  cudaError_t e;
  for (int s = 1; s <= kQuadMaxSlots; ++s) {
    const int most = (int)quad_smem_bytes(s, kMaxMinorDigits);
    if ((e = cudaFuncSetAttribute(kPermQuad[s], cudaFuncAttributeMaxDynamicSharedMemorySize, most))) return e;
    if ((e = cudaFuncSetAttribute(kMinorsQuad[s], cudaFuncAttributeMaxDynamicSharedMemorySize, most))) return e;
    for (int rows = 0; rows <= kMaxMinorDigits; ++rows) {
      int* occ[2] = {&g_quad_occ[0][s][rows], &g_quad_occ[1][s][rows]};
      const size_t b = quad_smem_bytes(s, rows);
      if (rows > 0 && b == quad_smem_bytes(s, rows - 1)) {  // the same block as before
        *occ[0] = occ[0][-1];
        *occ[1] = occ[1][-1];
        continue;
      }
      if ((e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(occ[0], kPermQuad[s], kQuadBlock, b))) return e;
      if ((e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(occ[1], kMinorsQuad[s], kQuadBlock, b))) return e;
    }
  }
  return cudaSuccess;
}

int64_t quad_resident_walkers(int nf, int rows, bool minors, int sm_count) {
  if (nf < 2 || nf > kMaxFactors) return kQuadWalkers;
  rows = minors ? std::min(std::max(rows, 0), kMaxMinorDigits) : 0;
  return (int64_t)std::max(1, g_quad_occ[minors ? 1 : 0][quad_slots(nf)][rows]) * sm_count * kQuadWalkers;
}

cudaError_t launch_quad_sweep(int nf, bool minors, const SweepLaunch& L, cudaStream_t st) {
  const unsigned grid = (unsigned)((L.total_threads + kQuadWalkers - 1) / kQuadWalkers);
  const int s = quad_slots(nf);
  if (minors)
    kMinorsQuad[s]<<<grid, kQuadBlock, quad_smem_bytes(s, L.rows), st>>>(L.probs, L.n_probs, L.pool, L.total_threads,
                                                                         L.partials, L.uniform_threads);
  else
    kPermQuad[s]<<<grid, kQuadBlock, quad_smem_bytes(s, 0), st>>>(L.probs, L.n_probs, L.pool, L.total_threads,
                                                                  L.partials);
  return cudaGetLastError();
}

}  // namespace boss
