// boss_grad.cu -- permanents with all their derivatives (Glynn's sum).
//
// With s_f the factors and w_b = mult_b - 2 r_b a digit's weight,
//     d perm / d U[mode f][mode b] = scale sum over the mode's copies f of
//     G_{b,f} = sum_r sign(r) prod C(mult, r) w_b(r) L_f(r),  L_f = prod_{f' != f} s_f'.
// w_b changes only when digit b moves, by -+2, so a running total R_f of the signed
// and weighted L_f is kept, a move of digit b adds +-2 R_. to its row G_b, and at
// the end every row takes w_b R_. (the held digit, weight 1, last).
//
// GB300 mapping.  In FP64 the three products per factor and code (prefix, suffix,
// their product) hold the FP64 pipe for 12 of the 14 instructions per factor; here
// they run on the integer pipe in block floating point (boss_sweep.cuh) and only R
// and G stay FP64: 4 instructions per factor and code.  Four lanes share a walker
// (boss_quad.cuh): lane k has factors 4 i + k, i < M = ceil(nf / 4) (padded with the
// constant 1), their sums, its suffix products and its R in registers.  A lane
// multiplies its own factors, the other three lanes' product comes from two
// shuffled products, and its leave-one-out products from a prefix that starts
// there.  No shared memory, 12 to 20 warps per SM.
//
// G lives in global memory, one slice per warp, entry (row * M + i) * 32 + lane, so
// that a warp whose walkers move the same digit (ranges are aligned, range_align)
// updates whole lines; a row is first written, not added to, when first touched.
#include <algorithm>

#include "boss_internal.h"
#include "boss_quad.cuh"

namespace boss {

struct GradMant {  // (re + i im) 2^e, normal (bf_renorm)
  long long re, im;
  int e;
};
__device__ __forceinline__ GradMant grad_norm(Cx64 s) {  // of a factor's sum (fully where |s| >= 2^32)
  GradMant r{s.re, s.im, 0};
  r.e = bf_renorm(r.re, r.im) - 29;
  return r;
}
__device__ __forceinline__ GradMant grad_mul(const GradMant& a, const GradMant& b) {
  GradMant r;
  bf_mul_high(a.re, a.im, b.re, b.im, r.re, r.im);
  r.e = a.e + b.e + 35 + bf_renorm(r.re, r.im);
  return r;
}
__device__ __forceinline__ GradMant grad_last(const GradMant& a, const GradMant& b) {  // a product that is only converted
  GradMant r;
  bf_mul_high(a.re, a.im, b.re, b.im, r.re, r.im);
  r.e = a.e + b.e + 64;
  return r;
}
__device__ __forceinline__ GradMant grad_from(const GradMant& a, int o) {  // lane ^ o's
  GradMant r;
  r.re = __shfl_xor_sync(0xffffffffu, a.re, o);
  r.im = __shfl_xor_sync(0xffffffffu, a.im, o);
  r.e = __shfl_xor_sync(0xffffffffu, a.e, o);
  return r;
}

// Layout of a sweep in the pool: rows, one per digit, F = 4 M packed entries u (factor
// f at f); base, F sums at r = 0 (2^61, the constant 1, for the padding); F int32
// fraction bits.  P.fx: minus their sum.
template <int M>
__global__ void __launch_bounds__(128, M <= 3 ? 5 : M <= 5 ? 4 : 3) grad_sweep_kernel(
    const SweepProblem* __restrict__ probs, int n_probs, const longlong2* __restrict__ pool, int64_t total_walkers,
    double2* __restrict__ gpart, double2* __restrict__ ppart) {
  constexpr int F = 4 * M;
  const int64_t at = (int64_t)blockIdx.x * kQuadWalkers + (threadIdx.x >> 2);
  const bool live = at < total_walkers;
  const int64_t walker = live ? at : total_walkers - 1;
  const SweepProblem& P = probs[find_problem(probs, n_probs, walker)];
  const QuadRange Q = quad_range(P, walker, live);
  const int kk = threadIdx.x & 3, lane = threadIdx.x & 31;
  const int nd = P.nd, nb = P.nb, ndt = P.nd + P.fixed_digit;
  const longlong2* rows = pool + P.mat_off;
  const longlong2* base = pool + P.base_off;
  const int32_t* fxs = reinterpret_cast<const int32_t*>(base + F);
  double2* G = gpart + P.part_off + (Q.q >> 3) * ((int64_t)ndt * M * 32) + lane;
  QuadWalk k;
  quad_walk_at(P, (uint64_t)(Q.len > 0 ? Q.a : 0), k);
  Cx64 s[M];
  int fx[M];
#pragma unroll
  for (int i = 0; i < M; ++i) {
    const longlong2 b = base[4 * i + kk];
    s[i] = cx(b.x, b.y);
    fx[i] = fxs[4 * i + kk];
  }
  auto move = [&](int d, int sg) {
    const longlong2* row = rows + (int64_t)d * F + kk;
#pragma unroll
    for (int i = 0; i < M; ++i) {
      const longlong2 u = __ldg(row + 4 * i);
      s[i] = cx(add_packed(s[i].re, u.x, sg), add_packed(s[i].im, u.y, sg));
    }
  };
  for (uint64_t bits = k.g; bits; bits &= bits - 1ull) move(__ffsll((long long)bits) - 1, -2);
  for (int d = nb; d < nd; ++d)
    if (k.r[d]) move(d, -2 * (int)k.r[d]);
  double2 R[M];
#pragma unroll
  for (int i = 0; i < M; ++i) R[i] = make_double2(0.0, 0.0);
  double pr = 0.0, pi = 0.0;
  uint64_t touched = 0;
  for (int64_t it = 0; it < Q.most; ++it) {
    if (it > 0 && it < Q.len) {
      int dr;
      const int b = quad_next(P, (uint64_t)(Q.a + it), k, dr);
      const double c = 2.0 * dr;  // w_b goes down by 2 when r goes up
      double2* Gb = G + (int64_t)b * M * 32;
      if ((touched >> b) & 1ull) {
#pragma unroll
        for (int i = 0; i < M; ++i) {
          double2 g = Gb[i * 32];
          g.x = fma(c, R[i].x, g.x);
          g.y = fma(c, R[i].y, g.y);
          Gb[i * 32] = g;
        }
      } else {
        touched |= 1ull << b;
#pragma unroll
        for (int i = 0; i < M; ++i) Gb[i * 32] = make_double2(c * R[i].x, c * R[i].y);
      }
      move(b, -2 * dr);
    }
    // suffixes within the lane, the lane's product, the other lanes'
    int least = 0;
    GradMant n[M], suf[M];  // the factors; suf[i]: factors after i of this lane (i < M - 1)
#pragma unroll
    for (int i = 0; i < M; ++i) {
      n[i] = grad_norm(s[i]);
      least = min(least, n[i].e);
    }
    if (least < -29) {  // rare: a factor below 2^32
#pragma unroll
      for (int i = 0; i < M; ++i) {
        const BFloat z = bf_norm(s[i].re, s[i].im, 0);
        n[i] = GradMant{z.re, z.im, z.e};
      }
    }
    GradMant A = n[M - 1];
#pragma unroll
    for (int i = M - 2; i >= 0; --i) {
      suf[i] = A;
      A = grad_mul(A, n[i]);
    }
    const GradMant A1 = grad_from(A, 1);
    const GradMant B = grad_mul(A, A1);
    GradMant pre = grad_mul(A1, grad_from(B, 2));
    const double w = it < Q.len ? xor_sign(k.w, k.parity << 31) : 0.0;
#pragma unroll
    for (int i = 0; i < M; ++i) {
      const GradMant L = i < M - 1 ? grad_last(pre, suf[i]) : pre;
      const int e = L.e + P.fx + fx[i];
      R[i].x = fma(w, bf_to_double(L.re, e), R[i].x);
      R[i].y = fma(w, bf_to_double(L.im, e), R[i].y);
      pre = grad_mul(pre, n[i]);
    }
    pr = fma(w, bf_to_double(pre.re, pre.e + P.fx), pr);
    pi = fma(w, bf_to_double(pre.im, pre.e + P.fx), pi);
  }
  for (int b = 0; b < ndt && live; ++b) {
    const double w = b < nb ? (((k.g >> b) & 1ull) ? -1.0 : 1.0)
                            : b < nd ? (double)P.mult[b] - 2.0 * (double)k.r[b] : 1.0;
    double2* Gb = G + (int64_t)b * M * 32;
    const bool had = b < nd && ((touched >> b) & 1ull);
#pragma unroll
    for (int i = 0; i < M; ++i) {
      const double2 g = had ? Gb[i * 32] : make_double2(0.0, 0.0);
      Gb[i * 32] = make_double2(fma(w, R[i].x, g.x), fma(w, R[i].y, g.y));
    }
  }
  // the warp's permanents: every lane of a walker has it; walkers in a fixed order
#pragma unroll
  for (int o = 4; o < 32; o <<= 1) {
    pr += __shfl_xor_sync(0xffffffffu, pr, o);
    pi += __shfl_xor_sync(0xffffffffu, pi, o);
  }
  if (live && lane == 0) ppart[walker >> 3] = make_double2(pr, pi);
}

// Sums of the warps' slices: block (sweep, 64 entries, part z of the walkers), entry
// e = (row * M + i) * 4 + lane & 3 by four threads, each every fourth walker of the
// part in order, then the four.  Bound by reading the slices; few sweeps fill the GPU
// only if a sweep's walkers are split over blocks (one gradient at n = 18: 312 us with
// one part, 154 with 51, of which most is the sweep).  One part writes the gradients and permanents, several
// write gridDim.z rows of row_stride + 1 sums a sweep (the permanent's last) to grad_out.
__global__ void __launch_bounds__(256) grad_reduce_kernel(const SweepProblem* __restrict__ probs,
                                                          const double2* __restrict__ gpart,
                                                          const double2* __restrict__ ppart,
                                                          double2* __restrict__ grad_out,
                                                          double2* __restrict__ perm_out, int row_stride, int F) {
  __shared__ double2 sum[256];
  const SweepProblem& P = probs[blockIdx.x];
  const int ne = (P.nd + P.fixed_digit) * F;
  const int64_t warps = P.n_threads >> 3, slice = (int64_t)ne * 8;
  const int parts = (int)gridDim.z;
  const int64_t w0 = warps * blockIdx.z / parts, w1 = warps * (blockIdx.z + 1) / parts;
  double2* g_out;
  double2* p_out;
  double scale;
  if (parts == 1) {
    g_out = grad_out + (size_t)P.out_idx * row_stride;
    p_out = perm_out + P.out_idx;
    scale = P.scale;
  } else {
    g_out = grad_out + ((size_t)blockIdx.x * parts + blockIdx.z) * (row_stride + 1);
    p_out = g_out + row_stride;
    scale = 1.0;
  }
  const int part = threadIdx.x >> 6, e = blockIdx.y * 64 + (threadIdx.x & 63);
  double ar = 0.0, ai = 0.0;
  if (e < ne) {
    const double2* g = gpart + P.part_off + (int64_t)(e >> 2) * 32 + (e & 3);
#pragma unroll 8  // independent loads in flight
    for (int64_t q = 8 * w0 + part; q < 8 * w1; q += 4) {
      const double2 v = g[(q >> 3) * slice + 4 * (q & 7)];
      ar += v.x;
      ai += v.y;
    }
  }
  sum[threadIdx.x] = make_double2(ar, ai);
  __syncthreads();
  if (part == 0 && e < ne) {
    for (int p = 1; p < 4; ++p) {
      ar += sum[threadIdx.x + 64 * p].x;
      ai += sum[threadIdx.x + 64 * p].y;
    }
    g_out[e] = make_double2(ar * scale, ai * scale);  // e = row F + 4 i + lane: the factor
  }
  if (blockIdx.y == 0) {
    __syncthreads();
    ar = ai = 0.0;
    for (int64_t q = w0 + threadIdx.x; q < w1; q += 256) {
      const double2 v = ppart[(P.thread_begin >> 3) + q];
      ar += v.x;
      ai += v.y;
    }
    sum[threadIdx.x] = make_double2(ar, ai);
    __syncthreads();
    for (int s = 128; s > 0; s >>= 1) {
      if ((int)threadIdx.x < s) {
        sum[threadIdx.x].x += sum[threadIdx.x + s].x;
        sum[threadIdx.x].y += sum[threadIdx.x + s].y;
      }
      __syncthreads();
    }
    if (threadIdx.x == 0) *p_out = make_double2(sum[0].x * scale, sum[0].y * scale);
  }
}

// The parts' sums: one thread per entry (the permanent's last), the parts in order.
__global__ void __launch_bounds__(128) grad_parts_kernel(const SweepProblem* __restrict__ probs,
                                                         const double2* __restrict__ mid, int parts,
                                                         double2* __restrict__ grad_out,
                                                         double2* __restrict__ perm_out, int row_stride, int F) {
  const SweepProblem& P = probs[blockIdx.x];
  const int e = blockIdx.y * 128 + threadIdx.x, ne = (P.nd + P.fixed_digit) * F;
  if (e > row_stride || (e >= ne && e < row_stride)) return;
  const double2* v = mid + (size_t)blockIdx.x * parts * (row_stride + 1) + e;
  double ar = 0.0, ai = 0.0;
#pragma unroll 8  // independent loads in flight
  for (int z = 0; z < parts; ++z) {
    const double2 x = v[(size_t)z * (row_stride + 1)];
    ar += x.x;
    ai += x.y;
  }
  double2* o = e == row_stride ? perm_out + P.out_idx : grad_out + (size_t)P.out_idx * row_stride + e;
  *o = make_double2(ar * P.scale, ai * P.scale);
}

constexpr int kGradMaxM = kMaxFactors / 4;
using GradKernel = void (*)(const SweepProblem*, int, const longlong2*, int64_t, double2*, double2*);
static const GradKernel kGrad[kGradMaxM + 1] = {nullptr,
                                                grad_sweep_kernel<1>,
                                                grad_sweep_kernel<2>,
                                                grad_sweep_kernel<3>,
                                                grad_sweep_kernel<4>,
                                                grad_sweep_kernel<5>,
                                                grad_sweep_kernel<6>,
                                                grad_sweep_kernel<7>,
                                                grad_sweep_kernel<8>};
static int g_grad_occ[kGradMaxM + 1];

cudaError_t prepare_grad_kernels() {
  for (int m = 1; m <= kGradMaxM; ++m) {
    const cudaError_t e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&g_grad_occ[m], kGrad[m], kQuadBlock, 0);
    if (e != cudaSuccess) return e;
  }
  return cudaSuccess;
}

int64_t grad_resident_walkers(int nf, int sm_count) {
  return (int64_t)std::max(1, g_grad_occ[grad_factors(nf) / 4]) * sm_count * kQuadWalkers;
}

cudaError_t launch_grad_sweep(int nf, const SweepProblem* probs, int n_probs, const longlong2* pool, int64_t walkers,
                              double2* gpart, double2* ppart, cudaStream_t st) {
  if (nf < 1 || nf > kMaxFactors) return cudaErrorInvalidValue;
  if (walkers <= 0) return cudaSuccess;
  kGrad[grad_factors(nf) / 4]<<<(unsigned)((walkers + kQuadWalkers - 1) / kQuadWalkers), kQuadBlock, 0, st>>>(
      probs, n_probs, pool, walkers, gpart, ppart);
  return cudaGetLastError();
}

int grad_reduce_parts(int64_t walkers, int n_probs, int row_stride, int sm_count) {
  const int64_t blocks = (int64_t)n_probs * ((row_stride + 63) / 64);
  const int64_t fill = (2 * sm_count + blocks - 1) / blocks;
  return (int)std::max<int64_t>(1, std::min<int64_t>(fill, walkers / n_probs / 128));
}

cudaError_t launch_grad_reduce(int nf, const SweepProblem* probs, int n_probs, const double2* gpart,
                               const double2* ppart, double2* mid, int parts, double2* grad_out, double2* perm_out,
                               int row_stride, cudaStream_t st) {
  if (n_probs <= 0) return cudaSuccess;
  grad_reduce_kernel<<<dim3((unsigned)n_probs, (unsigned)((row_stride + 63) / 64), (unsigned)parts), 256, 0, st>>>(
      probs, gpart, ppart, parts > 1 ? mid : grad_out, perm_out, row_stride, grad_factors(nf));
  if (parts > 1)
    grad_parts_kernel<<<dim3((unsigned)n_probs, (unsigned)(row_stride / 128 + 1)), 128, 0, st>>>(
        probs, mid, parts, grad_out, perm_out, row_stride, grad_factors(nf));
  return cudaGetLastError();
}

}  // namespace boss
