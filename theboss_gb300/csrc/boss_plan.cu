// boss_plan.cu -- the rows of many sweeps made on the GPU.
//
// The host decides a sweep's digits and factors; the fixed-point entries, the pairs'
// coefficients (exact 128-bit products, boss_quad.cuh) and the base sums are a few
// thousand integer multiplications per sweep, 2 to 5 microseconds each on one host
// core.  A batch uploads the matrix and the lists and one block per sweep makes
// them by the host's rules (fill_sweep): the same scales, entries and integer sums.
#include "boss_internal.h"
#include "boss_quad.cuh"

namespace boss {

__global__ void __launch_bounds__(128) plan_rows_kernel(const PlanItem* __restrict__ items,
                                                        const double2* __restrict__ U, int m,
                                                        longlong2* __restrict__ pool,
                                                        SweepProblem* __restrict__ probs) {
  extern __shared__ longlong2 plan_smem[];
  __shared__ int fxs[kMaxFactors + 3];
  __shared__ unsigned long long esum[kMaxFactors / 2][4];  // per pair: E+ re im, E- re im
  __shared__ int elow[kMaxFactors / 2][4];                  // and their low parts
  const PlanItem& I = items[blockIdx.x];
  const int nf = I.nf, nd = I.nd_all, tid = threadIdx.x;
  auto entry = [&](int a, int f) {
    return I.digits_are_outputs ? U[(size_t)I.digit[a] * m + I.factor[f]] : U[(size_t)I.factor[f] * m + I.digit[a]];
  };
  for (int f = tid; f < nf; f += 128) {
    double bound = 0.0;
#pragma unroll 4
    for (int a = 0; a < nd; ++a) {
      const double2 z = entry(a, f);
      bound += I.mult[a] * fmax(fabs(z.x), fabs(z.y));
    }
    int fx = 56;
    if (bound > 0.0 && isfinite(bound)) fx = max(-1000, min(61 - ilogb(bound * (1.0 + 0x1p-40)), 1000));
    fxs[f] = fx;
  }
  for (int g = tid; g < kMaxFactors * 2; g += 128) {
    esum[g >> 2][g & 3] = 0ull;
    elow[g >> 2][g & 3] = 0;
  }
  __syncthreads();
  longlong2* const us = plan_smem;  // the entries, [digit][factor]
  auto u = [&](int e) { return cx(us[e].x, us[e].y); };
  for (int e = tid; e < nd * nf; e += 128) {
    const int a = e / nf, f = e - a * nf;
    const double2 z = entry(a, f);
    const double h = I.glynn ? 1.0 : -0.5;  // Ryser's u = -U / 2
    us[e] = make_longlong2(__double2ll_rn(ldexp(h * z.x, fxs[f])), __double2ll_rn(ldexp(h * z.y, fxs[f])));
  }
  __syncthreads();
  longlong2* rows = pool + I.mat_off;
  longlong2* base = pool + I.base_off;
  auto packed = [](Cx64 v) { return make_longlong2(pack_row(v.re), pack_row(v.im)); };
  auto plain = [](Cx64 v) { return make_longlong2(v.re, v.im); };
  auto outer_sum = [&](int first, int f) {
    Cx64 o = cx(0, 0);
    for (int a = first; a < nd; ++a) o = cx_add(o, cx_times(u(a * nf + f), I.mult[a]));
    return o;
  };
  int fx_sum = 0;
  if (I.layout == kRowsGrad) {
    const int F = grad_factors(nf);
    int32_t* bits = reinterpret_cast<int32_t*>(base + F);
    for (int e = tid; e < I.nd * F; e += 128) {
      const int a = e / F, f = e - a * F;
      rows[e] = f < nf ? packed(u(a * nf + f)) : make_longlong2(0, 0);
    }
    for (int f = tid; f < F; f += 128) {
      base[f] = f < nf ? plain(outer_sum(0, f)) : make_longlong2(1ll << 61, 0);  // padding: the constant 1
      bits[f] = f < nf ? fxs[f] : 61;
    }
    fx_sum = 61 * (F - nf);
  } else {
    const int slots = quad_slots(nf), W = quad_width(nf), ndo = I.nd - 2;
    longlong2* consts = base + W;
    const Cx64 zero = cx(0, 0);
    auto at = [&](int a, int f) { return f < nf ? u(a * nf + f) : zero; };  // an odd last factor's partner
    for (int e = tid; e < (nd - 2) * slots; e += 128) {
      const int d = e / slots, g = e - d * slots, a = d + 2;
      const Cx64 uf = at(a, 2 * g), ug = at(a, 2 * g + 1);
      Cx64 ep, em;
      quad_row(uf, ug, at(0, 2 * g), at(1, 2 * g), at(0, 2 * g + 1), at(1, 2 * g + 1), ep, em);
      if (d < ndo) {  // the held digit, last, has no row
        longlong2* r = rows + (size_t)d * W + kQuadRow * g;
        r[0] = packed(uf);
        r[1] = packed(ug);
        r[2] = packed(ep);
        r[3] = packed(em);
        r[4] = quad_low(ep, em);
      }
      const unsigned long long k = I.mult[a];
      atomicAdd(&esum[g][0], k * (unsigned long long)ep.re);
      atomicAdd(&esum[g][1], k * (unsigned long long)ep.im);
      atomicAdd(&esum[g][2], k * (unsigned long long)em.re);
      atomicAdd(&esum[g][3], k * (unsigned long long)em.im);
      atomicAdd(&elow[g][0], (int)k * ep.fr);
      atomicAdd(&elow[g][1], (int)k * ep.fi);
      atomicAdd(&elow[g][2], (int)k * em.fr);
      atomicAdd(&elow[g][3], (int)k * em.fi);
    }
    __syncthreads();
    for (int g = tid; g < slots; g += 128) {
      const bool unit = 2 * g + 1 >= nf;
      const Cx64 f0 = at(0, 2 * g), f1 = at(1, 2 * g), g0 = at(0, 2 * g + 1), g1 = at(1, 2 * g + 1);
      Cx64 of, og, ep = Cx64{(long long)esum[g][0], (long long)esum[g][1], elow[g][0], elow[g][1]},
                   em = Cx64{(long long)esum[g][2], (long long)esum[g][3], elow[g][2], elow[g][3]};
      if (I.glynn) {
        of = outer_sum(2, 2 * g);
        og = unit ? zero : outer_sum(2, 2 * g + 1);
      } else {  // Ryser: no base, and r = (1 - d) / 2 leaves -(u0 + u1)
        of = cx_sub(zero, cx_add(f0, f1));
        og = cx_sub(zero, cx_add(g0, g1));
        quad_row(of, og, f0, f1, g0, g1, ep, em);
      }
      if (unit) {
        og = cx(kQuadOne, 0);
        quad_row(zero, og, f0, f1, zero, zero, ep, em);
      }
      longlong2* b = base + kQuadRow * g;
      b[0] = plain(of);
      b[1] = plain(og);
      b[2] = plain(ep);
      b[3] = plain(em);
      b[4] = quad_low(ep, em);
      quad_constants(f0, f1, g0, g1, consts + kQuadConst * g);
    }
    fx_sum = (nf & 1) ? 62 : 0;
  }
  if (tid == 0) {
    for (int f = 0; f < nf; ++f) fx_sum += fxs[f];
    probs[blockIdx.x].fx = -fx_sum;
  }
}

cudaError_t launch_plan_rows(const PlanItem* items, int n, const double2* U, int m, int max_entries, longlong2* pool,
                             SweepProblem* probs, cudaStream_t st) {
  plan_rows_kernel<<<n, 128, sizeof(longlong2) * (size_t)max_entries, st>>>(items, U, m, pool, probs);
  return cudaGetLastError();
}

}  // namespace boss
