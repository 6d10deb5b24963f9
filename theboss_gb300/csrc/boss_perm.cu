// boss_perm.cu -- dispatch of the NF-templated sweep kernels, the fixed-order
// reductions of their partials, and the thread partition shared by every caller.
#include <algorithm>
#include <cmath>

#include "boss_internal.h"

namespace boss {

cudaError_t sweep_nf_a_launch(int nf, SweepOp op, const SweepLaunch& L, cudaStream_t st);
cudaError_t sweep_nf_b_launch(int nf, SweepOp op, const SweepLaunch& L, cudaStream_t st);
cudaError_t sweep_nf_c_launch(int nf, SweepOp op, const SweepLaunch& L, cudaStream_t st);
cudaError_t sweep_nf_d_launch(int nf, SweepOp op, const SweepLaunch& L, cudaStream_t st);
cudaError_t sweep_nf_a_prepare(int* perm_occ, int* minors_occ, int* ff_occ, int* pff_occ);
cudaError_t sweep_nf_b_prepare(int* perm_occ, int* minors_occ, int* ff_occ, int* pff_occ);
cudaError_t sweep_nf_c_prepare(int* perm_occ, int* minors_occ, int* ff_occ, int* pff_occ);
cudaError_t sweep_nf_d_prepare(int* perm_occ, int* minors_occ, int* ff_occ, int* pff_occ);


static int g_perm_occ[kMaxFactors + 1];
static int g_perm_ff_occ[kMaxFactors + 1];
static int g_minors_occ[kMaxFactors + 1][kMaxMinorDigits + 1];     // [nf][rows of minors]
static int g_minors_ff_occ[kMaxFactors + 1][kMaxMinorDigits + 1];  // float-pair kernel; 0: none

cudaError_t prepare_sweep_kernels() {
  cudaError_t e;
  if ((e = sweep_nf_a_prepare(g_perm_occ + 1, &g_minors_occ[1][0], &g_minors_ff_occ[1][0], g_perm_ff_occ + 1)))
    return e;
  if ((e = sweep_nf_b_prepare(g_perm_occ + 9, &g_minors_occ[9][0], &g_minors_ff_occ[9][0], g_perm_ff_occ + 9)))
    return e;
  if ((e = sweep_nf_c_prepare(g_perm_occ + 17, &g_minors_occ[17][0], &g_minors_ff_occ[17][0], g_perm_ff_occ + 17)))
    return e;
  if ((e = sweep_nf_d_prepare(g_perm_occ + 25, &g_minors_occ[25][0], &g_minors_ff_occ[25][0], g_perm_ff_occ + 25)))
    return e;
  if ((e = prepare_quad_kernels())) return e;
  return prepare_grad_kernels();
}


bool minors_ff_available(int nf) { return nf >= 1 && nf <= kMaxFactors && g_minors_ff_occ[nf][kMaxMinorDigits] > 0; }

int64_t sweep_resident_minors(int nf, int rows, int sm_count, bool ff) {
  if (nf < 1 || nf > kMaxFactors) return 128;
  rows = std::min(std::max(rows, 1), kMaxMinorDigits);
  const int occ = ff ? g_minors_ff_occ[nf][rows] : g_minors_occ[nf][rows];
  return (int64_t)std::max(1, occ) * sm_count * 128;
}

int64_t sweep_resident_threads(int nf, SweepOp op, int sm_count) {
  if (nf < 1 || nf > kMaxFactors) return 128;
  const int occ = std::max(1, op == SweepOp::kPerm     ? g_perm_occ[nf]
                              : op == SweepOp::kPermFF ? g_perm_ff_occ[nf]
                                                       : g_minors_occ[nf][kMaxMinorDigits]);
  return (int64_t)occ * sm_count * 128;
}

cudaError_t launch_sweep(int nf, SweepOp op, const SweepLaunch& L, cudaStream_t st) {
  if (L.total_threads <= 0) return cudaSuccess;
  if (L.quad) return launch_quad_sweep(nf, op == SweepOp::kMinors, L, st);
  if (nf >= 1 && nf <= 8) return sweep_nf_a_launch(nf, op, L, st);
  if (nf <= 16) return sweep_nf_b_launch(nf, op, L, st);
  if (nf <= 24) return sweep_nf_c_launch(nf, op, L, st);
  if (nf <= 32) return sweep_nf_d_launch(nf, op, L, st);
  return cudaErrorInvalidValue;
}

void partition_threads(const std::vector<uint64_t>& n_codes, int64_t resident, std::vector<int64_t>& n_threads,
                       int64_t min_codes) {
  const size_t n = n_codes.size();
  n_threads.assign(n, 1);
  long double total = 0;
  for (uint64_t c : n_codes) total += (long double)c;
  if (total <= 0) return;
  long double want = std::min<long double>((long double)resident, total / (long double)min_codes);
  want = std::max<long double>(want, (long double)n);
  for (size_t p = 0; p < n; ++p) {
    long double t = want * (long double)n_codes[p] / total;
    int64_t k = (int64_t)std::floor(t);
    k = std::max<int64_t>(k, 1);
    k = std::min<int64_t>(k, (int64_t)std::max<uint64_t>(n_codes[p], 1));
    n_threads[p] = k;
  }
}

int range_align(int64_t n_codes, int64_t n_threads, int nb) {
  int c = 0;
  while (c < 6 && c < nb) {
    const int64_t units = (n_codes + (2ll << c) - 1) >> (c + 1);
    const int64_t longest = ((units + n_threads - 1) / n_threads) << (c + 1);
    if (32.0 * (double)longest * (double)n_threads > 33.0 * (double)n_codes) break;
    ++c;
  }
  return c;
}

// One block per sweep: fixed-order sum of its groups' partials.
// ff: the partials are float pairs (float4), as the float-pair sweep writes them.
__global__ void perm_reduce_kernel(const SweepProblem* __restrict__ probs, const double2* __restrict__ partials,
                                   double2* __restrict__ out, int ff) {
  __shared__ double sr[256], si[256];
  const SweepProblem& P = probs[blockIdx.x];
  double ar = 0.0, ai = 0.0;
  const int64_t parts = P.n_threads / P.group;
#pragma unroll 4  // independent loads in flight
  for (int64_t i = threadIdx.x; i < parts; i += blockDim.x) {
    double2 v;
    if (ff) {
      const float4 f = reinterpret_cast<const float4*>(partials)[P.part_off + i];
      v = make_double2(ff_to_double(f.x, f.y), ff_to_double(f.z, f.w));
    } else {
      v = partials[P.part_off + i];
    }
    ar += v.x;
    ai += v.y;
  }
  sr[threadIdx.x] = ar;
  si[threadIdx.x] = ai;
  __syncthreads();
  for (int s = blockDim.x >> 1; s > 0; s >>= 1) {
    if ((int)threadIdx.x < s) {
      sr[threadIdx.x] += sr[threadIdx.x + s];
      si[threadIdx.x] += si[threadIdx.x + s];
    }
    __syncthreads();
  }
  if (threadIdx.x == 0) out[P.out_idx] = make_double2(sr[0] * P.scale, si[0] * P.scale);
}

// One block per all-minors sweep and digit: a fixed-order tree sum over the
// groups' partials.
// ff: the partials are float pairs (float4), as the float-pair sweep writes them.
__global__ void __launch_bounds__(128) minors_reduce_kernel(const SweepProblem* __restrict__ probs,
                                                            const double2* __restrict__ partials,
                                                            double2* __restrict__ out, int nd_max, int ff) {
  __shared__ double sr[128], si[128];
  const SweepProblem& P = probs[blockIdx.x];
  const int nd = P.nd + P.low + P.fixed_digit, j = blockIdx.y;  // the held digit's row last
  if (j >= nd) return;
  const int64_t parts = P.n_threads / P.group;
  double ar = 0.0, ai = 0.0;
#pragma unroll 4  // independent loads in flight
  for (int64_t q = threadIdx.x; q < parts; q += 128) {
    double2 v;
    if (ff) {
      const float4 f = reinterpret_cast<const float4*>(partials)[P.part_off + q * nd + j];
      v = make_double2(ff_to_double(f.x, f.y), ff_to_double(f.z, f.w));
    } else {
      v = partials[P.part_off + q * nd + j];
    }
    ar += v.x;
    ai += v.y;
  }
  sr[threadIdx.x] = ar;
  si[threadIdx.x] = ai;
  __syncthreads();
  int s = 64;
  while (s >= parts) s >>= 1;  // few partials: the upper sums are zero
  for (; s > 0; s >>= 1) {
    if ((int)threadIdx.x < s) {
      sr[threadIdx.x] += sr[threadIdx.x + s];
      si[threadIdx.x] += si[threadIdx.x + s];
    }
    __syncthreads();
  }
  if (threadIdx.x == 0) out[(size_t)P.out_idx * nd_max + j] = make_double2(sr[0] * P.scale, si[0] * P.scale);
}

cudaError_t launch_perm_reduce(const SweepProblem* probs, int n_probs, const double2* partials, double2* out,
                               cudaStream_t st, bool ff) {
  if (n_probs <= 0) return cudaSuccess;
  perm_reduce_kernel<<<n_probs, 256, 0, st>>>(probs, partials, out, ff ? 1 : 0);
  return cudaGetLastError();
}

cudaError_t launch_minors_reduce(const SweepProblem* probs, int n_probs, int rows, const double2* partials,
                                 double2* out, int nd_max, cudaStream_t st, bool ff) {
  if (n_probs <= 0) return cudaSuccess;
  minors_reduce_kernel<<<dim3((unsigned)n_probs, (unsigned)rows), 128, 0, st>>>(probs, partials, out, nd_max, ff ? 1 : 0);
  return cudaGetLastError();
}

}  // namespace boss
