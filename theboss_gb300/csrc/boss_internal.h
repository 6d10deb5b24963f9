// boss_internal.h -- declarations shared by the CUDA translation units of
// libboss_gb300.so.  Not part of the public C ABI (that is include/boss.h).
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

#include <functional>
#include <string>
#include <vector>

#include "boss_sweep.cuh"

namespace boss {

enum class SweepOp { kPerm = 0, kMinors = 1, kMinorsFF = 2, kPermFF = 3 };  // FF: float pairs

// Everything one sweep launch needs (device pointers).
struct SweepLaunch {
  const SweepProblem* probs = nullptr;
  int n_probs = 0;
  const longlong2* pool = nullptr;
  int64_t total_threads = 0;
  double2* partials = nullptr;
  int grid = 1;
  int rows = 32;  // all-minors: shared-memory rows of minors per thread (nd + held digit, at most 32)
  bool quad = false;  // permanents, all-minors in FP64: the four-codes-per-step kernels (boss_quad.cuh)
  int64_t uniform_threads = 0;  // all-minors: > 0 when every sweep has this many threads and sweep p
                                // starts at thread p * uniform_threads (no search for the sweep)
};

// Sets kernel attributes and records occupancy (once per process, outside any capture).
cudaError_t prepare_sweep_kernels();
// Resident threads of one full wave of the sweep kernel for `nf` factors.
int64_t sweep_resident_threads(int nf, SweepOp op, int sm_count);
// Resident threads of the all-minors kernel (FP64, or the float-pair one) with
// `rows` rows of minors per thread.
int64_t sweep_resident_minors(int nf, int rows, int sm_count, bool ff = false);
// The same for the four-codes-per-step kernels (boss_quad.cu; rows matter to the
// all-minors kernel only).
cudaError_t prepare_quad_kernels();
int64_t quad_resident_walkers(int nf, int rows, bool minors, int sm_count);
cudaError_t launch_quad_sweep(int nf, bool minors, const SweepLaunch& L, cudaStream_t st);
// Gradient sweeps (boss_grad.cu) of nf factors: walkers resident at once; the sweep
// (grad_slice entries of gpart per warp of 8 walkers, one of ppart) and the
// reduction (grad_out: per sweep row_stride entries, digit by digit, factor by
// factor with the factor count padded to a multiple of 4).
cudaError_t prepare_grad_kernels();
int64_t grad_resident_walkers(int nf, int sm_count);
__host__ __device__ inline int grad_factors(int nf) { return (nf + 3) / 4 * 4; }
inline int64_t grad_slice(int rows, int nf) { return (int64_t)rows * grad_factors(nf) * 8; }
cudaError_t launch_grad_sweep(int nf, const SweepProblem* probs, int n_probs, const longlong2* pool, int64_t walkers,
                              double2* gpart, double2* ppart, cudaStream_t st);
// parts of the walkers that blocks of their own sum, into parts * (row_stride + 1)
// entries of mid per sweep: few sweeps leave SMs idle otherwise.
int grad_reduce_parts(int64_t walkers, int n_probs, int row_stride, int sm_count);
cudaError_t launch_grad_reduce(int nf, const SweepProblem* probs, int n_probs, const double2* gpart,
                               const double2* ppart, double2* mid, int parts, double2* grad_out, double2* perm_out,
                               int row_stride, cudaStream_t st);
// Whether the float-pair all-minors kernel exists for nf factors.
bool minors_ff_available(int nf);
cudaError_t launch_sweep(int nf, SweepOp op, const SweepLaunch& L, cudaStream_t st);
cudaError_t launch_perm_reduce(const SweepProblem* probs, int n_probs, const double2* partials, double2* out,
                               cudaStream_t st, bool ff = false);
// rows: the most digits (held one included) of a sweep.
cudaError_t launch_minors_reduce(const SweepProblem* probs, int n_probs, int rows, const double2* partials,
                                 double2* out, int nd_max, cudaStream_t st, bool ff = false);

// Splits `n_codes` codes over at most `resident` threads, proportionally, at
// least one thread per sweep and at least min_codes codes per thread.
constexpr int kFFMaxFactors = 24;      // float-pair all-minors: above this the sums exhaust the registers
constexpr int kFFPermMaxFactors = 32;  // float-pair permanents
constexpr int64_t kMinCodesPerThread = 8;
void partition_threads(const std::vector<uint64_t>& n_codes, int64_t resident, std::vector<int64_t>& n_threads,
                       int64_t min_codes = kMinCodesPerThread);
// The fewest codes (steps of four for the quad kernels) a thread takes in a launch of
// `codes`: `most` amortise a thread's first sums and its row of partials while the GPU
// is full, but below one block of `block` threads or walkers per SM the launch lasts as
// long as one thread's chain, so it halves down to `least`.  16 samples of 8 photons,
// two input modes doubly occupied: 15 kernels of 254 us in all with 8 codes a thread,
// 148 with one; one k = 10 all-minors call: 53 and 40 us.
inline int64_t min_codes_per_thread(double codes, int64_t most, int64_t least, int block, int sm_count) {
  int64_t c = most;
  while (c > least && codes < (double)c * block * sm_count) c >>= 1;
  return c;
}
// log2 of the codes every range of a sweep starts at a multiple of: the largest
// (at most 6, at most the nb binary digits) that makes the longest range at most
// 1/32 longer than an even split.  Lanes of a warp then flip the same low digit
// at each step and read the same row (one broadcast instead of several lines).
int range_align(int64_t n_codes, int64_t n_threads, int nb);

// ---------------------------------------------------------------------------
// Host-side sweep description.
// ---------------------------------------------------------------------------
// Factors from which a sweep with two binary digits takes four codes per step
// (boss_quad.cuh) instead of the templated kernel.  Permanents: always (sweeps of 64
// permanents: n = 12 18.4 against 17.7 us, n = 16 89 against 116, n = 18 416 against 433,
// n = 20 1.67 against 1.94 ms, n = 24 28.1 against 37.0).  All-minors: from 14, by the
// sampler's levels (300 samples of 18 photons, eta 0.9, with the line at 13, 14, 15, 16, none:
// 1.76, 1.77, 1.79, 1.84, 1.93 ms a call; 10^4 of 20 at 0.5: 2.72, 2.74, 2.73, 2.74, 2.69).
// Calls planned on the host share the line, though theirs would lie higher: one call of 14
// factors 44 against 40 us, of 17 66 against 54, of 20 112 against 125.
constexpr int kQuadMinFactors = 2;
constexpr int kQuadMinMinorFactors = 14;
enum RowLayout : int {
  kRowsPlain = 0,   // D (float pairs)
  kRowsPacked = 1,  // u = -D / 2 packed: the templated FP64 kernels
  kRowsQuad = 2,    // boss_quad.cuh: two binary digits and two factors at least
  kRowsGrad = 3     // boss_grad.cu
};
struct HostSweep {
  int layout = kRowsPlain;
  bool on_device = false;  // D and base are made by boss_plan.cu (D_size, base_size entries)
  size_t D_size = 0, base_size = 0;
  int kind = kRyser;
  int parity0 = 0;
  int nd = 0, nb = 0, nf = 0;
  int has_base = 0;
  int fx_sum = 0;              // sum of the factors' own fraction bits (permanents, all-minors)
  uint8_t mult[kMaxDigits] = {};
  std::vector<longlong2> D;     // nd x nf; kRowsQuad: (nd - 2) x quad_width(nf)
  std::vector<longlong2> base;  // nf (has_base); kRowsQuad: base and constants
  double scale = 1.0;
  uint64_t total_codes = 1;
  int digit_mode[kMaxDigits] = {};  // digit -> mode (all-minors results)
  int factor_mode[kMaxFactors] = {};  // factor -> mode (gradients)
  int fixed_mode = -1;                // mode of the digit held at r = 0 (Glynn halving), or -1
  bool digits_are_outputs = false;    // orientation of the sweep
  // Float-pair all-minors: factor f's bound 2^p <= max(sum mult |Re|, sum mult |Im|) < 2^(p+1)
  // over every digit (held one included), in fixed-point units; fx_to_ff takes 189 - p.
  std::vector<int> fbias;
  int ff_exp = 0;  // sum_f (p_f + 1 - fx_f): the float-pair products' scale
};

// What boss_plan.cu needs to make one sweep's rows on the GPU.
struct PlanItem {
  int32_t layout, nd, nd_all, nf;  // nd_all: with the held digit, last
  int32_t glynn, digits_are_outputs;
  int64_t mat_off, base_off;       // its rows and base in the pool
  uint16_t digit[kMaxDigits + 1], factor[kMaxFactors];
  uint8_t mult[kMaxDigits + 1];
};
// max_entries: the most digits x factors of an item (at most 65 x 32: 33 KB of shared memory).
cudaError_t launch_plan_rows(const PlanItem* items, int n, const double2* U, int m, int max_entries, longlong2* pool,
                             SweepProblem* probs, cudaStream_t st);

// Arithmetic of the all-minors sweeps (boss_minors_arithmetic): 0 float pairs
// where the kernel exists for the factor count, 1 FP64.
extern int g_minors_arith;
// Arithmetic of the single-permanent sweeps (boss_perm_arithmetic), same codes.
extern int g_perm_arith;
// x * 2^(fbias - 190) as a float pair, the host twin of fx_to_ff (same bits).
void host_fx_to_ff(long long x, int fbias, float& hi, float& lo);

// Status codes of the C ABI (include/boss.h repeats them).
enum Status : int {
  kOk = 0,
  kErrSize = 1,     // size mismatch: theboss raises AttributeError
  kErrLimit = 2,    // beyond this library's limits
  kErrCuda = 3,     // CUDA runtime error
  kErrArg = 4,      // invalid argument
  kErrPmf = 5,      // a pmf could not be normalised (theboss: ValueError in numpy.random.choice)
  kErrNoDevice = 6  // no CUDA device
};

void set_error(const std::string& msg);
int fail_cuda(cudaError_t e, const char* where);

// Per-process device context: non-blocking streams, SM count, grow-only buffers.
struct DeviceBuffer {
  void* ptr = nullptr;
  size_t bytes = 0;
};
// Runs fn(0 .. threads - 1) on the library's host threads (fn(0) on the caller) and
// returns when all have finished.
void host_parallel(int threads, const std::function<void(int)>& fn);

struct Context {
  bool ready = false;
  int device = 0;
  int sm_count = 0;
  cudaStream_t stream = nullptr;
  cudaStream_t sampler_streams[3] = {nullptr, nullptr, nullptr};  // the sampler's pipelined slots 1..3 (boss_gccb.cu)
  DeviceBuffer plans, pool, partials, out, counter, index, misc, gpart, pperm;
  DeviceBuffer gccb[32];  // the sampler's slots, 8 each
  DeviceBuffer dist[4];
  void* pinned = nullptr;
  size_t pinned_bytes = 0;
};
Context* context(int* status);
int ensure(DeviceBuffer& b, size_t bytes);
int ensure_pinned(Context* cx, size_t bytes);

// Uploads a list of sweeps (all of one sweep_class), launches the sweep
// and the reduction, copies the results back.  results: one complex per sweep
// (perms) or nd_max complex per sweep (all-minors).
int run_sweeps(Context* cx, const std::vector<HostSweep>& sweeps, bool minors, int nd_max, double2* results_host,
               const double* matrix = nullptr, int m = 0);  // the matrix of sweeps whose rows the device makes

// Permanents of at most kSmallPermMax particles, 1 to 128 GPU threads each (Glynn's
// formula in registers, no sweep planning; m <= 65536): by_l[l] lists the requests k with
// l = sum(S_k) = sum(T_k) particles; S, T are the callers' occupation rows.
constexpr int kSmallPermMax = 10;
int small_perm_batch(Context* cx, const double* matrix, int m, int len, const int32_t* S, const int32_t* T,
                     const std::vector<int>* by_l, double2* results);

// One permanent request (theboss's variant semantics).  Returns kOk and either
// fills `hs` (needs_sweep = true) or sets `value` for the edge cases theboss
// special-cases.
// What the sweep is planned for: any kernel, float pairs where they are chosen; the
// templated FP64 kernels only; FP64 always (the allocation-free entry point); the
// gradient kernel.
enum PlanFor : int { kPlanAny = 0, kPlanTemplated = 1, kPlanFP64 = 2, kPlanGrad = 3 };
int plan_permanent(const double* U, int m, const int32_t* S, const int32_t* T, int len, int variant, HostSweep& hs,
                   bool& needs_sweep, double2& value, PlanFor plan = kPlanAny, bool on_device = false);

// Sweeps of one launch share the factor count and the kernel: class 2 nf + quad.
constexpr int kSweepClasses = 2 * (kMaxFactors + 1);
inline int sweep_class(const HostSweep& h) { return 2 * h.nf + (h.layout == kRowsQuad ? 1 : 0); }

}  // namespace boss
