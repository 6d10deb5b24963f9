// boss_capi.cu -- host side of libboss_gb300.so: the per-process device context,
// the sweep planner (theboss calculator semantics -> SweepPlan segments) and the
// extern "C" entry points declared in include/boss.h.
#include <cuda_runtime.h>
#include <stdint.h>
#include <string.h>

#include <algorithm>
#include <cmath>
#include <mutex>
#include <string>
#include <vector>

#include "../../include/boss.h"
#include "boss_internal.h"
#include "boss_quad.cuh"

namespace boss {

static thread_local std::string g_last_error;
std::mutex g_api_mutex;

void set_error(const std::string& msg) { g_last_error = msg; }

int fail_cuda(cudaError_t e, const char* where) {
  set_error(std::string(where) + ": " + cudaGetErrorString(e));
  return kErrCuda;
}

static Context g_ctx;

Context* context(int* status) {
  *status = kOk;
  if (g_ctx.ready) return &g_ctx;
  int n = 0;
  cudaError_t e = cudaGetDeviceCount(&n);
  if (e != cudaSuccess || n == 0) {
    set_error("no CUDA device available");
    *status = kErrNoDevice;
    return nullptr;
  }
  if ((e = cudaGetDevice(&g_ctx.device)) != cudaSuccess) { *status = fail_cuda(e, "cudaGetDevice"); return nullptr; }
  if ((e = cudaDeviceGetAttribute(&g_ctx.sm_count, cudaDevAttrMultiProcessorCount, g_ctx.device)) != cudaSuccess) {
    *status = fail_cuda(e, "cudaDeviceGetAttribute");
    return nullptr;
  }
  if ((e = cudaStreamCreateWithFlags(&g_ctx.stream, cudaStreamNonBlocking)) != cudaSuccess) {
    *status = fail_cuda(e, "cudaStreamCreate");
    return nullptr;
  }
  for (cudaStream_t& st : g_ctx.sampler_streams)
    if ((e = cudaStreamCreateWithFlags(&st, cudaStreamNonBlocking)) != cudaSuccess) {
      *status = fail_cuda(e, "cudaStreamCreate");
      return nullptr;
    }
  if ((e = prepare_sweep_kernels()) != cudaSuccess) {
    *status = fail_cuda(e, "kernel attributes");
    return nullptr;
  }
  g_ctx.ready = true;
  return &g_ctx;
}

int ensure(DeviceBuffer& b, size_t bytes) {
  if (bytes <= b.bytes && b.ptr) return kOk;
  size_t want = std::max(bytes, b.bytes + b.bytes / 2);
  want = (want + 4095) & ~(size_t)4095;
  if (b.ptr) cudaFree(b.ptr);
  b.ptr = nullptr;
  b.bytes = 0;
  cudaError_t e = cudaMalloc(&b.ptr, want);
  if (e != cudaSuccess) return fail_cuda(e, "cudaMalloc");
  b.bytes = want;
  return kOk;
}

int ensure_pinned(Context* cx, size_t bytes) {
  if (bytes <= cx->pinned_bytes && cx->pinned) return kOk;
  size_t want = std::max(bytes, cx->pinned_bytes + cx->pinned_bytes / 2);
  want = (want + 4095) & ~(size_t)4095;
  if (cx->pinned) cudaFreeHost(cx->pinned);
  cx->pinned = nullptr;
  cx->pinned_bytes = 0;
  cudaError_t e = cudaMallocHost(&cx->pinned, want);
  if (e != cudaSuccess) return fail_cuda(e, "cudaMallocHost");
  cx->pinned_bytes = want;
  return kOk;
}

static inline size_t align_up(size_t x, size_t a) { return (x + a - 1) & ~(a - 1); }

// The device description of a planned sweep, but for its place in the launch.
static void describe_sweep(const HostSweep& h, int64_t n_threads, int group, SweepProblem& P) {
  memset(&P, 0, sizeof(P));
  P.low = h.layout == kRowsQuad ? 2 : 0;
  P.nd = h.nd - P.low;
  P.nb = h.nb - P.low;
  P.nf = h.nf;
  P.kind = h.kind;
  P.parity0 = h.parity0;
  P.fx = -h.fx_sum;
  P.has_base = h.has_base;
  P.n_codes = (int64_t)(h.total_codes >> P.low);
  P.n_threads = n_threads;
  P.align = range_align(P.n_codes, n_threads, P.nb);
  P.scale = h.scale;
  P.fixed_digit = (h.fixed_mode >= 0) ? 1 : 0;
  P.group = group;
  for (int i = 0; i < P.nd; ++i) P.mult[i] = h.mult[i + P.low];
}

// Threads (or walkers) for each of a launch's sweeps, all of one sweep_class, in
// aligned groups that sum their partials in the sweep (returned: the group's size):
// the largest that costs no sweep more than 2 % of its threads, so that the
// reduction reads that many times fewer rows (one k = 21 all-minors sweep: 21 rows of
// 39 k partials, 0.36 ms in the reduction without groups).  sm_count = 0: launches that
// leave SMs idle are not spread over them (fewer partials).
static int split_threads(const std::vector<HostSweep>& sweeps, int64_t resident, bool minors, int sm_count,
                         std::vector<int64_t>& nthr) {
  const int low = sweeps[0].layout == kRowsQuad ? 2 : 0;
  std::vector<uint64_t> codes(sweeps.size());
  double total = 0.0;
  for (size_t p = 0; p < sweeps.size(); ++p) total += (double)(codes[p] = sweeps[p].total_codes >> low);
  partition_threads(codes, resident, nthr,
                    min_codes_per_thread(total, kMinCodesPerThread >> low, 1, low ? kQuadWalkers : 128, sm_count));
  int G = minors ? 32 : low ? 8 : 1;  // what the kernels can sum
  for (int64_t t : nthr)
    while (G > 1 && (double)(t / G * G) < 0.98 * (double)t) G >>= 1;
  for (int64_t& t : nthr) t = t / G * G;
  return G;
}

static size_t rows_of(const HostSweep& h) { return h.on_device ? h.D_size : h.D.size(); }
static size_t base_of(const HostSweep& h) { return h.on_device ? h.base_size : h.base.size(); }

// Whether a call's sweeps have their rows made on the GPU: where planning them on the
// host (17 ns per digit and factor, judged by the first request) takes longer than the
// extra launch (15 us) and the matrix's way there (0.78 ns an entry).  Calls in us, host / GPU
// rows: 64 of n = 16 in 32 modes 443 / 178, 4 of n = 12 in 32 modes 42 / 49, in 512 modes
// 51 / 261, 64 there 379 / 462, 128 745 / 639.
static bool plan_on_device(int m, int count, int len, const int32_t* S, const int32_t* T) {
  if (count < 4 || m > 512) return false;
  int ni = 0, no = 0;
  for (int i = 0; i < len; ++i) {
    ni += std::max(S[i], 0);
    no += std::max(T[i], 0);
  }
  return 22.0 * count * ni * no > 20000.0 + (double)m * m;
}

static void describe_plan(const HostSweep& h, int64_t mat_off, int64_t base_off, PlanItem& I) {
  I.layout = h.layout;
  I.nd = h.nd;
  I.nd_all = h.nd + (h.fixed_mode >= 0 ? 1 : 0);
  I.nf = h.nf;
  I.glynn = h.kind == kGlynn ? 1 : 0;
  I.digits_are_outputs = h.digits_are_outputs ? 1 : 0;
  I.mat_off = mat_off;
  I.base_off = base_off;
  for (int a = 0; a < h.nd; ++a) {
    I.digit[a] = (uint16_t)h.digit_mode[a];
    I.mult[a] = h.mult[a];
  }
  if (h.fixed_mode >= 0) {
    I.digit[h.nd] = (uint16_t)h.fixed_mode;
    I.mult[h.nd] = 1;
  }
  for (int f = 0; f < h.nf; ++f) I.factor[f] = (uint16_t)h.factor_mode[f];
}

// A list of sweeps that share one factor count, uploaded and ready to launch.
struct SweepBatch {
  int n = 0, nf = 0;
  bool minors = false;
  bool ff = false;  // all-minors on float pairs
  int nd_max = 1;
  SweepLaunch L;
  size_t out_elems = 0;
  double2* out = nullptr;  // results, in page-locked memory that the reduction writes: no copy down
  double codes = 0.0;  // codes swept per launch
};

static int sweeps_prepare(Context* cx, const std::vector<HostSweep>& sweeps, bool minors, int nd_max, SweepBatch& B,
                          const double* matrix = nullptr, int m = 0) {
  const int n = (int)sweeps.size();
  B.n = n;
  B.nf = sweeps[0].nf;
  B.minors = minors;
  B.nd_max = nd_max;
  // Float pairs (planned as plain rows) only for Glynn-kind sweeps: the Ryser form's
  // alternating sum cancels far more (its FP64 error is already ~1e-10 at n = 20),
  // and float pairs would leave theboss's tolerance.
  B.ff = sweeps[0].layout == kRowsPlain;
  const bool quad = sweeps[0].layout == kRowsQuad;
  const SweepOp op = minors ? SweepOp::kMinors : (B.ff ? SweepOp::kPermFF : SweepOp::kPerm);
  B.codes = 0.0;
  int rows = 1;  // all-minors: rows of minors per thread
  for (int p = 0; p < n; ++p) {
    B.codes += (double)sweeps[p].total_codes;
    rows = std::max(rows, sweeps[p].nd + (sweeps[p].fixed_mode >= 0 ? 1 : 0));
  }
  std::vector<int64_t> nthr;
  const int G = split_threads(sweeps,
                              quad     ? quad_resident_walkers(B.nf, rows, minors, cx->sm_count)
                              : minors ? sweep_resident_minors(B.nf, rows, cx->sm_count, B.ff)
                                       : sweep_resident_threads(B.nf, op, cx->sm_count),
                              minors, cx->sm_count, nthr);
  std::vector<SweepProblem> probs(n);
  int64_t pool_n = 0, threads = 0, parts = 0;
  for (int p = 0; p < n; ++p) {
    const HostSweep& h = sweeps[p];
    SweepProblem& P = probs[p];
    describe_sweep(h, nthr[p], G, P);
    P.out_idx = p;
    P.thread_begin = threads;
    P.mat_off = pool_n;
    pool_n += (int64_t)rows_of(h);
    P.base_off = pool_n;
    pool_n += (int64_t)base_of(h);
    P.part_off = parts;
    if (B.ff) {  // float-pair rows of the binary digits, then the factors' biases
      P.ff_off = pool_n;
      pool_n += (int64_t)h.nb * h.nf + (h.nf + 3) / 4;
      P.scale = std::ldexp(h.scale, h.ff_exp);
    }
    threads += nthr[p];
    parts += nthr[p] / G * (minors ? h.nd + P.fixed_digit : 1);
  }
  // arena: problems | matrix and plan items (rows made on the device) | pool; `up` bytes
  // of it come from the host
  const bool device_rows = sweeps[0].on_device;  // all of a call's sweeps of a class alike
  size_t off = 0;
  const size_t o_probs = off; off = align_up(off + sizeof(SweepProblem) * n, 256);
  const size_t o_U = off; off = align_up(off + (device_rows ? sizeof(double2) * (size_t)m * m : 0), 256);
  const size_t o_items = off; off = align_up(off + (device_rows ? sizeof(PlanItem) * n : 0), 256);
  const size_t o_pool = off; off = align_up(off + sizeof(longlong2) * std::max<int64_t>(pool_n, 1), 256);
  const size_t arena_bytes = off, up = device_rows ? o_pool : arena_bytes;
  B.out_elems = (size_t)n * (minors ? nd_max : 1);
  int st;
  if ((st = ensure(cx->plans, arena_bytes))) return st;
  if ((st = ensure(cx->partials, sizeof(double2) * std::max<int64_t>(parts, 1)))) return st;
  const size_t o_out = align_up(up, 256);
  if ((st = ensure_pinned(cx, o_out + sizeof(double2) * B.out_elems))) return st;
  char* h = (char*)cx->pinned;
  B.out = (double2*)(h + o_out);
  memcpy(h + o_probs, probs.data(), sizeof(SweepProblem) * n);
  longlong2* hp = (longlong2*)(h + o_pool);
  int max_entries = 0;
  if (device_rows) memcpy(h + o_U, matrix, sizeof(double2) * (size_t)m * m);
  for (int p = 0; p < n && device_rows; ++p) {
    describe_plan(sweeps[p], probs[p].mat_off, probs[p].base_off, ((PlanItem*)(h + o_items))[p]);
    max_entries = std::max(max_entries, (sweeps[p].nd + 1) * B.nf);
  }
  for (int p = 0; p < n && !device_rows; ++p) {
    const HostSweep& hs = sweeps[p];
    std::copy(hs.D.begin(), hs.D.end(), hp + probs[p].mat_off);
    std::copy(hs.base.begin(), hs.base.end(), hp + probs[p].base_off);
    if (B.ff) {
      float4* df = reinterpret_cast<float4*>(hp + probs[p].ff_off);
      for (int d = 0; d < hs.nb; ++d)
        for (int f = 0; f < hs.nf; ++f) {
          const longlong2 v = hs.D[(size_t)d * hs.nf + f];
          float4& o = df[(size_t)d * hs.nf + f];
          host_fx_to_ff(v.x, hs.fbias[f], o.x, o.y);
          host_fx_to_ff(v.y, hs.fbias[f], o.z, o.w);
        }
      int* fb = reinterpret_cast<int*>(df + (size_t)hs.nb * hs.nf);
      for (int f = 0; f < hs.nf; ++f) fb[f] = hs.fbias[f];
    }
  }
  char* d = (char*)cx->plans.ptr;
  cudaError_t e = cudaMemcpyAsync(d, h, up, cudaMemcpyHostToDevice, cx->stream);
  if (e != cudaSuccess) return fail_cuda(e, "H2D sweeps");
  if (device_rows) {
    e = launch_plan_rows((const PlanItem*)(d + o_items), n, (const double2*)(d + o_U), m, max_entries,
                         (longlong2*)(d + o_pool), (SweepProblem*)(d + o_probs), cx->stream);
    if (e != cudaSuccess) return fail_cuda(e, "sweep rows");
  }
  B.L.probs = (const SweepProblem*)(d + o_probs);
  B.L.n_probs = n;
  B.L.pool = (const longlong2*)(d + o_pool);
  B.L.total_threads = threads;
  B.L.partials = (double2*)cx->partials.ptr;
  B.L.grid = (int)((threads + 127) / 128);
  B.L.rows = rows;
  B.L.quad = quad;
  return kOk;
}

static int sweeps_launch(Context* cx, const SweepBatch& B, cudaEvent_t after_sweep = nullptr) {
  const SweepOp op = B.minors ? (B.ff ? SweepOp::kMinorsFF : SweepOp::kMinors) : (B.ff ? SweepOp::kPermFF : SweepOp::kPerm);
  cudaError_t e = launch_sweep(B.nf, op, B.L, cx->stream);
  if (e != cudaSuccess) return fail_cuda(e, "sweep launch");
  if (after_sweep) cudaEventRecord(after_sweep, cx->stream);
  e = B.minors ? launch_minors_reduce(B.L.probs, B.n, B.L.rows, B.L.partials, B.out, B.nd_max, cx->stream, B.ff)
               : launch_perm_reduce(B.L.probs, B.n, B.L.partials, B.out, cx->stream, B.ff);
  return e == cudaSuccess ? kOk : fail_cuda(e, "reduce launch");
}

static int sweeps_collect(Context* cx, const SweepBatch& B, double2* results_host) {
  const cudaError_t e = cudaStreamSynchronize(cx->stream);
  if (e != cudaSuccess) return fail_cuda(e, "sweep");
  memcpy(results_host, B.out, sizeof(double2) * B.out_elems);
  return kOk;
}

int run_sweeps(Context* cx, const std::vector<HostSweep>& sweeps, bool minors, int nd_max, double2* results_host,
               const double* matrix, int m) {
  if (sweeps.empty()) return kOk;
  SweepBatch B;
  int st = sweeps_prepare(cx, sweeps, minors, nd_max, B, matrix, m);
  if (!st) st = sweeps_launch(cx, B);
  if (st) {
    cudaStreamSynchronize(cx->stream);  // nothing queued may outlive the call's staging
    return st;
  }
  return sweeps_collect(cx, B, results_host);
}

// ---------------------------------------------------------------------------
// Planner: theboss calculator semantics -> HostSweep
// ---------------------------------------------------------------------------
static inline double2 U_at(const double* U, int m, int row, int col) {
  const double* p = U + 2 * ((size_t)row * m + col);
  return make_double2(p[0], p[1]);
}

struct Side {
  int n = 0;                 // particles
  std::vector<int> modes;    // distinct occupied modes, binary first
  std::vector<int> mult;
  int nb = 0;
  uint64_t codes = 1;        // prod (mult + 1)
};

static Side make_side(const int32_t* occ, int len) {
  Side s;
  for (int i = 0; i < len; ++i)
    if (occ[i] == 1) { s.modes.push_back(i); s.mult.push_back(1); }
  s.nb = (int)s.modes.size();
  for (int i = 0; i < len; ++i)
    if (occ[i] > 1) { s.modes.push_back(i); s.mult.push_back(occ[i]); }
  for (int i = 0; i < len; ++i) s.n += std::max(occ[i], 0);
  for (size_t a = 0; a < s.mult.size(); ++a) {
    const uint64_t b = (uint64_t)s.mult[a] + 1;
    s.codes = (s.codes > (UINT64_MAX >> 2) / b) ? UINT64_MAX : s.codes * b;
  }
  return s;
}

// Fixed-point fraction bits for sums bounded by `bound` (|s| <= bound): the
// integer sums stay below 2^bits (with room for the entries' roundings).
static int choose_fx(double bound, int bits) {
  if (!(bound > 0.0) || !std::isfinite(bound)) return 56;
  int ex = 0;
  std::frexp(bound * (1.0 + 0x1p-40), &ex);  // bound < 2^ex
  return std::max(-1000, std::min(bits - ex, 1000));
}

// v * 2^fx rounded to the nearest integer (ties to even); |v * 2^fx| < 2^62.
static inline long long to_fixed(double v, double scale) {
  double x = v * scale;  // exact: scale is a power of two
  const double t = std::copysign(4503599627370496.0, x);  // 2^52: adding it rounds to an integer
  if (std::fabs(x) < 4503599627370496.0) x = (x + t) - t;
  return (long long)x;
}

// FP64 by default (theboss computes in float64); float pairs on request.
int g_minors_arith = 1;
int g_perm_arith = 1;

static longlong2 packed(Cx64 v) { return longlong2{pack_row(v.re), pack_row(v.im)}; }
static longlong2 plain(Cx64 v) { return longlong2{v.re, v.im}; }

// The rows, base and constants of boss_quad.cuh.  u[a * nf + f]: every digit's
// fixed-point u (binary digits first, the held one at `drop`).
static void fill_quad(HostSweep& hs, const Side& dig, int drop, bool glynn, const std::vector<Cx64>& u) {
  const int nf = hs.nf, slots = quad_slots(nf), W = quad_width(nf), nd_all = (int)dig.modes.size(), ndo = hs.nd - 2;
  const Cx64 zero{0, 0};
  hs.D.assign((size_t)ndo * W, longlong2{0, 0});
  hs.base.assign((size_t)quad_base(nf), longlong2{0, 0});
  longlong2* consts = hs.base.data() + W;
  for (int g = 0; g < slots; ++g) {
    const bool unit = 2 * g + 1 >= nf;  // an odd last factor's partner, the constant 1
    auto U = [&](int a, int k) { return k && unit ? zero : u[(size_t)a * nf + 2 * g + k]; };
    const Cx64 f0 = U(0, 0), f1 = U(1, 0), g0 = U(0, 1), g1 = U(1, 1);
    Cx64 of = zero, og = zero, ep = zero, em = zero;
    int row = 0;
    for (int a = 2; a < nd_all; ++a) {
      const Cx64 uf = U(a, 0), ug = U(a, 1);
      Cx64 rp, rm;
      quad_row(uf, ug, f0, f1, g0, g1, rp, rm);
      if (a != drop) {
        longlong2* r = &hs.D[(size_t)(row++) * W + kQuadRow * g];
        r[0] = packed(uf);
        r[1] = packed(ug);
        r[2] = packed(rp);
        r[3] = packed(rm);
        r[4] = quad_low(rp, rm);
      }
      of = cx_add(of, cx_times(uf, dig.mult[a]));
      og = cx_add(og, cx_times(ug, dig.mult[a]));
      ep = cx_add(ep, cx_times(rp, dig.mult[a]));
      em = cx_add(em, cx_times(rm, dig.mult[a]));
    }
    if (!glynn) {  // Ryser: no base, and r = (1 - d) / 2 leaves -(u0 + u1)
      of = cx_sub(zero, cx_add(f0, f1));
      og = cx_sub(zero, cx_add(g0, g1));
      quad_row(of, og, f0, f1, g0, g1, ep, em);
    }
    if (unit) {
      og = Cx64{kQuadOne, 0};
      quad_row(zero, og, f0, f1, zero, zero, ep, em);
    }
    longlong2* b = &hs.base[kQuadRow * g];
    b[0] = plain(of);
    b[1] = plain(og);
    b[2] = plain(ep);
    b[3] = plain(em);
    b[4] = quad_low(ep, em);
    quad_constants(f0, f1, g0, g1, consts + kQuadConst * g);
  }
  if (nf & 1) hs.fx_sum += 62;
}

// The rows, base and fraction bits of boss_grad.cu (Glynn kind).
static void fill_grad(HostSweep& hs, const Side& dig, int drop, const std::vector<Cx64>& u, const int* fxs) {
  const int nf = hs.nf, F = grad_factors(nf), nd_all = (int)dig.modes.size();
  hs.D.assign((size_t)hs.nd * F, longlong2{0, 0});
  hs.base.assign((size_t)F + F / 4, longlong2{0, 0});
  int32_t* bits = (int32_t*)(hs.base.data() + F);
  for (int f = 0; f < F; ++f) {
    bits[f] = f < nf ? fxs[f] : 61;
    if (f >= nf) hs.base[f] = longlong2{1ll << 61, 0};  // padding: the constant 1
  }
  int row = 0;
  for (int a = 0; a < nd_all; ++a) {
    for (int f = 0; f < nf; ++f) {
      const Cx64 v = u[(size_t)a * nf + f];
      if (a != drop) hs.D[(size_t)row * F + f] = packed(v);
      hs.base[f].x += (long long)dig.mult[a] * v.re;
      hs.base[f].y += (long long)dig.mult[a] * v.im;
    }
    if (a != drop) ++row;
  }
  hs.fx_sum += 61 * (F - nf);
}

// Fills a sweep that iterates `dig` and multiplies over the particles of `col`
// (a mode occupied p times gives p factors).  entry(a, l) is the matrix element
// between digit mode a and product mode l.  Every factor f has its own fixed-point
// scale 2^fx_f, chosen so that its largest possible sum fills the bits (a shared
// scale would leave the factors of small rows with fewer significant bits).
template <class F>
static int fill_sweep(HostSweep& hs, const Side& dig, const Side& col, int kind, bool halve, PlanFor plan, bool ff,
                      int quad_min, bool on_device, F entry) {
  int drop = -1;
  if (halve && dig.nb > 0) drop = dig.nb - 1;  // a binary digit fixed at r = 0
  hs.kind = kind;
  hs.nd = (int)dig.modes.size() - (drop >= 0 ? 1 : 0);
  hs.nb = dig.nb - (drop >= 0 ? 1 : 0);
  std::vector<int> fmode;
  for (size_t l = 0; l < col.modes.size(); ++l)
    for (int k = 0; k < col.mult[l]; ++k) fmode.push_back(col.modes[l]);
  hs.nf = (int)fmode.size();
  hs.fixed_mode = (drop >= 0) ? dig.modes[drop] : -1;
  for (int f = 0; f < (int)fmode.size() && f < kMaxFactors; ++f) hs.factor_mode[f] = fmode[f];
  if (hs.nd > kMaxDigits || hs.nf > kMaxFactors || hs.nf < 1) {
    set_error("sweep exceeds 64 distinct iterated modes or 32 product-side particles");
    return kErrLimit;
  }
  hs.total_codes = 1;
  int a_out = 0;
  for (size_t a = 0; a < dig.modes.size(); ++a) {
    if ((int)a == drop) continue;
    hs.mult[a_out] = (uint8_t)dig.mult[a];
    hs.digit_mode[a_out] = dig.modes[a];
    const uint64_t b = (uint64_t)dig.mult[a] + 1;
    if (hs.total_codes > (1ull << 62) / b) {
      set_error("code count exceeds 2^62");
      return kErrLimit;
    }
    hs.total_codes *= b;
    ++a_out;
  }
  const bool glynn = kind == kGlynn;
  hs.layout = plan == kPlanGrad                                         ? kRowsGrad
              : (ff && glynn && plan == kPlanAny)                       ? kRowsPlain
              : (plan != kPlanTemplated && hs.nb >= 2 && hs.nf >= quad_min)   ? kRowsQuad
                                                                       : kRowsPacked;
  hs.scale = glynn ? std::ldexp(1.0, -dig.n) * (drop >= 0 ? 2.0 : 1.0) : 1.0;
  hs.parity0 = glynn ? 0 : (dig.n & 1);
  hs.has_base = glynn;  // (the quad and gradient layouts carry one always)
  hs.on_device = on_device && (hs.layout == kRowsQuad || hs.layout == kRowsGrad);
  if (hs.on_device) {
    const int Fg = grad_factors(hs.nf), W = quad_width(hs.nf);
    hs.D_size = hs.layout == kRowsGrad ? (size_t)hs.nd * Fg : (size_t)(hs.nd - 2) * W;
    hs.base_size = hs.layout == kRowsGrad ? (size_t)Fg + Fg / 4 : (size_t)quad_base(hs.nf);
    return kOk;
  }
  // |row sum| <= sum_a mult_a * max component of the entries
  const int nf = hs.nf, nd_all = (int)dig.modes.size();
  double bound[kMaxFactors] = {};
  for (int a = 0; a < nd_all; ++a)
    for (int f = 0; f < nf; ++f) {
      const double2 z = entry(dig.modes[a], fmode[f]);
      bound[f] += dig.mult[a] * std::max(std::fabs(z.x), std::fabs(z.y));
    }
  const bool old_rows = hs.layout == kRowsPlain;
  const int bits = old_rows ? 61 : 62;  // plain rows hold D = -2 u, which needs the bit
  hs.fx_sum = 0;
  hs.ff_exp = 0;
  hs.fbias.assign(nf, 189);
  int fxs[kMaxFactors];
  std::vector<Cx64> u((size_t)nd_all * nf);
  for (int f = 0; f < nf; ++f) {
    const int fx = choose_fx(bound[f], bits);
    fxs[f] = fx;
    const double scale = std::ldexp(glynn || old_rows ? 1.0 : -0.5, fx);  // Ryser's u = -U / 2
    unsigned long long bx = 0, by = 0;
    for (int a = 0; a < nd_all; ++a) {
      const double2 z = entry(dig.modes[a], fmode[f]);
      const long long x = to_fixed(z.x, scale), y = to_fixed(z.y, scale);
      u[(size_t)a * nf + f] = Cx64{x, y};
      bx += (unsigned long long)dig.mult[a] * (unsigned long long)std::llabs(x);
      by += (unsigned long long)dig.mult[a] * (unsigned long long)std::llabs(y);
    }
    const unsigned long long b = std::max(bx, by);
    const int p = b ? 63 - __builtin_clzll(b) : 0;
    hs.fbias[f] = 189 - p;
    hs.ff_exp += p + 1 - fx;
    hs.fx_sum += fx;
  }
  if (hs.layout == kRowsQuad) {
    fill_quad(hs, dig, drop, glynn, u);
    return kOk;
  }
  if (hs.layout == kRowsGrad) {
    fill_grad(hs, dig, drop, u, fxs);
    return kOk;
  }
  hs.D.resize((size_t)hs.nd * nf);
  if (hs.has_base) hs.base.assign(nf, longlong2{0, 0});
  a_out = 0;
  for (int a = 0; a < nd_all; ++a) {
    for (int f = 0; f < nf; ++f) {
      const Cx64 v = u[(size_t)a * nf + f];
      if (a != drop)
        hs.D[(size_t)a_out * nf + f] = !old_rows ? packed(v) : glynn ? longlong2{-2 * v.re, -2 * v.im} : plain(v);
      if (glynn) {
        hs.base[f].x += (long long)dig.mult[a] * v.re;
        hs.base[f].y += (long long)dig.mult[a] * v.im;
      }
    }
    if (a != drop) ++a_out;
  }
  return kOk;
}

void host_fx_to_ff(long long x, int fbias, float& hi, float& lo) {
  const unsigned long long sgn = (unsigned long long)(x >> 63);
  const unsigned long long ax = ((unsigned long long)x ^ sgn) - sgn;
  if (!ax) {
    hi = lo = 0.0f;
    return;
  }
  const int lz = __builtin_clzll(ax);
  const unsigned long long y = ax << lz;
  const uint32_t yh = (uint32_t)(y >> 32);
  const int ex = fbias - lz;
  const uint32_t s32 = (uint32_t)sgn & 0x80000000u;
  const uint32_t hb = (((uint32_t)(ex - 1)) << 23) + (yh >> 8);
  const uint32_t nxt = (uint32_t)(y >> 17) & 0x7FFFFFu;
  const uint32_t eb = ((uint32_t)(ex - 23)) << 23;
  auto as_f = [](uint32_t u) {
    float f;
    memcpy(&f, &u, 4);
    return f;
  };
  auto as_u = [](float f) {
    uint32_t u;
    memcpy(&u, &f, 4);
    return u;
  };
  const float l = as_f(eb | nxt) - as_f(eb);
  hi = as_f(hb | s32);
  lo = as_f(as_u(l) ^ s32);
}

// One permanent request.  Returns kOk and either fills `hs` (needs_sweep = true)
// or sets `value` directly for the edge cases theboss special-cases.
int plan_permanent(const double* U, int m, const int32_t* S, const int32_t* T, int len, int variant,
                          HostSweep& hs, bool& needs_sweep, double2& value, PlanFor plan,
                          bool on_device) {
  needs_sweep = false;
  const bool ff = g_perm_arith == 0;  // float pairs: every factor count has the kernel (kFFPermMaxFactors)
  if (len > m || len < 0) {  // bs_permanent_calculator_base.py:61-72
    set_error("state length exceeds matrix dimension");
    return kErrSize;
  }
  for (int i = 0; i < len; ++i)
    if (S[i] < 0 || T[i] < 0 || S[i] > 255 || T[i] > 255) {
      set_error("occupations must be in [0, 255]");
      return kErrArg;
    }
  const Side in = make_side(S, len), out = make_side(T, len);
  auto entry_in_out = [&](int i_mode, int j_mode) { return U_at(U, m, j_mode, i_mode); };  // digit = input
  auto entry_out_in = [&](int j_mode, int i_mode) { return U_at(U, m, j_mode, i_mode); };  // digit = output
  switch (variant) {
    case BOSS_RYSER:
    case BOSS_CHIN_HUH: {
      if (out.modes.empty()) {  // empty product: (1 - 1)^n
        value = make_double2(in.n == 0 ? 1.0 : 0.0, 0.0);
        return kOk;
      }
      if (in.modes.empty()) {  // r = 0 only: prod of zero sums
        value = make_double2(0.0, 0.0);
        return kOk;
      }
      const bool ch = (variant == BOSS_CHIN_HUH);
      const int st = fill_sweep(hs, in, out, ch ? kGlynn : kRyser, ch && in.n == out.n, plan, ff, kQuadMinFactors, on_device, entry_in_out);
      if (st) return st;
      needs_sweep = true;
      return kOk;
    }
    case BOSS_GLYNN:
    case BOSS_CLASSIC: {
      if (variant == BOSS_CLASSIC && in.n == 0) {  // classic_permanent_calculator.py:29-33
        value = make_double2(out.n == 0 ? 1.0 : 0.0, 0.0);
        return kOk;
      }
      if (in.n == 0 || out.n == 0) {  // glynn_gray_permanent_calculator.py:52-53
        value = make_double2(1.0, 0.0);
        return kOk;
      }
      if (in.n != out.n) {
        set_error("effective scattering matrix is not square (sum of input != sum of output)");
        return kErrSize;
      }
      // Iterate the side with fewer codes (after fixing one binary digit).
      const uint64_t ci = in.nb ? in.codes / 2 : in.codes;
      const uint64_t co = out.nb ? out.codes / 2 : out.codes;
      int st;
      bool outs = co < ci;
      st = outs ? fill_sweep(hs, out, in, kGlynn, true, plan, ff, kQuadMinFactors, on_device, entry_out_in) : fill_sweep(hs, in, out, kGlynn, true, plan, ff, kQuadMinFactors, on_device, entry_in_out);
      if (st == kErrLimit) {  // try the other orientation
        outs = !outs;
        st = outs ? fill_sweep(hs, out, in, kGlynn, true, plan, ff, kQuadMinFactors, on_device, entry_out_in) : fill_sweep(hs, in, out, kGlynn, true, plan, ff, kQuadMinFactors, on_device, entry_in_out);
      }
      if (st) return st;
      hs.digits_are_outputs = outs;
      if (hs.nd == 0) {  // a single code
        // fall through to the sweep anyway: nd = 0 is a one-code sweep
      }
      needs_sweep = true;
      return kOk;
    }
    default:
      set_error("unknown permanent variant");
      return kErrArg;
  }
}

// All-minors request (bs_submatrices_permanent_calculator_base.py:150-189).
// results: len complex (minor of input mode i at position i).
static int plan_minors(const double* U, int m, const int32_t* S, const int32_t* T, int len, HostSweep& hs,
                       bool& needs_sweep, double2* direct) {
  needs_sweep = false;
  if (len > m || len <= 0) {
    set_error("state length must be in [1, matrix dimension]");
    return kErrSize;
  }
  for (int i = 0; i < len; ++i)
    if (S[i] < 0 || T[i] < 0 || S[i] > 255 || T[i] > 255) {
      set_error("occupations must be in [0, 255]");
      return kErrArg;
    }
  const Side in = make_side(S, len), out = make_side(T, len);
  if (in.n == 1) {  // bs_submatrices_permanent_calculator_base.py:157-158
    for (int i = 0; i < len; ++i) direct[i] = make_double2((double)S[i], 0.0);
    return kOk;
  }
  for (int i = 0; i < len; ++i) direct[i] = make_double2(0.0, 0.0);
  if (in.n == 0) return kOk;
  if (in.modes.size() > (size_t)kMaxMinorDigits || out.n > kMaxFactors) {
    set_error("all-minors sweep exceeds 32 distinct input modes or 32 output particles");
    return kErrLimit;
  }
  if (out.modes.empty()) {
    // Product over no columns is 1; theboss skips the r = 0 code
    // (bs_cc_ryser_submatrices_permanent_calculator.py:73-78), so every other code
    // adds (-1)^|r| C-weights.  Evaluated directly on the host.
    std::vector<int> r(in.modes.size(), 0), u(in.modes.size(), 1);
    double binom = 1.0;
    double sign = 1.0;
    const size_t nd = in.modes.size();
    uint64_t guard = 0;
    for (;;) {
      size_t idx = 0;
      int k = r[0] + u[0];
      bool done = false;
      while (k > in.mult[idx] || k < 0) {
        u[idx] = -u[idx];
        if (++idx == nd) { done = true; break; }
        k = r[idx] + u[idx];
      }
      if (done) break;
      const int last = r[idx];
      r[idx] = k;
      sign = -sign;
      binom = (k > last) ? binom * ((double)(in.mult[idx] - last) / k) : binom * ((double)last / (in.mult[idx] - k));
      for (size_t a = 0; a < nd; ++a) {
        if (r[a] == in.mult[a]) continue;
        const double ub = binom / ((double)in.mult[a] / (in.mult[a] - r[a]));
        direct[in.modes[a]].x += sign * ub;
      }
      if (++guard > (1ull << 24)) {
        set_error("degenerate all-minors request too large");
        return kErrLimit;
      }
    }
    return kOk;
  }
  // Glynn form: the coefficients of an appended row of variables (every S_i minor_i
  // from one sweep, one single-occupied digit held at r = 0); the kernel
  // accumulates half of each, hence the factor 2.
  auto entry = [&](int i_mode, int j_mode) { return U_at(U, m, j_mode, i_mode); };
  const int st = fill_sweep(hs, in, out, kGlynn, true, kPlanAny, g_minors_arith == 0 && out.n <= kFFMaxFactors,
                            kQuadMinMinorFactors, false, entry);
  if (st) return st;
  hs.scale *= 2.0;
  needs_sweep = true;
  return kOk;
}

}  // namespace boss

using namespace boss;

extern "C" {

const char* boss_last_error(void) { return g_last_error.c_str(); }

int boss_abi_version(void) { return BOSS_ABI_VERSION; }

int boss_select_device(int32_t device) {
  std::lock_guard<std::mutex> lk(g_api_mutex);
  if (g_ctx.ready) {
    if (g_ctx.device == device) return kOk;
    set_error("the library's context is already bound to another device");
    return kErrArg;
  }
  cudaError_t e = cudaSetDevice(device);
  return e == cudaSuccess ? kOk : fail_cuda(e, "cudaSetDevice");
}

int boss_device_sm_count(int32_t* sm_count) {
  std::lock_guard<std::mutex> lk(g_api_mutex);
  int st;
  Context* cx = context(&st);
  if (!cx) return st;
  *sm_count = cx->sm_count;
  return kOk;
}

int boss_perm_batch(const double* matrix, int32_t m, const int32_t* input_states, const int32_t* output_states,
                    int32_t len, int32_t count, int32_t variant, double* results) {
  if (!matrix || !input_states || !output_states || !results || m <= 0 || count < 0) {
    set_error("null pointer or bad size");
    return kErrArg;
  }
  std::lock_guard<std::mutex> lk(g_api_mutex);
  std::vector<HostSweep> by_class[kSweepClasses];
  std::vector<int> which[kSweepClasses];
  std::vector<int> small[kSmallPermMax + 1];  // by particle count; no planning
  bool any = false, any_small = false;
  const bool on_device = count > 0 && plan_on_device(m, count, len, input_states, output_states);
  if (variant < BOSS_RYSER || variant > BOSS_CLASSIC) {
    set_error("unknown permanent variant");
    return kErrArg;
  }
  for (int k = 0; k < count; ++k) {
    const int32_t* Sk = input_states + (size_t)k * len;
    const int32_t* Tk = output_states + (size_t)k * len;
    if (len <= m && m <= 65536) {  // equal particle counts up to kSmallPermMax: every variant is the permanent
      int ni = 0, no = 0;
      bool ok = true;
      for (int i = 0; i < len; ++i) {
        ok &= (Sk[i] >= 0 && Tk[i] >= 0 && Sk[i] <= 255 && Tk[i] <= 255);
        ni += Sk[i];
        no += Tk[i];
      }
      if (ok && ni == no && ni >= 1 && ni <= kSmallPermMax) {
        small[ni].push_back(k);
        any_small = true;
        continue;
      }
    }
    HostSweep hs;
    bool need = false;
    double2 v = make_double2(0.0, 0.0);
    const int st = plan_permanent(matrix, m, Sk, Tk, len, variant, hs, need, v, kPlanAny, on_device);
    if (st) return st;
    if (need) {
      const int c = sweep_class(hs);
      which[c].push_back(k);
      by_class[c].push_back(std::move(hs));
      any = true;
    } else {
      results[2 * k] = v.x;
      results[2 * k + 1] = v.y;
    }
  }
  if (!any && !any_small) return kOk;
  int st;
  Context* cx = context(&st);
  if (!cx) return st;
  if (any_small && (st = small_perm_batch(cx, matrix, m, len, input_states, output_states, small,
                                          (double2*)results)))
    return st;
  for (int c = 0; c < kSweepClasses; ++c) {
    if (by_class[c].empty()) continue;
    std::vector<double2> out(by_class[c].size());
    st = run_sweeps(cx, by_class[c], false, 1, out.data(), matrix, m);
    if (st) return st;
    for (size_t a = 0; a < out.size(); ++a) {
      results[2 * which[c][a]] = out[a].x;
      results[2 * which[c][a] + 1] = out[a].y;
    }
  }
  return kOk;
}

int boss_submatrices_batch(const double* matrix, int32_t m, const int32_t* input_states,
                           const int32_t* output_states, int32_t len, int32_t count, int32_t variant,
                           double* results) {
  if (!matrix || !input_states || !output_states || !results || m <= 0 || count < 0) {
    set_error("null pointer or bad size");
    return kErrArg;
  }
  if (variant != BOSS_RYSER && variant != BOSS_CHIN_HUH) {
    set_error("all-minors variant must be BOSS_RYSER or BOSS_CHIN_HUH");
    return kErrArg;
  }
  std::lock_guard<std::mutex> lk(g_api_mutex);
  std::vector<HostSweep> by_class[kSweepClasses];
  std::vector<int> which[kSweepClasses];
  double2* res = (double2*)results;
  bool any = false;
  for (int k = 0; k < count; ++k) {
    HostSweep hs;
    bool need = false;
    const int st = plan_minors(matrix, m, input_states + (size_t)k * len, output_states + (size_t)k * len, len, hs,
                               need, res + (size_t)k * len);
    if (st) return st;
    if (need) {
      const int c = sweep_class(hs);
      which[c].push_back(k);
      by_class[c].push_back(std::move(hs));
      any = true;
    }
  }
  if (!any) return kOk;
  int st;
  Context* cx = context(&st);
  if (!cx) return st;
  const int nd_max = kMaxMinorDigits;
  for (int c = 0; c < kSweepClasses; ++c) {
    if (by_class[c].empty()) continue;
    std::vector<double2> out(by_class[c].size() * nd_max);
    st = run_sweeps(cx, by_class[c], true, nd_max, out.data());
    if (st) return st;
    for (size_t a = 0; a < by_class[c].size(); ++a) {
      const HostSweep& hs = by_class[c][a];
      double2* row = res + (size_t)which[c][a] * len;
      for (int d = 0; d < hs.nd; ++d) {  // the sweep gives S_i minor_i
        const double2 v = out[a * nd_max + d];
        row[hs.digit_mode[d]] = make_double2(v.x / hs.mult[d], v.y / hs.mult[d]);
      }
      if (hs.fixed_mode >= 0) row[hs.fixed_mode] = out[a * nd_max + hs.nd];  // the held digit (S_i = 1)
    }
  }
  return kOk;
}

int boss_perm_grad_batch(const double* matrix, int32_t m, const int32_t* input_states,
                         const int32_t* output_states, int32_t len, int32_t count, double* perms, double* grads) {
  if (!matrix || !input_states || !output_states || !perms || !grads || m <= 0 || count < 0 || len <= 0) {
    set_error("null pointer or bad size");
    return kErrArg;
  }
  std::lock_guard<std::mutex> lk(g_api_mutex);
  double2* P2 = (double2*)perms;
  double2* G2 = (double2*)grads;
  std::fill(G2, G2 + (size_t)count * len * len, make_double2(0.0, 0.0));
  std::vector<HostSweep> by_nf[kMaxFactors + 1];
  std::vector<int> which[kMaxFactors + 1];
  bool any = false;
  const bool on_device = count > 0 && plan_on_device(m, count, len, input_states, output_states);
  for (int k = 0; k < count; ++k) {
    HostSweep hs;
    bool need = false;
    double2 v = make_double2(0.0, 0.0);
    const int32_t* S = input_states + (size_t)k * len;
    const int32_t* T = output_states + (size_t)k * len;
    int st = plan_permanent(matrix, m, S, T, len, BOSS_GLYNN, hs, need, v, kPlanGrad, on_device);
    if (st) return st;
    if (!need) {  // no particles: perm = 1, gradient 0
      P2[k] = v;
      continue;
    }
    if (hs.nd + 1 > kMaxDigits) {
      set_error("gradient sweep exceeds the digit limit");
      return kErrLimit;
    }
    which[hs.nf].push_back(k);
    by_nf[hs.nf].push_back(std::move(hs));
    any = true;
  }
  if (!any) return kOk;
  int st;
  Context* cx = context(&st);
  if (!cx) return st;
  for (int nf = 1; nf <= kMaxFactors; ++nf) {
    const std::vector<HostSweep>& sw = by_nf[nf];
    const int n = (int)sw.size();
    if (n == 0) continue;
    // walkers in proportion to the codes, at least 32 codes each (a walker also leaves
    // a (nd + 1) x nf slice; 4 where that leaves SMs idle: one gradient at n = 14 takes
    // 134 us with 32, 70 with 4), whole warps of 8, one wave of resident warps
    double total = 0.0;
    for (const HostSweep& h : sw) total += (double)h.total_codes;
    const int64_t resident = grad_resident_walkers(nf, cx->sm_count);
    const int64_t least = min_codes_per_thread(total, 32, 4, kQuadWalkers, cx->sm_count);
    const double want = std::max<double>(n, std::min<double>((double)resident, total / (double)least));
    const int F = grad_factors(nf);
    std::vector<SweepProblem> probs(n);
    int64_t pool_n = 0, walkers = 0, gparts = 0;
    int row = 0;  // entries of the largest sweep's gradient
    for (int p = 0; p < n; ++p) {
      const HostSweep& h = sw[p];
      SweepProblem& Pp = probs[p];
      const int64_t share = (int64_t)std::floor(want * (double)h.total_codes / total);
      describe_sweep(h, std::max<int64_t>(8, share / 8 * 8), 1, Pp);
      Pp.out_idx = p;
      Pp.thread_begin = walkers;
      Pp.mat_off = pool_n;
      pool_n += (int64_t)rows_of(h);
      Pp.base_off = pool_n;
      pool_n += (int64_t)base_of(h);
      Pp.part_off = gparts;
      const int rows = h.nd + Pp.fixed_digit;
      row = std::max(row, rows * F);
      walkers += Pp.n_threads;
      gparts += Pp.n_threads / 8 * grad_slice(rows, nf);
    }
    size_t off = 0;
    const size_t o_probs = off; off = align_up(off + sizeof(SweepProblem) * n, 256);
    const bool device_rows = sw[0].on_device;
    const size_t o_U = off; off = align_up(off + (device_rows ? sizeof(double2) * (size_t)m * m : 0), 256);
    const size_t o_items = off; off = align_up(off + (device_rows ? sizeof(PlanItem) * n : 0), 256);
    const size_t o_pool = off; off = align_up(off + sizeof(longlong2) * std::max<int64_t>(pool_n, 1), 256);
    const size_t arena_bytes = off, up = device_rows ? o_pool : arena_bytes;
    const size_t out_g = (size_t)n * row, out_p = (size_t)n;
    if ((st = ensure(cx->plans, arena_bytes))) return st;
    const int parts = grad_reduce_parts(walkers, n, row, cx->sm_count);
    const int64_t mid = parts > 1 ? (int64_t)n * parts * (row + 1) : 0;
    if ((st = ensure(cx->gpart, sizeof(double2) * std::max<int64_t>(gparts + mid, 1)))) return st;
    if ((st = ensure(cx->pperm, sizeof(double2) * std::max<int64_t>(walkers / 8, 1)))) return st;
    if ((st = ensure(cx->out, sizeof(double2) * (out_g + out_p)))) return st;
    if ((st = ensure_pinned(cx, std::max(up, sizeof(double2) * (out_g + out_p))))) return st;
    char* h = (char*)cx->pinned;
    memcpy(h + o_probs, probs.data(), sizeof(SweepProblem) * n);
    longlong2* hp = (longlong2*)(h + o_pool);
    int max_entries = 0;
    if (device_rows) memcpy(h + o_U, matrix, sizeof(double2) * (size_t)m * m);
    for (int p = 0; p < n; ++p) {
      if (device_rows) {
        describe_plan(sw[p], probs[p].mat_off, probs[p].base_off, ((PlanItem*)(h + o_items))[p]);
        max_entries = std::max(max_entries, (sw[p].nd + 1) * nf);
        continue;
      }
      std::copy(sw[p].D.begin(), sw[p].D.end(), hp + probs[p].mat_off);
      std::copy(sw[p].base.begin(), sw[p].base.end(), hp + probs[p].base_off);
    }
    char* d = (char*)cx->plans.ptr;
    cudaError_t e = cudaMemcpyAsync(d, h, up, cudaMemcpyHostToDevice, cx->stream);
    if (e != cudaSuccess) return fail_cuda(e, "H2D gradient sweeps");
    if (device_rows) {
      e = launch_plan_rows((const PlanItem*)(d + o_items), n, (const double2*)(d + o_U), m, max_entries,
                           (longlong2*)(d + o_pool), (SweepProblem*)(d + o_probs), cx->stream);
      if (e != cudaSuccess) return fail_cuda(e, "gradient rows");
    }
    const SweepProblem* dp = (const SweepProblem*)(d + o_probs);
    double2 *gpart = (double2*)cx->gpart.ptr, *ppart = (double2*)cx->pperm.ptr;
    if ((e = launch_grad_sweep(nf, dp, n, (const longlong2*)(d + o_pool), walkers, gpart, ppart, cx->stream)) !=
        cudaSuccess)
      return fail_cuda(e, "gradient sweep");
    double2* dout = (double2*)cx->out.ptr;
    if ((e = launch_grad_reduce(nf, dp, n, gpart, ppart, gpart + gparts, parts, dout, dout + out_g, row,
                                cx->stream)) != cudaSuccess)
      return fail_cuda(e, "gradient reduce");
    e = cudaMemcpyAsync(cx->pinned, dout, sizeof(double2) * (out_g + out_p), cudaMemcpyDeviceToHost, cx->stream);
    if (e != cudaSuccess) return fail_cuda(e, "D2H gradients");
    if ((e = cudaStreamSynchronize(cx->stream)) != cudaSuccess) return fail_cuda(e, "gradient sweep");
    const double2* hg = (const double2*)cx->pinned;
    const double2* hpm = hg + out_g;
    for (int p = 0; p < n; ++p) {
      const HostSweep& hs = sw[p];
      const int k = which[nf][p];
      P2[k] = hpm[p];
      double2* gk = G2 + (size_t)k * len * len;
      const int ndt = hs.nd + (hs.fixed_mode >= 0 ? 1 : 0);
      for (int b = 0; b < ndt; ++b) {
        const int bmode = (b < hs.nd) ? hs.digit_mode[b] : hs.fixed_mode;
        for (int f = 0; f < nf; ++f) {
          const int fmode = hs.factor_mode[f];
          const int j = hs.digits_are_outputs ? bmode : fmode;  // output mode
          const int i = hs.digits_are_outputs ? fmode : bmode;  // input mode
          const double2 v = hg[(size_t)p * row + (size_t)b * F + f];
          gk[(size_t)j * len + i].x += v.x;
          gk[(size_t)j * len + i].y += v.y;
        }
      }
    }
  }
  return kOk;
}

int boss_perm_bench(const double* matrix, int32_t m, const int32_t* input_states, const int32_t* output_states,
                    int32_t len, int32_t count, int32_t variant, int32_t n_warmup, int32_t n_steps,
                    int64_t flush_bytes, double* sweep_ms, double* info, double* results) {
  if (!matrix || !input_states || !output_states || m <= 0 || count <= 0 || n_steps <= 0 || !sweep_ms || !info) {
    set_error("null pointer or bad size");
    return kErrArg;
  }
  std::lock_guard<std::mutex> lk(g_api_mutex);
  std::vector<HostSweep> sweeps;
  PlanFor plan = kPlanAny;
  double flops = 0.0;
  for (int k = 0; k < count; ++k) {
    HostSweep hs;
    bool need = false;
    double2 v;
    const int st = plan_permanent(matrix, m, input_states + (size_t)k * len, output_states + (size_t)k * len, len,
                                  variant, hs, need, v, plan);
    if (st) return st;
    if (!need) {
      set_error("benchmark permanents must need a sweep");
      return kErrArg;
    }
    if (!sweeps.empty() && hs.nf != sweeps[0].nf) {
      set_error("benchmark permanents must share one product size");
      return kErrArg;
    }
    if (!sweeps.empty() && hs.layout != sweeps[0].layout && plan == kPlanAny) {  // one kernel for all: start over
      plan = kPlanTemplated;
      sweeps.clear();
      flops = 0.0;
      k = -1;
      continue;
    }
    // per code: nf complex adds, nf - 1 complex products, one signed complex add
    flops += (double)hs.total_codes * (8.0 * hs.nf - 4.0);
    sweeps.push_back(std::move(hs));
  }
  int st;
  Context* cx = context(&st);
  if (!cx) return st;
  SweepBatch B;
  if ((st = sweeps_prepare(cx, sweeps, false, 1, B))) return st;
  if (flush_bytes > 0 && (st = ensure(cx->misc, (size_t)flush_bytes))) return st;
  cudaEvent_t e0, e1;
  cudaEventCreate(&e0);
  cudaEventCreate(&e1);
  cudaError_t e = cudaSuccess;
  for (int it = 0; it < n_warmup + n_steps && !st; ++it) {
    if (flush_bytes > 0) e = cudaMemsetAsync(cx->misc.ptr, it & 0xff, (size_t)flush_bytes, cx->stream);
    if (e != cudaSuccess) break;
    cudaEventRecord(e0, cx->stream);
    st = sweeps_launch(cx, B, e1);
    if (st) break;
    e = cudaEventSynchronize(e1);
    if (e != cudaSuccess) break;
    if (it >= n_warmup) {
      float ms = 0.f;
      cudaEventElapsedTime(&ms, e0, e1);
      sweep_ms[it - n_warmup] = ms;
    }
  }
  cudaEventDestroy(e0);
  cudaEventDestroy(e1);
  if (!st && e != cudaSuccess) st = fail_cuda(e, "perm bench");
  if (st) return st;
  std::vector<double2> out(B.out_elems);
  if ((st = sweeps_collect(cx, B, out.data()))) return st;
  if (results)
    for (int k = 0; k < count; ++k) {
      results[2 * k] = out[k].x;
      results[2 * k + 1] = out[k].y;
    }
  info[0] = B.codes;
  info[1] = flops;
  info[2] = (double)B.L.total_threads;
  info[3] = (double)B.nf;
  // float pairs: nf - 1 renormalised complex products of 38, one complex sum of
  // 16, 15/16 of the codes 16 per factor to move the sums, 1/16 of them 2 per factor
  info[4] = B.ff ? B.codes * (53.125 * B.nf - 22.0) : 0.0;
  return kOk;
}

}  // extern "C"

// ---------------------------------------------------------------------------
// Allocation-free permanents.
//
// Some callers cannot let a library call cudaMalloc: processes that hand all of
// the GPU's memory to their own pool allocator up front and must account for
// every byte, services running under a hard memory cap where a surprise
// allocation can fail or fragment the pool, and latency-sensitive loops that
// avoid cudaMalloc's implicit device synchronisation.  For them
// boss_perm_batch_noalloc runs the same permanent sweep as boss_perm_batch with
// all of its scratch (sweep descriptors, fixed-point rows, per-thread partial
// sums) in one statically sized device array, g_noalloc_scratch below, and
// writes the results into a device buffer the caller owns.
// ---------------------------------------------------------------------------
namespace boss {

constexpr size_t kNoAllocScratchBytes = (size_t)8 << 20;  // 8 MiB, held by every GPU that loads the library
static __device__ __align__(256) unsigned char g_noalloc_scratch[kNoAllocScratchBytes];
// Host-side copy source, page-locked once (cudaHostRegister: no device memory) so
// that its copies are truly asynchronous; an event recorded after each copy is
// waited on before the array is refilled.
alignas(4096) static unsigned char g_noalloc_staging[kNoAllocScratchBytes];
static bool g_noalloc_staging_pinned = false;
static cudaEvent_t g_noalloc_staging_free = nullptr;  // recorded after the last copy out of the staging array

struct NoAllocDevice {
  bool ready = false;
  int sm_count = 0;
  unsigned char* scratch = nullptr;  // device address of g_noalloc_scratch on this device
  cudaEvent_t copied = nullptr;      // this device's staging-copy event
};
constexpr int kNoAllocMaxDevices = 64;
static NoAllocDevice g_noalloc_dev[kNoAllocMaxDevices];

// Once per device, with that device current: the device address of the scratch
// array (its host-side name is only a stand-in), the kernel attributes and the
// staging-copy event; once per process, the staging array is page-locked.
static int noalloc_setup(int device, NoAllocDevice*& out) {
  if (device < 0 || device >= kNoAllocMaxDevices) {
    set_error("device index out of range");
    return kErrArg;
  }
  NoAllocDevice& d = g_noalloc_dev[device];
  if (!d.ready) {
    void* p = nullptr;
    cudaError_t e = cudaGetSymbolAddress(&p, g_noalloc_scratch);
    if (e != cudaSuccess) return fail_cuda(e, "cudaGetSymbolAddress(g_noalloc_scratch)");
    if ((e = cudaDeviceGetAttribute(&d.sm_count, cudaDevAttrMultiProcessorCount, device)) != cudaSuccess)
      return fail_cuda(e, "cudaDeviceGetAttribute");
    if ((e = prepare_sweep_kernels()) != cudaSuccess) return fail_cuda(e, "kernel attributes");
    if ((e = cudaEventCreateWithFlags(&d.copied, cudaEventDisableTiming)) != cudaSuccess)
      return fail_cuda(e, "cudaEventCreate");
    if (!g_noalloc_staging_pinned) {
      e = cudaHostRegister(g_noalloc_staging, sizeof(g_noalloc_staging), cudaHostRegisterPortable);
      if (e != cudaSuccess) return fail_cuda(e, "cudaHostRegister(staging)");
      g_noalloc_staging_pinned = true;
    }
    d.scratch = (unsigned char*)p;
    d.ready = true;
  }
  out = &d;
  return kOk;
}

// Waits until the staging array's last copy has left it (from any device).
static int noalloc_staging_wait() {
  if (!g_noalloc_staging_free) return kOk;
  cudaError_t e = cudaEventSynchronize(g_noalloc_staging_free);
  return e == cudaSuccess ? kOk : fail_cuda(e, "staging copy");
}

// Queues the copy of the first `bytes` of the staging array into the device's
// scratch and marks the staging array busy until it has left.
static int noalloc_stage(NoAllocDevice* dev, size_t bytes, cudaStream_t s) {
  cudaError_t e = cudaMemcpyAsync(dev->scratch, g_noalloc_staging, bytes, cudaMemcpyHostToDevice, s);
  if (e != cudaSuccess) return fail_cuda(e, "H2D staging");
  if ((e = cudaEventRecord(dev->copied, s)) != cudaSuccess) return fail_cuda(e, "event record");
  g_noalloc_staging_free = dev->copied;
  return kOk;
}

// Results that need no sweep (theboss's empty-state rules): out[idx[i]] = val[i].
__global__ void noalloc_scatter_kernel(const int32_t* __restrict__ idx, const double2* __restrict__ val, int n,
                                       double2* __restrict__ out) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) out[idx[i]] = val[i];
}

// One product-size group of a request: its sweeps' layout in the scratch.
struct NoAllocGroup {
  int cls = 0;  // sweep_class
  std::vector<int64_t> nthr;
  int group = 1;
  int64_t threads = 0, parts = 0;
  size_t o_pool = 0, o_part = 0, bytes = 0;
};

}  // namespace boss

extern "C" int boss_perm_batch_noalloc(const double* matrix, int32_t m, const int32_t* input_states,
                                       const int32_t* output_states, int32_t len, int32_t count, int32_t variant,
                                       double* results_device, void* stream) {
  if (!matrix || !input_states || !output_states || !results_device || m <= 0 || count < 0) {
    set_error("null pointer or bad size");
    return kErrArg;
  }
  std::lock_guard<std::mutex> lk(g_api_mutex);
  int device = 0;
  cudaError_t e = cudaGetDevice(&device);
  if (e != cudaSuccess) return fail_cuda(e, "cudaGetDevice");
  NoAllocDevice* dev = nullptr;
  int st = noalloc_setup(device, dev);
  if (st) return st;
  cudaStream_t s = (cudaStream_t)stream;
  double2* out = (double2*)results_device;
  // (1) Plan every permanent and lay out every scratch image; reject the request
  // before anything is queued if one image exceeds the scratch.  The quad kernel's
  // rows take twice the templated kernels': a request too large for them is planned
  // again for those.
  std::vector<HostSweep> by_class[kSweepClasses];
  std::vector<int> which[kSweepClasses];
  std::vector<int32_t> direct_idx;
  std::vector<double2> direct_val;
  std::vector<NoAllocGroup> groups;
  size_t o_dval = 0, direct_bytes = 0, need_bytes = 0;
  // Before that the same plan is tried with more codes a thread (fewer partials).  A request
  // whose first permanent's rows fill the scratch when repeated is planned for the
  // templated kernels at once (6000 of 8 photons 24.7 -> 7.3 ms; 13.7 with one plan and one
  // layout).
  int attempt = 0;  // 0, 1: any kernel, codes spread over idle SMs or not; 2: templated kernels
  if (count > 0) {
    HostSweep hs;  // its sizes only
    bool need = false;
    double2 v;
    if (plan_permanent(matrix, m, input_states, output_states, len, variant, hs, need, v, kPlanFP64, true) == kOk &&
        need && hs.on_device &&
        (sizeof(SweepProblem) + sizeof(longlong2) * (rows_of(hs) + base_of(hs))) * (size_t)count > kNoAllocScratchBytes)
      attempt = 2;
  }
  for (; attempt < 3; ++attempt) {
  groups.clear();
  if (attempt != 1) {
    for (int c = 0; c < kSweepClasses; ++c) {
      by_class[c].clear();
      which[c].clear();
    }
    direct_idx.clear();
    direct_val.clear();
    for (int k = 0; k < count; ++k) {
      HostSweep hs;
      bool need = false;
      double2 v = make_double2(0.0, 0.0);
      st = plan_permanent(matrix, m, input_states + (size_t)k * len, output_states + (size_t)k * len, len, variant, hs,
                          need, v, attempt == 2 ? kPlanTemplated : kPlanFP64);
      if (st) return st;
      if (need) {
        const int c = sweep_class(hs);
        which[c].push_back(k);
        by_class[c].push_back(std::move(hs));
      } else {  // a permanent theboss defines without a sweep (empty states)
        direct_idx.push_back(k);
        direct_val.push_back(v);
      }
    }
  }
  o_dval = align_up(sizeof(int32_t) * direct_idx.size(), 256);
  direct_bytes = o_dval + sizeof(double2) * direct_val.size();
  for (int c = 0; c < kSweepClasses; ++c) {
    const std::vector<HostSweep>& sw = by_class[c];
    const int n = (int)sw.size();
    if (n == 0) continue;
    NoAllocGroup G;
    G.cls = c;
    const int nf = sw[0].nf;
    G.group = split_threads(sw,
                            sw[0].layout == kRowsQuad ? quad_resident_walkers(nf, 0, false, dev->sm_count)
                                                      : sweep_resident_threads(nf, SweepOp::kPerm, dev->sm_count),
                            false, attempt == 0 ? dev->sm_count : 0, G.nthr);
    int64_t pool_n = 0;
    for (int p = 0; p < n; ++p) {
      pool_n += (int64_t)(sw[p].D.size() + sw[p].base.size());
      G.threads += G.nthr[p];
      G.parts += G.nthr[p] / G.group;
    }
    G.o_pool = align_up(sizeof(SweepProblem) * n, 256);
    G.o_part = align_up(G.o_pool + sizeof(longlong2) * (size_t)std::max<int64_t>(pool_n, 1), 256);
    G.bytes = G.o_part + sizeof(double2) * (size_t)G.parts;
    groups.push_back(std::move(G));
  }
  need_bytes = direct_bytes;
  for (const NoAllocGroup& G : groups) need_bytes = std::max(need_bytes, G.bytes);
  if (need_bytes <= kNoAllocScratchBytes) break;
  }
  if (need_bytes > kNoAllocScratchBytes) {
    set_error("request needs " + std::to_string(need_bytes) + " bytes of scratch; the allocation-free entry "
              "point has " + std::to_string(kNoAllocScratchBytes) + " (split the batch)");
    return kErrLimit;
  }
  // (2) The direct results, through the staging array and a scatter kernel.
  if (!direct_idx.empty()) {
    if ((st = noalloc_staging_wait())) return st;
    memcpy(g_noalloc_staging, direct_idx.data(), sizeof(int32_t) * direct_idx.size());
    memcpy(g_noalloc_staging + o_dval, direct_val.data(), sizeof(double2) * direct_val.size());
    if ((st = noalloc_stage(dev, direct_bytes, s))) return st;
    const int nd = (int)direct_idx.size();
    noalloc_scatter_kernel<<<(nd + 127) / 128, 128, 0, s>>>((const int32_t*)dev->scratch,
                                                            (const double2*)(dev->scratch + o_dval), nd, out);
    if ((e = cudaGetLastError()) != cudaSuccess) return fail_cuda(e, "scatter launch");
  }
  // (3) One sweep launch per product size; each image reuses the scratch from its
  // start (stream order keeps it behind the previous image's kernels).
  for (const NoAllocGroup& G : groups) {
    const std::vector<HostSweep>& sw = by_class[G.cls];
    const int nf = sw[0].nf;
    const int n = (int)sw.size();
    if ((st = noalloc_staging_wait())) return st;
    SweepProblem* hp = (SweepProblem*)g_noalloc_staging;
    longlong2* hpool = (longlong2*)(g_noalloc_staging + G.o_pool);
    int64_t pool_at = 0, thread_at = 0;
    for (int p = 0; p < n; ++p) {
      const HostSweep& h = sw[p];
      SweepProblem& P = hp[p];
      describe_sweep(h, G.nthr[p], G.group, P);
      P.out_idx = which[G.cls][p];  // the reduction writes straight into the caller's buffer
      P.thread_begin = thread_at;
      P.mat_off = pool_at;
      std::copy(h.D.begin(), h.D.end(), hpool + pool_at);
      pool_at += (int64_t)h.D.size();
      P.base_off = pool_at;
      std::copy(h.base.begin(), h.base.end(), hpool + pool_at);
      pool_at += (int64_t)h.base.size();
      P.part_off = thread_at / G.group;
      thread_at += G.nthr[p];
    }
    if ((st = noalloc_stage(dev, G.o_part, s))) return st;
    SweepLaunch L;
    L.probs = (const SweepProblem*)dev->scratch;
    L.n_probs = n;
    L.pool = (const longlong2*)(dev->scratch + G.o_pool);
    L.total_threads = G.threads;
    L.partials = (double2*)(dev->scratch + G.o_part);
    L.grid = (int)((G.threads + 127) / 128);
    L.quad = sw[0].layout == kRowsQuad;
    if ((e = launch_sweep(nf, SweepOp::kPerm, L, s)) != cudaSuccess) return fail_cuda(e, "sweep launch");
    if ((e = launch_perm_reduce(L.probs, n, L.partials, out, s)) != cudaSuccess) return fail_cuda(e, "reduce launch");
  }
  return kOk;
}
