// Host runtime and C ABI of poremaps_gb300 (see include/poremaps.h).
//
// The calc_flow loop (reference src/calc_flow.cc:53-169) runs on the host and
// drives device sweeps in blocks that end exactly at the iterations where the
// reference evaluates convergence (it % it_eval == 0 && it > 1000), so the
// stopping iteration, the log rows and the final fields follow the reference's
// control flow.
#include <math.h>
#include <stdarg.h>
#include <stdio.h>
#include <stdlib.h>
#include <string.h>

#include <algorithm>
#include <atomic>
#include <array>
#include <chrono>
#include <map>
#include <mutex>
#include <string>
#include <thread>
#include <vector>

#include "../../include/poremaps.h"
#include "pm_api_internal.h"
#include "pm_compact.h"
#include "pm_internal.h"

using namespace pm;

namespace {

thread_local std::string g_err;

}  // namespace

namespace pm {

pm_status set_error(pm_status st, const char* fmt, ...) {
  char buf[512];
  va_list ap;
  va_start(ap, fmt);
  vsnprintf(buf, sizeof buf, fmt, ap);
  va_end(ap);
  g_err = buf;
  return st;
}

// Countdown of pm_debug_fail_alloc: the allocation that takes it from 1 to 0
// fails as cudaMalloc does when the device is out of memory.
std::atomic<int> g_fail_alloc{0};

// pm_debug_launch_forms: the form problems made from now on take, -1 their own.
std::atomic<int> g_force_form64{-1}, g_force_variant{-1};

// Device blocks of destroyed problems, kept for the next ones: a call that
// makes and destroys its problems (the tensor's three rotations, the server's
// samples) spends 0.2 to 2 ms a problem in cudaMalloc and cudaFree otherwise
// (the tensor of a 128^3 pack: 27.9 -> 26.9 ms, 24 server samples 63 -> 59 ms).
// At most kPoolBytes are kept; they count as free memory, an allocation of this
// library that fails gives them back to the device and is tried again, and
// pm_release_memory gives them back to others.  A block is put here only once
// no work uses it.
constexpr size_t kPoolBytes = 1ull << 30;
struct PoolBlock {
  void* p;
  size_t bytes;
  int dev;
};
std::mutex g_pool_mu;
std::vector<PoolBlock> g_pool;
std::map<void*, PoolBlock> g_pool_out;  // every block dev_alloc handed out
size_t g_pool_bytes = 0;

bool pool_give_back() {  // g_pool_mu held; whether there was any
  const bool any = !g_pool.empty();
  for (auto& b : g_pool) cudaFree(b.p);
  g_pool.clear();
  g_pool_bytes = 0;
  return any;
}

bool pool_release() {
  std::lock_guard<std::mutex> lk(g_pool_mu);
  return pool_give_back();
}

// An allocation, tried again when the kept blocks are given back; one that
// failed is reported by its own status only, not by the next launch's
// cudaGetLastError as well.
template <typename Alloc>
cudaError_t alloc_or_release(Alloc&& alloc, bool (*release)()) {
  cudaError_t e = alloc();
  if (e == cudaErrorMemoryAllocation) {
    cudaGetLastError();
    if (release()) e = alloc();
  }
  if (e != cudaSuccess) cudaGetLastError();
  return e;
}

cudaError_t cuda_alloc(void** p, size_t bytes) {
  return alloc_or_release([&] { return cudaMalloc(p, bytes); }, pool_release);
}

cudaError_t cuda_alloc_async(void** p, size_t bytes, cudaStream_t st) {
  return alloc_or_release([&] { return cudaMallocAsync(p, bytes, st); }, pool_release);
}

template <typename T>
cudaError_t dev_alloc(T** ptr, size_t bytes) {
  int n = g_fail_alloc.load();
  while (n > 0 && !g_fail_alloc.compare_exchange_weak(n, n - 1)) {
  }
  *ptr = nullptr;
  if (n == 1) return cudaErrorMemoryAllocation;
  int dev = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) return e;
  bytes = bytes > 0 ? bytes : 1;
  std::lock_guard<std::mutex> lk(g_pool_mu);
  size_t best = g_pool.size();  // the smallest that holds it and wastes at most a quarter
  for (size_t i = 0; i < g_pool.size(); ++i)
    if (g_pool[i].dev == dev && g_pool[i].bytes >= bytes && g_pool[i].bytes - bytes <= bytes / 4 &&
        (best == g_pool.size() || g_pool[i].bytes < g_pool[best].bytes))
      best = i;
  void* p = nullptr;
  if (best < g_pool.size()) {
    p = g_pool[best].p;
    bytes = g_pool[best].bytes;
    g_pool_bytes -= bytes;
    g_pool.erase(g_pool.begin() + best);
  } else {
    e = alloc_or_release([&] { return cudaMalloc(&p, bytes); }, pool_give_back);
    if (e != cudaSuccess) return e;
  }
  g_pool_out[p] = {p, bytes, dev};
  *ptr = (T*)p;
  return cudaSuccess;
}

// p: from dev_alloc, no longer used by any work; null does nothing.
void dev_free(void* p) {
  if (!p) return;
  std::lock_guard<std::mutex> lk(g_pool_mu);
  auto it = g_pool_out.find(p);
  const PoolBlock b = it->second;
  const size_t bytes = b.bytes;
  g_pool_out.erase(it);
  if (bytes > kPoolBytes) {
    cudaFree(p);
    return;
  }
  while (g_pool_bytes + bytes > kPoolBytes) {  // the oldest make room
    cudaFree(g_pool.front().p);
    g_pool_bytes -= g_pool.front().bytes;
    g_pool.erase(g_pool.begin());
  }
  g_pool.push_back(b);
  g_pool_bytes += bytes;
}

// Sub-buffers of one device allocation, each on a 256-byte boundary (the
// alignment cudaMalloc gives): a problem's fixed buffers and its compact
// store are one allocation each, so that concurrent set-ups (the tensor's
// three rotations, the server's admissions) make a few driver calls each
// instead of one per buffer.
struct Carve {
  size_t bytes = 0;
  size_t take(size_t n) {
    const size_t o = bytes;
    bytes = (bytes + n + 255) & ~(size_t)255;
    return o;
  }
};

// Pinned host result buffers (256 bytes per problem) from a process-wide pool
// of 64 KB slabs that lives until exit: cudaMallocHost is a slow driver call
// and cudaFreeHost waits for the device.  A buffer goes back to the pool only
// after its problem's stream is synchronised.
static std::mutex g_pin_mu;
static std::vector<double*> g_pin_free;

size_t pool_bytes() {
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess) return 0;
  std::lock_guard<std::mutex> lk(g_pool_mu);
  size_t n = 0;
  for (auto& b : g_pool)
    if (b.dev == dev) n += b.bytes;
  return n;
}

static cudaError_t pinned_slot(double** out) {
  std::lock_guard<std::mutex> lk(g_pin_mu);
  if (g_pin_free.empty()) {
    void* slab = nullptr;
    cudaError_t e = cudaMallocHost(&slab, 65536);
    if (e != cudaSuccess) return e;
    for (int i = 0; i < 65536 / 256; ++i) g_pin_free.push_back((double*)((char*)slab + 256 * i));
  }
  *out = g_pin_free.back();
  g_pin_free.pop_back();
  return cudaSuccess;
}

static void pinned_release(double* p) {
  if (!p) return;
  std::lock_guard<std::mutex> lk(g_pin_mu);
  g_pin_free.push_back(p);
}

pm_status cuda_error(cudaError_t e, const char* where) {
  if (e == cudaErrorMemoryAllocation)
    return set_error(PM_ERR_NOMEM, "%s: %s", where, cudaGetErrorString(e));
  return set_error(PM_ERR_CUDA, "%s: %s", where, cudaGetErrorString(e));
}

}  // namespace pm

#define CK(expr)                                        \
  do {                                                  \
    cudaError_t _e = (expr);                            \
    if (_e != cudaSuccess) return cuda_error(_e, #expr); \
  } while (0)

namespace {

pm_status validate(const pm_params* p) {
  if (!p) return set_error(PM_ERR_INVALID, "params is NULL");
  if (p->size[0] < 1 || p->size[1] < 1 || p->size[2] < 1)
    return set_error(PM_ERR_INVALID, "size_x_y_z must be positive (got %d %d %d)", p->size[0],
                     p->size[1], p->size[2]);
  if ((long long)p->size[0] * p->size[1] * p->size[2] > (1LL << 31) - 1)
    return set_error(PM_ERR_INVALID, "domain larger than 2^31 voxels");
  if (p->boundary_method < 0 || p->boundary_method > 4)
    return set_error(PM_ERR_INVALID, "boundary_method must be 0..4 (got %d)", p->boundary_method);
  if (p->solving_algorithm < 1 || p->solving_algorithm > 3)
    return set_error(PM_ERR_INVALID, "solving_algorithm must be 1, 2 or 3 (got %u)",
                     p->solving_algorithm);
  if (p->it_eval <= 0 || p->it_write <= 0)
    return set_error(PM_ERR_INVALID, "it_eval and it_write must be positive");
  if (p->order < -1 || p->order > 2) return set_error(PM_ERR_INVALID, "bad order %d", p->order);
  if (p->precision < 0 || p->precision > 1)
    return set_error(PM_ERR_INVALID, "bad precision %d", p->precision);
  if (!(p->eps_fixed_point >= 0) || !isfinite(p->eps_fixed_point))
    return set_error(PM_ERR_INVALID, "eps_fixed_point must be finite and >= 0");
  {
    const int* b = p->brick;
    const bool none = !b[0] && !b[1] && !b[2], all = b[0] > 0 && b[1] > 0 && b[2] > 0;
    if (!none && !all)
      return set_error(PM_ERR_INVALID, "brick must be 0 0 0 or three positive extents");
  }
  if (p->kernel < -1 || p->kernel > 13) return set_error(PM_ERR_INVALID, "bad kernel %d", p->kernel);
  if (p->kernel == 4 && p->brick[0] && pm::brick_shape_of(p->brick[0], p->brick[1], p->brick[2]) < 0)
    return set_error(PM_ERR_INVALID, "kernel 4 bricks are 32x8x8, 32x8x4 or 32x4x4");
  if (p->precision == PM_PREC_MIXED && p->solving_algorithm == 1)
    return set_error(PM_ERR_INVALID,
                     "mixed precision sweeps in Jacobi order, which diverges for solver 1 "
                     "(explicit pressure update); use solver 2/3 or precision fp64");
  return PM_OK;
}

// Whether sweeps go from one FP64 state to the other (whose solid voxels and
// wall halos no sweep writes, so both start as copies).  The mixed form has one
// and the reference order sweeps in place, its second state the exchange: a
// copy there was 1.3 of the 62.5 ms of 201 iterations of a 512^3 medium.
bool two_states(const pm_problem* pr) {
  return pr->precision == PM_PREC_FP64 && pr->order != PM_ORDER_REFERENCE;
}

pm_status device_sync(pm_problem* pr, const char* where) {
  cudaError_t e = cudaStreamSynchronize(pr->st);
  if (e != cudaSuccess) return cuda_error(e, where);
  int* flags[4] = {pr->zp ? zmarch_error_flag(pr->zp) : nullptr,
                   pr->bp ? brick_error_flag(pr->bp) : nullptr,
                   (pr->kern == 11 || pr->kern == 12) ? pr->cerr : nullptr,
                   pr->werr};
  for (int* f : flags) {
    if (!f) continue;
    int flag = 0;
    e = cudaMemcpy(&flag, f, sizeof(int), cudaMemcpyDeviceToHost);
    if (e != cudaSuccess) return cuda_error(e, where);
    if (flag) {
      cudaMemset(f, 0, sizeof(int));
      return set_error(PM_ERR_CUDA, "%s: a wait of the sweep timed out", where);
    }
  }
  return PM_OK;
}

// The FP32 correction sweep e_out = L(e_in) + r of the mixed form.
pm_status correction_sweep(pm_problem* pr, int src) {
  if (pr->kern == 13 && pr->crec) {
    CK(launch_dc_inner_cr(pr->Ec[src], pr->Ec[1 - src], pr->Rc, pr->crec, pr->cslot2, pr->nlist,
                          pr->solver, pr->cvar, pr->st));
  } else if (pr->kern == 13) {  // a medium whose offsets no record holds
    CK(launch_dc_inner_c(pr->Ec[src], pr->Ec[1 - src], pr->Rc, pr->cmeta, pr->cslot4,
                         pr->cslot2, pr->nlist, pr->solver, 5, pr->st));
  } else if (pr->kern == 11 || pr->kern == 12) {
    CK(launch_dc_inner_cb(pr->Ec[src], pr->Ec[1 - src], pr->Rc, pr->cmeta, pr->cslot4,
                          pr->cslot2, pr->nlist, pr->solver, pr->kern == 11 ? 5 : 4, pr->cerr,
                          pr->st));
  } else if (pr->compact()) {
    CK(launch_dc_inner_c(pr->Ec[src], pr->Ec[1 - src], pr->Rc, pr->cmeta, pr->cslot4,
                         pr->cslot2, pr->nlist, pr->solver, pr->kern - 5, pr->st));
  } else if (pr->zp) {
    CK(zmarch_inner(pr->zp, src, pr->E[1 - src], pr->g, pr->solver, pr->st));
  } else if (pr->bp) {
    CK(brick_inner(pr->bp, src, pr->E[1 - src], pr->R, pr->list, pr->g, pr->solver, pr->st));
  } else if (pr->kern >= 5) {
    CK(launch_dc_inner_pf(pr->E[src], pr->E[1 - src], pr->R, pr->codes, pr->list, pr->nlist,
                          pr->g, pr->solver, 9 - pr->kern, pr->st));
  } else if (pr->kern == 2) {
    CK(launch_dc_inner_occ(pr->E[src], pr->E[1 - src], pr->R, pr->codes, pr->list, pr->nlist,
                           pr->g, pr->solver, pr->st));
  } else {
    CK(launch_dc_inner(pr->E[src], pr->E[1 - src], pr->R, pr->codes, pr->list, pr->nlist, pr->g,
                       pr->solver, pr->st));
  }
  return PM_OK;
}

// Launch form of an FP64 phase over n voxels: the one that won alone
// (choose_fp64_shapes), or, for problems that share the device, what suits
// them all.  Where their states exceed L2, the whole stencil in plain launches:
// overlapped CTAs that wait take the place of other problems' CTAs, and the
// reduced loads gain little there (three 128^3 packs, red-black: 151 us against
// 167 with 2 CTAs per SM and 156 with 3; three 96^3 media 100, 115, 104; a tensor
// of a 128^3 pack 157 against 170).  Within L2, 3 CTAs per SM once the problems'
// blocks no longer fit beside each other (three 48^3 media, Jacobi: 12 us
// against 14 whole and 15.5 with 2; 56^3 red-black 19, 22.5, 24.6), else as alone.
int form64(const pm_problem* pr, int phase, int n) {
  if (pr->share <= 1 || pr->pf64_forced) return pr->pf64[phase];
  const size_t states = (size_t)pr->share * 2 * 4 * sizeof(double) * (size_t)pr->g.alloc64;
  if (states > kL2Bytes) return kForm64Whole;
  return (long long)pr->share * ((n + 255) / 256) > 3LL * sm_count() ? kForm64Three
                                                                     : pr->pf64[phase];
}

// An iteration's sweeps A -> B (fused exchange + reapply) of the FP64 forms.
pm_status sweeps64(pm_problem* pr, Fields<double> A, Fields<double> B) {
  auto sweep = [&](int phase, const int* list, int n) {
    return launch_sweep64(A, B, pr->codes, list, n, pr->g, pr->solver, pr->exact, phase, pr->st,
                          form64(pr, phase, n));
  };
  if (pr->order == PM_ORDER_JACOBI) {
    CK(sweep(0, pr->list, pr->nlist));
  } else {
    CK(sweep(1, pr->list, pr->nred));
    CK(sweep(2, pr->list + pr->nred, pr->nlist - pr->nred));
  }
  return PM_OK;
}

// One iteration of the FP64 forms: sweep, swap.
pm_status iterate64(pm_problem* pr) {
  pm_status s = sweeps64(pr, pr->F[pr->cur], pr->F[1 - pr->cur]);
  pr->cur = 1 - pr->cur;
  return s;
}

// Launch form of each FP64 phase (kForm64*), timed on the problem.  The whole
// stencil is kept unless another form is 1 % faster: it is, where the voxels are
// dense or their states exceed L2 (Jacobi of a 256^3 medium of porosity 0.6 538 us
// against 549 with the reduced loads, 512^3 4,253 against 4,346, red-black of
// 400^3 2,081 against 2,141), the reduced loads where they are not (red-black of
// a 48^3 medium 8.2 us against 11.4, of a 256^3 one of porosity 0.2 252 against
// 285), and the lists' lengths decide how evenly the waves of 2 and 3 end (a
// 97x61x118 pack sweeps in 21.9 us with 2 and 25.7 with 3, a 128^3 one in 59.8
// and 57.6).
// All give identical fields; the trials sweep the two states, which are set up
// again afterwards.
pm_status choose_fp64_shapes(pm_problem* pr) {
  if (pr->exact) return PM_OK;
  if (const int forced = g_force_form64.load(); forced >= 0) {
    for (int& f : pr->pf64) f = forced;
    pr->pf64_forced = true;
    return PM_OK;
  }
  static std::mutex mu;
  static std::map<std::array<long long, 7>, std::array<int, 3>> tuned;
  std::lock_guard<std::mutex> lock(mu);
  const std::array<long long, 7> key = {
      pr->g.nx, pr->g.ny, pr->g.nz, pr->solver, pr->prm.boundary_method, pr->order,
      (long long)llround(20.0 * (double)pr->nlist / (double)pr->g.nvox)};
  auto hit = tuned.find(key);
  if (hit != tuned.end()) {
    for (int i = 0; i < 3; ++i) pr->pf64[i] = hit->second[i];
    return PM_OK;
  }
  // whole iterations in turn between the two states, as a solve runs them: every
  // form once, then those within a tenth of the best again where iterations are
  // short; one voxel per thread only where they are very short (it wins by the
  // end of a wave if at all).  A 100^3 Jacobi problem of a new shape is set up in
  // 1.63 ms so, 2.24 with nine iterations of every form.
  constexpr float kShort = 0.25f, kVeryShort = 0.02f;  // ms an iteration
  float t[kForms64];
  auto set = [&](int form) { for (int& f : pr->pf64) f = form; };
  auto trial = [&](int form, int untimed, int timed) -> pm_status {
    set(form);
    pm_status s = PM_OK;
    for (int r = 0; r < untimed && s == PM_OK; ++r) s = iterate64(pr);
    if (s != PM_OK) return s;
    CK(cudaEventRecord(pr->ev0, pr->st));
    for (int r = 0; r < timed && s == PM_OK; ++r) s = iterate64(pr);
    CK(cudaEventRecord(pr->ev1, pr->st));
    if (s == PM_OK) s = device_sync(pr, "FP64 sweep shape");
    float ms = 0.f;
    if (s == PM_OK) CK(cudaEventElapsedTime(&ms, pr->ev0, pr->ev1));
    t[form] = std::min(t[form], ms / timed);
    return s;
  };
  for (float& x : t) x = 1e30f;
  pm_status s;
  for (int form = kForms64 - 1; form >= 0; --form)
    if (form != kForm64One || t[kForm64Whole] < kVeryShort)
      if ((s = trial(form, 1, 2)) != PM_OK) return s;
  const float near_best = 1.1f * *std::min_element(t, t + kForms64);
  for (int form = kForms64 - 1; form >= 0; --form)
    if (t[form] <= near_best && t[form] < kShort && (s = trial(form, 0, 4)) != PM_OK) return s;
  int best = kForm64Whole;
  for (int form = 0; form < kForm64Whole; ++form)
    if (t[form] < 0.99f * t[kForm64Whole] && t[form] < t[best]) best = form;
  set(best);
  pr->cur = 0;
  CK(launch_init64(pr->F[0], pr->codes, pr->g, pr->st));
  CK(launch_copy_fields64(pr->F[1], pr->F[0], pr->g, pr->st));
  tuned[key] = {pr->pf64[0], pr->pf64[1], pr->pf64[2]};
  return device_sync(pr, "FP64 sweep shape");
}

// Correction-sweep kernels of the mixed form: 0 TMA z-march with 32 x 16
// tiles, 3 the same with 32 x 8 tiles, 1 fluid-list gather, 2 fluid-list
// gather compiled for four blocks per SM, 4 TMA bricks (32x8x8, 32x8x4 or
// 32x4x4 voxels per CTA, the fluid list in the same brick order), 5,
// 6 and 7 persistent fluid-list gather with the list prefetched (4 / 3 / 2
// CTAs per SM), 8, 9 and 10 persistent sweep over the compact store
// (pm_compact.cu: fluid voxels only, six precomputed neighbour positions per
// voxel; 3 / 4 CTAs per SM with the next positions prefetched, 5 without),
// 11 and 12 the same sweep with each chunk's positions staged in shared
// memory by bulk copies (5 / 4 CTAs per SM), 13 the sweep over packed records
// of the compact store (16 bytes of index data per voxel instead of 28).
// kernel < 0 takes 13 and times its launch variants on this problem (a few
// launches each; the correction buffers are scratch until the first residual
// sweep); where the records cannot hold a medium's offsets it times the other
// list kernels and keeps the fastest.
pm_status zero_corrections(pm_problem* pr) {
  if (pr->E[0]) {
    CK(launch_zero4(pr->E[0], pr->g, pr->st));
    CK(launch_zero4(pr->E[1], pr->g, pr->st));
  }
  if (pr->Ec[0])
    CK(cudaMemsetAsync(pr->c_base, 0, 2 * sizeof(float4) * ((size_t)pr->nlist + 1), pr->st));
  return PM_OK;
}

// Frees the correction store the chosen kernel does not use.
void release_unused_store(pm_problem* pr) {
  if (pr->compact()) {
    cudaStreamSynchronize(pr->st);
    dev_free(pr->f32_base);
    pr->f32_base = nullptr;
    pr->E[0] = pr->E[1] = pr->R = nullptr;
  } else {
    cudaStreamSynchronize(pr->st);
    dev_free(pr->carena);
    dev_free(pr->crec_own);
    pr->carena = nullptr;
    pr->crec = pr->crec_own = nullptr;
    pr->compact_ready = false;
    pr->cerr = nullptr;
    pr->c_base = pr->Ec[0] = pr->Ec[1] = pr->Rc = nullptr;
    pr->cslot4 = nullptr;
    pr->cslot2 = nullptr;
    pr->cmeta = nullptr;
    pr->cwords = nullptr;
  }
}

// Tuned correction-sweep choices: (kernel, brick order of the fluid list) per
// (size, solver, boundary method, porosity bucket, whether the packed records
// hold the medium, which decides the candidates).  The choice depends on the
// medium's size, porosity and boundary family, not on its exact pattern, and
// every candidate gives bitwise identical fields: problems alike (e.g. the
// rotated runs of one tensor) share one tuning, and concurrent tunings are
// serialised instead of timing each other's noise.
struct Cand {
  int k, b[3];
  int var = 0;  // kernel 13: launch variant (launch_dc_inner_cr)
};
using TuneKey = std::array<long long, 7>;
std::mutex g_tune_mu;
std::map<TuneKey, Cand> g_tuned;

TuneKey tune_key(const pm_problem* pr) {
  return {pr->g.nx, pr->g.ny, pr->g.nz, pr->solver, pr->prm.boundary_method,
          (long long)llround(20.0 * (double)pr->nlist / (double)pr->g.nvox),
          compact_records_fit(pr->g, pr->nlist)};
}

// The kernel a problem will use if it is already known (pinned, the packed
// records, or tuned for a problem alike), else -1: problem creation then
// allocates only its store.
int known_kernel(const pm_problem* pr, int kernel) {
  if (kernel >= 0) return kernel;
  if (compact_records_fit(pr->g, pr->nlist)) return 13;
  std::lock_guard<std::mutex> lock(g_tune_mu);
  auto hit = g_tuned.find(tune_key(pr));
  return hit != g_tuned.end() ? hit->second.k : -1;
}

pm_status choose_correction_kernel(pm_problem* pr, int kernel) {
  const bool tma = zmarch_available() != 0;
  static const int kLex[3] = {0, 0, 0};
  // set up kernel k with the fluid list in brick order b (k 1, 2, 4); the
  // compact store (k 8) needs the lexicographic list
  auto make = [&](int k, const int* b) -> pm_status {
    if (pr->zp) { zmarch_destroy(pr->zp); pr->zp = nullptr; }
    if (pr->bp) { brick_destroy(pr->bp); pr->bp = nullptr; }
    pr->kern = k;
    const bool cpt = k >= 8 && k <= 13;
    if (!(cpt ? pr->c_base : pr->f32_base))
      return set_error(PM_ERR_INVALID, "the correction store of kernel %d is not allocated", k);
    if (cpt) b = kLex;
    // the list is rebuilt only when its order changes (creation builds it
    // lexicographic), and the compact store is set up once per list order
    if (b[0] != pr->brick[0] || b[1] != pr->brick[1] || b[2] != pr->brick[2]) {
      int* dcount = (int*)pr->dout;
      CK(launch_fluid_list(pr->codes, pr->g, pr->list, dcount, pr->st, b[0], b[1], b[2]));
      for (int i = 0; i < 3; ++i) pr->brick[i] = b[i];
      pr->compact_ready = false;
    }
    if (cpt && !pr->compact_ready) {
      CK(compact_setup(pr->codes, pr->g, pr->list, pr->nlist, pr->cwords, pr->cslot4,
                       pr->cslot2, pr->cmeta, pr->st));
      pr->compact_ready = true;
    }
    if (k == 13 && !pr->crec && compact_records_fit(pr->g, pr->nlist)) {
      // pinned: records of their own (the footprint counts them); else they
      // take the place of the slots
      pr->crec = pr->crec_own ? pr->crec_own : (uint4*)pr->cslot4;
      CK(compact_records(pr->cmeta, pr->cslot4, pr->cslot2, pr->nlist, pr->crec, pr->cslot2,
                         pr->st));
      // the first sweep may follow directly, and it reads records before it
      // waits for the launch before it (ld_record)
      pm_status s = device_sync(pr, "packed records");
      if (s != PM_OK) return s;
    }
    if (k == 0 || k == 3)
      CK(zmarch_create(&pr->zp, pr->g, pr->E[0], pr->E[1], pr->R, pr->codes, 0, k == 3));
    if (k == 4)
      CK(brick_create(&pr->bp, pr->g, pr->E[0], pr->E[1], pr->codes, pr->list, pr->nlist,
                      brick_shape_of(b[0], b[1], b[2]), pr->st));
    return PM_OK;
  };
  if (kernel >= 0) {
    if ((kernel == 0 || kernel == 3 || kernel == 4) && !tma) kernel = 1;
    const int* b = pr->prm.brick;
    static const int kBrick0[3] = {32, 8, 8};
    if (kernel == 4 && !b[0]) b = kBrick0;
    pm_status s = make(kernel, (kernel == 0 || kernel == 3) ? kLex : b);
    if (s != PM_OK) return s;
    return device_sync(pr, "kernel choice");
  }
  std::lock_guard<std::mutex> lock(g_tune_mu);
  const TuneKey key = tune_key(pr);
  auto hit = g_tuned.find(key);
  if (hit != g_tuned.end()) {
    pm_status s = make(hit->second.k, hit->second.b);
    if (s != PM_OK) return s;
    pr->cvar = hit->second.var;
    release_unused_store(pr);
    return device_sync(pr, "kernel choice");
  }
  // The packed records win on every medium measured (pm_compact.cu), so only
  // their launch variants are timed.  Without them: the TMA kernels (0, 3, 4)
  // and the bulk-staged compact sweeps (11, 12) lose on every medium and are
  // left to explicit choice.
  std::vector<Cand> cands;
  if (compact_records_fit(pr->g, pr->nlist))
    cands = {{13, {0, 0, 0}, 0}, {13, {0, 0, 0}, 1}, {13, {0, 0, 0}, 2}};
  else
    cands = {{10, {0, 0, 0}}, {9, {0, 0, 0}}, {8, {0, 0, 0}}, {6, {0, 0, 0}},
             {6, {32, 8, 8}}, {5, {0, 0, 0}}, {7, {0, 0, 0}}, {2, {0, 0, 0}}};
  const int nc = (int)cands.size();
  // Each candidate: the best of three timings of five sweeps.  Among the list
  // kernels the first is kept unless another one is at least 5 % faster: timed
  // alone 10, 9 and 8 come within 1 % of each other (10.4 us on the 128^3
  // sphere pack), but when problems share the device more resident warps win,
  // and they are ordered by those.  The launch variants of the records hold the
  // same warps: 2 % (512^3: 254 us with CTAs of 1024 threads, 267 with 256).
  const float margin = cands[0].k == 13 ? 0.98f : 0.95f;
  std::vector<float> t(nc);
  for (int i = 0; i < nc; ++i) {
    pm_status s;
    if ((s = make(cands[i].k, cands[i].b)) != PM_OK) return s;
    pr->cvar = cands[i].var;
    for (int w = 0; w < 2; ++w)
      if ((s = correction_sweep(pr, 0)) != PM_OK) return s;
    t[i] = 1e30f;
    for (int trial = 0; trial < 3; ++trial) {
      CK(cudaEventRecord(pr->ev0, pr->st));
      for (int r = 0; r < 5; ++r)
        if ((s = correction_sweep(pr, 0)) != PM_OK) return s;
      CK(cudaEventRecord(pr->ev1, pr->st));
      if ((s = device_sync(pr, "kernel autotune")) != PM_OK) return s;
      float ms = 0.f;
      CK(cudaEventElapsedTime(&ms, pr->ev0, pr->ev1));
      if (ms < t[i]) t[i] = ms;
    }
  }
  int bi = 0;
  for (int i = 1; i < nc; ++i)
    if (t[i] < t[bi]) bi = i;
  if (t[bi] > margin * t[0]) bi = 0;
  g_tuned[key] = cands[bi];
  pm_status s = make(cands[bi].k, cands[bi].b);
  if (s != PM_OK) return s;
  pr->cvar = cands[bi].var;
  if ((s = zero_corrections(pr)) != PM_OK) return s;
  if ((s = device_sync(pr, "kernel autotune")) != PM_OK) return s;
  release_unused_store(pr);
  return PM_OK;
}

pm_status dc_flush(pm_problem* pr) {
  if (pr->dc_pos > 0) {
    if (pr->compact())
      CK(launch_dc_correct_c(pr->F[pr->cur], pr->Ec[pr->ecur], pr->list, pr->nlist, pr->g,
                             pr->st));
    else
      CK(launch_dc_correct_list(pr->F[pr->cur], pr->E[pr->ecur], pr->list, pr->nlist, pr->g,
                                pr->st));
    pr->dc_pos = 0;
  }
  return PM_OK;
}

}  // namespace

pm_status pm::problem_flush(pm_problem* pr) { return dc_flush(pr); }

pm_status pm::problem_pack(pm_problem* pr) {
  if (!pr->compact() || pr->crec || !compact_records_fit(pr->g, pr->nlist)) return PM_OK;
  pr->crec = (uint4*)pr->cslot4;
  pr->kern = 13;
  CK(compact_records(pr->cmeta, pr->cslot4, pr->cslot2, pr->nlist, pr->crec, pr->cslot2, pr->st));
  return PM_OK;
}

namespace {

pm_status iterate_mixed(pm_problem* pr) {
  if (pr->dc_pos == 0) {
    if (pr->compact())
      CK(launch_dc_residual_c(pr->F[pr->cur], pr->Rc, pr->Ec[pr->ecur], pr->codes, pr->list,
                              pr->nlist, pr->g, pr->solver, pr->st));
    else
      CK(launch_dc_residual(pr->F[pr->cur], pr->R, pr->E[pr->ecur], pr->codes, pr->list,
                            pr->nlist, pr->g, pr->solver, pr->st));
  } else {
    pm_status s = correction_sweep(pr, pr->ecur);
    if (s != PM_OK) return s;
    pr->ecur = 1 - pr->ecur;
  }
  pr->dc_pos++;
  // the FP64 correction lands after every sweep whose iteration index is a
  // multiple of mixed_inner (with mixed_inner = it_eval: on every iteration
  // the reference evaluates convergence at)
  if (pr->iteration % pr->mixed_inner == 0) return dc_flush(pr);
  return PM_OK;
}

}  // namespace

namespace {

pm_status iterate_direct(pm_problem* pr, int n) {
  for (int i = 0; i < n; ++i) {
    if (pr->order == PM_ORDER_REFERENCE) {
      // in place: the second state's memory is the sweep's exchange
      CK(launch_wave(pr->F[0], pr->codes, pr->g, pr->solver, pr->f64_base[1], pr->werr,
                     pr->st));
    } else {
      pm_status s = pr->precision == PM_PREC_MIXED ? iterate_mixed(pr) : iterate64(pr);
      if (s != PM_OK) return s;
    }
    pr->iteration++;
    pr->sweeps_done++;
  }
  return PM_OK;
}

constexpr int kGraphMinSweeps = 16;  // shorter blocks are launched directly
constexpr size_t kGraphCache = 8;

}  // namespace

// A block of n sweeps runs as one CUDA graph: the
// first time a (length, parity state) occurs the launches are captured while
// the host bookkeeping advances as usual, later blocks with the same start
// state replay the graph and apply the recorded end state.  Graph launches
// cut the per-kernel launch cost that dominates small domains.
pm_status pm::iterate_n(pm_problem* pr, int n) {
  if (n <= 0) return PM_OK;
  // long runs go as it_eval-long chunks, whose graphs repeat
  const int chunk = std::max(kGraphMinSweeps, pr->prm.it_eval);
  while (n > chunk) {
    pm_status s = iterate_n(pr, chunk);
    if (s != PM_OK) return s;
    n -= chunk;
  }
  if (n < kGraphMinSweeps) return iterate_direct(pr, n);
  const int phase = pr->precision == PM_PREC_MIXED ? pr->iteration % pr->mixed_inner : 0;
  for (const auto& b : pr->graphs) {
    if (b.n == n && b.cur == pr->cur && b.ecur == pr->ecur && b.dc_pos == pr->dc_pos &&
        b.phase == phase && b.share == pr->share) {
      CK(cudaGraphLaunch(b.exec, pr->st));
      count_launches(b.launches);
      pr->cur = b.cur1;
      pr->ecur = b.ecur1;
      pr->dc_pos = b.dc_pos1;
      pr->iteration += n;
      pr->sweeps_done += n;
      return PM_OK;
    }
  }
  pm_problem::BlockGraph b;
  b.n = n; b.cur = pr->cur; b.ecur = pr->ecur; b.dc_pos = pr->dc_pos; b.phase = phase;
  b.share = pr->share;
  const unsigned long long l0 = launches_total();
  CK(cudaStreamBeginCapture(pr->st, cudaStreamCaptureModeThreadLocal));
  pm_status s = iterate_direct(pr, n);
  cudaGraph_t graph = nullptr;
  cudaError_t e = cudaStreamEndCapture(pr->st, &graph);
  if (s != PM_OK) {
    if (graph) cudaGraphDestroy(graph);
    return s;
  }
  if (e != cudaSuccess) return cuda_error(e, "sweep block capture");
  e = cudaGraphInstantiate(&b.exec, graph, 0);
  cudaGraphDestroy(graph);
  if (e != cudaSuccess) return cuda_error(e, "sweep block graph");
  b.launches = launches_total() - l0;  // counted once by the capture: this launch
  b.cur1 = pr->cur; b.ecur1 = pr->ecur; b.dc_pos1 = pr->dc_pos;
  CK(cudaGraphLaunch(b.exec, pr->st));
  if (pr->graphs.size() >= kGraphCache) {
    cudaGraphExecDestroy(pr->graphs.front().exec);
    pr->graphs.erase(pr->graphs.begin());
  }
  pr->graphs.push_back(b);
  return PM_OK;
}

namespace {

pm_status reduce_launch(pm_problem* pr, int full) {
  int mode = (pr->precision == PM_PREC_MIXED && pr->dc_pos > 0) ? 1 : 0;
  if (pr->order == PM_ORDER_REFERENCE) {
    CK(launch_reduce_serial(pr->F[pr->cur], full, pr->list, pr->nlist, pr->g,
                            pr->prm.dom_interest, pr->dout, pr->st));
    CK(cudaMemcpyAsync(pr->hout, pr->dout, sizeof(double) * kRedVals, cudaMemcpyDeviceToHost,
                       pr->st));
    return PM_OK;
  }
  const bool cpt = pr->compact();
  const float4* e = cpt ? pr->Ec[pr->ecur] : pr->E[pr->ecur];
  if (!full) {
    CK(launch_reduce_check(pr->F[pr->cur], e, mode, pr->list, pr->nlist, pr->g, pr->partials,
                           pr->dout, pr->st, cpt));
  } else {
    CK(launch_reduce(pr->F[pr->cur], e, mode, full, pr->order != PM_ORDER_REFERENCE, pr->codes,
                     pr->g, pr->prm.dom_interest, pr->partials, pr->dout, pr->st,
                     cpt ? pr->cwords : nullptr));
  }
  CK(cudaMemcpyAsync(pr->hout, pr->dout, sizeof(double) * kRedVals, cudaMemcpyDeviceToHost,
                     pr->st));
  return PM_OK;
}

}  // namespace

pm_status pm::reduce(pm_problem* pr, int full) {
  pm_status s = reduce_launch(pr, full);
  if (s != PM_OK) return s;
  return device_sync(pr, "reduce");
}

namespace {

// Initial state: fields as set up by allocate_initial_field + reapply.
pm_status reset_state(pm_problem* pr) {
  CK(launch_init64(pr->F[0], pr->codes, pr->g, pr->st));
  if (two_states(pr)) CK(launch_copy_fields64(pr->F[1], pr->F[0], pr->g, pr->st));
  if (pr->precision == PM_PREC_MIXED) {
    pm_status s = zero_corrections(pr);
    if (s != PM_OK) return s;
  }
  pr->cur = pr->ecur = pr->dc_pos = 0;
  pr->iteration = 0;
  pr->perm_prev = 0.0;
  pr->conv = 0.0;
  pr->conv_valid = false;
  pr->stop = pm::StopState{};
  pr->first_log = true;
  pr->device_ms = 0.0;
  pr->sweeps_done = 0;
  return device_sync(pr, "reset");
}

}  // namespace

// compute_convergence (evaluation.cc:216-262)
void pm::convergence_from(pm_problem* pr, double velz_sum, double* perm, double* conv) {
  int flcount = (int)(double)pr->counts.fluid;
  double sum = flcount == 0 ? 0.0 : velz_sum;
  double mean = sum / flcount;
  double cur = mean / kRe;
  *conv = fabs(cur - *perm) / cur;
  *perm = cur;
}

namespace {

// compute_permeability (evaluation.cc:54-211) from the device sums
void permeability_from(pm_problem* pr, const double* s, pm_result* r) {
  const int* di = pr->prm.dom_interest;
  bool dofi = di[0] | di[1] | di[2] | di[3] | di[4] | di[5];
  int wfl = (int)pr->counts.fluid;
  double wx = s[0], wy = s[1], wz = s[2], wmax = s[3];
  if (wfl == 0) { wx = wy = wz = 0.0; wmax = 0.0; }
  double phi = pr->phi, dx = pr->prm.voxel_size;
  if (dofi) {
    int fl = (int)pr->counts.box_fluid, p0f = (int)pr->counts.p0_fluid,
        pef = (int)pr->counts.pend_fluid;
    double vx = fl ? s[4] : 0.0, vy = fl ? s[5] : 0.0, vz = fl ? s[6] : 0.0;
    double p0 = p0f ? s[7] : 0.0, pe = pef ? s[8] : 0.0;
    double pgrad = ((pe / pef) - (p0 / p0f)) / (di[5] - di[4]);
    r->k13 = (vx / fl) * (1.0 / kRe) * phi * (1.0 / pgrad) * (dx * dx);
    r->k23 = (vy / fl) * (1.0 / kRe) * phi * (1.0 / pgrad) * (dx * dx);
    r->k33 = (vz / fl) * (1.0 / kRe) * phi * (1.0 / pgrad) * (dx * dx);
  } else {
    r->k13 = r->k23 = r->k33 = 0.0;
  }
  r->wk13 = (wx / wfl) * (1.0 / kRe) * phi * (dx * dx);
  r->wk23 = (wy / wfl) * (1.0 / kRe) * phi * (dx * dx);
  r->wk33 = (wz / wfl) * (1.0 / kRe) * phi * (dx * dx);
  r->wmean_velz = wz / wfl * dx;
  r->wmax_velz = wmax * dx;
  r->porosity = phi;
}

}  // namespace

namespace pm {

// write_logfile (output.cc:193-230): same header and "%i, %e, ..." row format.
pm_status write_log_row(const char* path, bool first, int iteration, double conv, double tps,
                        const pm_result& r) {
  FILE* f = fopen(path, "a");
  if (!f) return set_error(PM_ERR_IO, "cannot open log file %s", path);
  if (first)
    fprintf(f,
            "# iteration, conv, TPS [1/s], wmax_velz [m/s], wmean_velz [m/s], k13 [m^2], k23 "
            "[m^2], k33 [m^2], wk13 [m^2], wk23 [m^2], wk33 [m^2]\n");
  fprintf(f, "%i, %e, %e, %e, %e, %e, %e, %e, %e, %e, %e\n", iteration, conv, tps, r.wmax_velz,
          r.wmean_velz, r.k13, r.k23, r.k33, r.wk13, r.wk23, r.wk33);
  fclose(f);
  return PM_OK;
}

size_t problem_device_bytes(const pm_params* p) {
  Grid g = make_grid(p->size[0], p->size[1], p->size[2], p->boundary_method);
  size_t b = (size_t)g.allocc + 4 * (size_t)g.nvox + 2 * 4 * 8 * (size_t)g.alloc64;
  // the padded correction store, the compact one (fluid voxels <= voxels), or
  // both while the autotuner times kernels of either
  const bool cpt = p->kernel >= 8 && p->kernel <= 13;
  if (p->precision == PM_PREC_MIXED && !cpt) b += 3 * sizeof(float4) * (size_t)g.alloc4;
  if (p->precision == PM_PREC_MIXED && (cpt || p->kernel < 0))
    b += (3 * sizeof(float4) + sizeof(int4) + sizeof(int2) + sizeof(unsigned)) *
             ((size_t)g.nvox + 1) +
         sizeof(uint2) * (size_t)compact_words(g) + sizeof(int2) + 3 * sizeof(unsigned) +
         sizeof(int);
  if (p->precision == PM_PREC_MIXED && p->kernel == 13)
    b += sizeof(uint4) * ((size_t)g.nvox + 1);  // kernel 13's packed records
  b += 8 * (size_t)g.nvox;  // export scratch
  return b + (1 << 20);
}

}  // namespace pm

// ------------------------------------------------------------------ C ABI
extern "C" {

const char* pm_last_error(void) { return g_err.c_str(); }
size_t pm_last_error_copy(char* buf, size_t size) {
  const size_t n = g_err.size();
  if (buf && size > 0) {
    const size_t k = n < size - 1 ? n : size - 1;
    memcpy(buf, g_err.data(), k);
    buf[k] = '\0';
  }
  return n;
}
const char* pm_version(void) { return "poremaps_gb300 0.1 (sm_103a)"; }

pm_status pm_problem_footprint(const pm_params* p, size_t* bytes) {
  if (!bytes) return set_error(PM_ERR_INVALID, "bytes is NULL");
  pm_status s = validate(p);
  if (s != PM_OK) return s;
  *bytes = problem_device_bytes(p);
  return PM_OK;
}

pm_status pm_debug_tma_fail(int on) {
  zmarch_debug_fail(on);
  compact_debug_fail(on);
  wave_debug_fail(on);
  return PM_OK;
}

pm_status pm_debug_fail_alloc(int nth) {
  if (nth < 0) return set_error(PM_ERR_INVALID, "nth must be >= 0");
  g_fail_alloc.store(nth);
  return PM_OK;
}

pm_status pm_debug_launch_forms(int fp64_form, int record_variant) {
  if (fp64_form < -1 || fp64_form >= kForms64 || record_variant < -1 || record_variant > 2)
    return set_error(PM_ERR_INVALID, "forms: FP64 -1..%d, records -1..2", kForms64 - 1);
  g_force_form64.store(fp64_form);
  g_force_variant.store(record_variant);
  return PM_OK;
}

pm_status pm_params_default(pm_params* p) {
  if (!p) return set_error(PM_ERR_INVALID, "params is NULL");
  memset(p, 0, sizeof(*p));
  p->boundary_method = 0;
  p->voxel_size = 1e-5;
  p->max_iter = 100000001;
  p->it_eval = 100;
  p->it_write = 100;
  p->solving_algorithm = 2;
  p->eps = 1e-6;
  p->porosity = -1.0;
  p->order = PM_ORDER_DEFAULT;
  p->precision = PM_PREC_FP64;
  p->arith = PM_ARITH_FAST;
  p->write_log = 0;
  p->mixed_inner = 0;
  p->kernel = -1;
  return PM_OK;
}

pm_status pm_problem_create(const pm_params* p, const uint8_t* geom, pm_problem** out) {
  return problem_create(p, geom, -1, out);
}

}  // extern "C"

// pm_problem_create; rot_axis 0 / 1: geom is the unrotated volume of the
// tensor's x / y solve (sizes (nz', nx', ny') / (ny', nz', nx') for the
// problem's sizes (nx', ny', nz')), rotated on the device after the upload.
pm_status pm::problem_create(const pm_params* p, const uint8_t* geom, int rot_axis,
                             pm_problem** out) {
  if (!out) return set_error(PM_ERR_INVALID, "out is NULL");
  *out = nullptr;
  pm_status s = validate(p);
  if (s != PM_OK) return s;
  if (!geom) return set_error(PM_ERR_INVALID, "geometry is NULL");
  pm_problem* pr = new pm_problem();
  pr->prm = *p;
  pr->solver = (int)p->solving_algorithm;
  pr->order = p->order == PM_ORDER_DEFAULT ? PM_ORDER_REDBLACK : p->order;
  pr->precision = p->precision;
  if (pr->precision == PM_PREC_MIXED) pr->order = PM_ORDER_JACOBI;
  if (pr->order == PM_ORDER_REFERENCE) pr->precision = PM_PREC_FP64;
  pr->exact = p->arith == PM_ARITH_EXACT;
  pr->mixed_inner = p->mixed_inner > 0 ? p->mixed_inner : p->it_eval;
  pr->g = make_grid(p->size[0], p->size[1], p->size[2], p->boundary_method);
  const Grid& g = pr->g;
  auto fail = [&](pm_status st) {
    pm_problem_destroy(pr);
    return st;
  };
  size_t need = problem_device_bytes(p);
  size_t freeb = 0, totalb = 0;
  if (cudaMemGetInfo(&freeb, &totalb) != cudaSuccess)
    return fail(cuda_error(cudaGetLastError(), "cudaMemGetInfo"));
  freeb += pool_bytes();
  if (need > freeb)
    return fail(set_error(PM_ERR_NOMEM, "problem needs %zu bytes, %zu free", need, freeb));
  cudaError_t e;
#define CKF(expr)                                              \
  do {                                                         \
    if ((e = (expr)) != cudaSuccess) return fail(cuda_error(e, #expr)); \
  } while (0)
  CKF(cudaStreamCreateWithFlags(&pr->st, cudaStreamNonBlocking));
  sm_count();  // device query outside any later graph capture
  CKF(cudaEventCreate(&pr->ev0));
  CKF(cudaEventCreate(&pr->ev1));
  // the fixed buffers: codes, fluid list, the two FP64 states, reduction
  // partials and results, export scratch (one allocation)
  pr->scratch_bytes = 8 * (size_t)g.nvox;
  {
    Carve c;
    const size_t o_codes = c.take(g.allocc);
    const size_t o_list = c.take(sizeof(int) * (size_t)(g.nvox > 0 ? g.nvox : 1));
    const size_t o_f64[2] = {c.take(4 * sizeof(double) * (size_t)g.alloc64),
                             c.take(4 * sizeof(double) * (size_t)g.alloc64)};
    const size_t o_part = c.take(sizeof(double) * kRedBlocks * kRedVals + 64);
    const size_t o_dout = c.take(sizeof(double) * 16);
    const size_t o_scr = c.take(pr->scratch_bytes);
    const size_t o_werr = c.take(sizeof(int));
    CKF(dev_alloc((void**)&pr->arena, c.bytes));
    char* a = (char*)pr->arena;
    pr->codes_base = (uint8_t*)(a + o_codes);
    pr->list = (int*)(a + o_list);
    for (int b = 0; b < 2; ++b) pr->f64_base[b] = (double*)(a + o_f64[b]);
    pr->partials = (double*)(a + o_part);
    pr->dout = (double*)(a + o_dout);
    pr->scratch = a + o_scr;
    if (pr->order == PM_ORDER_REFERENCE) {
      pr->werr = (int*)(a + o_werr);
      CKF(cudaMemsetAsync(pr->werr, 0, sizeof(int), pr->st));
    }
  }
  pr->codes = pr->codes_base + kXoffC;
  CKF(cudaMemsetAsync(pr->codes_base, 0, g.allocc, pr->st));
  for (int b = 0; b < 2; ++b) {
    double* base = pr->f64_base[b];
    pr->F[b] = {base + kXoff64, base + g.alloc64 + kXoff64, base + 2 * g.alloc64 + kXoff64,
                base + 3 * g.alloc64 + kXoff64};
  }
  CKF(pinned_slot(&pr->hout));
  // geometry upload (through the export scratch, 8 bytes per voxel) -> codes
  // -> fluid list; a rotated solve rotates the upload into the scratch's
  // second voxel-sized part first
  const uint8_t* raw = (const uint8_t*)pr->scratch;
  CKF(cudaMemcpyAsync(pr->scratch, geom, (size_t)g.nvox, cudaMemcpyHostToDevice, pr->st));
  if (rot_axis == 0 || rot_axis == 1) {
    uint8_t* rot = (uint8_t*)pr->scratch + g.nvox;
    if (rot_axis == 0) CKF(launch_rotate_geom(raw, rot, 0, g.nz, g.nx, g.ny, pr->st));
    else CKF(launch_rotate_geom(raw, rot, 1, g.ny, g.nz, g.nx, pr->st));
    raw = rot;
  }
  CKF(launch_codes(raw, pr->codes, g, pr->st));
  int* dcount = (int*)pr->dout;
  CKF(launch_fluid_list(pr->codes, g, pr->list, dcount, pr->st));
  unsigned long long* dcnt = (unsigned long long*)((char*)pr->dout + 64);
  CKF(launch_counts(pr->codes, g, p->dom_interest, dcnt, pr->st));
  CKF(cudaMemcpyAsync(pr->hout, pr->dout, 96, cudaMemcpyDeviceToHost, pr->st));
  CKF(launch_init64(pr->F[0], pr->codes, g, pr->st));
  if (two_states(pr)) CKF(launch_copy_fields64(pr->F[1], pr->F[0], g, pr->st));
  CKF(cudaStreamSynchronize(pr->st));
  pr->nlist = *(int*)pr->hout;
  if (pr->order == PM_ORDER_REDBLACK) {
    // red voxels first, then black: each half-sweep walks only its own colour
    int* dc = (int*)pr->dout;
    CKF(launch_fluid_list(pr->codes, g, pr->list, dc, pr->st, 0, 0, 0, 0));
    CKF(cudaMemcpyAsync(pr->hout, pr->dout, sizeof(int), cudaMemcpyDeviceToHost, pr->st));
    CKF(cudaStreamSynchronize(pr->st));
    pr->nred = *(int*)pr->hout;
    CKF(launch_fluid_list(pr->codes, g, pr->list + pr->nred, dc, pr->st, 0, 0, 0, 1));
    CKF(cudaMemcpyAsync(pr->hout, pr->dout, sizeof(int), cudaMemcpyDeviceToHost, pr->st));
    CKF(cudaStreamSynchronize(pr->st));
    if (pr->nred + *(int*)pr->hout != pr->nlist)
      return fail(set_error(PM_ERR_CUDA, "red-black fluid lists do not add up"));
  }
  if (pr->precision == PM_PREC_MIXED) {
    // the correction store(s): only the one the kernel uses when it is known
    // (pinned, or tuned for a problem alike), both while the autotuner times
    // kernels of either
    const int kk = known_kernel(pr, p->kernel);
    const bool want_compact = kk < 0 || (kk >= 8 && kk <= 13);
    if (kk < 0 || !want_compact) {
      CKF(dev_alloc((void**)&pr->f32_base, 3 * sizeof(float4) * (size_t)g.alloc4));
      CKF(cudaMemsetAsync(pr->f32_base, 0, 3 * sizeof(float4) * (size_t)g.alloc4, pr->st));
      for (int k = 0; k < 3; ++k) {
        float4* f = pr->f32_base + k * g.alloc4 + kXoff4;
        if (k < 2) pr->E[k] = f;
        else pr->R = f;
      }
    }
    if (want_compact) {
      // e0, e1, r, slots, metadata, error flag, mask words (one allocation);
      // slots and metadata hold one and three entries more than positions,
      // which the bulk-staged sweep's copies (rounded up to 16 bytes) may read
      const size_t nl = (size_t)pr->nlist + 1;  // and the zero slot
      Carve c;
      const size_t o_e = c.take(3 * sizeof(float4) * nl);
      const size_t o_s4 = c.take(sizeof(int4) * nl);
      const size_t o_s2 = c.take(sizeof(int2) * (nl + 1));
      const size_t o_m = c.take(sizeof(unsigned) * (nl + 3));
      const size_t o_err = c.take(sizeof(int));
      const size_t o_w = c.take(sizeof(uint2) * (size_t)compact_words(g));
      CKF(dev_alloc((void**)&pr->carena, c.bytes));
      char* a = (char*)pr->carena;
      pr->c_base = (float4*)(a + o_e);
      pr->cslot4 = (int4*)(a + o_s4);
      pr->cslot2 = (int2*)(a + o_s2);
      pr->cmeta = (unsigned*)(a + o_m);
      pr->cerr = (int*)(a + o_err);
      pr->cwords = (uint2*)(a + o_w);
      // kernel 13's packed records, when pinned
      if (p->kernel == 13) CKF(dev_alloc((void**)&pr->crec_own, sizeof(uint4) * nl));
      CKF(cudaMemsetAsync(pr->c_base, 0, 3 * sizeof(float4) * nl, pr->st));
      CKF(cudaMemsetAsync(pr->cerr, 0, sizeof(int), pr->st));
      pr->Ec[0] = pr->c_base;
      pr->Ec[1] = pr->c_base + nl;
      pr->Rc = pr->c_base + 2 * nl;
    }
    pm_status ts = choose_correction_kernel(pr, p->kernel);
    if (ts != PM_OK) return fail(ts);
    if (const int forced = g_force_variant.load(); forced >= 0) pr->cvar = forced;
  }
  if (pr->precision == PM_PREC_FP64 && pr->order != PM_ORDER_REFERENCE) {
    pm_status ts = choose_fp64_shapes(pr);
    if (ts != PM_OK) return fail(ts);
  }
  unsigned long long* hc = (unsigned long long*)((char*)pr->hout + 64);
  pr->counts = {(long long)hc[0], (long long)hc[1], (long long)hc[2], (long long)hc[3]};
  // get_porosity (geometry.cc:335-364): fluid count / interior voxel count
  if (p->porosity == -1.0) {
    double vox = (double)((long long)g.nx * g.ny * g.nz);
    pr->phi = (double)pr->counts.fluid / vox;
  } else {
    pr->phi = p->porosity;
  }
#undef CKF
  *out = pr;
  return PM_OK;
}

extern "C" {

pm_status pm_problem_destroy(pm_problem* pr) {
  if (!pr) return PM_OK;
  if (pr->st) cudaStreamSynchronize(pr->st);
  for (auto& b : pr->graphs) cudaGraphExecDestroy(b.exec);
  zmarch_destroy(pr->zp);
  brick_destroy(pr->bp);
  dev_free(pr->arena);
  dev_free(pr->f32_base);
  dev_free(pr->carena);
  dev_free(pr->crec_own);
  pinned_release(pr->hout);
  if (pr->ev0) cudaEventDestroy(pr->ev0);
  if (pr->ev1) cudaEventDestroy(pr->ev1);
  if (pr->st) cudaStreamDestroy(pr->st);
  delete pr;
  return PM_OK;
}

pm_status pm_iterate(pm_problem* pr, int n) {
  if (!pr || n < 0) return set_error(PM_ERR_INVALID, "bad arguments");
  pm_status s = iterate_n(pr, n);
  if (s != PM_OK) return s;
  return device_sync(pr, "pm_iterate");
}

pm_status pm_compute_convergence(pm_problem* pr, double* permeability, double* conv) {
  if (!pr || !permeability || !conv) return set_error(PM_ERR_INVALID, "bad arguments");
  pm_status s = reduce(pr, 0);
  if (s != PM_OK) return s;
  convergence_from(pr, pr->hout[2], permeability, conv);
  return PM_OK;
}

pm_status pm_compute_permeability(pm_problem* pr, pm_result* res) {
  if (!pr || !res) return set_error(PM_ERR_INVALID, "bad arguments");
  pm_status s = reduce(pr, 1);
  if (s != PM_OK) return s;
  permeability_from(pr, pr->hout, res);
  return PM_OK;
}

pm_status pm_get_porosity(pm_problem* pr, double* porosity) {
  if (!pr || !porosity) return set_error(PM_ERR_INVALID, "bad arguments");
  *porosity = pr->phi;
  return PM_OK;
}

pm_status pm_get_iteration(pm_problem* pr, int* iteration) {
  if (!pr || !iteration) return set_error(PM_ERR_INVALID, "bad arguments");
  *iteration = pr->iteration;
  return PM_OK;
}

// calc_flow (calc_flow.cc:53-169)
pm_status pm_solve(pm_problem* pr, pm_result* res) {
  if (!pr || !res) return set_error(PM_ERR_INVALID, "bad arguments");
  auto t0 = std::chrono::steady_clock::now();
  const pm_params& p = pr->prm;
  memset(res, 0, sizeof(*res));
  double conv = pr->conv_valid ? pr->conv : 1.0 + p.eps;
  double perm = pr->perm_prev;
  pm_status s = PM_OK;
  float block_ms = 0.f;
  bool done = pr->conv_valid && stop_met(p, conv, pr->stop);
  while (pr->iteration < p.max_iter && !done) {
    // the next iteration at which the reference evaluates convergence
    long long it = pr->iteration;
    long long nxt = it;
    if (nxt <= 1000) nxt = 1001;
    nxt = ((nxt + p.it_eval - 1) / p.it_eval) * p.it_eval;
    long long last = nxt < p.max_iter ? nxt : (long long)p.max_iter - 1;
    int n = (int)(last - it + 1);
    const bool check = last == nxt;
    CK(cudaEventRecord(pr->ev0, pr->st));
    if ((s = iterate_n(pr, n)) != PM_OK) return s;
    CK(cudaEventRecord(pr->ev1, pr->st));
    // the convergence sums ride behind the block: one host synchronisation
    if (check && (s = reduce_launch(pr, 0)) != PM_OK) return s;
    if ((s = device_sync(pr, "sweep block")) != PM_OK) return s;
    CK(cudaEventElapsedTime(&block_ms, pr->ev0, pr->ev1));
    pr->device_ms += block_ms;
    if (check) {
      convergence_from(pr, pr->hout[2], &perm, &conv);
      stop_record(p, conv, pr->stop);
      done = stop_met(p, conv, pr->stop);
      res->iterations = (int)last;
      if (last % p.it_write == 0) {
        // the full permeability is only needed for a log row here; the
        // result's is computed once after the loop
        const bool log = p.write_log && p.log_file_name[0];
        if (log && (s = pm_compute_permeability(pr, res)) != PM_OK) return s;
        if (log) {
          double tps = block_ms > 0 ? 1000.0 * n / block_ms : 0.0;
          if ((s = write_log_row(p.log_file_name, pr->first_log, (int)last, conv, tps, *res)) !=
              PM_OK)
            return s;
        }
        pr->first_log = false;
      }
    }
  }
  pr->conv = conv;
  pr->conv_valid = true;
  pr->perm_prev = perm;
  pm_result keep = *res;
  if ((s = pm_compute_permeability(pr, res)) != PM_OK) return s;
  res->iterations = keep.iterations;
  res->sweeps = (int)pr->sweeps_done;
  res->conv = conv;
  res->converged = pr->conv_valid && stop_converged(p, conv, pr->stop);
  res->permeability = perm;
  res->device_ms = pr->device_ms;
  res->wall_ms =
      std::chrono::duration<double, std::milli>(std::chrono::steady_clock::now() - t0).count();
  res->glups = pr->device_ms > 0 ? (double)pr->g.nvox * pr->sweeps_done / (pr->device_ms * 1e6)
                                 : 0.0;
  if (!isfinite(res->wk33) || !isfinite(perm))
    return set_error(PM_ERR_NONFINITE, "non-finite permeability (conv=%g)", conv);
  return PM_OK;
}

pm_status pm_set_device(int device) {
  CK(cudaSetDevice(device));
  return PM_OK;
}

pm_status pm_release_memory(void) {
  pool_release();
  return PM_OK;
}

pm_status pm_problem_reset(pm_problem* pr) {
  if (!pr) return set_error(PM_ERR_INVALID, "bad arguments");
  return reset_state(pr);
}

pm_status pm_block_timed(pm_problem* pr, int n, int check, double* permeability, double* conv,
                         double* device_ms) {
  if (!pr || n < 0) return set_error(PM_ERR_INVALID, "bad arguments");
  pm_status s;
  CK(cudaEventRecord(pr->ev0, pr->st));
  if ((s = iterate_n(pr, n)) != PM_OK) return s;
  if (check && (s = reduce_launch(pr, 0)) != PM_OK) return s;
  CK(cudaEventRecord(pr->ev1, pr->st));
  if ((s = device_sync(pr, "pm_block_timed")) != PM_OK) return s;
  float ms = 0.f;
  CK(cudaEventElapsedTime(&ms, pr->ev0, pr->ev1));
  pr->device_ms += ms;
  if (device_ms) *device_ms = ms;
  if (check && permeability && conv) convergence_from(pr, pr->hout[2], permeability, conv);
  return PM_OK;
}

pm_status pm_block_group_timed(pm_problem** prs, int count, int n, int check,
                               double* permeability, double* conv, double* device_ms) {
  if (!prs || count <= 0 || n < 0) return set_error(PM_ERR_INVALID, "bad arguments");
  for (int i = 0; i < count; ++i)
    if (!prs[i]) return set_error(PM_ERR_INVALID, "bad arguments");
  pm_problem* lead = prs[0];
  // the sweeps of the group share the device until it is joined
  struct Share {
    pm_problem** prs;
    int count;
    Share(pm_problem** p, int n) : prs(p), count(n) { set(n); }
    ~Share() { set(1); }
    void set(int n) {
      for (int i = 0; i < count; ++i) prs[i]->share = n;
    }
  } share(prs, count);
  // fork: every stream starts after the start event on the first stream
  CK(cudaEventRecord(lead->ev0, lead->st));
  for (int i = 1; i < count; ++i) CK(cudaStreamWaitEvent(prs[i]->st, lead->ev0, 0));
  pm_status s;
  for (int i = 0; i < count; ++i) {
    if ((s = iterate_n(prs[i], n)) != PM_OK) return s;
    if (check && (s = reduce_launch(prs[i], 0)) != PM_OK) return s;
  }
  // join: the end event on the first stream follows every stream's block
  for (int i = 1; i < count; ++i) {
    CK(cudaEventRecord(prs[i]->ev1, prs[i]->st));
    CK(cudaStreamWaitEvent(lead->st, prs[i]->ev1, 0));
  }
  CK(cudaEventRecord(lead->ev1, lead->st));
  for (int i = count - 1; i >= 0; --i)
    if ((s = device_sync(prs[i], "pm_block_group_timed")) != PM_OK) return s;
  float ms = 0.f;
  CK(cudaEventElapsedTime(&ms, lead->ev0, lead->ev1));
  if (device_ms) *device_ms = ms;
  for (int i = 0; i < count; ++i) {
    prs[i]->device_ms += ms;
    if (check && permeability && conv)
      convergence_from(prs[i], prs[i]->hout[2], &permeability[i], &conv[i]);
  }
  return PM_OK;
}

pm_status pm_kernel_time(pm_problem* pr, int kernel, int n, double* avg_ms) {
  if (!pr || n <= 0 || !avg_ms) return set_error(PM_ERR_INVALID, "bad arguments");
  if (pr->order == PM_ORDER_REFERENCE)
    return set_error(PM_ERR_INVALID, "kernel timing is for the out-of-place forms");
  // Repeated launches read the current state and write the scratch buffer
  // (identical result every time), so the state is unchanged afterwards.
  CK(cudaEventRecord(pr->ev0, pr->st));
  for (int i = 0; i < n; ++i) {
    if (pr->precision == PM_PREC_MIXED) {
      if (kernel == 1) {
        if (pr->dc_pos != 0) return set_error(PM_ERR_INVALID, "residual timing needs dc_pos 0");
        if (pr->compact())
          CK(launch_dc_residual_c(pr->F[pr->cur], pr->Rc, pr->Ec[pr->ecur], pr->codes, pr->list,
                                  pr->nlist, pr->g, pr->solver, pr->st));
        else
          CK(launch_dc_residual(pr->F[pr->cur], pr->R, pr->E[pr->ecur], pr->codes, pr->list,
                                pr->nlist, pr->g, pr->solver, pr->st));
      } else {
        pm_status s = correction_sweep(pr, pr->ecur);
        if (s != PM_OK) return s;
      }
    } else {
      pm_status s = sweeps64(pr, pr->F[pr->cur], pr->F[1 - pr->cur]);
      if (s != PM_OK) return s;
    }
  }
  CK(cudaEventRecord(pr->ev1, pr->st));
  pm_status s;
  if ((s = device_sync(pr, "pm_kernel_time")) != PM_OK) return s;
  float ms = 0.f;
  CK(cudaEventElapsedTime(&ms, pr->ev0, pr->ev1));
  *avg_ms = ms / n;
  return PM_OK;
}

uint64_t pm_kernel_launches(void) { return (uint64_t)launches_total(); }

pm_status pm_get_kernel(pm_problem* pr, int* kernel) {
  if (!pr || !kernel) return set_error(PM_ERR_INVALID, "bad arguments");
  *kernel = pr->kern;
  return PM_OK;
}

pm_status pm_get_brick(pm_problem* pr, int brick[3]) {
  if (!pr || !brick) return set_error(PM_ERR_INVALID, "bad arguments");
  for (int i = 0; i < 3; ++i) brick[i] = pr->brick[i];
  return PM_OK;
}

pm_status pm_get_fields(pm_problem* pr, double* u, double* v, double* w, double* p) {
  if (!pr) return set_error(PM_ERR_INVALID, "bad arguments");
  pm_status s;
  if ((s = dc_flush(pr)) != PM_OK) return s;
  double* out[4] = {u, v, w, p};
  const Fields<double>& f = pr->F[pr->cur];
  const double* src[4] = {f.u, f.v, f.w, f.p};
  for (int k = 0; k < 4; ++k) {
    if (!out[k]) continue;
    CK(launch_pack64(src[k], pr->codes, k == 3 && pr->order != PM_ORDER_REFERENCE, pr->g,
                     (double*)pr->scratch, pr->st));
    CK(cudaMemcpyAsync(out[k], pr->scratch, sizeof(double) * pr->g.nvox, cudaMemcpyDeviceToHost,
                       pr->st));
    if ((s = device_sync(pr, "pm_get_fields")) != PM_OK) return s;
  }
  return PM_OK;
}

pm_status pm_set_fields(pm_problem* pr, const double* u, const double* v, const double* w,
                        const double* p, int iteration) {
  if (!pr || !u || !v || !w || !p || iteration < 0)
    return set_error(PM_ERR_INVALID, "bad arguments");
  pm_status s;
  if ((s = reset_state(pr)) != PM_OK) return s;
  // The state is a function of the interior: periodic halos are copies and
  // the pressure planes are reapplied.  The pre-reapply pressure of the last
  // interior plane is not in the dumps; the reapplied value stands in for it.
  const Fields<double>& f = pr->F[0];
  double* dst[4] = {f.u, f.v, f.w, f.p};
  const double* src[4] = {u, v, w, p};
  for (int k = 0; k < 4; ++k) {
    CK(cudaMemcpyAsync(pr->scratch, src[k], sizeof(double) * pr->g.nvox, cudaMemcpyHostToDevice,
                       pr->st));
    CK(launch_unpack64((const double*)pr->scratch, pr->g, dst[k], pr->st));
    // the staging buffer is reused: finish this field before the next copy
    if ((s = device_sync(pr, "pm_set_fields")) != PM_OK) return s;
  }
  CK(launch_halo64(f, pr->g, pr->st));
  CK(launch_reapply64(f.p, pr->codes, pr->g, pr->st));
  if (two_states(pr)) CK(launch_copy_fields64(pr->F[1], pr->F[0], pr->g, pr->st));
  pr->iteration = iteration;
  return device_sync(pr, "pm_set_fields");
}

pm_status pm_get_neighborhood(pm_problem* pr, int32_t* out) {
  if (!pr || !out) return set_error(PM_ERR_INVALID, "bad arguments");
  CK(launch_pack_codes(pr->codes, pr->g, (int*)pr->scratch, pr->st));
  CK(cudaMemcpyAsync(out, pr->scratch, sizeof(int32_t) * pr->g.nvox, cudaMemcpyDeviceToHost,
                     pr->st));
  return device_sync(pr, "pm_get_neighborhood");
}

}  // extern "C"

namespace pm {
const pm_params* problem_params(const pm_problem* pr) { return &pr->prm; }
long long problem_nvox(const pm_problem* pr) { return pr->g.nvox; }
cudaStream_t problem_stream(const pm_problem* pr) { return pr->st; }
}  // namespace pm
