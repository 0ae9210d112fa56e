// A stand-in for the CUDA runtime and the kernel launchers, so that the host
// runtime (pm_api.cpp, pm_server.cpp) runs on a machine without a GPU.  Device
// memory is host memory of a limited size per device, launches only note their
// name, and the order in which work reaches a stream is checked:
//   * set-up data that overlapped launches read before their wait (packed
//     records, fluid lists) has to be followed by a synchronisation or a plain
//     launch before such a launch ("unordered <launcher>" otherwise);
//   * a launcher's buffers must exist ("null <launcher>").
// Values are not computed: sums read back are zero, event times are the sums of
// the costs given to the launchers in between.
#include <string.h>
#include <sys/mman.h>

#include <map>
#include <set>
#include <string>
#include <vector>

#include "../poremaps_gb300/csrc/pm_api_internal.h"
#include "../poremaps_gb300/csrc/pm_batch.h"
#include "../poremaps_gb300/csrc/pm_compact.h"

namespace {

struct Block {
  size_t bytes;
  int dev;
};
struct Stream {
  int pending = 0;         // launches since the last synchronisation
  bool unordered = false;  // set-up data no plain launch or synchronisation follows yet
  double clock = 0.0;
};
struct Event {
  double clock = 0.0;
};

constexpr size_t kSmall = 1 << 20;  // copies and fills above this are left out

std::string g_trace;
std::map<void*, Block> g_blocks;
std::set<Stream*> g_streams;
std::map<std::string, double> g_cost;
size_t g_total[2] = {64ull << 30, 64ull << 30}, g_used[2] = {0, 0};
bool g_split = false;  // no block above half of a device's memory can be had
int g_dev = 0, g_fluid = 0, g_fail_launch = 0;
cudaError_t g_last = cudaSuccess;  // what cudaGetLastError returns, once
bool g_capture = false;

Stream* S(cudaStream_t st) { return (Stream*)st; }

void note(const std::string& s) { g_trace += s + "\n"; }

void settle(Stream* s) {
  s->pending = 0;
  s->unordered = false;
}

enum { kPlain = 0, kOverlapped = 1 };

cudaError_t launch(const char* name, cudaStream_t st, int how,
                   std::initializer_list<const void*> buffers) {
  if (g_fail_launch > 0 && --g_fail_launch == 0) return cudaErrorLaunchOutOfResources;
  // the launchers report cudaGetLastError
  if (const cudaError_t e = cudaGetLastError(); e != cudaSuccess) return e;
  note(name);
  for (const void* b : buffers)
    if (!b) note(std::string("null ") + name);
  if (how == kOverlapped && S(st)->unordered) note(std::string("unordered ") + name);
  if (how == kPlain) S(st)->unordered = false;
  if (!g_capture) S(st)->pending++;
  S(st)->clock += g_cost.count(name) ? g_cost[name] : 1.0;
  return cudaSuccess;
}

cudaError_t device_alloc(void** p, size_t n) {
  *p = nullptr;
  if (g_used[g_dev] + n > g_total[g_dev] || (g_split && n > g_total[g_dev] / 2)) {
    note("out of memory");
    return g_last = cudaErrorMemoryAllocation;
  }
  void* m = mmap(nullptr, n, PROT_READ | PROT_WRITE, MAP_PRIVATE | MAP_ANONYMOUS | MAP_NORESERVE,
                 -1, 0);
  if (m == MAP_FAILED) return cudaErrorMemoryAllocation;
  g_blocks[m] = {n, g_dev};
  g_used[g_dev] += n;
  *p = m;
  return cudaSuccess;
}

}  // namespace

extern "C" {

// ---- what the tests set and read
const char* fake_trace() { return g_trace.c_str(); }
void fake_reset_trace() { g_trace.clear(); }
void fake_set_fluid(int n) { g_fluid = n; }
void fake_set_cost(const char* name, double ms) { g_cost[name] = ms; }
void fake_set_memory(int dev, size_t bytes) { g_total[dev] = bytes; }
void fake_split_memory(int on) { g_split = on != 0; }
size_t fake_used(int dev) { return g_used[dev]; }
void fake_fail_launch(int nth) { g_fail_launch = nth; }
int fake_pending() {
  int n = 0;
  for (auto* s : g_streams) n += s->pending;
  return n;
}

// ---- CUDA runtime
cudaError_t cudaMalloc(void** p, size_t n) { return device_alloc(p, n); }
cudaError_t cudaMallocAsync(void** p, size_t n, cudaStream_t) { return device_alloc(p, n); }
cudaError_t cudaFree(void* p) {  // waits for the device, as the real one
  if (!p) return cudaSuccess;
  for (auto* s : g_streams) settle(s);
  auto it = g_blocks.find(p);
  if (it == g_blocks.end()) return cudaErrorInvalidValue;
  g_used[it->second.dev] -= it->second.bytes;
  munmap(p, it->second.bytes);
  g_blocks.erase(it);
  return cudaSuccess;
}
cudaError_t cudaMallocHost(void** p, size_t n) {
  *p = calloc(1, n);
  return cudaSuccess;
}
cudaError_t cudaFreeHost(void* p) {
  free(p);
  return cudaSuccess;
}
cudaError_t cudaMemGetInfo(size_t* fr, size_t* tot) {
  *tot = g_total[g_dev];
  *fr = g_total[g_dev] > g_used[g_dev] ? g_total[g_dev] - g_used[g_dev] : 0;
  return cudaSuccess;
}
cudaError_t cudaGetDevice(int* d) {
  *d = g_dev;
  return cudaSuccess;
}
cudaError_t cudaSetDevice(int d) {
  g_dev = d;
  return cudaSuccess;
}
cudaError_t cudaGetLastError() {
  const cudaError_t e = g_last;
  g_last = cudaSuccess;
  return e;
}
const char* cudaGetErrorString(cudaError_t e) {
  return e == cudaErrorMemoryAllocation ? "out of memory" : "error";
}
cudaError_t cudaMemcpyAsync(void* d, const void* s, size_t n, cudaMemcpyKind, cudaStream_t) {
  if (n <= kSmall && n > 0) memcpy(d, s, n);
  return cudaSuccess;
}
cudaError_t cudaMemcpy(void* d, const void* s, size_t n, cudaMemcpyKind k) {
  return cudaMemcpyAsync(d, s, n, k, nullptr);
}
cudaError_t cudaMemset(void* p, int v, size_t n) {
  if (n <= kSmall) memset(p, v, n);
  return cudaSuccess;
}
cudaError_t cudaMemsetAsync(void* p, int v, size_t n, cudaStream_t) { return cudaMemset(p, v, n); }
cudaError_t cudaStreamCreateWithFlags(cudaStream_t* st, unsigned) {
  Stream* s = new Stream();
  g_streams.insert(s);
  *st = (cudaStream_t)s;
  return cudaSuccess;
}
cudaError_t cudaStreamDestroy(cudaStream_t st) {
  g_streams.erase(S(st));
  delete S(st);
  return cudaSuccess;
}
cudaError_t cudaStreamSynchronize(cudaStream_t st) {
  settle(S(st));
  return cudaSuccess;
}
cudaError_t cudaStreamWaitEvent(cudaStream_t, cudaEvent_t, unsigned) { return cudaSuccess; }
cudaError_t cudaStreamBeginCapture(cudaStream_t, cudaStreamCaptureMode) {
  g_capture = true;
  return cudaSuccess;
}
cudaError_t cudaStreamEndCapture(cudaStream_t, cudaGraph_t* g) {
  g_capture = false;
  *g = (cudaGraph_t) new int(0);
  return cudaSuccess;
}
cudaError_t cudaGraphInstantiate(cudaGraphExec_t* x, cudaGraph_t, unsigned long long) {
  *x = (cudaGraphExec_t) new int(0);
  return cudaSuccess;
}
cudaError_t cudaGraphDestroy(cudaGraph_t g) {
  delete (int*)g;
  return cudaSuccess;
}
cudaError_t cudaGraphExecDestroy(cudaGraphExec_t x) {
  delete (int*)x;
  return cudaSuccess;
}
cudaError_t cudaGraphLaunch(cudaGraphExec_t, cudaStream_t st) {
  S(st)->pending++;
  return cudaSuccess;
}
cudaError_t cudaEventCreate(cudaEvent_t* e) {
  *e = (cudaEvent_t) new Event();
  return cudaSuccess;
}
cudaError_t cudaEventDestroy(cudaEvent_t e) {
  delete (Event*)e;
  return cudaSuccess;
}
cudaError_t cudaEventRecord(cudaEvent_t e, cudaStream_t st) {
  ((Event*)e)->clock = S(st)->clock;
  return cudaSuccess;
}
cudaError_t cudaEventSynchronize(cudaEvent_t) { return cudaSuccess; }
cudaError_t cudaEventElapsedTime(float* ms, cudaEvent_t a, cudaEvent_t b) {
  *ms = (float)(((Event*)b)->clock - ((Event*)a)->clock);
  return cudaSuccess;
}

}  // extern "C"

// ---- kernel launchers
namespace pm {

void count_launches(int) {}
unsigned long long launches_total() { return 0; }
int sm_count() { return 152; }

Grid make_grid(int nx, int ny, int nz, int) {
  Grid g;
  memset(&g, 0, sizeof g);
  g.nx = nx; g.ny = ny; g.nz = nz;
  g.NX = nx + 4; g.NY = ny + 4; g.NZ = nz + 4;
  g.nvox = (long long)nx * ny * nz;
  g.alloc64 = g.alloc32 = g.allocc = g.alloc4 = (long long)g.NX * g.NY * g.NZ + 64;
  return g;
}

cudaError_t launch_codes(const uint8_t*, uint8_t* c, const Grid&, cudaStream_t st) {
  return launch("codes", st, kPlain, {c});
}
cudaError_t launch_rotate_geom(const uint8_t*, uint8_t* d, int, int, int, int, cudaStream_t st) {
  return launch("rotate_geom", st, kPlain, {d});
}
cudaError_t launch_fluid_list(const uint8_t*, const Grid&, int* list, int* count, cudaStream_t st,
                              int, int, int, int parity) {
  const cudaError_t e = launch("fluid_list", st, kPlain, {list, count});
  S(st)->unordered = true;
  *count = parity < 0 ? g_fluid : parity == 0 ? g_fluid / 2 : g_fluid - g_fluid / 2;
  return e;
}
cudaError_t launch_counts(const uint8_t*, const Grid&, const int*, unsigned long long* out,
                          cudaStream_t st) {
  memset(out, 0, 4 * sizeof *out);
  out[0] = (unsigned long long)g_fluid;
  return launch("counts", st, kPlain, {out});
}
cudaError_t launch_init64(Fields<double> f, const uint8_t*, const Grid&, cudaStream_t st) {
  return launch("init64", st, kPlain, {f.u});
}
cudaError_t launch_copy_fields64(Fields<double> d, Fields<double>, const Grid&, cudaStream_t st) {
  return launch("copy_fields64", st, kPlain, {d.u});
}
cudaError_t launch_halo64(Fields<double> f, const Grid&, cudaStream_t st) {
  return launch("halo64", st, kPlain, {f.u});
}
cudaError_t launch_reapply64(double* p, const uint8_t*, const Grid&, cudaStream_t st) {
  return launch("reapply64", st, kPlain, {p});
}
cudaError_t launch_wave(Fields<double> f, const uint8_t*, const Grid&, int, double* x, int* err,
                        cudaStream_t st) {
  return launch("wave", st, kPlain, {f.u, x, err});
}
void wave_debug_fail(int) {}
cudaError_t launch_sweep64(Fields<double> A, Fields<double> B, const uint8_t*, const int* list,
                           int, const Grid&, int, int exact, int, cudaStream_t st, int form) {
  const std::string cost = "sweep64 form " + std::to_string(form);
  note(cost);
  g_cost["sweep64"] = g_cost.count(cost) ? g_cost[cost] : 1.0;
  const bool plain = exact || form == kForm64One || form == kForm64Whole;
  return launch("sweep64", st, plain ? kPlain : kOverlapped, {A.u, B.u, list});
}
cudaError_t launch_dc_correct_list(Fields<double> x, const float4* e, const int* list, int,
                                   const Grid&, cudaStream_t st) {
  return launch("dc_correct_list", st, kPlain, {x.u, e, list});
}
cudaError_t launch_dc_residual(Fields<double> x, float4* r, float4* e, const uint8_t*, const int*,
                               int, const Grid&, int, cudaStream_t st) {
  return launch("dc_residual", st, kPlain, {x.u, r, e});
}
cudaError_t launch_dc_inner(const float4* e, float4* e2, const float4* r, const uint8_t*,
                            const int*, int, const Grid&, int, cudaStream_t st) {
  return launch("dc_inner", st, kPlain, {e, e2, r});
}
cudaError_t launch_dc_inner_pf(const float4* e, float4* e2, const float4* r, const uint8_t*,
                               const int*, int, const Grid&, int, int, cudaStream_t st) {
  return launch("dc_inner_pf", st, kPlain, {e, e2, r});
}
cudaError_t launch_dc_inner_occ(const float4* e, float4* e2, const float4* r, const uint8_t*,
                                const int*, int, const Grid&, int, cudaStream_t st) {
  return launch("dc_inner_occ", st, kPlain, {e, e2, r});
}
cudaError_t launch_zero4(float4* e, const Grid&, cudaStream_t st) {
  return launch("zero4", st, kPlain, {e});
}
cudaError_t launch_reduce_check(Fields<double> x, const float4*, int, const int*, int, const Grid&,
                                double*, double* out, cudaStream_t st, int) {
  return launch("reduce_check", st, kPlain, {x.u, out});
}
cudaError_t launch_reduce(Fields<double> x, const float4*, int, int, int, const uint8_t*,
                          const Grid&, const int*, double*, double* out, cudaStream_t st,
                          const uint2*) {
  return launch("reduce", st, kPlain, {x.u, out});
}
cudaError_t launch_reduce_serial(Fields<double> x, int, const int* list, int, const Grid&,
                                 const int*, double* out, cudaStream_t st) {
  return launch("reduce_serial", st, kPlain, {x.u, list, out});
}
cudaError_t launch_pack64(const double* f, const uint8_t*, int, const Grid&, double* out,
                          cudaStream_t st) {
  return launch("pack64", st, kPlain, {f, out});
}
cudaError_t launch_unpack64(const double* in, const Grid&, double* f, cudaStream_t st) {
  return launch("unpack64", st, kPlain, {in, f});
}
cudaError_t launch_pack_codes(const uint8_t*, const Grid&, int* out, cudaStream_t st) {
  return launch("pack_codes", st, kPlain, {out});
}

long long compact_words(const Grid& g) { return (long long)((g.nx + 31) / 32) * g.ny * g.nz + 1; }
bool compact_records_fit(const Grid& g, int nlist) {
  return g.nx < (1 << 13) && nlist < (1 << 27) - 1;
}
cudaError_t compact_setup(const uint8_t*, const Grid&, const int*, int, uint2* w, int4* sa,
                          int2* sb, unsigned* m, cudaStream_t st) {
  return launch("compact_setup", st, kPlain, {w, sa, sb, m});
}
cudaError_t compact_records(const unsigned* m, const int4* sa, const int2* sb, int, uint4* rec,
                            int2* ya, cudaStream_t st) {
  const cudaError_t e = launch("compact_records", st, kPlain, {m, sa, sb, rec, ya});
  S(st)->unordered = true;
  return e;
}
cudaError_t launch_dc_inner_cr(const float4* e, float4* e2, const float4* r, const uint4* rec,
                               const int2* ya, int, int, int, cudaStream_t st) {
  return launch("dc_inner_cr", st, kOverlapped, {e, e2, r, rec, ya});
}
cudaError_t launch_dc_inner_c(const float4* e, float4* e2, const float4* r, const unsigned* m,
                              const int4* sa, const int2* sb, int, int, int, cudaStream_t st) {
  return launch("dc_inner_c", st, kPlain, {e, e2, r, m, sa, sb});
}
cudaError_t launch_dc_inner_cb(const float4* e, float4* e2, const float4* r, const unsigned* m,
                               const int4* sa, const int2* sb, int, int, int, int* err,
                               cudaStream_t st) {
  return launch("dc_inner_cb", st, kPlain, {e, e2, r, m, sa, sb, err});
}
void compact_debug_fail(int) {}
cudaError_t launch_dc_residual_c(Fields<double> x, float4* r, float4* e, const uint8_t*,
                                 const int*, int, const Grid&, int, cudaStream_t st) {
  return launch("dc_residual_c", st, kPlain, {x.u, r, e});
}
cudaError_t launch_dc_correct_c(Fields<double> x, const float4* e, const int*, int, const Grid&,
                                cudaStream_t st) {
  return launch("dc_correct_c", st, kPlain, {x.u, e});
}

cudaError_t launch_batch(int, const SampleDesc* d, const WorkItem* items, int, int, int, int,
                         double*, cudaStream_t st, int) {
  return launch("batch", st, kPlain, {d, items});
}
cudaError_t launch_batch_flat(const FlatSample* s, const int2* items, int, int, int,
                              cudaStream_t st) {
  return launch("batch_flat", st, kOverlapped, {s, items});
}
cudaError_t launch_batch_round(const SampleDesc* d, const WorkItem* items, int, int, int,
                               unsigned* sync, cudaStream_t st, int, unsigned, int, int, int) {
  return launch("batch_round", st, kPlain, {d, items, sync});
}

// the TMA kernels are not offered here (kernel 1 then stands in for them)
struct ZmarchPlan {};
int zmarch_available() { return 0; }
cudaError_t zmarch_create(ZmarchPlan**, const Grid&, float4*, float4*, float4*, const uint8_t*,
                          int, int) {
  return cudaErrorNotSupported;
}
void zmarch_destroy(ZmarchPlan*) {}
cudaError_t zmarch_inner(const ZmarchPlan*, int, float4*, const Grid&, int, cudaStream_t) {
  return cudaErrorNotSupported;
}
int* zmarch_error_flag(const ZmarchPlan*) { return nullptr; }
void zmarch_debug_fail(int) {}
struct BrickPlan {};
int brick_shape_of(int, int, int) { return 0; }
cudaError_t brick_create(BrickPlan**, const Grid&, float4*, float4*, const uint8_t*, const int*,
                         int, int, cudaStream_t) {
  return cudaErrorNotSupported;
}
void brick_destroy(BrickPlan*) {}
cudaError_t brick_inner(const BrickPlan*, int, float4*, const float4*, const int*, const Grid&,
                        int, cudaStream_t) {
  return cudaErrorNotSupported;
}
int* brick_error_flag(const BrickPlan*) { return nullptr; }

}  // namespace pm
