// Device memory, streams, graphs and the kernel launchers as host code, so that the host side of the library
// (ct_api.cu, compiled as C++) runs without a GPU. "Device" memory is host memory whose blocks are
// known by address and size; a launch does no work but checks that what it was given is there: every
// pointer lies in a live block with room for what the kernel would touch, and the exchange ring is long enough
// for the delays that it would meet. A captured launch is checked when its graph runs. What was found
// wrong is kept as text (host_device_report). Allocations can be made to fail by size, elapsed times
// can be scripted.
#include <cuda_runtime.h>
#include <dlfcn.h>
#include <pthread.h>

#include <algorithm>
#include <cerrno>
#include <cstdlib>
#include <cstring>
#include <map>
#include <mutex>
#include <new>
#include <set>
#include <string>
#include <utility>
#include <vector>

#include "../../cardiotrust_b200/csrc/ct_internal.cuh"

namespace {

constexpr int kCapacity = 4;  // co-resident CTAs of the recursion kernel
constexpr size_t kRecordBytes = 64;

struct Recorded {
  ct::WaveLaunch launch;
  bool adjoint;
  int grid;
};
// A gradient sweep, and whether its kernel takes blocks without a ring.
struct Sweep {
  const ct::DeviceScenario* d;
  bool any;
};
struct Graph {
  std::vector<Sweep> sweeps;
  std::vector<Recorded> launches;
  std::vector<std::pair<const ct::DeviceScenario*, const void*>> ranges;  // delay ranges, and the reverse table they covered
};

std::map<char*, size_t> g_blocks;
size_t g_live = 0;
size_t g_fail_from = ~size_t(0);      // device allocations of at least so many bytes fail
size_t g_host_fail_from = ~size_t(0) / 2;  // the library's host allocations of this size up to twice as much fail
bool g_no_threads = false;            // no thread can be started (with this library preloaded)
cudaError_t g_last = cudaSuccess;     // of this runtime, until it is asked for
std::string g_report;
Graph* g_capturing = nullptr;
std::vector<float> g_times;
size_t g_time = 0;
std::vector<int> g_orders;  // phases of every batched forward that ran
int g_landed = 0;  // what was recorded on a stream has happened: never, always, or once the stream was waited for
bool g_waited = false;
int g_captures = 0;     // epochs captured since the last count
int g_sweep_blocks = 0;     // of the last sweep
bool g_last_sweep = false;  // whether the last sweep takes blocks without a ring
int g_last_routes = 0;      // ct::WaveRoutes of the last forward
int g_routes[2][3];         // tiles of the last forward and adjoint: followed by progress, by tags, polled directly

void wrong(const std::string& what) {
  if (g_report.size() < 4000) g_report += what + "\n";
}

bool live(const void* p, size_t bytes) {
  auto it = g_blocks.upper_bound((char*)p);
  if (!p || it == g_blocks.begin()) return false;
  --it;
  return (char*)p + bytes <= it->first + it->second;
}
void need(const void* p, size_t bytes, const char* what) {
  if (!live(p, bytes)) wrong(std::string(what) + " is not in a live block");
}

// The rows that readers may still want: every step, or twice the largest delay and two. And a kernel that takes the delays
// and halos that it meets.
void check_ring(const ct::WaveScn& p, int routes, const char* form) {
  need(p.xch, sizeof(uint4) * ((size_t)p.xrows * p.V + 8 * (size_t)p.ntiles), form);
  if (!live(p.src, sizeof(int32_t) * p.V * ct::kOffsets) || !live(p.delays, sizeof(int32_t) * p.V * ct::kOffsets)) {
    wrong(std::string(form) + ": tables are not in a live block");
    return;
  }
  int64_t dmin = INT32_MAX, dmax = 1;
  for (int64_t i = 0; i < (int64_t)p.V * ct::kOffsets; ++i)
    if (p.src[i] >= 0) {
      const int64_t delay = p.delays[p.rows ? p.src[i] * ct::kOffsets + i % ct::kOffsets : i];
      dmin = std::min(dmin, delay);
      dmax = std::max(dmax, delay);
    }
  if (routes == ct::kStaged && dmax - dmin > ct::kFwdRingSpread) wrong(std::string(form) + ": delays too far apart for the staged ring");
  for (int t = 0; t < p.ntiles; ++t)
    if (routes != ct::kEvery && p.nhalo[t] < 0) wrong(std::string(form) + ": a halo too large for the staged ring");
  if (p.xrows >= p.T) return;
  if (p.xrows < 2 * dmax + 2) wrong(std::string(form) + ": the exchange ring is too short");
  // rows are written again: a tile that is read knows how far its reader is, by its items (polled) or its halo (staged)
  std::vector<std::set<int>> reads((size_t)p.ntiles), sees((size_t)p.ntiles);
  for (int64_t i = 0; i < (int64_t)p.V * ct::kOffsets; ++i)
    if (p.src[i] >= 0) reads[(size_t)(i / ct::kOffsets / ct::kFwdTileVoxels)].insert(p.src[i] / ct::kFwdTileVoxels);
  for (int t = 0; t < p.ntiles; ++t) {
    sees[(size_t)t] = reads[(size_t)t];
    for (int i = 0; routes == ct::kStaged && i < p.nhalo[t]; ++i)
      sees[(size_t)t].insert(p.halo[(size_t)t * ct::kFwdHaloMax + i] / ct::kFwdTileVoxels);
  }
  for (int t = 0; t < p.ntiles; ++t)
    for (int a : reads[(size_t)t])
      if (a != t && !sees[(size_t)a].count(t)) wrong(std::string(form) + ": a tile overwrites rows that are still read");
}
void check(const Recorded& r) {
  const ct::WaveLaunch& l = r.launch;
  if (!live(l.scns, sizeof(ct::WaveScn) * l.nscn) || !live(l.tiles, sizeof(int2) * l.ntiles) ||
      !live(l.phase_begin, sizeof(int) * (l.nphases + 1))) {
    wrong("batch tables are not in a live block");
    return;
  }
  if (l.phase_begin[0] != 0 || l.phase_begin[l.nphases] != l.ntiles) wrong("phases do not cover the tiles");
  if (!r.adjoint) g_orders.push_back(l.nphases);
  for (int f = 0; f < l.nphases; ++f) {
    const int begin = l.phase_begin[f], end = l.phase_begin[f + 1];
    if (end - begin > r.grid) need(l.record, (size_t)end * kRecordBytes, "a record of a tile that shares a CTA");
    for (int t = begin; t < end; ++t)
      if (l.tiles[t].x < 0 || l.tiles[t].x >= l.nscn) wrong("a tile of no scenario");
  }
  for (int i = 0; i < l.nscn; ++i) check_ring(l.scns[i], l.routes, r.adjoint ? "batched adjoint" : "batched forward");
}

void check_sweep(const Sweep& w) {
  int64_t dmin = INT32_MAX, dmax = 1;
  for (int64_t i = 0; i < w.d->V * ct::kOffsets; ++i)
    if (w.d->nbr[i] >= 0) {
      dmin = std::min<int64_t>(dmin, w.d->delays[i]);
      dmax = std::max<int64_t>(dmax, w.d->delays[i]);
    }
  if (!w.any && dmax - dmin > ct::kSweepRingSpread) wrong("delays too far apart for the sweep's ring");
  for (int b = 0; b < w.d->sweep_blocks; ++b)
    if (!w.any && w.d->snhalo[b] < 0) wrong("a halo too large for the sweep's ring");
}
cudaError_t sweep(const ct::DeviceScenario& d) {
  g_sweep_blocks = d.sweep_blocks;
  g_last_sweep = d.sweep_any;
  const Sweep w{&d, d.sweep_any};
  if (g_capturing)
    g_capturing->sweeps.push_back(w);
  else
    check_sweep(w);
  return cudaSuccess;
}

void count_routes(int (&n)[3], const ct::DeviceScenario& d, const int32_t* nhalo, const int32_t* near) {
  n[0] = n[1] = n[2] = 0;
  for (int t = 0; t < d.tiles; ++t) ++n[nhalo[t] < 0 ? 2 : nhalo[t] > 0 && near[t * ct::kNearTiles] < 0 ? 1 : 0];
}

}  // namespace

// ---- the library's host allocations
void* operator new(size_t n) {
  void* p = n >= g_host_fail_from && n < g_host_fail_from * 2 ? nullptr : std::malloc(n ? n : 1);
  if (!p) throw std::bad_alloc();
  return p;
}
void operator delete(void* p) noexcept { std::free(p); }
void operator delete(void* p, size_t) noexcept { std::free(p); }

extern "C" {

// ---- control
void host_device_fail_from(size_t bytes) { g_fail_from = bytes; }
void host_device_fail_host_from(size_t bytes) { g_host_fail_from = bytes; }
void host_device_no_threads(int on) { g_no_threads = on != 0; }
int pthread_create(pthread_t* t, const pthread_attr_t* a, void* (*f)(void*), void* p) {
  using Create = int (*)(pthread_t*, const pthread_attr_t*, void* (*)(void*), void*);
  static Create next = (Create)dlsym(RTLD_NEXT, "pthread_create");
  return g_no_threads ? EPERM : next(t, a, f, p);
}
size_t host_device_live() { return g_live; }
void host_device_times(const float* ms, int n) {
  g_times.assign(ms, ms + n);
  g_time = 0;
}
int host_device_report(char* out, int len) {  // and forget it
  std::strncpy(out, g_report.c_str(), (size_t)len - 1);
  out[len - 1] = 0;
  const int n = (int)g_report.size();
  g_report.clear();
  return n;
}
void host_device_landed(int when) { g_landed = when; }
int host_device_captures() { return std::exchange(g_captures, 0); }
int host_device_sweep_blocks() { return g_sweep_blocks; }
int host_device_last_sweep() { return g_last_sweep; }
int host_device_last_routes() { return g_last_routes; }
void host_device_routes(int* out) { std::memcpy(out, g_routes, sizeof(g_routes)); }
int host_device_phases(int* out, int len) {  // phases of the batched forwards since the last call
  const int n = (int)g_orders.size();
  for (int i = 0; i < n && i < len; ++i) out[i] = g_orders[(size_t)i];
  g_orders.clear();
  return n;
}

// ---- runtime
cudaError_t cudaMalloc(void** p, size_t n) {
  *p = nullptr;
  if (n >= g_fail_from) return g_last = cudaErrorMemoryAllocation;
  *p = std::calloc(n ? n : 1, 1);
  g_blocks[(char*)*p] = n;
  g_live += n;
  return cudaSuccess;
}
cudaError_t cudaFree(void* p) {
  if (!p) return cudaSuccess;
  auto it = g_blocks.find((char*)p);
  if (it == g_blocks.end()) return cudaErrorInvalidValue;
  g_live -= it->second;
  g_blocks.erase(it);  // the memory itself is not used again, so that a pointer kept too long is seen
  return cudaSuccess;
}
cudaError_t cudaMallocAsync(void** p, size_t n, cudaStream_t) { return cudaMalloc(p, n); }
cudaError_t cudaFreeAsync(void* p, cudaStream_t) { return cudaFree(p); }
cudaError_t cudaMallocHost(void** p, size_t n) {
  *p = std::calloc(n, 1);
  return cudaSuccess;
}
cudaError_t cudaFreeHost(void* p) {
  std::free(p);
  return cudaSuccess;
}
cudaError_t cudaMemcpy(void* d, const void* s, size_t n, cudaMemcpyKind) {
  std::memcpy(d, s, n);
  return cudaSuccess;
}
cudaError_t cudaMemcpyAsync(void* d, const void* s, size_t n, cudaMemcpyKind k, cudaStream_t) {
  return cudaMemcpy(d, s, n, k);
}
cudaError_t cudaMemset(void* d, int v, size_t n) {
  std::memset(d, v, n);
  return cudaSuccess;
}
cudaError_t cudaMemsetAsync(void* d, int v, size_t n, cudaStream_t) { return cudaMemset(d, v, n); }
cudaError_t cudaGetDeviceCount(int* n) { return *n = 1, cudaSuccess; }
cudaError_t cudaGetDevice(int* d) { return *d = 0, cudaSuccess; }
cudaError_t cudaSetDevice(int) { return cudaSuccess; }
cudaError_t cudaDeviceGetAttribute(int* v, cudaDeviceAttr, int) { return *v = kCapacity, cudaSuccess; }
cudaError_t cudaGetLastError() {
  const cudaError_t e = g_last;
  g_last = cudaSuccess;
  return e;
}
const char* cudaGetErrorString(cudaError_t) { return "made to fail"; }
cudaError_t cudaStreamCreateWithFlags(cudaStream_t* s, unsigned) { return *s = (cudaStream_t)1, cudaSuccess; }
cudaError_t cudaStreamDestroy(cudaStream_t) { return cudaSuccess; }
cudaError_t cudaStreamSynchronize(cudaStream_t) {
  g_waited = true;
  return cudaSuccess;
}
cudaError_t cudaStreamWaitEvent(cudaStream_t, cudaEvent_t, unsigned) { return cudaSuccess; }
cudaError_t cudaEventCreate(cudaEvent_t* e) { return *e = (cudaEvent_t)1, cudaSuccess; }
cudaError_t cudaEventCreateWithFlags(cudaEvent_t* e, unsigned) { return cudaEventCreate(e); }
cudaError_t cudaEventDestroy(cudaEvent_t) { return cudaSuccess; }
cudaError_t cudaEventRecord(cudaEvent_t, cudaStream_t) {
  g_waited = false;
  return cudaSuccess;
}
cudaError_t cudaEventQuery(cudaEvent_t) { return g_landed == 1 || (g_landed == 2 && g_waited) ? cudaSuccess : cudaErrorNotReady; }
cudaError_t cudaEventElapsedTime(float* ms, cudaEvent_t, cudaEvent_t) {
  *ms = g_time < g_times.size() ? g_times[g_time++] : 1.0f;
  return cudaSuccess;
}
cudaError_t cudaStreamBeginCapture(cudaStream_t, cudaStreamCaptureMode) {
  g_capturing = new Graph;
  ++g_captures;
  return cudaSuccess;
}
cudaError_t cudaStreamEndCapture(cudaStream_t, cudaGraph_t* g) {
  *g = (cudaGraph_t)g_capturing;
  g_capturing = nullptr;
  return cudaSuccess;
}
cudaError_t cudaGraphInstantiate(cudaGraphExec_t* e, cudaGraph_t g, unsigned long long) {
  *e = (cudaGraphExec_t) new Graph(*(Graph*)g);
  return cudaSuccess;
}
cudaError_t cudaGraphLaunch(cudaGraphExec_t e, cudaStream_t) {
  for (const Recorded& r : ((Graph*)e)->launches) check(r);
  for (const Sweep& w : ((Graph*)e)->sweeps) check_sweep(w);
  for (const auto& r : ((Graph*)e)->ranges)
    if (r.first->rev != r.second) wrong("a captured update leaves the adjoint's delay ranges behind");
  return cudaSuccess;
}
cudaError_t cudaGraphDestroy(cudaGraph_t g) {
  delete (Graph*)g;
  return cudaSuccess;
}
cudaError_t cudaGraphExecDestroy(cudaGraphExec_t e) {
  delete (Graph*)e;
  return cudaSuccess;
}
cudaError_t cudaGraphGetNodes(cudaGraph_t, cudaGraphNode_t*, size_t* n) { return *n = 0, cudaSuccess; }
cudaError_t cudaGraphNodeGetType(cudaGraphNode_t, cudaGraphNodeType* t) {
  return *t = cudaGraphNodeTypeKernel, cudaSuccess;
}
int ct_predict_measurements_noalloc(const float*, const float*, const float*, float*, float*, int64_t, int64_t, int64_t,
                                    void*) {
  return CT_ERR_NOT_SUPPORTED;
}
}  // extern "C"

namespace ct {

int wave_capacity(int) { return kCapacity; }
size_t wave_record_bytes() { return kRecordBytes; }
WaveScn wave_scenario(const DeviceScenario& d, bool adjoint, const WaveScalars&, float* part) {
  WaveScn a{};
  a.V = (int)d.V;
  a.T = (int)d.T;
  a.ntiles = d.tiles;
  a.xrows = d.xrows;
  a.src = adjoint ? d.rev : d.nbr;
  a.delays = d.delays;
  a.xch = d.xch;
  a.part = part;
  a.nhalo = adjoint ? d.rnhalo : d.nhalo;
  a.halo = adjoint ? d.rhalo : d.halo;
  a.rows = adjoint ? d.LX : nullptr;  // tells the directions apart here
  return a;
}
cudaError_t launch_wave(const WaveLaunch& l, bool adjoint, int grid, cudaStream_t) {
  const Recorded r{l, adjoint, grid};
  if (g_capturing)
    g_capturing->launches.push_back(r);
  else
    check(r);
  return cudaSuccess;
}
cudaError_t launch_forward(DeviceScenario& d, float, cudaStream_t) {
  g_last_routes = d.routes;
  check_ring(wave_scenario(d, false, WaveScalars{}, nullptr), d.routes, "forward");
  count_routes(g_routes[0], d, d.nhalo, d.near);
  if (d.tiles > d.wave_grid) need(d.record, (size_t)d.tiles * kRecordBytes, "forward record");
  return cudaSuccess;
}
cudaError_t launch_adjoint_states(DeviceScenario& d, const WaveScalars&, cudaStream_t) {
  check_ring(wave_scenario(d, true, WaveScalars{}, nullptr), d.rroutes, "adjoint");
  count_routes(g_routes[1], d, d.rnhalo, d.rnear);
  return cudaSuccess;
}
cudaError_t clear_exchange(DeviceScenario& d, cudaStream_t) {
  if (!g_capturing) need(d.xch, sizeof(uint4) * (size_t)d.xrows * d.V, "exchange ring");
  return cudaSuccess;
}
cudaError_t launch_delay_ranges(DeviceScenario& d, cudaStream_t) {
  if (g_capturing) g_capturing->ranges.push_back({&d, d.rev});
  d.dmin[0] = INT32_MAX;
  d.dmin[1] = INT32_MIN;
  for (int64_t i = 0; i < d.V * kOffsets; ++i)
    if (d.nbr[i] >= 0) {
      if (d.delays[i] < d.dmin[0]) d.dmin[0] = d.delays[i];
      if (d.delays[i] > d.dmin[1]) d.dmin[1] = d.delays[i];
    }
  return cudaSuccess;
}
cudaError_t launch_mirror_tables(DeviceScenario& d, cudaStream_t) {
  const int64_t n = (int64_t)d.tiles * kFwdTileVoxels * kOffsets;
  need(d.rev, sizeof(int32_t) * d.V * kOffsets, "reverse table");
  need(d.rhslot, sizeof(int16_t) * n, "reverse slots");
  for (int64_t i = 0; i < d.V * kOffsets; ++i) d.rev[i] = d.nbr[i / kOffsets * kOffsets + (kOffsets - 1 - i % kOffsets)];
  return cudaSuccess;
}
cudaError_t launch_permute_blocks(const void* src, void* dst, const int32_t* perm, int64_t V, int64_t words, bool gather,
                                  cudaStream_t) {
  for (int64_t u = 0; u < V; ++u)
    std::memcpy((int32_t*)dst + (gather ? u : perm[u]) * words, (const int32_t*)src + (gather ? perm[u] : u) * words,
                sizeof(int32_t) * (size_t)words);
  return cudaSuccess;
}

int measure_ksplit(int64_t, int64_t, int64_t, int) { return 1; }
bool umma_supported(int64_t) { return false; }
int umma_yn(int64_t) { return 64; }
int umma_ksplit(int64_t, int64_t, int64_t, int) { return 1; }
int64_t slice_pitch(int64_t k) { return k; }
int64_t slice_groups(int64_t) { return 1; }
int slice_ksplit(int64_t, int64_t, int64_t, int) { return 1; }
PostPlan post_plan(int64_t, int64_t, int) { return PostPlan{}; }
int plain_step_launches(const PlainScalars&) { return 1; }
float lead_field_factor(float) { return 1.0f; }
void connect_voxels_host(const int32_t*, const int32_t*, const float*, int64_t, int64_t, int64_t, const float*, float,
                         float*, float*) {}
void output_state_indices_host(const int32_t*, const int32_t*, int64_t, int64_t, int64_t, const std::vector<int64_t>&,
                               int32_t*) {}
cudaError_t umma_prepare(DeviceScenario&, cudaStream_t) { return cudaSuccess; }
cudaError_t slice_prepare(DeviceScenario&, cudaStream_t) { return cudaSuccess; }
cudaError_t launch_derive(DeviceScenario& d, const DeriveScalars&, cudaStream_t) { return sweep(d); }
cudaError_t launch_adjoint_gradients(DeviceScenario& d, const DeriveScalars&, cudaStream_t) { return sweep(d); }
cudaError_t launch_update(DeviceScenario&, const UpdateScalars&, cudaStream_t) { return cudaSuccess; }
cudaError_t launch_measure(DeviceScenario&, int64_t, bool, cudaStream_t) { return cudaGetLastError(); }
cudaError_t launch_map_residuals(DeviceScenario&, int64_t, cudaStream_t) { return cudaSuccess; }
cudaError_t launch_measure_umma(DeviceScenario&, int64_t, bool, int, cudaStream_t) { return cudaSuccess; }
cudaError_t launch_map_residuals_umma(DeviceScenario&, int64_t, int, cudaStream_t) { return cudaSuccess; }
cudaError_t launch_measure_sliced(DeviceScenario&, int64_t, bool, cudaStream_t) { return cudaSuccess; }
cudaError_t launch_map_residuals_sliced(DeviceScenario&, int64_t, cudaStream_t) { return cudaSuccess; }
cudaError_t launch_plain_beat(DeviceScenario&, int64_t, const PlainScalars&, cudaStream_t) { return cudaSuccess; }
cudaError_t launch_step_metrics(DeviceScenario&, float, cudaStream_t) { return cudaSuccess; }
cudaError_t launch_step_metrics_parts(DeviceScenario&, const float*, int, float, cudaStream_t) { return cudaSuccess; }
cudaError_t launch_batch_metrics(DeviceScenario&, int64_t, cudaStream_t) { return cudaSuccess; }
cudaError_t launch_batch_metrics_dev(DeviceScenario&, const int64_t*, cudaStream_t) { return cudaSuccess; }
cudaError_t launch_average_delays(DeviceScenario&, cudaStream_t) { return cudaSuccess; }
cudaError_t launch_smoothness(DeviceScenario&, float, cudaStream_t) { return cudaSuccess; }
cudaError_t launch_last_max_reg(DeviceScenario&, float, float*, cudaStream_t) { return cudaSuccess; }
cudaError_t launch_spherical(const DeviceScenario&, const PostBuffers&, const PostPlan&, bool, float, cudaStream_t) {
  return cudaSuccess;
}
cudaError_t launch_final_metrics(const PostBuffers&, const int32_t*, const int32_t*, int64_t, unsigned long long*, float*,
                                 int, cudaStream_t) {
  return cudaSuccess;
}
cudaError_t launch_lead_field(const float*, const int32_t*, int64_t, const float*, const float*, const float*, int64_t,
                              int64_t, float, float*, int64_t, int, cudaStream_t) {
  return cudaSuccess;
}
cudaError_t launch_delay_samples(const int32_t*, const int32_t*, const float*, int64_t, int64_t, int64_t, const float*,
                                 float, float*, int32_t*, float*, unsigned long long*, int, cudaStream_t) {
  return cudaSuccess;
}

}  // namespace ct
