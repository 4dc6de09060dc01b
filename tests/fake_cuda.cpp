// A stand-in for the CUDA runtime and the kernels behind csrc/api.cu, so that
// the host code of the C ABI runs on a machine without a GPU (test_host_abi.py
// compiles the two together).  Memory is host memory and copies happen at
// once.  It knows two devices, refuses a launch on a stream of a device that
// is not current, lets a test hold a stream's work back or make a call fail,
// and counts what the rules forbid: a graph destroyed while it may still run,
// a tile launch without tensor maps, memory freed twice.
#include "fake_prelude.h"

#include <condition_variable>
#include <cstring>
#include <map>
#include <mutex>
#include <set>
#include <string>

#include "split_common.cuh"

using namespace phono;

namespace {
struct Stream {
  int dev;
  bool held = false;
  std::set<void*> flying;    // graphs launched and not waited for
  std::set<Stream*> behind;  // streams whose work this one waits for
};
struct Event {
  Stream* at = nullptr;
};
struct Block {
  size_t bytes;
  int dev;
};
std::mutex g_m;
std::condition_variable g_cv;
std::map<char*, Block> g_mem, g_pinned;
std::map<std::string, int> g_fail, g_count;
std::set<Stream*> g_streams;
int g_broken = 0;
size_t g_limit = 0;  // bytes all allocations may take (0: any)
thread_local int g_dev = 0;
Stream* S(cudaStream_t s) { return reinterpret_cast<Stream*>(s); }
Event* E(cudaEvent_t e) { return reinterpret_cast<Event*>(e); }

bool fails(const char* what) {  // counts down to the call that fails
  std::lock_guard<std::mutex> hold(g_m);
  auto f = g_fail.find(what);
  if (f == g_fail.end() || f->second == 0) return false;
  return --f->second == 0;
}
void landed(Stream* s) {
  s->flying.clear();
  for (Stream* t : s->behind) t->flying.clear();
  s->behind.clear();
}
cudaError_t launch(const char* what, cudaStream_t st) {
  if (fails(what)) return cudaErrorUnknown;
  std::lock_guard<std::mutex> hold(g_m);
  if (S(st)->dev != g_dev) return cudaErrorInvalidResourceHandle;
  g_count[what]++;
  return cudaSuccess;
}
CUresult encode(CUtensorMap* t, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*, const cuuint64_t*, const cuuint32_t*,
                const cuuint32_t*, CUtensorMapInterleave, CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill) {
  if (fails("encode")) return CUDA_ERROR_UNKNOWN;
  t->opaque[0] = 1;
  return CUDA_SUCCESS;
}
template <class R>
cudaError_t step(const StepArgs<R>& a, cudaStream_t st) {
  if (!a.tm_u.opaque[0] || !a.tm_mat.opaque[0]) g_broken++;
  return launch("tile", st);
}
}  // namespace

void fake_launch(cudaStream_t st) { launch("other", st); }

namespace phono {
cudaError_t configure_step_f64(int) { return fails("configure") ? cudaErrorUnknown : cudaSuccess; }
cudaError_t configure_step_f32k(int) { return fails("configure") ? cudaErrorUnknown : cudaSuccess; }
cudaError_t configure_step_f64v(int) { return fails("configure") ? cudaErrorUnknown : cudaSuccess; }
cudaError_t launch_step_f64(const StepArgs<double>& a, int, int, cudaStream_t st) { return step(a, st); }
cudaError_t launch_step_f64v(const StepArgs<double>& a, int, int, cudaStream_t st) { return step(a, st); }
cudaError_t launch_step_f32k(const StepArgs<float>& a, int, int, cudaStream_t st) { return step(a, st); }
cudaError_t launch_split(int, const void*, bool, bool, cudaStream_t st) { return launch("split", st); }
cudaError_t launch_energy(const EnergyArgs&, double2*, int, double*, int, cudaStream_t st) { return launch("energy", st); }
cudaError_t launch_lattice_ids(uint8_t*, const Geo&, int, int, int, const double*, const uint8_t*, int, uint8_t, cudaStream_t st) {
  return launch("lattice", st);
}
cudaError_t launch_inclusion_ids(uint8_t*, const Geo&, const double*, const double*, const double4*, const int*, const uint8_t*, int,
                                 uint8_t, cudaStream_t st) {
  return launch("inclusions", st);
}
cudaError_t launch_unpack_ids(uint8_t* mat, const Geo& g, const uint8_t* dense, long long first, int rows, cudaStream_t st) {
  const cudaError_t e = launch("unpack", st);
  for (long long r = first; e == cudaSuccess && r < first + rows; r++)
    std::memcpy(mat + g.mo0 + r / g.ny * g.msx + r % g.ny * g.msy, dense + (r - first) * g.nz, g.nz);
  return e;
}
cudaError_t launch_readback(const void* in, long long sx, long long sy, int ex, int ey, int ez, int es, void* out, cudaStream_t st) {
  const cudaError_t e = launch("readback", st);
  for (int i = 0; e == cudaSuccess && i < ex; i++)
    for (int j = 0; j < ey; j++)
      std::memcpy((char*)out + ((size_t)i * ey + j) * ez * es, (const char*)in + (i * sx + j * sy) * es, (size_t)ez * es);
  return e;
}
}  // namespace phono

extern "C" {

// ---- controls ----
void fake_hold(void* s, int on) {
  std::lock_guard<std::mutex> hold(g_m);
  ((Stream*)s)->held = on;
  g_cv.notify_all();
}
void fake_fail(const char* what, int after) {  // the after-th call of its kind from now fails
  std::lock_guard<std::mutex> hold(g_m);
  g_fail[what] = after;
}
void fake_reset() {
  g_fail.clear();
  g_broken = 0;
  g_limit = 0;
}
void fake_limit(size_t bytes) { g_limit = bytes; }
void fake_device(int dev) { g_dev = dev; }
int fake_current() { return g_dev; }
int fake_broken() { return g_broken; }
int fake_count(const char* what) { return g_count[what]; }
size_t fake_bytes(int dev) {  // each allocation rounded up to 512 bytes
  size_t n = 0;
  for (auto& m : g_mem)
    if (m.second.dev == dev) n += (m.second.bytes + 511) / 512 * 512;
  return n;
}
void fake_pin(void* p, size_t bytes) { g_pinned[(char*)p] = Block{bytes, 0}; }

// ---- the runtime ----
const char* cudaGetErrorString(cudaError_t) { return "fake error"; }
cudaError_t cudaGetLastError() { return cudaSuccess; }
cudaError_t cudaGetDevice(int* d) { return *d = g_dev, cudaSuccess; }
cudaError_t cudaSetDevice(int d) { return g_dev = d, cudaSuccess; }
cudaError_t cudaDeviceGetAttribute(int* v, enum cudaDeviceAttr, int) { return *v = 152, cudaSuccess; }
cudaError_t cudaMalloc(void** p, size_t n) {
  if (fails("malloc") || (g_limit && fake_bytes(g_dev) + (n + 511) / 512 * 512 > g_limit)) return cudaErrorMemoryAllocation;
  *p = std::calloc(n, 1);
  std::lock_guard<std::mutex> hold(g_m);
  g_mem[(char*)*p] = Block{n, g_dev};
  return cudaSuccess;
}
cudaError_t cudaFree(void* p) {
  if (!p) return cudaSuccess;
  std::lock_guard<std::mutex> hold(g_m);
  if (!g_mem.erase((char*)p)) g_broken++;
  else std::free(p);
  return cudaSuccess;
}
cudaError_t cudaMemcpy(void* d, const void* s, size_t n, enum cudaMemcpyKind) { return std::memcpy(d, s, n), cudaSuccess; }
cudaError_t cudaMemcpyAsync(void* d, const void* s, size_t n, enum cudaMemcpyKind, cudaStream_t) {
  if (fails("copy")) return cudaErrorUnknown;
  return std::memcpy(d, s, n), cudaSuccess;
}
cudaError_t cudaMemsetAsync(void* d, int v, size_t n, cudaStream_t) { return std::memset(d, v, n), cudaSuccess; }
cudaError_t cudaMemcpy3DAsync(const struct cudaMemcpy3DParms* p, cudaStream_t) {
  for (size_t i = 0; i < p->extent.depth; i++)
    for (size_t j = 0; j < p->extent.height; j++)
      std::memcpy((char*)p->dstPtr.ptr + (i * p->dstPtr.ysize + j) * p->dstPtr.pitch,
                  (const char*)p->srcPtr.ptr + (i * p->srcPtr.ysize + j) * p->srcPtr.pitch, p->extent.width);
  return cudaSuccess;
}
cudaError_t cudaPointerGetAttributes(struct cudaPointerAttributes* a, const void* p) {
  *a = cudaPointerAttributes{};
  for (auto& m : g_pinned)
    if ((char*)p >= m.first && (char*)p < m.first + m.second.bytes) a->type = cudaMemoryTypeHost, a->devicePointer = (void*)p;
  return cudaSuccess;
}
cudaError_t cudaStreamCreateWithFlags(cudaStream_t* s, unsigned) {
  std::lock_guard<std::mutex> hold(g_m);
  Stream* t = new Stream{g_dev};
  g_streams.insert(t);
  *s = reinterpret_cast<cudaStream_t>(t);
  return cudaSuccess;
}
cudaError_t cudaStreamDestroy(cudaStream_t) { return cudaSuccess; }  // (kept: other streams may name it)
cudaError_t cudaStreamSynchronize(cudaStream_t s) {
  if (fails("sync")) return cudaErrorUnknown;
  std::unique_lock<std::mutex> hold(g_m);
  g_cv.wait(hold, [&] { return !S(s)->held; });
  landed(S(s));
  return cudaSuccess;
}
cudaError_t cudaStreamWaitEvent(cudaStream_t s, cudaEvent_t e, unsigned) {
  std::lock_guard<std::mutex> hold(g_m);
  if (E(e)->at) S(s)->behind.insert(E(e)->at);
  return cudaSuccess;
}
cudaError_t cudaStreamBeginCapture(cudaStream_t, enum cudaStreamCaptureMode) { return cudaSuccess; }
cudaError_t cudaStreamEndCapture(cudaStream_t, cudaGraph_t* g) {
  *g = reinterpret_cast<cudaGraph_t>(new int);
  return cudaSuccess;
}
cudaError_t cudaGraphInstantiate(cudaGraphExec_t* x, cudaGraph_t, unsigned long long) {
  *x = reinterpret_cast<cudaGraphExec_t>(new int);
  return cudaSuccess;
}
cudaError_t cudaGraphDestroy(cudaGraph_t g) { return delete reinterpret_cast<int*>(g), cudaSuccess; }
cudaError_t cudaGraphLaunch(cudaGraphExec_t x, cudaStream_t s) {
  std::lock_guard<std::mutex> hold(g_m);
  S(s)->flying.insert(x);
  g_count["graph"]++;
  return cudaSuccess;
}
cudaError_t cudaGraphExecDestroy(cudaGraphExec_t x) {
  std::lock_guard<std::mutex> hold(g_m);
  for (Stream* s : g_streams) g_broken += (int)s->flying.count(x);
  return cudaSuccess;  // (kept: its address stays its own)
}
cudaError_t cudaEventCreateWithFlags(cudaEvent_t* e, unsigned) {
  *e = reinterpret_cast<cudaEvent_t>(new Event);
  return cudaSuccess;
}
cudaError_t cudaEventCreate(cudaEvent_t* e) { return cudaEventCreateWithFlags(e, 0); }
cudaError_t cudaEventDestroy(cudaEvent_t e) { return delete E(e), cudaSuccess; }
cudaError_t cudaEventRecord(cudaEvent_t e, cudaStream_t s) {
  std::lock_guard<std::mutex> hold(g_m);
  E(e)->at = S(s);
  return cudaSuccess;
}
cudaError_t cudaEventSynchronize(cudaEvent_t) { return cudaSuccess; }
cudaError_t cudaEventElapsedTime(float* ms, cudaEvent_t, cudaEvent_t) { return *ms = 1.f, cudaSuccess; }
cudaError_t cudaGetDriverEntryPointByVersion(const char*, void** fn, unsigned, unsigned long long,
                                             enum cudaDriverEntryPointQueryResult* r) {
  *fn = (void*)encode;
  if (r) *r = cudaDriverEntryPointSuccess;
  return cudaSuccess;
}

}  // extern "C"
