// C ABI of libphono_gpu.so (declared in include/phono.h).
#include <cmath>
#include <climits>
#include <cstdio>
#include <cstring>
#include <mutex>
#include <string>
#include <vector>
#include <algorithm>

#include "../../include/phono.h"
#include <cudaTypedefs.h>
#include "split_common.cuh"

namespace phono {
cudaError_t configure_step_f64(int tj);
cudaError_t configure_step_f32k(int tj);
cudaError_t launch_step_f64(const StepArgs<double>& a, int tj, int n_face_blocks, cudaStream_t st);
cudaError_t launch_step_f32k(const StepArgs<float>& a, int tj, int n_face_blocks, cudaStream_t st);
cudaError_t configure_step_f64v(int tj);
cudaError_t launch_step_f64v(const StepArgs<double>& a, int tj, int n_face_blocks, cudaStream_t st);
cudaError_t launch_split(int precision, const void* args, bool stress, bool after_kernel, cudaStream_t st);
cudaError_t launch_energy(const EnergyArgs& a, double2* partial, int nblocks, double* out, int march_blocks, cudaStream_t st);
cudaError_t launch_lattice_ids(uint8_t* mat, const Geo& g, int pitch, int ncx, int ncy, const double* radius,
                               const uint8_t* kind, int depth, uint8_t host, cudaStream_t st);
cudaError_t launch_unpack_ids(uint8_t* mat, const Geo& g, const uint8_t* dense, long long first, int rows, cudaStream_t st);
cudaError_t launch_readback(const void* in, long long sx, long long sy, int ex, int ey, int ez, int es, void* out,
                            cudaStream_t st);
cudaError_t launch_inclusion_ids(uint8_t* mat, const Geo& g, const double* x, const double* y, const double4* incl,
                                 const int* kend, const uint8_t* id, int n, uint8_t host, cudaStream_t st);

__global__ void advance_step_kernel(int* p, int n) { *p += n; }
// a batched instance's step counter, stopping at its budget
__global__ void advance_clamped_kernel(int* p, int n, int end) { *p = min(*p + n, end); }
}  // namespace phono

using namespace phono;

static thread_local std::string g_err;

static int fail(int code, const std::string& msg) {
  g_err = msg;
  return code;
}

namespace phono {
void set_last_error(const char* msg) { g_err = msg; }
}  // namespace phono

#define CK(call)                                                                        \
  do {                                                                                  \
    cudaError_t e_ = (call);                                                            \
    if (e_ != cudaSuccess) return fail(PHONO_ERR_CUDA, std::string(#call) + ": " + cudaGetErrorString(e_)); \
  } while (0)

static const int kGraphSteps = 12;  // multiple of 2 and 3: buffer rotations line up
static const int kEnergyBlocks = 1024;
// FP32 meshes from here on sum their energy marching along x: smaller ones have
// too few columns for it (energy.cu: 42.8 us a call without and 53.2 with it at
// 108 k nodes, 78.3 and 67.1 at 207 k)
static const double kEnergyMarchNodes = 200000;

// the FP64 velocity form's two-launch step multiplies by constants in integer
// arithmetic from here on (split_step.cu: 35 k nodes 9.5 us a step without and
// 10.9 with it, 78 k nodes 13.9 and 13.4)
static const double kSoftVelNodes = 60000;

// tile decomposition of the tile pass and the TMA descriptors of its boxes
struct Tiling {
  int tj = 0, xseg = 64, ntj = 0, ntk = 0, nseg = 0, n_tile = 0;
  std::vector<int> seg_start;  // first plane of each x segment, + nx-1
  CUtensorMap tm_u{}, tm_mat{}, tm_pw0{}, tm_pw1{};
};

struct phono_handle {
  phono_desc d;  // scalar copy; pointers not kept
  int es = 8;
  Geo g{};
  size_t field_elems = 0;  // per array
  size_t mat_bytes = 0;
  std::vector<void*> allocs;
  int nbuf = 3;            // u buffers: 3 rotating (F64) or 2 ping-pong (F32K)
  char* ubase = nullptr;   // nbuf x 3 padded arrays, buffer-major
  char* vbase = nullptr;   // F32K: 2 x 3 velocity arrays
  char* cbase = nullptr;   // F32K: 2 x 3 Kahan arrays
  void* sp[6] = {};       // R spacings (F64 raw, F32K reciprocals)
  double* rsp64[6] = {};  // reciprocal double spacings 1/fd, 1/sd (energy)
  double h_sp0[6] = {};   // first elements (raw)
  DivTable dtab{};        // FP64 leapfrog: reciprocal pairs of the mesh's divisors (tab null: none)
  std::vector<double> sp_host[6];  // raw spacings (ABC coefficients)
  uint8_t* mat = nullptr;
  int dev = 0;               // the device the handle was made on
  bool in_stage = false;     // it counts among the users of that device's stage
  void* tab = nullptr;       // 16 R per material
  double* tab13 = nullptr;   // raw table (energy)
  double* src = nullptr;
  int nsrc = 0;
  void* surf = nullptr;
  int nrec_cap = 0;
  int* step_base = nullptr;
  int* err = nullptr;
  double2* partial = nullptr;
  double* energy_out = nullptr;
  double abc[8] = {};
  Tiling t;                    // the tile shape the caller knows
  Tiling own;                  // a default handle's own shape (own.tj 0: t)
  int own_limit = 0;           // longest segment of it in a batch (0: alone)
  bool lent = false;           // not a default handle: own is its batch's choice
  int separate_faces = 1;
  FaceTable faces{};
  // two-launch step (split_step.cu): stress window of `win` planes (0: this
  // mesh has none).  split: the handle steps that way (default tile shape);
  // the velocity forms' v and Kahan terms then stay in buffer 0
  int win = 0, tsy = 0;
  bool split = false;
  bool resplit = false;        // in a batch (tile pass): back to the two-launch form when it leaves
  char* stress = nullptr;      // leapfrog: the window
  SoftRec* rec = nullptr;      // FP64: table entries as records, 16 per material
  int shared = 0;              // leapfrog: the normal stresses share terms (split_step.cu)
  void* spd[6] = {};           // divisors of the two-launch step (FP64: records or factors, FP32: sp)
  double* vals = nullptr;      // leapfrog: values of all records
  cudaStream_t stream = nullptr;
  cudaGraphExec_t graph = nullptr;
  cudaEvent_t ev0 = nullptr, ev1 = nullptr;
  int steps_done = 0;
  int nmat = 0;
  bool timed = false;
  phono_batch* batch = nullptr;  // the batch that steps this handle, if any
  int wait_polls = 0;            // tile-pass wait budget (0: default)
  int skip_plane = -1;           // test hook of phono_test_wait_timeout (-1: off)
};

static long long round_up(long long x, long long m) { return (x + m - 1) / m * m; }

// a leapfrog handle that keeps to tiles has no use for its stress window
static cudaError_t drop_window(phono_handle* h) {
  if (!h->stress) return cudaSuccess;
  h->allocs.erase(std::find(h->allocs.begin(), h->allocs.end(), h->stress));
  const cudaError_t e = cudaFree(h->stress);
  h->stress = nullptr;
  h->win = 0;
  h->split = false;
  return e;
}

// memory of a handle that is being made: where it does not fit beside the stress
// window, the handle does without the window
static int dalloc(phono_handle* h, void** p, size_t bytes) {
  cudaError_t e = cudaMalloc(p, bytes);
  if (e != cudaSuccess && h->stress) {
    cudaGetLastError();
    drop_window(h);
    e = cudaMalloc(p, bytes);
  }
  if (e != cudaSuccess) {
    *p = nullptr;
    return fail(PHONO_ERR_NOMEM, std::string("cudaMalloc ") + std::to_string(bytes) + " bytes: " + cudaGetErrorString(e));
  }
  h->allocs.push_back(*p);
  return PHONO_OK;
}

static void batch_detach(phono_batch* b, const phono_handle* h);
static void leave_stage(phono_handle* h);

static void release(phono_handle* h) {
  if (!h) return;
  if (h->batch) batch_detach(h->batch, h);
  if (h->stream) cudaStreamSynchronize(h->stream);
  if (h->graph) cudaGraphExecDestroy(h->graph);
  for (void* p : h->allocs) cudaFree(p);
  leave_stage(h);
  if (h->ev0) cudaEventDestroy(h->ev0);
  if (h->ev1) cudaEventDestroy(h->ev1);
  if (h->stream) cudaStreamDestroy(h->stream);
  delete h;
}

// ABC coefficients in the reference order from the material at node (0,0,0)
// (base_solver.py:525-537): clx[-1] ctx[-1] cty[0] cly[0] cty[-1] cly[-1] ctz[-1] clz[-1]
static void abc_coeffs(const phono_handle* h, const double* row0, double out[8]) {
  double vl = std::sqrt(row0[0] / row0[12]);
  double vt = std::sqrt(row0[9] / row0[12]);
  double vld = vl * h->d.dt, vtd = vt * h->d.dt;
  const int nx = h->d.nx, ny = h->d.ny, nz = h->d.nz;
  const std::vector<double>&fdx = h->sp_host[0], &fdy = h->sp_host[1], &fdz = h->sp_host[2];
  const std::vector<double>&sdx = h->sp_host[3], &sdy = h->sp_host[4], &sdz = h->sp_host[5];
  out[0] = (vld - sdx[nx - 3]) / (vld + sdx[nx - 3]);
  out[1] = (vtd - fdx[nx - 2]) / (vtd + fdx[nx - 2]);
  out[2] = (vtd - fdy[0]) / (vtd + fdy[0]);
  out[3] = (vld - sdy[0]) / (vld + sdy[0]);
  out[4] = (vtd - fdy[ny - 2]) / (vtd + fdy[ny - 2]);
  out[5] = (vld - sdy[ny - 3]) / (vld + sdy[ny - 3]);
  out[6] = (vtd - fdz[nz - 2]) / (vtd + fdz[nz - 2]);
  out[7] = (vld - sdz[nz - 3]) / (vld + sdz[nz - 3]);
}

// the largest of n ids, 64 at a time: a byte at a time took most of a material
// upload (160x128x64 cells: 837 us with it, 416 without)
static int largest_id(const uint8_t* id, size_t n) {
  uint8_t m[64] = {};
  size_t p = 0;
  for (; p + 64 <= n; p += 64)
    for (int q = 0; q < 64; q++) m[q] = id[p + q] > m[q] ? id[p + q] : m[q];
  for (; p < n; p++) m[0] = std::max(m[0], id[p]);
  return *std::max_element(m, m + 64);
}

static int check_materials(const phono_handle* h, const uint8_t* mat, const double* table, int nmat) {
  if (!mat || !table) return fail(PHONO_ERR_ARG, "material ids or table is NULL");
  if (nmat < 1 || nmat > 256) return fail(PHONO_ERR_ARG, "nmat must be in 1..256");
  for (int q = 0; q < nmat * PHONO_TABLE_COLS; q++)
    if (!std::isfinite(table[q])) return fail(PHONO_ERR_ARG, "material table holds a non-finite value");
  for (int q = 0; q < nmat; q++)
    if (!(table[q * PHONO_TABLE_COLS + 12] > 0.0)) return fail(PHONO_ERR_ARG, "density must be > 0");
  size_t n = (size_t)h->d.nx * h->d.ny * h->d.nz;
  if (largest_id(mat, n) >= nmat) return fail(PHONO_ERR_ARG, "material id out of range");
  return PHONO_OK;
}

// From 256 KB on, ids pass through a stage of whole rows on the way to the
// padded layout, where a kernel puts them: a strided copy moves a row (65 bytes,
// say) at a time (us an upload, strided / staged: 160x128x64 cells 416 / 89,
// 256x256x128 2334 / 539, 512x512x256 11300 / 4100).  One stage a device, made at
// the first such upload and given back with the device's last handle; an upload
// holds it for its own copies alone: it waits for the handle's earlier work
// before.  Handles come and go meanwhile (an upload's handle is a user, so that
// the stage is not given back under it).
struct IdStage {
  std::mutex upload;  // held for an upload's copies
  std::mutex count;   // held while a handle joins or leaves
  int users = 0;
  uint8_t* p = nullptr;
};
static IdStage g_stage[32];
constexpr size_t kStageBytes = 4 << 20, kStagedFrom = 256 << 10;

static void join_stage(phono_handle* h) {
  if (h->dev < 0 || h->dev >= 32) return;
  std::lock_guard<std::mutex> hold(g_stage[h->dev].count);
  g_stage[h->dev].users++;
  h->in_stage = true;
}
static void leave_stage(phono_handle* h) {
  if (!h->in_stage) return;
  IdStage& g = g_stage[h->dev];
  std::lock_guard<std::mutex> hold(g.count);
  if (--g.users == 0 && g.p) {
    cudaFree(g.p);
    g.p = nullptr;
  }
  h->in_stage = false;
}

// A launch goes to a stream of the current device only; copies do not mind.
// Calls that were copies make the handle's device current for their launches.
struct OnDevice {
  int back = -1;
  cudaError_t err;
  explicit OnDevice(int dev) {
    int now = dev;
    err = cudaGetDevice(&now);
    if (err == cudaSuccess && now != dev && (err = cudaSetDevice(dev)) == cudaSuccess) back = now;
  }
  ~OnDevice() {
    if (back >= 0) cudaSetDevice(back);
  }
};

// `staged`: the ids are in place (else nothing was done)
static int upload_staged(phono_handle* h, const uint8_t* mat, bool& staged) {
  const int nz = h->d.nz;
  const long long rows = (long long)h->d.nx * h->d.ny, step = (long long)kStageBytes / nz;
  if (!h->in_stage || (size_t)rows * nz < kStagedFrom || step < 1) return PHONO_OK;
  const OnDevice here(h->dev);
  CK(here.err);
  CK(cudaStreamSynchronize(h->stream));
  IdStage& g = g_stage[h->dev];
  std::lock_guard<std::mutex> hold(g.upload);
  if (!g.p && cudaMalloc(&g.p, kStageBytes) != cudaSuccess) {
    g.p = nullptr;
    cudaGetLastError();
    return PHONO_OK;
  }
  cudaError_t e = cudaSuccess;
  for (long long first = 0; first < rows && e == cudaSuccess; first += step) {
    const int n = (int)std::min(step, rows - first);
    e = cudaMemcpyAsync(g.p, mat + first * nz, (size_t)n * nz, cudaMemcpyHostToDevice, h->stream);
    if (e == cudaSuccess) e = launch_unpack_ids(h->mat, h->g, g.p, first, n, h->stream);
  }
  const cudaError_t done = cudaStreamSynchronize(h->stream);
  CK(e);
  CK(done);
  staged = true;
  return PHONO_OK;
}

// ids into the padded layout, 16-entry device rows, raw rows, ABC coefficients
static int upload_table(phono_handle* h, const double* table, int nmat, int id000);

static int upload_materials(phono_handle* h, const uint8_t* mat, const double* table, int nmat) {
  const int nx = h->d.nx, ny = h->d.ny, nz = h->d.nz;
  bool staged = false;
  if (const int rc = upload_staged(h, mat, staged)) return rc;
  if (!staged) {
    cudaMemcpy3DParms p{};
    p.srcPtr = make_cudaPitchedPtr((void*)mat, nz, nz, ny);
    p.dstPtr = make_cudaPitchedPtr(h->mat + h->g.mo0, h->g.msy, h->g.msy, ny + 2);
    p.extent = make_cudaExtent(nz, ny, nx);
    p.kind = cudaMemcpyHostToDevice;
    CK(cudaMemcpy3DAsync(&p, h->stream));
  }
  return upload_table(h, table, nmat, mat[0]);
}

// the 16-entry device rows of the material table; id000 = the material at
// node (0, 0, 0), whose wave speeds set the absorbing-face coefficients
static int upload_table(phono_handle* h, const double* table, int nmat, int id000) {
  const double dt = h->d.dt;
  const double dt2 = dt * dt;
  const bool leapfrog = h->d.precision == PHONO_F64;
  std::vector<double> t(16 * nmat, 0.0);
  for (int m = 0; m < nmat; m++) {
    const double* row = table + m * PHONO_TABLE_COLS;
    for (int q = 0; q < 12; q++) t[m * 16 + q] = row[q];
    // (dt**2 / P) of base_solver.py:443 for the leapfrog, dt / P for the velocity form
    t[m * 16 + 12] = leapfrog ? dt2 / row[12] : dt / row[12];
    t[m * 16 + 13] = row[12];
    t[m * 16 + 14] = dt;
  }
  std::vector<float> t32;
  std::vector<SoftRec> rec;
  if (h->es == 8) {
    CK(cudaMemcpyAsync(h->tab, t.data(), t.size() * 8, cudaMemcpyHostToDevice, h->stream));
  } else {
    t32.assign(t.begin(), t.end());
    CK(cudaMemcpyAsync(h->tab, t32.data(), t32.size() * 4, cudaMemcpyHostToDevice, h->stream));
  }
  if (h->rec) {  // the same entries for the two-launch step
    for (size_t q = 0; q < t.size(); q++) rec.push_back(soft_record(t[q], false, (uint32_t)q));
    CK(cudaMemcpyAsync(h->rec, rec.data(), rec.size() * sizeof(SoftRec), cudaMemcpyHostToDevice, h->stream));
  }
  if (leapfrog) {
    h->shared = 1;
    for (int m = 0; m < nmat; m++) {
      const double* c = table + m * PHONO_TABLE_COLS;
      auto same = [&](int p, int q) { return soft_bits(c[p]) == soft_bits(c[q]); };  // zeros with their signs
      h->shared &= same(3, 6) && same(1, 7) && same(2, 5);
    }
    CK(cudaMemcpyAsync(h->vals, t.data(), t.size() * 8, cudaMemcpyHostToDevice, h->stream));
  }
  CK(cudaMemcpyAsync(h->tab13, table, (size_t)nmat * PHONO_TABLE_COLS * 8, cudaMemcpyHostToDevice, h->stream));
  CK(cudaStreamSynchronize(h->stream));
  h->nmat = nmat;
  abc_coeffs(h, table + (size_t)id000 * PHONO_TABLE_COLS, h->abc);
  return PHONO_OK;
}

template <class R>
static StepArgs<R> make_args(const phono_handle* h, const Tiling& t, int step_off) {
  StepArgs<R> a{};
  a.g = h->g;
  a.sp.fdx = (const R*)h->sp[0];
  a.sp.fdy = (const R*)h->sp[1];
  a.sp.fdz = (const R*)h->sp[2];
  a.sp.sdx = (const R*)h->sp[3];
  a.sp.sdy = (const R*)h->sp[4];
  a.sp.sdz = (const R*)h->sp[5];
  R s0[6];
  // the leapfrog divides by raw spacings; the velocity forms multiply by reciprocals
  const bool raw = h->d.precision == PHONO_F64;
  for (int q = 0; q < 6; q++) s0[q] = raw ? (R)h->h_sp0[q] : (R)(1.0 / h->h_sp0[q]);
  a.sp.fdx0 = s0[0];
  a.sp.fdy0 = s0[1];
  a.sp.fdz0 = s0[2];
  a.sp.sdx0 = s0[3];
  a.sp.sdy0 = s0[4];
  a.sp.sdz0 = s0[5];
  a.dtab = h->dtab;
  a.mat = h->mat;
  a.tab = (const R*)h->tab;
  a.src = h->src;
  a.tm_u = t.tm_u;
  a.tm_mat = t.tm_mat;
  a.tm_pw0 = t.tm_pw0;
  a.tm_pw1 = t.tm_pw1;
  a.nmat = h->nmat;
  a.ubase = (R*)h->ubase;
  a.vbase = (R*)h->vbase;
  a.cbase = (R*)h->cbase;
  for (int q = 0; q < 8; q++) a.abc[q] = (R)h->abc[q];
  a.dt = (R)h->d.dt;
  a.surf = (R*)h->surf;
  a.record_every = h->d.record_every;
  a.rec_base = 0;
  a.nrec_cap = h->nrec_cap;
  a.step_base = h->step_base;
  a.step_off = step_off;
  a.surface_mode = h->d.surface_mode;
  a.bc = h->d.bc;
  a.source_mode = h->d.source_mode;
  a.ntj = t.ntj;
  a.ntk = t.ntk;
  a.nseg = t.nseg;
  for (int q = 0; q <= SEG_TABLE && q < (int)t.seg_start.size(); q++) a.seg_start[q] = t.seg_start[q];
  a.xseg = t.xseg;
  a.n_tile_blocks = t.n_tile;
  a.faces = h->faces;
  a.err = h->err;
  a.step_end = 0x7fffffff;
  a.wait_polls = h->wait_polls;
  a.skip_plane = h->skip_plane;
  return a;
}

// Two-launch step: the stresses and the update of one chunk of planes after
// another (one chunk when the stress window holds the whole mesh).  A chunk's
// update reads the stresses from two planes behind it to one ahead.
template <class R, class D>
static cudaError_t split_step(const phono_handle* h, int step_off, int step_end, cudaStream_t st) {
  SplitArgs<R, D> a{};
  a.g = h->g;
  const D** sp[6] = {&a.fdx, &a.fdy, &a.fdz, &a.sdx, &a.sdy, &a.sdz};
  for (int q = 0; q < 6; q++) *sp[q] = (const D*)h->spd[q];
  a.mat = h->mat;
  a.tab = (const R*)h->tab;
  a.rec = h->rec;
  a.vals = h->vals;
  a.shared = h->shared;
  a.soft = (double)h->d.nx * h->d.ny * h->d.nz >= kSoftVelNodes;
  a.dtab = h->dtab;
  a.src = h->src;
  a.ubase = (R*)h->ubase;
  a.vbase = (R*)h->vbase;
  a.cbase = (R*)h->cbase;
  for (int q = 0; q < 8; q++) a.abc[q] = (R)h->abc[q];
  a.dt = (R)h->d.dt;
  a.surf = (R*)h->surf;
  a.record_every = h->d.record_every;
  a.nrec_cap = h->nrec_cap;
  a.step_base = h->step_base;
  a.step_off = step_off;
  a.step_end = step_end;
  a.surface_mode = h->d.surface_mode;
  a.bc = h->d.bc;
  a.source_mode = h->d.source_mode;
  a.err = h->err;
  const int nx = h->d.nx, ny = h->d.ny, nz = h->d.nz;
  a.W = h->win;
  if (h->stress) {  // leapfrog
    a.tsy = h->tsy;
    a.tsx = (unsigned)(ny * h->tsy);
    a.tcs = (long long)h->win * a.tsx;
    a.Ta = (R*)h->stress + SPLIT_KOFF;
    a.Tb = a.Ta + 3 * a.tcs;
  } else {  // velocity forms: the layout of the fields
    a.tsy = (int)h->g.sy;
    a.tsx = (unsigned)h->g.sx;
    a.tcs = h->g.fstride;
    a.Ta = a.vbase + 3 * a.tcs + h->g.o0;
    a.Tb = a.cbase + 3 * a.tcs + h->g.o0;
  }
  a.dz1 = fast_div(nz - 1);
  a.dy1 = fast_div(ny - 1);
  // points of each component on no face: nj rows (from 1), nk columns (from 0),
  // planes up to xn, the last of them and the outer rows and column next to a face
  int xn[3], nj[3], nk[3];
  for (int c = 0; c < 3; c++) {
    xn[c] = nx - 2 - (c == 0);
    nj[c] = ny - 2 - (c == 1);
    nk[c] = nz - 1 - (c == 2);
    a.uy_[c] = fast_div(std::max(nj[c] - 2, 1));
    a.uz_[c] = fast_div(std::max(nk[c] - 1, 1));
    a.per[c] = fast_div(std::min(nj[c], 2) * nk[c] + std::max(nj[c] - 2, 0));
    a.nk[c] = fast_div(nk[c]);
  }
  const int len = h->win >= nx ? nx : h->win - SPLIT_BEHIND;
  cudaError_t e = cudaSuccess;
  for (int p = 0, done = 0; p < nx && e == cudaSuccess; p += len) {
    a.pa = p;
    a.pb = std::min(p + len, nx);
    a.sa = done;
    a.sb = done = std::min(a.pb + 1, nx);
    for (int c = 0; c < 3; c++) {
      const int planes = std::max(0, std::min(a.pb, xn[c]) - p);
      a.off[c + 1] = a.off[c] + planes * a.per[c].d + (p <= xn[c] && xn[c] < a.pb ? nj[c] * nk[c] : 0);
    }
    for (int c = 0; c < 3; c++) {
      const int planes = std::max(0, std::min(a.pb, xn[c]) - p);
      a.off[c + 4] = a.off[c + 3] + planes * std::max(nj[c] - 2, 0) * (nk[c] - 1);
    }
    // the first launch of a chunk of steps waits for all before it
    e = launch_split(h->d.precision, &a, true, step_off > 0 || p > 0, st);
    if (e == cudaSuccess) e = launch_split(h->d.precision, &a, false, true, st);
  }
  return e;
}

static cudaError_t split_step_any(const phono_handle* h, int step_off, int step_end, cudaStream_t st) {
  if (h->d.precision == PHONO_F64) return split_step<double, SoftRec>(h, step_off, step_end, st);
  if (h->d.precision == PHONO_F64V) return split_step<double, SoftFactor>(h, step_off, step_end, st);
  return split_step<float, float>(h, step_off, step_end, st);
}

// one step of the tile pass, in a handle's own shape
static cudaError_t tile_step(const phono_handle* h, int step_off, int step_end, int form, cudaStream_t st) {
  const Tiling& t = h->own.tj ? h->own : h->t;
  if (h->d.precision == PHONO_F32K) {
    StepArgs<float> a = make_args<float>(h, t, step_off);
    a.step_end = step_end;
    return launch_step_f32k(a, t.tj, form, st);
  }
  StepArgs<double> a = make_args<double>(h, t, step_off);
  a.step_end = step_end;
  return h->d.precision == PHONO_F64 ? launch_step_f64(a, t.tj, form, st) : launch_step_f64v(a, t.tj, form, st);
}

// one time step (parts: the handle's form; or 2 tile launch only, 3 face launch only)
static cudaError_t launch_one(phono_handle* h, int step_off, int parts = -1) {
  if (h->split) return parts == 3 ? cudaSuccess : split_step_any(h, step_off, 0x7fffffff, h->stream);
  const int form = parts < 0 ? h->separate_faces : parts;
  return tile_step(h, step_off, 0x7fffffff, form, h->stream);
}

// Padded device layout: planes -1..nx, rows -1..ny, z rows with KPAD zeros
// behind them, rounded up to 128 bytes; material ids with an MKOFF front pad
// and 16-byte rows.
static long long field_row(int nz, int es) {
  return round_up((es == 8 ? Lay<double>::KPAD : Lay<float>::KPAD) + nz + 1, 128 / es);
}
static long long mat_row(int nz) { return round_up(MKOFF + nz + 1, 16); }

// Planes of the stress window of the two-launch step; 0: the mesh steps with
// the tile pass.
//  * FP64 (both schemes) is bound by the FP64 pipe: every mesh takes the
//    two-launch form (256x256x128 cells: 1.07 ms a step against 2.0 for the
//    best tile shape of the leapfrog, 0.84 against 1.17 for the velocity form).
//  * FP32 moves 60 more bytes a node than the tile pass, and wins only where
//    a launch is too short to fill its pipeline (us a step, two launches
//    against the default tiles: 7.5 / 10.1 at 78 k nodes, 9.2 / 9.7 at 139 k,
//    12.0 / 11.2 at 208 k, 16.2 / 12.8 at 310 k, 147 / 67 at 3.1 M).
// The velocity forms' stresses fit in the second buffers of v and the Kahan
// term.  The leapfrog's window is the whole mesh up to 128 MB, else the planes
// that fill 128 MB and at least 36: chunks cost a tail each (256x256x128: 1.08
// ms at 64 MB, 1.03 with all 463 MB), and the footprint should not grow by the
// six stresses of a large mesh.  With ny == 3 a face point can be the point
// another face's chain starts from (the tile pass's one-launch form has that).
constexpr long long kSplitF32Nodes = 170000;
static int split_window(int nx, int ny, int nz, int precision) {
  if (ny == 3) return 0;
  if (precision == PHONO_F32K && (long long)nx * ny * nz > kSplitF32Nodes) return 0;
  long long win = nx;
  if (precision == PHONO_F64)
    win = std::min(win, std::max<long long>((128LL << 20) / (6LL * ny * round_up(SPLIT_KOFF + nz, 8) * 8), 36));
  // flattened points of a launch are 31-bit
  return 3LL * win * ny * nz <= 0x7fff0000LL ? (int)win : 0;
}
// bytes of the leapfrog's window (the velocity forms need none)
static size_t split_bytes(int nx, int ny, int nz, int precision) {
  if (precision != PHONO_F64) return 0;
  return (size_t)6 * split_window(nx, ny, nz, precision) * ny * round_up(SPLIT_KOFF + nz, 8) * 8;
}

// One allocation holds what depends on the mesh alone: per axis the spacings
// as the kernels use them (with one value 1 before and two after, so that the
// tile pass reads the x spacings of its planes -1..nx without range tests;
// the padding only reaches values whose results are discarded), their FP64
// reciprocals (energy) and, for FP64, the records of the two-launch step (16 per
// material id first), for the leapfrog with their values and the divisor table.
struct ConstBlock {
  size_t sp[6], rsp[6], spd[6], div, rec, vals, bytes;
};
static ConstBlock const_block(int nx, int ny, int nz, int precision) {
  const int es = precision == PHONO_F32K ? 4 : 8;
  const int lens[6] = {nx - 1, ny - 1, nz - 1, nx - 2, ny - 2, nz - 2};
  ConstBlock c{};
  auto take = [&](size_t n) {
    const size_t at = c.bytes;
    c.bytes += (n + 511) / 512 * 512;
    return at;
  };
  for (int a = 0; a < 6; a++) c.sp[a] = take((size_t)(lens[a] + 3) * es);
  for (int a = 0; a < 6; a++) c.rsp[a] = take((size_t)lens[a] * 8);
  if (precision == PHONO_F64) {
    c.div = take(sizeof(double) * 4 * DIV_TABLE_SLOTS_MAX);
    size_t n = 256 * 16;
    for (int a = 0; a < 6; a++) {
      c.spd[a] = take((size_t)(lens[a] + 3) * sizeof(SoftRec));
      n += lens[a] + 1;
    }
    c.vals = take(n * 8);
  } else if (precision == PHONO_F64V) {
    for (int a = 0; a < 6; a++) c.spd[a] = take((size_t)(lens[a] + 3) * sizeof(SoftFactor));
  }
  if (es == 8) c.rec = take(256 * 16 * sizeof(SoftRec));
  return c;
}

// Bytes of device memory phono_create allocates for a handle (each cudaMalloc
// rounded up to 512 bytes).  shaped: it is made with a tile shape, and has no
// stress window.
static size_t handle_bytes(int nx, int ny, int nz, int precision, int max_steps, int record_every, bool shaped) {
  const int es = precision == PHONO_F32K ? 4 : 8;
  const int nbuf = precision == PHONO_F64 ? 3 : 2;
  auto r = [](size_t b) { return (b + 511) / 512 * 512; };
  const size_t field_elems = (size_t)(nx + 2) * (ny + 2) * field_row(nz, es);
  const size_t fb = field_elems * es * 3 * nbuf;
  size_t total = r(fb) * (precision == PHONO_F64 ? 1 : 3);
  total += r(const_block(nx, ny, nz, precision).bytes);
  total += r((size_t)(nx + 2) * (ny + 2) * mat_row(nz));
  total += r((size_t)256 * 16 * es) + r((size_t)256 * PHONO_TABLE_COLS * 8);
  const int cap = max_steps > 0 ? max_steps : 1;
  total += r((size_t)cap * 8);
  const int nrec = record_every > 0 ? max_steps / record_every : 0;
  if (nrec > 0) total += r((size_t)nrec * nx * ny * es);
  total += r(sizeof(int) * 2) + r(sizeof(double2) * kEnergyBlocks) + r(sizeof(double) * 2);
  if (!shaped) total += r(split_bytes(nx, ny, nz, precision));
  return total;
}

static int check_desc(const phono_desc* d) {
  if (!d) return fail(PHONO_ERR_ARG, "desc is NULL");
  if (d->nx < 3 || d->ny < 3 || d->nz < 3) return fail(PHONO_ERR_ARG, "nx, ny, nz must be >= 3 mesh nodes");
  if ((long long)d->nx * d->ny * d->nz > (1LL << 34)) return fail(PHONO_ERR_ARG, "grid too large");
  if (!d->fdx || !d->fdy || !d->fdz || !d->sdx || !d->sdy || !d->sdz) return fail(PHONO_ERR_ARG, "spacing array is NULL");
  if (!d->mat || !d->table) return fail(PHONO_ERR_ARG, "material ids or table is NULL");
  if (d->nmat < 1 || d->nmat > 256) return fail(PHONO_ERR_ARG, "nmat must be in 1..256");
  if (d->precision != PHONO_F64 && d->precision != PHONO_F32K && d->precision != PHONO_F64V)
    return fail(PHONO_ERR_ARG, "unknown precision");
  if (d->surface_mode < 0 || d->surface_mode > 1) return fail(PHONO_ERR_ARG, "unknown surface_mode");
  if (d->bc < 0 || d->bc > 1) return fail(PHONO_ERR_ARG, "unknown bc");
  if (d->source_mode < 0 || d->source_mode > 1) return fail(PHONO_ERR_ARG, "unknown source_mode");
  if (d->max_steps < 0 || d->record_every < 0) return fail(PHONO_ERR_ARG, "max_steps and record_every must be >= 0");
  if (!(d->dt > 0.0) || !std::isfinite(d->dt)) return fail(PHONO_ERR_ARG, "dt must be finite and > 0");
  if (d->tile_j != 0 && d->tile_j != 4 && d->tile_j != 8 && d->tile_j != 16) return fail(PHONO_ERR_ARG, "tile_j must be 0, 4, 8 or 16");
  if (d->x_segment < -4096) return fail(PHONO_ERR_ARG, "x_segment out of range");
  for (int q = 0; q < d->nmat * PHONO_TABLE_COLS; q++)
    if (!std::isfinite(d->table[q])) return fail(PHONO_ERR_ARG, "material table holds a non-finite value");
  for (int q = 0; q < d->nmat; q++)
    if (!(d->table[q * PHONO_TABLE_COLS + 12] > 0.0)) return fail(PHONO_ERR_ARG, "density must be > 0");
  const double* arrs[6] = {d->fdx, d->fdy, d->fdz, d->sdx, d->sdy, d->sdz};
  int lens[6] = {d->nx - 1, d->ny - 1, d->nz - 1, d->nx - 2, d->ny - 2, d->nz - 2};
  for (int a = 0; a < 6; a++)
    for (int q = 0; q < lens[a]; q++)
      if (!(arrs[a][q] > 0.0) || !std::isfinite(arrs[a][q])) return fail(PHONO_ERR_ARG, "spacings must be finite and > 0");
  size_t n = (size_t)d->nx * d->ny * d->nz;
  if (largest_id(d->mat, n) >= d->nmat) return fail(PHONO_ERR_ARG, "material id out of range");
  return PHONO_OK;
}

// fields from here on are read back into pinned memory by a kernel
constexpr size_t kReadbackBytes = 128 << 10;

// the device address of `bytes` bytes of pinned host memory at p; NULL where
// it is any other memory
static void* pinned_address(const void* p, size_t bytes) {
  cudaPointerAttributes a{}, z{};
  if (cudaPointerGetAttributes(&a, p) == cudaSuccess && a.type == cudaMemoryTypeHost && a.devicePointer &&
      cudaPointerGetAttributes(&z, (const char*)p + bytes - 1) == cudaSuccess && z.type == cudaMemoryTypeHost &&
      z.devicePointer == (char*)a.devicePointer + bytes - 1)
    return a.devicePointer;
  cudaGetLastError();
  return nullptr;
}

// 3-D copy between a dense host array (ex, ey, ez) and the padded device layout
static cudaError_t copy3d(phono_handle* h, void* dev, void* host, int c, bool to_dev) {
  int ex = h->d.nx - (c == 0), ey = h->d.ny - (c == 1), ez = h->d.nz - (c == 2);
  // pinned memory is written by a kernel (readback.cu); pageable memory, an
  // element off its own alignment and small fields take the strided copy (a run
  // of 6500 nodes FP64, 58 KB a field: 1284 us, 1309 with the kernel)
  const size_t bytes = (size_t)ex * ey * ez * h->es;
  if (!to_dev && bytes >= kReadbackBytes && (uintptr_t)host % h->es == 0) {
    const OnDevice here(h->dev);
    if (here.err != cudaSuccess) return here.err;
    if (void* to = pinned_address(host, bytes)) {
      cudaError_t e = launch_readback((char*)dev + h->g.o0 * h->es, h->g.sx, h->g.sy, ex, ey, ez, h->es, to, h->stream);
      return e == cudaSuccess ? cudaStreamSynchronize(h->stream) : e;
    }
  }
  cudaMemcpy3DParms p{};
  cudaPitchedPtr hp = make_cudaPitchedPtr(host, (size_t)ez * h->es, (size_t)ez * h->es, ey);
  cudaPitchedPtr dp = make_cudaPitchedPtr((char*)dev + h->g.o0 * h->es, (size_t)h->g.sy * h->es,
                                          (size_t)h->g.sy * h->es, h->d.ny + 2);
  p.extent = make_cudaExtent((size_t)ez * h->es, ey, ex);
  if (to_dev) {
    p.srcPtr = hp;
    p.dstPtr = dp;
    p.kind = cudaMemcpyHostToDevice;
  } else {
    p.srcPtr = dp;
    p.dstPtr = hp;
    p.kind = cudaMemcpyDeviceToHost;
  }
  cudaError_t e = cudaMemcpy3DAsync(&p, h->stream);
  if (e != cudaSuccess) return e;
  return cudaStreamSynchronize(h->stream);
}

// buffers holding the current state after steps_done steps
static void* arr(const phono_handle* h, char* base, int buf, int comp) {
  return base + (size_t)(buf * 3 + comp) * h->field_elems * h->es;
}

static void* field_ptr(phono_handle* h, int field) {
  int t = h->steps_done;
  int comp = field % 3;
  if (h->d.precision == PHONO_F64) {
    if (field <= PHONO_FIELD_UZ) return arr(h, h->ubase, (t + 1) % 3, comp);
    if (field <= PHONO_FIELD_UZ_OLD) return arr(h, h->ubase, t % 3, comp);
    return nullptr;
  }
  int b = t & 1;
  if (field <= PHONO_FIELD_UZ) return arr(h, h->ubase, b, comp);
  if (field <= PHONO_FIELD_UZ_OLD) return nullptr;
  if (h->split) b = 0;
  if (field <= PHONO_FIELD_VZ) return arr(h, h->vbase, b, comp);
  if (field <= PHONO_FIELD_CZ) return arr(h, h->cbase, b, comp);
  return nullptr;
}

// Switch a handle between the two-launch form (v and the Kahan term in buffer
// 0) and the tile pass (in the buffer of the step's parity).  On failure the
// handle keeps its form: what may have been copied is the state it does not use.
static cudaError_t set_split(phono_handle* h, bool on) {
  if (h->split == on) return cudaSuccess;
  cudaError_t e = cudaSuccess;
  if (h->vbase && (h->steps_done & 1)) {
    const size_t n = 3 * h->field_elems * h->es;
    for (char* b : {h->vbase, h->cbase})
      if (e == cudaSuccess)
        e = cudaMemcpyAsync(on ? b : b + n, on ? b + n : b, n, cudaMemcpyDeviceToDevice, h->stream);
  }
  if (e == cudaSuccess) h->split = on;
  return e;
}

// Tile decomposition of a handle: tile_j rows x 32 z-points per block, the
// x axis cut into segments of x_segment planes, and the face-pass work list.
// x_segment > 0: segments of x_segment planes (the last one shorter).
// x_segment = -L: tapered segments -- L planes while more than 2L planes are
// left, then the rest in four nearly equal parts -- so that the blocks a
// launch dispatches last are short and the tail of the last wave is short.
static std::vector<int> segment_starts(int planes, int xseg) {
  std::vector<int> st{0};
  if (xseg > 0) {
    for (int p = xseg; p < planes; p += xseg) st.push_back(p);
  } else {
    const int len = -xseg;
    int p = 0;
    while (planes - p > 2 * len) st.push_back(p += len);
    const int rem = planes - p, parts = rem >= 4 ? 4 : (rem > 0 ? rem : 0);
    for (int q = 1; q < parts; q++) st.push_back(p + (int)((long long)rem * q / parts));
  }
  st.push_back(planes);
  return st;
}

// h->xseg of a handle whose segments were given as a list (phono_set_segments)
constexpr int kExplicitSegments = INT_MIN;

// tile height tj and x segments starting at starts[0..n) (+ nx-1 at the end)
static int apply_tiling(phono_handle* h, Tiling& t, int tj, int xseg, const std::vector<int>& starts) {
  const int nx = h->d.nx, ny = h->d.ny, nz = h->d.nz;
  const int ntj = (ny - 1 + tj - 1) / tj, ntk = (nz - 1 + TK - 1) / TK, nseg = (int)starts.size() - 1;
  if (xseg <= 0 && nseg > SEG_TABLE) return fail(PHONO_ERR_ARG, "tapered or listed x segments: more than 64 segments");
  long long ntile = (long long)ntj * ntk * nseg;
  // face points left to the face pass, per component: z=N only where it meets
  // an x / y face (2*ex + ey-2; the tile pass writes the rest), y=N and y=0
  // (ex*(ez-1)), x=N ((ey-2)*(ez-1))
  FaceTable faces{};
  long long acc = 0;
  for (int c = 0; c < 3; c++) {
    long long ex = nx - (c == 0), ey = ny - (c == 1), ez = nz - (c == 2);
    long long cnt[4] = {2 * ex + (ey - 2), ex * (ez - 1), ex * (ez - 1), (ey - 2) * (ez - 1)};
    for (int p = 0; p < 4; p++) {
      faces.off[c * 4 + p] = (int)acc;
      acc += cnt[p];
    }
  }
  faces.off[12] = (int)acc;
  const long long nface = (acc + TK * tj - 1) / (TK * tj);
  if (ntile + nface > 0x7fffffffLL || acc > 0x7fffffffLL) return fail(PHONO_ERR_ARG, "grid too large for one launch");
  t.tj = tj;
  t.xseg = xseg;
  t.seg_start = starts;
  t.ntj = ntj;
  t.ntk = ntk;
  t.nseg = nseg;
  t.n_tile = (int)ntile;
  h->faces = faces;
  // faces in a second launch that reads the tile pass's interior values; the
  // chain end of a face point can itself be a face point only when ny == 3
  h->separate_faces = ny >= 4 ? 1 : 0;
  return PHONO_OK;
}

static int set_tiling(phono_handle* h, int tj, int xseg) {
  return apply_tiling(h, h->t, tj, xseg, segment_starts(h->d.nx - 1, xseg));
}

static int sm_count() {
  int dev = 0, nsm = 152;
  if (cudaGetDevice(&dev) == cudaSuccess) cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev);
  cudaGetLastError();
  return nsm;
}

// Segments that keep the resident blocks busy to the end: every wave of blocks
// takes segments of one length, the last the shortest, since blocks of equal
// length that share the memory bandwidth drift apart and leave it idle at the
// end.  For `depth` planes a block slot and at most `waves` waves; the lengths
// grow by 1/0.6 from the shortest up to 17 planes.
static std::vector<double> wave_lengths(double depth, int waves, double shortest) {
  std::vector<double> len{shortest};
  double sum = shortest;
  while ((int)len.size() < waves) {
    const double next = std::min(len.back() / 0.6, 17.0);
    if (sum + next > depth) break;
    len.push_back(next);
    sum += next;
  }
  for (double& l : len) l *= depth / sum;
  std::reverse(len.begin(), len.end());
  return len;
}

// A default FP32 handle's own tiles: the vectorised tile pass at height 16,
// which needs no face launch, or 8 where 16 rows waste more than half of
// the y extent (us a step at 8 / 16: 8 rows, 1399x8x16 cells 13.5 / 15.5; 24
// rows 23.9 / 23.5, 130 rows 25.6 / 22.4, 256 rows 124 / 118).  Segments: at least as many as fill one wave of resident
// blocks (3 an SM of height 16, 5 of height 8; 160x128x64 cells: 31 us with 448
// blocks of 456, 37 with 480); meshes of a few waves in lengths that fall from
// wave to wave (us a step, even segments before: 256x256x128 129 / 122,
// 329x199x149 146 / 138, 119x149x288 83 / 78, 193x161x97 63 / 61); where less
// than three segments fill a wave, even ones of about 12 planes (a segment
// reads two planes more than it updates; long ones let neighbouring blocks
// drift apart until their common halo rows have left L2: 512x512x256 cells 802
// us at 12 planes, 917 at 57). Beside other
// instances (a batch) there is no last wave to fill: even segments of at most
// `limit` planes (0: alone), see batch_rebuild.
static int own_tiling(phono_handle* h, Tiling& t, int limit) {
  const int nsm = sm_count();
  const int planes = h->d.nx - 1, rows = h->d.ny - 1;
  const long long r16 = round_up(rows, 16), r8 = round_up(rows, 8);
  const int tj = r16 > r8 + r8 / 2 ? 8 : 16;
  const long long tiles = (tj == 16 ? r16 : r8) / tj * ((h->d.nz - 1 + TK - 1) / TK), wave = (long long)nsm * (tj == 16 ? 3 : 5);
  std::vector<int> starts;
  auto even = [&](int nseg) {
    for (int q = 0; q <= nseg; q++) starts.push_back((int)((long long)planes * q / nseg));
  };
  const int fill = (int)std::min<long long>(wave / tiles, planes);  // segments that fill a wave
  if (limit) {
    even((planes + limit - 1) / limit);
  } else if (fill >= 3) {
    double at = 0;
    starts.push_back(0);
    for (double l : wave_lengths((double)planes / fill, SEG_TABLE / fill, tj == 16 ? 3.6 : 4.4))
      for (int q = 0; q < fill; q++) starts.push_back((int)std::lround(at += l));
    starts.back() = planes;
  } else {
    const long long want = tiles * ((planes + 11) / 12), waves = (want + wave - 1) / wave;
    even((int)std::min<long long>(std::max<long long>(waves * wave / tiles, 1), planes));
  }
  const int nseg = (int)starts.size() - 1;
  // more segments than a launch describes by table: even ones
  if (nseg > SEG_TABLE) return apply_tiling(h, t, tj, (planes + nseg - 1) / nseg, segment_starts(planes, (planes + nseg - 1) / nseg));
  return apply_tiling(h, t, tj, kExplicitSegments, starts);
}

// TMA descriptors: a 4-D (k, j, i, array) map over the u allocation with a
// (KW, TJ+2, 1, 3) box (one plane tile of the three components of a buffer)
// and a 3-D (k, j, i) map over the material ids with a (48, TJ+2, 1) box.
static int encode_tensor_maps(const phono_handle* h, Tiling& t) {
  static PFN_cuTensorMapEncodeTiled_v12000 encode = nullptr;
  if (!encode) {
    void* fn = nullptr;
    cudaDriverEntryPointQueryResult q;
    CK(cudaGetDriverEntryPointByVersion("cuTensorMapEncodeTiled", &fn, 12000, cudaEnableDefault, &q));
    if (q != cudaDriverEntryPointSuccess || !fn) return fail(PHONO_ERR_CUDA, "cuTensorMapEncodeTiled not available");
    encode = (PFN_cuTensorMapEncodeTiled_v12000)fn;
  }
  const int es = h->es;
  const int kw = es == 8 ? Lay<double>::KW : Lay<float>::KW;
  cuuint64_t dims[4] = {(cuuint64_t)h->g.sy, (cuuint64_t)(h->d.ny + 2), (cuuint64_t)(h->d.nx + 2),
                        (cuuint64_t)(h->nbuf * 3)};
  cuuint64_t strides[3] = {(cuuint64_t)h->g.sy * es, (cuuint64_t)h->g.sx * es, (cuuint64_t)h->field_elems * es};
  cuuint32_t box[4] = {(cuuint32_t)kw, (cuuint32_t)(t.tj + 2), 1, 3};
  cuuint32_t estr[4] = {1, 1, 1, 1};
  CUresult r = encode(&t.tm_u, es == 8 ? CU_TENSOR_MAP_DATA_TYPE_FLOAT64 : CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 4,
                      h->ubase, dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_NONE,
                      CU_TENSOR_MAP_L2_PROMOTION_L2_128B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  if (r != CUDA_SUCCESS) return fail(PHONO_ERR_CUDA, "cuTensorMapEncodeTiled (fields) failed: " + std::to_string(r));
  cuuint64_t mdims[3] = {(cuuint64_t)h->g.msy, (cuuint64_t)(h->d.ny + 2), (cuuint64_t)(h->d.nx + 2)};
  cuuint64_t mstr[2] = {(cuuint64_t)h->g.msy, (cuuint64_t)h->g.msx};
  cuuint32_t mbox[3] = {(cuuint32_t)MKW, (cuuint32_t)(t.tj + 2), 1};
  r = encode(&t.tm_mat, CU_TENSOR_MAP_DATA_TYPE_UINT8, 3, h->mat, mdims, mstr, mbox, estr,
             CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_L2_128B,
             CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  if (r != CUDA_SUCCESS) return fail(PHONO_ERR_CUDA, "cuTensorMapEncodeTiled (materials) failed: " + std::to_string(r));
  // pointwise state, own points only: a (32, TJ, 1, 3) box over u_old (F64)
  // or over v and the Kahan terms (velocity forms)
  cuuint32_t pbox[4] = {(cuuint32_t)TK, (cuuint32_t)t.tj, 1, 3};
  const bool f64 = h->d.precision == PHONO_F64;
  void* pw[2] = {f64 ? h->ubase : h->vbase, f64 ? h->ubase : h->cbase};
  CUtensorMap* maps[2] = {&t.tm_pw0, &t.tm_pw1};
  for (int q = 0; q < 2; q++) {
    r = encode(maps[q], es == 8 ? CU_TENSOR_MAP_DATA_TYPE_FLOAT64 : CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 4, pw[q], dims,
               strides, pbox, estr, CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_NONE,
               CU_TENSOR_MAP_L2_PROMOTION_L2_128B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    if (r != CUDA_SUCCESS) return fail(PHONO_ERR_CUDA, "cuTensorMapEncodeTiled (pointwise) failed: " + std::to_string(r));
  }
  return PHONO_OK;
}

extern "C" {

int phono_abi_version(void) { return PHONO_ABI_VERSION; }

int phono_footprint_shaped(int nx, int ny, int nz, int precision, int max_steps, int record_every, int tile_j, int x_segment,
                           size_t* bytes) {
  if (!bytes) return fail(PHONO_ERR_ARG, "bytes is NULL");
  if (nx < 3 || ny < 3 || nz < 3) return fail(PHONO_ERR_ARG, "nx, ny, nz must be >= 3 mesh nodes");
  if ((long long)nx * ny * nz > (1LL << 34)) return fail(PHONO_ERR_ARG, "grid too large");
  if (precision != PHONO_F64 && precision != PHONO_F32K && precision != PHONO_F64V)
    return fail(PHONO_ERR_ARG, "unknown precision");
  if (max_steps < 0 || record_every < 0) return fail(PHONO_ERR_ARG, "max_steps and record_every must be >= 0");
  *bytes = handle_bytes(nx, ny, nz, precision, max_steps, record_every, tile_j || x_segment);
  return PHONO_OK;
}

int phono_footprint(int nx, int ny, int nz, int precision, int max_steps, int record_every, size_t* bytes) {
  return phono_footprint_shaped(nx, ny, nz, precision, max_steps, record_every, 0, 0, bytes);
}

const char* phono_last_error(void) { return g_err.c_str(); }

int phono_create(const phono_desc* d, phono_handle** out) {
  if (!out) return fail(PHONO_ERR_ARG, "out is NULL");
  *out = nullptr;
  int rc = check_desc(d);
  if (rc) return rc;
  phono_handle* h = new phono_handle();
  h->d = *d;
  h->d.fdx = h->d.fdy = h->d.fdz = h->d.sdx = h->d.sdy = h->d.sdz = nullptr;
  h->d.mat = nullptr;
  h->d.table = nullptr;
  const bool f64 = d->precision == PHONO_F64;  // leapfrog state (u_old, u, u_new)
  h->es = d->precision == PHONO_F32K ? 4 : 8;
  const int nx = d->nx, ny = d->ny, nz = d->nz;
  // padded layout: planes -1..nx, rows -1..ny
  const long long pz = field_row(nz, h->es);
  h->nbuf = f64 ? 3 : 2;
  h->g.nx = nx;
  h->g.ny = ny;
  h->g.nz = nz;
  h->g.sy = pz;
  h->g.sx = (long long)(ny + 2) * pz;
  h->g.o0 = h->g.sx + h->g.sy;
  h->field_elems = (size_t)(nx + 2) * h->g.sx;
  if (h->field_elems >= (1ull << 32)) {  // the tile pass addresses an array with 32-bit offsets
    delete h;
    return fail(PHONO_ERR_ARG, "grid too large: one padded array exceeds 2^32 elements");
  }
  h->g.fstride = (long long)h->field_elems;
  const long long mpz = mat_row(nz);
  h->g.msy = mpz;
  h->g.msx = (long long)(ny + 2) * mpz;
  h->g.mo0 = h->g.msx + h->g.msy + MKOFF;
  h->mat_bytes = (size_t)(nx + 2) * h->g.msx;

  // tiles: the shape the caller knows by default is height 4 for FP32, 8 for
  // FP64, and 24 planes per segment
  int rt = set_tiling(h, d->tile_j ? d->tile_j : (d->precision == PHONO_F32K ? 4 : 8), d->x_segment ? d->x_segment : 24);
  if (!rt && d->precision == PHONO_F32K && !d->tile_j && !d->x_segment) rt = own_tiling(h, h->own, 0);
  if (rt) {
    std::string m_ = g_err;
    delete h;
    g_err = m_;
    return PHONO_ERR_ARG;
  }

  cudaError_t e = cudaGetDevice(&h->dev);
  if (e == cudaSuccess) e = cudaStreamCreateWithFlags(&h->stream, cudaStreamNonBlocking);
  if (e != cudaSuccess) {
    delete h;
    return fail(PHONO_ERR_CUDA, std::string("cudaStreamCreate: ") + cudaGetErrorString(e));
  }
#define TRY(x)            \
  do {                    \
    int r_ = (x);         \
    if (r_) {             \
      std::string m_ = g_err; \
      release(h);         \
      g_err = m_;         \
      return r_;          \
    }                     \
  } while (0)
#define TRYC(x)                                                                         \
  do {                                                                                  \
    cudaError_t e_ = (x);                                                               \
    if (e_ != cudaSuccess) {                                                            \
      release(h);                                                                       \
      return fail(PHONO_ERR_CUDA, std::string(#x) + ": " + cudaGetErrorString(e_));     \
    }                                                                                   \
  } while (0)
  TRYC(f64 ? configure_step_f64(h->t.tj)
           : (d->precision == PHONO_F64V ? configure_step_f64v(h->t.tj) : configure_step_f32k(h->t.tj)));
  if (h->own.tj) TRYC(configure_step_f32k(h->own.tj));
  TRYC(cudaEventCreate(&h->ev0));
  TRYC(cudaEventCreate(&h->ev1));
  const size_t fb = h->field_elems * h->es * 3 * h->nbuf;
  TRY(dalloc(h, (void**)&h->ubase, fb));
  TRYC(cudaMemsetAsync(h->ubase, 0, fb, h->stream));
  if (!f64) {
    TRY(dalloc(h, (void**)&h->vbase, fb));
    TRY(dalloc(h, (void**)&h->cbase, fb));
    TRYC(cudaMemsetAsync(h->vbase, 0, fb, h->stream));
    TRYC(cudaMemsetAsync(h->cbase, 0, fb, h->stream));
  }

  // spacings and what derives from them, in one allocation and one copy
  const double* arrs[6] = {d->fdx, d->fdy, d->fdz, d->sdx, d->sdy, d->sdz};
  int lens[6] = {nx - 1, ny - 1, nz - 1, nx - 2, ny - 2, nz - 2};
  {
    const ConstBlock cb = const_block(nx, ny, nz, d->precision);
    std::vector<char> host(cb.bytes, 0);
    char* dev = nullptr;
    TRY(dalloc(h, (void**)&dev, cb.bytes));
    std::vector<double> divisors{1.0};
    uint32_t nval = 256 * 16;  // the table's values come first (upload_table)
    double* vals = f64 ? (double*)(host.data() + cb.vals) : nullptr;
    for (int a = 0; a < 6; a++) {
      h->h_sp0[a] = arrs[a][0];
      h->sp_host[a].assign(arrs[a], arrs[a] + lens[a]);
      h->sp[a] = dev + cb.sp[a] + h->es;
      const bool f64v = d->precision == PHONO_F64V;
      h->spd[a] = f64 ? (void*)((SoftRec*)(dev + cb.spd[a]) + 1) : f64v ? (void*)((SoftFactor*)(dev + cb.spd[a]) + 1) : h->sp[a];
      h->rsp64[a] = (double*)(dev + cb.rsp[a]);
      SoftRec* rec = (SoftRec*)(host.data() + cb.spd[a]);
      const uint32_t one = nval;  // the padding's divisor
      if (f64) vals[nval++] = 1.0;
      for (int q = -1; q < lens[a] + 2; q++) {
        const bool in = q >= 0 && q < lens[a];
        const double v = in ? arrs[a][q] : 1.0;
        // F64: raw spacings; the velocity forms: reciprocals
        if (h->es == 4) ((float*)(host.data() + cb.sp[a]))[q + 1] = (float)(1.0 / v);
        else ((double*)(host.data() + cb.sp[a]))[q + 1] = f64 ? v : 1.0 / v;
        if (in) ((double*)(host.data() + cb.rsp[a]))[q] = 1.0 / v;
        if (f64) {
          rec[q + 1] = soft_record(v, true, in ? nval : one);
          if (in) vals[nval++] = v;
        }
        if (f64v) ((SoftFactor*)rec)[q + 1] = SoftFactor{soft_record(1.0 / v, false, 0), 1.0 / v, 0.0};
      }
      divisors.insert(divisors.end(), arrs[a], arrs[a] + lens[a]);
    }
    if (h->es == 8) h->rec = (SoftRec*)(dev + cb.rec);
    if (f64) {
      h->vals = (double*)(dev + cb.vals);
      // divisor table (div_tab in div_table.cuh) over the distinct spacing
      // values and 1.0, the divisors the step uses
      std::vector<double> tbl;
      if (build_div_table(divisors, tbl, &h->dtab.mult, &h->dtab.shift)) {
        std::memcpy(host.data() + cb.div, tbl.data(), tbl.size() * sizeof(double));
        h->dtab.tab = (const double*)(dev + cb.div);
      }
    }
    TRYC(cudaMemcpy(dev, host.data(), host.size(), cudaMemcpyHostToDevice));
  }
  // materials: padded id layout and the 16-entry device rows (capacity 256 ids)
  TRY(dalloc(h, (void**)&h->mat, h->mat_bytes));
  TRYC(cudaMemsetAsync(h->mat, 0, h->mat_bytes, h->stream));
  join_stage(h);
  TRY(dalloc(h, &h->tab, (size_t)256 * 16 * h->es));
  // two-launch step (a handle made with a tile shape never takes it); the
  // leapfrog's window is zero outside the points the stress pass writes, and a
  // mesh whose window does not fit keeps to the tiles.  (Made after the rest, small
  // windows lie where the steps take 1% longer.)
  const bool shaped = d->tile_j || d->x_segment;
  h->win = shaped ? 0 : split_window(nx, ny, nz, d->precision);
  if (const size_t sb = shaped ? 0 : split_bytes(nx, ny, nz, d->precision)) {
    h->tsy = (int)round_up(SPLIT_KOFF + nz, 8);
    if (dalloc(h, (void**)&h->stress, sb)) {
      h->win = 0;
      cudaGetLastError();
      g_err.clear();
    } else {
      TRYC(cudaMemsetAsync(h->stress, 0, sb, h->stream));
    }
  }
  h->split = h->win > 0;
  TRY(dalloc(h, (void**)&h->tab13, (size_t)256 * PHONO_TABLE_COLS * 8));
  TRY(upload_materials(h, d->mat, d->table, d->nmat));
  TRY(encode_tensor_maps(h, h->t));
  if (h->own.tj) TRY(encode_tensor_maps(h, h->own));
  // source table, surface records, counters
  int cap = d->max_steps > 0 ? d->max_steps : 1;
  TRY(dalloc(h, (void**)&h->src, (size_t)cap * 8));
  TRYC(cudaMemsetAsync(h->src, 0, (size_t)cap * 8, h->stream));
  h->nrec_cap = d->record_every > 0 ? d->max_steps / d->record_every : 0;
  if (h->nrec_cap > 0) {
    size_t sb = (size_t)h->nrec_cap * nx * ny * h->es;
    TRY(dalloc(h, &h->surf, sb));
    TRYC(cudaMemsetAsync(h->surf, 0, sb, h->stream));
  }
  TRY(dalloc(h, (void**)&h->step_base, sizeof(int) * 2));
  h->err = h->step_base + 1;
  TRYC(cudaMemsetAsync(h->step_base, 0, sizeof(int) * 2, h->stream));
  TRY(dalloc(h, (void**)&h->partial, sizeof(double2) * kEnergyBlocks));
  TRY(dalloc(h, (void**)&h->energy_out, sizeof(double) * 2));
  TRYC(cudaStreamSynchronize(h->stream));
#undef TRY
#undef TRYC
  *out = h;
  return PHONO_OK;
}

int phono_set_source(phono_handle* h, const double* samples, int n) {
  if (!h || (!samples && n > 0)) return fail(PHONO_ERR_ARG, "NULL argument");
  if (n < 0 || n > (h->d.max_steps > 0 ? h->d.max_steps : 1)) return fail(PHONO_ERR_ARG, "n exceeds max_steps");
  for (int q = 0; q < n; q++)
    if (!std::isfinite(samples[q])) return fail(PHONO_ERR_ARG, "source sample is not finite");
  CK(cudaMemcpyAsync(h->src, samples, (size_t)n * 8, cudaMemcpyHostToDevice, h->stream));
  CK(cudaStreamSynchronize(h->stream));
  h->nsrc = n;
  return PHONO_OK;
}

static int build_graph(phono_handle* h) {
  cudaGraph_t g = nullptr;
  CK(cudaStreamBeginCapture(h->stream, cudaStreamCaptureModeThreadLocal));
  cudaError_t e = cudaSuccess;
  for (int s = 0; s < kGraphSteps && e == cudaSuccess; s++) e = launch_one(h, s);
  if (e == cudaSuccess) {
    advance_step_kernel<<<1, 1, 0, h->stream>>>(h->step_base, kGraphSteps);
    e = cudaGetLastError();
  }
  cudaError_t e2 = cudaStreamEndCapture(h->stream, &g);
  if (e != cudaSuccess) {
    if (g) cudaGraphDestroy(g);
    return fail(PHONO_ERR_CUDA, std::string("graph capture: ") + cudaGetErrorString(e));
  }
  if (e2 != cudaSuccess) return fail(PHONO_ERR_CUDA, std::string("cudaStreamEndCapture: ") + cudaGetErrorString(e2));
  e = cudaGraphInstantiate(&h->graph, g, 0);
  cudaGraphDestroy(g);
  if (e != cudaSuccess) return fail(PHONO_ERR_CUDA, std::string("cudaGraphInstantiate: ") + cudaGetErrorString(e));
  return PHONO_OK;
}

int phono_step(phono_handle* h, int nsteps) {
  if (!h) return fail(PHONO_ERR_ARG, "handle is NULL");
  if (h->batch) return fail(PHONO_ERR_STATE, "handle is in a batch: step it with phono_batch_step");
  if (nsteps < 0) return fail(PHONO_ERR_ARG, "nsteps < 0");
  if (h->steps_done + nsteps > h->nsrc)
    return fail(PHONO_ERR_STATE, "not enough source samples: call phono_set_source with max_steps samples");
  if (nsteps == 0) return PHONO_OK;
  if (!h->graph && nsteps >= kGraphSteps) {
    int rc = build_graph(h);
    if (rc) return rc;
  }
  CK(cudaEventRecord(h->ev0, h->stream));
  int full = nsteps / kGraphSteps, rem = nsteps % kGraphSteps;
  for (int q = 0; q < full; q++) CK(cudaGraphLaunch(h->graph, h->stream));
  for (int s = 0; s < rem; s++) CK(launch_one(h, s));
  if (rem) {
    advance_step_kernel<<<1, 1, 0, h->stream>>>(h->step_base, rem);
    CK(cudaGetLastError());
  }
  CK(cudaEventRecord(h->ev1, h->stream));
  h->timed = true;
  h->steps_done += nsteps;
  return PHONO_OK;
}

int phono_time_kernels(phono_handle* h, int nsteps, float* tile_ms, float* face_ms) {
  if (!h || !tile_ms || !face_ms) return fail(PHONO_ERR_ARG, "NULL argument");
  if (h->batch) return fail(PHONO_ERR_STATE, "handle is in a batch");
  if (nsteps < 1) return fail(PHONO_ERR_ARG, "nsteps must be >= 1");
  if (h->steps_done + nsteps > h->nsrc)
    return fail(PHONO_ERR_STATE, "not enough source samples: call phono_set_source with max_steps samples");
  const bool sep = h->separate_faces != 0;
  std::vector<cudaEvent_t> ev(3 * (size_t)nsteps, nullptr);
  cudaError_t e = cudaSuccess;
  for (size_t q = 0; q < ev.size() && e == cudaSuccess; q++) e = cudaEventCreate(&ev[q]);
  for (int s = 0; s < nsteps && e == cudaSuccess; s++) {
    e = cudaEventRecord(ev[3 * s], h->stream);
    if (e == cudaSuccess) e = launch_one(h, s, sep ? 2 : 0);
    if (e == cudaSuccess) e = cudaEventRecord(ev[3 * s + 1], h->stream);
    if (e == cudaSuccess && sep) e = launch_one(h, s, 3);
    if (e == cudaSuccess) e = cudaEventRecord(ev[3 * s + 2], h->stream);
  }
  if (e == cudaSuccess) {
    advance_step_kernel<<<1, 1, 0, h->stream>>>(h->step_base, nsteps);
    e = cudaGetLastError();
  }
  if (e == cudaSuccess) e = cudaStreamSynchronize(h->stream);
  float t = 0.f, f = 0.f;
  for (int s = 0; s < nsteps && e == cudaSuccess; s++) {
    float a = 0.f, b = 0.f;
    e = cudaEventElapsedTime(&a, ev[3 * s], ev[3 * s + 1]);
    if (e == cudaSuccess) e = cudaEventElapsedTime(&b, ev[3 * s + 1], ev[3 * s + 2]);
    t += a;
    f += b;
  }
  for (cudaEvent_t x : ev)
    if (x) cudaEventDestroy(x);
  if (e != cudaSuccess) return fail(PHONO_ERR_CUDA, std::string("phono_time_kernels: ") + cudaGetErrorString(e));
  h->steps_done += nsteps;
  *tile_ms = t;
  *face_ms = f;
  return PHONO_OK;
}

int phono_steps_done(const phono_handle* h) { return h ? h->steps_done : fail(PHONO_ERR_ARG, "handle is NULL"); }

// the device error word of a handle: bit 2 a tile-pass wait ran out, bit 1 a
// non-finite surface value
static int device_error(int err) {
  if (err & 2) return fail(PHONO_ERR_TIMEOUT, "a tile-pass pipeline wait ran out; the state of that step is invalid");
  if (err & 1) return fail(PHONO_ERR_NUMERIC, "non-finite value in the recorded surface");
  return PHONO_OK;
}

int phono_sync(phono_handle* h) {
  if (!h) return fail(PHONO_ERR_ARG, "handle is NULL");
  CK(cudaStreamSynchronize(h->stream));
  int err = 0;
  CK(cudaMemcpy(&err, h->err, sizeof(int), cudaMemcpyDeviceToHost));
  return device_error(err);
}

int phono_test_wait_timeout(phono_handle* h, int polls, int skip_plane) {
  if (!h) return fail(PHONO_ERR_ARG, "handle is NULL");
  if (h->batch) return fail(PHONO_ERR_STATE, "handle is in a batch");
  if (polls < 0 || skip_plane < -1 || skip_plane > h->d.nx) return fail(PHONO_ERR_ARG, "polls >= 0, skip_plane in -1..nx");
  CK(cudaStreamSynchronize(h->stream));
  if (polls || skip_plane >= 0) CK(set_split(h, false));  // the two-launch form waits for nothing
  h->wait_polls = polls;
  h->skip_plane = skip_plane;
  if (h->graph) {  // the hook is a kernel argument baked into the graph
    cudaGraphExecDestroy(h->graph);
    h->graph = nullptr;
  }
  return PHONO_OK;
}

int phono_last_step_ms(phono_handle* h, float* ms) {
  if (!h || !ms) return fail(PHONO_ERR_ARG, "NULL argument");
  if (!h->timed) return fail(PHONO_ERR_STATE, "no step timed yet");
  CK(cudaEventSynchronize(h->ev1));
  CK(cudaEventElapsedTime(ms, h->ev0, h->ev1));
  return PHONO_OK;
}

int phono_read_surface(phono_handle* h, int first, int count, void* host_out) {
  if (!h || (!host_out && count > 0)) return fail(PHONO_ERR_ARG, "NULL argument");
  if (first < 0 || count < 0 || first + count > h->nrec_cap) return fail(PHONO_ERR_ARG, "record range out of bounds");
  if (count == 0) return PHONO_OK;
  size_t rec = (size_t)h->d.nx * h->d.ny * h->es;
  CK(cudaMemcpyAsync(host_out, (char*)h->surf + (size_t)first * rec, (size_t)count * rec, cudaMemcpyDeviceToHost,
                     h->stream));
  CK(cudaStreamSynchronize(h->stream));
  return PHONO_OK;
}

int phono_set_steps_done(phono_handle* h, int steps) {
  if (!h) return fail(PHONO_ERR_ARG, "handle is NULL");
  if (h->batch) return fail(PHONO_ERR_STATE, "handle is in a batch");
  if (steps < 0 || steps > h->nsrc) return fail(PHONO_ERR_ARG, "steps must be in 0..(source samples set)");
  CK(cudaStreamSynchronize(h->stream));
  CK(cudaMemcpy(h->step_base, &steps, sizeof(int), cudaMemcpyHostToDevice));
  h->steps_done = steps;
  return PHONO_OK;
}

int phono_upload_surface(phono_handle* h, int first, int count, const void* host_in) {
  if (!h || (!host_in && count > 0)) return fail(PHONO_ERR_ARG, "NULL argument");
  if (h->batch) return fail(PHONO_ERR_STATE, "handle is in a batch");
  if (first < 0 || count < 0 || first + count > h->nrec_cap) return fail(PHONO_ERR_ARG, "record range out of bounds");
  if (count == 0) return PHONO_OK;
  size_t rec = (size_t)h->d.nx * h->d.ny * h->es;
  CK(cudaMemcpyAsync((char*)h->surf + (size_t)first * rec, host_in, (size_t)count * rec, cudaMemcpyHostToDevice,
                     h->stream));
  CK(cudaStreamSynchronize(h->stream));
  return PHONO_OK;
}

static int field_check(phono_handle* h, int field, const void* host, size_t bytes, void** dev) {
  if (!h || !host) return fail(PHONO_ERR_ARG, "NULL argument");
  if (field < 0 || field > PHONO_FIELD_CZ) return fail(PHONO_ERR_ARG, "unknown field");
  *dev = field_ptr(h, field);
  if (!*dev) return fail(PHONO_ERR_ARG, "field not held by this precision");
  int c = field % 3;
  size_t n = (size_t)(h->d.nx - (c == 0)) * (h->d.ny - (c == 1)) * (h->d.nz - (c == 2));
  if (bytes != n * h->es) return fail(PHONO_ERR_ARG, "byte count does not match the field shape");
  return PHONO_OK;
}

int phono_download(phono_handle* h, int field, void* host, size_t bytes) {
  void* dev;
  int rc = field_check(h, field, host, bytes, &dev);
  if (rc) return rc;
  CK(cudaStreamSynchronize(h->stream));
  CK(copy3d(h, dev, host, field % 3, false));
  return PHONO_OK;
}

int phono_upload(phono_handle* h, int field, const void* host, size_t bytes) {
  if (h && h->batch) return fail(PHONO_ERR_STATE, "handle is in a batch");
  void* dev;
  int rc = field_check(h, field, host, bytes, &dev);
  if (rc) return rc;
  CK(cudaStreamSynchronize(h->stream));
  CK(copy3d(h, dev, (void*)host, field % 3, true));
  return PHONO_OK;
}

int phono_elem_size(const phono_handle* h) { return h ? h->es : fail(PHONO_ERR_ARG, "handle is NULL"); }

int phono_energy(phono_handle* h, double out[2]) {
  if (!h || !out) return fail(PHONO_ERR_ARG, "NULL argument");
  EnergyArgs a{};
  a.g = h->g;
  a.ux = field_ptr(h, PHONO_FIELD_UX);
  a.uy = field_ptr(h, PHONO_FIELD_UY);
  a.uz = field_ptr(h, PHONO_FIELD_UZ);
  const bool f64 = h->d.precision == PHONO_F64;
  a.vx = field_ptr(h, f64 ? PHONO_FIELD_UX_OLD : PHONO_FIELD_VX);
  a.vy = field_ptr(h, f64 ? PHONO_FIELD_UY_OLD : PHONO_FIELD_VY);
  a.vz = field_ptr(h, f64 ? PHONO_FIELD_UZ_OLD : PHONO_FIELD_VZ);
  a.f32 = h->es == 4 ? 1 : 0;
  a.vgiven = f64 ? 0 : 1;
  a.inv_dt = 1.0 / h->d.dt;
  a.rfdx = h->rsp64[0];
  a.rfdy = h->rsp64[1];
  a.rfdz = h->rsp64[2];
  a.rsdx = h->rsp64[3];
  a.rsdy = h->rsp64[4];
  a.rsdz = h->rsp64[5];
  a.mat = h->mat;
  a.tab = h->tab13;
  a.nmat = h->nmat;
  const bool march = h->es == 4 && (double)h->d.nx * h->d.ny * h->d.nz >= kEnergyMarchNodes;
  CK(launch_energy(a, h->partial, kEnergyBlocks, h->energy_out, march ? 2 * sm_count() : 0, h->stream));
  CK(cudaMemcpyAsync(out, h->energy_out, sizeof(double) * 2, cudaMemcpyDeviceToHost, h->stream));
  CK(cudaStreamSynchronize(h->stream));
  return PHONO_OK;
}

int phono_reset(phono_handle* h) {
  if (!h) return fail(PHONO_ERR_ARG, "handle is NULL");
  if (h->batch) return fail(PHONO_ERR_STATE, "handle is in a batch");
  const size_t fb = h->field_elems * h->es * 3 * h->nbuf;
  CK(cudaMemsetAsync(h->ubase, 0, fb, h->stream));
  if (h->vbase) CK(cudaMemsetAsync(h->vbase, 0, fb, h->stream));
  if (h->cbase) CK(cudaMemsetAsync(h->cbase, 0, fb, h->stream));
  if (h->surf) CK(cudaMemsetAsync(h->surf, 0, (size_t)h->nrec_cap * h->d.nx * h->d.ny * h->es, h->stream));
  CK(cudaMemsetAsync(h->step_base, 0, sizeof(int) * 2, h->stream));
  h->steps_done = 0;
  return PHONO_OK;
}

int phono_set_materials(phono_handle* h, const uint8_t* mat, const double* table, int nmat) {
  if (!h) return fail(PHONO_ERR_ARG, "handle is NULL");
  if (h->batch) return fail(PHONO_ERR_STATE, "handle is in a batch");
  int rc = check_materials(h, mat, table, nmat);
  if (rc) return rc;
  rc = upload_materials(h, mat, table, nmat);
  if (rc) return rc;
  // the absorbing-face coefficients are kernel arguments baked into the graph
  if (h->graph) {
    CK(cudaStreamSynchronize(h->stream));
    cudaGraphExecDestroy(h->graph);
    h->graph = nullptr;
  }
  return PHONO_OK;
}

int phono_set_lattice(phono_handle* h, const phono_lattice* lat, const double* table, int nmat) {
  if (!h || !lat || !table || !lat->radius || !lat->kind) return fail(PHONO_ERR_ARG, "NULL argument");
  if (h->batch) return fail(PHONO_ERR_STATE, "handle is in a batch");
  if (nmat < 1 || nmat > 256) return fail(PHONO_ERR_ARG, "nmat must be in 1..256");
  if (lat->pitch < 1 || lat->ncx < 1 || lat->ncy < 1) return fail(PHONO_ERR_ARG, "pitch and cell counts must be >= 1");
  if (lat->host < 0 || lat->host >= nmat) return fail(PHONO_ERR_ARG, "host material id out of range");
  const int ncell = lat->ncx * lat->ncy;
  for (int q = 0; q < ncell; q++) {
    if (lat->kind[q] >= nmat) return fail(PHONO_ERR_ARG, "hole material id out of range");
    if (!(lat->radius[q] >= 0.0) || !std::isfinite(lat->radius[q])) return fail(PHONO_ERR_ARG, "radius must be finite and >= 0");
  }
  for (int q = 0; q < nmat * PHONO_TABLE_COLS; q++)
    if (!std::isfinite(table[q])) return fail(PHONO_ERR_ARG, "material table holds a non-finite value");
  for (int q = 0; q < nmat; q++)
    if (!(table[q * PHONO_TABLE_COLS + 12] > 0.0)) return fail(PHONO_ERR_ARG, "density must be > 0");
  CK(cudaStreamSynchronize(h->stream));
  double* d_r = nullptr;
  uint8_t* d_k = nullptr;
  CK(cudaMalloc(&d_r, sizeof(double) * ncell));
  cudaError_t e = cudaMalloc(&d_k, ncell);
  if (e == cudaSuccess) e = cudaMemcpy(d_r, lat->radius, sizeof(double) * ncell, cudaMemcpyHostToDevice);
  if (e == cudaSuccess) e = cudaMemcpy(d_k, lat->kind, ncell, cudaMemcpyHostToDevice);
  if (e == cudaSuccess) e = launch_lattice_ids(h->mat, h->g, lat->pitch, lat->ncx, lat->ncy, d_r, d_k, lat->depth,
                                               (uint8_t)lat->host, h->stream);
  if (e == cudaSuccess) e = cudaStreamSynchronize(h->stream);
  cudaFree(d_r);
  cudaFree(d_k);
  if (e != cudaSuccess) return fail(PHONO_ERR_CUDA, std::string("lattice ids: ") + cudaGetErrorString(e));
  // node (0, 0, 0): inside the hole of cell (0, 0) only if its radius exceeds
  // the distance to the cell centre (the same test as the kernel's)
  const double c0 = 0.5 * lat->pitch, r0 = lat->radius[0];
  const int id000 = (c0 * c0 + c0 * c0 < r0 * r0 && lat->depth >= 0) ? lat->kind[0] : lat->host;
  int rc = upload_table(h, table, nmat, id000);
  if (rc) return rc;
  if (h->graph) {  // the absorbing-face coefficients are kernel arguments baked into the graph
    CK(cudaStreamSynchronize(h->stream));
    cudaGraphExecDestroy(h->graph);
    h->graph = nullptr;
  }
  return PHONO_OK;
}

// z extent of each inclusion as simulation/grid.py:171-174 computes it.  The
// first inclusion keeps the z nodes with z <= t.z (the float32 depth widened
// to double).  That line rebinds the loop's `z` to the kept index array, so
// every later inclusion keeps the positions p of the previous selection with
// p <= t.z.  With ascending node coordinates every selection is a prefix of
// the z nodes: kend[t] is its length.
static std::vector<int> inclusion_z_extents(const double* z, int nz, const float* tz, int n) {
  std::vector<int> kend(n);
  int prev = nz;
  for (int t = 0; t < n; t++) {
    const double depth = (double)tz[t];
    int cnt = 0;
    if (t == 0) {
      for (int k = 0; k < nz; k++) cnt += z[k] <= depth;
    } else {
      for (int p = 0; p < prev; p++) cnt += (double)p <= depth;
    }
    kend[t] = cnt;
    prev = cnt;
  }
  return kend;
}

int phono_set_inclusions(phono_handle* h, const phono_inclusions* inc, const double* table, int nmat) {
  if (!h || !inc || !table || !inc->x || !inc->y || !inc->z) return fail(PHONO_ERR_ARG, "NULL argument");
  if (h->batch) return fail(PHONO_ERR_STATE, "handle is in a batch");
  const int nx = h->d.nx, ny = h->d.ny, nz = h->d.nz, n = inc->n;
  if (n < 0) return fail(PHONO_ERR_ARG, "n must be >= 0");
  if (n > 0 && (!inc->tx || !inc->ty || !inc->tz || !inc->tr)) return fail(PHONO_ERR_ARG, "NULL inclusion array");
  if (nmat < 1 || nmat > 256) return fail(PHONO_ERR_ARG, "nmat must be in 1..256");
  if (inc->host < 0 || inc->host >= nmat) return fail(PHONO_ERR_ARG, "host material id out of range");
  if (!inc->id && (inc->inside < 0 || inc->inside >= nmat)) return fail(PHONO_ERR_ARG, "inside material id out of range");
  for (int q = 0; q < n; q++)
    if (inc->id && inc->id[q] >= nmat) return fail(PHONO_ERR_ARG, "inclusion material id out of range");
  const double* axes[3] = {inc->x, inc->y, inc->z};
  const int ns[3] = {nx, ny, nz};
  for (int a = 0; a < 3; a++)
    for (int q = 0; q < ns[a]; q++) {
      if (!std::isfinite(axes[a][q])) return fail(PHONO_ERR_ARG, "node coordinates must be finite");
      if (q > 0 && !(axes[a][q] > axes[a][q - 1])) return fail(PHONO_ERR_ARG, "node coordinates must ascend");
    }
  for (int q = 0; q < nmat * PHONO_TABLE_COLS; q++)
    if (!std::isfinite(table[q])) return fail(PHONO_ERR_ARG, "material table holds a non-finite value");
  for (int q = 0; q < nmat; q++)
    if (!(table[q * PHONO_TABLE_COLS + 12] > 0.0)) return fail(PHONO_ERR_ARG, "density must be > 0");
  const std::vector<int> kend = inclusion_z_extents(inc->z, nz, inc->tz, n);
  std::vector<double4> incl(n);
  std::vector<uint8_t> ids(n);
  for (int q = 0; q < n; q++) {
    incl[q] = make_double4((double)inc->tx[q], (double)inc->ty[q], (double)inc->tr[q], 0.0);
    ids[q] = inc->id ? inc->id[q] : (uint8_t)inc->inside;
  }
  // the material at node (0, 0, 0), by the kernel's test (its wave speeds set
  // the absorbing-face coefficients)
  int id000 = inc->host;
  for (int q = n - 1; q >= 0; q--) {
    if (kend[q] < 1) continue;
    const double dx = inc->x[0] - incl[q].x, dy = inc->y[0] - incl[q].y;
    if (std::sqrt(dx * dx + dy * dy) < incl[q].z) {
      id000 = ids[q];
      break;
    }
  }
  CK(cudaStreamSynchronize(h->stream));
  // one scratch allocation: coordinates, inclusions, extents, ids
  const size_t bx = (size_t)nx * 8, by = (size_t)ny * 8, bi = (size_t)n * sizeof(double4), bk = (size_t)n * 4;
  const size_t total = bx + by + bi + bk + n + 64;
  char* d = nullptr;
  CK(cudaMalloc(&d, total));
  double* dx = (double*)d;
  double* dy = (double*)(d + bx);
  double4* di = (double4*)(d + round_up(bx + by, 32));
  int* dk = (int*)((char*)di + bi);
  uint8_t* did = (uint8_t*)(dk + n);
  cudaError_t e = cudaMemcpy(dx, inc->x, bx, cudaMemcpyHostToDevice);
  if (e == cudaSuccess) e = cudaMemcpy(dy, inc->y, by, cudaMemcpyHostToDevice);
  if (e == cudaSuccess && n > 0) e = cudaMemcpy(di, incl.data(), bi, cudaMemcpyHostToDevice);
  if (e == cudaSuccess && n > 0) e = cudaMemcpy(dk, kend.data(), bk, cudaMemcpyHostToDevice);
  if (e == cudaSuccess && n > 0) e = cudaMemcpy(did, ids.data(), n, cudaMemcpyHostToDevice);
  if (e == cudaSuccess) e = launch_inclusion_ids(h->mat, h->g, dx, dy, di, dk, did, n, (uint8_t)inc->host, h->stream);
  if (e == cudaSuccess) e = cudaStreamSynchronize(h->stream);
  cudaFree(d);
  if (e != cudaSuccess) return fail(PHONO_ERR_CUDA, std::string("inclusion ids: ") + cudaGetErrorString(e));
  int rc = upload_table(h, table, nmat, id000);
  if (rc) return rc;
  if (h->graph) {  // the absorbing-face coefficients are kernel arguments baked into the graph
    CK(cudaStreamSynchronize(h->stream));
    cudaGraphExecDestroy(h->graph);
    h->graph = nullptr;
  }
  return PHONO_OK;
}

int phono_download_materials(phono_handle* h, uint8_t* host, size_t bytes) {
  if (!h || !host) return fail(PHONO_ERR_ARG, "NULL argument");
  const int nx = h->d.nx, ny = h->d.ny, nz = h->d.nz;
  if (bytes != (size_t)nx * ny * nz) return fail(PHONO_ERR_ARG, "byte count does not match nx*ny*nz");
  CK(cudaStreamSynchronize(h->stream));
  cudaMemcpy3DParms p{};
  p.srcPtr = make_cudaPitchedPtr(h->mat + h->g.mo0, h->g.msy, h->g.msy, ny + 2);
  p.dstPtr = make_cudaPitchedPtr((void*)host, nz, nz, ny);
  p.extent = make_cudaExtent(nz, ny, nx);
  p.kind = cudaMemcpyDeviceToHost;
  CK(cudaMemcpy3DAsync(&p, h->stream));
  CK(cudaStreamSynchronize(h->stream));
  return PHONO_OK;
}

void* phono_stream(phono_handle* h) { return h ? (void*)h->stream : nullptr; }

// switch a handle to tile height tj and the given x segments, keeping the old
// shape if the new one cannot be set up
static int retile(phono_handle* h, int tj, int xseg, const std::vector<int>& starts) {
  if (!h->split && !h->own.tj && tj == h->t.tj && starts == h->t.seg_start) {
    h->t.xseg = xseg;
    return PHONO_OK;
  }
  CK(cudaStreamSynchronize(h->stream));
  const int p = h->d.precision;
  CK(p == PHONO_F64 ? configure_step_f64(tj) : (p == PHONO_F64V ? configure_step_f64v(tj) : configure_step_f32k(tj)));
  Tiling t;
  int rc = apply_tiling(h, t, tj, xseg, starts);
  if (!rc) rc = encode_tensor_maps(h, t);
  if (rc) return rc;
  h->t = t;
  h->own = Tiling();
  CK(set_split(h, false));
  CK(drop_window(h));
  if (h->graph) {  // the captured launches hold the old grid and tensor maps
    cudaGraphExecDestroy(h->graph);
    h->graph = nullptr;
  }
  return PHONO_OK;
}

int phono_set_tiling(phono_handle* h, int tile_j, int x_segment) {
  if (!h) return fail(PHONO_ERR_ARG, "handle is NULL");
  if (h->batch) return fail(PHONO_ERR_STATE, "handle is in a batch");
  const bool keep = tile_j == 0;
  if (tile_j == 0) tile_j = h->t.tj;
  if (tile_j != 4 && tile_j != 8 && tile_j != 16) return fail(PHONO_ERR_ARG, "tile_j must be 0, 4, 8 or 16");
  if (x_segment < -4096) return fail(PHONO_ERR_ARG, "x_segment out of range");
  if (x_segment == 0 && keep) return PHONO_OK;
  if (x_segment == 0)  // keep the current segments (a list included)
    return retile(h, tile_j, h->t.xseg, h->t.seg_start);
  return retile(h, tile_j, x_segment, segment_starts(h->d.nx - 1, x_segment));
}

int phono_set_segments(phono_handle* h, int tile_j, const int* lengths, int n) {
  if (!h || !lengths) return fail(PHONO_ERR_ARG, "NULL argument");
  if (h->batch) return fail(PHONO_ERR_STATE, "handle is in a batch");
  if (tile_j == 0) tile_j = h->t.tj;
  if (tile_j != 4 && tile_j != 8 && tile_j != 16) return fail(PHONO_ERR_ARG, "tile_j must be 0, 4, 8 or 16");
  if (n < 1 || n > PHONO_MAX_SEGMENTS) return fail(PHONO_ERR_ARG, "n must be 1..PHONO_MAX_SEGMENTS");
  std::vector<int> starts{0};
  long long sum = 0;
  for (int q = 0; q < n; q++) {
    if (lengths[q] < 1) return fail(PHONO_ERR_ARG, "segment lengths must be >= 1");
    sum += lengths[q];
    if (sum > h->d.nx - 1) break;
    starts.push_back((int)sum);
  }
  if (sum != h->d.nx - 1) return fail(PHONO_ERR_ARG, "segment lengths must add up to nx - 1 planes");
  return retile(h, tile_j, kExplicitSegments, starts);
}

void phono_destroy(phono_handle* h) { release(h); }

}  // extern "C"

// ---------------------------------------------------------------------------
// batches
// ---------------------------------------------------------------------------
struct phono_batch {
  int cap = 0, precision = 0, tj = 8;
  std::vector<phono_handle*> slot;
  std::vector<int> remaining;
  cudaStream_t stream = nullptr;
  cudaEvent_t ev0 = nullptr, ev1 = nullptr;
  bool timed = false, dirty = true;
  int streams = 0;  // PHONO_BATCH_STREAMS: this many workers, every instance in its own shape; 0: the default scheme
  std::vector<cudaStream_t> workers;
  std::vector<cudaEvent_t> joins;
  cudaEvent_t fork = nullptr;
  std::vector<int> order;     // active slots, costliest first
  std::vector<int> step_end;  // per slot: the instance's budget end
  std::vector<cudaGraphExec_t> igraph;  // per slot, 12 steps with its budget baked in
  cudaStream_t capture = nullptr;       // capture stream (always idle)
};
constexpr int kBatchWorkers = 64;  // worker streams of the default scheme, at most one an instance

static void drop_igraph(phono_batch* b, int s) {
  if (s < (int)b->igraph.size() && b->igraph[s]) {
    cudaGraphExecDestroy(b->igraph[s]);
    b->igraph[s] = nullptr;
  }
}

// a handle destroyed while in a batch leaves it (the batch's work list is
// rebuilt before its next step)
static void batch_detach(phono_batch* b, const phono_handle* h) {
  if (b->stream) cudaStreamSynchronize(b->stream);
  for (int s = 0; s < b->cap; s++)
    if (b->slot[s] == h) {
      b->slot[s] = nullptr;
      b->remaining[s] = 0;
      b->dirty = true;
      drop_igraph(b, s);
    }
}

// a default FP32 handle's tiles for single steps (0) or, with segments of at
// most `limit` planes, for steps beside others; it keeps those it has when the
// new ones cannot be set up
static int reshape_own(phono_handle* h, int limit) {
  Tiling own;
  int rc = own_tiling(h, own, limit);
  if (!rc) rc = encode_tensor_maps(h, own);
  if (rc) return rc;
  h->own = own;
  h->own_limit = limit;
  if (h->graph && !h->lent) {  // (a lent shape's is that of t)
    cudaGraphExecDestroy(h->graph);
    h->graph = nullptr;
  }
  return PHONO_OK;
}

// The batch's work is done: the handle is on its own again.  Where its own
// tiles or form cannot be set up anew it steps on in those of the batch.
static int leave_batch(phono_handle* h) {
  h->batch = nullptr;
  if (h->lent) h->own = Tiling{}, h->lent = false;
  const bool resplit = h->resplit;
  h->resplit = false;
  int rc = h->own.tj ? reshape_own(h, 0) : PHONO_OK;
  if (resplit) {
    const cudaError_t e = set_split(h, true);
    if (e != cudaSuccess) rc = fail(PHONO_ERR_CUDA, std::string("leaving a batch: ") + cudaGetErrorString(e));
  }
  if (rc && h->graph) {  // captured in the form it had before
    cudaGraphExecDestroy(h->graph);
    h->graph = nullptr;
  }
  return rc;
}

static void batch_release(phono_batch* b) {
  if (!b) return;
  if (b->stream) cudaStreamSynchronize(b->stream);
  for (phono_handle* h : b->slot)
    if (h) leave_batch(h);
  for (cudaGraphExec_t g : b->igraph)
    if (g) cudaGraphExecDestroy(g);
  if (b->ev0) cudaEventDestroy(b->ev0);
  if (b->ev1) cudaEventDestroy(b->ev1);
  for (cudaEvent_t e : b->joins) cudaEventDestroy(e);
  if (b->fork) cudaEventDestroy(b->fork);
  for (cudaStream_t w : b->workers) cudaStreamDestroy(w);
  if (b->capture) cudaStreamDestroy(b->capture);
  if (b->stream) cudaStreamDestroy(b->stream);
  delete b;
}

static_assert(PHONO_MAX_SEGMENTS == SEG_TABLE, "segment list limit and the kernel table differ");

// worker streams: as many as asked for, kept for the batch's lifetime
static int need_workers(phono_batch* b, int want) {
  if (!b->fork) CK(cudaEventCreateWithFlags(&b->fork, cudaEventDisableTiming));
  if (!b->capture) CK(cudaStreamCreateWithFlags(&b->capture, cudaStreamNonBlocking));
  while ((int)b->workers.size() < want) {
    cudaStream_t w = nullptr;
    cudaEvent_t j = nullptr;
    CK(cudaStreamCreateWithFlags(&w, cudaStreamNonBlocking));
    cudaError_t e = cudaEventCreateWithFlags(&j, cudaEventDisableTiming);
    if (e != cudaSuccess) {
      cudaStreamDestroy(w);
      return fail(PHONO_ERR_CUDA, std::string("cudaEventCreateWithFlags: ") + cudaGetErrorString(e));
    }
    b->workers.push_back(w);
    b->joins.push_back(j);
  }
  return PHONO_OK;
}

// The active instances, the most node updates left first (each instance's
// chunks are queued before the next one's), and the segment length of those
// that pick their own tiles: as many blocks in all as stay resident (three an
// SM), in segments of 3 to 24 planes.  A step of a small batch is the march of
// one block (6 crystals of 55 k nodes: 15 us a step in segments of 3 planes,
// 53 in 24), while a large one pays for the planes that segments share (24
// crystals of 1.2 M nodes: 552 us in segments of 4 planes, 432 in 24).  An
// instance's segments are cut anew, and its graph captured again, when the
// length has changed by more than a factor of two.
static int batch_rebuild(phono_batch* b) {
  std::vector<int> act;
  double planes = 0;  // of all tile columns
  for (int s = 0; s < b->cap; s++)
    if (b->slot[s] && b->remaining[s] > 0) {
      act.push_back(s);
      const phono_handle* h = b->slot[s];
      const Tiling& t = h->own.tj ? h->own : h->t;
      planes += (double)t.ntj * t.ntk * (h->d.nx - 1);
    }
  auto cost = [&](int x) {
    const phono_handle* h = b->slot[x];
    return (long long)h->d.nx * h->d.ny * h->d.nz * b->remaining[x];
  };
  std::sort(act.begin(), act.end(), [&](int x, int y) {
    const long long cx = cost(x), cy = cost(y);
    return cx != cy ? cx > cy : x < y;
  });
  const int limit = (int)std::min(std::max(planes / (3.0 * sm_count()), 3.0), 24.0);
  for (int s : act) {
    phono_handle* h = b->slot[s];
    if (!h->own.tj || h->split || (h->own_limit && limit <= 2 * h->own_limit && h->own_limit <= 2 * limit)) continue;
    if (b->igraph[s]) CK(cudaStreamSynchronize(b->stream));  // its graph may still run
    int rc = reshape_own(h, limit);
    if (rc) return rc;
    drop_igraph(b, s);
  }
  b->order = act;
  b->dirty = false;
  return PHONO_OK;
}

// one step of instance s on stream st, with the handle's own kernels and tiles
static cudaError_t chain_launch(phono_batch* b, int s, int step_off, cudaStream_t st) {
  phono_handle* h = b->slot[s];
  if (h->split) return split_step_any(h, step_off, b->step_end[s], st);
  return tile_step(h, step_off, b->step_end[s], h->separate_faces, st);
}

// The 12-step graph of the instance in slot s (its own step
// kernels, as phono_step launches them, and a step-counter update clamped at
// its budget), captured on the batch's idle capture stream
static int capture_instance(phono_batch* b, int s) {
  cudaGraph_t g = nullptr;
  CK(cudaStreamBeginCapture(b->capture, cudaStreamCaptureModeThreadLocal));
  cudaError_t e = cudaSuccess;
  for (int q = 0; q < kGraphSteps && e == cudaSuccess; q++) e = chain_launch(b, s, q, b->capture);
  if (e == cudaSuccess) {
    advance_clamped_kernel<<<1, 1, 0, b->capture>>>(b->slot[s]->step_base, kGraphSteps, b->step_end[s]);
    e = cudaGetLastError();
  }
  cudaError_t e2 = cudaStreamEndCapture(b->capture, &g);
  if (e != cudaSuccess || e2 != cudaSuccess) {
    if (g) cudaGraphDestroy(g);
    return fail(PHONO_ERR_CUDA, std::string("instance graph capture: ") + cudaGetErrorString(e != cudaSuccess ? e : e2));
  }
  e = cudaGraphInstantiate(&b->igraph[s], g, 0);
  cudaGraphDestroy(g);
  if (e != cudaSuccess) return fail(PHONO_ERR_CUDA, std::string("cudaGraphInstantiate: ") + cudaGetErrorString(e));
  return PHONO_OK;
}

// n steps of every active instance.  Instance q (costliest
// first) runs on worker q mod W; the host issues chunk by chunk (a 12-step
// instance graph each, then the remainder step by step) across the instances
// so that the workers progress together, and joins the workers back into the
// batch stream only after the last chunk: an instance's next chunk starts as
// soon as its previous one is done, whatever the others are doing.
static cudaError_t streams_steps(phono_batch* b, int n) {
  const int na = (int)b->order.size(), nw = std::min(na, b->streams ? b->streams : (int)b->workers.size());
  cudaError_t e = cudaEventRecord(b->fork, b->stream);
  for (int w = 0; w < nw && e == cudaSuccess; w++) e = cudaStreamWaitEvent(b->workers[w], b->fork, 0);
  const int full = n / kGraphSteps, rem = n % kGraphSteps;
  for (int c = 0; c < full && e == cudaSuccess; c++)
    for (int q = 0; q < na && e == cudaSuccess; q++) {
      const int s = b->order[q];
      if (b->remaining[s] > c * kGraphSteps) e = cudaGraphLaunch(b->igraph[s], b->workers[q % nw]);
    }
  for (int t = 0; t < rem && e == cudaSuccess; t++)
    for (int q = 0; q < na && e == cudaSuccess; q++) {
      const int s = b->order[q];
      if (b->remaining[s] > full * kGraphSteps + t) e = chain_launch(b, s, t, b->workers[q % nw]);
    }
  for (int q = 0; rem && q < na && e == cudaSuccess; q++) {
    const int s = b->order[q];
    if (b->remaining[s] <= full * kGraphSteps) continue;
    advance_clamped_kernel<<<1, 1, 0, b->workers[q % nw]>>>(b->slot[s]->step_base, rem, b->step_end[s]);
    e = cudaGetLastError();
  }
  for (int w = 0; w < nw && e == cudaSuccess; w++) {
    e = cudaEventRecord(b->joins[w], b->workers[w]);
    if (e == cudaSuccess) e = cudaStreamWaitEvent(b->stream, b->joins[w], 0);
  }
  return e;
}

extern "C" {

int phono_batch_create(int capacity, int precision, int tile_j, phono_batch** out) {
  if (!out) return fail(PHONO_ERR_ARG, "out is NULL");
  *out = nullptr;
  if (capacity < 1 || capacity > (1 << 20)) return fail(PHONO_ERR_ARG, "capacity must be in 1..2^20");
  if (precision != PHONO_F64 && precision != PHONO_F32K && precision != PHONO_F64V)
    return fail(PHONO_ERR_ARG, "unknown precision");
  if (tile_j == 0) tile_j = 8;
  if (tile_j != 4 && tile_j != 8 && tile_j != 16) return fail(PHONO_ERR_ARG, "tile_j must be 4, 8 or 16");
  phono_batch* b = new phono_batch();
  b->cap = capacity;
  b->precision = precision;
  b->tj = tile_j;
  b->slot.assign(capacity, nullptr);
  b->remaining.assign(capacity, 0);
  b->step_end.assign(capacity, 0);
  b->igraph.assign(capacity, nullptr);
#define BTRYC(x)                                                                      \
  do {                                                                                \
    cudaError_t e_ = (x);                                                             \
    if (e_ != cudaSuccess) {                                                          \
      batch_release(b);                                                               \
      return fail(PHONO_ERR_CUDA, std::string(#x) + ": " + cudaGetErrorString(e_));   \
    }                                                                                 \
  } while (0)
  BTRYC(cudaStreamCreateWithFlags(&b->stream, cudaStreamNonBlocking));
  BTRYC(cudaEventCreate(&b->ev0));
  BTRYC(cudaEventCreate(&b->ev1));
#undef BTRYC
  *out = b;
  return PHONO_OK;
}

int phono_batch_set_mode(phono_batch* b, int mode, int streams) {
  if (!b) return fail(PHONO_ERR_ARG, "batch is NULL");
  if (mode != PHONO_BATCH_PERSISTENT && mode != PHONO_BATCH_STREAMS) return fail(PHONO_ERR_ARG, "unknown batch mode");
  if (mode == PHONO_BATCH_STREAMS && (streams < 1 || streams > 256))
    return fail(PHONO_ERR_ARG, "streams must be in 1..256");
  for (phono_handle* h : b->slot)
    if (h) return fail(PHONO_ERR_STATE, "the launch scheme of a batch is set while it is empty");
  CK(cudaStreamSynchronize(b->stream));
  const int want = mode == PHONO_BATCH_STREAMS ? streams : 0;
  if (want) {
    int rc = need_workers(b, want);
    if (rc) return rc;
  }
  b->streams = want;
  b->dirty = true;
  return PHONO_OK;
}

int phono_batch_add(phono_batch* b, phono_handle* h, int nsteps) {
  if (!b || !h) return fail(PHONO_ERR_ARG, "NULL argument");
  if (h->batch) return fail(PHONO_ERR_ARG, h->batch == b ? "handle already in the batch" : "handle is in another batch");
  if (h->d.precision != b->precision) return fail(PHONO_ERR_ARG, "handle precision differs from the batch");
  if (!b->streams && h->t.tj != b->tj) return fail(PHONO_ERR_ARG, "handle tile_j differs from the batch");
  if (!h->separate_faces) return fail(PHONO_ERR_ARG, "batched instances need ny >= 4");
  if (h->nmat > BATCH_TAB_ROWS)
    return fail(PHONO_ERR_ARG, "batched instances hold at most " + std::to_string(BATCH_TAB_ROWS) + " materials");
  if (nsteps < 0 || h->steps_done + nsteps > h->nsrc)
    return fail(PHONO_ERR_STATE, "not enough source samples for the requested steps");
  int s = -1;
  for (int q = 0; q < b->cap; q++) {
    if (b->slot[q] == h) return fail(PHONO_ERR_ARG, "handle already in the batch");
    if (s < 0 && !b->slot[q]) s = q;
  }
  if (s < 0) return fail(PHONO_ERR_NOMEM, "batch is full");
  if (!b->streams) {
    int members = 1;
    for (const phono_handle* x : b->slot) members += x != nullptr;
    int rc = need_workers(b, std::min(members, kBatchWorkers));
    if (rc) return rc;
  }
  // In the default scheme FP32 instances step in tiles of the batch's choice
  // (12 crystals of 6.2 M nodes: 98 us a step, 108 at height 8, 177 in one
  // launch a step whose blocks took tiles of all instances from a list).
  const bool lend = !h->own.tj && !b->streams && b->precision == PHONO_F32K;
  Tiling own;
  if (lend) {
    int rc = own_tiling(h, own, 24);  // (its tensor maps come with the next work list)
    if (rc) return rc;
    CK(configure_step_f32k(own.tj));
  }
  CK(cudaStreamSynchronize(h->stream));
  CK(cudaStreamSynchronize(b->stream));
  // beside others FP32's two launches only move more bytes (12 crystals: 120 us
  // a step, 142 with the small ones split)
  const bool resplit = h->split && b->precision == PHONO_F32K;
  if (resplit) CK(set_split(h, false));
  // nothing fails from here on: the handle is the batch's
  h->resplit = resplit;
  if (lend) h->own = own, h->lent = true;
  h->own_limit = 0;  // cut with the next work list
  b->slot[s] = h;
  b->remaining[s] = nsteps;
  b->step_end[s] = h->steps_done + nsteps;
  b->dirty = true;
  h->batch = b;
  return s;
}

int phono_batch_remove(phono_batch* b, int s) {
  if (!b || s < 0 || s >= b->cap || !b->slot[s]) return fail(PHONO_ERR_ARG, "no instance in that slot");
  CK(cudaStreamSynchronize(b->stream));
  phono_handle* h = b->slot[s];
  b->slot[s] = nullptr;
  b->remaining[s] = 0;
  b->dirty = true;
  drop_igraph(b, s);
  return leave_batch(h);
}

int phono_batch_remaining(const phono_batch* b, int s) {
  if (!b || s < 0 || s >= b->cap || !b->slot[s]) return fail(PHONO_ERR_ARG, "no instance in that slot");
  return b->remaining[s];
}

int phono_batch_step(phono_batch* b, int nsteps) {
  if (!b) return fail(PHONO_ERR_ARG, "batch is NULL");
  if (nsteps < 0) return fail(PHONO_ERR_ARG, "nsteps < 0");
  if (nsteps == 0) return PHONO_OK;
  if (b->dirty) {
    for (int s = 0; s < b->cap; s++)
      if (b->slot[s]) CK(cudaStreamSynchronize(b->slot[s]->stream));
    int rc = batch_rebuild(b);
    if (rc) return rc;
  }
  if (nsteps >= kGraphSteps)
    for (int s : b->order)
      if (!b->igraph[s]) {
        int rc = capture_instance(b, s);
        if (rc) return rc;
      }
  CK(cudaEventRecord(b->ev0, b->stream));
  CK(streams_steps(b, nsteps));
  CK(cudaEventRecord(b->ev1, b->stream));
  b->timed = true;
  for (int s = 0; s < b->cap; s++) {
    if (!b->slot[s] || b->remaining[s] <= 0) continue;
    const int adv = std::min(nsteps, b->remaining[s]);
    b->remaining[s] -= adv;
    b->slot[s]->steps_done += adv;
    if (b->remaining[s] == 0) b->dirty = true;
  }
  return PHONO_OK;
}

int phono_batch_sync(phono_batch* b) {
  if (!b) return fail(PHONO_ERR_ARG, "batch is NULL");
  CK(cudaStreamSynchronize(b->stream));
  for (int s = 0; s < b->cap; s++) {
    if (!b->slot[s]) continue;
    int err = 0;
    CK(cudaMemcpy(&err, b->slot[s]->err, sizeof(int), cudaMemcpyDeviceToHost));
    if (err & 2) return fail(PHONO_ERR_TIMEOUT, "instance " + std::to_string(s) + ": a tile-pass pipeline wait ran out");
    if (err) return fail(PHONO_ERR_NUMERIC, "instance " + std::to_string(s) + ": non-finite surface value");
  }
  return PHONO_OK;
}

int phono_batch_last_step_ms(phono_batch* b, float* ms) {
  if (!b || !ms) return fail(PHONO_ERR_ARG, "NULL argument");
  if (!b->timed) return fail(PHONO_ERR_STATE, "no step timed yet");
  CK(cudaEventSynchronize(b->ev1));
  CK(cudaEventElapsedTime(ms, b->ev0, b->ev1));
  return PHONO_OK;
}

void phono_batch_destroy(phono_batch* b) { batch_release(b); }

}  // extern "C"
