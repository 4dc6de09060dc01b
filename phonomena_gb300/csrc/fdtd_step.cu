// Elastic FDTD step for GB300 (sm_103a).
//
// One time step of phonomena's staggered-grid solver
// (simulation/base_solver.py:245-266) as a tile pass; the other form, which FP64
// and small FP32 handles take by default, is split_step.cu's.
//
//  * tile blocks: a (TJ x 32) tile of the (y, z) plane marches along x over a
//    segment of planes.  Planes of u (all three components, 1-node halo), of
//    the material ids and of the pointwise state of the own points (u_old, or v
//    and the Kahan term) stream into a shared-memory ring through TMA
//    (cp.async.bulk.tensor, completion on an mbarrier per slot).  Each iteration
//    evaluates the six stresses of the current plane once (plus the halo
//    stresses the neighbours need) and writes the new state of the plane.
//    Stresses are never written to global memory.  FP32 tiles of height 8 and 16
//    hold them in registers (tile_vec.cuh: four z points a thread, a 3-slot
//    ring), the others in shared memory (tile_rows.cuh: one z point a thread, a
//    4-slot ring).  The tile pass also writes the z = N face point above every
//    (i, j) that is on no x / y face, and in FP32 at height 16 (ny >= 5) all
//    face points: then a step is this launch alone.
//
//  * face points otherwise (fdtd_face_kernel, a second launch; for ny == 3,
//    extra blocks of the same launch): the x = N, y = 0, y = N faces and the z = N
//    points on them (simulation/base_solver.py:540-554).  The reference
//    applies the faces one after another, each reading the plane next to it
//    as left by the earlier faces; the final value of a face point is thus a
//    chain of at most four face formulas ending at the interior value of one
//    point q.  The face thread walks that chain from q's new value (written
//    by the tile pass; evaluated from the input state in the one-launch form).
//
// Three arithmetic schemes share this structure:
//  F64  - the reference leapfrog u' = (2u - u_old) + (dt^2/P) * div T with the
//         reference's IEEE operation order (explicit _rn intrinsics, true
//         division), bit-identical to the reference CPU solver.
//  F32K - FP32 velocity form v' = v + (dt/P) div T, u' = u + dt v' with a
//         Kahan-compensated displacement sum; explicit fmaf only.
//  F64V - the F32K scheme in FP64.
//
#include <cstdio>
#include "scheme.cuh"

namespace phono {

// ---------------------------------------------------------------------------
// fetchers
// ---------------------------------------------------------------------------
template <class R>
struct GlobalFetch {
  const R* ux;
  const R* uy;
  const R* uz;
  const uint8_t* mat;
  const R* tab;
  Geo g;
  R s;
  int wall;
  __device__ __forceinline__ R x(int i, int j, int k) const { return __ldg(ux + fidx(g, i, j, k)); }
  __device__ __forceinline__ R y(int i, int j, int k) const { return __ldg(uy + fidx(g, i, j, k)); }
  __device__ __forceinline__ R z(int i, int j, int k) const {
    if (i == 0 && (wall || k == 0)) return s;  // source overwrite (base_solver.py:251)
    return __ldg(uz + fidx(g, i, j, k));
  }
  __device__ __forceinline__ const R* row(int i, int j, int k) const {
    return tab + 16 * __ldg(mat + g.mo0 + (long long)i * g.msx + (long long)j * g.msy + k);
  }
};

// Geometry of one ring slot of a (TJ x 32) tile: a u component tile is
// TJ+2 rows (1-row halo) of KW values starting KB before the tile's first z
// point; the three components follow each other (CW apart); SU and SM are the
// slot strides of u and of the material ids, rounded to 128 bytes.
template <class R, int TJ>
struct TileShape {
  static constexpr int KW = Lay<R>::KW, KB = Lay<R>::KB;
  static constexpr int CW = (TJ + 2) * KW;                       // component stride in a slot
  static constexpr int SU = ((3 * CW * (int)sizeof(R) + 127) / 128) * 128 / (int)sizeof(R);  // slot stride
  static constexpr int SM = (((TJ + 2) * MKW + 127) / 128) * 128;                               // mat slot stride
};

// interior (V0) value of u_new at a point, evaluated from global memory
template <class S>
__device__ typename S::R v0_global(const StepArgs<typename S::R>& a, const Roles<typename S::R>& r,
                                   const GlobalFetch<typename S::R>& f, int c, int i, int j, int k) {
  using R = typename S::R;
  const Geo& g = a.g;
  long long off = fidx(g, i, j, k);
  if (!in_v0(g, c, i, j, k)) return __ldg(r.cur(c) + off);  // u_new not written this step: last value
  const R* row;
  R dv, u;
  if (c == 0) {
    dv = div_x<S>(a, f, i, j, k, t1_at<S>(a, f, i + 1, j, k, 0), t1_at<S>(a, f, i, j, k, 0), t6_at<S>(a, f, i, j, k),
                  t6_at<S>(a, f, i, j - 1, k), t5_at<S>(a, f, i, j, k), t5_at<S>(a, f, i, j, k - 1), row);
    u = f.x(i, j, k);
  } else if (c == 1) {
    dv = div_y<S>(a, f, i, j, k, t6_at<S>(a, f, i, j, k), t6_at<S>(a, f, i - 1, j, k), t1_at<S>(a, f, i, j + 1, k, 1),
                  t1_at<S>(a, f, i, j, k, 1), t4_at<S>(a, f, i, j, k), t4_at<S>(a, f, i, j, k - 1), row);
    u = f.y(i, j, k);
  } else {
    dv = div_z<S>(a, f, i, j, k, t5_at<S>(a, f, i, j, k), t5_at<S>(a, f, i - 1, j, k), t4_at<S>(a, f, i, j, k),
                  t4_at<S>(a, f, i, j - 1, k), t1_at<S>(a, f, i, j, k + 1, 2), t1_at<S>(a, f, i, j, k, 2), row);
    u = f.z(i, j, k);
  }
  R vn, cn;
  return update_value<S>(u, load_pw<S>(r, c, off), dv, row, vn, cn);
}

// final value of a face point: walk z=N, y=N, y=0, x=N (reverse of the
// reference order), evaluate the interior value at the end, apply the faces
// from_out: the interior value of the chain end is read from the new state,
// which the tile pass has already written (separate face pass); otherwise it
// is evaluated here from the input state (fused launch).  The chain end is
// never a face point when ny >= 4, which is when the separate pass is used.
template <class S>
__device__ typename S::R face_value(const StepArgs<typename S::R>& a, const Roles<typename S::R>& r,
                                    const GlobalFetch<typename S::R>& f, int c, int i, int j, int k,
                                    bool from_out) {
  using R = typename S::R;
  const Geo& g = a.g;
  const int xi = ext_x(g, c) - 1, jN = ext_y(g, c) - 1, kz = ext_z(g, c) - 1;
  int ci = i, cj = j, ck = k;
  const bool sz = ck == kz;  // z = N face at (i, j, kz)
  if (sz) ck -= 1;
  const bool syn = cj == jN;  // y = N face at (i, jN, ck)
  const int kyn = ck;
  if (syn) cj -= 1;
  const bool sy0 = cj == 0;  // y = 0 face at (i, 0, ck)
  if (sy0) cj += 1;
  const bool sx = ci == xi;  // x = N face at (xi, cj, ck)
  if (sx) ci -= 1;
  auto U = [&](int ii, int jj, int kk) -> R {
    return c == 0 ? f.x(ii, jj, kk) : (c == 1 ? f.y(ii, jj, kk) : f.z(ii, jj, kk));
  };
  R val = from_out ? r.out(c)[fidx(g, ci, cj, ck)] : v0_global<S>(a, r, f, c, ci, cj, ck);
  if (sx) val = S::abc(c == 0 ? a.abc[0] : a.abc[1], val, U(xi, cj, ck), U(xi - 1, cj, ck));
  if (sy0) val = S::abc(c == 1 ? a.abc[3] : a.abc[2], val, U(i, 0, kyn), U(i, 1, kyn));
  if (syn) val = S::abc(c == 1 ? a.abc[5] : a.abc[4], val, U(i, jN, kyn), U(i, jN - 1, kyn));
  if (sz) val = S::abc(c == 2 ? a.abc[7] : a.abc[6], val, U(i, j, kz), U(i, j, kz - 1));
  return val;
}

// one face point: flattened index -> (component, plane, i, j, k), final value,
// state store and surface record
template <class S>
__device__ __forceinline__ void face_point(const StepArgs<typename S::R>& a, const Roles<typename S::R>& r,
                                           const typename S::R s, const int tt, const int idx, const bool from_out) {
  using R = typename S::R;
  const Geo& g = a.g;
  if (idx >= a.faces.off[12]) return;
  int q = 0;
  while (q < 11 && idx >= a.faces.off[q + 1]) q++;
  const int c = q >> 2, pl = q & 3, rr = idx - a.faces.off[q];
  const int ex = ext_x(g, c), ey = ext_y(g, c), ez = ext_z(g, c);
  int i, j, k;
  if (pl == 0) {  // z = N points that are also on an x / y face (the rest: tile pass)
    k = ez - 1;
    if (rr < ex) { i = rr; j = 0; }
    else if (rr < 2 * ex) { i = rr - ex; j = ey - 1; }
    else { i = ex - 1; j = 1 + rr - 2 * ex; }
  }
  else if (pl == 1) { i = rr / (ez - 1); k = rr - i * (ez - 1); j = ey - 1; }
  else if (pl == 2) { i = rr / (ez - 1); k = rr - i * (ez - 1); j = 0; }
  else { j = rr / (ez - 1); k = rr - j * (ez - 1); j += 1; i = ex - 1; }
  GlobalFetch<R> f{r.cur(0), r.cur(1), r.cur(2), a.mat, a.tab, g, s, a.source_mode};
  R val = a.bc == 1 ? R(0) : face_value<S>(a, r, f, c, i, j, k, from_out);
  long long off = fidx(g, i, j, k);
  store_point<S>(r, c, off, val, R(0), R(0));
  if (c == 2 && k == 0) record(a, tt, i, j, val);
}

// separate face pass: runs after the tile-only step launch on the same stream
template <class S>
__global__ void __launch_bounds__(256) fdtd_face_kernel(const __grid_constant__ StepArgs<typename S::R> a) {
  using R = typename S::R;
  const int tt = __ldg(a.step_base) + a.step_off;
  if (tt >= a.step_end) return;
  const Roles<R> r = roles<S>(a, tt);
  face_point<S>(a, r, (R)__ldg(a.src + tt), tt, blockIdx.x * 256 + threadIdx.x, true);
}

// ---------------------------------------------------------------------------
// TMA + mbarrier helpers (inline PTX)
// ---------------------------------------------------------------------------
__device__ __forceinline__ uint32_t smem_u32(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }

__device__ __forceinline__ void mbar_init(uint64_t* bar, int count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(bar)), "r"(count) : "memory");
}
__device__ __forceinline__ void mbar_expect_tx(uint64_t* bar, uint32_t bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_u32(bar)), "r"(bytes)
               : "memory");
}
__device__ __forceinline__ bool mbar_try_wait(uint64_t* bar, uint32_t parity) {
  uint32_t ok;
  asm volatile(
      "{\n .reg .pred p;\n mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n selp.u32 %0, 1, 0, p;\n}\n"
      : "=r"(ok)
      : "r"(smem_u32(bar)), "r"(parity)
      : "memory");
  return ok != 0;
}
// bounded wait: false if the phase did not complete within `limit` polls
// (limit <= 0: 2^22 polls, about 0.3 s with the back-off below)
__device__ __forceinline__ bool mbar_wait(uint64_t* bar, uint32_t parity, int limit = 0) {
  if (limit <= 0) limit = 1 << 22;
  for (int it = 0; it < limit; it++) {
    if (mbar_try_wait(bar, parity)) return true;
    if (it > 64) __nanosleep(64);
  }
  return false;
}
__device__ __forceinline__ void tma_load_4d(void* dst, const CUtensorMap* tm, int c0, int c1, int c2, int c3,
                                            uint64_t* bar) {
  asm volatile(
      "cp.async.bulk.tensor.4d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3, %4, %5}], "
      "[%6];" ::"r"(smem_u32(dst)),
      "l"(tm), "r"(c0), "r"(c1), "r"(c2), "r"(c3), "r"(smem_u32(bar))
      : "memory");
}
__device__ __forceinline__ void tma_load_3d(void* dst, const CUtensorMap* tm, int c0, int c1, int c2,
                                            uint64_t* bar) {
  asm volatile(
      "cp.async.bulk.tensor.3d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3, %4}], "
      "[%5];" ::"r"(smem_u32(dst)),
      "l"(tm), "r"(c0), "r"(c1), "r"(c2), "r"(smem_u32(bar))
      : "memory");
}

// Shared memory of a tile block: mbarriers, the u ring (NSLOT planes of the
// three components with a 1-node halo), the pointwise ring (own points of
// u_old, or of v and the Kahan terms, for the same planes), the material-id
// ring, the stress planes and, last, the material table (its size depends on
// the number of materials, so it is the only variable part).
template <class S, int TJ>
struct SmemPlan {
  using R = typename S::R;
  using TF = TileShape<R, TJ>;
  static constexpr int W = TK + 2, PL = W * (TJ + 2);
  static constexpr int NPW = S::kahan ? 2 : 1;  // pointwise arrays: v and c, or u_old
  static constexpr int PWC = TJ * TK;           // one component of a pointwise tile
  static constexpr int PWS = NPW * 3 * PWC;     // one pointwise slot
  static constexpr size_t BARS = 128;
  static constexpr size_t UR = (size_t)NSLOT * TF::SU * sizeof(R);
  static constexpr size_t PWR = (size_t)NSLOT * PWS * sizeof(R);
  static constexpr size_t MR = (size_t)NSLOT * TF::SM;
  static constexpr size_t TS = ((7 * PL * sizeof(R) + 127) / 128) * 128;
  static constexpr size_t off_u = BARS, off_pw = off_u + UR, off_m = off_pw + PWR, off_t = off_m + MR;
  static constexpr size_t off_tab = off_t + TS;
  static constexpr size_t fixed = off_tab + 128;  // + alignment slack
  static constexpr size_t bytes(int table_rows) { return fixed + (size_t)table_rows * 16 * sizeof(R); }
  static constexpr uint32_t tx_bytes = (uint32_t)(3 * (TJ + 2) * Lay<R>::KW * sizeof(R) + (TJ + 2) * MKW);
  static constexpr uint32_t pw_bytes = (uint32_t)(PWS * sizeof(R));
  static_assert((PWC * sizeof(R)) % 128 == 0 && (TF::SU * sizeof(R)) % 128 == 0, "ring tiles must stay 128-byte aligned");
};

// FP32 tiles of height 8 and 16 take the vectorised pass (tile_vec.cuh); at
// height 4 one updating warp does not pay for the halo warp (256x256x128
// cells: 192 us a step against 154 with one row a thread).
template <class S, int TJ>
__host__ __device__ constexpr bool vec_tile() { return sizeof(typename S::R) == 4 && TJ >= VEC_TJ; }

#include "tile_rows.cuh"
#include "tile_vec.cuh"

// the tile pass of one block
template <class S, int TJ>
__device__ __forceinline__ void run_tile(const StepArgs<typename S::R>& a, unsigned char* base,
                                         const Roles<typename S::R>& r, const typename S::R s, const int tt,
                                         const int tid, const int b) {
  if constexpr (vec_tile<S, TJ>()) tile_block_vec<TJ>(a, base, r, s, tt, tid, b);
  else tile_block_rows<S, TJ>(a, base, r, s, tt, tid, b);
}

// ---------------------------------------------------------------------------
// the step kernel
// ---------------------------------------------------------------------------
// Resident blocks per SM the register allocation is made for (measured on
// GB300 for the 256x256x128 crystal and the 64-crystal batch).  FP32: tile
// height 4, 6 blocks of 128 threads (up to 85 registers); heights 8 and 16, 5
// blocks of 96 or 3 of 160 threads (up to 128 registers).  FP64: 16 warps per
// SM.
template <class R, int TJ>
struct MinBlocks {
  static constexpr int value = sizeof(R) == 8 ? (TJ < 16 ? 16 / TJ : 1) : (TJ == 4 ? 6 : (TJ == 8 ? 5 : 3));
};
template <class S, int TJ>
__host__ __device__ constexpr int step_threads() {
  return vec_tile<S, TJ>() ? VecPlan<TJ>::NT : TK * TJ;
}
template <class S, int TJ>
__host__ __device__ constexpr size_t step_smem(int table_rows) {
  return vec_tile<S, TJ>() ? VecPlan<TJ>::bytes(table_rows) : SmemPlan<S, TJ>::bytes(table_rows);
}
template <class S, int TJ>
__global__ void __launch_bounds__(step_threads<S, TJ>(), MinBlocks<typename S::R, TJ>::value)
    fdtd_step_kernel(const __grid_constant__ StepArgs<typename S::R> a) {
  using R = typename S::R;
  extern __shared__ __align__(128) unsigned char smem_raw[];
  // 128-byte aligned start, derived by pointer arithmetic on the shared array
  // so that every access below stays a shared-memory access (an integer
  // round trip would turn them into generic loads)
  unsigned char* base = smem_raw + ((128u - (smem_u32(smem_raw) & 127u)) & 127u);

  const int tt = __ldg(a.step_base) + a.step_off;
  if (tt >= a.step_end) {  // a batched instance past its budget
    last_launch_done();
    return;
  }
  const Roles<R> r = roles<S>(a, tt);
  const R s = (R)__ldg(a.src + tt);
  const int tid = threadIdx.y * TK + threadIdx.x;

  if ((int)blockIdx.x >= a.n_tile_blocks) {
    // ---------------- face blocks (fused launch) ----------------
    face_point<S>(a, r, s, tt, ((int)blockIdx.x - a.n_tile_blocks) * step_threads<S, TJ>() + tid, false);
    return;
  }

  // ---------------- tile blocks ----------------
  run_tile<S, TJ>(a, base, r, s, tt, tid, blockIdx.x);
}

// ---------------------------------------------------------------------------
// host-side launch helpers (called by the C ABI in api.cu)
// ---------------------------------------------------------------------------
template <class S, int TJ>
static cudaError_t configure_tj() {
  return cudaFuncSetAttribute(fdtd_step_kernel<S, TJ>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                              (int)step_smem<S, TJ>(TAB_ROWS_MAX));
}

template <class S>
cudaError_t configure_step(int tj) {
  switch (tj) {
    case 4: return configure_tj<S, 4>();
    case 8: return configure_tj<S, 8>();
    case 16: return configure_tj<S, 16>();
    default: return cudaErrorInvalidValue;
  }
}

// separate_faces: 0 one fused launch (face points in extra blocks), 1 the tile
// launch then the face launch; 2 only the tile launch and 3 only the face
// launch of the separate form (phono_time_kernels times them apart).  No face
// launch where the tile pass writes the faces.
template <class S, int TJ>
static cudaError_t launch_tj(const StepArgs<typename S::R>& a, int separate_faces, cudaStream_t st) {
  const int nfaces = writes_faces(sizeof(typename S::R) == 4, TJ, a.g.ny) ? 0 : a.faces.off[12];
  constexpr int NT = step_threads<S, TJ>();
  dim3 block(TK, NT / TK);
  // fused: face points handled by extra blocks of the same launch
  dim3 grid(a.n_tile_blocks + (separate_faces ? 0 : (nfaces + NT - 1) / NT));
  if (separate_faces != 3) {
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = grid;
    cfg.blockDim = block;
    cfg.dynamicSmemBytes = step_smem<S, TJ>(a.nmat);
    cfg.stream = st;
    cudaLaunchAttribute at{};
    at.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at.val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = &at;
    // behind the tile launch of the step before, which wrote its faces too
    cfg.numAttrs = separate_faces == 1 && nfaces == 0 && a.step_off > 0 ? 1 : 0;
    cudaError_t e = cudaLaunchKernelEx(&cfg, fdtd_step_kernel<S, TJ>, a);
    if (e != cudaSuccess) return e;
  }
  if ((separate_faces == 1 || separate_faces == 3) && nfaces > 0)
    fdtd_face_kernel<S><<<(nfaces + 255) / 256, 256, 0, st>>>(a);
  return cudaGetLastError();
}

template <class S>
cudaError_t launch_step(const StepArgs<typename S::R>& a, int tj, int separate_faces, cudaStream_t st) {
  switch (tj) {
    case 4: return launch_tj<S, 4>(a, separate_faces, st);
    case 8: return launch_tj<S, 8>(a, separate_faces, st);
    case 16: return launch_tj<S, 16>(a, separate_faces, st);
    default: return cudaErrorInvalidValue;
  }
}

// non-template entry points for the C ABI translation unit
cudaError_t configure_step_f64(int tj) { return configure_step<F64>(tj); }
cudaError_t configure_step_f32k(int tj) { return configure_step<F32K>(tj); }
cudaError_t launch_step_f64(const StepArgs<double>& a, int tj, int nf, cudaStream_t st) {
  return launch_step<F64>(a, tj, nf, st);
}
cudaError_t launch_step_f32k(const StepArgs<float>& a, int tj, int nf, cudaStream_t st) {
  return launch_step<F32K>(a, tj, nf, st);
}
cudaError_t configure_step_f64v(int tj) { return configure_step<F64V>(tj); }
cudaError_t launch_step_f64v(const StepArgs<double>& a, int tj, int nf, cudaStream_t st) {
  return launch_step<F64V>(a, tj, nf, st);
}

}  // namespace phono
