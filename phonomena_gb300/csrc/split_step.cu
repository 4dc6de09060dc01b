// Two-launch step: all stresses of a chunk of planes into a stress window in
// global memory, then every displacement point of the chunk, faces included.
//
// Each stress is computed once and each thread owns one point of a flattened
// box, so no lane idles on a ragged z or y extent, no block waits at a barrier
// and a mesh of a few thousand nodes still spreads over all SMs.  The stresses
// cost a write and a read of 24 (FP32) or 48 bytes a node.  The velocity forms
// keep them in the second buffers of v and of the Kahan term; the leapfrog has
// a window of at most a few dozen planes of a large mesh, and a step walks
// through it in chunks.  The result is that of the tile pass, bit for bit.
//
// Bound (one GB300, us a step, the best tile shape of the tile pass first):
// the FP64 leapfrog by latency: of 1214 instructions a stress point 18 are FP64,
// and with the 25 warps an SM that the registers leave (28 in the update) issue
// is 60% busy, ALU 59 (45), FP64 pipe 58 (56), with 2.6 stalls an issue on a
// dependent instruction and 2.7 (3.3) on loads; the FP64 velocity form by the
// FP64 pipe; small meshes by two dependent launches (1.2 us each) of three or
// four L2 latencies.
//   nodes       25x21x13   41x41x21   61x61x21   150x131x47  194x162x98  257x257x129
//   F64         25 / 8.4   32 / 10.8  47 / 13.5  354 / 102   969 / 337   2012 / 924
//   F64V        13 / 7.2   21 / 9.1   29 / 13.4  197 / 98    559 / 307   1174 / 838
//   F32K        9 / 5.3    10 / 5.7   12 / 6.7   (split_f32.cu; larger meshes: tile_vec.cuh)
#include "split_point.cuh"

namespace phono {

// an operand of a product in integer arithmetic: its value, and taken apart
// where the integer path may take it
struct SoftArg {
  double x;
  SoftNum n;
  bool ok;
};
__device__ __forceinline__ SoftArg soft_arg(double x) {
  SoftArg v;
  v.x = x;
  v.n = soft_split(x, v.ok);
  return v;
}
__device__ __forceinline__ bool is_zero(double x) {
  return ((uint32_t)__double2hiint(x) << 1 | (uint32_t)__double2loint(x)) == 0u;
}
// a zero's quotient or product keeps its sign (flip: the other operand's, in the top bit)
__device__ __forceinline__ double signed_zero(double x, uint32_t flip) {
  return soft_double(((uint32_t)__double2hiint(x) ^ flip) & 0x80000000u, 0u);
}

// a call, so that nothing multiplies ahead of the branches around it
__device__ __noinline__ double slow_mul(double x, double c) { return __dmul_rn(x, c); }

// the velocity form in FP64: reciprocal spacings, coefficients as stored.  Of
// its 63 FP64 operations a node 15 are products with a constant that no sum
// takes in; SOFT: those run in integer arithmetic, 24 FP64 instructions a
// stress point and 33 a node's update becoming 18 and 30 (the FP64 pipe, 85%
// busy before, is still the bound at 78 and 67%).  A product is a chain of 25
// instructions, so that meshes whose launches are a latency keep the plain
// form.  us a step, plain / SOFT: 41x41x21 nodes 9.5 / 10.9, 61x61x21 13.9 /
// 13.4, 81x71x31 26.1 / 22.7, 194x162x98 387 / 307, 257x257x129 1078 / 838.
template <bool SOFT>
struct VelOps {
  using Base = F64V;
  using R = double;
  using D = SoftFactor;
  using Args = SplitArgs<R, D>;
  // resident blocks the registers are allotted for (SOFT, us a step on
  // 256x256x128 cells): 9 and 8 838, 8 and 8 844, 6 and 7 877, 8 and 9 885
  static constexpr int STRESS_BLOCKS = SOFT ? 9 : 6, UPDATE_BLOCKS = SOFT ? 8 : 7;
  static constexpr bool SMALL = !SOFT;  // stress points may be shared by threads
  // x * c.  The result of a product may go into another one: the range that
  // soft_arg tests leaves room for two factors (soft_f64.cuh).
  template <class V>
  static __device__ __forceinline__ SoftArg product(const SoftArg& x, const SoftRec& c, V value) {
    SoftArg p;
    if constexpr (!SOFT) {
      p.x = __dmul_rn(x.x, value());
      return p;
    }
    const bool fits = (int)c.hi < 0;
    p.ok = x.ok && fits;
    if (p.ok) {
      p.n = soft_mul(x.n, c);
      p.x = soft_join(p.n);
    } else if (fits && is_zero(x.x)) {
      p.x = signed_zero(x.x, soft_sign(c));
    } else {
      p.x = slow_mul(x.x, value());
    }
    return p;
  }
  static __device__ __forceinline__ SoftArg product(R x, const D& c) {
    return product(soft_arg(x), c.rec, [&] { return c.v; });
  }
  static __device__ __forceinline__ void normals(const Args& a, int id, R d1, R d2, R d3, const D& x, const D& y, const D& z,
                                                 R* t) {
    const R* c = a.tab + 16 * id;
    const SoftRec* rec = a.rec + 16 * id;
    const R e1 = product(d1, x).x, e2 = product(d2, y).x;
    const SoftArg e3 = product(d3, z);
#pragma unroll
    for (int q = 0; q < 3; q++)
      t[q] = __fma_rn(__ldg(c + 3 * q), e1,
                      __fma_rn(__ldg(c + 3 * q + 1), e2, product(e3, ldd(rec + 3 * q + 2), [&] { return __ldg(c + 3 * q + 2); }).x));
  }
  static __device__ __forceinline__ R normal(const Args& a, int id, int q, R d1, R d2, R d3, const D& x, const D& y, const D& z) {
    const R* c = a.tab + 16 * id + 3 * q;
    const R e1 = product(d1, x).x, e2 = product(d2, y).x;
    const SoftArg e3 = product(d3, z);
    return __fma_rn(__ldg(c), e1, __fma_rn(__ldg(c + 1), e2, product(e3, ldd(a.rec + 16 * id + 3 * q + 2), [&] { return __ldg(c + 2); }).x));
  }
  static __device__ __forceinline__ R shear(const Args& a, int id, int col, R d1, const D& x, R d2, const D& y) {
    const R s = __fma_rn(d1, x.v, product(d2, y).x);
    return product(soft_arg(s), ldd(a.rec + 16 * id + col), [&] { return __ldg(a.tab + 16 * id + col); }).x;
  }
  static __device__ __forceinline__ R div3(const Args& a, R d1, const D& x, R d2, const D& y, R d3, const D& z) {
    return __fma_rn(d1, x.v, __fma_rn(d2, y.v, product(d3, z).x));
  }
  static __device__ __forceinline__ R update(const Args& a, int id, R u, Pw<R> pw, R dv, R& vn, R& cn) {
    return update_value<F64V>(u, pw, dv, __ldg(a.tab + 16 * id + 12), a.dt, vn, cn);
  }
};

// the leapfrog: multiplications by constants and divisions in integer
// arithmetic (soft_f64.cuh), additions on the FP64 pipe
__device__ __noinline__ double slow_div(double x, double b, DivTable k) { return k.tab ? div_tab(x, b, k) : __ddiv_rn(x, b); }

// SHARED: every material has c10 = c20, c01 = c21 and c02 = c12 (isotropic and
// cubic ones do), so that the normal stresses share three of their nine terms
// (256x256x128 cells: 924 us a step, 1008 without).
template <bool SHARED>
struct LeapOps {
  using Base = F64;
  using R = double;
  using D = SoftRec;
  using Args = SplitArgs<double, SoftRec>;
  // resident blocks the registers are allotted for (us a step on 256x256x128
  // cells): 7 and 8 924, 6 and 8 954, 8 and 8 926, 7 and 7 962
  static constexpr int STRESS_BLOCKS = 7, UPDATE_BLOCKS = 8;
  static constexpr bool SMALL = true;
  static __device__ __forceinline__ double divide(const Args& a, double x, const SoftRec& d) {
    const SoftArg v = soft_arg(x);
    if (v.ok && (int)d.hi < 0) return soft_join(soft_div(v.n, d, [&] { return __ldg(a.vals + d.idx); }));
    return is_zero(x) ? signed_zero(x, 0u) : slow_div(x, __ldg(a.vals + d.idx), a.dtab);
  }
  static __device__ __forceinline__ double times(const Args& a, double x, const SoftRec& c) {
    const SoftArg v = soft_arg(x);
    if (v.ok && (int)c.hi < 0) return soft_join(soft_mul(v.n, c));
    return is_zero(x) ? signed_zero(x, soft_sign(c)) : __dmul_rn(__ldg(a.vals + c.idx), x);
  }
  // (c * x) / d, both roundings
  static __device__ __forceinline__ double scaled(const Args& a, const SoftArg& v, const SoftRec& c, const SoftRec& d) {
    if (v.ok && (int)(c.hi & d.hi) < 0)
      return soft_join(soft_div(soft_mul(v.n, c), d, [&] { return __ldg(a.vals + d.idx); }));
    if (is_zero(v.x)) return signed_zero(v.x, soft_sign(c));
    const double y = __dmul_rn(__ldg(a.vals + c.idx), v.x);
    return is_zero(y) ? y : slow_div(y, __ldg(a.vals + d.idx), a.dtab);
  }
  static __device__ __forceinline__ void normals(const Args& a, int id, R d1, R d2, R d3, const D& x, const D& y,
                                                 const D& z, R* t) {
    const SoftRec* c = a.rec + 16 * id;
    const SoftArg v1 = soft_arg(d1), v2 = soft_arg(d2), v3 = soft_arg(d3);
    if constexpr (SHARED) {
      const R x1 = scaled(a, v1, ldd(c + 3), x), y0 = scaled(a, v2, ldd(c + 1), y), z0 = scaled(a, v3, ldd(c + 2), z);
      t[0] = __dadd_rn(__dadd_rn(scaled(a, v1, ldd(c), x), y0), z0);
      t[1] = __dadd_rn(__dadd_rn(x1, scaled(a, v2, ldd(c + 4), y)), z0);
      t[2] = __dadd_rn(__dadd_rn(x1, y0), scaled(a, v3, ldd(c + 8), z));
    } else {
      // not unrolled: the instructions of three copies miss the cache (1033 us
      // a step on 256x256x128 cells, 1008 so)
#pragma unroll 1
      for (int q = 0; q < 3; q++)
        t[q] = __dadd_rn(__dadd_rn(scaled(a, v1, ldd(c + 3 * q), x), scaled(a, v2, ldd(c + 3 * q + 1), y)),
                         scaled(a, v3, ldd(c + 3 * q + 2), z));
    }
  }
  static __device__ __forceinline__ R normal(const Args& a, int id, int q, R d1, R d2, R d3, const D& x, const D& y, const D& z) {
    const SoftRec* c = a.rec + 16 * id + 3 * q;
    return __dadd_rn(__dadd_rn(scaled(a, soft_arg(d1), ldd(c), x), scaled(a, soft_arg(d2), ldd(c + 1), y)),
                     scaled(a, soft_arg(d3), ldd(c + 2), z));
  }
  static __device__ __forceinline__ R shear(const Args& a, int id, int col, R d1, const D& x, R d2, const D& y) {
    return times(a, __dadd_rn(divide(a, d1, x), divide(a, d2, y)), ldd(a.rec + 16 * id + col));
  }
  static __device__ __forceinline__ R div3(const Args& a, R d1, const D& x, R d2, const D& y, R d3, const D& z) {
    return __dadd_rn(__dadd_rn(divide(a, d1, x), divide(a, d2, y)), divide(a, d3, z));
  }
  static __device__ __forceinline__ R update(const Args& a, int id, R u, Pw<R> pw, R dv, R& vn, R& cn) {
    vn = cn = 0;
    // 2u is exact, so the FMA rounds as the reference's 2u - u_old
    return __dadd_rn(__fma_rn(2.0, u, -pw.p0), times(a, dv, ldd(a.rec + 16 * id + 12)));
  }
};

// ---------------------------------------------------------------------------
// stresses of planes [sa, sb): one thread per node of [sa, sb) x [0, ny-1) x
// [0, nz-1).  Zero where the reference never writes (base_solver.py:329-433).
//
// PARTS: threads that share a point, in blocks of their own (blockIdx.y).  On a
// mesh of few blocks the pass is the 1220 instructions of one thread after
// another: two parts (normal and shear stresses) or six (a stress each)
// shorten that chain, until the work done twice fills the chip.  us a step
// with 1 / 2 / 6 parts: F64 25x21x13 nodes 11.9 / 9.8 / 8.4, 41x41x21 12.5 /
// 10.8 / 10.8, 61x61x21 14.3 / 14.4 / 15.6, 101x101x41 44 / 46 / 58; F64V
// 25x21x13 8.3 / 7.6 / 7.2, 41x41x21 9.5 / 9.5 / 9.8.
// ---------------------------------------------------------------------------
template <class O, int PARTS>
__global__ void __launch_bounds__(SPLIT_THREADS, O::STRESS_BLOCKS) split_stress_kernel(const __grid_constant__ typename O::Args a) {
  using R = typename O::R;
  using B = typename O::Base;
  last_launch_done();
  const int tt = __ldg(a.step_base) + a.step_off;
  if (tt >= a.step_end) return;
  const Geo& g = a.g;
  const int nx = g.nx;
  int n = blockIdx.x * SPLIT_THREADS + threadIdx.x;
  const int q1 = fdiv(n, a.dz1), k = n - q1 * a.dz1.d;
  const int q2 = fdiv(q1, a.dy1), j = q1 - q2 * a.dy1.d;
  const int i = a.sa + q2;
  if (i >= a.sb) return;
  const Roles<R> r = roles<B>(a, tt);
  const unsigned sx = (unsigned)g.sx, sy = (unsigned)g.sy;
  const unsigned o = (unsigned)g.o0 + (unsigned)i * sx + (unsigned)j * sy + (unsigned)k;
  const R *X = r.u_cur + o, *Y = X + r.fs, *Z = Y + r.fs;
  const uint8_t* M = a.mat + g.mo0 + (long long)i * g.msx + (long long)j * g.msy + k;
  const bool kz = k == 0;
  const int up = kz ? 0 : 1;  // shear moduli of T4, T5: one layer down, except in the z = 0 row
  const bool i_n = i >= 1 && i <= nx - 2, i_s = i <= nx - 2, j_n = j >= 1;
  const int part = PARTS == 1 ? 0 : (int)blockIdx.y;
  // the stresses of this block, T1..T6
  auto mine = [&](int q) { return PARTS == 1 || (PARTS == 2 ? part == q / 3 : part == q); };
  const R x0 = X[0], y0 = Y[0];
  R z0 = Z[0];
  if (i == 0 && (a.source_mode == 1 || kz)) z0 = (R)__ldg(a.src + tt);  // source overwrite (base_solver.py:251)
  const R x_k = mine(4) ? X[1] : R(0), x_j = mine(5) ? X[sy] : R(0), y_k = mine(3) ? Y[1] : R(0),
          y_i = mine(5) ? Y[sx] : R(0), z_j = mine(3) ? Z[sy] : R(0), z_i = mine(4) ? Z[sx] : R(0);
  R t[6] = {R(0), R(0), R(0), R(0), R(0), R(0)};
  if (i_n && j_n && (mine(0) || mine(1) || mine(2))) {
    const R d1 = B::sub(x0, *(X - sx)), d2 = B::sub(y0, *(Y - sy)), d3 = B::sub(z0, Z[-1]);
    const auto ax = ldd(a.sdx + (kz ? 0 : i - 1));
    const auto ay = ldd(a.sdy + (kz ? 0 : j - 1));
    const auto az = ldd(a.sdz + (kz ? 0 : k - 1));
    if constexpr (PARTS == 6) t[0] = O::normal(a, M[0], part, d1, d2, d3, ax, ay, az);
    else O::normals(a, M[0], d1, d2, d3, ax, ay, az, t);
  }
  if (kz) t[PARTS == 6 ? 0 : 2] = PARTS == 6 && part != 2 ? t[0] : R(0);  // base_solver.py:418
  // shears; the z = 0 row's substituted spacings are base_solver.py:420-433's
  if (i_n && mine(3))
    t[3] = O::shear(a, M[g.msy + up], 9, B::sub(y_k, y0), ldd(kz ? a.fdy : a.fdz + k), B::sub(z_j, z0),
                    ldd(kz ? a.fdz : a.fdy + j));
  if (i_s && j_n && mine(4))
    t[4] = O::shear(a, M[g.msx + up], 10, B::sub(x_k, x0), ldd(kz ? a.fdx : a.fdz + k), B::sub(z_i, z0),
                    ldd(kz ? a.fdz : a.fdx + i));
  if (i_s && mine(5))
    t[5] = O::shear(a, M[g.msx + g.msy], 11, B::sub(x_j, x0), ldd(kz ? a.fdx : a.fdy + j), B::sub(y_i, y0),
                    ldd(kz ? a.fdz : a.fdx + i));
  const unsigned to = (unsigned)(i % a.W) * a.tsx + (unsigned)(j * a.tsy + k);
  if constexpr (PARTS == 6) {
    if (part < 3) a.Ta[to + part * a.tcs] = t[0];
    else a.Tb[to + (part - 3) * a.tcs] = part == 3 ? t[3] : part == 4 ? t[4] : t[5];
    return;
  }
#pragma unroll
  for (int q = 0; q < 3; q++) {
    if (mine(q)) a.Ta[to + q * a.tcs] = t[q];
    if (mine(q + 3)) a.Tb[to + q * a.tcs] = t[q + 3];
  }
}

// ---------------------------------------------------------------------------
// new state of planes [pa, pb): one thread per point of each component that is
// on no face, those next to a face first.  A face point's value is a chain of at most four face formulas
// (base_solver.py:540-554, in the order x=N, y=0, y=N, z=N) from the new value
// of one such point: the thread of that point writes it (in warps of their own:
// with the z = N points in the lanes above them, the FP64 step was 20% slower).
// The velocity forms
// update v and the Kahan term in place (no other thread reads them), which
// leaves their second buffers to the stresses.
// ---------------------------------------------------------------------------
template <class O>
__global__ void __launch_bounds__(SPLIT_THREADS, O::UPDATE_BLOCKS) split_update_kernel(const __grid_constant__ typename O::Args a) {
  using R = typename O::R;
  using B = typename O::Base;
  last_launch_done();
  const int tt = __ldg(a.step_base) + a.step_off;
  if (tt >= a.step_end) return;
  const Geo& g = a.g;
  int n = blockIdx.x * SPLIT_THREADS + threadIdx.x;
  if (n >= a.off[6]) return;
  int c, i, j, k;
  const bool edge = update_point(a, g, n, c, i, j, k);
  Roles<R> r = roles<B>(a, tt);
  if constexpr (B::kahan) {
    r.v_in = r.v_out = a.vbase;
    r.c_in = r.c_out = a.cbase;
  }
  const unsigned o = (unsigned)g.o0 + (unsigned)i * (unsigned)g.sx + (unsigned)j * (unsigned)g.sy + (unsigned)k;
  const R* uc = r.cur(c);
  const R u = uc[o];
  // old values for the face points, read early: they are off the path of the update
  FacePoints<B, typename O::Args> faces(a, r, uc, c, i, j, k, tt, o, edge);
  if (edge) faces.read();
  R val, vn = R(0), cn = R(0);
  if (c == 0 || i >= 1) {
    const bool kz = k == 0;
    Pw<R> pw;
    if constexpr (B::kahan) pw = Pw<R>{r.v_in[c * r.fs + o], r.c_in[c * r.fs + o]};
    else pw = Pw<R>{r.old(c)[o], R(0)};
    const unsigned s0 = (unsigned)i % a.W, sp = s0 + 1 == a.W ? 0 : s0 + 1, sm = s0 == 0 ? a.W - 1 : s0 - 1;
    const unsigned ro = (unsigned)(j * a.tsy + k);
    const R *A = a.Ta + ro, *Bc = a.Tb + ro + s0 * a.tsx, *Bm = a.Tb + ro + sm * a.tsx;  // T4..T6 of planes i, i-1
    const R* Ac = A + s0 * a.tsx;
    const long long tc = a.tcs;
    const uint8_t* M = a.mat + g.mo0 + (long long)i * g.msx + (long long)j * g.msy + k;
    R d1, d2, d3;
    const typename O::D *ax, *ay, *az;
    int id;
    if (c == 0) {  // base_solver.py:441-447, 495-501
      d1 = B::sub(*(A + sp * a.tsx), Ac[0]);
      d2 = B::sub(Bc[2 * tc], *(Bc + 2 * tc - a.tsy));
      d3 = B::sub(Bc[tc], *(Bc + tc - 1));
      ax = a.fdx + (kz ? 0 : i), ay = a.sdy + (kz ? 0 : j - 1), az = a.sdz + (kz ? 0 : k - 1);
      id = M[g.msx];
    } else if (c == 1) {  // base_solver.py:449-455, 503-509
      d1 = B::sub(Bc[2 * tc], Bm[2 * tc]);
      d2 = B::sub(*(Ac + tc + a.tsy), Ac[tc]);
      d3 = B::sub(Bc[0], *(Bc - 1));
      ax = a.sdx + (kz ? 0 : i - 1), ay = a.fdy + (kz ? 0 : j), az = a.sdz + (kz ? 0 : k - 1);
      id = M[g.msy];
    } else {  // base_solver.py:457-463, 511-516: as written, :516 adds T3[..,1] undivided
      d1 = B::sub(Bc[tc], Bm[tc]);
      d2 = B::sub(Bc[0], *(Bc - a.tsy));
      d3 = B::sub(Ac[2 * tc + 1], Ac[2 * tc]);
      ax = a.sdx + (kz ? 0 : i - 1), ay = a.sdy + (kz ? 0 : j - 1);
      az = a.fdz + (kz ? (a.surface_mode == 0 ? -1 : 0) : k);
      id = kz ? M[0] : M[1];
    }
    const R dv = O::div3(a, d1, ldd(ax), d2, ldd(ay), d3, ldd(az));
    val = O::update(a, id, u, pw, dv, vn, cn);
    store_point<B>(r, c, o, val, vn, cn);
  } else {  // uy, uz at i = 0: not written by the reference, keeps its state
    val = u;
    r.out(c)[o] = u;
  }
  if (c == 2 && k == 0) record(a, tt, i, j, val);
  if (edge) faces.write(val);
}

template <class O>
static cudaError_t launch_pass(const void* args, bool stress, bool after_kernel, cudaStream_t st) {
  const typename O::Args& a = *(const typename O::Args*)args;
  if (!stress) return split_launch(split_update_kernel<O>, a, a.off[6], after_kernel, st);
  const long long points = (long long)(a.sb - a.sa) * a.dy1.d * a.dz1.d;
  if constexpr (O::SMALL) {
    if (points < 20000) return split_launch(split_stress_kernel<O, 6>, a, points, after_kernel, st, 6);
    if (points < 60000) return split_launch(split_stress_kernel<O, 2>, a, points, after_kernel, st, 2);
  }
  return split_launch(split_stress_kernel<O, 1>, a, points, after_kernel, st);
}

cudaError_t launch_split_f32(const void* args, bool stress, bool after_kernel, cudaStream_t st);

// one pass over the planes set in the arguments; precision as in phono.h;
// after_kernel: the launch before it on the stream is a pass of the same chunk
// of steps (nothing between the two changed a constant or the step counter)
cudaError_t launch_split(int precision, const void* args, bool stress, bool after_kernel, cudaStream_t st) {
  if (precision == 0) {
    if (((const LeapOps<false>::Args*)args)->shared) return launch_pass<LeapOps<true>>(args, stress, after_kernel, st);
    return launch_pass<LeapOps<false>>(args, stress, after_kernel, st);
  }
  if (precision == 2) {
    if (((const VelOps<true>::Args*)args)->soft) return launch_pass<VelOps<true>>(args, stress, after_kernel, st);
    return launch_pass<VelOps<false>>(args, stress, after_kernel, st);
  }
  return launch_split_f32(args, stress, after_kernel, st);
}

}  // namespace phono
