// Arithmetic schemes, addressing and pointwise operations shared by the step
// kernels (fdtd_step.cu, split_step.cu).
#pragma once
#include "fdtd_common.cuh"

namespace phono {

// ---------------------------------------------------------------------------
// arithmetic schemes
// ---------------------------------------------------------------------------
struct F64 {
  using R = double;
  static constexpr bool kahan = false;
  __device__ __forceinline__ static R sub(R a, R b) { return __dsub_rn(a, b); }
  // x / b with IEEE rounding, through the divisor table when the handle has one
  __device__ __forceinline__ static R dv(const DivTable& k, R x, R b) { return k.tab ? div_tab(x, b, k) : __ddiv_rn(x, b); }
  // normal stresses ((C0*d1)/a + (C1*d2)/b) + (C2*d3)/d   (base_solver.py:329-351)
  __device__ __forceinline__ static R tn1(const DivTable& k, const R* c, R d1, R d2, R d3, R a, R b, R d) {
    return __dadd_rn(__dadd_rn(dv(k, __dmul_rn(c[0], d1), a), dv(k, __dmul_rn(c[1], d2), b)),
                     dv(k, __dmul_rn(c[2], d3), d));
  }
  // shear stress C * (d1/a + d2/b)   (base_solver.py:353-372)
  __device__ __forceinline__ static R ts(const DivTable& k, R cs, R d1, R a, R d2, R b) {
    return __dmul_rn(cs, __dadd_rn(dv(k, d1, a), dv(k, d2, b)));
  }
  // (d1/a + d2/b) + d3/c   (base_solver.py:444-446)
  __device__ __forceinline__ static R div3(const DivTable& k, R d1, R a, R d2, R b, R d3, R c) {
    return __dadd_rn(__dadd_rn(dv(k, d1, a), dv(k, d2, b)), dv(k, d3, c));
  }
  // uz z=0 row as written at base_solver.py:516: ((d1/a + d2/b) + T3[..,1]) - T3[..,0]/fdz
  // with T3[..,0] == +0, so the last subtraction is exact and dropped.
  __device__ __forceinline__ static R div_surf_ref(const DivTable& k, R d1, R a, R d2, R b, R t31) {
    return __dadd_rn(__dadd_rn(dv(k, d1, a), dv(k, d2, b)), t31);
  }
  // u[b-+1] + c * (u_new[b-+1] - u[b])   (base_solver.py:540-554)
  __device__ __forceinline__ static R abc(R coef, R nbr_new, R self_old, R nbr_old) {
    return __dadd_rn(nbr_old, __dmul_rn(coef, __dsub_rn(nbr_new, self_old)));
  }
};

struct F32K {
  using R = float;
  static constexpr bool kahan = true;
  __device__ __forceinline__ static R sub(R a, R b) { return __fsub_rn(a, b); }
  // strains e = d * (1/spacing); T = fmaf(C0, e1, fmaf(C1, e2, C2 * e3))
  __device__ __forceinline__ static R tn1(const DivTable&, const R* c, R d1, R d2, R d3, R a, R b, R d) {
    return __fmaf_rn(c[0], __fmul_rn(d1, a), __fmaf_rn(c[1], __fmul_rn(d2, b), __fmul_rn(c[2], __fmul_rn(d3, d))));
  }
  __device__ __forceinline__ static R ts(const DivTable&, R cs, R d1, R a, R d2, R b) {
    return __fmul_rn(cs, __fmaf_rn(d1, a, __fmul_rn(d2, b)));
  }
  __device__ __forceinline__ static R div3(const DivTable&, R d1, R a, R d2, R b, R d3, R c) {
    return __fmaf_rn(d1, a, __fmaf_rn(d2, b, __fmul_rn(d3, c)));
  }
  // reference-precedence z = 0 row: T3[..,1] as the third term with factor 1
  __device__ __forceinline__ static R div_surf_ref(const DivTable& k, R d1, R a, R d2, R b, R t31) {
    return div3(k, d1, a, d2, b, t31, 1.0f);
  }
  __device__ __forceinline__ static R abc(R coef, R nbr_new, R self_old, R nbr_old) {
    return __fmaf_rn(coef, __fsub_rn(nbr_new, self_old), nbr_old);
  }
  __device__ __forceinline__ static R fma(R a, R b, R c) { return __fmaf_rn(a, b, c); }
  __device__ __forceinline__ static R add(R a, R b) { return __fadd_rn(a, b); }
};

// The F32K scheme carried out in FP64: the fast FP64 reference for judging
// the FP32 error (same operation sequence, double rounding).
struct F64V {
  using R = double;
  static constexpr bool kahan = true;
  __device__ __forceinline__ static R sub(R a, R b) { return __dsub_rn(a, b); }
  __device__ __forceinline__ static R tn1(const DivTable&, const R* c, R d1, R d2, R d3, R a, R b, R d) {
    return __fma_rn(c[0], __dmul_rn(d1, a), __fma_rn(c[1], __dmul_rn(d2, b), __dmul_rn(c[2], __dmul_rn(d3, d))));
  }
  __device__ __forceinline__ static R ts(const DivTable&, R cs, R d1, R a, R d2, R b) {
    return __dmul_rn(cs, __fma_rn(d1, a, __dmul_rn(d2, b)));
  }
  __device__ __forceinline__ static R div3(const DivTable&, R d1, R a, R d2, R b, R d3, R c) {
    return __fma_rn(d1, a, __fma_rn(d2, b, __dmul_rn(d3, c)));
  }
  __device__ __forceinline__ static R div_surf_ref(const DivTable& k, R d1, R a, R d2, R b, R t31) {
    return div3(k, d1, a, d2, b, t31, 1.0);
  }
  __device__ __forceinline__ static R abc(R coef, R nbr_new, R self_old, R nbr_old) {
    return __fma_rn(coef, __dsub_rn(nbr_new, self_old), nbr_old);
  }
  __device__ __forceinline__ static R fma(R a, R b, R c) { return __fma_rn(a, b, c); }
  __device__ __forceinline__ static R add(R a, R b) { return __dadd_rn(a, b); }
};

// ---------------------------------------------------------------------------
// addressing
// ---------------------------------------------------------------------------
__device__ __forceinline__ long long fidx(const Geo& g, int i, int j, int k) {
  return g.o0 + (long long)i * g.sx + (long long)j * g.sy + k;
}

// component extents and face coordinates
__device__ __forceinline__ int ext_x(const Geo& g, int c) { return g.nx - (c == 0); }
__device__ __forceinline__ int ext_y(const Geo& g, int c) { return g.ny - (c == 1); }
__device__ __forceinline__ int ext_z(const Geo& g, int c) { return g.nz - (c == 2); }
// points the reference's interior update or z=0 row writes
// (base_solver.py:441-463,495-516)
__device__ __forceinline__ bool in_v0(const Geo& g, int c, int i, int j, int k) {
  if (c == 0) return j >= 1 && j <= g.ny - 2 && k >= 0 && k <= g.nz - 2;
  if (c == 1) return i >= 1 && i <= g.nx - 2 && k >= 0 && k <= g.nz - 2;
  return i >= 1 && i <= g.nx - 2 && j >= 1 && j <= g.ny - 2;
}

// ---------------------------------------------------------------------------
// stress at a point, given a fetcher F: x/y/z(i,j,k) -> u, row(i,j,k) -> the
// 16-entry material row.  Zero wherever the reference never writes the
// stress array.
// ---------------------------------------------------------------------------
template <class S, class F>
__device__ __forceinline__ typename S::R t1_at(const StepArgs<typename S::R>& a, const F& f, int i, int j, int k,
                                               int which) {  // which: 0 T1, 1 T2, 2 T3
  using R = typename S::R;
  const Geo& g = a.g;
  if (i < 1 || i > g.nx - 2 || j < 1 || j > g.ny - 2 || k < 0 || k > g.nz - 2) return R(0);
  if (k == 0 && which == 2) return R(0);  // T3[1:-1,1:-1,0] = 0 (base_solver.py:418)
  const R* c = f.row(i, j, k) + 3 * which;
  R d1 = S::sub(f.x(i, j, k), f.x(i - 1, j, k));
  R d2 = S::sub(f.y(i, j, k), f.y(i, j - 1, k));
  if (k == 0)  // base_solver.py:408-416: uz - 0, first-element spacings
    return S::tn1(a.dtab, c, d1, d2, f.z(i, j, 0), a.sp.sdx0, a.sp.sdy0, a.sp.sdz0);
  return S::tn1(a.dtab, c, d1, d2, S::sub(f.z(i, j, k), f.z(i, j, k - 1)), __ldg(a.sp.sdx + i - 1),
                __ldg(a.sp.sdy + j - 1), __ldg(a.sp.sdz + k - 1));
}

template <class S, class F>
__device__ __forceinline__ void t123_at(const StepArgs<typename S::R>& a, const F& f, int i, int j, int k,
                                        typename S::R& T1, typename S::R& T2, typename S::R& T3) {
  using R = typename S::R;
  const Geo& g = a.g;
  if (i < 1 || i > g.nx - 2 || j < 1 || j > g.ny - 2 || k < 0 || k > g.nz - 2) {
    T1 = T2 = T3 = R(0);
    return;
  }
  const R* c = f.row(i, j, k);
  R d1 = S::sub(f.x(i, j, k), f.x(i - 1, j, k));
  R d2 = S::sub(f.y(i, j, k), f.y(i, j - 1, k));
  if (k == 0) {
    R d3 = f.z(i, j, 0);
    T1 = S::tn1(a.dtab, c, d1, d2, d3, a.sp.sdx0, a.sp.sdy0, a.sp.sdz0);
    T2 = S::tn1(a.dtab, c + 3, d1, d2, d3, a.sp.sdx0, a.sp.sdy0, a.sp.sdz0);
    T3 = R(0);
  } else {
    R d3 = S::sub(f.z(i, j, k), f.z(i, j, k - 1));
    R sa = __ldg(a.sp.sdx + i - 1), sb = __ldg(a.sp.sdy + j - 1), sd = __ldg(a.sp.sdz + k - 1);
    T1 = S::tn1(a.dtab, c, d1, d2, d3, sa, sb, sd);
    T2 = S::tn1(a.dtab, c + 3, d1, d2, d3, sa, sb, sd);
    T3 = S::tn1(a.dtab, c + 6, d1, d2, d3, sa, sb, sd);
  }
}

template <class S, class F>
__device__ __forceinline__ typename S::R t4_at(const StepArgs<typename S::R>& a, const F& f, int i, int j, int k) {
  using R = typename S::R;
  const Geo& g = a.g;
  if (i < 1 || i > g.nx - 2 || j < 0 || j > g.ny - 2 || k < 0 || k > g.nz - 2) return R(0);
  if (k == 0)  // base_solver.py:420-423
    return S::ts(a.dtab, f.row(i, j + 1, 0)[9], S::sub(f.y(i, j, 1), f.y(i, j, 0)), a.sp.fdy0,
                 S::sub(f.z(i, j + 1, 0), f.z(i, j, 0)), a.sp.fdz0);
  return S::ts(a.dtab, f.row(i, j + 1, k + 1)[9], S::sub(f.y(i, j, k + 1), f.y(i, j, k)), __ldg(a.sp.fdz + k),
               S::sub(f.z(i, j + 1, k), f.z(i, j, k)), __ldg(a.sp.fdy + j));
}

template <class S, class F>
__device__ __forceinline__ typename S::R t5_at(const StepArgs<typename S::R>& a, const F& f, int i, int j, int k) {
  using R = typename S::R;
  const Geo& g = a.g;
  if (i < 0 || i > g.nx - 2 || j < 1 || j > g.ny - 2 || k < 0 || k > g.nz - 2) return R(0);
  if (k == 0)  // base_solver.py:425-428
    return S::ts(a.dtab, f.row(i + 1, j, 0)[10], S::sub(f.x(i, j, 1), f.x(i, j, 0)), a.sp.fdx0,
                 S::sub(f.z(i + 1, j, 0), f.z(i, j, 0)), a.sp.fdz0);
  return S::ts(a.dtab, f.row(i + 1, j, k + 1)[10], S::sub(f.x(i, j, k + 1), f.x(i, j, k)), __ldg(a.sp.fdz + k),
               S::sub(f.z(i + 1, j, k), f.z(i, j, k)), __ldg(a.sp.fdx + i));
}

template <class S, class F>
__device__ __forceinline__ typename S::R t6_at(const StepArgs<typename S::R>& a, const F& f, int i, int j, int k) {
  using R = typename S::R;
  const Geo& g = a.g;
  if (i < 0 || i > g.nx - 2 || j < 0 || j > g.ny - 2 || k < 0 || k > g.nz - 2) return R(0);
  if (k == 0)  // base_solver.py:430-433
    return S::ts(a.dtab, f.row(i + 1, j + 1, 0)[11], S::sub(f.x(i, j + 1, 0), f.x(i, j, 0)), a.sp.fdx0,
                 S::sub(f.y(i + 1, j, 0), f.y(i, j, 0)), a.sp.fdz0);
  return S::ts(a.dtab, f.row(i + 1, j + 1, k)[11], S::sub(f.x(i, j + 1, k), f.x(i, j, k)), __ldg(a.sp.fdy + j),
               S::sub(f.y(i + 1, j, k), f.y(i, j, k)), __ldg(a.sp.fdx + i));
}

// divergence terms of the three components (base_solver.py:441-463,495-516)
// and the material row whose density applies
template <class S, class F>
__device__ __forceinline__ typename S::R div_x(const StepArgs<typename S::R>& a, const F& f, int i, int j, int k,
                                               typename S::R t1p, typename S::R t1m, typename S::R t6a,
                                               typename S::R t6b, typename S::R t5a, typename S::R t5b,
                                               const typename S::R*& row) {
  if (k == 0) {
    row = f.row(i + 1, j, 0);
    return S::div3(a.dtab, S::sub(t1p, t1m), a.sp.fdx0, S::sub(t6a, t6b), a.sp.sdy0, t5a, a.sp.sdz0);
  }
  row = f.row(i + 1, j, k);
  return S::div3(a.dtab, S::sub(t1p, t1m), __ldg(a.sp.fdx + i), S::sub(t6a, t6b), __ldg(a.sp.sdy + j - 1),
                 S::sub(t5a, t5b), __ldg(a.sp.sdz + k - 1));
}
template <class S, class F>
__device__ __forceinline__ typename S::R div_y(const StepArgs<typename S::R>& a, const F& f, int i, int j, int k,
                                               typename S::R t6a, typename S::R t6b, typename S::R t2p,
                                               typename S::R t2m, typename S::R t4a, typename S::R t4b,
                                               const typename S::R*& row) {
  if (k == 0) {
    row = f.row(i, j + 1, 0);
    return S::div3(a.dtab, S::sub(t6a, t6b), a.sp.sdx0, S::sub(t2p, t2m), a.sp.fdy0, t4a, a.sp.sdz0);
  }
  row = f.row(i, j + 1, k);
  return S::div3(a.dtab, S::sub(t6a, t6b), __ldg(a.sp.sdx + i - 1), S::sub(t2p, t2m), __ldg(a.sp.fdy + j),
                 S::sub(t4a, t4b), __ldg(a.sp.sdz + k - 1));
}
template <class S, class F>
__device__ __forceinline__ typename S::R div_z(const StepArgs<typename S::R>& a, const F& f, int i, int j, int k,
                                               typename S::R t5a, typename S::R t5b, typename S::R t4a,
                                               typename S::R t4b, typename S::R t3p, typename S::R t3m,
                                               const typename S::R*& row) {
  if (k == 0) {
    row = f.row(i, j, 0);  // density at z index 0 (base_solver.py:513)
    if (a.surface_mode == 0) return S::div_surf_ref(a.dtab, S::sub(t5a, t5b), a.sp.sdx0, S::sub(t4a, t4b), a.sp.sdy0, t3p);
    return S::div3(a.dtab, S::sub(t5a, t5b), a.sp.sdx0, S::sub(t4a, t4b), a.sp.sdy0, t3p, a.sp.fdz0);
  }
  row = f.row(i, j, k + 1);
  return S::div3(a.dtab, S::sub(t5a, t5b), __ldg(a.sp.sdx + i - 1), S::sub(t4a, t4b), __ldg(a.sp.sdy + j - 1),
                 S::sub(t3p, t3m), __ldg(a.sp.fdz + k));
}

// state arrays of global step tt: buffer indices, pointers formed on use
// (no pointer arrays, which would live in local memory)
template <class R>
struct Roles {
  // component-0 array of each role (component c at + c * fs), set once per
  // launch: an access is the point's offset added to a block-uniform base
  R *u_cur, *u_old, *u_out, *v_in, *v_out, *c_in, *c_out;
  long long fs;
  int rold, rcur, rout;  // buffer indices: u at tt-1 (F64), tt, tt+1
  __device__ __forceinline__ const R* cur(int c) const { return u_cur + c * fs; }
  __device__ __forceinline__ const R* old(int c) const { return u_old + c * fs; }
  __device__ __forceinline__ R* out(int c) const { return u_out + c * fs; }
  __device__ __forceinline__ const R* vin(int c) const { return v_in + c * fs; }
  __device__ __forceinline__ const R* cin(int c) const { return c_in + c * fs; }
  __device__ __forceinline__ R* vout(int c) const { return v_out + c * fs; }
  __device__ __forceinline__ R* cout(int c) const { return c_out + c * fs; }
};

template <class S, class A>
__device__ __forceinline__ Roles<typename S::R> roles(const A& a, int tt) {
  Roles<typename S::R> r;
  r.fs = a.g.fstride;
  if (!S::kahan) {
    r.rold = tt % 3;
    r.rcur = (tt + 1) % 3;
    r.rout = (tt + 2) % 3;
  } else {
    r.rcur = tt & 1;
    r.rout = r.rcur ^ 1;
    r.rold = r.rcur;
  }
  const long long f3 = 3 * r.fs;
  r.u_cur = a.ubase + r.rcur * f3;
  r.u_old = a.ubase + r.rold * f3;
  r.u_out = a.ubase + r.rout * f3;
  r.v_in = a.vbase + r.rcur * f3;
  r.v_out = a.vbase + r.rout * f3;
  r.c_in = a.cbase + r.rcur * f3;
  r.c_out = a.cbase + r.rout * f3;
  return r;
}

// pointwise state of a V0 point that the update needs besides u itself
template <class R>
struct Pw {
  R p0, p1;  // F64: u_old, -; F32K: v, c
};

template <class S>
__device__ __forceinline__ Pw<typename S::R> load_pw(const Roles<typename S::R>& r, int c, long long off) {
  Pw<typename S::R> p;
  if constexpr (!S::kahan) {
    p.p0 = __ldg(r.old(c) + off);
    p.p1 = 0;
  } else {
    p.p0 = __ldg(r.vin(c) + off);
    p.p1 = __ldg(r.cin(c) + off);
  }
  return p;
}

// new state of one V0 point: F64 leapfrog / F32K Kahan velocity update.
// q = the table's column 12 at the point (dt^2/P or dt/P), dt = column 14.
template <class S>
__device__ __forceinline__ typename S::R update_value(typename S::R u, Pw<typename S::R> pw, typename S::R dv,
                                                      typename S::R q, typename S::R dt, typename S::R& vn,
                                                      typename S::R& cn) {
  using R = typename S::R;
  if constexpr (!S::kahan) {
    // (2u - u_old) + (dt^2/P) * div   (base_solver.py:441-443)
    vn = cn = 0;
    return __dadd_rn(__dsub_rn(__dmul_rn(2.0, u), pw.p0), __dmul_rn(q, dv));
  } else {
    R v2 = S::fma(q, dv, pw.p0);   // v + (dt/P) div
    R y = S::fma(dt, v2, -pw.p1);  // dt v - c
    R t = S::add(u, y);
    cn = S::sub(S::sub(t, u), y);
    vn = v2;
    return t;
  }
}
template <class S>
__device__ __forceinline__ typename S::R update_value(typename S::R u, Pw<typename S::R> pw, typename S::R dv,
                                                      const typename S::R* row, typename S::R& vn,
                                                      typename S::R& cn) {
  return update_value<S>(u, pw, dv, row[12], row[14], vn, cn);
}

// OFF: element offset inside one array; the tile path passes a 32-bit
// unsigned offset (one multiply-add per address), the face path 64-bit
template <class S, class OFF>
__device__ __forceinline__ void store_point(const Roles<typename S::R>& r, int c, OFF off, typename S::R un,
                                            typename S::R vn, typename S::R cn) {
  r.out(c)[off] = un;
  if constexpr (S::kahan) {
    r.vout(c)[off] = vn;
    r.cout(c)[off] = cn;
  }
}

// a point the reference does not write this step keeps its state; returns u
template <class S, class OFF>
__device__ __forceinline__ typename S::R store_stale(const Roles<typename S::R>& r, int c, OFF off) {
  const typename S::R u = __ldg(r.cur(c) + off);
  r.out(c)[off] = u;
  if constexpr (S::kahan) {
    r.vout(c)[off] = __ldg(r.vin(c) + off);
    r.cout(c)[off] = __ldg(r.cin(c) + off);
  }
  return u;
}

template <class A, class R>
__device__ __forceinline__ void record(const A& a, int tt, int i, int j, R val) {
  if (a.record_every > 0 && (tt + 1) % a.record_every == 0) {
    int slot = (tt + 1) / a.record_every - 1 - a.rec_base;
    if (slot >= 0 && slot < a.nrec_cap) a.surf[((long long)slot * a.g.nx + i) * a.g.ny + j] = val;
  }
  if (!isfinite(val)) atomicOr(a.err, 1);
}

// Programmatic launches: a launch may start (its index arithmetic and reads of
// constants: material rows, spacings, the step counter, which changes between
// chunks of launches only) once the blocks of the one ahead have ended or let
// it, and waits here until that is complete before it touches the state.  The
// state is read with plain loads from then on: it is not read-only over such a
// launch's lifetime, as the non-coherent loads (__ldg) would need.  A block
// that has nothing to do waits too: the launch behind it relies on this one
// for all that came before.
__device__ __forceinline__ void last_launch_done() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
__device__ __forceinline__ void let_next_launch() { asm volatile("griddepcontrol.launch_dependents;"); }

}  // namespace phono
