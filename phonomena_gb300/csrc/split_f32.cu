// The two-launch step in FP32 (small meshes): the passes of split_step.cu, with
// every constant (material rows, spacings, the step counter) read before the
// wait for the launch ahead, so that only the state's loads and the arithmetic
// remain behind it.  (The FP64 kernels need those registers for arithmetic.)
// us a step, plain launches with the constants read on the way, and now: 6.5 /
// 5.3 at 25x21x13 nodes, 7.0 / 5.7 at 41x41x21, 7.9 / 6.7 at 61x61x21 (with the
// next launch allowed from a block's start instead of its end 5.2 / 6.1 / 7.8).
#include "split_point.cuh"

namespace phono {

using F32Args = SplitArgs<float, float>;

// ---------------------------------------------------------------------------
// stresses of planes [sa, sb): one thread per node of [sa, sb) x [0, ny-1) x
// [0, nz-1).  Zero where the reference never writes (base_solver.py:329-433).
// ---------------------------------------------------------------------------
__global__ void __launch_bounds__(SPLIT_THREADS, 8) split_stress_f32_kernel(const __grid_constant__ F32Args a) {
  using R = float;
  using B = F32K;
  const Geo& g = a.g;
  const int nx = g.nx;
  int n = blockIdx.x * SPLIT_THREADS + threadIdx.x;
  const int q1 = fdiv(n, a.dz1), k = n - q1 * a.dz1.d;
  const int q2 = fdiv(q1, a.dy1), j = q1 - q2 * a.dy1.d;
  const int i = a.sa + q2;
  if (i >= a.sb) return;
  const int tt = __ldg(a.step_base) + a.step_off;
  const bool kz = k == 0;
  const int up = kz ? 0 : 1;  // shear moduli of T4, T5: one layer down, except in the z = 0 row
  const bool i_n = i >= 1 && i <= nx - 2, i_s = i <= nx - 2, j_n = j >= 1;
  // what no step changes: material rows and spacings (the z = 0 row's
  // substitutions are base_solver.py:408-433's; the arrays are padded)
  const uint8_t* M = a.mat + g.mo0 + (long long)i * g.msx + (long long)j * g.msy + k;
  const R* row = a.tab + 16 * M[0];
  const float4 r0 = __ldg(reinterpret_cast<const float4*>(row)), r1 = __ldg(reinterpret_cast<const float4*>(row) + 1);
  const R rn[9] = {r0.x, r0.y, r0.z, r0.w, r1.x, r1.y, r1.z, r1.w, __ldg(row + 8)};
  const R c4 = __ldg(a.tab + 16 * M[g.msy + up] + 9), c5 = __ldg(a.tab + 16 * M[g.msx + up] + 10),
          c6 = __ldg(a.tab + 16 * M[g.msx + g.msy] + 11);
  const R dx = __ldg(a.sdx + (kz ? 0 : i - 1)), dy = __ldg(a.sdy + (kz ? 0 : j - 1)), dz = __ldg(a.sdz + (kz ? 0 : k - 1));
  const R a4 = __ldg(kz ? a.fdy : a.fdz + k), b4 = __ldg(kz ? a.fdz : a.fdy + j), a5 = __ldg(kz ? a.fdx : a.fdz + k),
          b5 = __ldg(kz ? a.fdz : a.fdx + i), a6 = __ldg(kz ? a.fdx : a.fdy + j);
  const R src = (R)__ldg(a.src + tt);
  const Roles<R> r = roles<B>(a, tt);
  const unsigned sx = (unsigned)g.sx, sy = (unsigned)g.sy;
  const unsigned o = (unsigned)g.o0 + (unsigned)i * sx + (unsigned)j * sy + (unsigned)k;
  const R *X = r.u_cur + o, *Y = X + r.fs, *Z = Y + r.fs;
  last_launch_done();
  if (tt >= a.step_end) return;
  const R x0 = X[0], y0 = Y[0];
  const R x_k = X[1], x_j = X[sy], y_k = Y[1], y_i = Y[sx], z_j = Z[sy], z_i = Z[sx];
  R z0 = Z[0];
  if (i == 0 && (a.source_mode == 1 || kz)) z0 = src;  // source overwrite (base_solver.py:251)
  R t[6] = {R(0), R(0), R(0), R(0), R(0), R(0)};
  if (i_n && j_n) {
    const R d1 = B::sub(x0, *(X - sx)), d2 = B::sub(y0, *(Y - sy)), d3 = B::sub(z0, Z[-1]);
    for (int q = 0; q < 3; q++) t[q] = B::tn1(a.dtab, rn + 3 * q, d1, d2, d3, dx, dy, dz);
  }
  if (kz) t[2] = R(0);  // base_solver.py:418
  if (i_n) t[3] = B::ts(a.dtab, c4, B::sub(y_k, y0), a4, B::sub(z_j, z0), b4);
  if (i_s && j_n) t[4] = B::ts(a.dtab, c5, B::sub(x_k, x0), a5, B::sub(z_i, z0), b5);
  if (i_s) t[5] = B::ts(a.dtab, c6, B::sub(x_j, x0), a6, B::sub(y_i, y0), b5);
  const unsigned to = (unsigned)i * a.tsx + (unsigned)(j * a.tsy + k);
#pragma unroll
  for (int c = 0; c < 3; c++) {
    a.Ta[to + c * a.tcs] = t[c];
    a.Tb[to + c * a.tcs] = t[c + 3];
  }
}

// ---------------------------------------------------------------------------
// new state of planes [pa, pb): one thread per point of each component that is
// on no face, with the face points next to it; v and the Kahan term in place
// ---------------------------------------------------------------------------
__global__ void __launch_bounds__(SPLIT_THREADS, 7) split_update_f32_kernel(const __grid_constant__ F32Args a) {
  using R = float;
  using B = F32K;
  const Geo& g = a.g;
  int n = blockIdx.x * SPLIT_THREADS + threadIdx.x;
  if (n >= a.off[6]) return;
  const int tt = __ldg(a.step_base) + a.step_off;
  int c, i, j, k;
  const bool edge = update_point(a, g, n, c, i, j, k);
  Roles<R> r = roles<B>(a, tt);
  r.v_in = r.v_out = a.vbase;
  r.c_in = r.c_out = a.cbase;
  const unsigned o = (unsigned)g.o0 + (unsigned)i * (unsigned)g.sx + (unsigned)j * (unsigned)g.sy + (unsigned)k;
  const R* uc = r.cur(c);
  // what no step changes (the arrays are padded; as written, base_solver.py:516
  // adds T3[..,1] undivided)
  const bool kz = k == 0;
  const uint8_t* M = a.mat + g.mo0 + (long long)i * g.msx + (long long)j * g.msy + k;
  const R rq = __ldg(a.tab + 16 * (c == 0 ? M[g.msx] : c == 1 ? M[g.msy] : kz ? M[0] : M[1]) + 12);
  const R dx = __ldg(c == 0 ? a.fdx + (kz ? 0 : i) : a.sdx + (kz ? 0 : i - 1));
  const R dy = __ldg(c == 1 ? a.fdy + (kz ? 0 : j) : a.sdy + (kz ? 0 : j - 1));
  const R dz = __ldg(c == 2 ? a.fdz + (kz ? (a.surface_mode == 0 ? -1 : 0) : k) : a.sdz + (kz ? 0 : k - 1));
  last_launch_done();
  if (tt >= a.step_end) return;
  const R u = uc[o];
  // old values for the face points, read early: they are off the path of the update
  FacePoints<B, F32Args> faces(a, r, uc, c, i, j, k, tt, o, edge);
  if (edge) faces.read();
  R val, vn = R(0), cn = R(0);
  if (c == 0 || i >= 1) {
    const Pw<R> pw{r.v_in[c * r.fs + o], r.c_in[c * r.fs + o]};
    const unsigned s0 = (unsigned)i, sp = s0 + 1, sm = s0 - 1;  // the window holds the whole mesh
    const unsigned ro = (unsigned)(j * a.tsy + k);
    const R *A = a.Ta + ro, *Bc = a.Tb + ro + s0 * a.tsx, *Bm = a.Tb + ro + sm * a.tsx;  // T4..T6 of planes i, i-1
    const R* Ac = A + s0 * a.tsx;
    const long long tc = a.tcs;
    R d1, d2, d3;
    if (c == 0) {  // base_solver.py:441-447, 495-501
      d1 = B::sub(*(A + sp * a.tsx), Ac[0]);
      d2 = B::sub(Bc[2 * tc], *(Bc + 2 * tc - a.tsy));
      d3 = B::sub(Bc[tc], *(Bc + tc - 1));
    } else if (c == 1) {  // base_solver.py:449-455, 503-509
      d1 = B::sub(Bc[2 * tc], Bm[2 * tc]);
      d2 = B::sub(*(Ac + tc + a.tsy), Ac[tc]);
      d3 = B::sub(Bc[0], *(Bc - 1));
    } else {  // base_solver.py:457-463, 511-516
      d1 = B::sub(Bc[tc], Bm[tc]);
      d2 = B::sub(Bc[0], *(Bc - a.tsy));
      d3 = B::sub(Ac[2 * tc + 1], Ac[2 * tc]);
    }
    val = update_value<B>(u, pw, B::div3(a.dtab, d1, dx, d2, dy, d3, dz), rq, a.dt, vn, cn);
    store_point<B>(r, c, o, val, vn, cn);
  } else {  // uy, uz at i = 0: not written by the reference, keeps its state
    val = u;
    r.out(c)[o] = u;
  }
  if (c == 2 && k == 0) record(a, tt, i, j, val);
  if (edge) faces.write(val);
}

cudaError_t launch_split_f32(const void* args, bool stress, bool after_kernel, cudaStream_t st) {
  const F32Args& a = *(const F32Args*)args;
  return stress ? split_launch(split_stress_f32_kernel, a, (long long)(a.sb - a.sa) * a.dy1.d * a.dz1.d, after_kernel, st)
                : split_launch(split_update_f32_kernel, a, a.off[6], after_kernel, st);
}

}  // namespace phono
