// Device parts shared by the two-launch kernels (split_step.cu, split_f32.cu).
#pragma once
#include "scheme.cuh"
#include "split_common.cuh"

namespace phono {

__device__ __forceinline__ float ldd(const float* p) { return __ldg(p); }
__device__ __forceinline__ double ldd(const double* p) { return __ldg(p); }
__device__ __forceinline__ SoftRec ldd(const SoftRec* p) {
  const uint4 v = __ldg(reinterpret_cast<const uint4*>(p));
  return SoftRec{v.x, v.y, v.z, v.w};
}

// (a caller that uses one part loads that part alone)
__device__ __forceinline__ SoftFactor ldd(const SoftFactor* p) { return SoftFactor{ldd(&p->rec), ldd(&p->v), 0.0}; }

__device__ __forceinline__ int fdiv(int n, const FastDiv& f) { return (int)(__umulhi(2u * (unsigned)n, f.mult) >> f.shift); }

// point n of an update launch: component and indices; whether it is next to a face
template <class A>
__device__ __forceinline__ bool update_point(const A& a, const Geo& g, int n, int& c, int& i, int& j, int& k) {
  const bool edge = n < a.off[3];
  if (!edge) {
    c = (n >= a.off[4]) + (n >= a.off[5]);
    n -= a.off[3 + c];
    const FastDiv fz = a.uz_[c], fy = a.uy_[c];
    const int q1 = fdiv(n, fz), q2 = fdiv(q1, fy);
    k = n - q1 * fz.d, j = q1 - q2 * fy.d + 2, i = a.pa + q2;
  } else {  // points next to a face: per plane the rows j = 1 and jN-1, then the rest of k = kN-1
    c = (n >= a.off[1]) + (n >= a.off[2]);
    n -= a.off[c];
    const int xi = ext_x(g, c) - 1, nj = ext_y(g, c) - 2, nk = ext_z(g, c) - 1, rows = min(nj, 2) * nk;
    const int planes = max(min(a.pb, xi - 1) - a.pa, 0);
    i = fdiv(n, a.per[c]);
    if (i < planes) {
      n -= i * a.per[c].d;
      i += a.pa;
      if (n < nk) j = 1, k = n;
      else if (n < rows) j = nj, k = n - nk;
      else j = 2 + n - rows, k = nk - 1;
    } else {  // the plane next to x = N: all of it
      n -= planes * a.per[c].d;
      i = xi - 1;
      j = fdiv(n, a.nk[c]);
      k = n - j++ * nk;
    }
  }
  return edge;
}

// The face points whose chain of face formulas (base_solver.py:540-554) starts
// at a point: x = N first, then y = 0 or N, then z = N.
template <class B, class A>
struct FacePoints {
  using R = typename B::R;
  const A& a;
  const Roles<R>& r;
  const R* uc;
  int c, i, j, k, tt, nfx, nfz, fj;
  unsigned o;
  bool two_y;
  R old[8];  // old values of the up to 2 x 2 x 2 points they span, [z][y][x]

  __device__ __forceinline__ FacePoints(const A& a_, const Roles<R>& r_, const R* uc_, int c_, int i_, int j_, int k_, int tt_,
                                        unsigned o_, bool edge)
      : a(a_), r(r_), uc(uc_), c(c_), i(i_), j(j_), k(k_), tt(tt_), o(o_) {
    const Geo& g = a.g;
    nfx = edge && i == ext_x(g, c) - 2, nfz = edge && k == ext_z(g, c) - 2;
    fj = !edge ? 0 : j == 1 ? -1 : j == ext_y(g, c) - 2 ? 1 : 0;
    two_y = fj < 0 && j == ext_y(g, c) - 2;
  }
  __device__ __forceinline__ unsigned at(bool fx, bool fy, bool fk) const {
    return o + (fx ? (unsigned)a.g.sx : 0u) + (fy ? (unsigned)(fj * (int)a.g.sy) : 0u) + (fk ? 1u : 0u);
  }
  __device__ __forceinline__ void read() {
    const R s = (R)__ldg(a.src + tt);
#pragma unroll
    for (int q = 0; q < 8; q++) {
      const bool fx = q & 1, fy = q & 2, fk = q & 4;
      if ((fx && !nfx) || (fy && !fj) || (fk && !nfz)) continue;
      old[q] = uc[at(fx, fy, fk)];
      if (c == 2 && i == 0 && !fx && (a.source_mode == 1 || (k == 0 && !fk))) old[q] = s;  // source overwrite (base_solver.py:251)
    }
  }
  __device__ __forceinline__ void write(R val) {
    for (;;) {
      R w[8];
      w[0] = val;
#pragma unroll
      for (int q = 1; q < 8; q++) {
        const bool fx = q & 1, fy = q & 2, fk = q & 4;
        if ((fx && !nfx) || (fy && !fj) || (fk && !nfz)) continue;
        const int from = q & (fk ? 3 : fy ? 1 : 0);
        const R f = fk ? (c == 2 ? a.abc[7] : a.abc[6])
                       : !fy ? (c == 0 ? a.abc[0] : a.abc[1])
                             : fj < 0 ? (c == 1 ? a.abc[3] : a.abc[2]) : (c == 1 ? a.abc[5] : a.abc[4]);
        w[q] = a.bc == 1 ? R(0) : B::abc(f, w[from], old[q], old[from]);
        store_point<B>(r, c, at(fx, fy, fk), w[q], R(0), R(0));
        if (c == 2 && k == 0 && !fk) record(a, tt, i + fx, fy ? j + fj : j, w[q]);
      }
      if (!two_y || fj > 0) break;
      fj = 1;  // a single row between the two y faces
      read();
    }
  }
};

// the stress or update launch of the planes set in the arguments
template <class F, class A>
inline cudaError_t split_launch(F* kernel, const A& a, long long points, bool after_kernel, cudaStream_t st,
                                int parts = 1) {
  if (points <= 0) return cudaSuccess;
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = dim3((unsigned)((points + SPLIT_THREADS - 1) / SPLIT_THREADS), (unsigned)parts);
  cfg.blockDim = dim3(SPLIT_THREADS);
  cfg.stream = st;
  cudaLaunchAttribute at{};
  at.id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at.val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = &at;
  cfg.numAttrs = after_kernel ? 1 : 0;
  return cudaLaunchKernelEx(&cfg, kernel, a);
}

}  // namespace phono
