// Arguments of the two-launch step (split_step.cu), shared with the C ABI.
#pragma once
#include "fdtd_common.cuh"
#include "soft_f64.cuh"

namespace phono {

constexpr int SPLIT_THREADS = 128;
constexpr int SPLIT_KOFF = 4;     // front pad of a stress row of the leapfrog's window: k = -1 reads zero
constexpr int SPLIT_BEHIND = 3;   // planes behind a chunk that its update pass still reads

// n / d for 0 <= n < 2^31, d >= 1: umulhi(2n, mult) >> shift with
// mult = floor(2^(31+shift) / d) + 1 and shift = ceil(log2 d)
struct FastDiv {
  unsigned mult;
  int shift, d;
};
inline FastDiv fast_div(int d) {
  int s = 0;
  while ((1ll << s) < d) s++;
  return FastDiv{(unsigned)((1ull << (31 + s)) / (unsigned)d + 1), s, d};
}

// a factor with its record (soft_f64.cuh)
struct alignas(16) SoftFactor {
  SoftRec rec;
  double v, unused;
};

// R: element type; D: divisor as the scheme uses it (FP32: reciprocal; FP64
// velocity form: reciprocal with its record; leapfrog: record).  Spacing
// arrays carry the value 1 at index -1 and two after the end.
template <class R, class D>
struct SplitArgs {
  Geo g;
  const D *fdx, *fdy, *fdz, *sdx, *sdy, *sdz;
  const uint8_t* mat;
  const R* tab;          // velocity forms: 16 entries per material id
  const SoftRec* rec;    // FP64: the same entries as records
  const double* vals;    // leapfrog: values of the records (fallback division)
  int shared;            // leapfrog: c10 = c20, c01 = c21, c02 = c12 in every material
  int soft;              // FP64 velocity form: products in integer arithmetic
  DivTable dtab;
  const double* src;
  R *ubase, *vbase, *cbase;
  R abc[8];
  R dt;
  R* surf;
  int record_every, rec_base, nrec_cap;
  const int* step_base;
  int step_off, step_end;
  int surface_mode, bc, source_mode;
  int* err;
  // stress window: W planes (plane p in slot p % W) of rows of tsy elements;
  // component q at Ta + q * tcs (T1..T3) or Tb + (q - 3) * tcs (T4..T6)
  R *Ta, *Tb;
  int W, tsy;
  unsigned tsx;            // elements per plane
  long long tcs;           // elements per component
  int sa, sb;              // stress planes of this launch
  int pa, pb;              // update planes of this launch
  FastDiv dz1, dy1;        // nz-1, ny-1 (stress box)
  FastDiv uz_[3], uy_[3];  // update points away from the faces: z and y extents of each component
  FastDiv per[3], nk[3];   // points next to a face: per plane, per row of the plane next to x = N
  int off[7];              // first point of each component next to a face, then of the others, total
};

}  // namespace phono
