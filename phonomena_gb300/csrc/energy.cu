// Energy reduction of an FDTD state (FP64 accumulation, deterministic order).
//
// E_kin = 1/2 sum rho v^2 over the displacement points the interior update
// writes, E_str = 1/2 sum T . e over the stress points the reference computes
// (normal stresses at nodes, shears at edges; simulation/base_solver.py:323-433)
// with unit weights.  v is the half-step velocity: (u - u_old)/dt for the
// leapfrog state, the stored v for the velocity form.  Used only to measure the
// error of the FP32 path against the FP64 path; the reference has no energy.
//
// Pass 1 writes one partial pair per block into a scratch array; pass 2 sums
// the partials in block order in one block, so the result does not depend on
// scheduling.
#include <cstdio>

#include "fdtd_common.cuh"

namespace phono {

__device__ __forceinline__ double ld(const void* p, int f32, long long off) {
  return f32 ? (double)__ldg((const float*)p + off) : __ldg((const double*)p + off);
}

constexpr int EN_THREADS = 256;
constexpr int EN_WARPS = EN_THREADS / 32;

// Material row of the reductions: the quadratic form of the normal strains
// (c00, c11, c22, c01 + c10, c02 + c20, c12 + c21), the shear moduli, rho.
constexpr int EN_COLS = 10;
__device__ __forceinline__ double en_coef(const double* row, int q) {
  switch (q) {
    case 0: return __ldg(row);
    case 1: return __ldg(row + 4);
    case 2: return __ldg(row + 8);
    case 3: return __dadd_rn(__ldg(row + 1), __ldg(row + 3));
    case 4: return __dadd_rn(__ldg(row + 2), __ldg(row + 6));
    case 5: return __dadd_rn(__ldg(row + 5), __ldg(row + 7));
    default: return __ldg(row + 3 + q);  // 6..8: columns 9..11; 9: rho
  }
}

// sums of the block's threads, halved, into its partial
__device__ __forceinline__ void block_partial(double ek, double es, double2* partial) {
  __shared__ double sk[EN_THREADS], ss[EN_THREADS];
  sk[threadIdx.x] = 0.5 * ek;
  ss[threadIdx.x] = 0.5 * es;
  __syncthreads();
  for (int w = EN_THREADS / 2; w > 0; w >>= 1) {
    if ((int)threadIdx.x < w) {
      sk[threadIdx.x] += sk[threadIdx.x + w];
      ss[threadIdx.x] += ss[threadIdx.x + w];
    }
    __syncthreads();
  }
  if (threadIdx.x == 0) *partial = make_double2(sk[0], ss[0]);
}

// One warp per (i, j) row of the mesh, lanes along k (coalesced loads of every
// array), rows dealt to the warps of the grid in a fixed order.  Spacings come
// as FP64 reciprocals (the strain is a difference times 1/spacing) and the
// material table is staged in shared memory, so a node costs about 40 FP64
// operations, which bounds the kernel (one FP64 instruction takes a
// multiprocessor 16 cycles): 0.57 ms of FP64 pipe at 8.5 M nodes, 0.70 ms
// measured (0.79 with two resident blocks instead of four), 1.27 with separate
// multiplications and additions and all nine stiffnesses.  Element type T of the displacement / velocity arrays.
template <class T>
__global__ void __launch_bounds__(EN_THREADS, 4) energy_partial_kernel(EnergyArgs a, double2* __restrict__ partial) {
  extern __shared__ double etab[];  // nmat rows of EN_COLS
  for (int q = threadIdx.x; q < a.nmat * EN_COLS; q += EN_THREADS)
    etab[q] = en_coef(a.tab + 13 * (q / EN_COLS), q % EN_COLS);
  __syncthreads();
  const Geo& g = a.g;
  const int nx = g.nx, ny = g.ny, nz = g.nz;
  const int lane = threadIdx.x & 31;
  const int nwarps = gridDim.x * EN_WARPS;
  const T* ux = (const T*)a.ux;
  const T* uy = (const T*)a.uy;
  const T* uz = (const T*)a.uz;
  const T* vx = (const T*)a.vx;
  const T* vy = (const T*)a.vy;
  const T* vz = (const T*)a.vz;
  const uint8_t* mat = a.mat;
  double ek = 0.0, es = 0.0;  // sums of rho v^2 (leapfrog: of rho (u - u_old)^2) and of T . e
  for (int r = blockIdx.x * EN_WARPS + (threadIdx.x >> 5); r < nx * ny; r += nwarps) {
    const int i = r / ny, j = r - (r / ny) * ny;
    const long long o = g.o0 + (long long)i * g.sx + (long long)j * g.sy;      // field (i, j, 0)
    const long long mo = g.mo0 + (long long)i * g.msx + (long long)j * g.msy;  // material (i, j, 0)
    // row predicates of the point sets below
    const bool ix_in = i <= nx - 3, iyz_in = i >= 1 && i <= nx - 2, ish = i <= nx - 2;
    const bool jx_in = j >= 1 && j <= ny - 2, jy_in = j >= 1 && j <= ny - 3, jsh = j <= ny - 2;
    const double rsdx = iyz_in ? __ldg(a.rsdx + i - 1) : 0.0, rfdx = ish ? __ldg(a.rfdx + i) : 0.0;
    const double rsdy = jx_in ? __ldg(a.rsdy + j - 1) : 0.0, rfdy = jsh ? __ldg(a.rfdy + j) : 0.0;
    for (int k = lane; k < nz; k += 32) {
      const long long p = o + k;
      const bool kin = k <= nz - 2, kn = k >= 1 && k <= nz - 2;
      const double rsdz = kn ? __ldg(a.rsdz + k - 1) : 0.0, rfdz = kn ? __ldg(a.rfdz + k) : 0.0;
      auto at = [&](const T* f, long long q) { return (double)__ldg(f + q); };
      // kinetic energy at the interior displacement points, absorbing faces excluded
      auto vel = [&](const T* u, const T* v) { return a.vgiven ? at(v, p) : at(u, p) - at(v, p); };
      auto square = [&](double& sum, double c, double x) { sum = __fma_rn(__dmul_rn(c, x), x, sum); };
      if (ix_in && jx_in && kin) square(ek, etab[EN_COLS * mat[mo + g.msx + k] + 9], vel(ux, vx));
      if (iyz_in && jy_in && kin) square(ek, etab[EN_COLS * mat[mo + g.msy + k] + 9], vel(uy, vy));
      if (iyz_in && jx_in && k <= nz - 3) square(ek, etab[EN_COLS * mat[mo + k + 1] + 9], vel(uz, vz));
      if (!kn) continue;  // every strain term below needs 1 <= k <= nz-2
      const double x0 = at(ux, p), y0 = at(uy, p), z0 = at(uz, p);
      // strain energy: normal stresses at interior nodes
      if (iyz_in && jx_in) {
        const double* c = etab + EN_COLS * mat[mo + k];
        const double e1 = (x0 - at(ux, p - g.sx)) * rsdx, e2 = (y0 - at(uy, p - g.sy)) * rsdy, e3 = (z0 - at(uz, p - 1)) * rsdz;
        es = __fma_rn(__fma_rn(c[0], e1, __fma_rn(c[3], e2, __dmul_rn(c[4], e3))), e1, es);
        es = __fma_rn(__fma_rn(c[1], e2, __dmul_rn(c[5], e3)), e2, es);
        square(es, c[2], e3);
      }
      // shears at edges
      if (iyz_in && jsh)
        square(es, etab[EN_COLS * mat[mo + g.msy + k + 1] + 6],
               __fma_rn(at(uy, p + 1) - y0, rfdz, __dmul_rn(at(uz, p + g.sy) - z0, rfdy)));
      if (ish && jx_in)
        square(es, etab[EN_COLS * mat[mo + g.msx + k + 1] + 7],
               __fma_rn(at(ux, p + 1) - x0, rfdz, __dmul_rn(at(uz, p + g.sx) - z0, rfdx)));
      if (ish && jsh)
        square(es, etab[EN_COLS * mat[mo + g.msx + g.msy + k] + 8],
               __fma_rn(at(ux, p + g.sy) - x0, rfdy, __dmul_rn(at(uy, p + g.sx) - y0, rfdx)));
    }
  }
  block_partial(a.vgiven ? ek : ek * (a.inv_dt * a.inv_dt), es, partial + blockIdx.x);
}

// ---------------------------------------------------------------------------
// FP32 fields of large meshes: the same FP64 sums, marching along x with the
// values of the last plane in registers, and FP32 values widened by integer
// instructions: the conversion instruction runs at the FP64 pipe's rate.
// ---------------------------------------------------------------------------
// a call, so that the conversion is not done ahead of the branches around it
__device__ __noinline__ double convert(float x) { return (double)x; }
__device__ __forceinline__ double widen(float x) {
  const uint32_t u = __float_as_uint(x);
  if ((u & 0x7fffffffu) - 0x00800000u < 0x7f000000u)  // normal: the exponent rebiased, the fraction moved
    return __hiloint2double((int)((((uint32_t)((int)u >> 3)) & 0x8fffffffu) + 0x38000000u), (int)(u << 29));
  return u << 1 ? convert(x) : __hiloint2double((int)u, 0);
}

constexpr int EN_PLANES = 64;  // most planes of an item

// what plane i of a column adds to the last plane's values
struct EnPlane {
  float x0, xk, xj;      // ux(i), ux(i, k+1), ux(i, j+1)
  float y1, yk, yj;      // uy(i+1), uy(i, k+1), uy(i, j-1)
  float z1, zk, zj;      // uz(i+1), uz(i, k-1), uz(i, j+1)
  float vx, vy, vz;
  int id, id_z, id_y, id_yz;  // plane i+1: own, k+1, j+1, both
};

// A block takes (column tile of 8 rows x 32 z, 1/nit of the planes) items in a
// fixed order; a warp owns a row of the tile, a lane a z column, and marches
// along x with the values of the last plane in registers and those of the next
// one on their way.  Bound by the FP64 pipe: 39 operations a node, 0.54 ms of
// its issue at 257x257x129 nodes.  us a call, energy_partial_kernel<float> / here:
// 55 k nodes 40.0 / 53.9, 108 k 42.8 / 53.2, 207 k 78.3 / 67.1, 845 k 166 / 116,
// 8.5 M 1066 / 633.  (Terms formed in pairs of floats took 216 there, but a
// term was off by up to 2^-45, which shows when a state is a few values; here
// it is as good as the other form's.)
__global__ void __launch_bounds__(EN_THREADS, 2) energy_march_kernel(EnergyArgs a, int nit, double2* __restrict__ partial) {
  extern __shared__ double etab[];  // nmat rows of EN_COLS constants, then the x spacings of an item
  double* px = etab + a.nmat * EN_COLS;
  for (int q = threadIdx.x; q < a.nmat * EN_COLS; q += EN_THREADS) etab[q] = en_coef(a.tab + 13 * (q / EN_COLS), q % EN_COLS);
  const Geo& g = a.g;
  const int nx = g.nx, ny = g.ny, nz = g.nz;
  const int lane = threadIdx.x & 31, row = threadIdx.x >> 5;
  const int nkt = (nz - 1 + 31) / 32, njt = (ny - 1 + EN_WARPS - 1) / EN_WARPS;
  const long long sx = g.sx, sy = g.sy, msx = g.msx, msy = g.msy;
  double ek = 0.0, es = 0.0;
  for (int item = blockIdx.x; item < nkt * njt * nit; item += gridDim.x) {
    const int kt = item % nkt, rest = item / nkt, jt = rest % njt, part = rest / njt;
    const int i0 = (int)((long long)(nx - 1) * part / nit), i1 = (int)((long long)(nx - 1) * (part + 1) / nit);
    __syncthreads();
    for (int q = threadIdx.x; q < 2 * (i1 - i0); q += EN_THREADS) {
      const int i = i0 + (q >> 1);  // 1/sdx[i-1], 1/fdx[i]
      px[q] = q & 1 ? __ldg(a.rfdx + i) : (i >= 1 && i <= nx - 2 ? __ldg(a.rsdx + i - 1) : 0.0);
    }
    __syncthreads();
    const int j = jt * EN_WARPS + row, k = kt * 32 + lane;
    if (j > ny - 2 || k > nz - 2) continue;  // no term there
    const bool j_n = j >= 1, jy = j >= 1 && j <= ny - 3, kn = k >= 1, kz = k <= nz - 3;
    const double rsy = j_n ? __ldg(a.rsdy + j - 1) : 0.0, rfy = __ldg(a.rfdy + j);
    const double rsz = kn ? __ldg(a.rsdz + k - 1) : 0.0, rfz = __ldg(a.rfdz + k);
    const long long o = g.o0 + (long long)i0 * sx + (long long)j * sy + k;
    const float *ux = (const float*)a.ux + o, *uy = (const float*)a.uy + o, *uz = (const float*)a.uz + o;
    const float *vx = (const float*)a.vx + o, *vy = (const float*)a.vy + o, *vz = (const float*)a.vz + o;
    const uint8_t* m = a.mat + g.mo0 + (long long)i0 * msx + (long long)j * msy + k;
    double xm = widen(__ldg(ux - sx)), y0 = widen(__ldg(uy)), z0 = widen(__ldg(uz));
    int id = m[0], id_z = m[1], id_y = m[msy], id_yz = m[msy + 1];
    // the padding makes every neighbour of planes up to nx-1 readable
    auto read = [&] {
      EnPlane p;
      p.x0 = __ldg(ux), p.xk = __ldg(ux + 1), p.xj = __ldg(ux + sy);
      p.y1 = __ldg(uy + sx), p.yk = __ldg(uy + 1), p.yj = __ldg(uy - sy);
      p.z1 = __ldg(uz + sx), p.zk = __ldg(uz - 1), p.zj = __ldg(uz + sy);
      p.vx = __ldg(vx), p.vy = __ldg(vy), p.vz = __ldg(vz);
      p.id = m[msx], p.id_z = m[msx + 1], p.id_y = m[msx + msy], p.id_yz = m[msx + msy + 1];
      ux += sx, uy += sx, uz += sx, vx += sx, vy += sx, vz += sx, m += msx;
      return p;
    };
    auto square = [&](double& sum, int mid, int q, double x) { sum = __fma_rn(__dmul_rn(etab[EN_COLS * mid + q], x), x, sum); };
    EnPlane next = read();
    for (int i = i0; i < i1; i++) {
      const EnPlane p = next;
      if (i + 1 < i1) next = read();
      const bool i_n = i >= 1, in = i_n && j_n;  // i <= nx-2 here
      const double x0 = widen(p.x0), y1 = widen(p.y1), z1 = widen(p.z1);
      // kinetic energy
      if (j_n && i <= nx - 3) square(ek, p.id, 9, widen(p.vx));
      if (i_n && jy) square(ek, id_y, 9, widen(p.vy));
      if (in && kz) square(ek, id_z, 9, widen(p.vz));
      if (kn) {
        const double rsx = px[2 * (i - i0)], rfx = px[2 * (i - i0) + 1];
        if (in) {
          const double* c = etab + EN_COLS * id;
          const double e1 = __dmul_rn(__dsub_rn(x0, xm), rsx), e2 = __dmul_rn(__dsub_rn(y0, widen(p.yj)), rsy),
                       e3 = __dmul_rn(__dsub_rn(z0, widen(p.zk)), rsz);
          es = __fma_rn(__fma_rn(c[0], e1, __fma_rn(c[3], e2, __dmul_rn(c[4], e3))), e1, es);
          es = __fma_rn(__fma_rn(c[1], e2, __dmul_rn(c[5], e3)), e2, es);
          square(es, id, 2, e3);
        }
        auto shear = [&](int mid, int q, double d1, double r1, double d2, double r2) {
          square(es, mid, q, __fma_rn(d1, r1, __dmul_rn(d2, r2)));
        };
        if (i_n) shear(id_yz, 6, __dsub_rn(widen(p.yk), y0), rfz, __dsub_rn(widen(p.zj), z0), rfy);
        if (j_n) shear(p.id_z, 7, __dsub_rn(widen(p.xk), x0), rfz, __dsub_rn(z1, z0), rfx);
        shear(p.id_y, 8, __dsub_rn(widen(p.xj), x0), rfy, __dsub_rn(y1, y0), rfx);
      }
      xm = x0, y0 = y1, z0 = z1;
      id = p.id, id_z = p.id_z, id_y = p.id_y, id_yz = p.id_yz;
    }
  }
  block_partial(ek, es, partial + blockIdx.x);
}

__global__ void __launch_bounds__(EN_THREADS) energy_final_kernel(const double2* __restrict__ partial, int n,
                                                                    double* __restrict__ out) {
  __shared__ double sk[EN_THREADS], ss[EN_THREADS];
  double ek = 0.0, es = 0.0;
  for (int q = threadIdx.x; q < n; q += EN_THREADS) {
    ek += partial[q].x;
    es += partial[q].y;
  }
  sk[threadIdx.x] = ek;
  ss[threadIdx.x] = es;
  __syncthreads();
  for (int w = EN_THREADS / 2; w > 0; w >>= 1) {
    if ((int)threadIdx.x < w) {
      sk[threadIdx.x] += sk[threadIdx.x + w];
      ss[threadIdx.x] += ss[threadIdx.x + w];
    }
    __syncthreads();
  }
  if (threadIdx.x == 0) {
    out[0] = sk[0];
    out[1] = ss[0];
  }
}

// partial must hold nblocks double2 values; out two doubles (device).
// march_blocks > 0: FP32 fields by energy_march_kernel in that many blocks
// (at most nblocks)
cudaError_t launch_energy(const EnergyArgs& a, double2* partial, int nblocks, double* out, int march_blocks, cudaStream_t st) {
  if (march_blocks > 0) {
    const size_t smem = ((size_t)a.nmat * EN_COLS + 2 * EN_PLANES) * sizeof(double);
    nblocks = nblocks < march_blocks ? nblocks : march_blocks;
    // x parts: as many items as fill the blocks' last round best
    const int tiles = ((a.g.nz + 30) / 32) * ((a.g.ny - 1 + EN_WARPS - 1) / EN_WARPS);
    const int least = (a.g.nx - 1 + EN_PLANES - 1) / EN_PLANES, most = (a.g.nx - 1 + 7) / 8;
    int nit = least;
    double best = 0.0;
    for (int n = least; n <= most && n <= least + 16; n++) {
      const int rounds = (tiles * n + nblocks - 1) / nblocks;
      // a round takes its planes and about two more for the start of a column
      const double use = 1.0 / (rounds * ((double)(a.g.nx - 1) / n + 2.0));
      if (use > best) best = use, nit = n;
    }
    energy_march_kernel<<<nblocks, EN_THREADS, smem, st>>>(a, nit, partial);
  } else {
    const size_t smem = (size_t)a.nmat * EN_COLS * sizeof(double);
    // no block without a row: its table and its sums took longer than the rows
    // of a small mesh (us a call: 2.0 k nodes 32.4 / 27.7, 35 k 40.4 / 31.3); the
    // partials left out are zeros
    const long long rows = ((long long)a.g.nx * a.g.ny + EN_WARPS - 1) / EN_WARPS;
    if (rows < nblocks) nblocks = (int)rows;
    if (a.f32)
      energy_partial_kernel<float><<<nblocks, EN_THREADS, smem, st>>>(a, partial);
    else
      energy_partial_kernel<double><<<nblocks, EN_THREADS, smem, st>>>(a, partial);
  }
  energy_final_kernel<<<1, EN_THREADS, 0, st>>>(partial, nblocks, out);
  return cudaGetLastError();
}

}  // namespace phono

// ---------------------------------------------------------------------------
// Allocation-free variant (phono_energy_static in include/phono.h).
//
// Same energy as energy_partial_kernel, over caller-owned dense arrays in the
// reference shapes, one block per x plane; the per-plane partials go to the
// file-scope scratch array below instead of a buffer from cudaMalloc, and
// energy_final_kernel sums them in plane order.  Host code must not pass the
// array's name to a kernel (it is a host-side stand-in): the device address
// is looked up once per device with cudaGetSymbolAddress.
// ---------------------------------------------------------------------------
#include <atomic>

#include "../../include/phono.h"

namespace phono {

static __device__ __align__(256) double2 g_energy_scratch[PHONO_ENERGY_STATIC_MAX_NX];

__global__ void __launch_bounds__(EN_THREADS) energy_plane_kernel(phono_energy_dense a, double2* __restrict__ partial) {
  const int nx = a.nx, ny = a.ny, nz = a.nz;
  const int i = blockIdx.x;
  const int f32 = a.precision == PHONO_F32K;
  const int vgiven = a.precision != PHONO_F64;
  const double inv_dt = 1.0 / a.dt;
  const unsigned nmat = (unsigned)a.nmat;
  bool bad_id = false;  // a material id at or past the table's end: no table read, NaN result
  auto ix = [&](int ii, int jj, int kk) { return ((long long)ii * ny + jj) * nz + kk; };          // ux, mat
  auto iy = [&](int ii, int jj, int kk) { return ((long long)ii * (ny - 1) + jj) * nz + kk; };    // uy
  auto iz = [&](int ii, int jj, int kk) { return ((long long)ii * ny + jj) * (nz - 1) + kk; };    // uz
  auto C = [&](int ii, int jj, int kk, int e) {
    const unsigned id = a.mat[ix(ii, jj, kk)];
    if (id >= nmat) {
      bad_id = true;
      return 0.0;
    }
    return a.table[id * 13 + e];
  };
  auto rho = [&](int ii, int jj, int kk) { return C(ii, jj, kk, 12); };
  auto vel = [&](const void* u, const void* v, long long off) {
    double x = ld(v, f32, off);
    return vgiven ? x : (ld(u, 0, off) - x) * inv_dt;
  };
  double ek = 0.0, es = 0.0;
  for (int q = threadIdx.x; q < ny * nz; q += EN_THREADS) {
    const int j = q / nz, k = q - j * nz;
    if (i <= nx - 3 && j >= 1 && j <= ny - 2 && k <= nz - 2) {
      double v = vel(a.ux, a.vx, ix(i, j, k));
      ek += 0.5 * rho(i + 1, j, k) * v * v;
    }
    if (i >= 1 && i <= nx - 2 && j >= 1 && j <= ny - 3 && k <= nz - 2) {
      double v = vel(a.uy, a.vy, iy(i, j, k));
      ek += 0.5 * rho(i, j + 1, k) * v * v;
    }
    if (i >= 1 && i <= nx - 2 && j >= 1 && j <= ny - 2 && k <= nz - 3) {
      double v = vel(a.uz, a.vz, iz(i, j, k));
      ek += 0.5 * rho(i, j, k + 1) * v * v;
    }
    if (i >= 1 && i <= nx - 2 && j >= 1 && j <= ny - 2 && k >= 1 && k <= nz - 2) {
      double e1 = (ld(a.ux, f32, ix(i, j, k)) - ld(a.ux, f32, ix(i - 1, j, k))) / a.sdx[i - 1];
      double e2 = (ld(a.uy, f32, iy(i, j, k)) - ld(a.uy, f32, iy(i, j - 1, k))) / a.sdy[j - 1];
      double e3 = (ld(a.uz, f32, iz(i, j, k)) - ld(a.uz, f32, iz(i, j, k - 1))) / a.sdz[k - 1];
      double t1 = C(i, j, k, 0) * e1 + C(i, j, k, 1) * e2 + C(i, j, k, 2) * e3;
      double t2 = C(i, j, k, 3) * e1 + C(i, j, k, 4) * e2 + C(i, j, k, 5) * e3;
      double t3 = C(i, j, k, 6) * e1 + C(i, j, k, 7) * e2 + C(i, j, k, 8) * e3;
      es += 0.5 * (t1 * e1 + t2 * e2 + t3 * e3);
    }
    if (i >= 1 && i <= nx - 2 && j <= ny - 2 && k >= 1 && k <= nz - 2) {
      double gam = (ld(a.uy, f32, iy(i, j, k + 1)) - ld(a.uy, f32, iy(i, j, k))) / a.fdz[k] +
                   (ld(a.uz, f32, iz(i, j + 1, k)) - ld(a.uz, f32, iz(i, j, k))) / a.fdy[j];
      es += 0.5 * C(i, j + 1, k + 1, 9) * gam * gam;
    }
    if (i <= nx - 2 && j >= 1 && j <= ny - 2 && k >= 1 && k <= nz - 2) {
      double gam = (ld(a.ux, f32, ix(i, j, k + 1)) - ld(a.ux, f32, ix(i, j, k))) / a.fdz[k] +
                   (ld(a.uz, f32, iz(i + 1, j, k)) - ld(a.uz, f32, iz(i, j, k))) / a.fdx[i];
      es += 0.5 * C(i + 1, j, k + 1, 10) * gam * gam;
    }
    if (i <= nx - 2 && j <= ny - 2 && k >= 1 && k <= nz - 2) {
      double gam = (ld(a.ux, f32, ix(i, j + 1, k)) - ld(a.ux, f32, ix(i, j, k))) / a.fdy[j] +
                   (ld(a.uy, f32, iy(i + 1, j, k)) - ld(a.uy, f32, iy(i, j, k))) / a.fdx[i];
      es += 0.5 * C(i + 1, j + 1, k, 11) * gam * gam;
    }
  }
  const bool any_bad = __syncthreads_or(bad_id);
  __shared__ double sk[EN_THREADS], ss[EN_THREADS];
  sk[threadIdx.x] = ek;
  ss[threadIdx.x] = es;
  __syncthreads();
  for (int w = EN_THREADS / 2; w > 0; w >>= 1) {
    if ((int)threadIdx.x < w) {
      sk[threadIdx.x] += sk[threadIdx.x + w];
      ss[threadIdx.x] += ss[threadIdx.x + w];
    }
    __syncthreads();
  }
  if (threadIdx.x == 0) partial[i] = any_bad ? make_double2(__longlong_as_double(0x7ff8000000000000LL),
                                                            __longlong_as_double(0x7ff8000000000000LL))
                                             : make_double2(sk[0], ss[0]);
}

}  // namespace phono

namespace phono {
void set_last_error(const char* msg);  // api.cu: message behind phono_last_error()
}

namespace {
// Device address of g_energy_scratch, looked up on the first call made with
// that device current.  Two host threads making their first call on one
// device at the same time both look it up and store the same value; the
// atomics make that well defined.  The address belongs to the device's
// primary context: after cudaDeviceReset the cache is stale, so a process
// that resets a device must not call phono_energy_static on it again.
constexpr int kMaxDevices = 64;
std::atomic<void*> g_scratch_addr[kMaxDevices];
}  // namespace

extern "C" int phono_energy_static(const phono_energy_dense* in, double* out_dev, void* stream) {
  using namespace phono;
  auto fail = [](int code, const char* msg) {
    set_last_error(msg);
    return code;
  };
  if (!in || !out_dev) return fail(PHONO_ERR_ARG, "NULL argument");
  if (in->nx < 3 || in->ny < 3 || in->nz < 3) return fail(PHONO_ERR_ARG, "nx, ny, nz must be >= 3 mesh nodes");
  if (in->nx > PHONO_ENERGY_STATIC_MAX_NX)
    return fail(PHONO_ERR_ARG, "nx exceeds PHONO_ENERGY_STATIC_MAX_NX, the planes of the static scratch array");
  if ((long long)in->ny * in->nz > 0x7fffffffLL) return fail(PHONO_ERR_ARG, "ny * nz too large");
  if (in->precision != PHONO_F64 && in->precision != PHONO_F32K && in->precision != PHONO_F64V)
    return fail(PHONO_ERR_ARG, "unknown precision");
  if (!in->ux || !in->uy || !in->uz || !in->vx || !in->vy || !in->vz || !in->mat || !in->table || !in->fdx ||
      !in->fdy || !in->fdz || !in->sdx || !in->sdy || !in->sdz)
    return fail(PHONO_ERR_ARG, "NULL device pointer in the input");
  if (!(in->dt > 0.0)) return fail(PHONO_ERR_ARG, "dt must be > 0");
  if (in->nmat < 1 || in->nmat > 256) return fail(PHONO_ERR_ARG, "nmat must be in 1..256");
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= kMaxDevices)
    return fail(PHONO_ERR_CUDA, "cudaGetDevice failed");
  void* addr = g_scratch_addr[dev].load(std::memory_order_acquire);
  if (!addr) {
    cudaError_t e = cudaGetSymbolAddress(&addr, g_energy_scratch);
    if (e != cudaSuccess || !addr) return fail(PHONO_ERR_CUDA, "cudaGetSymbolAddress of the energy scratch failed");
    g_scratch_addr[dev].store(addr, std::memory_order_release);
  }
  double2* partial = static_cast<double2*>(addr);
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  energy_plane_kernel<<<in->nx, EN_THREADS, 0, st>>>(*in, partial);
  energy_final_kernel<<<1, EN_THREADS, 0, st>>>(partial, in->nx, out_dev);
  cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) return fail(PHONO_ERR_CUDA, cudaGetErrorString(e));
  return PHONO_OK;
}
