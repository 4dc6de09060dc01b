// Tile pass of the FP32 velocity form (included by fdtd_step.cu).
//
// A block owns a (TJ x 32) tile of the (y, z) plane and marches along x over
// planes [ib, ie).  TJ/4 warps update it: a thread owns four consecutive z
// points of one row (8 lanes span the tile's 32 columns, a warp four rows),
// so that ring reads, state and stores are 128-bit and everything that does
// not depend on the point (ring slots, range tests, x spacings, material rows
// of a homogeneous neighbourhood) is shared by four nodes.  One more warp
// evaluates the stresses of the tile's halo (row above and below, column left
// and right) and issues the TMA copies.
//
// Stage p of the 3-slot ring holds plane p of u (three components, 1-node
// halo) and of the material ids, and plane p-1 of the pointwise state (v and
// the Kahan term of the own points), on one mbarrier.  Per plane i:
//   A  read u of planes i and i+1, evaluate the six stresses, update ux of
//      plane i-1 (its x difference was the last stress missing), publish the
//      stresses that another warp needs;
//   -- one barrier; the slot of plane i is refilled with stage i+3 --
//   B  fetch the neighbours' stresses (shuffles inside the warp, shared memory
//      across warps, double-buffered), update uy and uz of plane i, form what
//      ux of plane i will need.
// Segment ends need only T1 of the first plane behind them.
//
// The face points are written here too (height 16, five rows of nodes and
// more).  The halo warp of a block with a row next to y = 0 or y = N evaluates
// that face's points of plane i-1 from the new state the block has just
// written: it reads it behind the barrier of iteration i and uses it before
// the next one.  The x = N points come after the last plane, from the threads
// of the rows.  A face launch of its own costs 4 to 5 us a step (with it and
// without, us a step: 512x512x256 cells 805 / 778, 256x256x128 122 / 118,
// 160x128x64 25.8 / 24.5); the same from the registers of the updating threads
// made their loop slower for every block (256x256x128: 138).  At height 8 the
// halo warp has half the time for it, and the launch is the better one (193x161x97
// cells 62.5 us a step with it, 61.2 without, 12 crystals of 6.2 M nodes stepped
// together 174 and 208).
//
// With the faces written here a step is one launch, and the next one is let in
// when a block has finished its planes: its start (barriers, tables, spacings)
// runs beside the last blocks of this one (whole runs without and with:
// 160x128x64 cells, 300 steps 8.91 / 8.31 ms, 256x256x128, 360 steps 44.2 /
// 43.7; let in at the start of a block, or one or two planes earlier, less).
//
// Bound by DRAM traffic on large meshes (512x512x256 cells: 778 us a step,
// 6.37 TB/s of the 73 bytes a node, 94% of the measured copy bandwidth), and by
// the latency of a plane (1.7 us for a block alone) with the ramp and tail of
// the launch on small ones.  The form before it, one node a thread with all
// stresses exchanged through shared memory and two barriers a plane, issued
// 507 instructions a node against 220 here and was bound by that.  Rows start
// on 128-byte lines, so that a row of the tile's state is one line for the
// copies in and for the stores (87 bytes of DRAM traffic a node when rows
// started 32 bytes into a line, 80 now).  us a step, best tiles of the form
// before, this form, with aligned rows, now: 512x512x256 1043 / 850 / 805 /
// 778, 256x256x128 154 / 138 / 128 / 118, 193x161x97 80 / 66 / 63 / 59,
// 160x128x64 39.5 / 31 / 26 / 24.5.
// Included inside namespace phono, after the TMA helpers and the schemes.
#pragma once

template <int TJ>
struct VecPlan {
  static constexpr int NW = TJ / 4;          // updating warps
  static constexpr int NT = 32 * (NW + 1);   // threads of a block
  static constexpr int NS = 3;               // ring slots
  static constexpr int KW = Lay<float>::KW, KB = Lay<float>::KB, CW = (TJ + 2) * KW;
  static constexpr int SU = (3 * CW * 4 + 127) / 128 * 32;           // u slot (floats)
  static constexpr int SM = ((TJ + 2) * MKW + 127) / 128 * 128;      // id slot (bytes)
  static constexpr int PWC = TJ * TK, PWS = 6 * PWC;                 // pointwise component, slot (floats)
  static constexpr int EX = (NW + 1) * 32;                           // one exchanged row set (floats)
  static constexpr size_t off_u = 128, off_pw = off_u + (size_t)NS * SU * 4, off_m = off_pw + (size_t)NS * PWS * 4;
  static constexpr size_t off_e = off_m + (size_t)NS * SM;           // rows: T2, T4, T6, two buffers each
  static constexpr size_t off_c = off_e + (size_t)6 * EX * 4;        // columns: T3, T4, T5, two buffers of 16 each
  static constexpr size_t off_tab = off_c + 6 * 16 * 4;
  static constexpr size_t bytes(int table_rows) { return off_tab + 128 + (size_t)table_rows * 64; }
  static constexpr uint32_t tx_bytes = (uint32_t)(3 * CW * 4 + (TJ + 2) * MKW), pw_bytes = (uint32_t)(PWS * 4);
  static_assert(off_tab % 16 == 0 && (PWC * 4) % 128 == 0, "alignment of the shared arrays");
};

// New state of component c's four points from z = k on at offset o; `last` is
// the z of the row's last inner point.  Above that comes the z = N face point
// (base_solver.py:552-554; old: the old values, old4 the one above them), then
// padding, which stays zero.
__device__ __forceinline__ void store_vec(const Roles<float>& r, int c, unsigned o, int w, bool rigid, float face,
                                          const float (&old)[4], float old4, float (&u)[4], float (&v)[4], float (&kc)[4]) {
  // w = last - k
  if (w <= 3) {
    const float f1 = F32K::abc(face, u[0], old[1], old[0]), f2 = F32K::abc(face, u[1], old[2], old[1]),
                f3 = F32K::abc(face, u[2], old[3], old[2]);
    if (w == 3) store_point<F32K>(r, c, o + 4, rigid ? 0.f : F32K::abc(face, u[3], old4, old[3]), 0.f, 0.f);
    u[1] = w < 1 ? (w == 0 && !rigid ? f1 : 0.f) : u[1];
    u[2] = w < 2 ? (w == 1 && !rigid ? f2 : 0.f) : u[2];
    u[3] = w < 3 ? (w == 2 && !rigid ? f3 : 0.f) : u[3];
#pragma unroll
    for (int q = 1; q < 4; q++) v[q] = w < q ? 0.f : v[q], kc[q] = w < q ? 0.f : kc[q];
  }
  if (w < 0) return;
  *reinterpret_cast<float4*>(r.out(c) + o) = make_float4(u[0], u[1], u[2], u[3]);
  *reinterpret_cast<float4*>(r.vout(c) + o) = make_float4(v[0], v[1], v[2], v[3]);
  *reinterpret_cast<float4*>(r.cout(c) + o) = make_float4(kc[0], kc[1], kc[2], kc[3]);
}

// Four points of a face row, or of a row next to one, of component c: plane p,
// row j, from z = k on.
struct FaceRow {
  float v[4], v4;  // old values (uz of plane 0: the source), and the one above
  __device__ __forceinline__ void read(const StepArgs<float>& a, const Roles<float>& r, const float s, int c, int p, int j, int k) {
    const float* src = r.cur(c) + fidx(a.g, p, j, k);
    const float4 t = *reinterpret_cast<const float4*>(src);
    v[0] = t.x, v[1] = t.y, v[2] = t.z, v[3] = t.w, v4 = src[4];
    if (c == 2 && p == 0) {  // source overwrite (base_solver.py:251)
      if (a.source_mode == 1) v[0] = v[1] = v[2] = v[3] = v4 = s;
      else if (k == 0) v[0] = s;
    }
  }
  // u: new values of the points; stored with the z = N point above them
  __device__ __forceinline__ void write(const StepArgs<float>& a, const Roles<float>& r, int tt, int c, int p, int j, int k,
                                        float (&u)[4]) const {
    if (c == 2 && k == 0) record(a, tt, p, j, u[0]);
    float vn[4] = {0.f, 0.f, 0.f, 0.f}, cn[4] = {0.f, 0.f, 0.f, 0.f};
    store_vec(r, c, (unsigned)fidx(a.g, p, j, k), (c == 2 ? a.g.nz - 3 : a.g.nz - 2) - k, a.bc == 1, c == 2 ? a.abc[7] : a.abc[6],
              v, v4, u, vn, cn);
  }
  // new values from those of the next row inward, `in` and its old values
  __device__ __forceinline__ void face(const StepArgs<float>& a, const float f, const float (&in)[4], const FaceRow& old,
                                       float (&u)[4]) const {
#pragma unroll
    for (int q = 0; q < 4; q++) u[q] = a.bc == 1 ? 0.f : F32K::abc(f, in[q], v[q], old.v[q]);
  }
};
__device__ __forceinline__ float y_face_coef(const StepArgs<float>& a, int c, int dj) {
  return dj < 0 ? a.abc[c == 1 ? 3 : 2] : a.abc[c == 1 ? 5 : 4];
}

// The block's barrier for its two kinds of warps, which reach it at statements
// of their own: __syncthreads() has to be one statement for all threads, while
// PTX's barrier counts those that arrive at barrier 0, wherever that is.
// Aligned: the lanes of a warp are of one kind and come together (us for 360
// steps on 256x256x128 cells: 43150, 52940 without).
__device__ __forceinline__ void block_wait() { asm volatile("barrier.cta.sync.aligned 0;" ::: "memory"); }
__device__ __forceinline__ bool block_any(bool x) {
  uint32_t any;
  asm volatile(
      "{\n .reg .pred p, q;\n setp.ne.u32 p, %1, 0;\n barrier.cta.red.or.pred.aligned q, 0, p;\n selp.u32 %0, 1, 0, q;\n}\n"
      : "=r"(any)
      : "r"((uint32_t)x)
      : "memory");
  return any != 0;
}

template <int TJ>
__device__ __forceinline__ void tile_block_vec(const StepArgs<float>& a, unsigned char* base, const Roles<float>& r,
                                               const float s, const int tt, const int tid, const int b) {
  using P = VecPlan<TJ>;
  using S = F32K;
  constexpr int KW = P::KW, KB = P::KB, CW = P::CW, YO = CW, ZO = 2 * CW, NS = P::NS;
  uint64_t* bars = reinterpret_cast<uint64_t*>(base);
  float* uring = reinterpret_cast<float*>(base + P::off_u);
  float* pwring = reinterpret_cast<float*>(base + P::off_pw);
  uint8_t* mring = reinterpret_cast<uint8_t*>(base + P::off_m);
  float* ex = reinterpret_cast<float*>(base + P::off_e);
  float* cx = reinterpret_cast<float*>(base + P::off_c);
  float* tab = reinterpret_cast<float*>(base + P::off_tab);

  const Geo& g = a.g;
  const int nx = g.nx, ny = g.ny, nz = g.nz;
  const int kt = b % a.ntk, rest = b / a.ntk, jt = rest % a.ntj, seg = rest / a.ntj;
  const int j0 = jt * TJ, k0 = kt * TK;
  const int ib = a.nseg <= SEG_TABLE ? a.seg_start[seg] : seg * a.xseg;
  const int ie = a.nseg <= SEG_TABLE ? a.seg_start[seg + 1] : min(ib + a.xseg, nx - 1);
  const int lane = tid & 31, warp = tid >> 5;
  const bool halo = warp == P::NW;

  for (int q = tid; q < a.nmat * 16; q += P::NT) tab[q] = __ldg(a.tab + q);

  // -------- ring --------
  const int sbuf = r.rcur * 3;
  auto issue = [&](int p, int sl) {  // stage p into slot sl (one thread)
    const bool pw = p - 1 >= ib;
    mbar_expect_tx(&bars[sl], P::tx_bytes + (pw ? P::pw_bytes : 0u));
    // test hook (skip_plane >= 0; -1 is off): armed, no copy, so the wait on it runs out
    if (a.skip_plane >= 0 && p == a.skip_plane) return;
    tma_load_4d(uring + sl * P::SU, &a.tm_u, k0 - KB, j0, p + 1, sbuf, &bars[sl]);
    tma_load_3d(mring + sl * P::SM, &a.tm_mat, k0, j0, p + 1, &bars[sl]);
    if (pw) {
      float* d = pwring + sl * P::PWS;
      tma_load_4d(d, &a.tm_pw0, k0, j0 + 1, p, sbuf, &bars[sl]);
      tma_load_4d(d + 3 * P::PWC, &a.tm_pw1, k0, j0 + 1, p, sbuf, &bars[sl]);
    }
  };
  if (tid == 0) {
    for (int q = 0; q < NS; q++) mbar_init(&bars[q], 1);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  __syncthreads();
  last_launch_done();
  int issued = ib - 2;  // last stage issued (halo warp's lane 0)
  const bool producer = halo && lane == 0;
  if (producer)
    for (int p = ib - 1; p <= min(ib + 1, ie); p++) {
      issue(p, p - ib + 1);
      issued = p;
    }
  // one verdict per warp: what depends on it has warp-wide operations
  auto arrived = [&](int sl, uint32_t parity) { return __all_sync(0xffffffffu, mbar_wait(&bars[sl], parity, a.wait_polls)) != 0; };
  bool ok = arrived(0, 0);
  if (ok) ok = arrived(1, 0);
  if (ib <= 1) {  // source patch: plane 0 is stage ib or ib-1
    float* zt = uring + (1 - ib) * P::SU + ZO;
    if (a.source_mode == 1) {
      for (int q = tid; q < CW; q += P::NT) zt[q] = s;
    } else if (k0 == 0) {
      for (int q = tid; q < TJ + 2; q += P::NT) zt[q * KW + KB] = s;
    }
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
  }
  // one verdict per block before anything is refilled: a slot whose stage never
  // arrived must not be armed a second time
  if (__syncthreads_or(!ok)) ok = false;

  // The (padded) x spacings fdx[p], sdx[p-1] of 32 planes at a time, one plane
  // a lane: a load per plane would wait for L2 in every iteration (stores
  // stream through what L1 the ring leaves).
  float fxv = 0.f, sxv = 0.f;
  auto spacings = [&](int p0) {
    const int p = min(p0 + lane, nx);
    fxv = __ldg(a.sp.fdx + p);
    sxv = __ldg(a.sp.sdx + min(p, nx - 1) - 1);
  };
  spacings(ib);
  float fx_prev = __ldg(a.sp.fdx + ib - 1), fx_cur = __shfl_sync(0xffffffffu, fxv, 0), sx_cur = __shfl_sync(0xffffffffu, sxv, 0);
  // those of plane i+1, at the end of iteration i
  auto advance = [&](int i) {
    const int n = (i + 1 - ib) & 31;
    if (n == 0) spacings(i + 1);
    fx_prev = fx_cur;
    fx_cur = __shfl_sync(0xffffffffu, fxv, n);
    sx_cur = __shfl_sync(0xffffffffu, sxv, n);
  };
  int s0 = 1, s1 = 2;  // slots of stages i, i+1
  uint32_t par = 0;    // phase parity of slot s1

  if (halo) {
    // ---------------- halo warp ----------------
    // rounds 0..2: one row each, lane = column; 3: columns k0-1; 4: column k0+32
    const int kk = k0 + lane, l = lane & 15;
    const bool kz = kk == 0, kin = kk <= nz - 2;
    const int jt2 = j0 + TJ, jb = j0 - 1, jc = j0 + l, kc = k0 - 1, kr = k0 + TK;
    const float sdz_k = kz ? a.sp.sdz0 : (kin ? __ldg(a.sp.sdz + kk - 1) : 1.f);
    const float t2_b = kz ? a.sp.sdy0 : (jt2 <= ny - 2 ? __ldg(a.sp.sdy + jt2 - 1) : 1.f);
    const float fdy_b = jb >= 0 ? __ldg(a.sp.fdy + jb) : 1.f;
    const float t6_a = kz ? a.sp.fdx0 : fdy_b;
    const float t4_a = kz ? a.sp.fdy0 : (kin ? __ldg(a.sp.fdz + kk) : 1.f), t4_b = kz ? a.sp.fdz0 : fdy_b;
    const float col_a = kc >= 0 && kc <= nz - 2 ? __ldg(a.sp.fdz + kc) : 1.f;
    const float col_b = jc <= ny - 2 ? __ldg(a.sp.fdy + jc) : 1.f;
    const float t3_b = jc >= 1 && jc <= ny - 2 ? __ldg(a.sp.sdy + jc - 1) : 1.f;
    const float t3_c = kr <= nz - 2 ? __ldg(a.sp.sdz + kr - 1) : 1.f;
    const bool col = l < TJ;
    const int u_top = (TJ + 1) * KW + KB + lane, u_bot = KB + lane, u_col = (l + 1) * KW + KB - 1, u_right = u_col + 1 + TK;
    const int m_top = (TJ + 1) * MKW + MKOFF + lane, m_bot = MKW + MKOFF + lane;
    const int m_t4c = (l + 2) * MKW + MKOFF, m_t5c = (l + 1) * MKW + MKOFF, m_right = m_t5c + TK;
    // y faces: a lane takes four points of a component's row next to y = 0 or,
    // from the end, y = N; a tile with both does the second on the spot
    const int fc = lane >> 3, fk = k0 + 4 * (lane & 7), f_hi = ny - 2 - (fc == 1 ? 1 : 0);
    const bool f_on = writes_faces(true, TJ, ny) && fc < 3 && fk <= nz - 2, hi = f_on && f_hi >= j0 && f_hi < j0 + TJ;
    const int fd = !f_on ? 0 : j0 == 0 ? -1 : hi ? 1 : 0, fj = fd < 0 ? 1 : f_hi;
    float fn[4];
    FaceRow f_in, f_out;
    auto face_read = [&](int p, int j, int dj) {
      const float4 t = *reinterpret_cast<const float4*>(r.out(fc) + fidx(g, p, j, fk));
      fn[0] = t.x, fn[1] = t.y, fn[2] = t.z, fn[3] = t.w;
      f_in.read(a, r, s, fc, p, j, fk);
      f_out.read(a, r, s, fc, p, j + dj, fk);
    };
    auto face_write = [&](int p, int j, int dj) {
      float u[4];
      f_out.face(a, y_face_coef(a, fc, dj), fn, f_in, u);
      f_out.write(a, r, tt, fc, p, j + dj, fk, u);
    };
    // plane p's points, their values read before; then those of the other face
    auto face_rows = [&](int p, bool read) {
#pragma unroll 1
      for (int j = fj, dj = fd; dj; read = true) {
        if (read) face_read(p, j, dj);
        face_write(p, j, dj);
        dj = dj < 0 && hi ? 1 : 0, j = f_hi;
      }
    };
    float xt_m = 0.f, xr_m = 0.f;  // ux one plane back at u_top, u_right
    {
      const float* U = uring;
      if (ok) xt_m = U[u_top], xr_m = col ? U[u_right] : 0.f;
    }
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    block_wait();  // stage ib-1 is read
    if (producer && ok && ib + 2 <= ie) {
      issue(ib + 2, 0);
      issued = ib + 2;
    }
    for (int i = ib; i < ie; i++) {
      if (ok) ok = arrived(s1, par);
      const int buf = i & 1;
      if (ok) {
        const float *U0 = uring + s0 * P::SU, *U1 = uring + s1 * P::SU;
        const uint8_t *M0 = mring + s0 * P::SM, *M1 = mring + s1 * P::SM;
        const float sx5 = kz ? a.sp.fdz0 : fx_cur;
        {  // T2 row above
          const float x = U0[u_top];
          const float* c = tab + 16 * M0[m_top] + 3;
          ex[buf * P::EX + P::NW * 32 + lane] =
              S::tn1(a.dtab, c, S::sub(x, xt_m), S::sub(U0[YO + u_top], U0[YO + u_top - KW]),
                     S::sub(U0[ZO + u_top], U0[ZO + u_top - 1]), kz ? a.sp.sdx0 : sx_cur, t2_b, sdz_k);
          xt_m = x;
        }
        // T4, T6 row below
        ex[(2 + buf) * P::EX + lane] =
            S::ts(a.dtab, tab[16 * M0[m_bot + (kz ? 0 : 1)] + 9], S::sub(U0[YO + u_bot + 1], U0[YO + u_bot]), t4_a,
                  S::sub(U0[ZO + u_bot + KW], U0[ZO + u_bot]), t4_b);
        ex[(4 + buf) * P::EX + lane] =
            S::ts(a.dtab, tab[16 * M1[m_bot] + 11], S::sub(U0[u_bot + KW], U0[u_bot]), t6_a,
                  S::sub(U1[YO + u_bot], U0[YO + u_bot]), sx5);
        if (col) {  // T4 (lanes 0..15) and T5 (16..31) column left; T3 column right
          const bool t5 = lane >= 16;
          const float* D = U0 + (t5 ? 0 : YO) + u_col;
          const float zc = U0[ZO + u_col];
          const float d2 = S::sub(t5 ? U1[ZO + u_col] : U0[ZO + u_col + KW], zc);
          const float v = S::ts(a.dtab, tab[16 * (t5 ? M1[m_t5c] : M0[m_t4c]) + (t5 ? 10 : 9)], S::sub(D[1], D[0]), col_a,
                                d2, t5 ? fx_cur : col_b);
          cx[(2 + 2 * (t5 ? 1 : 0) + buf) * 16 + l] = k0 == 0 ? 0.f : v;
          if (!t5) {
            const float x = U0[u_right];
            const float* c = tab + 16 * M0[m_right] + 6;
            cx[buf * 16 + l] = S::tn1(a.dtab, c, S::sub(x, xr_m), S::sub(U0[YO + u_right], U0[YO + u_right - KW]),
                                      S::sub(U0[ZO + u_right], U0[ZO + u_right - 1]), sx_cur, t3_b, t3_c);
            xr_m = x;
          }
        }
        if (fd && i >= ib + 2) face_rows(i - 2, false);
      }
      // The slot of plane i is refilled by TMA (async proxy) after the
      // barrier: order this thread's reads of it first (a barrier orders
      // shared-memory accesses of the block's threads only).
      asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
      if (block_any(!ok)) {
        ok = false;
        break;
      }
      if (producer && i + 3 <= ie) {
        issue(i + 3, s0);
        issued = i + 3;
      }
      if (fd && i > ib) face_read(i - 1, fj, fd);  // plane i-1 is complete
      s0 = s1;
      if (++s1 == NS) s1 = 0, par ^= 1;
      advance(i);
    }
    if (ok && fd && ie - ib >= 2) face_rows(ie - 2, false);
    let_next_launch();
    block_wait();  // the last plane is written
    if (ok && fd && !(fc == 0 && ie == nx - 1)) face_rows(ie - 1, true);  // ux ends at plane nx-2, its x = N face
  } else {
    // ---------------- updating warps ----------------
    const int lr = lane >> 3, lc = lane & 7, jl = 4 * warp + lr, j = j0 + jl, k = k0 + 4 * lc;
    const int Lu = (jl + 1) * KW + KB + 4 * lc, Lm = (jl + 1) * MKW + MKOFF + 4 * lc, Lp = jl * TK + 4 * lc;
    const bool kz = k == 0, j_n = j >= 1 && j <= ny - 2;
    // spacings of the four points; in the z = 0 row the reference's
    // substitutions (base_solver.py:408-433, 495-516), kept apart as *0
    float sdz[4], fdz[4];
#pragma unroll
    for (int q = 0; q < 4; q++) {
      sdz[q] = k + q == 0 ? a.sp.sdz0 : (k + q <= nz - 2 ? __ldg(a.sp.sdz + k + q - 1) : 1.f);
      fdz[q] = k + q <= nz - 2 ? __ldg(a.sp.fdz + k + q) : 1.f;
    }
    const float sb = j_n ? __ldg(a.sp.sdy + j - 1) : 1.f, fdyj = j <= ny - 2 ? __ldg(a.sp.fdy + j) : 1.f;
    const float sb0 = kz ? a.sp.sdy0 : sb, t4a0 = kz ? a.sp.fdy0 : fdz[0], t4b0 = kz ? a.sp.fdz0 : fdyj;
    const float t5a0 = kz ? a.sp.fdx0 : fdz[0], t6a0 = kz ? a.sp.fdx0 : fdyj, uyb0 = kz ? a.sp.fdy0 : fdyj;
    const float uzc0 = kz ? (a.surface_mode == 0 ? 1.f : a.sp.fdz0) : fdz[0];
    const unsigned zsel = kz ? 0x4320u : 0x4321u;  // ids one layer down; the z = 0 row: its own
    // rows of each component (uy has its y = N face at ny-2), and whether a
    // component's last inner point may be among the four
    const bool row = j_n && k <= nz - 2, row_y = row && j <= ny - 3;
    const bool edge = k + 3 >= nz - 3;
    const bool rigid = a.bc == 1;
    const unsigned off_j = (unsigned)(g.o0 + (long long)j * g.sy + k), sxu = (unsigned)g.sx;
    float* rec = nullptr;  // the surface record this step writes
    if (kz && row && a.record_every > 0 && (tt + 1) % a.record_every == 0) {
      const int slot = (tt + 1) / a.record_every - 1 - a.rec_base;
      if (slot >= 0 && slot < a.nrec_cap) rec = a.surf + ((long long)slot * nx) * ny + j;
    }

    auto ld4 = [](const float* p, float (&v)[4]) {
      const float4 t = *reinterpret_cast<const float4*>(p);
      v[0] = t.x, v[1] = t.y, v[2] = t.z, v[3] = t.w;
    };
    auto id_of = [](unsigned w, int q) { return (int)((w >> (8 * q)) & 0xffu); };
    // ids of a plane: own points, one layer down, next row, next row one layer down
    struct Ids {
      unsigned c, z, y, yz;
    };
    auto read_ids = [&](const uint8_t* M) {
      const unsigned c = *reinterpret_cast<const unsigned*>(M + Lm), c4 = *reinterpret_cast<const unsigned*>(M + Lm + 4);
      const unsigned y = *reinterpret_cast<const unsigned*>(M + Lm + MKW), y4 = *reinterpret_cast<const unsigned*>(M + Lm + MKW + 4);
      return Ids{c, __byte_perm(c, c4, zsel), y, __byte_perm(y, y4, zsel)};
    };
    float xm[4], t1m[4], t5m[4], t6m[4], px[4], y0[4], z0[4], xm4;
    Ids id;
    {  // plane ib-1: T5, T6; values of plane ib
      const float *U0 = uring, *U1 = uring + P::SU;
      ld4(U0 + Lu, xm);
      ld4(U1 + YO + Lu, y0);
      ld4(U1 + ZO + Lu, z0);
      id = read_ids(mring + P::SM);
      float xj[4], ym[4], zm[4];
      ld4(U0 + Lu + KW, xj);
      ld4(U0 + YO + Lu, ym);
      ld4(U0 + ZO + Lu, zm);
      const float xk = xm4 = U0[Lu + 4];
      const float sx0 = kz ? a.sp.fdz0 : fx_prev;
#pragma unroll
      for (int q = 0; q < 4; q++) {
        t1m[q] = px[q] = t5m[q] = t6m[q] = 0.f;
        if (ok && ib >= 1) {
          t5m[q] = S::ts(a.dtab, tab[16 * id_of(id.z, q) + 10], S::sub(q < 3 ? xm[q < 3 ? q + 1 : 3] : xk, xm[q]),
                         q ? fdz[q] : t5a0, S::sub(z0[q], zm[q]), q ? fx_prev : sx0);
          t6m[q] = S::ts(a.dtab, tab[16 * id_of(id.y, q) + 11], S::sub(xj[q], xm[q]), q ? fdyj : t6a0,
                         S::sub(y0[q], ym[q]), q ? fx_prev : sx0);
        }
      }
    }
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    block_wait();  // stage ib-1 is read: its slot is refilled with stage ib+2

    // ux of plane i-1 from T1 of plane i (base_solver.py:441-447, 495-501)
    auto update_x = [&](int i, const float (&t1)[4], const float* pw, const float (&qd)[4], const float fxm) {
      float v[4], kc[4], un[4], vn[4], cn[4];
      ld4(pw + Lp, v);
      ld4(pw + 3 * P::PWC + Lp, kc);
      const float f0 = kz ? a.sp.fdx0 : fxm;
#pragma unroll
      for (int q = 0; q < 4; q++) {
        const float dv = __fmaf_rn(S::sub(t1[q], t1m[q]), q ? fxm : f0, px[q]);
        un[q] = update_value<S>(xm[q], Pw<float>{v[q], kc[q]}, dv, qd[q], a.dt, vn[q], cn[q]);
      }
      if (row) store_vec(r, 0, off_j + (unsigned)(i - 1) * sxu, nz - 2 - k, rigid, a.abc[6], xm, xm4, un, vn, cn);
    };

    for (int i = ib; i < ie; i++) {
      if (ok) ok = arrived(s1, par);
      const int buf = i & 1;
      float t2[4], t3[4], t4[4], t5[4], t6[4], y1[4], z1[4], x0[4], qy[4], qz[4], y4 = 0.f, z4 = 0.f;
      Ids id1 = id;
      const float sa0 = kz ? a.sp.sdx0 : sx_cur;
      if (ok) {
        const float *U0 = uring + s0 * P::SU, *U1 = uring + s1 * P::SU;
        float xj[4], yj[4], zj[4], t1[4], qx[4];
        ld4(U0 + Lu, x0);
        ld4(U0 + Lu + KW, xj);
        ld4(U0 + YO + Lu - KW, yj);
        ld4(U0 + ZO + Lu + KW, zj);
        ld4(U1 + YO + Lu, y1);
        ld4(U1 + ZO + Lu, z1);
        const float xk = U0[Lu + 4], yk = U0[YO + Lu + 4], zk = U0[ZO + Lu - 1];
        y4 = yk;
        if (edge) z4 = U0[ZO + Lu + 4];
        id1 = read_ids(mring + s1 * P::SM);
        const float sx0 = kz ? a.sp.fdz0 : fx_cur;
        // material rows: one lookup where the neighbourhood is of one material
        const unsigned sp = (id.c & 0xffu) * 0x01010101u;
        const bool uni = (((id.c ^ sp) | (id.z ^ sp) | (id.y ^ sp)) | ((id.yz ^ sp) | (id1.z ^ sp) | (id1.y ^ sp))) == 0u;
        auto point = [&](const int q, const float* c, const float c4, const float c5, const float c6) {
          const float e1 = S::sub(x0[q], xm[q]), e2 = S::sub(y0[q], yj[q]), e3 = S::sub(z0[q], q ? z0[q ? q - 1 : 0] : zk);
          const float A = q ? sx_cur : sa0, Bq = q ? sb : sb0;
          t1[q] = S::tn1(a.dtab, c, e1, e2, e3, A, Bq, sdz[q]);
          t2[q] = S::tn1(a.dtab, c + 3, e1, e2, e3, A, Bq, sdz[q]);
          t3[q] = S::tn1(a.dtab, c + 6, e1, e2, e3, A, Bq, sdz[q]);
          t4[q] = S::ts(a.dtab, c4, S::sub(q < 3 ? y0[q < 3 ? q + 1 : 3] : yk, y0[q]), q ? fdz[q] : t4a0, S::sub(zj[q], z0[q]),
                        q ? fdyj : t4b0);
          t5[q] = S::ts(a.dtab, c5, S::sub(q < 3 ? x0[q < 3 ? q + 1 : 3] : xk, x0[q]), q ? fdz[q] : t5a0, S::sub(z1[q], z0[q]),
                        q ? fx_cur : sx0);
          t6[q] = S::ts(a.dtab, c6, S::sub(xj[q], x0[q]), q ? fdyj : t6a0, S::sub(y1[q], y0[q]), q ? fx_cur : sx0);
        };
        if (__all_sync(0xffffffffu, uni)) {
          const float4* row4 = reinterpret_cast<const float4*>(tab + 16 * (id.c & 0xffu));
          const float4 c0 = row4[0], c1 = row4[1], c2 = row4[2];
          const float qd = tab[16 * (id.c & 0xffu) + 12];
          const float c[9] = {c0.x, c0.y, c0.z, c0.w, c1.x, c1.y, c1.z, c1.w, c2.x};
#pragma unroll
          for (int q = 0; q < 4; q++) {
            point(q, c, c2.y, c2.z, c2.w);
            qx[q] = qy[q] = qz[q] = qd;
          }
        } else {
#pragma unroll
          for (int q = 0; q < 4; q++) {
            const float* rw = tab + 16 * id_of(id.c, q);
            const float4 c0 = reinterpret_cast<const float4*>(rw)[0], c1 = reinterpret_cast<const float4*>(rw)[1];
            const float c[9] = {c0.x, c0.y, c0.z, c0.w, c1.x, c1.y, c1.z, c1.w, rw[8]};
            point(q, c, tab[16 * id_of(id.yz, q) + 9], tab[16 * id_of(id1.z, q) + 10], tab[16 * id_of(id1.y, q) + 11]);
            qx[q] = rw[12];
            qy[q] = tab[16 * id_of(id.y, q) + 12];
            qz[q] = tab[16 * id_of(id.z, q) + 12];
          }
        }
        if (kz) t3[0] = 0.f;  // T3[1:-1,1:-1,0] = 0 (base_solver.py:418)
        if (i == 0) t1[0] = t1[1] = t1[2] = t1[3] = 0.f;
        if (i > ib) update_x(i, t1, pwring + s0 * P::PWS, qx, fx_prev);
#pragma unroll
        for (int q = 0; q < 4; q++) t1m[q] = t1[q], xm[q] = x0[q];
        xm4 = xk;
        if (lr == 0)
          *reinterpret_cast<float4*>(ex + buf * P::EX + warp * 32 + 4 * lc) = make_float4(t2[0], t2[1], t2[2], t2[3]);
        if (lr == 3) {
          *reinterpret_cast<float4*>(ex + (2 + buf) * P::EX + (warp + 1) * 32 + 4 * lc) = make_float4(t4[0], t4[1], t4[2], t4[3]);
          *reinterpret_cast<float4*>(ex + (4 + buf) * P::EX + (warp + 1) * 32 + 4 * lc) = make_float4(t6[0], t6[1], t6[2], t6[3]);
        }
      }
      asm volatile("fence.proxy.async.shared::cta;" ::: "memory");  // before the refill of plane i's slot (see above)
      if (block_any(!ok)) {
        ok = false;
        break;
      }
      // the neighbours' stresses
      float t2j[4], t4j[4], t6j[4];
#pragma unroll
      for (int q = 0; q < 4; q++) {
        t2j[q] = __shfl_down_sync(0xffffffffu, t2[q], 8);
        t4j[q] = __shfl_up_sync(0xffffffffu, t4[q], 8);
        t6j[q] = __shfl_up_sync(0xffffffffu, t6[q], 8);
      }
      float t3k = __shfl_down_sync(0xffffffffu, t3[0], 1), t4k = __shfl_up_sync(0xffffffffu, t4[3], 1),
            t5k = __shfl_up_sync(0xffffffffu, t5[3], 1);
      if (lr == 3) ld4(ex + buf * P::EX + (warp + 1) * 32 + 4 * lc, t2j);
      if (lr == 0) {
        ld4(ex + (2 + buf) * P::EX + warp * 32 + 4 * lc, t4j);
        ld4(ex + (4 + buf) * P::EX + warp * 32 + 4 * lc, t6j);
      }
      if (lc == 7) t3k = cx[buf * 16 + jl];
      if (lc == 0) t4k = cx[(2 + buf) * 16 + jl], t5k = cx[(4 + buf) * 16 + jl];
      const float* pw = pwring + s1 * P::PWS + Lp;
      const unsigned o = off_j + (unsigned)i * sxu;
      {  // uy (base_solver.py:449-455, 503-509)
        float v[4], kc[4], un[4], vn[4], cn[4];
        ld4(pw + P::PWC, v);
        ld4(pw + 4 * P::PWC, kc);
#pragma unroll
        for (int q = 0; q < 4; q++) {
          const float dv = S::div3(a.dtab, S::sub(t6[q], t6m[q]), q ? sx_cur : sa0, S::sub(t2j[q], t2[q]), q ? fdyj : uyb0,
                                   S::sub(t4[q], q ? t4[q ? q - 1 : 0] : t4k), sdz[q]);
          un[q] = update_value<S>(y0[q], Pw<float>{v[q], kc[q]}, dv, qy[q], a.dt, vn[q], cn[q]);
          if (i == 0) un[q] = y0[q], vn[q] = v[q], cn[q] = kc[q];  // not written by the reference: keeps its state
        }
        if (row_y) store_vec(r, 1, o, nz - 2 - k, rigid, a.abc[6], y0, y4, un, vn, cn);
      }
      {  // uz (base_solver.py:457-463, 511-516)
        float v[4], kc[4], un[4], vn[4], cn[4];
        ld4(pw + 2 * P::PWC, v);
        ld4(pw + 5 * P::PWC, kc);
#pragma unroll
        for (int q = 0; q < 4; q++) {
          const float dv = S::div3(a.dtab, S::sub(t5[q], t5m[q]), q ? sx_cur : sa0, S::sub(t4[q], t4j[q]), q ? sb : sb0,
                                   S::sub(q < 3 ? t3[q < 3 ? q + 1 : 3] : t3k, t3[q]), q ? fdz[q] : uzc0);
          un[q] = update_value<S>(z0[q], Pw<float>{v[q], kc[q]}, dv, qz[q], a.dt, vn[q], cn[q]);
          if (i == 0) {  // z0 holds the source there: the state itself is in global memory
            // (__ldcg: a plain load here costs registers, and the loop 4%)
            un[q] = row && k + q <= nz - 2 ? __ldcg(r.cur(2) + o + q) : 0.f;
            vn[q] = v[q], cn[q] = kc[q];
          }
        }
        if (row) store_vec(r, 2, o, nz - 3 - k, rigid, a.abc[7], z0, z4, un, vn, cn);
        if (kz && row) {  // surface uz (base_solver.py:114-116) and the non-finite guard
          if (rec) rec[(long long)i * ny] = un[0];
          if (!isfinite(un[0])) atomicOr(a.err, 1);
        }
      }
#pragma unroll
      for (int q = 0; q < 4; q++) {
        // what ux of plane i needs besides its x difference
        px[q] = __fmaf_rn(S::sub(t6[q], t6j[q]), q ? sb : sb0, __fmul_rn(S::sub(t5[q], q ? t5[q ? q - 1 : 0] : t5k), sdz[q]));
        t5m[q] = t5[q], t6m[q] = t6[q], y0[q] = y1[q], z0[q] = z1[q];
      }
      id = id1;
      s0 = s1;
      if (++s1 == NS) s1 = 0, par ^= 1;
      advance(i);
    }
    if (ok && ie < nx - 1) {  // ux of the last plane (x = N belongs to the face pass): T1 of plane ie
      const float* U0 = uring + s0 * P::SU;
      float x0[4], yj[4], t1[4], qx[4];
      ld4(U0 + Lu, x0);
      ld4(U0 + YO + Lu - KW, yj);
      const float zk = U0[ZO + Lu - 1], sa0 = kz ? a.sp.sdx0 : sx_cur;
#pragma unroll
      for (int q = 0; q < 4; q++) {
        const float* rw = tab + 16 * id_of(id.c, q);
        t1[q] = S::tn1(a.dtab, rw, S::sub(x0[q], xm[q]), S::sub(y0[q], yj[q]), S::sub(z0[q], q ? z0[q ? q - 1 : 0] : zk),
                       q ? sx_cur : sa0, q ? sb : sb0, sdz[q]);
        qx[q] = rw[12];
      }
      update_x(ie, t1, pwring + s0 * P::PWS, qx, fx_prev);
    }
    let_next_launch();
    // x = N (with its y = 0, y = N and z = N edges): the rows of the plane next
    // to it, as written above (ux of plane nx-3 may be the segment before's)
    if (ok && ie >= nx - 2 && row && writes_faces(true, TJ, ny)) {
#pragma unroll 1
      for (int c = 0; c < 3; c++) {
        if (c == 1 && !row_y) continue;
        const int p = c == 0 ? nx - 3 : nx - 2;
        if (p < ib || p >= ie) continue;
        const float4 t = *reinterpret_cast<const float4*>(r.out(c) + fidx(g, p, j, k));
        const float un[4] = {t.x, t.y, t.z, t.w};
        FaceRow in, out, edge_old;
        in.read(a, r, s, c, p, j, k);
        out.read(a, r, s, c, p + 1, j, k);
        const int dj = j == 1 ? -1 : j == ny - 2 - (c == 1 ? 1 : 0) ? 1 : 0;
        float u[4], w[4];
        out.face(a, a.abc[c == 0 ? 0 : 1], un, in, u);
        if (dj) {
          edge_old.read(a, r, s, c, p + 1, j + dj, k);
          edge_old.face(a, y_face_coef(a, c, dj), u, out, w);
          edge_old.write(a, r, tt, c, p + 1, j + dj, k, w);
        }
        out.write(a, r, tt, c, p + 1, j, k, u);
      }
    }
    block_wait();  // see the halo warp
  }
  if (!ok && producer) {
    // A wait ran out: flag it and drain the copies this block issued, so that
    // none writes into its shared memory after it returns (a copy that was
    // issued completes).  A stage armed without a copy (the test hook) has
    // nothing in flight.
    atomicOr(a.err, 2);
    for (int p = max(ib - 1, issued - NS + 1); p <= issued; p++) {
      if (a.skip_plane >= 0 && p == a.skip_plane) continue;
      const int q = p - ib + 1;
      mbar_wait(&bars[q % NS], (q / NS) & 1);
    }
  }
}
