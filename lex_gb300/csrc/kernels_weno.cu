// kernels_weno.cu - slow-mode WENO5 advection of one RK stage, as vertical marches.
//
// Flux-form advection of the prognostic fields (advection.py:9-149, fluxes :305-1281):
//
//   tendency(phi) = ( -sum_d d(m_d * phi_face)/dx_d + phi * div_at_phi ) / rho_at_phi
//
// Two kernels: k_weno_scalars_zm advects theta and qv together (their mass fluxes are the same
// rho0*u, rho0*v, rho0*w on the cell faces), k_weno_momentum_zm advects u, v and w together (their
// mass fluxes are averages of the three winds).  The upwind stencil is selected from the sign of
// the mass flux before the reconstruction; each face is evaluated once.
//
// Outputs (one_step_integration.py:258-296):
//   theta, qv : phi_next = phi^0 + dt_s * adv (+ dt_s * sgs); optional record of adv (+ sgs)
//   u         : R_u = adv + f v (Coriolis, pressure_gradient_coriolis.py:80-113) + sgs_u
//   v         : R_v = adv - f u + sgs_v
//   w         : R_w = adv + b8w (buoyancy at faces, pressure_equations.py:162-172) + sgs_w, with
//               adv = 0 on the bottom and lid faces (advection.py:146-147); wmode 1: adv only,
//               wmode 2: b8w only (diagnostics).
#include "lexgb_internal.cuh"

namespace lexgb {

namespace {

__device__ __forceinline__ int pmod(int i, int n) {
  i %= n;
  return i < 0 ? i + n : i;
}

// face value through column face H (between entries H-1 and H of an n-entry column), given
// s(H-3..H+2); entries outside 0..n-1 are never used; zero on the end faces.  Near-boundary
// rules of vertical_flux_scalar2 and friends (advection.py:327-406).  B2: weno5's, on the upward face next to
// the upper end (u and v on rows of other lengths than multiples of 4, as the boxes rounded it).
template <bool B2 = false>
__device__ __forceinline__ float vflux6(float m, float sm3, float sm2, float sm1, float s0, float sp1, float sp2, int H,
                                        int n, float eps) {
  if (H <= 0 || H >= n) return 0.f;
  const bool up = m >= 0.f;
  float r;
  if (H >= 3 && H <= n - 3) {
    r = weno5(up ? sm3 : sp2, up ? sm2 : sp1, up ? sm1 : s0, up ? s0 : sm1, up ? sp1 : sm2, eps);
  } else if (up) {
    if (H == 1)
      r = 0.5f * (sm1 + s0);
    else if (H == 2 || H == n - 1)
      r = weno3(sm2, sm1, s0, eps);
    else  // H == n-2
      r = weno5<B2>(sm3, sm2, sm1, s0, sp1, eps);
  } else {
    if (H == n - 1)
      r = 0.5f * (s0 + sm1);
    else if (H == 1 || H == n - 2)
      r = weno3(sp1, s0, sm1, eps);
    else  // H == 2
      r = weno5(sp2, sp1, s0, sm1, sm2, eps);
  }
  return m * r;
}

// ================================================================================================
// theta and qv
// ================================================================================================
struct ScalarArgs {
  const float* div;
  const float* T0;  // values at the start of the big step (may alias the outputs)
  const float* q0;
  const float* sgsT;
  const float* sgsQ;
  float* Tn;
  float* qn;
  float* recT;
  float* recQ;
  float dts;
  float* div_out;   // when set, div(rho0 u) and theta_rho of the state are computed here (div then
  float* trho_out;  // unused as an input) and written out
};

__device__ __forceinline__ float2 vflux6x2(float m, float2 sm3, float2 sm2, float2 sm1, float2 s0, float2 sp1,
                                           float2 sp2, int H, int n, float2 eps) {
  if (H <= 0 || H >= n) return f2(0.f);
  const bool up = m >= 0.f;
  float2 r;
  if (H >= 3 && H <= n - 3) {
    r = weno5x2(sel2(up, sm3, sp2), sel2(up, sm2, sp1), sel2(up, sm1, s0), sel2(up, s0, sm1), sel2(up, sp1, sm2), eps);
  } else if (up) {
    if (H == 1)
      r = mul2(f2(0.5f), add2(sm1, s0));
    else if (H == 2 || H == n - 1)
      r = weno3x2(sm2, sm1, s0, eps);
    else  // H == n-2
      r = weno5x2(sm3, sm2, sm1, s0, sp1, eps);
  } else {
    if (H == n - 1)
      r = mul2(f2(0.5f), add2(s0, sm1));
    else if (H == 1 || H == n - 2)
      r = weno3x2(sp1, s0, sm1, eps);
    else  // H == 2
      r = weno5x2(sp2, sp1, s0, sm1, sm2, eps);
  }
  return mul2(f2(m), r);
}

// ================================================================================================
// theta and qv, vertical march
//
// A block owns 32 x 8 columns (one thread each) and marches up a chunk of levels (zm_chunk).  For the x and
// y faces of a level it stages that level's plane of theta and qv with a 3-cell halo (40 x 14
// values, x widened to 4-aligned 16-byte pieces) by cp.async into a two-slot ring, the next level's
// plane in flight while the current one is used; the vertical stencil of a thread's own column
// slides through registers (s(k-3) .. s(k+2)), so no z halo is staged.  Each face flux is evaluated
// once: a thread its point's west, south and bottom faces; warp 0 also the 8 east-edge x faces,
// (the mass-flux winds and the stencil's next column value are loaded one level ahead)
// warp 1 the 32 north-edge y faces.  The bottom face of level k+1 is the top face of level k, so a
// level's tendency is completed in the next iteration.  Rows that do not start on 16-byte
// boundaries (nx % 4 != 0) are staged in 4-byte pieces (Stager): 102x75x59 22.5 us (theta, qv) and
// 36.9 us (u, v, w); one 32 x 4 x 4 box with a 3-D halo per block took 27.2 (with a kernel of its own
// for the divergence) and 37.5.  On such rows (V16 false) the marches keep the boxes' arithmetic, bit
// for bit: divisions by rho0, u, v and w reconstructed one by one, products and sums contracted as diff,
// sum2 and sum3 say.  In the other rows' arithmetic (reciprocals, packed reconstructions) u, v and w
// took 31.8 us, and the states differed in their last bits: that much moves the sign of a mass flux
// somewhere, where an adjoint jumps (up to 3e-3 of its rms at single points).
// ================================================================================================
constexpr int ZX = 32, ZY = 8, ZHX = 4, ZHY = 3;
constexpr int ZPX = ZX + 2 * ZHX, ZPY = ZY + 2 * ZHY;   // staged plane 40 x 14
constexpr int ZNT = ZX * ZY;
constexpr int kScalarsZmBlocks = 3;   // resident blocks per SM the theta/qv march is compiled for (measured
                                      // 92 us at 3, 120 us at 4 for 192 x 192 x 96)

// resident blocks on the device (SMs x blocks per SM) of the momentum and theta/qv marches, set by
// init_weno_attributes
int g_zm_slots = 304, g_zs_slots = 608;

// levels per block of a vertical march: as many level chunks as make one wave of resident blocks, down
// to single levels, and at most nine levels.  A chunk costs about one level more than it owns, but a small
// grid is bound by the serial march: theta/qv + u,v,w at 16x16x12 take 53 us in chunks of 8 levels and
// 14.5 us in chunks of 1, 32^3 39 and 14.5, 64^3 41 and 31 (chunks of 3).  And where one wave leaves SMs
// with a block less than others, for the whole march, short chunks even that out; a step with one wave,
// 6, 9 and 16 levels: 240x240x120 (240 tiles on 456 places) 4.74, 4.21, 4.16, 4.16 ms, 320x200x60 2.53,
// 2.32, 2.29, 2.32, 256x256x64 3.04, 2.82, 2.79, 2.83, 192x192x96 2.16, 2.17, 2.14, 2.16, 128x128x64
// 0.68, 0.69, 0.67, 0.68.
inline int zm_chunk(const Dims& d, int slots) {
  const int tiles = ((d.nx + 31) / 32) * ((d.ny + 7) / 8);
  const int nch = max(1, min(slots / tiles, d.nz));
  return min((d.nz + nch - 1) / nch, 9);
}

__device__ __forceinline__ void cp_async16(unsigned sa, const void* gmem) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(sa), "l"(gmem) : "memory");
}
__device__ __forceinline__ void cp_async4(unsigned sa, const void* gmem) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(sa), "l"(gmem) : "memory");
}
__device__ __forceinline__ unsigned smem_addr(const void* p) { return (unsigned)__cvta_generic_to_shared(p); }
constexpr unsigned kSlotBytes = ZPY * ZPX * sizeof(float);   // one staged plane
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N>
__device__ __forceinline__ void cp_async_wait() { asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory"); }

// Staging of planes by cp.async, at the same in-plane offsets on every level.  Rows on 16-byte
// boundaries (V16, nx % 4 == 0): thread t < 140 copies piece t (row t / 10, x piece t % 10).
constexpr int ZCHUNKS = ZPY * (ZPX / 4);                 // 16-byte pieces of one field's plane
template <bool V16>
struct Stager {
  bool stager;
  int sr, sc, soff;
  __device__ __forceinline__ Stager(int tid, int i0, int j0, int nx, int ny) {
    stager = tid < ZCHUNKS;
    sr = stager ? tid / (ZPX / 4) : 0;
    sc = 4 * (tid % (ZPX / 4));
    soff = pmod(j0 - ZHY + sr, ny) * nx + pmod(i0 - ZHX + sc, nx);
  }
  // the thread's first piece of a plane in shared memory
  __device__ __forceinline__ unsigned at(const float (&plane)[ZPY][ZPX]) const { return smem_addr(&plane[sr][sc]); }
  static __device__ __forceinline__ void cp(unsigned dst, const float* src) { cp_async16(dst, src); }
  // f(offset in the level's plane, byte offset from at()) for each of the thread's pieces
  template <class F>
  __device__ __forceinline__ void each(const F& f) const {
    if (stager) f(soff, 0u);
  }
};
// Rows on any 4-byte boundary: thread t copies values t, t + 256 and t + 512 of the 560.
template <>
struct Stager<false> {
  int goff[3], tid;
  __device__ __forceinline__ Stager(int t, int i0, int j0, int nx, int ny) : tid(t) {
#pragma unroll
    for (int m = 0; m < 3; ++m) {
      const int e = t + m * ZNT;
      goff[m] = pmod(j0 - ZHY + e / ZPX, ny) * nx + pmod(i0 - ZHX + e % ZPX, nx);
    }
  }
  __device__ __forceinline__ unsigned at(const float (&plane)[ZPY][ZPX]) const { return smem_addr(plane) + 4 * tid; }
  static __device__ __forceinline__ void cp(unsigned dst, const float* src) { cp_async4(dst, src); }
  template <class F>
  __device__ __forceinline__ void each(const F& f) const {
#pragma unroll
    for (int m = 0; m < 3; ++m)
      if (tid + m * ZNT < ZPY * ZPX) f(goff[m], 4u * m * ZNT);
  }
};

// the per-point values a level needs beyond the staged plane (loaded one level ahead)
struct ZLevel {
  float u, v, w, ue, ve;
  float2 top;   // the column value three levels up, for the register stencil
};

// Products and sums of the marches on rows of other lengths than multiples of 4, each rounded as written.
// r a - s b and a da + b db + c dc:
__device__ __forceinline__ float diff(float r, float a, float s, float b) { return __fmaf_rn(r, a, -__fmul_rn(s, b)); }
__device__ __forceinline__ float sum2(float a, float da, float b, float db) { return __fmaf_rn(a, da, __fmul_rn(b, db)); }
__device__ __forceinline__ float sum3(float a, float da, float b, float db, float c, float dc) {
  return __fmaf_rn(c, dc, sum2(a, da, b, db));
}

// FUSED: also form div(rho0 u) and theta_rho of the state (a.div_out, a.trho_out) instead of reading a.div
template <bool FUSED, bool V16>
__global__ void __launch_bounds__(ZNT, kScalarsZmBlocks) k_weno_scalars_zm(Dims d, Phys ph, Cols c, State s,
                                                                          ScalarArgs a, int zc) {
  __shared__ __align__(16) float pT[2][ZPY][ZPX];
  __shared__ __align__(16) float pQ[2][ZPY][ZPX];
  __shared__ float2 xF[ZY][ZX + 1];
  __shared__ float2 yF[ZY + 1][ZX];
  __shared__ float sMx[ZY][ZX + 1];  // FUSED: rho0 u on the west faces of the level's cells and the east edge
  __shared__ float sMy[ZY + 1][ZX];  //        rho0 v on the south faces and the north edge
  const int nx = d.nx, ny = d.ny, nz = d.nz, plane = d.plane();
  const int tx = threadIdx.x & 31, ty = threadIdx.x >> 5, tid = threadIdx.x;
  const int i0 = blockIdx.x * ZX, j0 = blockIdx.y * ZY;
  const int kb = blockIdx.z * zc, ke = min(kb + zc, nz);
  constexpr bool fused = FUSED;
  const int i = i0 + tx, j = j0 + ty;
  const bool col_own = i < nx && j < ny;
  // wrapped coordinates by full modulo: a tile and its halo may reach several periods past a
  // narrow grid (nx, ny >= 4)
  const int ic = pmod(i, nx), jc = pmod(j, ny);   // in-range column for loads
  const int cidx = jc * nx + ic;
  const int eidx = pmod(j0 + tx, ny) * nx + pmod(i0 + ZX, nx);  // warp 0: row tx's east-edge face
  const int nidx = pmod(j0 + ZY, ny) * nx + pmod(i0 + tx, nx);  // warp 1: column tx's north-edge face
  const float2 eps = make_float2(kWepsTheta, kWepsQv);

  const Stager<V16> sg(tid, i0, j0, nx, ny);
  const unsigned aT = sg.at(pT[0]), aQ = sg.at(pQ[0]);
  auto stage = [&](int k, int b) {
    sg.each([&](int g, unsigned e) {
      const size_t o = (size_t)k * plane + g;
      sg.cp(aT + b * kSlotBytes + e, s.T + o);
      sg.cp(aQ + b * kSlotBytes + e, s.q + o);
    });
    cp_async_commit();
  };
  auto colv = [&](int k) {
    const size_t g = (size_t)clampi(k, 0, nz - 1) * plane + cidx;
    return make_float2(__ldg(s.T + g), __ldg(s.q + g));
  };
  // level k's loads (k <= ke; level ke only needs w and the stencil value)
  auto fetch = [&](int k) {
    ZLevel L{0.f, 0.f, 0.f, 0.f, 0.f, make_float2(0.f, 0.f)};
    const size_t base = (size_t)min(k, nz - 1) * plane;
    if (k < nz) {
      L.u = __ldg(s.u + base + cidx);
      L.v = __ldg(s.v + base + cidx);
      if (ty == 0 && tx < ZY) L.ue = __ldg(s.u + base + eidx);
      if (ty == 1) L.ve = __ldg(s.v + base + nidx);
    }
    // faces 0 and nz carry no mass flux but enter the divergence as stored (k_div_trho reads them too)
    if (col_own && (fused || (k >= 1 && k < nz))) L.w = __ldg(s.w + (size_t)k * plane + cidx);
    L.top = colv(k + 3);
    return L;
  };

  stage(kb, 0);
  float2 cl[6];
#pragma unroll
  for (int m = 0; m < 6; ++m) cl[m] = colv(kb - 3 + m);
  ZLevel cur = fetch(kb);
  float2 zprev = f2(0.f), inner = f2(0.f), own = f2(0.f);
  float dv = 0.f, sT = 0.f, sQ = 0.f, T0 = 0.f, Q0 = 0.f;
  for (int k = kb; k <= ke; ++k) {
    const bool lev = k < ke;
    const ZLevel nxt = lev ? fetch(k + 1) : cur;   // one level ahead
    // bottom face of level k (top face of level k-1)
    const float mz = (col_own && k >= 1 && k < nz) ? c.rho_face[k] * cur.w : 0.f;
    const float2 zf = vflux6x2(mz, cl[0], cl[1], cl[2], cl[3], cl[4], cl[5], k, nz, eps);
    if (k > kb && col_own) {  // level k-1 complete
      const int km = k - 1;
      const size_t id = (size_t)km * plane + cidx;
      const float ri = V16 ? c.rho_inv[km] : c.rho[km];
      const float2 cv = fma2(sub2(zf, zprev), f2(-ph.rdz), inner);
      // 1/rho0 as a correctly rounded column value, or a division
      const float advT = V16 ? (cv.x + own.x * dv) * ri : (cv.x + own.x * dv) / ri;
      const float advQ = V16 ? (cv.y + own.y * dv) * ri : (cv.y + own.y * dv) / ri;
      float Tn = T0 + advT * a.dts, Qn = Q0 + advQ * a.dts, rT = advT, rQ = advQ;
      if (a.sgsT) {
        Tn = Tn + sT * a.dts;
        Qn = Qn + sQ * a.dts;
        rT = rT + sT;
        rQ = rQ + sQ;
      }
      if (a.Tn) a.Tn[id] = Tn;
      if (a.qn) a.qn[id] = Qn;
      if (a.recT) a.recT[id] = rT;
      if (a.recQ) a.recQ[id] = rQ;
    }
    zprev = zf;
    if (!lev) break;
    // x and y faces of level k; threads past the grid's end (partial tiles) evaluate the wrapped
    // faces: their west / south face is the periodic east / north face of the last column / row
    const bool next = k + 1 < ke;
    if (next) stage(k + 1, (k + 1 - kb) & 1);
    const float r = c.rho[k];
    const float mx = r * cur.u, my = r * cur.v, mxe = r * cur.ue, mye = r * cur.ve;
    if (col_own) {  // used when the level is completed, in the next iteration
      const size_t id = (size_t)k * plane + cidx;
      if (!fused) dv = __ldg(a.div + id);
      if (a.sgsT) {
        sT = __ldg(a.sgsT + id);
        sQ = __ldg(a.sgsQ + id);
      }
      T0 = a.T0[id];  // may alias the output: plain loads, same thread, before its write
      Q0 = a.q0[id];
    }
    if (next) cp_async_wait<1>(); else cp_async_wait<0>();
    __syncthreads();
    const int b = (k - kb) & 1;
    const float(&PT)[ZPY][ZPX] = pT[b];
    const float(&PQ)[ZPY][ZPX] = pQ[b];
    auto v2 = [&](int ry, int rx) { return make_float2(PT[ry][rx], PQ[ry][rx]); };
    const int lx = tx + ZHX, ly = ty + ZHY;
    own = v2(ly, lx);
    float dvz = 0.f;
    if (fused) {
      sMx[ty][tx] = V16 ? mx : cur.u;
      sMy[ty][tx] = V16 ? my : cur.v;
      if (ty == 0 && tx < ZY) sMx[tx][ZX] = V16 ? mxe : cur.ue;
      if (ty == 1) sMy[ZY][tx] = V16 ? mye : cur.ve;
      dvz = V16 ? (c.rho_face0[k + 1] * nxt.w - c.rho_face0[k] * cur.w) * ph.rdz
                : diff(c.rho_face0[k + 1], nxt.w, c.rho_face0[k], cur.w);
    }
    xF[ty][tx] = weno_flux_x2(mx, v2(ly, lx - 3), v2(ly, lx - 2), v2(ly, lx - 1), v2(ly, lx), v2(ly, lx + 1),
                              v2(ly, lx + 2), eps);
    yF[ty][tx] = weno_flux_x2(my, v2(ly - 3, lx), v2(ly - 2, lx), v2(ly - 1, lx), v2(ly, lx), v2(ly + 1, lx),
                              v2(ly + 2, lx), eps);
    if (ty == 0 && tx < ZY) {  // east-edge x face of row tx
      const int ry = tx + ZHY, rx = ZX + ZHX;
      xF[tx][ZX] = weno_flux_x2(mxe, v2(ry, rx - 3), v2(ry, rx - 2), v2(ry, rx - 1), v2(ry, rx), v2(ry, rx + 1),
                                v2(ry, rx + 2), eps);
    }
    if (ty == 1) {  // north-edge y face of column tx
      const int ry = ZY + ZHY, rx = tx + ZHX;
      yF[ZY][tx] = weno_flux_x2(mye, v2(ry - 3, rx), v2(ry - 2, rx), v2(ry - 1, rx), v2(ry, rx), v2(ry + 1, rx),
                                v2(ry + 2, rx), eps);
    }
    __syncthreads();
    inner = fma2(sub2(yF[ty + 1][tx], yF[ty][tx]), f2(-ph.rdy), mul2(sub2(xF[ty][tx + 1], xF[ty][tx]), f2(-ph.rdx)));
    if (fused && col_own) {  // get_divergence (advection.py:200-226) and theta_rho, as k_div_trho forms them
      if (V16) {
        const float dvx = (sMx[ty][tx + 1] - sMx[ty][tx]) * ph.rdx;
        const float dvy = (sMy[ty + 1][tx] - sMy[ty][tx]) * ph.rdy;
        dv = dvx + dvy + dvz;
      } else {
        dv = sum3(diff(r, sMx[ty][tx + 1], r, sMx[ty][tx]), ph.rdx, diff(r, sMy[ty + 1][tx], r, sMy[ty][tx]), ph.rdy,
                  dvz, ph.rdz);
      }
      const size_t id = (size_t)k * plane + cidx;
      a.div_out[id] = dv;
      a.trho_out[id] = theta_rho(own.x, own.y, ph.theta_ref);
    }
    // slide the column stencil up one level
#pragma unroll
    for (int m = 0; m < 5; ++m) cl[m] = cl[m + 1];
    cl[5] = cur.top;
    cur = nxt;
  }
}

// ================================================================================================
// u, v, w
// ================================================================================================
struct MomentumArgs {
  const float* div;
  const float* sgs_u;
  const float* sgs_v;
  const float* sgs_w;
  float* Ru;
  float* Rv;
  float* Rw;
  int wmode;
};

// ================================================================================================
// u, v and w, vertical march
//
// The tiling of k_weno_scalars_zm: a block owns 32 x 8 columns (one thread each) and marches up a
// chunk of levels.  Level k stages the planes of u and v at cell level k and of w at face level k
// (40 x 14 with halo, cp.async, two-slot ring; the next level's planes in flight while the current
// ones are used); the own columns of u, v and w slide through registers for the vertical stencils.
// Per thread and level: the x and y faces of u, of v and of w as three packed FP32x2 pairs (x face,
// y face, each upwinded by its own mass flux), the bottom faces of u and v as one more pair and the
// bottom face of w alone.  Edge faces: warp 0 the east x faces of u and v, warp 1 the north y faces
// of u and v, warp 2 the north y faces of w, warp 3 the east x faces of w.  Level k-1's tendencies
// are completed once the bottom faces of level k are known; the chunk at the lid adds w's face nz
// (no advection there).
// ================================================================================================
__device__ __forceinline__ float2 sel2m(bool p, bool q, float2 a, float2 b) {
  return make_float2(p ? a.x : b.x, q ? a.y : b.y);
}

// (m.x * upwind WENO5 of stencil .x, m.y * upwind WENO5 of stencil .y): two faces with mass fluxes of
// their own
template <bool PACKED>
__device__ __forceinline__ float2 weno_flux_2m(float2 m, float2 sm3, float2 sm2, float2 sm1, float2 s0, float2 sp1,
                                               float2 sp2, float2 eps) {
  if (!PACKED)
    return make_float2(weno_flux(m.x, sm3.x, sm2.x, sm1.x, s0.x, sp1.x, sp2.x, eps.x),
                       weno_flux(m.y, sm3.y, sm2.y, sm1.y, s0.y, sp1.y, sp2.y, eps.y));
  const bool p = m.x >= 0.f, q = m.y >= 0.f;
  return mul2(m, weno5x2(sel2m(p, q, sm3, sp2), sel2m(p, q, sm2, sp1), sel2m(p, q, sm1, s0), sel2m(p, q, s0, sm1),
                         sel2m(p, q, sp1, sm2), eps));
}

// vflux6 for two columns at the same face H: packed away from the ends, where each column's
// direction picks its own near-boundary rule
template <bool PACKED>
__device__ __forceinline__ float2 vflux6_2m(float2 m, float2 sm3, float2 sm2, float2 sm1, float2 s0, float2 sp1,
                                            float2 sp2, int H, int n, float eps) {
  if (H <= 0 || H >= n) return f2(0.f);
  if (PACKED && H >= 3 && H <= n - 3) return weno_flux_2m<true>(m, sm3, sm2, sm1, s0, sp1, sp2, f2(eps));
  return make_float2(vflux6<!PACKED>(m.x, sm3.x, sm2.x, sm1.x, s0.x, sp1.x, sp2.x, H, n, eps),
                     vflux6<!PACKED>(m.y, sm3.y, sm2.y, sm1.y, s0.y, sp1.y, sp2.y, H, n, eps));
}


template <bool V16>
__global__ void __launch_bounds__(ZNT, 3) k_weno_momentum_zm(Dims d, Phys ph, Cols c, State s, MomentumArgs a,
                                                              int zc) {
  __shared__ __align__(16) float pU[2][ZPY][ZPX];
  __shared__ __align__(16) float pV[2][ZPY][ZPX];
  __shared__ __align__(16) float pW[2][ZPY][ZPX];
  __shared__ float2 xUV[ZY][ZX + 1];   // x faces of (u, v)
  __shared__ float2 yUV[ZY + 1][ZX];   // y faces of (u, v)
  __shared__ float xW[ZY][ZX + 1];
  __shared__ float yW[ZY + 1][ZX];
  const int nx = d.nx, ny = d.ny, nz = d.nz, plane = d.plane();
  const int tx = threadIdx.x & 31, ty = threadIdx.x >> 5, tid = threadIdx.x;
  const int i0 = blockIdx.x * ZX, j0 = blockIdx.y * ZY;
  const int kb = blockIdx.z * zc, ke = min(kb + zc, nz);
  const int i = i0 + tx, j = j0 + ty;
  const bool col_own = i < nx && j < ny;
  const int cidx = pmod(j, ny) * nx + pmod(i, nx);     // threads past the grid's end: the wrapped column
  const int xmidx = pmod(j, ny) * nx + pmod(i - 1, nx);
  const int ymidx = pmod(j - 1, ny) * nx + pmod(i, nx);
  const int eidx = pmod(j0 + tx, ny) * nx + pmod(i0 + ZX, nx);  // warp 3: row tx's east point
  const int nidx = pmod(j0 + ZY, ny) * nx + pmod(i0 + tx, nx);  // warp 2: column tx's north point
  const float eps = kWepsMom;
  const Stager<V16> sg(tid, i0, j0, nx, ny);
  const unsigned sU = sg.at(pU[0]), sV = sg.at(pV[0]), sW = sg.at(pW[0]);
  // stage level k into slot b: u and v at cell level k (the lid's level for k = nz), w at face k
  auto stage = [&](int k, int b) {
    sg.each([&](int g, unsigned e) {
      const size_t ouv = (size_t)min(k, nz - 1) * plane + g, ow = (size_t)k * plane + g;
      sg.cp(sU + e + b * kSlotBytes, s.u + ouv);
      sg.cp(sV + e + b * kSlotBytes, s.v + ouv);
      sg.cp(sW + e + b * kSlotBytes, s.w + ow);
    });
    cp_async_commit();
  };
  auto col = [&](const float* f, int k, int top) { return __ldg(f + (size_t)clampi(k, 0, top) * plane + cidx); };
  auto bq = [&](int k) {
    const size_t q = (size_t)k * plane + cidx;
    return buoyancy_at(__ldg(s.T + q), __ldg(s.q + q), k, c);
  };

  stage(kb, 0);
  float su[6], sv[6], sw[6];   // own columns: levels k-3 .. k+2 (u, v) and faces k-3 .. k+2 (w)
#pragma unroll
  for (int m = 0; m < 6; ++m) {
    su[m] = col(s.u, kb - 3 + m, nz - 1);
    sv[m] = col(s.v, kb - 3 + m, nz - 1);
    sw[m] = col(s.w, kb - 3 + m, nz);
  }
  // edge lanes of w's faces: the level below's u at the east point (warp 3), v at the north point (warp 2)
  float eprev = 0.f;
  if (kb >= 1 && ty == 3 && tx < ZY) eprev = __ldg(s.u + (size_t)(kb - 1) * plane + eidx);
  if (kb >= 1 && ty == 2) eprev = __ldg(s.v + (size_t)(kb - 1) * plane + nidx);
  // the level being completed: x + y flux differences, Coriolis, div (own, i-1, j-1), the level
  // below's div, SGS, buoyancy (and the level below's)
  float2 inUV = f2(0.f);
  float inW = 0.f, corU = 0.f, corV = 0.f, dcC = 0.f, dxC = 0.f, dyC = 0.f, dzC = 0.f;
  float sgU = 0.f, sgV = 0.f, sgW = 0.f, bC = 0.f, bP = 0.f;
  if (kb >= 1 && col_own) {
    dcC = __ldg(a.div + (size_t)(kb - 1) * plane + cidx);
    if (a.wmode != 1) bC = bq(kb - 1);
  }
  float2 zpUV = f2(0.f);   // bottom faces of the level being completed
  float zpW = 0.f;
  const int lx = tx + ZHX, ly = ty + ZHY;
  for (int k = kb; k <= ke; ++k) {
    const bool lev = k < ke;
    const bool more = k + 1 <= ke;
    // the stencils' next column values and this level's per-point inputs, loaded ahead of their use
    const float tu = col(s.u, k + 3, nz - 1), tv = col(s.v, k + 3, nz - 1), tw = col(s.w, k + 3, nz);
    if (more) stage(k + 1, (k + 1 - kb) & 1);
    float dcN = 0.f, dxN = 0.f, dyN = 0.f, sgUN = 0.f, sgVN = 0.f, sgWN = 0.f, TN = 0.f, QN = 0.f;
    if (lev && col_own) {
      const size_t o = (size_t)k * plane;
      dcN = __ldg(a.div + o + cidx);
      dxN = __ldg(a.div + o + xmidx);
      dyN = __ldg(a.div + o + ymidx);
      if (a.sgs_u) {
        sgUN = __ldg(a.sgs_u + o + cidx);
        sgVN = __ldg(a.sgs_v + o + cidx);
      }
      if (a.sgs_w) sgWN = __ldg(a.sgs_w + o + cidx);
      if (a.wmode != 1) {
        TN = __ldg(s.T + o + cidx);
        QN = __ldg(s.q + o + cidx);
      }
    }
    if (more) cp_async_wait<1>(); else cp_async_wait<0>();
    __syncthreads();
    const int b = (k - kb) & 1;
    const float(&PU)[ZPY][ZPX] = pU[b];
    const float(&PV)[ZPY][ZPX] = pV[b];
    const float(&PW)[ZPY][ZPX] = pW[b];
    // bottom faces of level k: u and v through the face between cells k-1 and k (mass flux from w
    // on face k), w through cell k-1
    float2 zUV = f2(0.f);
    if (k >= 1 && k < nz) {
      const float rf = c.rho_face[k];
      const float2 m = make_float2(mass_flux(rf, PW[ly][lx - 1], rf, PW[ly][lx]),
                                   mass_flux(rf, PW[ly - 1][lx], rf, PW[ly][lx]));
      zUV = vflux6_2m<V16>(m, make_float2(su[0], sv[0]), make_float2(su[1], sv[1]), make_float2(su[2], sv[2]),
                           make_float2(su[3], sv[3]), make_float2(su[4], sv[4]), make_float2(su[5], sv[5]), k, nz, eps);
    }
    const float zW = (k >= 1) ? vflux6(mass_flux(sw[2], sw[3], c.rho[k - 1]), sw[0], sw[1], sw[2], sw[3], sw[4],
                                       sw[5], k, nz + 1, eps)
                              : 0.f;
    if (k > kb && col_own) {  // level k-1 complete
      const int kk = k - 1;
      const size_t id = (size_t)kk * plane + cidx;
      float Ru, Rv;
      if (V16) {
        const float ri = c.rho_inv[kk];   // 1/rho0, 1/rho0 on the face: correctly rounded column values
        const float2 cuv = fma2(sub2(zUV, zpUV), f2(-ph.rdz), inUV);
        Ru = (cuv.x + su[2] * (0.5f * (dxC + dcC))) * ri;
        Rv = (cuv.y + sv[2] * (0.5f * (dyC + dcC))) * ri;
        if (ph.cor_opt) {
          Ru = Ru + corU;
          Rv = Rv - corV;
        }
      } else {
        const float r1 = c.rho[kk];
        Ru = (su[2] * (0.5f * (dxC + dcC)) - __fmaf_rn(__fsub_rn(zUV.x, zpUV.x), ph.rdz, inUV.x)) / r1;
        Rv = (sv[2] * (0.5f * (dyC + dcC)) - __fmaf_rn(__fsub_rn(zUV.y, zpUV.y), ph.rdz, inUV.y)) / r1;
        if (ph.cor_opt) {
          Ru = __fmaf_rn(ph.f_cor * 0.25f, corU, Ru);
          Rv = __fmaf_rn(-ph.f_cor, corV, Rv);
        }
      }
      if (a.sgs_u) {
        Ru = Ru + sgU;
        Rv = Rv + sgV;
      }
      a.Ru[id] = Ru;
      a.Rv[id] = Rv;
      float adv = 0.f;   // w on face kk
      if (kk >= 1) {
        if (V16) {
          const float cw = fmaf(zW - zpW, -ph.rdz, inW);
          adv = (cw + sw[2] * (0.5f * (dzC + dcC))) * c.rho_w_inv[kk];
        } else {
          adv = (sw[2] * (0.5f * (dzC + dcC)) - __fmaf_rn(zW - zpW, ph.rdz, inW)) / (0.5f * (c.rho[kk - 1] + c.rho[kk]));
        }
      }
      float Rw = adv;
      if (a.wmode != 1) {
        const float b8w = kk == 0 ? 1.875f * bq(0) - 1.25f * bq(1) + 0.375f * bq(2) : 0.5f * (bP + bC);
        if (a.wmode == 2) {
          Rw = b8w;
        } else {
          Rw = adv + b8w;
          if (a.sgs_w) Rw = Rw + sgW;
        }
      }
      a.Rw[id] = Rw;
    }
    zpUV = zUV;
    zpW = zW;
    if (!lev) break;
    // x and y faces of level k
    const float r = c.rho[k], rm = k >= 1 ? c.rho[k - 1] : 0.f;
    auto xs = [&](const float(&P)[ZPY][ZPX], int ry, int rx, int o) { return P[ry][rx + o]; };
    {
      const float2 mu = make_float2(mass_flux(PU[ly][lx - 1], PU[ly][lx], r),          // cell between u's
                                    mass_flux(r, PV[ly][lx - 1], r, PV[ly][lx]));      // corner
      const float2 fu = weno_flux_2m<V16>(mu, make_float2(PU[ly][lx - 3], PU[ly - 3][lx]),
                                          make_float2(PU[ly][lx - 2], PU[ly - 2][lx]),
                                          make_float2(PU[ly][lx - 1], PU[ly - 1][lx]), make_float2(PU[ly][lx], PU[ly][lx]),
                                          make_float2(PU[ly][lx + 1], PU[ly + 1][lx]),
                                          make_float2(PU[ly][lx + 2], PU[ly + 2][lx]), f2(eps));
      const float2 mv = make_float2(mass_flux(r, PU[ly - 1][lx], r, PU[ly][lx]),       // corner
                                    mass_flux(PV[ly - 1][lx], PV[ly][lx], r));         // cell between v's
      const float2 fv = weno_flux_2m<V16>(mv, make_float2(PV[ly][lx - 3], PV[ly - 3][lx]),
                                          make_float2(PV[ly][lx - 2], PV[ly - 2][lx]),
                                          make_float2(PV[ly][lx - 1], PV[ly - 1][lx]), make_float2(PV[ly][lx], PV[ly][lx]),
                                          make_float2(PV[ly][lx + 1], PV[ly + 1][lx]),
                                          make_float2(PV[ly][lx + 2], PV[ly + 2][lx]), f2(eps));
      xUV[ty][tx] = make_float2(fu.x, fv.x);
      yUV[ty][tx] = make_float2(fu.y, fv.y);
    }
    if (k >= 1 && k < nz) {  // w's lateral faces on interior face levels
      const float2 mw = make_float2(mass_flux(rm, su[2], r, su[3]), mass_flux(rm, sv[2], r, sv[3]));
      const float2 fw = weno_flux_2m<V16>(mw, make_float2(PW[ly][lx - 3], PW[ly - 3][lx]),
                                          make_float2(PW[ly][lx - 2], PW[ly - 2][lx]),
                                          make_float2(PW[ly][lx - 1], PW[ly - 1][lx]), make_float2(PW[ly][lx], PW[ly][lx]),
                                          make_float2(PW[ly][lx + 1], PW[ly + 1][lx]),
                                          make_float2(PW[ly][lx + 2], PW[ly + 2][lx]), f2(eps));
      xW[ty][tx] = fw.x;
      yW[ty][tx] = fw.y;
    } else {
      xW[ty][tx] = 0.f;
      yW[ty][tx] = 0.f;
    }
    float corUN = 0.f, corVN = 0.f;
    if (ph.cor_opt) {  // f v at u points, f u at v points (4-point averages)
      if (V16) {
        corUN = ph.f_cor * 0.25f * (PV[ly][lx - 1] + PV[ly + 1][lx - 1] + PV[ly][lx] + PV[ly + 1][lx]);
        const float fu = 0.25f * (PU[ly - 1][lx] + PU[ly][lx] + PU[ly - 1][lx + 1] + PU[ly][lx + 1]);
        corVN = ph.cor_opt == 2 ? ph.f_cor * (fu - 1.0f) : ph.f_cor * fu;
      } else {   // without the factors, which come with the sum they are added to
        corUN = PV[ly][lx - 1] + PV[ly + 1][lx - 1] + PV[ly][lx] + PV[ly + 1][lx];
        corVN = 0.25f * (PU[ly - 1][lx] + PU[ly][lx] + PU[ly - 1][lx + 1] + PU[ly][lx + 1]);
        if (ph.cor_opt == 2) corVN = corVN - 1.0f;
      }
    }
    if (ty == 0 && tx < ZY) {  // east x faces of u and v, row tx
      const int ry = tx + ZHY, rx = ZX + ZHX;
      const float2 m = make_float2(mass_flux(PU[ry][rx - 1], PU[ry][rx], r),
                                   mass_flux(r, PU[ry - 1][rx], r, PU[ry][rx]));
      xUV[tx][ZX] = weno_flux_2m<V16>(m, make_float2(xs(PU, ry, rx, -3), xs(PV, ry, rx, -3)),
                                      make_float2(xs(PU, ry, rx, -2), xs(PV, ry, rx, -2)),
                                      make_float2(xs(PU, ry, rx, -1), xs(PV, ry, rx, -1)),
                                      make_float2(xs(PU, ry, rx, 0), xs(PV, ry, rx, 0)),
                                      make_float2(xs(PU, ry, rx, 1), xs(PV, ry, rx, 1)),
                                      make_float2(xs(PU, ry, rx, 2), xs(PV, ry, rx, 2)), f2(eps));
    } else if (ty == 1) {  // north y faces of u and v, column tx
      const int ry = ZY + ZHY, rx = tx + ZHX;
      const float2 m = make_float2(mass_flux(r, PV[ry][rx - 1], r, PV[ry][rx]),
                                   mass_flux(PV[ry - 1][rx], PV[ry][rx], r));
      yUV[ZY][tx] = weno_flux_2m<V16>(m, make_float2(PU[ry - 3][rx], PV[ry - 3][rx]),
                                      make_float2(PU[ry - 2][rx], PV[ry - 2][rx]),
                                      make_float2(PU[ry - 1][rx], PV[ry - 1][rx]), make_float2(PU[ry][rx], PV[ry][rx]),
                                      make_float2(PU[ry + 1][rx], PV[ry + 1][rx]),
                                      make_float2(PU[ry + 2][rx], PV[ry + 2][rx]), f2(eps));
    } else if (ty == 2) {  // north y faces of w, column tx
      const int ry = ZY + ZHY, rx = tx + ZHX;
      float f = 0.f;
      if (k >= 1 && k < nz)
        f = weno_flux(mass_flux(rm, eprev, r, PV[ry][rx]),
                      PW[ry - 3][rx], PW[ry - 2][rx], PW[ry - 1][rx],
                      PW[ry][rx], PW[ry + 1][rx], PW[ry + 2][rx], eps);
      yW[ZY][tx] = f;
      eprev = PV[ry][rx];
    } else if (ty == 3 && tx < ZY) {  // east x faces of w, row tx
      const int ry = tx + ZHY, rx = ZX + ZHX;
      float f = 0.f;
      if (k >= 1 && k < nz)
        f = weno_flux(mass_flux(rm, eprev, r, PU[ry][rx]),
                      PW[ry][rx - 3], PW[ry][rx - 2], PW[ry][rx - 1],
                      PW[ry][rx], PW[ry][rx + 1], PW[ry][rx + 2], eps);
      xW[tx][ZX] = f;
      eprev = PU[ry][rx];
    }
    __syncthreads();
    if (V16) {
      inUV = fma2(sub2(yUV[ty + 1][tx], yUV[ty][tx]), f2(-ph.rdy), mul2(sub2(xUV[ty][tx + 1], xUV[ty][tx]), f2(-ph.rdx)));
      inW = fmaf(yW[ty + 1][tx] - yW[ty][tx], -ph.rdy, (xW[ty][tx + 1] - xW[ty][tx]) * -ph.rdx);
    } else {
      const float2 xd = sub2(xUV[ty][tx + 1], xUV[ty][tx]), yd = sub2(yUV[ty + 1][tx], yUV[ty][tx]);
      inUV = make_float2(sum2(xd.x, ph.rdx, yd.x, ph.rdy), sum2(xd.y, ph.rdx, yd.y, ph.rdy));
      inW = sum2(xW[ty][tx + 1] - xW[ty][tx], ph.rdx, yW[ty + 1][tx] - yW[ty][tx], ph.rdy);
    }
    corU = corUN;
    corV = corVN;
    dzC = dcC;
    dcC = dcN;
    dxC = dxN;
    dyC = dyN;
    sgU = sgUN;
    sgV = sgVN;
    sgW = sgWN;
    bP = bC;
    if (a.wmode != 1 && col_own) bC = buoyancy_at(TN, QN, k, c);
#pragma unroll
    for (int m = 0; m < 5; ++m) {
      su[m] = su[m + 1];
      sv[m] = sv[m + 1];
      sw[m] = sw[m + 1];
    }
    su[5] = tu;
    sv[5] = tv;
    sw[5] = tw;
  }
  if (ke == nz && col_own) {  // w on the lid: no advection
    const size_t id = (size_t)nz * plane + cidx;
    float Rw = 0.f;
    if (a.wmode != 1) {
      const float b8w = 1.875f * bq(nz - 1) - 1.25f * bq(nz - 2) + 0.375f * bq(nz - 3);
      Rw = b8w;
      if (a.wmode == 0) {
        Rw = 0.f + b8w;
        if (a.sgs_w) Rw = Rw + __ldg(a.sgs_w + id);
      }
    }
    a.Rw[id] = Rw;
  }
}

}  // namespace

template <bool FUSED>
static void run_scalars(const Dims& d, const Phys& ph, const Cols& c, State in, const ScalarArgs& a, cudaStream_t st) {
  const int zc = zm_chunk(d, g_zs_slots);
  const dim3 g((d.nx + ZX - 1) / ZX, (d.ny + ZY - 1) / ZY, (d.nz + zc - 1) / zc);
  if (d.nx % 4 == 0)
    k_weno_scalars_zm<FUSED, true><<<g, ZNT, 0, st>>>(d, ph, c, in, a, zc);
  else
    k_weno_scalars_zm<FUSED, false><<<g, ZNT, 0, st>>>(d, ph, c, in, a, zc);
}

cudaError_t launch_adv_scalars(const Dims& d, const Phys& ph, const Cols& c, State in, const float* div,
                               const float* T0, const float* q0, Sgs sgs, float dts, SlowOut out, cudaStream_t st,
                               float* div_out, float* trho_out) {
  const ScalarArgs a{div, T0, q0, sgs.T, sgs.q, out.T_next, out.q_next, out.dT, out.dq, dts, div_out, trho_out};
  if (div_out)
    run_scalars<true>(d, ph, c, in, a, st);
  else
    run_scalars<false>(d, ph, c, in, a, st);
  return cudaGetLastError();
}

cudaError_t launch_adv_momentum(const Dims& d, const Phys& ph, const Cols& c, State in, const float* div, Sgs sgs,
                                float* Ru, float* Rv, float* Rw, int wmode, cudaStream_t st) {
  const MomentumArgs a{div, sgs.u, sgs.v, sgs.w, Ru, Rv, Rw, wmode};
  const int zc = zm_chunk(d, g_zm_slots);
  const dim3 g((d.nx + ZX - 1) / ZX, (d.ny + ZY - 1) / ZY, (d.nz + zc - 1) / zc);
  if (d.nx % 4 == 0)
    k_weno_momentum_zm<true><<<g, ZNT, 0, st>>>(d, ph, c, in, a, zc);
  else
    k_weno_momentum_zm<false><<<g, ZNT, 0, st>>>(d, ph, c, in, a, zc);
  return cudaGetLastError();
}

cudaError_t init_weno_attributes() {
  cudaError_t e;
  int dev = 0, sms = 0, nb = 0;
  if ((e = cudaGetDevice(&dev)) != cudaSuccess) return e;
  if ((e = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev)) != cudaSuccess) return e;
  if ((e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&nb, k_weno_momentum_zm<true>, ZNT, 0)) != cudaSuccess) return e;
  g_zm_slots = sms * max(nb, 1);
  if ((e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&nb, k_weno_scalars_zm<true, true>, ZNT, 0)) != cudaSuccess)
    return e;
  g_zs_slots = sms * max(nb, 1);
  return cudaSuccess;
}

}  // namespace lexgb
