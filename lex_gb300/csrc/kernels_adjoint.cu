// kernels_adjoint.cu - vector-Jacobian products (reverse mode) of the big-step operators.
//
// A thread owns the adjoint values it writes and sums the contributions of the forward outputs that
// depend on them, so there are no atomics and the results do not depend on scheduling.  The forward
// operators and their reference counterparts:
//
//   acoustic sub-step        one_step_integration.py:519-556 (k_acoustic_vec)
//   WENO flux divergence     advection.py:9-149, fluxes :305-1281 (k_weno_scalars_zm/momentum_zm)
//   mass divergence          advection.py:200-226 (k_div_trho)
//   theta_rho, buoyancy      one_step_integration.py:269, pressure_equations.py:162-172
//   Coriolis                 pressure_gradient_coriolis.py:80-113
//
// WENO adjoint: for each direction and every flux of the five advected fields (u, v, w, theta, qv), the
// flux adjoint Fbar = (cbar(right) - cbar(left)) / dx, the reconstruction W and its derivatives with
// respect to its stencil.  Fbar * m * dW/ds goes, as six slots, to the points p-3 .. p+2 of the flux between
// p-1 and p (k_adv_row_vjp, k_adv_march_vjp); the mass-flux adjoints Fbar * W go to the winds whose mass
// flux they are in a second kernel (k_adv_mass_vjp).
#include "lexgb_adjoint.cuh"
#include "smag_ops.cuh"

namespace lexgb {

namespace {

constexpr int AB = 256;
#define LD(p, idx) __ldg((p) + (idx))

constexpr float kHalfCp = (float)(0.5 * kCp);
constexpr float kRdCvA = (float)(kRd / kCv);

__device__ __forceinline__ int wrapx(int i, int n) { return i < 0 ? i + n : (i >= n ? i - n : i); }

// ---------------------------------------------------------------------------------------------
// reconstruction derivatives
// ---------------------------------------------------------------------------------------------
// W = weno5(a..e) (same formulas as weno5 in lexgb_internal.cuh) and dW/d(a..e) into g[0..4].
__device__ __forceinline__ float weno5_grad(float a, float b, float c, float d, float e, float eps, float* g) {
  const float t1 = a - 2.f * b + c, t2 = a - 4.f * b + 3.f * c;
  const float t3 = b - 2.f * c + d, t4 = b - d;
  const float t5 = c - 2.f * d + e, t6 = 3.f * c - 4.f * d + e;
  const float b1 = (13.f / 12.f) * t1 * t1 + 0.25f * t2 * t2;
  const float b2 = (13.f / 12.f) * t3 * t3 + 0.25f * t4 * t4;
  const float b3 = (13.f / 12.f) * t5 * t5 + 0.25f * t6 * t6;
  const float dd = b1 - b3, tau = fabsf(dd), sg = dd >= 0.f ? 1.f : -1.f;
  // one approximate reciprocal per denominator (the forward divides with div_approx)
  const float i1 = rcp_approx(b1 + eps), i2 = rcp_approx(b2 + eps), i3 = rcp_approx(b3 + eps);
  const float q1r = tau * i1, q2r = tau * i2, q3r = tau * i3;
  const float r1 = fminf(kRatioCap, q1r), r2 = fminf(kRatioCap, q2r), r3 = fminf(kRatioCap, q3r);
  const float w1 = 0.1f * (1.f + r1 * r1), w2 = 0.6f * (1.f + r2 * r2), w3 = 0.3f * (1.f + r3 * r3);
  const float q1 = (2.f / 6.f) * a + (-7.f / 6.f) * b + (11.f / 6.f) * c;
  const float q2 = (-1.f / 6.f) * b + (5.f / 6.f) * c + (2.f / 6.f) * d;
  const float q3 = (2.f / 6.f) * c + (5.f / 6.f) * d + (-1.f / 6.f) * e;
  const float iS = rcp_approx(w1 + w2 + w3);
  const float W = (w1 * q1 + w2 * q2 + w3 * q3) * iS;
  // reverse
  const float qb1 = w1 * iS, qb2 = w2 * iS, qb3 = w3 * iS;
  const float wb1 = (q1 - W) * iS, wb2 = (q2 - W) * iS, wb3 = (q3 - W) * iS;
  const float rb1 = q1r < kRatioCap ? wb1 * 0.2f * r1 : 0.f;
  const float rb2 = q2r < kRatioCap ? wb2 * 1.2f * r2 : 0.f;
  const float rb3 = q3r < kRatioCap ? wb3 * 0.6f * r3 : 0.f;
  const float taub = rb1 * i1 + rb2 * i2 + rb3 * i3;
  const float bb1 = -rb1 * r1 * i1 + taub * sg;
  const float bb2 = -rb2 * r2 * i2;
  const float bb3 = -rb3 * r3 * i3 - taub * sg;
  const float tb1 = bb1 * (13.f / 6.f) * t1, tb2 = bb1 * 0.5f * t2;
  const float tb3 = bb2 * (13.f / 6.f) * t3, tb4 = bb2 * 0.5f * t4;
  const float tb5 = bb3 * (13.f / 6.f) * t5, tb6 = bb3 * 0.5f * t6;
  g[0] = tb1 + tb2 + (2.f / 6.f) * qb1;
  g[1] = -2.f * tb1 - 4.f * tb2 + tb3 + tb4 + (-7.f / 6.f) * qb1 + (-1.f / 6.f) * qb2;
  g[2] = tb1 + 3.f * tb2 - 2.f * tb3 + tb5 + 3.f * tb6 + (11.f / 6.f) * qb1 + (5.f / 6.f) * qb2 + (2.f / 6.f) * qb3;
  g[3] = tb3 - tb4 - 2.f * tb5 - 4.f * tb6 + (2.f / 6.f) * qb2 + (5.f / 6.f) * qb3;
  g[4] = tb5 + tb6 + (-1.f / 6.f) * qb3;
  return W;
}

// W = weno3(a, b, c) and dW/d(a, b, c) into g[0..2].
__device__ __forceinline__ float weno3_grad(float a, float b, float c, float eps, float* g) {
  const float dab = a - b, dbc = b - c;
  const float b1 = dab * dab, b2 = dbc * dbc;
  const float dd = b1 - b2, tau = fabsf(dd), sg = dd >= 0.f ? 1.f : -1.f;
  const float i1 = rcp_approx(b1 + eps), i2 = rcp_approx(b2 + eps);
  const float q1r = tau * i1, q2r = tau * i2;
  const float r1 = fminf(kRatioCap, q1r), r2 = fminf(kRatioCap, q2r);
  const float w1 = (1.f / 3.f) * (1.f + r1 * r1), w2 = (2.f / 3.f) * (1.f + r2 * r2);
  const float q1 = -0.5f * a + 1.5f * b, q2 = 0.5f * b + 0.5f * c;
  const float iS = rcp_approx(w1 + w2);
  const float W = (w1 * q1 + w2 * q2) * iS;
  const float qb1 = w1 * iS, qb2 = w2 * iS;
  const float wb1 = (q1 - W) * iS, wb2 = (q2 - W) * iS;
  const float rb1 = q1r < kRatioCap ? wb1 * (2.f / 3.f) * r1 : 0.f;
  const float rb2 = q2r < kRatioCap ? wb2 * (4.f / 3.f) * r2 : 0.f;
  const float taub = rb1 * i1 + rb2 * i2;
  const float bb1 = -rb1 * r1 * i1 + taub * sg;
  const float bb2 = -rb2 * r2 * i2 - taub * sg;
  g[0] = bb1 * 2.f * dab - 0.5f * qb1;
  g[1] = -bb1 * 2.f * dab + bb2 * 2.f * dbc + 1.5f * qb1 + 0.5f * qb2;
  g[2] = -bb2 * 2.f * dbc + 0.5f * qb2;
  return W;
}

// Lateral face between s[2] and s[3] of s[0..5] (cells p-3 .. p+2): W and dW/ds into g[0..5].
__device__ __forceinline__ float lateral_grad(float m, const float* s, float eps, float* g) {
  float h[5];
  for (int q = 0; q < 6; ++q) g[q] = 0.f;
  if (m >= 0.f) {
    const float W = weno5_grad(s[0], s[1], s[2], s[3], s[4], eps, h);
    for (int q = 0; q < 5; ++q) g[q] = h[q];
    return W;
  }
  const float W = weno5_grad(s[5], s[4], s[3], s[2], s[1], eps, h);
  for (int q = 0; q < 5; ++q) g[5 - q] = h[q];
  return W;
}

// Vertical face H of an n-entry column (between entries H-1 and H), s[0..5] = entries H-3 .. H+2
// (entries outside 0..n-1 are never used); rules of vflux6 in kernels_weno.cu.
__device__ __forceinline__ float vertical_grad(float m, const float* s, int H, int n, float eps, float* g) {
  float h[5];
  for (int q = 0; q < 6; ++q) g[q] = 0.f;
  if (H <= 0 || H >= n) return 0.f;
  const bool up = m >= 0.f;
  if (H >= 3 && H <= n - 3) return lateral_grad(m, s, eps, g);
  if (up) {
    if (H == 1) {
      g[2] = 0.5f;
      g[3] = 0.5f;
      return 0.5f * (s[2] + s[3]);
    }
    if (H == 2 || H == n - 1) {
      const float W = weno3_grad(s[1], s[2], s[3], eps, h);
      g[1] = h[0]; g[2] = h[1]; g[3] = h[2];
      return W;
    }
    const float W = weno5_grad(s[0], s[1], s[2], s[3], s[4], eps, h);  // H == n-2
    for (int q = 0; q < 5; ++q) g[q] = h[q];
    return W;
  }
  if (H == n - 1) {
    g[3] = 0.5f;
    g[2] = 0.5f;
    return 0.5f * (s[3] + s[2]);
  }
  if (H == 1 || H == n - 2) {
    const float W = weno3_grad(s[4], s[3], s[2], eps, h);
    g[4] = h[0]; g[3] = h[1]; g[2] = h[2];
    return W;
  }
  const float W = weno5_grad(s[5], s[4], s[3], s[2], s[1], eps, h);  // H == 2
  for (int q = 0; q < 5; ++q) g[5 - q] = h[q];
  return W;
}

// ---------------------------------------------------------------------------------------------
// acoustic sub-step
// ---------------------------------------------------------------------------------------------
// Values one cell's reverse sub-step reads; neighbour index 0 cell, 1 west, 2 east, 3 south,
// 4 north, 5 below, 6 above.
struct AcNbr {
  float A[7];    // kDivDamp * dtau * adjoint of the output pi'
  float s[7];    // pi'_s
  float p[7];    // input pi'
  float t[7];    // theta_rho
  float unb_w, unb_e, vnb_s, vnb_n, wnb_b, wnb_t;  // adjoints of the output winds on the six faces
  float un_w, un_e, vn_s, vn_n, wn_b, wn_t;        // output winds on the six faces
};
struct AcCol {  // column constants of level k (rho* and their correctly rounded reciprocals *i)
  float pi0m, pi0, pi0p, rhom, rho, rhop, rhomi, rhoi, rhopi, rfb, rft, dzb, dzt;
  bool hb, ht;
};
struct AcOut {
  float ub, vb, wb, pb, tb, sb;
};

__device__ __forceinline__ AcOut acoustic_vjp_cell(const AcNbr& n, const AcCol& k, float pnb0, float rdx, float rdy,
                                                   float rdz, float dtau) {
  const float* A = n.A;
  const float* s = n.s;
  auto divb = [&](int q, float pi0) { return -A[q] * kRdCvA * (pi0 + s[q]); };
  const float D0 = divb(0, k.pi0), DW = divb(1, k.pi0), DE = divb(2, k.pi0), DS = divb(3, k.pi0), DN = divb(4, k.pi0);
  const float DB = k.hb ? divb(5, k.pi0m) : 0.f, DT = k.ht ? divb(6, k.pi0p) : 0.f;
  const float Gw = (s[0] - s[1]) * rdx, Ge = (s[2] - s[0]) * rdx, Gs = (s[0] - s[3]) * rdy, Gn = (s[4] - s[0]) * rdy;
  const float Uw = n.unb_w + (DW - D0) * rdx - 0.5f * Gw * (A[0] + A[1]);
  const float Ue = n.unb_e + (D0 - DE) * rdx - 0.5f * Ge * (A[2] + A[0]);
  const float Vs = n.vnb_s + (DS - D0) * rdy - 0.5f * Gs * (A[0] + A[3]);
  const float Vn = n.vnb_n + (D0 - DN) * rdy - 0.5f * Gn * (A[4] + A[0]);
  float Wb = 0.f, Wt = 0.f;
  if (k.hb) {
    const float Z = k.dzb + (s[0] - s[5]) * rdz;
    Wb = n.wnb_b + (DB - D0) * rdz - 0.5f * Z * k.rfb * (A[0] * k.rhoi + A[5] * k.rhomi);
  }
  if (k.ht) {
    const float Z = k.dzt + (s[6] - s[0]) * rdz;
    Wt = n.wnb_t + (D0 - DT) * rdz - 0.5f * Z * k.rft * (A[6] * k.rhopi + A[0] * k.rhoi);
  }
  AcOut o;
  o.ub = Uw;
  o.vb = Vs;
  o.wb = Wb;
  // pressure-gradient terms of the input pi' and theta_rho
  const float c0 = -kHalfCp * dtau;
  const float* p = n.p;
  const float* t = n.t;
  float pb = pnb0, tb = 0.f;
  pb += Uw * c0 * (t[0] + t[1]) * rdx - Ue * c0 * (t[2] + t[0]) * rdx;
  tb += Uw * c0 * (p[0] - p[1]) * rdx + Ue * c0 * (p[2] - p[0]) * rdx;
  pb += Vs * c0 * (t[0] + t[3]) * rdy - Vn * c0 * (t[4] + t[0]) * rdy;
  tb += Vs * c0 * (p[0] - p[3]) * rdy + Vn * c0 * (p[4] - p[0]) * rdy;
  if (k.hb) {
    pb += Wb * c0 * (t[0] + t[5]) * rdz;
    tb += Wb * c0 * (p[0] - p[5]) * rdz;
  }
  if (k.ht) {
    pb -= Wt * c0 * (t[6] + t[0]) * rdz;
    tb += Wt * c0 * (p[6] - p[0]) * rdz;
  }
  o.pb = pb;
  o.tb = tb;
  // pi'_s: the divergence factor and advection_pi of this cell and its six neighbours
  const float uw = n.un_w, ue = n.un_e, vs = n.vn_s, vn = n.vn_n;
  const float wbn = k.hb ? n.wn_b : 0.f, wtn = k.ht ? n.wn_t : 0.f;
  const float div = (ue - uw) * rdx + (vn - vs) * rdy + (wtn - wbn) * rdz;
  const float dap = -(0.5f * (-ue * rdx + uw * rdx) + 0.5f * (-vn * rdy + vs * rdy) +
                      ((k.hb ? 0.5f * k.rfb * wbn * rdz : 0.f) - (k.ht ? 0.5f * k.rft * wtn * rdz : 0.f)) * k.rhoi);
  float sb = A[0] * (-kRdCvA * div + dap);
  sb += A[2] * 0.5f * ue * rdx - A[1] * 0.5f * uw * rdx;
  sb += A[4] * 0.5f * vn * rdy - A[3] * 0.5f * vs * rdy;
  if (k.ht) sb += A[6] * 0.5f * k.rft * wtn * rdz * k.rhopi;
  if (k.hb) sb -= A[5] * 0.5f * k.rfb * wbn * rdz * k.rhomi;
  o.sb = sb;
  return o;
}

__device__ __forceinline__ AcCol acoustic_col(const Cols& c, int k, int nz) {
  AcCol q;
  q.hb = k > 0;
  q.ht = k + 1 < nz;
  q.pi0 = c.pi0[k];
  q.rho = c.rho[k];
  q.rhoi = c.rho_inv[k];
  q.pi0m = q.hb ? c.pi0[k - 1] : 0.f;
  q.rhom = q.hb ? c.rho[k - 1] : 1.f;
  q.rhomi = q.hb ? c.rho_inv[k - 1] : 1.f;
  q.pi0p = q.ht ? c.pi0[k + 1] : 0.f;
  q.rhop = q.ht ? c.rho[k + 1] : 1.f;
  q.rhopi = q.ht ? c.rho_inv[k + 1] : 1.f;
  q.rfb = c.rho_face[k];
  q.rft = c.rho_face[k + 1];
  q.dzb = c.dpi0dz[k];
  q.dzt = c.dpi0dz[k + 1];
  return q;
}

// V consecutive x cells per thread with V-wide row loads (nx % V == 0), blocks as k_acoustic_vec's.  Ten
// fields read, four written, five accumulated: 96 bytes a cell, 84 on average with the wind accumulators
// updated every other sub-step, from the sub-step's result and from its input, which is the result of the
// one before.  Bound by the memory's latency (162 registers, 12 warps an SM, DRAM at 41 %): 192x192x96
// 66.3 us a sub-step (launch list; 109 when the kernel read the accumulators after the stores, in every
// sub-step and through a persisting window of their own), 68.1 without their lines on the way to L2 from the
// start, 72.6 with the winds' updated in every sub-step.  Slower, by 2 to 4 % of the pass: the accumulators in
// registers from the start (198 of them), two cells a thread and twice the warps; programmatic dependent
// launch gained nothing.
template <int V>
struct VecF;
template <>
struct VecF<4> {
  typedef float4 T;
};
template <>
struct VecF<2> {
  typedef float2 T;
};
template <>
struct VecF<1> {
  typedef float T;
};
template <int V>
__device__ __forceinline__ void ldvec(const float* p, int i, float (&o)[V]) {
  typedef typename VecF<V>::T T;
  const T t = __ldg(reinterpret_cast<const T*>(p + i));
  const float* f = reinterpret_cast<const float*>(&t);
#pragma unroll
  for (int l = 0; l < V; ++l) o[l] = f[l];
}
template <int V>
__device__ __forceinline__ void ldv(const float* p, int i, float (&o)[V]) {
  typedef typename VecF<V>::T T;
  const T t = *reinterpret_cast<const T*>(p + i);
  const float* f = reinterpret_cast<const float*>(&t);
#pragma unroll
  for (int l = 0; l < V; ++l) o[l] = f[l];
}
template <int V>
__device__ __forceinline__ void stvec(float* p, int i, const float (&v)[V]) {
  typedef typename VecF<V>::T T;
  T t;
  float* f = reinterpret_cast<float*>(&t);
#pragma unroll
  for (int l = 0; l < V; ++l) f[l] = v[l];
  *reinterpret_cast<T*>(p + i) = t;
}
__device__ __forceinline__ void prefetch_l2(const float* p) { asm volatile("prefetch.global.L2 [%0];" ::"l"(p)); }

constexpr int VJP_T = 64;   // threads of a block

template <int V>
__global__ void __launch_bounds__(VJP_T) k_acoustic_vjpv(Dims d, Phys ph, Cols c, AcousticVjpArgs a, float dtau, int flat,
                                                      int k0) {
  const int nq = d.nx / V;
  int qx, j;
  if (flat) {
    const int t = blockIdx.x * blockDim.x + threadIdx.x;
    j = t / nq;
    qx = t - j * nq;
  } else {
    qx = blockIdx.x * blockDim.x + threadIdx.x;
    j = blockIdx.y * blockDim.y + threadIdx.y;
  }
  const int k = k0 + blockIdx.z;
  if (j >= d.ny) return;
  const int nx = d.nx, ny = d.ny, nz = d.nz, plane = d.plane();
  const int i0 = V * qx;
  const int r0 = k * plane + j * nx, rs = k * plane + wrapx(j - 1, ny) * nx, rn = k * plane + wrapx(j + 1, ny) * nx;
  const int iw = wrapx(i0 - 1, nx), ie = wrapx(i0 + V, nx);
  const AcCol col = acoustic_col(c, k, nz);
  const int rb = col.hb ? r0 - plane : r0, rt = col.ht ? r0 + plane : r0;
  const float K = kDivDamp * dtau;
  // rows: 0 centre, 1 south, 2 north, 3 below, 4 above
  const int rows[5] = {r0, rs, rn, rb, rt};
  float PN[5][V], PS[5][V], PP[5][V], TT[5][V];
#pragma unroll
  for (int r = 0; r < 5; ++r) {
    ldvec<V>(a.pnb, rows[r] + i0, PN[r]);
    ldvec<V>(a.ps, rows[r] + i0, PS[r]);
    ldvec<V>(a.p, rows[r] + i0, PP[r]);
    ldvec<V>(a.trho, rows[r] + i0, TT[r]);
  }
  const float pnW = LD(a.pnb, r0 + iw), pnE = LD(a.pnb, r0 + ie);
  const float psW = LD(a.ps, r0 + iw), psE = LD(a.ps, r0 + ie);
  const float ppW = LD(a.p, r0 + iw), ppE = LD(a.p, r0 + ie);
  const float ttW = LD(a.trho, r0 + iw), ttE = LD(a.trho, r0 + ie);
  float UNB[V], VNB[V], VNBn[V], WNB[V], WNBt[V], UN[V], VN[V], VNn[V], WN[V], WNt[V];
  ldvec<V>(a.unb, r0 + i0, UNB);
  ldvec<V>(a.vnb, r0 + i0, VNB);
  ldvec<V>(a.vnb, rn + i0, VNBn);
  ldvec<V>(a.wnb, r0 + i0, WNB);
  ldvec<V>(a.wnb, r0 + plane + i0, WNBt);
  ldvec<V>(a.un, r0 + i0, UN);
  ldvec<V>(a.vn, r0 + i0, VN);
  ldvec<V>(a.vn, rn + i0, VNn);
  ldvec<V>(a.wn, r0 + i0, WN);
  ldvec<V>(a.wn, r0 + plane + i0, WNt);
  const float unbE = LD(a.unb, r0 + ie), unE = LD(a.un, r0 + ie);
  // the accumulators on their way from memory while the inputs are: they are read after the results are
  // stored, and without registers for them until then
  if (a.acc) {
    prefetch_l2(a.Rub + r0 + i0);
    prefetch_l2(a.Rvb + r0 + i0);
    prefetch_l2(a.Rwb + r0 + i0);
  }
  prefetch_l2(a.trhob + r0 + i0);
  prefetch_l2(a.psb + r0 + i0);
  float ob[V], vb[V], wb[V], pb[V], tb[V], sb[V];
#pragma unroll
  for (int l = 0; l < V; ++l) {
    AcNbr n;
    // x neighbours inside the vector or the scalar ends
    const float pnw = l == 0 ? pnW : PN[0][l - 1], pne = l == V - 1 ? pnE : PN[0][l + 1];
    const float psw = l == 0 ? psW : PS[0][l - 1], pse = l == V - 1 ? psE : PS[0][l + 1];
    const float ppw = l == 0 ? ppW : PP[0][l - 1], ppe = l == V - 1 ? ppE : PP[0][l + 1];
    const float ttw = l == 0 ? ttW : TT[0][l - 1], tte = l == V - 1 ? ttE : TT[0][l + 1];
    n.A[0] = K * PN[0][l]; n.A[1] = K * pnw; n.A[2] = K * pne;
    n.A[3] = K * PN[1][l]; n.A[4] = K * PN[2][l];
    n.A[5] = col.hb ? K * PN[3][l] : 0.f; n.A[6] = col.ht ? K * PN[4][l] : 0.f;
    n.s[0] = PS[0][l]; n.s[1] = psw; n.s[2] = pse; n.s[3] = PS[1][l]; n.s[4] = PS[2][l];
    n.s[5] = PS[3][l]; n.s[6] = PS[4][l];
    n.p[0] = PP[0][l]; n.p[1] = ppw; n.p[2] = ppe; n.p[3] = PP[1][l]; n.p[4] = PP[2][l];
    n.p[5] = PP[3][l]; n.p[6] = PP[4][l];
    n.t[0] = TT[0][l]; n.t[1] = ttw; n.t[2] = tte; n.t[3] = TT[1][l]; n.t[4] = TT[2][l];
    n.t[5] = TT[3][l]; n.t[6] = TT[4][l];
    n.unb_w = UNB[l]; n.unb_e = l == V - 1 ? unbE : UNB[l + 1];
    n.vnb_s = VNB[l]; n.vnb_n = VNBn[l];
    n.wnb_b = WNB[l]; n.wnb_t = WNBt[l];
    n.un_w = UN[l]; n.un_e = l == V - 1 ? unE : UN[l + 1];
    n.vn_s = VN[l]; n.vn_n = VNn[l];
    n.wn_b = WN[l]; n.wn_t = WNt[l];
    const AcOut o = acoustic_vjp_cell(n, col, PN[0][l], ph.rdx, ph.rdy, ph.rdz, dtau);
    ob[l] = o.ub; vb[l] = o.vb; wb[l] = o.wb; pb[l] = o.pb; tb[l] = o.tb; sb[l] = o.sb;
  }
  stvec<V>(a.ub, r0 + i0, ob);
  stvec<V>(a.vb, r0 + i0, vb);
  stvec<V>(a.wb, r0 + i0, wb);
  stvec<V>(a.pb, r0 + i0, pb);
  if (k == nz - 1) {
    float z[V];
#pragma unroll
    for (int l = 0; l < V; ++l) z[l] = 0.f;
    stvec<V>(a.wb, r0 + plane + i0, z);
  }
  float au[V], av[V], aw[V], at[V], as[V];
  ldv<V>(a.trhob, r0 + i0, at);
  ldv<V>(a.psb, r0 + i0, as);
  if (a.acc) {
    ldv<V>(a.Rub, r0 + i0, au);
    ldv<V>(a.Rvb, r0 + i0, av);
    ldv<V>(a.Rwb, r0 + i0, aw);
#pragma unroll
    for (int l = 0; l < V; ++l) {
      if (a.acc == 2) {
        ob[l] += UNB[l];
        vb[l] += VNB[l];
        wb[l] += WNB[l];
      }
      au[l] += ob[l] * dtau;
      av[l] += vb[l] * dtau;
      if (col.hb) aw[l] += wb[l] * dtau;
    }
    stvec<V>(a.Rub, r0 + i0, au);
    stvec<V>(a.Rvb, r0 + i0, av);
    stvec<V>(a.Rwb, r0 + i0, aw);
  }
#pragma unroll
  for (int l = 0; l < V; ++l) {
    at[l] += tb[l];
    as[l] += sb[l];
  }
  stvec<V>(a.trhob, r0 + i0, at);
  stvec<V>(a.psb, r0 + i0, as);
}

// ---------------------------------------------------------------------------------------------
// pointwise part of a stage's reverse pass (after the acoustic loop):
//   cbar of the five advected fields, the phi*div terms, Coriolis, buoyancy, theta_rho,
//   pi'_s, SGS adjoints and the identity paths to xi0
// ---------------------------------------------------------------------------------------------
// Bound by memory: 40 fields read, 17 written, 230 bytes a cell.  Every read is issued before the first
// store, which the compiler may not move one across, and xsb is written here first, so it is neither cleared
// nor read: 192x192x96 258 -> 146 us.
__global__ void __launch_bounds__(AB) k_stage_pointwise_vjp(Dims d, Phys ph, Cols c, StageVjpArgs a) {
  const unsigned t = blockIdx.x * AB + threadIdx.x;
  const int nx = d.nx, ny = d.ny, nz = d.nz, plane = d.plane();
  if (t >= d.faces()) return;
  const int i = (int)(t % nx), j = (int)((t / nx) % ny), k = (int)(t / plane);
  const int id = (int)t, row = k * plane;
  const bool cell = k < nz, in_w = k >= 1 && cell, up = k + 1 < nz, sgs = a.sgsb_w != nullptr;
  const int ia = up ? id + plane : id;
  const int iw = row + j * nx + wrapx(i - 1, nx), ie = row + j * nx + wrapx(i + 1, nx);
  const int is = row + wrapx(j - 1, ny) * nx + i, in = row + wrapx(j + 1, ny) * nx + i;
  const float Rw = LD(a.Rwb, id), aw = LD(a.acb[2], id), x0w = a.x0b.w[id];
  const float sw = sgs && in_w ? a.sgsb_w[id] : 0.f;
  const float dvm = in_w ? LD(a.div, id - plane) : 0.f, dv = cell ? LD(a.div, id) : 0.f;
  if (!cell) {   // the lid: w = 0 there
    a.cb[2][id] = 0.f;
    a.xsb.w[id] = 0.f;
    a.x0b.w[id] = x0w + aw;
    return;
  }
  const float au = LD(a.acb[0], id), av = LD(a.acb[1], id), ap = LD(a.acb[3], id);
  const float Tb = LD(a.Tnb, id), Qb = LD(a.qnb, id), T = LD(a.xs.T, id), q = LD(a.xs.q, id);
  const float Ru = LD(a.Rub, id), Rue = LD(a.Rub, ie), Rv = LD(a.Rvb, id), Rvn = LD(a.Rvb, in);
  const float Rwt = up ? LD(a.Rwb, ia) : 0.f;
  const float u = LD(a.xs.u, id), ue = LD(a.xs.u, ie), v = LD(a.xs.v, id), vn = LD(a.xs.v, in);
  const float w = LD(a.xs.w, id), wt = LD(a.xs.w, ia);
  const float dvw = LD(a.div, iw), dvs = LD(a.div, is);
  const float trb = LD(a.trhob, id), psb = LD(a.psb, id);
  const float x0u = a.x0b.u[id], x0v = a.x0b.v[id], x0p = a.x0b.p[id], x0T = a.x0b.T[id], x0q = a.x0b.q[id];
  float su = 0.f, sv = 0.f, sT = 0.f, sq = 0.f;
  if (sgs) {
    su = a.sgsb_u[id];
    sv = a.sgsb_v[id];
    sT = a.sgsb_T[id];
    sq = a.sgsb_q[id];
  }
  float Rus = 0.f, Ruse = 0.f, Rvw = 0.f, Rvnw = 0.f;
  if (ph.cor_opt) {
    Rus = LD(a.Rub, is);
    Ruse = LD(a.Rub, row + wrapx(j - 1, ny) * nx + wrapx(i + 1, nx));
    Rvw = LD(a.Rvb, iw);
    Rvnw = LD(a.Rvb, row + wrapx(j + 1, ny) * nx + wrapx(i - 1, nx));
  }
  const float ri = c.rho_inv[k];   // products with the correctly rounded 1 / rho0 instead of divisions
  const float deni = c.rho_w_inv[k], denit = up ? c.rho_w_inv[k + 1] : 0.f;   // 1 / (0.5 (rho0(k-1) + rho0(k)))
  // ---- w point (face k): cbar_w, the w*div term; the acoustic loop starts from the big step's input
  a.cb[2][id] = in_w ? Rw * deni : 0.f;
  a.xsb.w[id] = in_w ? Rw * 0.5f * (dvm + dv) * deni : 0.f;
  a.x0b.w[id] = x0w + aw;
  if (sgs && in_w) a.sgsb_w[id] = sw + Rw;
  a.x0b.u[id] = x0u + au;
  a.x0b.v[id] = x0v + av;
  a.x0b.p[id] = x0p + ap;
  // ---- scalars
  const float cT = a.dts * Tb * ri, cQ = a.dts * Qb * ri;
  a.cb[3][id] = cT;
  a.cb[4][id] = cQ;
  float dvb = cT * T + cQ * q;
  float Tsb = cT * dv, qsb = cQ * dv;
  a.x0b.T[id] = x0T + Tb;
  a.x0b.q[id] = x0q + Qb;
  if (sgs) {
    a.sgsb_T[id] = sT + a.dts * Tb;
    a.sgsb_q[id] = sq + a.dts * Qb;
    a.sgsb_u[id] = su + Ru;
    a.sgsb_v[id] = sv + Rv;
  }
  // ---- u, v points
  a.cb[0][id] = Ru * ri;
  a.cb[1][id] = Rv * ri;
  float ub = Ru * 0.5f * (dvw + dv) * ri;
  float vb = Rv * 0.5f * (dvs + dv) * ri;
  // divergence adjoint of this cell from the phi*div terms of its u, v, w points
  dvb += 0.5f * ri * (Ru * u + Rue * ue);
  dvb += 0.5f * ri * (Rv * v + Rvn * vn);
  if (in_w) dvb += 0.5f * Rw * w * deni;
  if (up) dvb += 0.5f * Rwt * wt * denit;
  // Coriolis: R_u += f v4, R_v -= f u4 (both cor_opt 1 and 2 are linear in the winds)
  if (ph.cor_opt) {
    const float f4 = 0.25f * ph.f_cor;
    vb += f4 * (Ru + Rue + Rus + Ruse);
    ub -= f4 * (Rv + Rvn + Rvw + Rvnw);
  }
  a.xsb.u[id] = ub;
  a.xsb.v[id] = vb;
  a.divb[id] = dvb;
  // buoyancy b(k) enters b8w on faces k and k+1 (the end faces' extrapolations meet a zero R_w
  // adjoint: the acoustic sub-step pins w there)
  {
    const float bb = 0.5f * ((k >= 1 ? Rw : 0.f) + Rwt);
    const float th0 = c.theta0[k], q0 = c.qv0[k], tr0 = c.trho0[k];
    const float reps = (float)kReps;
    const float num = th0 * (float)(kReps - 1.0) * (q - q0) + (T - c.d0[k]) * (1.f + reps * q) * (1.f + q0);
    const float den = (1.f + q) * (1.f + q0);
    const float g = (float)kG / tr0;
    Tsb += bb * g * (1.f + reps * q) * (1.f + q0) / den;
    const float dnum = th0 * (float)(kReps - 1.0) + (T - c.d0[k]) * reps * (1.f + q0);
    qsb += bb * g * (dnum * den - num * (1.f + q0)) / (den * den);
  }
  // theta_rho = (theta_ref + T)(1 + reps q)/(1 + q)
  {
    const float reps = (float)kReps;
    Tsb += trb * (1.f + reps * q) / (1.f + q);
    qsb += trb * (ph.theta_ref + T) * (reps - 1.f) / ((1.f + q) * (1.f + q));
  }
  a.xsb.T[id] = Tsb;
  a.xsb.q[id] = qsb;
  a.xsb.p[id] = psb;
}

// mass divergence: xsb winds += div^T(divb)
// and, with x0b (the first stage, whose input is the big step's input): x0b += xsb, all six fields
__global__ void __launch_bounds__(AB) k_massdiv_vjp(Dims d, Phys ph, Cols c, const float* __restrict__ divb, State xsb,
                                                    State x0b) {
  const unsigned t = blockIdx.x * AB + threadIdx.x;
  const int nx = d.nx, ny = d.ny, nz = d.nz, plane = d.plane();
  if (t >= d.faces()) return;
  const int i = (int)(t % nx), j = (int)((t / nx) % ny), k = (int)(t / plane);
  const int id = (int)t;
  if (k >= 1 && k < nz) xsb.w[id] += c.rho_face0[k] * (LD(divb, id - plane) - LD(divb, id)) * ph.rdz;
  if (x0b.w) x0b.w[id] += xsb.w[id];
  if (k >= nz) return;
  const float r = c.rho[k];
  const int row = k * plane;
  xsb.u[id] += r * (LD(divb, row + j * nx + wrapx(i - 1, nx)) - LD(divb, id)) * ph.rdx;
  xsb.v[id] += r * (LD(divb, row + wrapx(j - 1, ny) * nx + i) - LD(divb, id)) * ph.rdy;
  if (x0b.u) {
    x0b.u[id] += xsb.u[id];
    x0b.v[id] += xsb.v[id];
    x0b.T[id] += xsb.T[id];
    x0b.q[id] += xsb.q[id];
    x0b.p[id] += xsb.p[id];
  }
}

// ---------------------------------------------------------------------------------------------
// WENO advection adjoint, one direction
// ---------------------------------------------------------------------------------------------
// Flux adjoints of a direction, fields 0 u, 1 v, 2 w, 3 theta, 4 qv: the flux between points p-1 and p names the
// six points p-3 .. p+2 in its slots, and each point adds up the slots that name it; the adjoint of a face's
// mass flux goes to mb[f].  No slot is stored: 30 fields a direction written and read back otherwise.

// Direction x: a block takes whole rows (nx <= ROW_T) or a segment of one with the five faces beside it, a
// thread a face, field after field, and the slots meet in shared memory.  Bound by the WENO derivatives'
// arithmetic (about 350 instructions a face): 192x192x96 315 us a stage with the slots in memory and gathered
// by another kernel, now 298; 64x64x64 28.4, now 25.9 (with the mass-flux part).  A field a block: 320.
constexpr int ROW_T = 256;
__global__ void __launch_bounds__(ROW_T) k_adv_row_vjp(Dims d, Phys ph, Cols c, AdvVjpArgs a, int rows) {
  __shared__ float slots[2][6][ROW_T];   // two fields' in turn: one barrier a field
  const int nx = d.nx, ny = d.ny, nz = d.nz, plane = d.plane();
  const int t = threadIdx.x;
  // the thread's face: row r = (k, j), column i; lo: the row's first slot; own: the face, and the point on its
  // right, are the block's to store
  int r, i, lo;
  bool own, live;
  if (rows > 0) {
    r = (int)blockIdx.x * rows + t / nx;
    i = t % nx;
    lo = t - i;
    live = own = t < rows * nx && r < ny * (nz + 1);
  } else {
    const int x0 = (int)blockIdx.y * (ROW_T - 5), np = min(ROW_T - 5, nx - x0);
    r = (int)blockIdx.x;
    i = wrapx(x0 - 2 + t, nx);
    lo = 0;
    live = t < np + 5;
    own = t >= 2 && t < np + 2;
  }
  const int j = r % ny, k = r / ny, row = k * plane + j * nx, id = row + i, im = row + wrapx(i - 1, nx);
  const bool cell = live && k < nz;
  int at[6], from[6];
#pragma unroll
  for (int q = 0; q < 6; ++q) {
    at[q] = row + wrapx(i + q - 3, nx);
    from[q] = rows > 0 ? lo + wrapx(i + 3 - q, nx) : t + 3 - q;   // the flux at point p+3-q names p in its slot q
  }
  const float* const u = a.xs.u;
  const float rk = cell ? c.rho[k] : 0.f, u0 = cell ? LD(u, id) : 0.f;
#pragma unroll 1
  for (int f = 0; f < 5; ++f) {
    float* const out = f == 0 ? a.xsb.u : f == 1 ? a.xsb.v : f == 2 ? a.xsb.w : f == 3 ? a.xsb.T : a.xsb.q;
    const bool mine = own && k < nz + (f == 2);
    const float o = mine ? out[id] : 0.f;
    float sl[6] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
    if (cell && (f != 2 || k >= 1)) {
      float m = rk * u0;
      if (f == 0)
        m = mass_flux(LD(u, im), u0, rk);
      else if (f == 1)
        m = mass_flux(rk, LD(u, k * plane + wrapx(j - 1, ny) * nx + i), rk, u0);
      else if (f == 2)
        m = mass_flux(c.rho[k - 1], LD(u, id - plane), rk, u0);
      const float Fb = (LD(a.cb[f], id) - LD(a.cb[f], im)) * ph.rdx;
      float s[6], g[6];
#pragma unroll
      for (int q = 0; q < 6; ++q) s[q] = LD(a.phi[f], at[q]);
      const float W = lateral_grad(m, s, f < 3 ? kWepsMom : (f == 3 ? kWepsTheta : kWepsQv), g);
#pragma unroll
      for (int q = 0; q < 6; ++q) sl[q] = Fb * m * g[q];
      if (own) a.mb[f][id] = Fb * W;
    }
#pragma unroll
    for (int q = 0; q < 6; ++q) slots[f & 1][q][t] = sl[q];
    __syncthreads();
    if (!mine) continue;
    float acc = 0.f;
#pragma unroll
    for (int q = 0; q < 6; ++q) acc += slots[f & 1][q][from[q]];
    out[id] = o + acc;
  }
}

// Directions y and z (D = 1, 2) of the flux adjoints in one pass: a thread walks a chunk of a column along D
// for one field, with the six points of the stencil and the six adjoints that still receive slots in
// registers: 192x192x96 320 us a direction and stage with the slots in memory, now 245; 64x64x64 29.5, now 28.
// Bound like the rows.  A chunk of n points takes n + 5 faces.
constexpr int MARCH_T = 128;
template <int D>
__global__ void __launch_bounds__(MARCH_T) k_adv_march_vjp(Dims d, Phys ph, Cols c, AdvVjpArgs a, int chunk) {
  const int nx = d.nx, ny = d.ny, nz = d.nz, plane = d.plane();
  const int f = blockIdx.z;
  const unsigned col = blockIdx.x * MARCH_T + threadIdx.x;
  if (col >= (unsigned)(D == 1 ? nx * nz : plane)) return;
  const int i = (int)(col % nx), r = (int)(col / nx);   // r: level (y) or row (z)
  if (D == 1 && f == 2 && r == 0) return;               // w = 0 on the ground
  const int n = D == 1 ? ny : (f == 2 ? nz + 1 : nz), stride = D == 1 ? nx : plane;
  const int base = D == 1 ? r * plane + i : r * nx + i;
  const int p0 = blockIdx.y * chunk, p1 = min(p0 + chunk, n);
  if (p0 >= p1) return;
  const float* const phi = a.phi[f];
  const float* const cb = a.cb[f];
  const float* const wind = D == 1 ? a.xs.v : a.xs.w;
  float* const out = f == 0 ? a.xsb.u : f == 1 ? a.xsb.v : f == 2 ? a.xsb.w : f == 3 ? a.xsb.T : a.xsb.q;
  float* const mb = a.mb[f];
  const float rd = D == 1 ? ph.rdy : ph.rdz, eps = f < 3 ? kWepsMom : (f == 3 ? kWepsTheta : kWepsQv);
  // rows -5 .. ny + 4 of at least four
  auto at = [&](int p) { return base + (D == 1 ? wrapx(wrapx(p, ny), ny) : p) * stride; };
  auto inside = [&](int p) { return D == 1 || (p >= 0 && p < n); };
  // the two winds of a face's mass flux (theta and qv: one)
  const int da = f == 0 ? wrapx(i - 1, nx) - i : D == 2 && f == 1 ? (wrapx(r - 1, ny) - r) * nx : D == 1 && f == 2 ? -plane : 0;
  const int ha = f == D ? 1 : 0;   // the wind's own field: the points on either side of the face
  const float ra = D == 1 ? (f == 2 ? c.rho[r - 1] : c.rho[r]) : 0.f, rb = D == 1 ? c.rho[r] : 0.f;
  // faces p0 - 2 .. p1 + 2 touch the chunk's points
  float s[6], acc[6];
#pragma unroll
  for (int q = 0; q < 6; ++q) {
    acc[q] = 0.f;
    s[q] = q > 0 && inside(p0 - 6 + q) ? LD(phi, at(p0 - 6 + q)) : 0.f;   // points H - 4 .. H + 1 of the first face
  }
  float cbm = inside(p0 - 3) ? LD(cb, at(p0 - 3)) : 0.f;
  float nphi, ncb, nwa, nw, nout;
  auto load = [&](int H) {   // what face H adds to the window
    const bool face = D == 1 || (H >= 1 && H < n);
    nphi = inside(H + 2) ? LD(phi, at(H + 2)) : 0.f;
    ncb = inside(H) ? LD(cb, at(H)) : 0.f;
    nw = face ? LD(wind, at(H)) : 0.f;
    nwa = face && f < 3 ? LD(wind, at(H - ha) + da) : 0.f;
    nout = H - 3 >= p0 ? out[at(H - 3)] : 0.f;
  };
  load(p0 - 2);
#pragma unroll 1
  for (int H = p0 - 2; H <= p1 + 2; ++H) {
#pragma unroll
    for (int q = 0; q < 5; ++q) s[q] = s[q + 1];
    s[5] = nphi;
    const float cbp = ncb, wa = nwa, wp = nw, o = nout;
    if (H < p1 + 2) load(H + 1);
    if (D == 1 || (H >= 1 && H < n)) {
      const float rc = D == 1 ? rb : f == 2 ? c.rho[H - 1] : c.rho_face[H];
      const float m = f == D ? mass_flux(wa, wp, rc) : f > 2 ? rc * wp : mass_flux(D == 1 ? ra : rc, wa, rc, wp);
      const float Fb = (cbp - cbm) * rd;
      float g[6];
      const float W = D == 1 ? lateral_grad(m, s, eps, g) : vertical_grad(m, s, H, n, eps, g);
      const float fm = Fb * m;
#pragma unroll
      for (int q = 0; q < 6; ++q) acc[q] += fm * g[q];
      if (H >= p0 && H < p1) mb[at(H)] = Fb * W;
    }
    cbm = cbp;
    if (H - 3 >= p0) out[at(H - 3)] = o + acc[0];
#pragma unroll
    for (int q = 0; q < 5; ++q) acc[q] = acc[q + 1];
    acc[5] = 0.f;
  }
}

// The mass-flux adjoints of direction D into its wind
template <int D>
__global__ void __launch_bounds__(AB) k_adv_mass_vjp(Dims d, Phys ph, Cols c, AdvVjpArgs a) {
  const unsigned t = blockIdx.x * AB + threadIdx.x;
  const int nx = d.nx, ny = d.ny, nz = d.nz, plane = d.plane();
  if (t >= d.faces()) return;
  const int i = (int)(t % nx), j = (int)((t / nx) % ny), k = (int)(t / plane);
  const int id = (int)t;
  const int ip = wrapx(i + 1, nx), jp = wrapx(j + 1, ny);
  if (D == 0) {
    if (k >= nz) return;
    const float r = c.rho[k];
    const int row = k * plane;
    float ub = r * (LD(a.mb[3], id) + LD(a.mb[4], id));                                                     // theta, qv
    ub += 0.5f * r * (LD(a.mb[0], id) + LD(a.mb[0], row + j * nx + ip));                // u
    ub += 0.5f * r * (LD(a.mb[1], id) + LD(a.mb[1], row + wrapx(j + 1, ny) * nx + i));  // v (corner)
    ub += 0.5f * r * ((k >= 1 ? LD(a.mb[2], id) : 0.f) + (k + 1 < nz ? LD(a.mb[2], id + plane) : 0.f));  // w
    a.xsb.u[id] += ub;
  } else if (D == 1) {
    if (k >= nz) return;
    const float r = c.rho[k];
    const int row = k * plane;
    float vb = r * (LD(a.mb[3], id) + LD(a.mb[4], id));
    vb += 0.5f * r * (LD(a.mb[0], id) + LD(a.mb[0], row + j * nx + ip));
    vb += 0.5f * r * (LD(a.mb[1], id) + LD(a.mb[1], row + jp * nx + i));
    vb += 0.5f * r * ((k >= 1 ? LD(a.mb[2], id) : 0.f) + (k + 1 < nz ? LD(a.mb[2], id + plane) : 0.f));
    a.xsb.v[id] += vb;
  } else {
    const int row = k * plane;
    float wb = 0.f;
    if (k >= 1 && k < nz) {
      const float rf = c.rho_face[k];
      wb += rf * (LD(a.mb[3], id) + LD(a.mb[4], id));
      wb += 0.5f * rf * (LD(a.mb[0], id) + LD(a.mb[0], row + j * nx + ip));
      wb += 0.5f * rf * (LD(a.mb[1], id) + LD(a.mb[1], row + jp * nx + i));
    }
    if (k >= 1) wb += 0.5f * c.rho[k - 1] * LD(a.mb[2], id);
    if (k + 1 <= nz) wb += 0.5f * c.rho[k] * LD(a.mb[2], id + plane);
    a.xsb.w[id] += wb;
  }
}

// ---------------------------------------------------------------------------------------------
// Smagorinsky (turbulence.py:9-111, :298-446) backwards
// ---------------------------------------------------------------------------------------------
// weight of the edge value e13 / e23 on w face f in s13 / s23 of cell level k (without rho):
// corner averages inside, the quadratic end extrapolation in the bottom and top cells
__device__ __forceinline__ float w_edge(int k, int f, int nz) {
  if (k == 0) return f == 1 ? 0.5f * 1.875f : (f == 2 ? 0.5f * -1.25f : (f == 3 ? 0.5f * 0.375f : 0.f));
  if (k == nz - 1) return f == nz - 1 ? 0.5f * 1.875f : (f == nz - 2 ? 0.5f * -1.25f : (f == nz - 3 ? 0.5f * 0.375f : 0.f));
  return (f == k || f == k + 1) ? 0.25f : 0.f;
}
// weight of n2_face(f) in N^2 of cell level k
__device__ __forceinline__ float w_n2(int k, int f, int nz) {
  if (k == 0) return f == 1 ? 1.875f : (f == 2 ? -1.25f : (f == 3 ? 0.375f : 0.f));
  if (k == nz - 1) return f == nz - 1 ? 1.875f : (f == nz - 2 ? -1.25f : (f == nz - 3 ? 0.375f : 0.f));
  return (f == k || f == k + 1) ? 0.5f : 0.f;
}
// the cell levels whose s13 / s23 / N^2 read face f: f-1, f and the two end cells (distinct)
__device__ __forceinline__ int face_cells(int f, int nz, int* ks) {
  int n = 0;
  ks[n++] = f - 1;
  ks[n++] = f;
  if (f - 1 != 0 && f != 0) ks[n++] = 0;
  if (f - 1 != nz - 1 && f != nz - 1) ks[n++] = nz - 1;
  return n;
}

// forward quantities of compute_deformation / compute_nm / compute_k at every cell (as k_smag_a)
__global__ void __launch_bounds__(AB) k_smag_lin(Dims d, Phys ph, Cols c, State s, SmagLin o) {
  using namespace smag;
  const unsigned t = blockIdx.x * AB + threadIdx.x;
  if (t >= d.cells()) return;
  const int nx = d.nx, ny = d.ny, nz = d.nz;
  const int i = (int)(t % nx), j = (int)((t / nx) % ny), k = (int)(t / d.plane());
  const int id = (int)t;
  const float r = c.rho[k], ri = c.rho_inv[k];
  const int ip = wrap(i + 1, nx), jp = wrap(j + 1, ny);
  const float s11 = r * (LD(s.u, d.at(ip, j, k)) - LD(s.u, id)) * ph.rdx;
  const float s22 = r * (LD(s.v, d.at(i, jp, k)) - LD(s.v, id)) * ph.rdy;
  const float s33 = r * (LD(s.w, d.at(i, j, k + 1)) - LD(s.w, id)) * ph.rdz;
  const float s12 = r * (0.25f * (e12(d, ph, s, i, j, k) + e12(d, ph, s, i + 1, j + 1, k) + e12(d, ph, s, i, j + 1, k) +
                                  e12(d, ph, s, i + 1, j, k)));
  float s13 = 0.f, s23 = 0.f, n2 = 0.f;
  // faces with nonzero weight: k, k+1 inside, 1..3 / nz-3..nz-1 in the end cells
  const int f0 = k == 0 ? 1 : (k == nz - 1 ? nz - 3 : k), f1 = k == 0 ? 3 : (k == nz - 1 ? nz - 1 : k + 1);
  for (int f = f0; f <= f1; ++f) {
    const float we = w_edge(k, f, nz), wn = w_n2(k, f, nz);
    if (we != 0.f) {
      s13 += we * (e13(d, ph, s, i, j, f) + e13(d, ph, s, i + 1, j, f));
      s23 += we * (e23(d, ph, s, i, j, f) + e23(d, ph, s, i, j + 1, f));
    }
    if (wn != 0.f) n2 += wn * n2_face(d, ph, s, i, j, f);
  }
  s13 *= r;
  s23 *= r;
  const float s2 = (2.f * (s11 * s11 + s22 * s22 + s33 * s33) + 4.f * (s12 * s12 + s13 * s13 + s23 * s23)) * (ri * ri);
  const float s2n2 = s2 - n2 * kInvPrandtl;
  const float km = s2n2 > 0.f ? ph.smag_l2 * sqrtf(s2n2) : 0.f;
  o.s[0][id] = s11; o.s[1][id] = s22; o.s[2][id] = s33; o.s[3][id] = s12; o.s[4][id] = s13; o.s[5][id] = s23;
  o.km[id] = km;
  o.kS[id] = s2n2 > 0.f ? 0.5f * ph.smag_l2 / sqrtf(s2n2) : 0.f;
}

// adjoint of compute_smag: tau_ij, K_h and the direct theta / qv terms of the scalar diffusion
__global__ void __launch_bounds__(AB) k_smag_tau_vjp(Dims d, Phys ph, Cols c, State s, SmagLin l, SmagVjpArgs a) {
  const unsigned t = blockIdx.x * AB + threadIdx.x;
  if (t >= d.cells()) return;
  const int nx = d.nx, ny = d.ny, nz = d.nz, plane = d.plane();
  const int i = (int)(t % nx), j = (int)((t / nx) % ny), k = (int)(t / plane);
  const int id = (int)t;
  const int im = wrapx(i - 1, nx), ip = wrapx(i + 1, nx), jm = wrapx(j - 1, ny), jp = wrapx(j + 1, ny);
  const float rdx = ph.rdx, rdy = ph.rdy, rdz = ph.rdz;
  const float r = c.rho[k], ri = c.rho_inv[k];   // ri: the correctly rounded 1 / rho0, multiplied instead of divided
  auto at = [&](int ii, int jj, int kk) { return (kk * ny + jj) * nx + ii; };
  const float* U = a.gu;
  const float* V = a.gv;
  const float* W = a.gw;
  // tau11, tau22, tau33
  a.tb[0][id] = (LD(U, at(ip, j, k)) - LD(U, id)) * rdx * ri;
  a.tb[1][id] = (LD(V, at(i, jp, k)) - LD(V, id)) * rdy * ri;
  float t33 = 0.f;
  if (k >= 1) t33 -= LD(W, id) * rdz * c.rho_wext_inv[k];
  if (k + 1 <= nz - 1) t33 += LD(W, id + plane) * rdz * c.rho_wext_inv[k + 1];
  a.tb[2][id] = t33;
  // tau12 through d12v (sgs_u) and d12u (sgs_v)
  {
    auto d12v = [&](int cc, int jf) {  // adjoint of (t12(cc,jf) - t12(cc,jf-1)) rdy
      const int c1 = wrapx(cc + 1, nx), c0 = wrapx(cc, nx), j0 = wrapx(jf, ny), j1 = wrapx(jf - 1, ny);
      return -0.25f * ri * (LD(U, at(c1, j0, k)) + LD(U, at(c0, j1, k)) + LD(U, at(c1, j1, k)) + LD(U, at(c0, j0, k)));
    };
    auto d12u = [&](int q, int rr) {  // adjoint of (t12(q,rr) - t12(q-1,rr)) rdx
      const int q0 = wrapx(q, nx), q1 = wrapx(q - 1, nx), r0 = wrapx(rr, ny), r1 = wrapx(rr + 1, ny);
      return -0.25f * ri * (LD(V, at(q0, r1, k)) + LD(V, at(q1, r0, k)) + LD(V, at(q0, r0, k)) + LD(V, at(q1, r1, k)));
    };
    a.tb[3][id] = rdy * (d12v(i, j) - d12v(i, j + 1)) + rdx * (d12u(i, j) - d12u(i + 1, j));
  }
  // tau13, tau23: sgs_w (centred lateral differences averaged to faces) and sgs_u / sgs_v
  {
    float t13 = 0.f, t23 = 0.f;
    for (int kf = k; kf <= k + 1; ++kf) {
      if (kf < 1 || kf > nz - 1) continue;
      const float cw = -0.5f * c.rho_wext_inv[kf];
      t13 += cw * (LD(W, at(im, j, kf)) - LD(W, at(ip, j, kf))) / (2.f * ph.dx);
      t23 += cw * (LD(W, at(i, jm, kf)) - LD(W, at(i, jp, kf))) / (2.f * ph.dy);
      // d13s(cc, k') = (to_w0(t13(cc), k'+1) - to_w0(t13(cc), k')) rdz enters sgs_u(cc), sgs_u(cc+1)
      auto d13s = [&](int kk) { return -0.5f * c.rho_inv[kk] * (LD(U, at(ip, j, kk)) + LD(U, at(i, j, kk))); };
      auto d23s = [&](int kk) { return -0.5f * c.rho_inv[kk] * (LD(V, at(i, jp, kk)) + LD(V, at(i, j, kk))); };
      t13 += 0.5f * rdz * (d13s(kf - 1) - d13s(kf));
      t23 += 0.5f * rdz * (d23s(kf - 1) - d23s(kf));
    }
    a.tb[4][id] = t13;
    a.tb[5][id] = t23;
  }
  // scalar diffusion of theta and qv: direct terms and K_h
  {
    const float khc = LD(l.km, id) * kInvPrandtl;
    auto kh = [&](int q) { return LD(l.km, q) * kInvPrandtl; };
    const int nb[4] = {at(im, j, k), at(ip, j, k), at(i, jm, k), at(i, jp, k)};
    float khb = 0.f;
    for (int fld = 0; fld < 2; ++fld) {
      const float* A = fld == 0 ? s.T : s.q;
      const float* G = fld == 0 ? a.gT : a.gq;
      const float a0 = LD(A, id), g0 = LD(G, id);
      float ab = 0.f;
      // x faces i (west) and i+1 (east), y faces j and j+1
      {
        const float fw = (g0 - LD(G, nb[0])) * rdx * ri, fe = (LD(G, nb[1]) - g0) * rdx * ri;
        const float k8w = 0.5f * (khc + kh(nb[0])), k8e = 0.5f * (kh(nb[1]) + khc);
        ab += -r * rdx * (fw * k8w - fe * k8e);
        khb += 0.5f * (fw * (-r * (a0 - LD(A, nb[0])) * rdx) + fe * (-r * (LD(A, nb[1]) - a0) * rdx));
        const float fs = (g0 - LD(G, nb[2])) * rdy * ri, fn = (LD(G, nb[3]) - g0) * rdy * ri;
        const float k8s = 0.5f * (khc + kh(nb[2])), k8n = 0.5f * (kh(nb[3]) + khc);
        ab += -r * rdy * (fs * k8s - fn * k8n);
        khb += 0.5f * (fs * (-r * (a0 - LD(A, nb[2])) * rdy) + fn * (-r * (LD(A, nb[3]) - a0) * rdy));
      }
      if (k >= 1) {  // bottom face k
        const float fb = g0 * rdz * ri - LD(G, id - plane) * rdz * c.rho_inv[k - 1];
        const float k8 = 0.5f * (kh(id - plane) + khc);
        ab += -c.rho_wext[k] * k8 * rdz * fb;
        khb += 0.5f * fb * (-c.rho_wext[k] * (a0 - LD(A, id - plane)) * rdz);
      }
      if (k + 1 <= nz - 1) {  // top face k+1
        const float ft = LD(G, id + plane) * rdz * c.rho_inv[k + 1] - g0 * rdz * ri;
        const float k8 = 0.5f * (khc + kh(id + plane));
        ab += c.rho_wext[k + 1] * k8 * rdz * ft;
        khb += 0.5f * ft * (-c.rho_wext[k + 1] * (LD(A, id + plane) - a0) * rdz);
      }
      (fld == 0 ? a.x0b.T : a.x0b.q)[id] += ab;
    }
    a.khb[id] = khb;
  }
}

// adjoint of compute_k and of the S^2 / N^2 combination: sbar_ij and N^2 bar at every cell
__global__ void __launch_bounds__(AB) k_smag_s_vjp(Dims d, Cols c, SmagLin l, SmagVjpArgs a) {
  const unsigned t = blockIdx.x * AB + threadIdx.x;
  if (t >= d.cells()) return;
  const int id = (int)t, k = (int)(t / d.plane());
  const float ri = c.rho_inv[k], km = LD(l.km, id);
  float s[6], tb[6];
  float kmb = LD(a.khb, id) * kInvPrandtl;
  for (int q = 0; q < 6; ++q) {
    s[q] = LD(l.s[q], id);
    tb[q] = LD(a.tb[q], id);
    kmb += -2.f * s[q] * tb[q];
  }
  if (a.kmkb) a.kmkb[id] = kmb * km;
  const float S2b = kmb * LD(l.kS, id);
  for (int q = 0; q < 6; ++q) a.sb[q][id] = -2.f * km * tb[q] + S2b * (q < 3 ? 4.f : 8.f) * s[q] * (ri * ri);
  a.n2b[id] = -S2b * kInvPrandtl;
}

// adjoint of compute_deformation and compute_nm: winds and theta / qv
__global__ void __launch_bounds__(AB) k_smag_state_vjp(Dims d, Phys ph, Cols c, State s, SmagVjpArgs a) {
  const unsigned t = blockIdx.x * AB + threadIdx.x;
  if (t >= d.faces()) return;
  const int nx = d.nx, ny = d.ny, nz = d.nz, plane = d.plane();
  const int i = (int)(t % nx), j = (int)((t / nx) % ny), k = (int)(t / plane);
  const int id = (int)t;
  const float rdx = ph.rdx, rdy = ph.rdy, rdz = ph.rdz;
  auto at = [&](int ii, int jj, int kk) { return (kk * ny + wrapx(jj, ny)) * nx + wrapx(ii, nx); };
  // adjoint of e12 at (u point q, v face jf), level kk
  auto e12b = [&](int q, int jf, int kk) {
    const float* S = a.sb[3];
    return 0.25f * c.rho[kk] * (LD(S, at(q, jf, kk)) + LD(S, at(q - 1, jf - 1, kk)) + LD(S, at(q, jf - 1, kk)) +
                                LD(S, at(q - 1, jf, kk)));
  };
  // adjoint of e13 at (u point q, row jj, w face f) / e23 at (column ii, v face jf, w face f)
  auto e13b = [&](int q, int jj, int f) {
    if (f < 1 || f > nz - 1) return 0.f;
    int ks[4];
    const int n = face_cells(f, nz, ks);
    float acc = 0.f;
    for (int m = 0; m < n; ++m) {
      const int kk = ks[m];
      if (kk < 0 || kk > nz - 1) continue;
      const float w = w_edge(kk, f, nz);
      if (w != 0.f) acc += w * c.rho[kk] * (LD(a.sb[4], at(q - 1, jj, kk)) + LD(a.sb[4], at(q, jj, kk)));
    }
    return acc;
  };
  auto e23b = [&](int ii, int jf, int f) {
    if (f < 1 || f > nz - 1) return 0.f;
    int ks[4];
    const int n = face_cells(f, nz, ks);
    float acc = 0.f;
    for (int m = 0; m < n; ++m) {
      const int kk = ks[m];
      if (kk < 0 || kk > nz - 1) continue;
      const float w = w_edge(kk, f, nz);
      if (w != 0.f) acc += w * c.rho[kk] * (LD(a.sb[5], at(ii, jf - 1, kk)) + LD(a.sb[5], at(ii, jf, kk)));
    }
    return acc;
  };
  // ---- w on face k
  {
    float wb = 0.f;
    if (k >= 1) wb += c.rho[k - 1] * rdz * LD(a.sb[2], id - plane);
    if (k <= nz - 1) wb -= c.rho[k] * rdz * LD(a.sb[2], id);
    wb += 0.5f * rdx * (e13b(i, j, k) - e13b(i + 1, j, k));
    wb += 0.5f * rdy * (e23b(i, j, k) - e23b(i, j + 1, k));
    a.x0b.w[id] += wb;
  }
  if (k >= nz) return;
  const float r = c.rho[k];
  // ---- u (west face of cell i)
  {
    float ub = r * rdx * (LD(a.sb[0], at(i - 1, j, k)) - LD(a.sb[0], id));
    ub += 0.5f * rdy * (e12b(i, j, k) - e12b(i, j + 1, k));
    ub += 0.5f * rdz * (e13b(i, j, k) - e13b(i, j, k + 1));
    a.x0b.u[id] += ub;
  }
  // ---- v (south face of cell j)
  {
    float vb = r * rdy * (LD(a.sb[1], at(i, j - 1, k)) - LD(a.sb[1], id));
    vb += 0.5f * rdx * (e12b(i, j, k) - e12b(i + 1, j, k));
    vb += 0.5f * rdz * (e23b(i, j, k) - e23b(i, j, k + 1));
    a.x0b.v[id] += vb;
  }
  // ---- theta, qv through N^2 = g/dz log(theta_rho_m(f) / theta_rho_m(f-1)) on faces k, k+1
  {
    auto n2fb = [&](int f) {
      if (f < 1 || f > nz - 1) return 0.f;
      int ks[4];
      const int n = face_cells(f, nz, ks);
      float acc = 0.f;
      for (int m = 0; m < n; ++m) {
        const int kk = ks[m];
        if (kk < 0 || kk > nz - 1) continue;
        const float w = w_n2(kk, f, nz);
        if (w != 0.f) acc += w * LD(a.n2b, at(i, j, kk));
      }
      return acc;
    };
    const float T = LD(s.T, id), q = LD(s.q, id);
    const float r1 = (float)kRepsm1;
    const float trm = (ph.theta_ref + T) * (1.f + r1 * q);
    const float trmb = (float)kG * rdz * (n2fb(k) - n2fb(k + 1)) / trm;
    a.x0b.T[id] += trmb * (1.f + r1 * q);
    a.x0b.q[id] += trmb * (ph.theta_ref + T) * r1;
  }
}

}  // namespace

template <int V>
static cudaError_t launch_vjpv(const Dims& d, const Phys& ph, const Cols& c, const AcousticVjpArgs& a, float dtau,
                               cudaStream_t st) {
  // blocks as the forward sub-step's
  const int nq = d.nx / V;
  constexpr int kMaxGrid = 65535;
  constexpr int BXT = V == 1 ? 32 : 16;
  const bool flat = nq % BXT != 0 || d.ny / (VJP_T / BXT) >= kMaxGrid / 2;
  const dim3 b = flat ? dim3(VJP_T) : dim3(BXT, VJP_T / BXT);
  dim3 g = flat ? dim3((nq * d.ny + VJP_T - 1) / VJP_T) : dim3(nq / BXT, (d.ny + b.y - 1) / b.y);
  for (int k0 = 0; k0 < d.nz; k0 += kMaxGrid) {   // one launch, but for grids of more than 65535 levels
    g.z = d.nz - k0 < kMaxGrid ? d.nz - k0 : kMaxGrid;
    k_acoustic_vjpv<V><<<g, b, 0, st>>>(d, ph, c, a, dtau, (int)flat, k0);
  }
  return cudaGetLastError();
}

cudaError_t launch_acoustic_vjp(const Dims& d, const Phys& ph, const Cols& c, const AcousticVjpArgs& a, float dtau,
                                cudaStream_t st) {
  if (d.nx % 4 == 0) return launch_vjpv<4>(d, ph, c, a, dtau, st);
  if (d.nx % 2 == 0) return launch_vjpv<2>(d, ph, c, a, dtau, st);
  return launch_vjpv<1>(d, ph, c, a, dtau, st);
}

cudaError_t launch_stage_pointwise_vjp(const Dims& d, const Phys& ph, const Cols& c, const StageVjpArgs& a,
                                       cudaStream_t st) {
  const unsigned g = (unsigned)((d.faces() + AB - 1) / AB);
  k_stage_pointwise_vjp<<<g, AB, 0, st>>>(d, ph, c, a);
  return cudaGetLastError();
}

cudaError_t launch_massdiv_vjp(const Dims& d, const Phys& ph, const Cols& c, const float* divb, State xsb,
                               cudaStream_t st, State x0b) {
  const unsigned g = (unsigned)((d.faces() + AB - 1) / AB);
  k_massdiv_vjp<<<g, AB, 0, st>>>(d, ph, c, divb, xsb, x0b);
  return cudaGetLastError();
}

// out += scale * sum(x): per-thread FP64 partial sums, a block reduction, one atomic a block
__global__ void __launch_bounds__(256) k_sum_scaled(long long n, const float* __restrict__ x, double scale,
                                                    double* __restrict__ out) {
  __shared__ double part[8];
  double acc = 0.0;
  for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x)
    acc += (double)x[i];
  for (int o = 16; o > 0; o >>= 1) acc += __shfl_down_sync(0xffffffffu, acc, o);
  if ((threadIdx.x & 31) == 0) part[threadIdx.x >> 5] = acc;
  __syncthreads();
  if (threadIdx.x == 0) {
    double s = 0.0;
    for (int wv = 0; wv < 8; ++wv) s += part[wv];
    atomicAdd(out, scale * s);
  }
}

cudaError_t launch_sum_scaled(long long n, const float* x, double scale, double* out, cudaStream_t st) {
  if (n <= 0) return cudaSuccess;
  long long b = (n + 255) / 256;
  if (b > 1024) b = 1024;
  k_sum_scaled<<<(unsigned)b, 256, 0, st>>>(n, x, scale, out);
  return cudaGetLastError();
}

cudaError_t launch_smag_vjp(const Dims& d, const Phys& ph, const Cols& c, State x0, const SmagLin& l,
                            const SmagVjpArgs& a, cudaStream_t st) {
  const unsigned gc = (unsigned)((d.cells() + AB - 1) / AB), gf = (unsigned)((d.faces() + AB - 1) / AB);
  k_smag_lin<<<gc, AB, 0, st>>>(d, ph, c, x0, l);
  k_smag_tau_vjp<<<gc, AB, 0, st>>>(d, ph, c, x0, l, a);
  k_smag_s_vjp<<<gc, AB, 0, st>>>(d, c, l, a);
  k_smag_state_vjp<<<gf, AB, 0, st>>>(d, ph, c, x0, a);
  return cudaGetLastError();
}

// Chunks of a column: ten blocks an SM, and at least 16 points, of which a chunk takes 21 faces (64x64x64, two
// steps and their reverse pass, 1, 2, 4, 8 chunks: 3.20, 3.05, 3.03, 3.08 ms; 192x192x96, one step, 1, 2, 3, 8:
// 9.54, 9.44, 9.44, 9.60)
template <int D>
static cudaError_t launch_march(const Dims& d, const Phys& ph, const Cols& c, const AdvVjpArgs& a, cudaStream_t st) {
  int dev = 0, sms = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e == cudaSuccess) e = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  if (e != cudaSuccess) return e;
  const int n = D == 1 ? d.ny : d.nz + 1;
  const long long cols = ((long long)(D == 1 ? d.nx * d.nz : d.plane()) + MARCH_T - 1) / MARCH_T;
  const long long want = (10LL * sms + 5 * cols - 1) / (5 * cols), most = n / 16 > 1 ? n / 16 : 1;
  const int chunk = (int)((n + (want < most ? want : most) - 1) / (want < most ? want : most));
  const unsigned count = (unsigned)((n + chunk - 1) / chunk);
  k_adv_march_vjp<D><<<dim3((unsigned)cols, count, 5), MARCH_T, 0, st>>>(d, ph, c, a, chunk);
  return cudaGetLastError();
}

// whole rows, as many as ROW_T threads take, or segments of long ones
static cudaError_t launch_rows(const Dims& d, const Phys& ph, const Cols& c, const AdvVjpArgs& a, cudaStream_t st) {
  const int rows = d.nx <= ROW_T ? ROW_T / d.nx : 0;
  const long long all = (long long)d.ny * (d.nz + 1);
  const dim3 g((unsigned)(rows ? (all + rows - 1) / rows : all), rows ? 1 : (d.nx + ROW_T - 6) / (ROW_T - 5));
  const int threads = rows ? (rows * d.nx + 31) / 32 * 32 : ROW_T;
  k_adv_row_vjp<<<g, threads, 0, st>>>(d, ph, c, a, rows);
  return cudaGetLastError();
}

cudaError_t launch_adv_vjp(const Dims& d, const Phys& ph, const Cols& c, const AdvVjpArgs& a, cudaStream_t st) {
  const unsigned g = (unsigned)((d.faces() + AB - 1) / AB);
  cudaError_t e = launch_rows(d, ph, c, a, st);
  if (e != cudaSuccess) return e;
  k_adv_mass_vjp<0><<<g, AB, 0, st>>>(d, ph, c, a);
  if ((e = launch_march<1>(d, ph, c, a, st)) != cudaSuccess) return e;
  k_adv_mass_vjp<1><<<g, AB, 0, st>>>(d, ph, c, a);
  if ((e = launch_march<2>(d, ph, c, a, st)) != cudaSuccess) return e;
  k_adv_mass_vjp<2><<<g, AB, 0, st>>>(d, ph, c, a);
  return cudaGetLastError();
}

}  // namespace lexgb

namespace lexgb {
namespace {
__global__ void k_axpy(float* __restrict__ y, const float* __restrict__ x, size_t n) {
  for (size_t t = (size_t)blockIdx.x * blockDim.x + threadIdx.x; t < n; t += (size_t)gridDim.x * blockDim.x)
    y[t] += x[t];
}
}  // namespace

cudaError_t launch_axpy(float* y, const float* x, size_t n, cudaStream_t st) {
  const unsigned g = (unsigned)((n + 255) / 256 < 8192 ? (n + 255) / 256 : 8192);
  k_axpy<<<g > 0 ? g : 1, 256, 0, st>>>(y, x, n);
  return cudaGetLastError();
}
}  // namespace lexgb

namespace lexgb {
namespace {
__global__ void k_shift(float* __restrict__ y, float c, size_t n) {
  for (size_t t = (size_t)blockIdx.x * blockDim.x + threadIdx.x; t < n; t += (size_t)gridDim.x * blockDim.x)
    y[t] += c;
}
}  // namespace

cudaError_t launch_shift(float* y, float c, size_t n, cudaStream_t st) {
  const unsigned g = (unsigned)((n + 255) / 256 < 8192 ? (n + 255) / 256 : 8192);
  k_shift<<<g > 0 ? g : 1, 256, 0, st>>>(y, c, n);
  return cudaGetLastError();
}
}  // namespace lexgb
