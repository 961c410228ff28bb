// kernels_cnn.cu - the learned SGS correction's 3-D CNN (simpleCNN, dl_models.py:19-30):
// four 3x3x3 convolutions (5 -> 32 -> 32 -> 32 -> 5 channels, zero padding, tanh-GELU between).
//
// Activations are stored channels-innermost, [z][y][x][C] in BF16, with C padded to a multiple of
// 16 for a convolution's input (the k16 of the MMA) and of 8 for its output (the n8).  Weights
// are [27 offsets][Cout][Cin] BF16 (Cin innermost), offset (dz+1)*9 + (dy+1)*3 + (dx+1).
//
//   k_conv3d       implicit GEMM on the BF16 tensor cores (mma.sync m16n8k16, FP32 accumulation):
//                  a warp owns 16 consecutive x points and every output channel; for each of the
//                  27 offsets and 16-channel slice it loads the shifted input rows as the A
//                  fragment and the weights as B.  Epilogue: + bias, optional FP32 pre-activation,
//                  optional GELU, BF16 and/or FP32 output.  The input gradient of a convolution is
//                  the same kernel run with the offsets mirrored and Cin/Cout swapped.
//   k_gelu_bwd     g = dy * GELU'(pre), to BF16 with the channel padding of the next backward conv
//   k_conv3d_dw    weight gradient dW[o][co][ci] = sum_p g[p][co] x[p+o][ci], FP32 on the CUDA
//                  cores (a small reduction: 27 * Cout * Cin outputs); each block reduces a slab of
//                  points for one offset and adds its partial sums atomically
//   k_bias_grad    db[co] = sum_p g[p][co]
//   k_adam         Adam update of FP32 master weights and their BF16 copies
//   k_sgs_pack     the network's input from the device-layout state (dl_models.py:125-155)
//   k_sgs_unpack   the re-staggered, scaled correction added to the state
//                  (dl_models.py:158-182, one_sprint_functions.py:136-151)
#include <cuda_bf16.h>
#include <stdint.h>

#include <type_traits>

#include "lexgb_cnn.cuh"

namespace lexgb {

namespace {

__device__ __forceinline__ float gelu_tanh(float x) {
  const float k0 = 0.7978845608028654f;  // sqrt(2/pi)
  return 0.5f * x * (1.f + tanhf(k0 * (x + 0.044715f * x * x * x)));
}
// forward GELU with the hardware tanh (tanh.approx.f32, relative error about 2^-11, below the
// BF16 precision the activations are stored in)
__device__ __forceinline__ float tanh_fast(float x) {
  float y;
  asm("tanh.approx.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}
__device__ __forceinline__ float gelu_tanh_fast(float x) {
  const float k0 = 0.7978845608028654f;  // sqrt(2/pi)
  return 0.5f * x * (1.f + tanh_fast(k0 * (x + 0.044715f * x * x * x)));
}
__device__ __forceinline__ void mma_bf16(float (&d)[4], const uint32_t (&a)[4], const uint32_t (&b)[2]) {
  asm volatile(
      "mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, "
      "{%0,%1,%2,%3};"
      : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
      : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b[0]), "r"(b[1]));
}

__device__ __forceinline__ uint32_t ld32(const __nv_bfloat16* p) { return *reinterpret_cast<const uint32_t*>(p); }

// NT: output-channel tiles of 8 (Cout = 8 * NT).  One warp: 16 points x Cout.
template <int NT>
__global__ void __launch_bounds__(128) k_conv3d(int nx, int ny, int nz, int cin, const __nv_bfloat16* __restrict__ x,
                                                const __nv_bfloat16* __restrict__ w, const float* __restrict__ bias,
                                                float* __restrict__ pre, __nv_bfloat16* __restrict__ ybf,
                                                float* __restrict__ yf, int gelu, int creal) {
  constexpr int COUT = 8 * NT;
  const int lane = threadIdx.x & 31;
  const long long warp = ((long long)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const int rows_x = nx / 16;
  const long long ntiles = (long long)rows_x * ny * nz;
  if (warp >= ntiles) return;
  const int tx = (int)(warp % rows_x), y = (int)((warp / rows_x) % ny), z = (int)(warp / ((long long)rows_x * ny));
  const int x0 = tx * 16;
  const int g = lane >> 2, t = lane & 3;
  float acc[NT][4];
#pragma unroll
  for (int n = 0; n < NT; ++n)
#pragma unroll
    for (int q = 0; q < 4; ++q) acc[n][q] = 0.f;
  for (int off = 0; off < 27; ++off) {
    const int dz = off / 9 - 1, dy = (off / 3) % 3 - 1, dx = off % 3 - 1;
    const int zz = z + dz, yy = y + dy;
    if (zz < 0 || zz >= nz || yy < 0 || yy >= ny) continue;  // zero padding: the whole slice is 0
    const int xa = x0 + g + dx, xb = x0 + g + 8 + dx;
    const bool va = xa >= 0 && xa < nx, vb = xb >= 0 && xb < nx;
    const long long rowbase = ((long long)zz * ny + yy) * nx;
    const __nv_bfloat16* pa = x + (rowbase + (va ? xa : 0)) * cin;
    const __nv_bfloat16* pb = x + (rowbase + (vb ? xb : 0)) * cin;
    const __nv_bfloat16* wo = w + (long long)off * COUT * cin;
    for (int kc = 0; kc < cin; kc += 16) {
      uint32_t a[4];
      a[0] = va ? ld32(pa + kc + 2 * t) : 0u;
      a[1] = vb ? ld32(pb + kc + 2 * t) : 0u;
      a[2] = va ? ld32(pa + kc + 2 * t + 8) : 0u;
      a[3] = vb ? ld32(pb + kc + 2 * t + 8) : 0u;
#pragma unroll
      for (int n = 0; n < NT; ++n) {
        const __nv_bfloat16* pw = wo + (long long)(n * 8 + g) * cin + kc + 2 * t;
        uint32_t b[2] = {ld32(pw), ld32(pw + 8)};
        mma_bf16(acc[n], a, b);
      }
    }
  }
  // epilogue: rows g and g+8, channels n*8 + 2t, 2t+1
  const long long p0 = (((long long)z * ny + y) * nx + x0 + g), p1 = p0 + 8;
#pragma unroll
  for (int n = 0; n < NT; ++n) {
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      const int co = n * 8 + 2 * t + (q & 1);
      const long long p = q < 2 ? p0 : p1;
      float v = acc[n][q] + (bias ? bias[co] : 0.f);
      if (pre) pre[p * COUT + co] = v;
      if (gelu) v = gelu_tanh(v);
      if (co >= creal) v = 0.f;  // padding channels stay zero
      if (ybf) ybf[p * COUT + co] = __float2bfloat16(v);
      if (yf) yf[p * COUT + co] = v;
    }
  }
}

__device__ __forceinline__ void ldsm_x4(uint32_t (&r)[4], const __nv_bfloat16* p) {
  const unsigned a = (unsigned)__cvta_generic_to_shared(p);
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0,%1,%2,%3}, [%4];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3])
               : "r"(a));
}
__device__ __forceinline__ void ldsm_x2(uint32_t (&r)[2], const __nv_bfloat16* p) {
  const unsigned a = (unsigned)__cvta_generic_to_shared(p);
  asm volatile("ldmatrix.sync.aligned.m8n8.x2.shared.b16 {%0,%1}, [%2];" : "=r"(r[0]), "=r"(r[1]) : "r"(a));
}

// programmatic dependent launch: let the next kernel of the stream start its prologue / wait
// until the previous kernel has completed and its writes are visible (both no-ops for kernels
// launched without the programmatic-serialisation attribute)
__device__ __forceinline__ void pdl_launch_dependents() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }
__device__ __forceinline__ void pdl_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }

// 16-byte asynchronous copy global -> shared; valid = false writes zeros (no bytes read)
__device__ __forceinline__ void cp_async16(void* smem, const void* gmem, bool valid) {
  const unsigned sa = (unsigned)__cvta_generic_to_shared(smem);
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(sa), "l"(gmem), "r"(valid ? 16 : 0));
}
__device__ __forceinline__ void cp_async_wait_all() { asm volatile("cp.async.wait_all;" ::: "memory"); }

// Shared-memory convolution (CIN 16 or 32, COUT 8, 16 or 32): a persistent block of 12 warps
// stages the layer's weights once ([27][COUT][CIN + 8]: the 8 padding channels put the 16-byte
// rows of an 8x8 matrix in distinct banks), then loops over tiles of 16 x 8 x 1 points (x, y, z),
// staging each tile's input with its halo ([3][10][18][CIN + 8], zero outside the grid) by
// cp.async.  Warp (d, r) takes the 9 offsets of the input plane z + d - 1 for rows y0 + r and
// y0 + r + 4, 16 points each, and every output channel (one A fragment feeds COUT / 8 MMAs, one
// B fragment two); fragments are read with ldmatrix.  The three planes' partial sums meet in
// shared memory and are added in plane order.
constexpr int CONV_RP = 4, CONV_MR = 2, CONV_TY = CONV_RP * CONV_MR, CONV_WARPS = 3 * CONV_RP;

template <int CIN, int COUT>
struct ConvSmem {
  static constexpr int CP = CIN + 8;
  static constexpr int NT = COUT / 8;
  static constexpr int THREADS = 32 * CONV_WARPS;
  static constexpr int W_ELEMS = 27 * COUT * CP;
  static constexpr int A_BYTES = 3 * (CONV_TY + 2) * 18 * CP * 2;
  static constexpr int PS = COUT + 4;                          // partial-sum row stride (floats)
  static constexpr int P_BYTES = CONV_TY * 16 * PS * 4;         // [128 points][PS]
  // buffers of partial sums: one a plane where two blocks still share an SM, else for planes 0 and 1
  static constexpr int NB = (size_t)W_ELEMS * 2 + 3 * P_BYTES <= 112 * 1024 ? 3 : 2;
  static constexpr size_t BYTES = (size_t)W_ELEMS * 2 + (A_BYTES > NB * P_BYTES ? A_BYTES : NB * P_BYTES);
};

// The weights, [27 COUT][CIN + 8], by the block: 16-byte pieces in the order of both memories, each block
// from another part of them on, as all blocks read the same ones (a correction at 32^3: 0.9 us)
template <int CIN, int COUT, int THREADS>
__device__ __forceinline__ void stage_taps(__nv_bfloat16* ws, const __nv_bfloat16* w) {
  constexpr int CH = CIN / 8, RT = THREADS / CH, N = 27 * COUT;
  constexpr int NI = (N + RT - 1) / RT;
  const int row = (int)(threadIdx.x / CH), c = (int)(threadIdx.x % CH);
  __nv_bfloat16* const d = ws + row * (CIN + 8) + c * 8;
  const __nv_bfloat16* const g = w + row * CIN + c * 8;
  int k = (int)(blockIdx.x % NI);
#pragma unroll
  for (int i = 0; i < NI; ++i) {
    if (row + k * RT < N) cp_async16(d + k * RT * (CIN + 8), g + k * RT * CIN, true);
    if (++k == NI) k = 0;
  }
}

// One input plane of a tile with its halo, [CONV_TY + 2][18][CIN + 8], zero outside the grid, by the
// CONV_RP warps that read it: thread t of 32 CONV_RP, 16-byte pieces in the order of both memories
template <int CIN>
__device__ __forceinline__ void stage_plane(__nv_bfloat16* ap, const __nv_bfloat16* x, int nx, int ny, int nz, int x0,
                                            int y0, int zz, unsigned t) {
  constexpr int CH = CIN / 8, RT = 32 * CONV_RP / CH, N = (CONV_TY + 2) * 18;
  const bool inz = zz >= 0 && zz < nz;
  const int c = (int)(t % CH);
  int q = (int)(t / CH), hy = q / 18, hx = q - 18 * hy;
  const __nv_bfloat16* const xp = x + (((long long)(inz ? zz : 0) * ny + y0 - 1) * nx + x0 - 1) * CIN + c * 8;
  __nv_bfloat16* const d = ap + q * (CIN + 8) + c * 8;
#pragma unroll
  for (int i = 0; i < (N + RT - 1) / RT; ++i) {
    if ((i + 1) * RT <= N || q + i * RT < N) {
      const bool in = inz && (unsigned)(x0 + hx - 1) < (unsigned)nx && (unsigned)(y0 + hy - 1) < (unsigned)ny;
      cp_async16(d + i * RT * (CIN + 8), in ? xp + (hy * nx + hx) * CIN : x, in);
    }
    hx += RT % 18;
    hy += RT / 18;
    if (hx >= 18) hx -= 18, ++hy;
  }
}

// (a + *b) + *c
__device__ __forceinline__ float4 sum3(float4 a, const float* b, const float* c) {
  const float4 u = *reinterpret_cast<const float4*>(b), v = *reinterpret_cast<const float4*>(c);
  return make_float4((a.x + u.x) + v.x, (a.y + u.y) + v.y, (a.z + u.z) + v.z, (a.w + u.w) + v.w);
}

// The epilogue of a tile of 16 x CONV_TY points over a whole block: four channels of a point at a time
// (a thread's channels are the same in every pass).
template <int COUT, int THREADS, int LV = 1>
struct ConvEpi {
  static constexpr int CPP = COUT / 4, PTS = LV * CONV_TY * 16, IT = (PTS * CPP + THREADS - 1) / THREADS;
  int co;
  float4 b4, db;   // the thread's biases, its sums for ConvEpilogue::db
  bool vec;        // 16-byte aligned outputs
  __device__ __forceinline__ explicit ConvEpi(const ConvEpilogue& o) : co((int)(4 * (threadIdx.x % CPP))) {
    b4 = o.bias ? make_float4(o.bias[co], o.bias[co + 1], o.bias[co + 2], o.bias[co + 3])
                : make_float4(0.f, 0.f, 0.f, 0.f);
    db = make_float4(0.f, 0.f, 0.f, 0.f);
    vec = (((uintptr_t)o.pre | (uintptr_t)o.yf | (uintptr_t)o.gpre | (uintptr_t)o.ybf) & 15) == 0;
  }
  __device__ __forceinline__ void st4(float* d, float4 v) const {
    if (vec) {
      *reinterpret_cast<float4*>(d) = v;
    } else {
      d[0] = v.x; d[1] = v.y; d[2] = v.z; d[3] = v.w;
    }
  }
  __device__ __forceinline__ float4 ld4(const float* d) const {
    return vec ? __ldg(reinterpret_cast<const float4*>(d)) : make_float4(d[0], d[1], d[2], d[3]);
  }
  // sum(pt, channel): the convolution's four sums at point pt of the tile's LV levels
  template <class F>
  __device__ __forceinline__ void tile(const ConvEpilogue& o, int nx, int ny, int nz, int x0, int y0, int z, const F& sum) {
#pragma unroll
    for (int i = 0; i < IT; ++i) {
      const unsigned pt = threadIdx.x / CPP + i * (THREADS / CPP);
      const int y = y0 + (int)(pt / 16 % CONV_TY), zl = z + (LV > 1 ? (int)(pt / (16 * CONV_TY)) : 0);
      if (pt >= PTS || y >= ny || zl >= nz) continue;
      // two levels: a grid of at most two tiles an SM
      const std::conditional_t<(LV > 1), int, long long> row = (std::conditional_t<(LV > 1), int, long long>)zl * ny + y;
      const long long p = row * nx + x0 + (int)(pt % 16);
      float4 gp = make_float4(0.f, 0.f, 0.f, 0.f);
      if (o.gpre) gp = ld4(o.gpre + p * COUT + co);
      float4 a = sum(pt, co);
      a = make_float4(a.x + b4.x, a.y + b4.y, a.z + b4.z, a.w + b4.w);
      if (o.pre) st4(o.pre + p * COUT + co, a);
      if (o.gelu) a = make_float4(gelu_tanh_fast(a.x), gelu_tanh_fast(a.y), gelu_tanh_fast(a.z), gelu_tanh_fast(a.w));
      if (o.gpre)
        a = make_float4(a.x * gelu_tanh_grad(gp.x), a.y * gelu_tanh_grad(gp.y), a.z * gelu_tanh_grad(gp.z),
                        a.w * gelu_tanh_grad(gp.w));
      if (co + 3 >= o.creal) {
        if (co >= o.creal) a.x = 0.f;
        if (co + 1 >= o.creal) a.y = 0.f;
        if (co + 2 >= o.creal) a.z = 0.f;
        a.w = 0.f;
      }
      if (o.ybf) {
        const __nv_bfloat162 lo = __floats2bfloat162_rn(a.x, a.y), hi = __floats2bfloat162_rn(a.z, a.w);
        __nv_bfloat16* const d = reinterpret_cast<__nv_bfloat16*>(o.ybf) + p * COUT + co;
        if (vec) {
          uint2 qq;
          qq.x = *reinterpret_cast<const uint32_t*>(&lo);
          qq.y = *reinterpret_cast<const uint32_t*>(&hi);
          *reinterpret_cast<uint2*>(d) = qq;
        } else {
          reinterpret_cast<__nv_bfloat162*>(d)[0] = lo;
          reinterpret_cast<__nv_bfloat162*>(d)[1] = hi;
        }
        const float2 l = __bfloat1622float2(lo), h = __bfloat1622float2(hi);
        db = make_float4(db.x + l.x, db.y + l.y, db.z + h.x, db.w + h.y);
      }
      if (o.yf && !o.compact) {
        st4(o.yf + p * COUT + co, a);
      } else if (o.yf) {
        float* const d = o.yf + p * o.creal + co;
        if (co < o.creal) d[0] = a.x;
        if (co + 1 < o.creal) d[1] = a.y;
        if (co + 2 < o.creal) d[2] = a.z;
        if (co + 3 < o.creal) d[3] = a.w;
      }
    }
  }
  // the block's sums of o.db, by one addition a channel (one a warp and channel, 2000 to an address, held a
  // gradient layer at 32^3 up for 5 us); scratch: THREADS / 32 * COUT floats of shared memory no longer read
  __device__ __forceinline__ void finish(const ConvEpilogue& o, float* scratch) {
    if (!o.db) return;
#pragma unroll
    for (int m = CPP; m < 32; m *= 2) {
      db.x += __shfl_xor_sync(0xffffffffu, db.x, m);
      db.y += __shfl_xor_sync(0xffffffffu, db.y, m);
      db.z += __shfl_xor_sync(0xffffffffu, db.z, m);
      db.w += __shfl_xor_sync(0xffffffffu, db.w, m);
    }
    __syncthreads();
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    if (lane < CPP) *reinterpret_cast<float4*>(scratch + warp * COUT + 4 * lane) = db;
    __syncthreads();
    if (threadIdx.x < COUT) {
      float v = 0.f;
      for (int w = 0; w < THREADS / 32; ++w) v += scratch[w * COUT + threadIdx.x];
      atomicAdd(o.db + threadIdx.x, v);
    }
  }
};

template <int CIN, int COUT>
__global__ void __launch_bounds__(ConvSmem<CIN, COUT>::THREADS)
    k_conv3d_smem(int nx, int ny, int nz, const __nv_bfloat16* __restrict__ x, const __nv_bfloat16* __restrict__ w,
                  const ConvEpilogue o, int early_weights) {
  using L = ConvSmem<CIN, COUT>;
  constexpr int CP = L::CP, NT = L::NT, KC = CIN / 16;
  extern __shared__ __align__(16) __nv_bfloat16 conv_smem[];
  __nv_bfloat16* Ws = conv_smem;
  __nv_bfloat16* As = conv_smem + L::W_ELEMS;
  float* Ps = reinterpret_cast<float*>(As);  // partial sums, after the tile's reads of As
  const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
  const int dz = wid / CONV_RP, rp = wid % CONV_RP;
  // early_weights: the weights are not written by the previous kernel of the stream, so their
  // staging overlaps that kernel's tail (launched as a programmatic dependent); the input is
  // read only after pdl_wait
  pdl_launch_dependents();
  if (!early_weights) pdl_wait();
  stage_taps<CIN, COUT, L::THREADS>(Ws, w);
  if (early_weights) pdl_wait();
  const int tiles_x = nx / 16, tiles_y = (ny + CONV_TY - 1) / CONV_TY;
  const long long ntiles = (long long)tiles_x * tiles_y * nz;
  const int g = lane >> 2, t = lane & 3;
  // ldmatrix row addresses: A (x4): matrix m = lane/8 -> rows (m & 1) * 8 + lane % 8, k half m >> 1
  const int a_row = ((lane >> 3) & 1) * 8 + (lane & 7), a_k = (lane >> 4) * 8;
  // B (x4, two n8 tiles): matrix m -> tile m >> 1, k half m & 1; (x2) matrix m -> k half m
  const int b_row = (lane >> 4) * 8 + (lane & 7), b_k = ((lane >> 3) & 1) * 8;
  ConvEpi<COUT, L::THREADS> ep(o);
  for (long long tile = blockIdx.x; tile < ntiles; tile += gridDim.x) {
    const int tx = (int)(tile % tiles_x), ty = (int)((tile / tiles_x) % tiles_y);
    const int z = (int)(tile / ((long long)tiles_x * tiles_y));
    const int x0 = tx * 16, y0 = ty * CONV_TY;
    __syncthreads();  // the previous tile's reads of As / Ps are done
    stage_plane<CIN>(As + dz * (CONV_TY + 2) * 18 * CP, x, nx, ny, nz, x0, y0, z + dz - 1, rp * 32 + lane);
    cp_async_wait_all();
    __syncthreads();
    const int ya = y0 + rp, yb = ya + CONV_RP;  // the warp's two rows
    const bool plane = z + dz - 1 >= 0 && z + dz - 1 < nz;
    float acc[CONV_MR][NT][4];
#pragma unroll
    for (int m = 0; m < CONV_MR; ++m)
#pragma unroll
      for (int n = 0; n < NT; ++n)
#pragma unroll
        for (int q = 0; q < 4; ++q) acc[m][n][q] = 0.f;
    if (plane && ya < ny) {
#pragma unroll 1
      for (int dy = 0; dy < 3; ++dy) {
        const bool ina = ya + dy - 1 >= 0 && ya + dy - 1 < ny, inb = yb + dy - 1 >= 0 && yb + dy - 1 < ny;
        if (!ina && !inb) continue;
        const __nv_bfloat16* arow = As + ((dz * (CONV_TY + 2) + rp + dy) * 18) * CP;
#pragma unroll
        for (int dx = 0; dx < 3; ++dx) {
          const __nv_bfloat16* wo = Ws + ((dz * 9 + dy * 3 + dx) * COUT) * CP;
#pragma unroll
          for (int kc = 0; kc < KC; ++kc) {
            uint32_t a[CONV_MR][4];
#pragma unroll
            for (int m = 0; m < CONV_MR; ++m)
              ldsm_x4(a[m], arow + (m * CONV_RP * 18 + dx + a_row) * CP + kc * 16 + a_k);
            if constexpr (NT == 1) {
              uint32_t b[2];
              ldsm_x2(b, wo + (lane & 7) * CP + kc * 16 + ((lane >> 3) & 1) * 8);
#pragma unroll
              for (int m = 0; m < CONV_MR; ++m) mma_bf16(acc[m][0], a[m], b);
            } else {
#pragma unroll
              for (int n2 = 0; n2 < NT / 2; ++n2) {
                uint32_t b4[4];
                ldsm_x4(b4, wo + (n2 * 16 + b_row) * CP + kc * 16 + b_k);
                const uint32_t b0[2] = {b4[0], b4[1]}, b1[2] = {b4[2], b4[3]};
#pragma unroll
                for (int m = 0; m < CONV_MR; ++m) {
                  mma_bf16(acc[m][2 * n2], a[m], b0);
                  mma_bf16(acc[m][2 * n2 + 1], a[m], b1);
                }
              }
            }
          }
        }
      }
    }
    __syncthreads();  // every warp is done with As: it becomes the partial sums [point][channel]
    // the planes' sums meet as (plane 0 + plane 1) + plane 2 (zeros where a plane does not exist):
    // in the epilogue, or with two buffers plane 2's warps add theirs to the other two
    constexpr int PS = L::PS, PB = CONV_TY * 16 * PS;
    auto each = [&](const auto& f) {
#pragma unroll
      for (int m = 0; m < CONV_MR; ++m)
#pragma unroll
        for (int n = 0; n < NT; ++n)
#pragma unroll
          for (int h = 0; h < 2; ++h)
            f(reinterpret_cast<float2*>(Ps + ((rp + m * CONV_RP) * 16 + g + 8 * h) * PS + n * 8 + 2 * t),
              make_float2(acc[m][n][2 * h], acc[m][n][2 * h + 1]));
    };
    if (dz < L::NB) each([&](float2* d, float2 v) { d[dz * (PB / 2)] = v; });
    __syncthreads();
    if (L::NB == 2) {
      if (dz == 2)
        each([&](float2* d, float2 v) {
          const float2 a = d[0], b = d[PB / 2];
          d[0] = make_float2((a.x + b.x) + v.x, (a.y + b.y) + v.y);
        });
      __syncthreads();
    }
    ep.tile(o, nx, ny, nz, x0, y0, z, [&](int pt, int c) {
      const float* const r = Ps + pt * PS + c;
      const float4 a = *reinterpret_cast<const float4*>(r);
      return L::NB == 3 ? sum3(a, r + PB, r + 2 * PB) : a;
    });
  }
  ep.finish(o, reinterpret_cast<float*>(conv_smem));
}

// The same convolution, two levels a block, once over the grid: where that gives each SM one block, the
// weights cross once a block instead of once a level, the levels share two of their four input planes,
// and a warp's A fragments feed both levels: 32^3, 9.1 -> 7.7 us a layer 16 -> 32, 11.5 -> 9.7 (32 -> 32),
// 6.8 -> 5.5 (32 -> 8).  Of the 9.7 us the products take 4.1 (one mma.sync in 8 cycles a scheduler is the
// tensor pipe's rate, 3.6 us here), staging 2.2, the sums and the epilogue 2.3, one after another with one
// block an SM.  Warp (p, r) takes input plane z0 + p - 1 for the levels it feeds; the sums are those of
// k_conv3d_smem, bit for bit.  PACK (16 -> 32): the input made from the state where it is staged, for the
// halo too, in place of a kernel that writes it: 2.0 us of a correction.
template <int CIN, int COUT>
struct ConvSmem2 {
  using S = ConvSmem<CIN, COUT>;
  static constexpr int PS = COUT == 8 ? 12 : COUT + 8;   // floats a point of partial sums: stores of 8 bytes in distinct banks
  static constexpr int WARPS = 4 * CONV_RP, THREADS = 32 * WARPS;
  static constexpr size_t A_BYTES = (size_t)4 * (CONV_TY + 2) * 18 * S::CP * 2;
  static constexpr size_t IN = (size_t)S::W_ELEMS * 2 + A_BYTES, OUT = (size_t)6 * CONV_TY * 16 * PS * 4;   // OUT over IN
  static constexpr size_t BYTES = IN > OUT ? IN : OUT;
};

template <int CIN, int COUT, bool PACK>
__global__ void __launch_bounds__(ConvSmem2<CIN, COUT>::THREADS)
    k_conv3d_smem2(int nx, int ny, int nz, const __nv_bfloat16* __restrict__ x, const PackIn in,
                   const __nv_bfloat16* __restrict__ w, const ConvEpilogue o, int early_weights) {
  using L = ConvSmem2<CIN, COUT>;
  using S1 = ConvSmem<CIN, COUT>;
  constexpr int CP = S1::CP, NT = S1::NT, KC = CIN / 16, PS = L::PS, PB = CONV_TY * 16 * PS;
  extern __shared__ __align__(16) __nv_bfloat16 conv_smem[];
  __nv_bfloat16* Ws = conv_smem;
  __nv_bfloat16* As = conv_smem + S1::W_ELEMS;
  float* Ps = reinterpret_cast<float*>(conv_smem);   // partial sums [level][tap plane], over everything
  const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
  const int pl = wid / CONV_RP, rp = wid % CONV_RP;
  pdl_launch_dependents();
  if (!early_weights) pdl_wait();
  stage_taps<CIN, COUT, L::THREADS>(Ws, w);
  ConvEpi<COUT, L::THREADS, 2> ep(o);
  const int tiles_x = nx / 16, tiles_y = (ny + CONV_TY - 1) / CONV_TY;
  const int tx = blockIdx.x % tiles_x, ty = (blockIdx.x / tiles_x) % tiles_y;
  const int x0 = tx * 16, y0 = ty * CONV_TY, z0 = 2 * (blockIdx.x / (tiles_x * tiles_y));
  std::conditional_t<PACK, PackNorm, int> nrm{};
  if constexpr (PACK) nrm = PackNorm(in, min(max(z0 + pl - 1, 0), nz - 1), nz);   // constant, like the weights
  if (early_weights) pdl_wait();
  __nv_bfloat16* const ap = As + pl * (CONV_TY + 2) * 18 * CP;
  if constexpr (PACK) {
    const int zz = z0 + pl - 1;
    constexpr int PTS = (CONV_TY + 2) * 18, T = 32 * CONV_RP, IT = (PTS + T - 1) / T;
    const bool inz = zz >= 0 && zz < nz;
    PackPoint f[IT];
    bool ok[IT];
#pragma unroll
    for (int i = 0; i < IT; ++i) {
      const int e = rp * 32 + lane + i * T, xx = x0 + e % 18 - 1, yy = y0 + e / 18 - 1;
      ok[i] = inz && e < PTS && xx >= 0 && xx < nx && yy >= 0 && yy < ny;
      if (ok[i]) f[i].load(in, xx, yy, zz, nx, ny);
    }
#pragma unroll
    for (int i = 0; i < IT; ++i) {
      const int e = rp * 32 + lane + i * T;
      if (e >= PTS) continue;
      uint4* const d = reinterpret_cast<uint4*>(ap + e * CP);
      d[0] = ok[i] ? f[i].channels(in, nrm) : make_uint4(0u, 0u, 0u, 0u);
      d[1] = make_uint4(0u, 0u, 0u, 0u);
    }
  } else {
    stage_plane<CIN>(ap, x, nx, ny, nz, x0, y0, z0 + pl - 1, rp * 32 + lane);
  }
  cp_async_wait_all();
  __syncthreads();
  const int g = lane >> 2, t = lane & 3;
  const int a_row = ((lane >> 3) & 1) * 8 + (lane & 7), a_k = (lane >> 4) * 8;
  const int b_row = (lane >> 4) * 8 + (lane & 7), b_k = ((lane >> 3) & 1) * 8;
  const int ya = y0 + rp, yb = ya + CONV_RP;
  float acc[2][CONV_MR][NT][4];
#pragma unroll
  for (int l = 0; l < 2; ++l)
#pragma unroll
    for (int m = 0; m < CONV_MR; ++m)
#pragma unroll
      for (int n = 0; n < NT; ++n)
#pragma unroll
        for (int q = 0; q < 4; ++q) acc[l][m][n][q] = 0.f;
  // the products of a plane that feeds levels LA..LB
  auto products = [&](auto la, auto lb) {
    constexpr int LA = decltype(la)::value, LB = decltype(lb)::value;
#pragma unroll 1
    for (int dy = 0; dy < 3; ++dy) {
      const bool ina = ya + dy - 1 >= 0 && ya + dy - 1 < ny, inb = yb + dy - 1 >= 0 && yb + dy - 1 < ny;
      if (!ina && !inb) continue;
      const __nv_bfloat16* arow = As + ((pl * (CONV_TY + 2) + rp + dy) * 18 + a_row) * CP + a_k;
      const __nv_bfloat16* wrow = Ws + ((pl * 9 + dy * 3) * COUT + (NT == 1 ? lane & 7 : b_row)) * CP + b_k;
      if constexpr (NT == 1) {   // few products: every load first
        uint32_t a[3 * KC][CONV_MR][4], b[3 * KC][2][2];
#pragma unroll
        for (int i = 0; i < 3 * KC; ++i) {
#pragma unroll
          for (int m = 0; m < CONV_MR; ++m)
            ldsm_x4(a[i][m], arow + (m * CONV_RP * 18 + i / KC) * CP + i % KC * 16);
#pragma unroll
          for (int l = LA; l <= LB; ++l) ldsm_x2(b[i][l], wrow + (i / KC - 9 * l) * COUT * CP + i % KC * 16);
        }
#pragma unroll
        for (int i = 0; i < 3 * KC; ++i)
#pragma unroll
          for (int l = LA; l <= LB; ++l)
#pragma unroll
            for (int m = 0; m < CONV_MR; ++m) mma_bf16(acc[l][m][0], a[i][m], b[i][l]);
        continue;
      }
#pragma unroll
      for (int dx = 0; dx < 3; ++dx) {
#pragma unroll
        for (int kc = 0; kc < KC; ++kc) {
          uint32_t a[CONV_MR][4];
#pragma unroll
          for (int m = 0; m < CONV_MR; ++m) ldsm_x4(a[m], arow + (m * CONV_RP * 18 + dx) * CP + kc * 16);
#pragma unroll
          for (int l = LA; l <= LB; ++l) {   // the plane is tap dz = pl - l of level z0 + l
            const __nv_bfloat16* wo = wrow + (dx - 9 * l) * COUT * CP + kc * 16;
#pragma unroll
            for (int n2 = 0; n2 < NT / 2; ++n2) {
              uint32_t b4[4];
              ldsm_x4(b4, wo + n2 * 16 * CP);
              const uint32_t b0[2] = {b4[0], b4[1]}, b1[2] = {b4[2], b4[3]};
#pragma unroll
              for (int m = 0; m < CONV_MR; ++m) {
                mma_bf16(acc[l][m][2 * n2], a[m], b0);
                mma_bf16(acc[l][m][2 * n2 + 1], a[m], b1);
              }
            }
          }
        }
      }
    }
  };
  if (z0 + pl - 1 >= 0 && z0 + pl - 1 < nz && ya < ny) {
    constexpr std::integral_constant<int, 0> lo{};
    constexpr std::integral_constant<int, 1> hi{};
    if (pl == 0)
      products(lo, lo);
    else if (pl == 3)
      products(hi, hi);
    else
      products(lo, hi);
  }
  __syncthreads();   // every warp is done with the weights and planes: the partial sums replace them
#pragma unroll
  for (int l = 0; l < 2; ++l) {
    const int dz = pl - l;
    if (dz < 0 || dz > 2) continue;
    float* const d = Ps + (l * 3 + dz) * PB;
#pragma unroll
    for (int m = 0; m < CONV_MR; ++m)
#pragma unroll
      for (int n = 0; n < NT; ++n)
#pragma unroll
        for (int h = 0; h < 2; ++h)
          *reinterpret_cast<float2*>(d + ((rp + m * CONV_RP) * 16 + g + 8 * h) * PS + n * 8 + 2 * t) =
              make_float2(acc[l][m][n][2 * h], acc[l][m][n][2 * h + 1]);
  }
  __syncthreads();
  ep.tile(o, nx, ny, nz, x0, y0, z0, [&](int pt, int c) {
    const float* const r = Ps + (pt / (16 * CONV_TY)) * 2 * PB + pt * PS + c;
    return sum3(*reinterpret_cast<const float4*>(r), r + PB, r + 2 * PB);
  });
  ep.finish(o, reinterpret_cast<float*>(conv_smem));
}

// [npts][5] FP32 -> [npts][16] BF16, the padding zero: the network's input, and the gradient at its
// output; db (8 channels) += the sums of the rounded values, one addition a block and channel (one a warp
// and channel, 9700 to an address, took most of the gradient's 75 us at 128x128x64, now 13; 54 MB moved).
__global__ void __launch_bounds__(256) k_pad5(long long npts, const float* __restrict__ in, uint4* __restrict__ out,
                                              float* __restrict__ db) {
  float s[5] = {0.f, 0.f, 0.f, 0.f, 0.f};
  for (long long p = (long long)blockIdx.x * blockDim.x + threadIdx.x; p < npts; p += (long long)gridDim.x * blockDim.x) {
    unsigned short h[6];
#pragma unroll
    for (int c = 0; c < 5; ++c) {
      const __nv_bfloat16 b = __float2bfloat16_rn(__ldg(in + p * 5 + c));
      h[c] = __bfloat16_as_ushort(b);
      s[c] += __bfloat162float(b);
    }
    out[2 * p] = make_uint4(h[0] | (uint32_t)h[1] << 16, h[2] | (uint32_t)h[3] << 16, h[4], 0u);
    out[2 * p + 1] = make_uint4(0u, 0u, 0u, 0u);
  }
  if (!db) return;
  __shared__ float part[5][8];
#pragma unroll
  for (int c = 0; c < 5; ++c) {
#pragma unroll
    for (int m = 16; m > 0; m /= 2) s[c] += __shfl_xor_sync(0xffffffffu, s[c], m);
    if ((threadIdx.x & 31) == 0) part[c][threadIdx.x >> 5] = s[c];
  }
  __syncthreads();
  if (threadIdx.x < 5) {
    float v = 0.f;
    for (int w = 0; w < 8; ++w) v += part[threadIdx.x][w];
    atomicAdd(db + threadIdx.x, v);
  }
}

// The input-gradient weights of the four layers: [27][cout][cin] -> [27][cin][g], offsets reversed,
// the g gradient channels cout padded with zeros (16 for the last layer's 8).
struct MirrorArgs {
  const __nv_bfloat16* w[4];
  __nv_bfloat16* out[4];
  int cin[4], cout[4], g[4], end[4];   // end: running total of the outputs
};
__global__ void k_mirror(MirrorArgs a) {
  int t = blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= a.end[3]) return;
  const int l = t < a.end[0] ? 0 : t < a.end[1] ? 1 : t < a.end[2] ? 2 : 3;
  if (l) t -= a.end[l - 1];
  const int co = t % a.g[l], ci = t / a.g[l] % a.cin[l], tap = t / (a.g[l] * a.cin[l]);
  a.out[l][t] = co < a.cout[l] ? a.w[l][((26 - tap) * a.cout[l] + co) * a.cin[l] + ci] : __float2bfloat16_rn(0.f);
}

// g[p][c] = dy[p][c] * GELU'(pre[p][c]) for c < C (pre and dy have C channels, FP32), written
// as BF16 with Cpad >= C channels (the padding zero)
__global__ void k_gelu_bwd(long long npts, int C, int Cpad, const float* __restrict__ dy, const float* __restrict__ pre,
                           __nv_bfloat16* __restrict__ g) {
  const long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= npts * Cpad) return;
  const long long p = t / Cpad;
  const int c = (int)(t - p * Cpad);
  float v = 0.f;
  if (c < C) v = dy[p * C + c] * (pre ? gelu_tanh_grad(pre[p * C + c]) : 1.f);
  g[t] = __float2bfloat16(v);
}

// dW[off][co][ci] += sum over a slab of points p of g[p][co] * x[p+off][ci] (zero outside).
// Block: one offset, SLAB consecutive points, threads over (co, ci).
constexpr int SLAB = 128;  // (cin + cout) * SLAB * 4 B <= 32 KB of shared memory
__global__ void k_conv3d_dw(int nx, int ny, int nz, int cin, int cout, int gstride, const __nv_bfloat16* __restrict__ x,
                            const __nv_bfloat16* __restrict__ g, float* __restrict__ dw) {
  extern __shared__ float sm[];
  float* gs = sm;                 // [SLAB][cout]
  float* xs = sm + SLAB * cout;   // [SLAB][cin]
  const int off = blockIdx.y;
  const int dz = off / 9 - 1, dy = (off / 3) % 3 - 1, dx = off % 3 - 1;
  const long long npts = (long long)nx * ny * nz;
  const long long p0 = (long long)blockIdx.x * SLAB;
  for (int e = threadIdx.x; e < SLAB * cout; e += blockDim.x) {
    const long long p = p0 + e / cout;
    gs[e] = p < npts ? __bfloat162float(g[p * gstride + e % cout]) : 0.f;
  }
  for (int e = threadIdx.x; e < SLAB * cin; e += blockDim.x) {
    const long long p = p0 + e / cin;
    float v = 0.f;
    if (p < npts) {
      const int i = (int)(p % nx), j = (int)((p / nx) % ny), k = (int)(p / ((long long)nx * ny));
      const int ii = i + dx, jj = j + dy, kk = k + dz;
      if (ii >= 0 && ii < nx && jj >= 0 && jj < ny && kk >= 0 && kk < nz)
        v = __bfloat162float(x[(((long long)kk * ny + jj) * nx + ii) * cin + e % cin]);
    }
    xs[e] = v;
  }
  __syncthreads();
  for (int e = threadIdx.x; e < cout * cin; e += blockDim.x) {
    const int co = e / cin, ci = e % cin;
    float acc = 0.f;
    for (int q = 0; q < SLAB; ++q) acc += gs[q * cout + co] * xs[q * cin + ci];
    atomicAdd(&dw[((long long)off * cout + co) * cin + ci], acc);
  }
}

// db[co] += sum_p g[p][co]
__global__ void k_bias_grad(long long npts, int cout, int gstride, const __nv_bfloat16* __restrict__ g,
                            float* __restrict__ db) {
  const int co = threadIdx.x % cout;
  const int lanes = blockDim.x / cout;
  float acc = 0.f;
  for (long long p = (long long)blockIdx.x * lanes + threadIdx.x / cout; p < npts; p += (long long)gridDim.x * lanes)
    acc += __bfloat162float(g[p * gstride + co]);
  if (threadIdx.x < lanes * cout) atomicAdd(&db[co], acc);
}

// Adam (bias-corrected moments) on FP32 master parameters, with an optional BF16 copy
__global__ void k_adam(long long n, float* __restrict__ w, const float* __restrict__ gw, float* __restrict__ m,
                       float* __restrict__ v, __nv_bfloat16* __restrict__ wbf, float lr, float b1, float b2, float eps,
                       float c1, float c2) {
  const long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= n) return;
  const float gg = gw[t];
  const float mm = b1 * m[t] + (1.f - b1) * gg;
  const float vv = b2 * v[t] + (1.f - b2) * gg * gg;
  m[t] = mm;
  v[t] = vv;
  const float ww = w[t] - lr * (mm / c1) / (sqrtf(vv / c2) + eps);
  w[t] = ww;
  if (wbf) wbf[t] = __float2bfloat16(ww);
}

// Input of the network (PackPoint), one thread per cell, 16 BF16 channels (32 bytes)
__global__ void k_sgs_pack(int nx, int ny, int nz, const PackIn in, uint4* __restrict__ x16) {
  pdl_launch_dependents();
  pdl_wait();
  const long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  const long long plane = (long long)nx * ny;
  if (t >= plane * nz) return;
  const int k = (int)(t / plane);
  PackPoint f;
  f.load(in, (int)(t % nx), (int)((t / nx) % ny), k, nx, ny);
  x16[2 * t] = f.channels(in, PackNorm(in, k, nz));
  x16[2 * t + 1] = make_uint4(0u, 0u, 0u, 0u);
}

// The correction corr[p][0..4] (FP32, 8 channels a point) back on the grid as
// dl_models.correct_array2tuple and one_sprint_functions.py:139-151 apply it: theta and qv at the
// cell; u (v) on the west (south) face i >= 1 as the mean of the two cells beside it and on face 0
// the value of face nx-1 (stagger_uvw copies the face next to the far end onto the end face,
// dl_models.py:172-182); w on the interior faces 1..nz-1 as the mean of the cells below and above
// (bottom and lid untouched); each times the output range at its own point, rout[f][l][j][i]
// (stride nz+1 levels: cells for theta and qv, west / south faces for u / v, faces 0..nz for w).
// One thread per cell; it writes only its own cell and its own west, south and bottom faces.  corr is
// still being written when the kernel's blocks start (no __restrict__: its loads stay behind pdl_wait).
__global__ void k_sgs_unpack(int nx, int ny, int nz, const float* corr, const float* __restrict__ rout,
                             float* __restrict__ T, float* __restrict__ u, float* __restrict__ v, float* __restrict__ w,
                             float* __restrict__ q) {
  const long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  const long long plane = (long long)nx * ny, cells = plane * nz, rstride = plane * (nz + 1);
  if (t >= cells) return;
  const int i = (int)(t % nx), j = (int)((t / nx) % ny), k = (int)(t / plane);
  float r[5];   // the ranges are the context's copies, like the weights: read while the network finishes
#pragma unroll
  for (int f = 0; f < 5; ++f) r[f] = __ldg(rout + f * rstride + t);
  // the two cells beside the west (south) face; face 0 takes cells nx-2, nx-1 (ny-2, ny-1)
  const long long ua = i > 0 ? t - 1 : t + (nx - 2), ub = i > 0 ? t : t + (nx - 1);
  const long long va = j > 0 ? t - nx : t + (long long)(ny - 2) * nx, vb = j > 0 ? t : t + (long long)(ny - 1) * nx;
  pdl_wait();
  auto c = [&](long long p, int f) { return corr[p * 8 + f]; };
  T[t] = __fadd_rn(T[t], __fmul_rn(c(t, 0), r[0]));
  u[t] = __fadd_rn(u[t], __fmul_rn(__fmul_rn(0.5f, __fadd_rn(c(ua, 1), c(ub, 1))), r[1]));
  v[t] = __fadd_rn(v[t], __fmul_rn(__fmul_rn(0.5f, __fadd_rn(c(va, 2), c(vb, 2))), r[2]));
  if (k > 0) w[t] = __fadd_rn(w[t], __fmul_rn(__fmul_rn(0.5f, __fadd_rn(c(t - plane, 3), c(t, 3))), r[3]));
  q[t] = __fadd_rn(q[t], __fmul_rn(c(t, 4), r[4]));
}
}  // namespace

// Persistent-grid size of k_conv3d_smem<CIN, COUT> (resident blocks on the current device), set
// up once per device: the dynamic shared-memory opt-in and the occupancy query are not stream
// operations, so they run here (conv_prepare) before any graph capture.
constexpr int CONV_MAX_DEVICES = 64;

template <int CIN, int COUT>
cudaError_t conv_grid(int* cap, int* nsm) {
  static int grid_cap[CONV_MAX_DEVICES] = {}, sm_count[CONV_MAX_DEVICES] = {};
  int dev = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) return e;
  if (dev < 0 || dev >= CONV_MAX_DEVICES) return cudaErrorInvalidDevice;
  if (!grid_cap[dev]) {
    using L = ConvSmem<CIN, COUT>;
    constexpr cudaFuncAttribute dyn = cudaFuncAttributeMaxDynamicSharedMemorySize;
    const int two = (int)ConvSmem2<CIN, COUT>::BYTES;
    if ((e = cudaFuncSetAttribute(k_conv3d_smem<CIN, COUT>, dyn, (int)L::BYTES)) != cudaSuccess) return e;
    if ((e = cudaFuncSetAttribute(k_conv3d_smem2<CIN, COUT, false>, dyn, two)) != cudaSuccess) return e;
    if constexpr (CIN == 16 && COUT == 32)
      if ((e = cudaFuncSetAttribute(k_conv3d_smem2<CIN, COUT, true>, dyn, two)) != cudaSuccess) return e;
    int sms = 0, per = 0;
    if ((e = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev)) != cudaSuccess) return e;
    if ((e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per, k_conv3d_smem<CIN, COUT>, L::THREADS, L::BYTES)) !=
        cudaSuccess)
      return e;
    sm_count[dev] = sms;
    grid_cap[dev] = sms * (per > 0 ? per : 1);
  }
  *cap = grid_cap[dev];
  *nsm = sm_count[dev];
  return cudaSuccess;
}

// One level a block where every block has an SM of its own, two where that still gives each SM one block,
// else tiles in turn on the resident blocks (a correction at 32^3: 40.0 us in turn, 34.5 in pairs)
static long long conv_tiles(int nx, int ny, int nz) { return (long long)(nx / 16) * ((ny + CONV_TY - 1) / CONV_TY) * nz; }
static bool conv_pairs(int nx, int ny, int nz, int sms) {
  const long long t = conv_tiles(nx, ny, nz);
  return t > sms && t / nz * ((nz + 1) / 2) <= sms;
}

// pdl: launch as a programmatic dependent of the previous kernel of the stream, staging the
// weights before waiting for it (the caller guarantees that kernel does not write them).  pack: the
// state the input is made of in place (16 -> 32 channels where conv_pairs).
template <int CIN, int COUT>
cudaError_t launch_conv_smem(int nx, int ny, int nz, const __nv_bfloat16* x, const __nv_bfloat16* w,
                             const ConvEpilogue& o, cudaStream_t st, bool pdl, const PackIn* pack = nullptr) {
  int cap = 0, sms = 0;
  cudaError_t e = conv_grid<CIN, COUT>(&cap, &sms);
  if (e != cudaSuccess) return e;
  const long long ntiles = conv_tiles(nx, ny, nz);
  using L = ConvSmem<CIN, COUT>;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)(ntiles < cap ? ntiles : cap));
  cfg.blockDim = dim3(L::THREADS);
  cfg.dynamicSmemBytes = L::BYTES;
  cfg.stream = st;
  cudaLaunchAttribute at[1];
  at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = at;
  cfg.numAttrs = pdl ? 1 : 0;
  if (!conv_pairs(nx, ny, nz, sms))
    return cudaLaunchKernelEx(&cfg, k_conv3d_smem<CIN, COUT>, nx, ny, nz, x, w, o, pdl ? 1 : 0);
  cfg.gridDim = dim3((unsigned)(ntiles / nz * ((nz + 1) / 2)));
  cfg.blockDim = dim3(ConvSmem2<CIN, COUT>::THREADS);
  cfg.dynamicSmemBytes = ConvSmem2<CIN, COUT>::BYTES;
  if constexpr (CIN == 16 && COUT == 32)
    if (pack)
      return cudaLaunchKernelEx(&cfg, k_conv3d_smem2<CIN, COUT, true>, nx, ny, nz, x, *pack, w, o, pdl ? 1 : 0);
  return cudaLaunchKernelEx(&cfg, k_conv3d_smem2<CIN, COUT, false>, nx, ny, nz, x, PackIn{}, w, o, pdl ? 1 : 0);
}

// which convolution kernel conv3d uses (LEXGB_CNN_AUTO: tcgen05 where the grid fits its 8 x 16 tiles and
// has at least kConvTcMinPoints points, else mma.sync); process-wide, set by lexgb_cnn_set_kernel.  The
// line is where the two sum in different orders for a caller's results: below it tcgen05 is now the
// faster one as well (the four layers at 64x64x32: 55 us against 103), but its last
// bits, rounded to BF16 between layers, are other ones.
int g_conv_kernel = LEXGB_CNN_AUTO;
constexpr long long kConvTcMinPoints = 1ll << 18;

static cudaError_t conv3d(int nx, int ny, int nz, int cin, int cout, const void* x, const void* w,
                          const ConvEpilogue& o, cudaStream_t st, bool pdl) {
  const bool big = (long long)nx * ny * nz >= kConvTcMinPoints;
  if (conv_tc_fits(nx, ny, nz, cin, cout, x, o) &&
      (g_conv_kernel == LEXGB_CNN_TCGEN05 || (g_conv_kernel == LEXGB_CNN_AUTO && big)))
    return launch_conv_tc(nx, ny, nz, cin, cout, x, w, o, st, pdl);
  if (g_conv_kernel == LEXGB_CNN_TCGEN05) return cudaErrorInvalidValue;
  if (!(cin == 16 || cin == 32) || !(cout == 8 || cout == 16 || cout == 32) || nx % 16) return cudaErrorInvalidValue;
  const __nv_bfloat16* xb = (const __nv_bfloat16*)x;
  const __nv_bfloat16* wb = (const __nv_bfloat16*)w;
#define LEXGB_CONV(CI, CO) launch_conv_smem<CI, CO>(nx, ny, nz, xb, wb, o, st, pdl)
  if (cin == 16) return cout == 8 ? LEXGB_CONV(16, 8) : cout == 16 ? LEXGB_CONV(16, 16) : LEXGB_CONV(16, 32);
  return cout == 8 ? LEXGB_CONV(32, 8) : cout == 16 ? LEXGB_CONV(32, 16) : LEXGB_CONV(32, 32);
#undef LEXGB_CONV
}

cudaError_t launch_cnn_conv3d(int nx, int ny, int nz, int cin, int cout, const void* x, const void* w,
                              const float* bias, float* pre, void* ybf, float* yf, int gelu, int creal,
                              cudaStream_t st, bool pdl) {
  ConvEpilogue o;
  o.bias = bias;
  o.pre = pre;
  o.ybf = ybf;
  o.yf = yf;
  o.gelu = gelu;
  o.creal = creal;
  return conv3d(nx, ny, nz, cin, cout, x, w, o, st, pdl);
}

// dw[27][cout][cin] += sum_p g[p][co] x[p+off][ci] on the kernel that fits
static cudaError_t weight_grad(int nx, int ny, int nz, int cin, int cout, int gstride, const void* x, const void* g,
                               float* dw, cudaStream_t st) {
  if (g_conv_kernel != LEXGB_CNN_MMA && conv_dw_tc_fits(nx, ny, nz, cin, cout, gstride, x, g, dw))
    return launch_conv_dw_tc(nx, ny, nz, cin, cout, gstride, x, g, dw, st);
  if (g_conv_kernel == LEXGB_CNN_TCGEN05) return cudaErrorInvalidValue;
  const long long npts = (long long)nx * ny * nz;
  const dim3 grid((unsigned)((npts + SLAB - 1) / SLAB), 27);
  const size_t smem = (size_t)SLAB * (cin + cout) * sizeof(float);
  k_conv3d_dw<<<grid, 256, smem, st>>>(nx, ny, nz, cin, cout, gstride, (const __nv_bfloat16*)x,
                                       (const __nv_bfloat16*)g, dw);
  return cudaGetLastError();
}

cudaError_t conv_prepare() {
  int cap, sms;
  cudaError_t e;
  if ((e = conv_tc_prepare()) != cudaSuccess) return e;
  if ((e = conv_grid<16, 8>(&cap, &sms)) != cudaSuccess) return e;
  if ((e = conv_grid<16, 16>(&cap, &sms)) != cudaSuccess) return e;
  if ((e = conv_grid<16, 32>(&cap, &sms)) != cudaSuccess) return e;
  if ((e = conv_grid<32, 8>(&cap, &sms)) != cudaSuccess) return e;
  if ((e = conv_grid<32, 16>(&cap, &sms)) != cudaSuccess) return e;
  return conv_grid<32, 32>(&cap, &sms);
}

cudaError_t launch_sgs_input(int nx, int ny, int nz, const float* T, const float* u, const float* v, const float* w,
                             const float* q, float theta_ref, const float* lo, const float* rin, void* x16,
                             const void* w0, const float* b0, void* out, cudaStream_t st, bool pdl) {
  PackIn in;
  in.T = T;
  in.u = u;
  in.v = v;
  in.w = w;
  in.q = q;
  in.theta_ref = theta_ref;
  in.lo = lo;
  in.rin = rin;
  ConvEpilogue o;
  o.bias = b0;
  o.ybf = out;
  o.gelu = 1;
  o.creal = 32;
  int cap = 0, sms = 0;
  cudaError_t e = conv_grid<16, 32>(&cap, &sms);
  if (e != cudaSuccess) return e;
  const long long n = (long long)nx * ny * nz;
  if (nx % 16 == 0 && n < kConvTcMinPoints && g_conv_kernel != LEXGB_CNN_TCGEN05 && conv_pairs(nx, ny, nz, sms))
    return launch_conv_smem<16, 32>(nx, ny, nz, (const __nv_bfloat16*)x16, (const __nv_bfloat16*)w0, o, st, pdl, &in);
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)((n + 255) / 256));
  cfg.blockDim = dim3(256);
  cfg.stream = st;
  cudaLaunchAttribute at[1];
  at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = at;
  cfg.numAttrs = pdl ? 1 : 0;
  e = cudaLaunchKernelEx(&cfg, k_sgs_pack, nx, ny, nz, in, (uint4*)x16);
  return e != cudaSuccess ? e : conv3d(nx, ny, nz, 16, 32, x16, w0, o, st, pdl);
}

cudaError_t launch_sgs_unpack(int nx, int ny, int nz, const float* corr, const float* rout, float* T, float* u,
                              float* v, float* w, float* q, cudaStream_t st, bool pdl) {
  const long long n = (long long)nx * ny * nz;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)((n + 255) / 256));
  cfg.blockDim = dim3(256);
  cfg.stream = st;
  cudaLaunchAttribute at[1];
  at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = at;
  cfg.numAttrs = pdl ? 1 : 0;
  return cudaLaunchKernelEx(&cfg, k_sgs_unpack, nx, ny, nz, corr, rout, T, u, v, w, q);
}
}  // namespace lexgb

// ------------------------------------------------------------------------------------------------
// C ABI (include/lexgb.h); device pointers, ordered on `stream` (0: the legacy default stream)
// ------------------------------------------------------------------------------------------------
namespace lexgb {
void record_error(const std::string& msg);
}

namespace {
int cnn_status(cudaError_t e, const char* what) {
  if (e == cudaSuccess) return LEXGB_OK;
  lexgb::record_error(std::string(what) + ": " + cudaGetErrorString(e));
  return LEXGB_ERR_CUDA;
}
bool aligned(const void* p, uintptr_t to) { return (uintptr_t)p % to == 0; }
int cnn_arg(const char* msg) {
  lexgb::record_error(msg);
  return LEXGB_ERR_ARG;
}
}  // namespace

extern "C" int lexgb_cnn_conv3d(int nx, int ny, int nz, int cin, int cout, const void* x, const void* w,
                                const float* bias, float* pre, void* y_bf16, float* y_f32, int gelu, int creal,
                                void* stream) {
  using namespace lexgb;
  if (nx <= 0 || ny <= 0 || nz <= 0 || nx % 16) return cnn_arg("lexgb_cnn_conv3d: need nx a positive multiple of 16");
  if (cin <= 0 || cin % 16) return cnn_arg("lexgb_cnn_conv3d: cin must be a positive multiple of 16");
  if (!(cout == 8 || cout == 16 || cout == 32)) return cnn_arg("lexgb_cnn_conv3d: cout must be 8, 16 or 32");
  if (!x || !w || (!y_bf16 && !y_f32 && !pre)) return cnn_arg("lexgb_cnn_conv3d: null argument");
  // x and w are read, and y_bf16 is stored, in pieces of 16 and 4 bytes (4 and 2 for more input channels)
  const bool wide = cin == 16 || cin == 32;
  if (!aligned(x, wide ? 16 : 4) || !aligned(w, wide ? 16 : 4) || !aligned(y_bf16, wide ? 4 : 2) ||
      !aligned(bias, 4) || !aligned(pre, 4) || !aligned(y_f32, 4))
    return cnn_arg("lexgb_cnn_conv3d: x and w must be 16-byte aligned (cin 16 or 32), bias and outputs 4-byte");
  const long long warps = (long long)(nx / 16) * ny * nz;
  const unsigned blocks = (unsigned)((warps + 3) / 4);
  cudaStream_t st = (cudaStream_t)stream;
  const __nv_bfloat16* xb = (const __nv_bfloat16*)x;
  const __nv_bfloat16* wb = (const __nv_bfloat16*)w;
  __nv_bfloat16* yb = (__nv_bfloat16*)y_bf16;
  if (cin == 16 || cin == 32)
    return cnn_status(launch_cnn_conv3d(nx, ny, nz, cin, cout, x, w, bias, pre, y_bf16, y_f32, gelu, creal, st, false),
                      "lexgb_cnn_conv3d");
  if (cout == 8)
    k_conv3d<1><<<blocks, 128, 0, st>>>(nx, ny, nz, cin, xb, wb, bias, pre, yb, y_f32, gelu, creal);
  else if (cout == 16)
    k_conv3d<2><<<blocks, 128, 0, st>>>(nx, ny, nz, cin, xb, wb, bias, pre, yb, y_f32, gelu, creal);
  else
    k_conv3d<4><<<blocks, 128, 0, st>>>(nx, ny, nz, cin, xb, wb, bias, pre, yb, y_f32, gelu, creal);
  return cnn_status(cudaGetLastError(), "lexgb_cnn_conv3d");
}

extern "C" int lexgb_cnn_set_kernel(int which) {
  using namespace lexgb;
  if (which != LEXGB_CNN_AUTO && which != LEXGB_CNN_MMA && which != LEXGB_CNN_TCGEN05)
    return cnn_arg("lexgb_cnn_set_kernel: unknown kernel");
  g_conv_kernel = which;
  return LEXGB_OK;
}

extern "C" int lexgb_cnn_take_timeouts(unsigned int* n) {
  using namespace lexgb;
  if (!n) return cnn_arg("lexgb_cnn_take_timeouts: null output");
  return cnn_status(conv_tc_take_timeouts(n), "lexgb_cnn_take_timeouts");
}

extern "C" int lexgb_cnn_gelu_bwd(long long npts, int c, int cpad, const float* dy, const float* pre, void* g_bf16,
                                  void* stream) {
  using namespace lexgb;
  if (npts <= 0 || c <= 0 || cpad < c || !dy || !g_bf16) return cnn_arg("lexgb_cnn_gelu_bwd: bad argument");
  const long long n = npts * cpad;
  k_gelu_bwd<<<(unsigned)((n + 255) / 256), 256, 0, (cudaStream_t)stream>>>(npts, c, cpad, dy, pre,
                                                                           (__nv_bfloat16*)g_bf16);
  return cnn_status(cudaGetLastError(), "lexgb_cnn_gelu_bwd");
}

extern "C" int lexgb_cnn_conv3d_dw(int nx, int ny, int nz, int cin, int cout, int gstride, const void* x,
                                   const void* g, float* dw, float* db, void* stream) {
  using namespace lexgb;
  if (nx <= 0 || ny <= 0 || nz <= 0 || cin <= 0 || cout <= 0 || cin > 32 || cout > 32 || 256 % cout ||
      gstride < cout || !x || !g || !dw)
    return cnn_arg("lexgb_cnn_conv3d_dw: bad argument (cin, cout <= 32, cout divides 256, gstride >= cout)");
  const long long npts = (long long)nx * ny * nz;
  cudaStream_t st = (cudaStream_t)stream;
  if (g_conv_kernel == LEXGB_CNN_TCGEN05 && !conv_dw_tc_fits(nx, ny, nz, cin, cout, gstride, x, g, dw))
    return cnn_arg("lexgb_cnn_conv3d_dw: the tcgen05 kernel needs cin 16 or 32, gstride 16 or 32, cout <= gstride "
                   "and 16-byte aligned x and g");
  const cudaError_t e = weight_grad(nx, ny, nz, cin, cout, gstride, x, g, dw, st);
  if (e != cudaSuccess) return cnn_status(e, "lexgb_cnn_conv3d_dw");
  if (db) k_bias_grad<<<256, 256, 0, st>>>(npts, cout, gstride, (const __nv_bfloat16*)g, db);
  return cnn_status(cudaGetLastError(), "lexgb_cnn_conv3d_dw");
}

// ------------------------------------------------------------------------------------------------
// the network's training pass
// ------------------------------------------------------------------------------------------------
namespace {
constexpr int NET_CIN[4] = {16, 32, 32, 32}, NET_COUT[4] = {32, 32, 32, 8};
constexpr int NET_REAL = 5;

unsigned pad_blocks(long long n) {
  const long long b = (n + 255) / 256;
  return (unsigned)(b < 1216 ? b : 1216);   // few additions to db: 8 blocks on each of 152 SMs
}
// the grid; n16 pointers that move in 16-byte pieces (16-byte aligned), and n4 of floats
bool net_args(int nx, int ny, int nz, const void* const* p16, int n16, const void* const* p4, int n4) {
  if (nx <= 0 || ny <= 0 || nz <= 0 || nx % 16) return false;
  for (int i = 0; i < n16; ++i)
    if (!p16[i] || !aligned(p16[i], 16)) return false;
  for (int i = 0; i < n4; ++i)
    if (!p4[i] || !aligned(p4[i], 4)) return false;
  return true;
}
}  // namespace

extern "C" int lexgb_cnn_net_forward(int nx, int ny, int nz, const float* x, const void* const w[4],
                                     const float* const b[4], void* const act[4], float* const pre[3], float* out,
                                     void* stream) {
  using namespace lexgb;
  if (!w || !b || !act || !pre || !out) return cnn_arg("lexgb_cnn_net_forward: null argument");
  const void* p16[8] = {w[0], w[1], w[2], w[3], act[0], act[1], act[2], act[3]};
  const void* p4[9] = {b[0], b[1], b[2], b[3], pre[0], pre[1], pre[2], out, x ? x : out};
  if (!net_args(nx, ny, nz, p16, 8, p4, 9))
    return cnn_arg("lexgb_cnn_net_forward: null argument, nx not a positive multiple of 16, or w or act not 16-byte aligned");
  cudaStream_t st = (cudaStream_t)stream;
  const long long n = (long long)nx * ny * nz;
  if (x) {
    k_pad5<<<pad_blocks(n), 256, 0, st>>>(n, x, (uint4*)act[0], nullptr);
    if (cudaError_t e = cudaGetLastError()) return cnn_status(e, "lexgb_cnn_net_forward");
  }
  for (int l = 0; l < 4; ++l) {
    const bool last = l == 3;
    ConvEpilogue o;
    o.bias = b[l];
    o.pre = last ? nullptr : pre[l];
    o.ybf = last ? nullptr : act[l + 1];
    o.yf = last ? out : nullptr;
    o.gelu = !last;
    o.creal = last ? NET_REAL : NET_COUT[l];
    o.compact = last;
    // each layer stages its weights, which no kernel of this call writes, while the previous one drains;
    // not the first with x NULL: the kernel before it is the caller's, and may be the one that writes them
    const cudaError_t e = conv3d(nx, ny, nz, NET_CIN[l], NET_COUT[l], act[l], w[l], o, st, l > 0 || x);
    if (e != cudaSuccess) return cnn_status(e, "lexgb_cnn_net_forward");
  }
  return LEXGB_OK;
}

extern "C" int lexgb_cnn_net_backward(int nx, int ny, int nz, const float* gout, const void* const w[4],
                                      const void* const act[4], const float* const pre[3], void* work, float* grads,
                                      float* dx, void* stream) {
  using namespace lexgb;
  if (!gout || !w || !act || !pre || !work || !grads || !dx) return cnn_arg("lexgb_cnn_net_backward: null argument");
  const void* p16[9] = {w[0], w[1], w[2], w[3], act[0], act[1], act[2], act[3], work};
  const void* p4[6] = {pre[0], pre[1], pre[2], gout, grads, dx};
  if (!net_args(nx, ny, nz, p16, 9, p4, 6))
    return cnn_arg("lexgb_cnn_net_backward: null argument, nx not a positive multiple of 16, or w, act or work not "
                   "16-byte aligned");
  cudaStream_t st = (cudaStream_t)stream;
  const long long n = (long long)nx * ny * nz;
  // work: two gradients of 32 channels (the first also holds the 16 channels at the output), then the
  // mirrored weights; grads: dw of the four layers, then db
  __nv_bfloat16* const g[2] = {(__nv_bfloat16*)work, (__nv_bfloat16*)work + n * 32};
  MirrorArgs m;
  __nv_bfloat16* wm = g[1] + n * 32;
  float *dw[4], *db[4], *q = grads;
  int end = 0;
  for (int l = 0; l < 4; ++l) {
    m.w[l] = (const __nv_bfloat16*)w[l];
    m.cin[l] = NET_CIN[l];
    m.cout[l] = NET_COUT[l];
    m.g[l] = l == 3 ? 16 : 32;
    m.out[l] = wm + end;
    m.end[l] = end += 27 * m.cin[l] * m.g[l];
    dw[l] = q;
    q += 27 * NET_CIN[l] * NET_COUT[l];
  }
  for (int l = 0; l < 4; ++l) {
    db[l] = q;
    q += NET_COUT[l];
  }
  cudaError_t e = cudaMemsetAsync(grads, 0, (size_t)(q - grads) * sizeof(float), st);
  if (e == cudaSuccess) {
    k_mirror<<<(end + 255) / 256, 256, 0, st>>>(m);
    k_pad5<<<pad_blocks(n), 256, 0, st>>>(n, gout, (uint4*)g[0], db[3]);
    e = cudaGetLastError();
  }
  for (int l = 3; l >= 0 && e == cudaSuccess; --l) {
    const __nv_bfloat16* in = g[(3 - l) & 1];
    e = weight_grad(nx, ny, nz, NET_CIN[l], NET_COUT[l], m.g[l], act[l], in, dw[l], st);
    if (e != cudaSuccess) break;
    // the input gradient, times GELU' of the layer below, as that layer's output gradient
    ConvEpilogue o;
    o.creal = l ? NET_CIN[l] : NET_REAL;
    o.compact = l == 0;
    if (l) {
      o.gpre = pre[l - 1];
      o.ybf = g[(4 - l) & 1];
      o.db = db[l - 1];
    } else {
      o.yf = dx;
    }
    e = conv3d(nx, ny, nz, m.g[l], NET_CIN[l], in, m.out[l], o, st, true);
  }
  return cnn_status(e, "lexgb_cnn_net_backward");
}

extern "C" int lexgb_cnn_adam(long long n, float* w, const float* gw, float* m, float* v, void* w_bf16, float lr,
                              float beta1, float beta2, float eps, int step, void* stream) {
  using namespace lexgb;
  if (n <= 0 || !w || !gw || !m || !v || step < 1) return cnn_arg("lexgb_cnn_adam: bad argument");
  const float c1 = 1.f - powf(beta1, (float)step), c2 = 1.f - powf(beta2, (float)step);
  k_adam<<<(unsigned)((n + 255) / 256), 256, 0, (cudaStream_t)stream>>>(n, w, gw, m, v, (__nv_bfloat16*)w_bf16, lr,
                                                                       beta1, beta2, eps, c1, c2);
  return cnn_status(cudaGetLastError(), "lexgb_cnn_adam");
}
