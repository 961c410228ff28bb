// lexgb_cnn.cuh - common includes of the learned SGS correction's CNN kernels.
#pragma once
#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <stdint.h>

#include <string>

#include "../../include/lexgb.h"

namespace lexgb {
// What a convolution does with its sums s (FP32, [npts][cout]): v = s + bias, stored to `pre`; then GELU
// (gelu), or the product with GELU'(gpre) (gpre: FP32 [npts][cout], a backward pass through the
// activation); channels >= creal zero; stored to ybf (BF16 [npts][cout]) and yf (FP32 [npts][cout], or
// with `compact` [npts][creal]); db[c] += the sum over the points of the values stored to ybf.
struct ConvEpilogue {
  const float* bias = nullptr;
  float* pre = nullptr;
  void* ybf = nullptr;
  float* yf = nullptr;
  const float* gpre = nullptr;
  float* db = nullptr;
  int gelu = 0, creal = 0, compact = 0;
};

// d/dx of the tanh GELU
__device__ __forceinline__ float gelu_tanh_grad(float x) {
  const float k0 = 0.7978845608028654f;   // sqrt(2/pi)
  const float u = k0 * (x + 0.044715f * x * x * x);
  const float t = tanhf(u);
  return 0.5f * (1.f + t) + 0.5f * x * (1.f - t * t) * k0 * (1.f + 3.f * 0.044715f * x * x);
}

// State fields the network's input is made of, and its normalisation.
struct PackIn {
  const float *T = nullptr, *u, *v, *w, *q;
  float theta_ref;
  const float *lo, *rin;   // [5][nz+1]
};

// The normalisation of level k: lo and rin of the five fields, of w on its lower and upper face
struct PackNorm {
  float lo[6], rin[6];
  PackNorm() = default;
  __device__ __forceinline__ PackNorm(const PackIn& a, int k, int nz) {
    constexpr int F[6] = {0, 1, 2, 3, 4, 3};
#pragma unroll
    for (int i = 0; i < 6; ++i) {
      lo[i] = __ldg(a.lo + F[i] * (nz + 1) + k + (i == 5));
      rin[i] = __ldg(a.rin + F[i] * (nz + 1) + k + (i == 5));
    }
  }
  __device__ __forceinline__ float operator()(float x, int i) const { return __fdiv_rn(__fsub_rn(x, lo[i]), rin[i]); }
};

// Network input of cell (i, j, k), as dl_models.phys_state_tuple2array makes it (dl_models.py:125-155):
// every field is min-max normalised on its own grid points with per-level constants lo[f][l] and
// rin[f][l] (stride nz+1: w's constants are per face level 0..nz), then the normalised winds are
// averaged to the cell centre (unstagger_uvw; u and v periodic): the first 8 of 16 BF16 channels, 5
// used.  The arithmetic is the element-wise sequence of the PyTorch packing of the same state, rounded
// the same way (no contractions), so both give the same BF16 inputs.
struct PackPoint {
  float T, u0, u1, v0, v1, w0, w1, q;
  __device__ __forceinline__ void load(const PackIn& a, int i, int j, int k, int nx, int ny) {
    const long long plane = (long long)nx * ny, t = plane * k + (long long)j * nx + i;
    T = a.T[t];
    u0 = a.u[t];
    u1 = a.u[t - i + (i + 1 == nx ? 0 : i + 1)];
    v0 = a.v[t];
    v1 = a.v[t + (long long)((j + 1 == ny ? 0 : j + 1) - j) * nx];
    w0 = a.w[t];
    w1 = a.w[t + plane];
    q = a.q[t];
  }
  __device__ __forceinline__ uint4 channels(const PackIn& a, const PackNorm& nrm) const {
    float f[6];
    f[0] = nrm(__fadd_rn(T, a.theta_ref), 0);
    f[1] = __fmul_rn(0.5f, __fadd_rn(nrm(u0, 1), nrm(u1, 1)));
    f[2] = __fmul_rn(0.5f, __fadd_rn(nrm(v0, 2), nrm(v1, 2)));
    f[3] = __fmul_rn(0.5f, __fadd_rn(nrm(w0, 3), nrm(w1, 5)));
    f[4] = nrm(q, 4);
    f[5] = 0.f;
    auto two = [&](int c) {
      return (uint32_t)__bfloat16_as_ushort(__float2bfloat16_rn(f[c])) |
             ((uint32_t)__bfloat16_as_ushort(__float2bfloat16_rn(f[c + 1])) << 16);
    };
    return make_uint4(two(0), two(2), two(4), 0u);
  }
};

// tcgen05 convolution (kernels_cnn_tc.cu): shape rule, launch, one-time set-up, timeout count
bool conv_tc_fits(int nx, int ny, int nz, int cin, int cout, const void* x, const ConvEpilogue& o);
cudaError_t launch_conv_tc(int nx, int ny, int nz, int cin, int cout, const void* x, const void* w,
                           const ConvEpilogue& o, cudaStream_t st, bool pdl);
cudaError_t conv_tc_prepare();
cudaError_t conv_tc_take_timeouts(unsigned int* n);
// tcgen05 weight gradient (kernels_cnn_tc.cu): dw[27][cout][cin] += sum_p g[p][co] x[p+off][ci]
bool conv_dw_tc_fits(int nx, int ny, int nz, int cin, int cout, int gstride, const void* x, const void* g,
                     const float* dw);
cudaError_t launch_conv_dw_tc(int nx, int ny, int nz, int cin, int cout, int gstride, const void* x, const void* g,
                              float* dw, cudaStream_t st);
}  // namespace lexgb
