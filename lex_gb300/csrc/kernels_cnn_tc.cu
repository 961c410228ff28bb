// kernels_cnn_tc.cu - the learned SGS correction's 3x3x3 convolution on the 5th-generation tensor
// cores (tcgen05.mma, accumulators in tensor memory), as an implicit GEMM per tile of points, one
// input plane at a time:
//
//   D[128 points][3 NP] += A[128 points][Cin] (input plane p shifted by (dy, dx))
//                          x B[Cin][3 NP]     (the weights of the taps (dz, dy, dx), dz = -1, 0, +1)
//
// so that one MMA adds plane p's share to the three output levels it feeds (p+1, p, p-1): each
// input tile is read by the tensor cores 9 x Cin/16 times per plane instead of 27 x Cin/16.
// A block owns a column of 8 (x) x 16 (y) points and marches up a chunk of levels, with its
// warps specialised:
//   the producer warp  loads each input plane the chunk needs (10 x 18 points with the one-point
//                      halo, zero outside the grid by the tensor map's out-of-bounds fill) by TMA
//                      (cp.async.bulk.tensor, one box per 8-channel group) into a ring of plane
//                      slots; a slot's full barrier completes on the bytes' arrival;
//   the MMA warp       for plane p issues the 9 x Cin/16 MMAs (M = 128, N = 3 NP, K = 16, BF16
//                      in, FP32 accumulate) into the columns of output levels p+1, p, p-1: the
//                      tensor memory is a ring of Q level slots of NP columns in descending level
//                      order, so the three are adjacent (where they wrap round the ring, the MMA
//                      is split in two; rows of levels outside the chunk are left out of N); it
//                      frees the plane's slot and marks level p-1 summed;
//   the epilogue warps (one per tensor-memory lane quarter and 16 channels) zero the ring first (the windows of
//                      neighbouring planes overlap, so every MMA accumulates), then for each level
//                      wait for it, read their 32 rows (tcgen05.ld), zero the level slot again if
//                      a later level of the chunk uses it, hand it back to the MMA warp and apply
//                      the epilogue (ConvEpilogue).  A lane's tensor-memory row is one point's
//                      channels; stored from there, a store instruction would touch 32 lines with
//                      16 bytes each, so the rows go through shared memory first and each
//                      instruction moves 64 consecutive bytes of FP32 of 8 points.
// What bounds it at 128x128x64 (two blocks per SM, 256 blocks of 32 levels): taken apart by leaving
// one part out of a copy, the epilogue and the MMAs of a plane each took 66 us for 32 -> 32 channels
// when four warps stored whole rows, together 95 us; loads do not matter.  The MMAs (9 Cin/16 of
// 128 x 96 x 16 a plane) are bound by reading A: a core matrix (8 points, 128 bytes) starts off a
// 128-byte boundary for every shift, two shared-memory passes instead of one.  Eight epilogue warps
// of 16 channels: 78 us (82 with the FP32 pre-activation; 120 and 182 with direct 16-byte stores and
// chunks of 5 levels).
// Every wait is bounded: one that gives up counts a timeout in g_tc_timeouts and sets the block's
// abort flag, which ends the other roles' waits; the block then waits (bounded) for the MMAs it
// issued and the copies in flight, frees its tensor memory and returns.
//
// Shared-memory layouts (16-byte pieces; the tensor cores' canonical K-major layout without
// swizzle, core matrix = 8 rows of 16 bytes):
//   weights  Wsm[9][CIN/8][3 NP][8]        (dy dx), input group, row t NP + co of tap (t - 1, dy,
//                                          dx) and output channel co; core matrix = 8 rows x 8
//                                          inputs; K step 3 NP x 16 B (LBO), next 8 rows 128 B (SBO)
//   planes   Psm[R][CIN/8][18][10][8]      slot, channel group (its box padded to 128-byte
//                                          alignment), row, x; core matrix = 8 consecutive x
//                                          points; K step = the next channel group's box (LBO),
//                                          next row of the tile 160 B (SBO)
#include <cuda.h>
#include <cuda_bf16.h>
#include <stdint.h>

#include "lexgb_cnn.cuh"

namespace lexgb {

__device__ unsigned int g_tc_timeouts = 0;   // bounded waits of k_conv3d_tc that gave up

namespace {

constexpr int TC_TX = 8, TC_TY = 16, TC_HX = TC_TX + 2, TC_HY = TC_TY + 2;
constexpr int TC_THREADS = 192;               // 4 epilogue warps, the producer, the MMA warp
constexpr long long TC_POLLS = 1ll << 24;     // mbarrier polls before a wait gives up
constexpr int TC_BOX_BYTES = TC_HY * TC_HX * 16;                  // one channel group's box: 2880
constexpr int TC_GROUP_BYTES = (TC_BOX_BYTES + 127) / 128 * 128;  // padded to 128 bytes: 2944

template <int CIN, int COUT>
struct TcLayout {
  static constexpr int NP = COUT < 16 ? 16 : COUT;  // output channels of one level in N (16 or 32)
  static constexpr int N3 = 3 * NP;                 // N of the MMA: output levels p+1, p, p-1
  static constexpr int CG = CIN / 8;                // channel groups of 8 (16 bytes)
  static constexpr int R = CIN * COUT == 1024 ? 3 : 4;   // plane slots (each plane is read once; two blocks per SM)
  static constexpr int TMEM_COLS = 256;             // two blocks per SM
  static constexpr int Q = TMEM_COLS / NP;          // level slots of NP columns (8 or 16)
  static constexpr int W_BYTES = 9 * CG * N3 * 16;
  static constexpr int PLANE_BYTES = CG * TC_GROUP_BYTES;
  static constexpr int P_BYTES = R * PLANE_BYTES;
  static constexpr int A_LBO = TC_GROUP_BYTES;      // next channel group
  static constexpr int A_SBO = TC_HX * 16;          // next row of the tile (8 points on)
  static constexpr int B_LBO = N3 * 16;             // next input-channel group
  static constexpr int B_SBO = 128;                 // next 8 rows of N
  static constexpr int HC = COUT < 16 ? COUT : 16;  // output channels of an epilogue warp
  static constexpr int EPI = 4 * (COUT / HC);       // epilogue warps: one per tensor-memory lane quarter and channel part
  static constexpr int THREADS = 32 * (EPI + 2);    // + the producer and the MMA warp
  static constexpr int NBAR = 2 * R + 2 * Q + 1;    // full[R], empty[R], summed[Q], freed[Q], done
  static constexpr int BAR_BYTES = (NBAR * 8 + 16 + 15) / 16 * 16;   // + tensor-memory address, abort flag
  // + alignment slack, barriers, tensor-memory address, abort flag, bias; at least 80 KB, so that
  // no more blocks share an SM than its tensor memory holds
  static constexpr int SR = HC + 4;                 // staged epilogue row (floats): conflict-free 16-byte accesses
  static constexpr int ST_OFF = (W_BYTES + P_BYTES + BAR_BYTES + 2 * NP * 4 + 15) / 16 * 16;   // bias, db sums before it
  static constexpr size_t NEED = 128 + (size_t)ST_OFF + EPI * 32 * SR * 4;
  static constexpr size_t BYTES = NEED < 80 * 1024 ? 80 * 1024 : NEED;
};

__device__ __forceinline__ uint32_t smem_u32(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }

__device__ __forceinline__ void cp16(uint32_t dst, const void* src, bool valid) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst), "l"(src), "r"(valid ? 16 : 0));
}

// canonical K-major, no-swizzle shared-memory matrix descriptor
__device__ __forceinline__ uint64_t smem_desc(uint32_t addr, uint32_t lbo, uint32_t sbo) {
  uint64_t d = (uint64_t)((addr & 0x3FFFFu) >> 4);
  d |= (uint64_t)((lbo >> 4) & 0x3FFFu) << 16;
  d |= (uint64_t)((sbo >> 4) & 0x3FFFu) << 32;
  d |= 1ull << 46;  // descriptor version
  return d;         // base offset 0, swizzle none
}

// instruction descriptor of kind::f16: D FP32, A and B BF16, both K-major, M x N
__host__ __device__ constexpr uint32_t tc_idesc(int m, int n) {
  return (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(n >> 3) << 17) | ((uint32_t)(m >> 4) << 24);
}

__device__ __forceinline__ void mma_bf16_tc(uint32_t tmem_d, uint64_t adesc, uint64_t bdesc, uint32_t idesc,
                                            uint32_t accumulate) {
  asm volatile(
      "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}" ::"r"(tmem_d),
      "l"(adesc), "l"(bdesc), "r"(idesc), "r"(accumulate));
}

// One lane of the (converged) warp.  Inside `if (elect_one())` the compiler knows a single thread runs
// and keeps the MMA descriptors in uniform registers; behind `lane == 0` each MMA moved its descriptors
// there first, 107 cycles an MMA whatever its size.
__device__ __forceinline__ bool elect_one() {
  uint32_t p;
  asm volatile("{\n\t.reg .pred q;\n\telect.sync _|q, 0xffffffff;\n\tselp.u32 %0, 1, 0, q;\n\t}" : "=r"(p));
  return p != 0;
}

__device__ __forceinline__ void mbar_init(uint32_t bar, uint32_t count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(bar), "r"(count) : "memory");
}
__device__ __forceinline__ void mbar_arrive(uint32_t bar) {
  asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(bar) : "memory");
}
__device__ __forceinline__ void mbar_expect_tx(uint32_t bar, uint32_t bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(bytes) : "memory");
}
__device__ __forceinline__ void mma_commit(uint32_t bar) {
  asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(bar) : "memory");
}

// Bounded wait for phase `parity` of an mbarrier; gives up early when the block's abort flag is set.
__device__ __forceinline__ bool mbar_wait(uint32_t bar, uint32_t parity, const volatile int* abort) {
  for (long long i = 0; i < TC_POLLS; ++i) {
    uint32_t done;
    asm volatile(
        "{\n\t.reg .pred p;\n\tmbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(done)
        : "r"(bar), "r"(parity)
        : "memory");
    if (done) return true;
    if ((i & 1023) == 1023 && *abort) return false;
  }
  return false;
}

// Bounded wait with a back-off between polls (about a second at most), for the warps that wait out
// the whole of a block's work; gives up early when the block's abort flag is set (if checked).
__device__ __forceinline__ bool mbar_wait_long(uint32_t bar, uint32_t parity, const volatile int* abort) {
  for (long long i = 0; i < (1ll << 22); ++i) {
    uint32_t done;
    asm volatile(
        "{\n\t.reg .pred p;\n\tmbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(done)
        : "r"(bar), "r"(parity)
        : "memory");
    if (done) return true;
    if (abort && *abort) return false;
    __nanosleep(256);
  }
  return false;
}

// a 4-D box (channel, x, y, z) of a tensor map into shared memory, completing on an mbarrier
__device__ __forceinline__ void tma_load_4d(uint32_t dst, const CUtensorMap* map, int c, int x, int y, int z,
                                            uint32_t bar) {
  asm volatile(
      "cp.async.bulk.tensor.4d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3, %4, "
      "%5}], [%6];" ::"r"(dst),
      "l"(reinterpret_cast<unsigned long long>(map)), "r"(c), "r"(x), "r"(y), "r"(z), "r"(bar)
      : "memory");
}

__device__ __forceinline__ float gelu_fast(float x) {
  const float k0 = 0.7978845608028654f;  // sqrt(2/pi)
  float t;
  asm("tanh.approx.f32 %0, %1;" : "=f"(t) : "f"(k0 * (x + 0.044715f * x * x * x)));
  return 0.5f * x * (1.f + t);
}

__device__ __forceinline__ void tmem_load16(uint32_t taddr, float* v) {
  uint32_t r[16];
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
        "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
      : "r"(taddr));
#pragma unroll
  for (int i = 0; i < 16; ++i) v[i] = __uint_as_float(r[i]);
}


__device__ __forceinline__ void tmem_zero16(uint32_t taddr) {
  const uint32_t z = 0;
  asm volatile(
      "tcgen05.st.sync.aligned.32x32b.x16.b32 [%0], {%1,%1,%1,%1,%1,%1,%1,%1,%1,%1,%1,%1,%1,%1,%1,%1};" ::"r"(taddr),
      "r"(z)
      : "memory");
}
__device__ __forceinline__ void tmem_zero8(uint32_t taddr) {
  const uint32_t z = 0;
  asm volatile("tcgen05.st.sync.aligned.32x32b.x8.b32 [%0], {%1,%1,%1,%1,%1,%1,%1,%1};" ::"r"(taddr), "r"(z)
               : "memory");
}
__device__ __forceinline__ void tmem_load8(uint32_t taddr, float* v) {
  uint32_t r[8];
  asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7])
               : "r"(taddr));
#pragma unroll
  for (int i = 0; i < 8; ++i) v[i] = __uint_as_float(r[i]);
}
// CW consecutive columns of this warp's lanes: load / zero
template <int CW>
__device__ __forceinline__ void tmem_load_cols(uint32_t taddr, float* v) {
#pragma unroll
  for (int c = 0; c < CW; c += 16) {
    if (CW - c >= 16) tmem_load16(taddr + (uint32_t)c, v + c);
    else tmem_load8(taddr + (uint32_t)c, v + c);
  }
}
template <int CW>
__device__ __forceinline__ void tmem_zero_cols(uint32_t taddr) {
#pragma unroll
  for (int c = 0; c < CW; c += 16) {
    if (CW - c >= 16) tmem_zero16(taddr + (uint32_t)c);
    else tmem_zero8(taddr + (uint32_t)c);
  }
}

// Shared memory of a block's tile (addresses in the shared window where the tensor cores or TMA use them)
struct TcSmem {
  uint32_t w, p, bar;     // the layer's weights, plane slots, barriers
  volatile int* abort;
  float *bias, *db;       // NP floats each: the layer's biases, the block's sums for ConvEpilogue::db
  float* stage;           // the epilogue warps' staged rows
};

// Barriers of a tile: full[R], empty[R], summed[Q] (a level slot's sums are complete), freed[Q] (read,
// and zeroed if reused), done
template <class L>
__device__ __forceinline__ void tc_barriers(uint32_t bar, int lane) {   // a warp
  for (int b = lane; b < L::NBAR; b += 32)
    mbar_init(bar + 8u * b, b >= 2 * L::R + L::Q && b < 2 * L::R + 2 * L::Q ? L::EPI : 1);
  asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
}

// weights Wsm[dy dx][cg][n][8] from w[tap][COUT][CIN]: row n = t NP + co holds the tap
// (dz = t - 1, dy, dx) of output channel co (rows co >= COUT zero), so that one MMA on input
// plane p adds to output levels p+1 (t = 0), p (t = 1) and p-1 (t = 2)
template <class L, int CIN, int COUT>
__device__ __forceinline__ void tc_stage_weights(uint32_t dst, const __nv_bfloat16* w, int warp, int lane) {
  // a warp per tap, whose COUT x CIN weights lie together: 512 bytes of them an instruction (one that
  // took a column of 16-byte pieces, as the rows lie in shared memory, spent 5 us on 55 KB)
  constexpr int WARPS = L::THREADS / 32;
  for (int tap = warp; tap < 27; tap += WARPS) {
    const int t = tap / 9, yx = tap - 9 * t;
#pragma unroll
    for (int c0 = 0; c0 < L::NP * L::CG; c0 += 32) {
      const int c = c0 + lane, co = c / L::CG, cg = c % L::CG;
      const bool ok = co < COUT;
      cp16(dst + (uint32_t)(((yx * L::CG + cg) * L::N3 + t * L::NP + co) * 16),
           w + (ok ? tap * COUT * CIN + c * 8 : 0), ok);
    }
  }
}

// epilogue warps: zero this warp's lanes and channels of the level slots in use (the MMA windows of
// neighbouring planes overlap, so they all accumulate)
template <class L>
__device__ __forceinline__ void tc_zero(uint32_t tmem, int warp, int levels) {
  if (warp >= L::EPI) return;
  const uint32_t at = tmem + ((uint32_t)(32 * (warp & 3)) << 16) + (uint32_t)((warp >> 2) * 16);
  for (int q = L::Q - min(levels, L::Q); q < L::Q; ++q) tmem_zero_cols<16>(at + (uint32_t)(q * L::NP));
  asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
}

// One tile of 8 x 16 points and the levels z0 .. z1-1: the roles of the block's warps, from
// initialised barriers, staged weights and zeroed level slots.
template <class L, int CIN, int COUT>
__device__ __forceinline__ void tc_tile(const CUtensorMap& xmap, int nx, int ny, int x0, int y0, int z0, int z1,
                                        const TcSmem& m, uint32_t tmem, const ConvEpilogue& o) {
  constexpr int NP = L::NP, N3 = L::N3, CG = L::CG, R = L::R, Q = L::Q, EPI = L::EPI;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  volatile int* const abort = m.abort;
  auto full = [&](int s) { return m.bar + 8u * s; };
  auto empty = [&](int s) { return m.bar + 8u * (R + s); };
  auto summed = [&](int q) { return m.bar + 8u * (2 * R + q); };
  auto freed = [&](int q) { return m.bar + 8u * (2 * R + Q + q); };
  const uint32_t done = m.bar + 8u * (2 * R + 2 * Q);
  // epilogue warp w: lanes 32 (w % 4) .., columns part .. part + CW - 1 of every level
  constexpr int CW = 16;
  const uint32_t lanes = (uint32_t)(32 * (warp & 3)) << 16;
  const int part = (warp >> 2) * CW;
  const int p0 = z0 - 1;   // first plane of the chunk; plane p uses slot (p - p0) % R, fill (p - p0) / R
  // Output level z of the chunk lives in level slot Q - 1 - (z - z0) mod Q, its (z - z0) / Q-th use:
  // the slots of levels p+1, p, p-1 follow one another except where they wrap round
  auto lslot = [&](int z) { return Q - 1 - (z - z0) % Q; };
  auto luse = [&](int z) { return (z - z0) / Q; };

  if (warp == EPI) {
    // ---------------- producer: planes z0-1 .. z1 ----------------
    if (elect_one()) {
      int p = p0;
      for (; p <= z1; ++p) {
        const int s = (p - p0) % R, k = (p - p0) / R;
        if (k > 0 && !mbar_wait(empty(s), (k - 1) & 1, abort)) {
          atomicAdd(&g_tc_timeouts, 1u);
          *abort = 1;
          break;
        }
        mbar_expect_tx(full(s), CG * TC_BOX_BYTES);
        for (int cg = 0; cg < CG; ++cg)
          tma_load_4d(m.p + s * L::PLANE_BYTES + cg * TC_GROUP_BYTES, &xmap, cg * 8, x0 - 1, y0 - 1, p, full(s));
      }
      // the copies this thread issued have landed before the block's memory goes (bounded)
      for (int q = p - 1; q >= p0 && q >= p - R; --q) mbar_wait_long(full((q - p0) % R), ((q - p0) / R) & 1, nullptr);
    }
  } else if (warp == EPI + 1) {
    // ---------------- MMA issuer: one plane at a time ----------------
    if (elect_one()) {
      // descriptors: the start address is the low field (16-byte units), so an operand at a fixed
      // offset from a base is the base's descriptor plus the offset / 16
      const uint64_t b0 = smem_desc(m.w, L::B_LBO, L::B_SBO);
      bool ok = true;
      int s = 0, k = 0;   // plane slot and fill
      for (int p = p0; p <= z1 && ok; ++p) {
        ok = mbar_wait(full(s), k & 1, abort);
        // level p+1 is new in its slot: the level that used the slot before has been read and zeroed
        if (ok && p + 1 < z1 && luse(p + 1) > 0) ok = mbar_wait(freed(lslot(p + 1)), (luse(p + 1) - 1) & 1, abort);
        if (!ok) {
          atomicAdd(&g_tc_timeouts, 1u);
          *abort = 1;
          break;
        }
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        // the rows t = 0, 1, 2 of N add to levels p+1, p, p-1; those of the chunk are t = ta .. tb-1
        const int ta = max(0, p + 2 - z1), tb = min(3, p + 2 - z0);
        const int q0 = lslot(p + 1 - ta);           // level p+1-ta's slot; the next rows' slots follow
        const int n1 = min(tb - ta, Q - q0);        // rows before the window wraps to column 0
        const int n2 = tb - ta - n1;
        const uint32_t c_hi = tmem + (uint32_t)(q0 * NP), c_lo = tmem;
        const uint32_t id1 = tc_idesc(128, n1 * NP), id2 = tc_idesc(128, n2 * NP);
        const uint64_t a0 = smem_desc(m.p + s * L::PLANE_BYTES, L::A_LBO, L::A_SBO);
        const uint64_t b1 = b0 + (uint64_t)((ta * NP * 16) >> 4), b2 = b1 + (uint64_t)((n1 * NP * 16) >> 4);
        auto taps = [&](uint32_t col, uint64_t bd, uint32_t id) {
#pragma unroll
          for (int dy = 0; dy < 3; ++dy)
#pragma unroll
            for (int dx = 0; dx < 3; ++dx)
#pragma unroll
              for (int ks = 0; ks < CIN / 16; ++ks)
                mma_bf16_tc(col, a0 + (uint64_t)((2 * ks * TC_GROUP_BYTES + (dy * TC_HX + dx) * 16) >> 4),
                            bd + (uint64_t)((((dy * 3 + dx) * CG + 2 * ks) * N3 * 16) >> 4), id, 1u);
        };
        taps(c_hi, b1, id1);
        if (n2 > 0) taps(c_lo, b2, id2);
        mma_commit(empty(s));               // plane p is not read again
        if (p > z0) mma_commit(summed(lslot(p - 1)));   // level p-1 has all three of its planes
        if (++s == R) {
          s = 0;
          ++k;
        }
      }
      mma_commit(done);
      mbar_wait_long(done, 0, nullptr);   // the MMAs are complete before the tensor memory goes
    }
  } else if (warp < EPI) {
    // ---------------- epilogue: warps 0 .. EPI-1 ----------------
    // row r of the tile <-> point (x0 + r % 8, y0 + r / 8); stores: pass i of a level takes points
    // i PPP + lane / CPP of the warp's 32, a lane 4 channels from ch
    constexpr int HC = L::HC, CPP = HC / 4, PPP = 32 / CPP;
    const int c4 = 4 * (lane % CPP), ch = part + c4, pl = lane / CPP;
    float* const st = m.stage + warp * 32 * L::SR;
    const float4 b4 = *reinterpret_cast<const float4*>(m.bias + ch);
    float4 sum = make_float4(0.f, 0.f, 0.f, 0.f);
    // the lane's point of pass i is at + i step (PPP points are PPP / 8 rows of the tile)
    const int r0 = 32 * (warp & 3) + pl;
    const long long at0 = (long long)(y0 + r0 / TC_TX) * nx + x0 + r0 % TC_TX, step = (long long)(PPP / TC_TX) * nx;
    const bool masked = ch + 3 >= o.creal;
    for (int z = z0; z < z1; ++z) {
      const int q = lslot(z);
      const long long at = (long long)z * ny * nx + at0;
      float4 gp[CPP];
      if (o.gpre) {   // in flight while the level is summed
#pragma unroll
        for (int i = 0; i < CPP; ++i)
          gp[i] = __ldg(reinterpret_cast<const float4*>(o.gpre + (at + i * step) * COUT + ch));
      }
      if (!__all_sync(0xffffffffu, mbar_wait(summed(q), luse(z) & 1, abort))) {   // warp-uniform
        if (lane == 0) {
          atomicAdd(&g_tc_timeouts, 1u);
          *abort = 1;
        }
        break;
      }
      asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
      float v[CW];
      const uint32_t cols = tmem + lanes + (uint32_t)(q * NP + part);
      tmem_load_cols<CW>(cols, v);
      asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
      if (z + Q < z1) {   // the slot's next level is in this chunk: zero it for that level
        tmem_zero_cols<CW>(cols);
        asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
      }
      asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
      __syncwarp();
      if (lane == 0) mbar_arrive(freed(q));
#pragma unroll
      for (int c = 0; c < HC; c += 4)
        *reinterpret_cast<float4*>(st + lane * L::SR + c) = make_float4(v[c], v[c + 1], v[c + 2], v[c + 3]);
      __syncwarp();
      float4 a[CPP];
#pragma unroll
      for (int i = 0; i < CPP; ++i) {
        a[i] = *reinterpret_cast<const float4*>(st + (i * PPP + pl) * L::SR + c4);
        a[i] = make_float4(a[i].x + b4.x, a[i].y + b4.y, a[i].z + b4.z, a[i].w + b4.w);
      }
      __syncwarp();   // the staged rows are read before the next level's replace them
      if (o.pre) {
#pragma unroll
        for (int i = 0; i < CPP; ++i) *reinterpret_cast<float4*>(o.pre + (at + i * step) * COUT + ch) = a[i];
      }
      if (o.gelu) {
#pragma unroll
        for (int i = 0; i < CPP; ++i)
          a[i] = make_float4(gelu_fast(a[i].x), gelu_fast(a[i].y), gelu_fast(a[i].z), gelu_fast(a[i].w));
      }
      if (o.gpre) {
#pragma unroll
        for (int i = 0; i < CPP; ++i)
          a[i] = make_float4(a[i].x * gelu_tanh_grad(gp[i].x), a[i].y * gelu_tanh_grad(gp[i].y),
                             a[i].z * gelu_tanh_grad(gp[i].z), a[i].w * gelu_tanh_grad(gp[i].w));
      }
      if (masked) {
#pragma unroll
        for (int i = 0; i < CPP; ++i) {
          if (ch >= o.creal) a[i].x = 0.f;
          if (ch + 1 >= o.creal) a[i].y = 0.f;
          if (ch + 2 >= o.creal) a[i].z = 0.f;
          a[i].w = 0.f;
        }
      }
      if (o.ybf) {
        __nv_bfloat16* const y = reinterpret_cast<__nv_bfloat16*>(o.ybf) + at * COUT + ch;
#pragma unroll
        for (int i = 0; i < CPP; ++i) {
          const __nv_bfloat162 lo = __floats2bfloat162_rn(a[i].x, a[i].y), hi = __floats2bfloat162_rn(a[i].z, a[i].w);
          uint2 qq;
          qq.x = *reinterpret_cast<const uint32_t*>(&lo);
          qq.y = *reinterpret_cast<const uint32_t*>(&hi);
          *reinterpret_cast<uint2*>(y + i * step * COUT) = qq;
          const float2 l = __bfloat1622float2(lo), h = __bfloat1622float2(hi);
          sum = make_float4(sum.x + l.x, sum.y + l.y, sum.z + h.x, sum.w + h.y);
        }
      }
      if (o.yf && !o.compact) {
#pragma unroll
        for (int i = 0; i < CPP; ++i) *reinterpret_cast<float4*>(o.yf + (at + i * step) * COUT + ch) = a[i];
      } else if (o.yf) {
#pragma unroll
        for (int i = 0; i < CPP; ++i) {
          float* const y = o.yf + (at + i * step) * o.creal + ch;
          if (ch < o.creal) y[0] = a[i].x;
          if (ch + 1 < o.creal) y[1] = a[i].y;
          if (ch + 2 < o.creal) y[2] = a[i].z;
          if (ch + 3 < o.creal) y[3] = a[i].w;
        }
      }
    }
    if (o.db) {   // lanes with the same channels, then the block's warps
#pragma unroll
      for (int m = CPP; m < 32; m *= 2) {
        sum.x += __shfl_xor_sync(0xffffffffu, sum.x, m);
        sum.y += __shfl_xor_sync(0xffffffffu, sum.y, m);
        sum.z += __shfl_xor_sync(0xffffffffu, sum.z, m);
        sum.w += __shfl_xor_sync(0xffffffffu, sum.w, m);
      }
      if (lane < CPP) {
        atomicAdd(m.db + ch, sum.x);
        atomicAdd(m.db + ch + 1, sum.y);
        atomicAdd(m.db + ch + 2, sum.z);
        atomicAdd(m.db + ch + 3, sum.w);
      }
    }
  }
}

template <int CIN, int COUT>
__global__ void __launch_bounds__(TcLayout<CIN, COUT>::THREADS, 2)
    k_conv3d_tc(const __grid_constant__ CUtensorMap xmap, int nx, int ny, int nz, int zc,
                const __nv_bfloat16* __restrict__ w, const ConvEpilogue o, int early_weights) {
  using L = TcLayout<CIN, COUT>;
  extern __shared__ unsigned char tc_raw[];
  const uint32_t raw_s = smem_u32(tc_raw);
  unsigned char* smem = tc_raw + ((128u - (raw_s & 127u)) & 127u);   // 128-byte aligned for TMA
  TcSmem m;
  m.w = smem_u32(smem);
  m.p = m.w + L::W_BYTES;
  m.bar = m.p + L::P_BYTES;
  uint32_t* tslot = reinterpret_cast<uint32_t*>(smem + L::W_BYTES + L::P_BYTES + L::NBAR * 8);
  m.abort = reinterpret_cast<volatile int*>(tslot + 1);
  m.bias = reinterpret_cast<float*>(smem + L::W_BYTES + L::P_BYTES + L::BAR_BYTES);
  m.db = m.bias + L::NP;
  m.stage = reinterpret_cast<float*>(smem + L::ST_OFF);
  const int tid = threadIdx.x, warp = tid >> 5;

  // the weights' copies leave first: they, the tensor memory and the barriers are the whole of a small
  // launch's start
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
  if (!early_weights) asm volatile("griddepcontrol.wait;" ::: "memory");
  tc_stage_weights<L, CIN, COUT>(m.w, w, warp, tid & 31);
  if (warp == L::EPI + 1) {  // tensor memory: Q level slots of NP columns
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tslot)),
                 "r"(L::TMEM_COLS)
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  if (warp == 1) {
    if ((tid & 31) == 0) *m.abort = 0;
    tc_barriers<L>(m.bar, tid & 31);
  }
  if (tid < L::NP) {   // the bias lands with the weights
    if (o.bias && tid < COUT)
      asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(smem_u32(m.bias + tid)), "l"(o.bias + tid) : "memory");
    else
      m.bias[tid] = 0.f;
    m.db[tid] = 0.f;
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  const uint32_t tmem = *tslot;
  tc_zero<L>(tmem, warp, zc);
  asm volatile("cp.async.wait_all;" ::: "memory");
  asm volatile("fence.proxy.async.shared::cta;" ::: "memory");   // weights -> the tensor cores
  const int tiles_x = nx / TC_TX, tiles_y = ny / TC_TY;
  const int tx = blockIdx.x % tiles_x, ty = (blockIdx.x / tiles_x) % tiles_y, ch = blockIdx.x / (tiles_x * tiles_y);
  const int x0 = tx * TC_TX, y0 = ty * TC_TY, z0 = ch * zc, z1 = min(z0 + zc, nz);
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  // the threads that read the previous kernel's output or write over what it read (all but the MMA
  // warp's) wait for it themselves: the first plane's copy leaves as soon as it can
  if (early_weights && warp != L::EPI + 1) asm volatile("griddepcontrol.wait;" ::: "memory");
  tc_tile<L, CIN, COUT>(xmap, nx, ny, x0, y0, z0, z1, m, tmem, o);

  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  if (o.db && tid < COUT) atomicAdd(o.db + tid, m.db[tid]);
  if (warp == L::EPI + 1) {
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(L::TMEM_COLS) : "memory");
  }
}

// ---------------------------------------------------------------------------------------------
// Weight gradient on the tensor cores:
//
//   dW[tap][co][ci] += sum over points p of g[p][co] x[p + off(tap)][ci]
//
// as D[M][N] += A[M][K] B[K][N] with K = the 128 points of an 8 (x) x 16 (y) tile at one level,
// N = the gradient's channels co (16 or 32) at up to three levels and M = 128 rows (dy shift s, input
// channel ci): the rows of A are the input plane read 16 / CG (4 or 8) rows apart, so one MMA covers the
// y offsets -1, 0, +1 (and spare shifts whose rows are dropped), and with the gradient planes below, at and
// above the input plane side by side in B the three z offsets too.  A costs the same however wide N is (its
// reads from shared memory, about 60 cycles an MMA): with one MMA for each (dz, dx) a level took 72 of
// them, and 32 -> 32 channels on 128x128x64 127 us; with 24, 66 us (62 in longer chains, launch_dw).  Each of the nine (dx, dz) pairs has
// its own accumulator in tensor memory; a block keeps them over all the (tile, level chunk) items
// it takes and adds them to dW once, at the end.  Both operands are MN-major (the channels are
// the contiguous 16 bytes of a core matrix; its 8 rows are 8 consecutive points along x):
//   x planes  Xsm[R][HY][CG][10][8]  halo rows y0-1 .. y0+14+SH, all channel groups of a row
//                                  together (a 5-D tensor map with the channel group as its own
//                                  dimension), so the next M block (next channel group, or the
//                                  next row after the last group) is 160 bytes on (SBO) and the
//                                  next K block (the next row of the tile) one halo row on (LBO)
//   gradient  Gsm[R+2][NP/8][16][8][8]  next N block = next channel group, then the next plane, 2048
//                                  bytes (SBO); next K block = next row, 128 bytes (LBO).  Planes R, R+1
//                                  hold planes 0, 1 again, so that three planes in a row are adjacent
//                                  wherever they begin
// Step j of an item takes input plane p = z0 - 1 + j.  Warp 4 loads it (with its halo; zero outside the
// grid) and gradient plane p + 1, where the item has it, into slot j % R; warp 5 issues the 24 MMAs of a
// step (3 dx x 8 pairs of rows) on gradient planes p - 1 .. p + 1; warps 0-3 clear the accumulators, wait
// for the last MMA, read their lane quarter of them and add the rows of the y offsets -1..+1 to dW
// (atomicAdd).
template <int CG, int NP>
struct DwLayout {
  static constexpr int SH = 16 / CG;                        // y shifts in the 128 rows of M
  static constexpr int HY = TC_TY + SH - 1;                 // halo rows of an x plane
  static constexpr int ROW_BYTES = CG * TC_HX * 16;         // one halo row, all channel groups
  static constexpr int X_BYTES = HY * ROW_BYTES;
  static constexpr int X_PAD = (X_BYTES + 127) / 128 * 128;
  static constexpr int G_GROUP = TC_TY * TC_TX * 16;        // one 8-channel group of a gradient tile
  static constexpr int G_BYTES = NP / 8 * G_GROUP;
  static constexpr int R = 6;                               // ring slots
  static constexpr int G_AT = R * X_PAD, BAR_AT = G_AT + (R + 2) * G_BYTES;
  static constexpr int TMEM_COLS = 9 * NP <= 256 ? 256 : 512;
  static constexpr int BAR_BYTES = (2 * R + 1) * 8 + 16;
  // + 4 KB after the barriers: an operand's core matrices, read with the two descriptor strides
  // either way round, stay inside the allocation
  static constexpr size_t NEED = 128 + (size_t)BAR_AT + BAR_BYTES + 4096;
  // at most 512 / TMEM_COLS blocks per SM, so that no block waits for another's tensor memory
  static constexpr size_t FLOOR = TMEM_COLS == 512 ? 120 * 1024 : 80 * 1024;
  static constexpr size_t BYTES = NEED < FLOOR ? FLOOR : NEED;
};

// a 5-D box into shared memory, completing on an mbarrier
__device__ __forceinline__ void tma_load_5d(uint32_t dst, const CUtensorMap* map, int c0, int c1, int c2, int c3,
                                            int c4, uint32_t bar) {
  asm volatile(
      "cp.async.bulk.tensor.5d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3, %4, "
      "%5, %6}], [%7];" ::"r"(dst),
      "l"(reinterpret_cast<unsigned long long>(map)), "r"(c0), "r"(c1), "r"(c2), "r"(c3), "r"(c4), "r"(bar)
      : "memory");
}

template <int CG, int NP>
__global__ void __launch_bounds__(TC_THREADS, 1)
    k_conv3d_dw_tc(const __grid_constant__ CUtensorMap xmap, const __grid_constant__ CUtensorMap gmap, int nx,
                   int ny, int nz, int zc, int cin, int cout, float* __restrict__ dw) {
  using L = DwLayout<CG, NP>;
  constexpr int R = L::R;
  extern __shared__ unsigned char tc_raw[];
  const uint32_t raw_s = smem_u32(tc_raw);
  unsigned char* smem = tc_raw + ((128u - (raw_s & 127u)) & 127u);
  const uint32_t x_s = smem_u32(smem), g_s = x_s + L::G_AT, bar_s = x_s + L::BAR_AT;
  auto slot = [&](long long j) { return (uint32_t)(j % R); };
  auto full = [&](long long j) { return bar_s + 8u * slot(j); };
  auto empty = [&](long long j) { return bar_s + 8u * (R + slot(j)); };
  const uint32_t done = bar_s + 8u * (2 * R);
  uint32_t* tslot = reinterpret_cast<uint32_t*>(smem + L::BAR_AT + (2 * R + 1) * 8);
  volatile int* abort = reinterpret_cast<volatile int*>(tslot + 1);
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;

  if (warp == 5) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tslot)),
                 "r"(L::TMEM_COLS)
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  if (tid == 0) {
    for (int s = 0; s < R; ++s) {
      mbar_init(full(s), 1);
      mbar_init(empty(s), 1);
    }
    mbar_init(done, 1);
    *abort = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  const uint32_t tmem = *tslot;
  if (warp < 4) {   // warp-aligned lane quarters
    for (int q = 0; q < 9 * NP / 16; ++q) tmem_zero_cols<16>(tmem + ((uint32_t)(32 * warp) << 16) + (uint32_t)(16 * q));
    asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");

  const int tiles_x = (nx + TC_TX - 1) / TC_TX, tiles_y = (ny + TC_TY - 1) / TC_TY;
  const int chunks = (nz + zc - 1) / zc, items = tiles_x * tiles_y * chunks;

  if (warp == 4) {
    // ---------------- producer ----------------
    if (elect_one()) {
      long long j = 0;
      bool ok = true;
      for (int it = blockIdx.x; it < items && ok; it += gridDim.x) {
        const int x0 = (it % tiles_x) * TC_TX, y0 = ((it / tiles_x) % tiles_y) * TC_TY;
        const int z0 = (it / (tiles_x * tiles_y)) * zc, z1 = min(z0 + zc, nz);
        for (int p = z0 - 1; p <= z1; ++p, ++j) {
          // the slot's gradient plane, loaded at step j - R, is last read at step j - R + 2
          const long long m = j - R + 2;
          if (m >= 0 && !mbar_wait(empty(m), (uint32_t)((m / R) & 1), abort)) {
            atomicAdd(&g_tc_timeouts, 1u);
            *abort = 1;
            ok = false;
            break;
          }
          const uint32_t q = slot(j);
          const int copies = p + 1 < z1 ? (q < 2 ? 2 : 1) : 0;
          mbar_expect_tx(full(j), L::X_BYTES + copies * L::G_BYTES);
          tma_load_5d(x_s + q * L::X_PAD, &xmap, 0, x0 - 1, 0, y0 - 1, p, full(j));
          for (int n = 0; n < copies; ++n)
            for (int cg = 0; cg < NP / 8; ++cg)
              tma_load_4d(g_s + (q + n * R) * L::G_BYTES + cg * L::G_GROUP, &gmap, cg * 8, x0, y0, p + 1, full(j));
        }
      }
      // the copies this thread issued have landed before the block's memory goes (bounded)
      for (long long jj = j - 1; jj >= 0 && jj >= j - R; --jj) mbar_wait_long(full(jj), (uint32_t)((jj / R) & 1), nullptr);
    }
  } else if (warp == 5) {
    // ---------------- MMA issuer ----------------
    if (elect_one()) {
      long long j = 0;
      bool ok = true;
      for (int it = blockIdx.x; it < items && ok; it += gridDim.x) {
        const int z0 = (it / (tiles_x * tiles_y)) * zc, z1 = min(z0 + zc, nz);
        const long long jb = j;
        for (int p = z0 - 1; p <= z1; ++p, ++j) {
          ok = mbar_wait(full(j), (uint32_t)((j / R) & 1), abort);
          if (!ok) {
            atomicAdd(&g_tc_timeouts, 1u);
            *abort = 1;
            break;
          }
          asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
          // gradient planes p - 1 + n, n0 <= n < n1, of the item; plane z was loaded at step jb + z - z0
          const int n0 = max(0, z0 + 1 - p), n1 = min(3, z1 + 1 - p);
          const uint32_t idesc = tc_idesc(128, (n1 - n0) * NP) | (1u << 15) | (1u << 16);   // A and B MN-major
          const uint64_t a0 = smem_desc(x_s + slot(j) * L::X_PAD, L::ROW_BYTES, TC_HX * 16);
          const uint64_t b0 = smem_desc(g_s + slot(jb + (p - 1 + n0 - z0)) * L::G_BYTES, 128, L::G_GROUP);
          const uint32_t col = tmem + (uint32_t)(n0 * NP);
#pragma unroll
          for (int dx = 0; dx < 3; ++dx)
#pragma unroll
            for (int m = 0; m < 8; ++m) {
              const uint64_t ad = a0 + (uint64_t)((2 * m * L::ROW_BYTES + dx * 16) >> 4);
              const uint64_t bd = b0 + (uint64_t)((2 * m * 128) >> 4);
              mma_bf16_tc(col + (uint32_t)(dx * 3 * NP), ad, bd, idesc, 1u);
            }
          mma_commit(empty(j));
        }
      }
      mma_commit(done);
      mbar_wait_long(done, 0, nullptr);   // the MMAs are complete before the tensor memory goes
    }
  } else {
    // ---------------- warps 0-3: the accumulators into dW ----------------
    const bool got = __all_sync(0xffffffffu, mbar_wait_long(done, 0, abort));
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    const int r = 32 * warp + lane, b = r >> 3, s = b / CG, ci = (b % CG) * 8 + (r & 7);
    if (got && !*abort && (4 * warp) / CG <= 2) {   // the warp holds rows of the y offsets -1..+1
      const bool mine = s <= 2 && ci < cin;
#pragma unroll 1
      for (int acc = 0; acc < 9; ++acc) {
        float v[NP];
#pragma unroll
        for (int c = 0; c < NP; c += 16) tmem_load16(tmem + ((uint32_t)(32 * warp) << 16) + (uint32_t)(acc * NP + c), v + c);
        asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
        if (mine) {
          const int tap = (2 - acc % 3) * 9 + s * 3 + acc / 3;   // gradient plane n of a step: dz = 2 - n
          float* d = dw + (long long)tap * cout * cin + ci;
#pragma unroll
          for (int co = 0; co < NP; ++co)
            if (co < cout) atomicAdd(d + (long long)co * cin, v[co]);
        }
      }
    }
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  if (warp == 5) {
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(L::TMEM_COLS) : "memory");
  }
}

constexpr int TC_MAX_DEVICES = 64;

template <int CIN, int COUT>
cudaError_t tc_setup(int* sms) {
  static int count[TC_MAX_DEVICES] = {};
  int dev = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) return e;
  if (dev < 0 || dev >= TC_MAX_DEVICES) return cudaErrorInvalidDevice;
  if (!count[dev]) {
    using L = TcLayout<CIN, COUT>;
    e = cudaFuncSetAttribute(k_conv3d_tc<CIN, COUT>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)L::BYTES);
    if (e != cudaSuccess) return e;
    e = cudaFuncSetAttribute(k_conv3d_tc<CIN, COUT>, cudaFuncAttributePreferredSharedMemoryCarveout,
                             (int)cudaSharedmemCarveoutMaxShared);
    if (e != cudaSuccess) return e;
    int n = 0;
    if ((e = cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev)) != cudaSuccess) return e;
    count[dev] = n;
  }
  *sms = count[dev];
  return cudaSuccess;
}

typedef CUresult (*EncodeTiledFn)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*,
                                  const cuuint64_t*, const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave,
                                  CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

EncodeTiledFn tc_encoder() {
  static EncodeTiledFn fn = nullptr;
  static bool tried = false;
  if (!tried) {
    tried = true;
    void* p = nullptr;
    cudaDriverEntryPointQueryResult q;
    if (cudaGetDriverEntryPointByVersion("cuTensorMapEncodeTiled", &p, 12000, cudaEnableDefault, &q) ==
            cudaSuccess &&
        q == cudaDriverEntryPointSuccess)
      fn = reinterpret_cast<EncodeTiledFn>(p);
    else
      cudaGetLastError();
  }
  return fn;
}

// activations [z][y][x][cin] BF16 as a 4-D tensor (channel, x, y, z); box = one 8-channel group of
// a 10 x 18 plane with halo; out-of-bounds elements read as zero
bool make_xmap(CUtensorMap* map, const void* x, int nx, int ny, int nz, int cin) {
  EncodeTiledFn enc = tc_encoder();
  if (!enc) return false;
  const cuuint64_t dims[4] = {(cuuint64_t)cin, (cuuint64_t)nx, (cuuint64_t)ny, (cuuint64_t)nz};
  const cuuint64_t strides[3] = {(cuuint64_t)cin * 2, (cuuint64_t)nx * cin * 2, (cuuint64_t)ny * nx * cin * 2};
  const cuuint32_t box[4] = {8, TC_HX, TC_HY, 1};
  const cuuint32_t estr[4] = {1, 1, 1, 1};
  return enc(map, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 4, const_cast<void*>(x), dims, strides, box, estr,
             CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
             CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

// Levels per block: a block takes zc + 2 planes (and about one more for its weights and its last
// epilogue), an SM holds two blocks and takes their planes one after another; a lone block leaves
// gaps, about 1.6 times the time, and with 55 KB of weights a block (wbytes) more where blocks on most
// SMs fetch them at once.  (32 -> 32 channels, us: 128x128x64 with 5 levels 125, 10: 103, 32, which this
// picks: 96; 64^3 4: 43, 8, picked: 36, 16: 43; 64x64x32 4, picked: 25, 8: 27; with this kernel forced, a
// corrected step at 32^3 with 2 levels 154.4, 3, picked: 151.9, 4: 155.3.)
int tc_levels(int tiles, int nz, int sms, int wbytes) {
  int zc = nz;
  double best = -1.0;
  for (int nch = 1; nch <= nz; ++nch) {
    const int z = (nz + nch - 1) / nch;
    const long long blocks = (long long)tiles * ((nz + z - 1) / z), per_sm = (blocks + sms - 1) / sms;
    const double alone = wbytes > 32 * 1024 && 3 * blocks > 2 * sms ? 2.0 : 1.6;
    const double cost = (z + 3) * (per_sm == 1 ? alone : (double)per_sm);
    if (best < 0 || cost < best) {
      best = cost;
      zc = z;
    }
  }
  return zc;
}

template <int CIN, int COUT>
cudaError_t launch_tc(int nx, int ny, int nz, const void* x, const __nv_bfloat16* w, const ConvEpilogue& o,
                      cudaStream_t st, bool pdl) {
  int sms = 0;
  cudaError_t e = tc_setup<CIN, COUT>(&sms);
  if (e != cudaSuccess) return e;
  CUtensorMap xmap;
  if (!make_xmap(&xmap, x, nx, ny, nz, CIN)) return cudaErrorInvalidValue;
  using L = TcLayout<CIN, COUT>;
  const int tiles = (nx / TC_TX) * (ny / TC_TY), zc = tc_levels(tiles, nz, sms, L::W_BYTES);
  if ((long long)tiles * ((nz + zc - 1) / zc) > 0x7fffffffll) return cudaErrorInvalidValue;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)(tiles * ((nz + zc - 1) / zc)));
  cfg.blockDim = dim3(L::THREADS);
  cfg.dynamicSmemBytes = L::BYTES;
  cfg.stream = st;
  cudaLaunchAttribute at[1];
  at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = at;
  cfg.numAttrs = pdl ? 1 : 0;
  return cudaLaunchKernelEx(&cfg, k_conv3d_tc<CIN, COUT>, xmap, nx, ny, nz, zc, w, o, pdl ? 1 : 0);
}


// activations [z][y][x][cin] BF16 as a 5-D tensor (8 channels, x, channel group, y, z): a box is a
// plane tile of 10 x hy points with all cin / 8 groups of each row side by side
bool make_dw_xmap(CUtensorMap* map, const void* x, int nx, int ny, int nz, int cin, int hy) {
  EncodeTiledFn enc = tc_encoder();
  if (!enc) return false;
  const cuuint64_t dims[5] = {8, (cuuint64_t)nx, (cuuint64_t)(cin / 8), (cuuint64_t)ny, (cuuint64_t)nz};
  const cuuint64_t strides[4] = {(cuuint64_t)cin * 2, 16, (cuuint64_t)nx * cin * 2, (cuuint64_t)ny * nx * cin * 2};
  const cuuint32_t box[5] = {8, TC_HX, (cuuint32_t)(cin / 8), (cuuint32_t)hy, 1};
  const cuuint32_t estr[5] = {1, 1, 1, 1, 1};
  return enc(map, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 5, const_cast<void*>(x), dims, strides, box, estr,
             CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
             CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

// gradient [z][y][x][c] BF16 as a 4-D tensor (channel, x, y, z); box = one 8-channel group of an
// 8 x 16 tile
bool make_dw_gmap(CUtensorMap* map, const void* g, int nx, int ny, int nz, int c) {
  EncodeTiledFn enc = tc_encoder();
  if (!enc) return false;
  const cuuint64_t dims[4] = {(cuuint64_t)c, (cuuint64_t)nx, (cuuint64_t)ny, (cuuint64_t)nz};
  const cuuint64_t strides[3] = {(cuuint64_t)c * 2, (cuuint64_t)nx * c * 2, (cuuint64_t)ny * nx * c * 2};
  const cuuint32_t box[4] = {8, TC_TX, TC_TY, 1};
  const cuuint32_t estr[4] = {1, 1, 1, 1};
  return enc(map, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 4, const_cast<void*>(g), dims, strides, box, estr,
             CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
             CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

template <int CG, int NP>
cudaError_t dw_grid(int* cap) {
  static int grid_cap[TC_MAX_DEVICES] = {};
  int dev = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) return e;
  if (dev < 0 || dev >= TC_MAX_DEVICES) return cudaErrorInvalidDevice;
  if (!grid_cap[dev]) {
    using L = DwLayout<CG, NP>;
    e = cudaFuncSetAttribute(k_conv3d_dw_tc<CG, NP>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)L::BYTES);
    if (e != cudaSuccess) return e;
    e = cudaFuncSetAttribute(k_conv3d_dw_tc<CG, NP>, cudaFuncAttributePreferredSharedMemoryCarveout,
                             (int)cudaSharedmemCarveoutMaxShared);
    if (e != cudaSuccess) return e;
    int sms = 0, per = 0;
    if ((e = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev)) != cudaSuccess) return e;
    if ((e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per, k_conv3d_dw_tc<CG, NP>, TC_THREADS, L::BYTES)) !=
        cudaSuccess)
      return e;
    per = per < 1 ? 1 : per;
    if (per > 512 / L::TMEM_COLS) per = 512 / L::TMEM_COLS;
    grid_cap[dev] = sms * per;
  }
  *cap = grid_cap[dev];
  return cudaSuccess;
}

template <int CG, int NP>
cudaError_t launch_dw(int nx, int ny, int nz, int cin, int cout, const void* x, const void* g, float* dw,
                      cudaStream_t st) {
  using L = DwLayout<CG, NP>;
  int cap = 0;
  cudaError_t e = dw_grid<CG, NP>(&cap);
  if (e != cudaSuccess) return e;
  CUtensorMap xmap, gmap;
  if (!make_dw_xmap(&xmap, x, nx, ny, nz, cin, L::HY) || !make_dw_gmap(&gmap, g, nx, ny, nz, NP))
    return cudaErrorInvalidValue;
  // level chunks: the count that ends soonest when every block takes ceil(items / blocks) items
  // of chunk + 1 steps (ties: fewer items).  An item takes chunk + 2; counted so, 128x128x64 would be a
  // quicker split by 2 % of a training pass (128 blocks of 64 levels for 152 of 56), but each MMA rounds its
  // accumulator towards zero, and the longer chain is less exact (2.9e-5 of the sum against 2.6e-5).
  const long long tiles = (long long)((nx + TC_TX - 1) / TC_TX) * ((ny + TC_TY - 1) / TC_TY);
  int zc = nz;
  long long best = -1;
  for (int nch = 1; nch <= nz; ++nch) {
    const int z = (nz + nch - 1) / nch;
    const long long items = tiles * ((nz + z - 1) / z), blocks = items < cap ? items : cap;
    const long long cost = (items + blocks - 1) / blocks * (z + 1);
    if (best < 0 || cost < best) {
      best = cost;
      zc = z;
    }
  }
  const long long items = tiles * ((nz + zc - 1) / zc);
  if (items > 0x7fffffffll) return cudaErrorInvalidValue;
  const unsigned blocks = (unsigned)(items < cap ? items : cap);
  k_conv3d_dw_tc<CG, NP><<<blocks, TC_THREADS, L::BYTES, st>>>(xmap, gmap, nx, ny, nz, zc, cin, cout, dw);
  return cudaGetLastError();
}
}  // namespace

bool conv_tc_fits(int nx, int ny, int nz, int cin, int cout, const void* x, const ConvEpilogue& o) {
  const uintptr_t align = (uintptr_t)x | (uintptr_t)o.pre | (uintptr_t)o.ybf | (o.compact ? 0 : (uintptr_t)o.yf) |
                          (uintptr_t)o.gpre;   // 16-byte TMA / loads / stores
  return (cin == 16 || cin == 32) && (cout == 8 || cout == 16 || cout == 32) && nx > 0 && ny > 0 && nz > 0 &&
         nx % TC_TX == 0 && ny % TC_TY == 0 && (align & 15) == 0 && tc_encoder() != nullptr;
}

cudaError_t launch_conv_tc(int nx, int ny, int nz, int cin, int cout, const void* x, const void* w,
                           const ConvEpilogue& o, cudaStream_t st, bool pdl) {
  if (!conv_tc_fits(nx, ny, nz, cin, cout, x, o)) return cudaErrorInvalidValue;
  const __nv_bfloat16* wb = (const __nv_bfloat16*)w;
#define LEXGB_TC(CI, CO) launch_tc<CI, CO>(nx, ny, nz, x, wb, o, st, pdl)
  if (cin == 16) return cout == 8 ? LEXGB_TC(16, 8) : cout == 16 ? LEXGB_TC(16, 16) : LEXGB_TC(16, 32);
  return cout == 8 ? LEXGB_TC(32, 8) : cout == 16 ? LEXGB_TC(32, 16) : LEXGB_TC(32, 32);
#undef LEXGB_TC
}

cudaError_t conv_tc_prepare() {
  int cap;
  cudaError_t e;
  if ((e = tc_setup<16, 8>(&cap)) != cudaSuccess) return e;
  if ((e = tc_setup<16, 16>(&cap)) != cudaSuccess) return e;
  if ((e = tc_setup<16, 32>(&cap)) != cudaSuccess) return e;
  if ((e = tc_setup<32, 8>(&cap)) != cudaSuccess) return e;
  if ((e = tc_setup<32, 16>(&cap)) != cudaSuccess) return e;
  if ((e = tc_setup<32, 32>(&cap)) != cudaSuccess) return e;
  if ((e = dw_grid<2, 16>(&cap)) != cudaSuccess) return e;
  if ((e = dw_grid<2, 32>(&cap)) != cudaSuccess) return e;
  if ((e = dw_grid<4, 16>(&cap)) != cudaSuccess) return e;
  return dw_grid<4, 32>(&cap);
}

bool conv_dw_tc_fits(int nx, int ny, int nz, int cin, int cout, int gstride, const void* x, const void* g,
                     const float* dw) {
  const uintptr_t align = (uintptr_t)x | (uintptr_t)g;   // 16-byte TMA bases
  return (cin == 16 || cin == 32) && (gstride == 16 || gstride == 32) && cout > 0 && cout <= gstride && nx > 0 &&
         ny > 0 && nz > 0 && (align & 15) == 0 && dw && tc_encoder() != nullptr;
}

cudaError_t launch_conv_dw_tc(int nx, int ny, int nz, int cin, int cout, int gstride, const void* x, const void* g,
                              float* dw, cudaStream_t st) {
  if (!conv_dw_tc_fits(nx, ny, nz, cin, cout, gstride, x, g, dw)) return cudaErrorInvalidValue;
  if (cin == 16) return gstride == 16 ? launch_dw<2, 16>(nx, ny, nz, cin, cout, x, g, dw, st)
                                      : launch_dw<2, 32>(nx, ny, nz, cin, cout, x, g, dw, st);
  return gstride == 16 ? launch_dw<4, 16>(nx, ny, nz, cin, cout, x, g, dw, st)
                       : launch_dw<4, 32>(nx, ny, nz, cin, cout, x, g, dw, st);
}

cudaError_t conv_tc_take_timeouts(unsigned int* n) {
  unsigned int zero = 0;
  cudaError_t e = cudaMemcpyFromSymbol(n, g_tc_timeouts, sizeof(unsigned int));
  if (e != cudaSuccess) return e;
  return cudaMemcpyToSymbol(g_tc_timeouts, &zero, sizeof(unsigned int));
}

}  // namespace lexgb
