// The warm-start network: a per-particle MLP 16 -> 64 -> 64 -> 64 -> 1 with
// SiLU activations, BF16 weights and FP32 accumulation, run on the tcgen05
// tensor cores (operands in shared memory, accumulators in TMEM).
//
// A CTA of 128 threads owns a tile of 128 rows (one row per thread, TMEM
// lane = row), so each layer is one M=128, N=64 MMA chain (K = 16 or 64 in
// steps of 16) followed by an epilogue in which every thread reads its own
// row back from TMEM, adds the bias, applies SiLU and writes the bf16 row
// of the next layer's A tile. The 64 -> 1 output layer is a per-thread dot
// product in FP32.
//
// Training (hand-written backward), one kernel per step and tile of 128 rows:
//   the forward pass keeps the activations and silu' on chip; backward forms
//   dy = 2 (y - t) / B, dz3 = (dy w4) * silu'(z3), and the activation gradients
//   dh2 = dz3 W3, dh1 = dz2 W2 on the tensor cores (A = bf16 dz, B = W^T
//   tiles); weight gradients dW = dz^T h are FP32 sums over the CTA's rows into
//   per-CTA partials. A second kernel adds the partials in a fixed order,
//   applies Adam to the FP32 master weights and repacks them as BF16 tiles.
//
// Every mbarrier wait is bounded; on expiry the kernel raises an error bit,
// stops issuing work and still releases its TMEM.
#include <cuda_bf16.h>

#include "chain.cuh"
#include "tc.cuh"
#include "xpbi_math.cuh"

namespace xpbi {

namespace {

constexpr int kRows = 128;
constexpr int kIn = 16;
constexpr int kHid = 64;
constexpr uint32_t kSpin = 1u << 24;
constexpr int kErrMma = 2;

// Parameter vector (f32 master): W1[64][16] b1[64] W2[64][64] b2 W3[64][64] b3 w4[64] b4
constexpr int oW1 = 0, oB1 = oW1 + kHid * kIn, oW2 = oB1 + kHid, oB2 = oW2 + kHid * kHid, oW3 = oB2 + kHid,
              oB3 = oW3 + kHid * kHid, oW4 = oB3 + kHid, oB4 = oW4 + kHid, kParams = oB4 + 1;
static_assert(kParams == 9473, "parameter count");

// Packed blob (device): bf16 core-layout tiles, then f32 vectors.
constexpr uint32_t bW1 = 0;                          // 64 x 16 bf16  = 2 KB
constexpr uint32_t bW2 = bW1 + kHid * kIn * 2;       // 64 x 64       = 8 KB
constexpr uint32_t bW3 = bW2 + kHid * kHid * 2;      // 64 x 64
constexpr uint32_t bW2T = bW3 + kHid * kHid * 2;     // W2 transposed
constexpr uint32_t bW3T = bW2T + kHid * kHid * 2;    // W3 transposed
constexpr uint32_t bF32 = bW3T + kHid * kHid * 2;    // b1 b2 b3 w4(bf16-rounded) b4 as f32
constexpr uint32_t kBlobBytes = bF32 + (4 * kHid + 4) * 4;
// shared-memory image of the forward kernel: A tile, W1, W2, W3, f32 vectors
constexpr uint32_t sA = 0;                           // 128 x 64 bf16 = 16 KB
constexpr uint32_t sW1 = sA + kRows * kHid * 2;
constexpr uint32_t sW2 = sW1 + kHid * kIn * 2;
constexpr uint32_t sW3 = sW2 + kHid * kHid * 2;
constexpr uint32_t sF32 = sW3 + kHid * kHid * 2;
constexpr uint32_t kFwdSmem = sF32 + (4 * kHid + 4) * 4;

// The sigmoid with the MUFU exponential and reciprocal (a few ulp): training's
// SiLU is z sigm(z), its derivative sigm(z) (1 + z (1 - sigm(z))).
__device__ __forceinline__ float sigm(float z) { return __fdividef(1.f, 1.f + __expf(-z)); }
// SiLU for inference: z sigmoid(z) = h + h tanh(h) with h = z / 2 and the
// MUFU tanh (one special-function op instead of an exponential and a
// reciprocal). Its ~5e-4 relative error lies below the bf16 rounding every
// activation gets; training keeps the exact form its backward pass uses.
__device__ __forceinline__ float tanhMufu(float x) {
  float y;
  asm("tanh.approx.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}
__device__ __forceinline__ float siluFast(float z) {
  const float h = 0.5f * z;
  return fmaf(h, tanhMufu(h), h);
}

// One f32 parameter into the packed blob.
__device__ __forceinline__ void packParam(uint8_t* __restrict__ blob, int q, float v) {
  auto tile = [&](uint32_t base, int r, int k, int K) {
    *reinterpret_cast<__nv_bfloat16*>(blob + base + tc::coreOffset(r, k, K)) = __float2bfloat16_rn(v);
  };
  float* f = reinterpret_cast<float*>(blob + bF32);
  if (q < oB1) {
    tile(bW1, q / kIn, q % kIn, kIn);  // W[out][in]
  } else if (q < oW2) {
    f[q - oB1] = v;
  } else if (q < oB2) {
    const int t = q - oW2;
    tile(bW2, t / kHid, t % kHid, kHid);
    tile(bW2T, t % kHid, t / kHid, kHid);  // row = in, col = out
  } else if (q < oW3) {
    f[kHid + q - oB2] = v;
  } else if (q < oB3) {
    const int t = q - oW3;
    tile(bW3, t / kHid, t % kHid, kHid);
    tile(bW3T, t % kHid, t / kHid, kHid);
  } else if (q < oW4) {
    f[2 * kHid + q - oB3] = v;
  } else if (q < oB4) {
    f[3 * kHid + q - oW4] = __bfloat162float(__float2bfloat16_rn(v));
  } else {
    f[4 * kHid] = v;
  }
}
__global__ void k_mlp_pack(const float* __restrict__ p, uint8_t* __restrict__ blob) {
  const int q = blockIdx.x * blockDim.x + threadIdx.x;
  if (q < kParams) packParam(blob, q, p[q]);
}

// Forward over `rows` feature rows X[rows][16] (f32).
__global__ void __launch_bounds__(kRows) k_mlp_fwd(const float* __restrict__ X, uint32_t rows,
                                                   const uint8_t* __restrict__ blob, float* __restrict__ y_out,
                                                   int* err, int skipZero) {
  extern __shared__ __align__(1024) uint8_t sm[];
  __shared__ __align__(8) uint64_t bar;
  __shared__ uint32_t tbase;
  const int tid = threadIdx.x, warp = tid >> 5;
  // weights -> shared memory (straight copy of the packed tiles)
  {
    const uint4* src = reinterpret_cast<const uint4*>(blob);
    uint4* dst = reinterpret_cast<uint4*>(sm + sW1);
    for (uint32_t q = tid; q < (bW2T - bW1) / 16u; q += kRows) dst[q] = src[q];  // W1, W2, W3
    const float* fs = reinterpret_cast<const float*>(blob + bF32);
    float* fd = reinterpret_cast<float*>(sm + sF32);
    for (uint32_t q = tid; q < 4 * kHid + 1; q += kRows) fd[q] = fs[q];
  }
  if (warp == 0) tc::tmemAlloc(&tbase, 64);
  if (tid == 0) tc::mbarInit(&bar, 1);
  tc::fenceBeforeSync();
  __syncthreads();
  tc::fenceAfterSync();
  const uint32_t tmem = tbase;
  const uint32_t tRow = tmem + ((uint32_t)(warp * 32) << 16);
  const float* F = reinterpret_cast<const float*>(sm + sF32);
  const uint32_t aAddr = tc::smemAddr(sm + sA), w1Addr = tc::smemAddr(sm + sW1), w2Addr = tc::smemAddr(sm + sW2),
                 w3Addr = tc::smemAddr(sm + sW3);
  constexpr uint32_t idesc = tc::idescBf16F32(kRows, kHid);
  uint32_t phase = 0;
  bool ok = true;
  const uint32_t ntiles = (rows + kRows - 1) / kRows;
  for (uint32_t tile = blockIdx.x; tile < ntiles && ok; tile += gridDim.x) {
    const uint32_t row = tile * kRows + tid;
    // ---- layer 1 input: features as bf16, K = 16
    bool active = false;
    {
      float x[kIn];
      if (row < rows) {
        const float4* xr = reinterpret_cast<const float4*>(X + (size_t)row * kIn);
#pragma unroll
        for (int q = 0; q < 4; ++q) {
          const float4 v = __ldg(xr + q);
          x[4 * q] = v.x; x[4 * q + 1] = v.y; x[4 * q + 2] = v.z; x[4 * q + 3] = v.w;
        }
      } else {
#pragma unroll
        for (int q = 0; q < kIn; ++q) x[q] = 0.f;
      }
#pragma unroll
      for (int q = 0; q < kIn; ++q) active |= x[q] != 0.f;
#pragma unroll
      for (int c = 0; c < kIn / 8; ++c) {
        __align__(16) __nv_bfloat16 h[8];
#pragma unroll
        for (int e = 0; e < 8; ++e) h[e] = __float2bfloat16_rn(x[8 * c + e]);
        *reinterpret_cast<uint4*>(sm + sA + tc::coreOffset(tid, 8 * c, kIn)) = *reinterpret_cast<uint4*>(h);
      }
    }
    // the solver's tiles of water particles (all-zero feature rows) need no
    // prediction: their output is defined as 0
    if (skipZero && !__syncthreads_or(active)) {
      if (row < rows) y_out[row] = 0.f;
      continue;
    }
    float y = F[4 * kHid];
    for (int layer = 0; layer < 3 && ok; ++layer) {
      tc::fenceProxyAsync();
      tc::fenceBeforeSync();
      __syncthreads();  // A written by every thread; every warp done with the accumulator
      if (tid == 0) {
        tc::fenceAfterSync();
        const uint32_t K = layer == 0 ? kIn : kHid;
        const uint32_t wAddr = layer == 0 ? w1Addr : (layer == 1 ? w2Addr : w3Addr);
        const uint32_t sbo = (K / 8) * 128;
        for (uint32_t ks = 0; ks < K / 16; ++ks)
          tc::mma(tmem, tc::smemDesc(aAddr + ks * 256, 128, sbo), tc::smemDesc(wAddr + ks * 256, 128, sbo), idesc,
                  ks > 0);
        tc::commit(&bar);
      }
      if (!tc::mbarWait(&bar, phase, kSpin)) {
        if (tid == 0) atomicOr(err, kErrMma);
        ok = false;
      }
      phase ^= 1u;
      tc::fenceAfterSync();
      // epilogue, 16 columns of this thread's row at a time; the MMA that read
      // A has completed, so the next layer's A row is written in place
      const float* bias = F + layer * kHid;
      const float* w4 = F + 3 * kHid;
#pragma unroll 1
      for (int c = 0; c < kHid / 16; ++c) {
        float z[16];
        tc::ld16(tRow + 16 * c, z);
#pragma unroll
        for (int j = 0; j < 16; ++j) z[j] += bias[16 * c + j];
        if (layer < 2) {
#pragma unroll
          for (int h8 = 0; h8 < 2; ++h8) {
            __align__(16) __nv_bfloat16 h[8];
#pragma unroll
            for (int e = 0; e < 8; ++e) h[e] = __float2bfloat16_rn(siluFast(z[8 * h8 + e]));
            *reinterpret_cast<uint4*>(sm + sA + tc::coreOffset(tid, 16 * c + 8 * h8, kHid)) =
                *reinterpret_cast<uint4*>(h);
          }
        } else {
#pragma unroll
          for (int j = 0; j < 16; ++j) y += siluFast(z[j]) * w4[16 * c + j];
        }
      }
    }
    if (ok && row < rows) y_out[row] = y;
  }
  tc::fenceBeforeSync();
  __syncthreads();
  tc::fenceAfterSync();
  if (warp == 0) tc::tmemDealloc(tmem, 64);
}

// One training step's forward and backward over a tile of 128 rows per CTA:
// per-CTA weight-gradient partials and the squared error.
//
// 256 threads: thread (row, half) holds 32 of its row's 64 columns, so a
// warp's lanes are the TMEM lanes of its quadrant. The activations h1, h2 (the
// bf16 values the next layer sees, as f32) and the derivatives silu'(z1),
// silu'(z2) stay in shared memory between the passes, rows padded to 68 floats
// so that 16-byte accesses of a row per lane meet every bank once. The weight
// gradients dW = dz^T h are f32 products (dz is not rounded), 16 outputs per
// thread in packed f32x2. Every sum over rows or CTAs adds its terms in
// order, one after the other: a step rounds weights and activations to bf16,
// so sums in another order, 1e-7 apart, are 1e-4 apart after some 20 steps
// (four partial sums of 32 rows took 2 us less). One CTA per SM; a step is
// bound by the chain of layers and the weight gradients' shared-memory reads.
// (A call of 24 steps of 8192 rows: 0.94 ms against 4.7 with the forward and
// backward kernels it replaces, whose per-thread arrays lived in local
// memory; the same bits.)
constexpr int kStepThreads = 256;
constexpr int kLd = 68;  // row stride of the f32 buffers
constexpr uint32_t tA = 0;                              // A tile, bf16
constexpr uint32_t tW = tA + kRows * kHid * 2;          // W1 W2 W3 W2T W3T as in the blob
constexpr uint32_t tF = tW + bF32;                      // f32 vectors
constexpr uint32_t tH1 = tF + (4 * kHid + 4) * 4;
constexpr uint32_t kBuf = kRows * kLd * 4;
constexpr uint32_t tH2 = tH1 + kBuf, tD1 = tH2 + kBuf, tD2 = tD1 + kBuf, tDZ = tD2 + kBuf;
constexpr uint32_t tRed = tDZ + kBuf;                   // [3][128] f32 scratch
constexpr uint32_t kStepSmem = tRed + 3 * kRows * 4;
static_assert(kStepSmem <= 227 * 1024, "one CTA's shared memory");
static_assert(tH1 % 16 == 0 && bF32 % 16 == 0, "16-byte aligned buffers");
constexpr int kPartStride = (kParams + 31) & ~31;       // floats per CTA's partial

// out[j * kCols + i] = sum over the CTA's rows of dz[r][j] h[r][i] and outB[j] =
// sum of dz[r][j], for h with kCols columns; each sum adds its rows in order
// (rows past the batch hold dz = 0). Bound by shared-memory reads: a warp takes
// 8 outputs j, so that its reads of dz are one address for all lanes (for 16
// columns, one per half), and its lanes the columns, two each (16 columns: one
// column, 4 of the warp's j). (2 x 8 outputs per thread, reading 16-byte groups
// of h, took 9,800 cycles for 64 columns and 6,250 for 16.)
template <int kCols>
__device__ __forceinline__ void wgrad(const float* dz, const float* h, float* __restrict__ out,
                                      float* __restrict__ outB) {
  static_assert(kStepThreads == 256 && kHid == 64 && (kCols == 64 || kCols == 16), "8 warps of 8 outputs j");
  constexpr int kI = kCols == 64 ? 2 : 1;  // columns per lane
  constexpr int kP = kCols == 64 ? 4 : 2;  // pairs of j per lane
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int i0 = kCols == 64 ? 2 * lane : lane & 15, j0 = warp * 8 + (kCols == 64 ? 0 : (lane >> 4) * 4);
  F2 acc[kP][kI], bias[kP];
#pragma unroll
  for (int p = 0; p < kP; ++p) {
    bias[p] = 0ull;
#pragma unroll
    for (int i = 0; i < kI; ++i) acc[p][i] = 0ull;
  }
#pragma unroll 8
  for (int r = 0; r < kRows; ++r) {
    F2 d[kP];
#pragma unroll
    for (int p = 0; p < kP; p += 2) {
      const ulonglong2 v = *reinterpret_cast<const ulonglong2*>(dz + r * kLd + j0 + 2 * p);
      d[p] = v.x;
      d[p + 1] = v.y;
    }
    float x[kI];
    if constexpr (kI == 2) {
      const float2 v = *reinterpret_cast<const float2*>(h + r * kLd + i0);
      x[0] = v.x;
      x[1] = v.y;
    } else {
      x[0] = h[r * kLd + i0];
    }
#pragma unroll
    for (int p = 0; p < kP; ++p) {
      bias[p] = add2(bias[p], d[p]);
#pragma unroll
      for (int i = 0; i < kI; ++i) acc[p][i] = fma2(d[p], f2(x[i], x[i]), acc[p][i]);
    }
  }
#pragma unroll
  for (int p = 0; p < kP; ++p) {
    float* o0 = out + (j0 + 2 * p) * kCols + i0;
    if constexpr (kI == 2) {
      *reinterpret_cast<float2*>(o0) = make_float2(lo2(acc[p][0]), lo2(acc[p][1]));
      *reinterpret_cast<float2*>(o0 + kCols) = make_float2(hi2(acc[p][0]), hi2(acc[p][1]));
    } else {
      o0[0] = lo2(acc[p][0]);
      o0[kCols] = hi2(acc[p][0]);
    }
    if (i0 == 0) {
      outB[j0 + 2 * p] = lo2(bias[p]);
      outB[j0 + 2 * p + 1] = hi2(bias[p]);
    }
  }
}

__global__ void __launch_bounds__(kStepThreads) k_mlp_step(const float* __restrict__ X, const float* __restrict__ T,
                                                           uint32_t rows, const uint8_t* blob,
                                                           float* __restrict__ partial, float* __restrict__ sqerr,
                                                           int* err) {
  extern __shared__ __align__(1024) uint8_t sm[];
  __shared__ __align__(8) uint64_t bar;
  __shared__ uint32_t tbase;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, half = warp >> 2;
  const int r = (warp & 3) * 32 + lane;  // row within the tile
  const int c0 = half * 32;              // first of this thread's columns
  const uint32_t row = blockIdx.x * kRows + r;
  const bool valid = row < rows;
  float* const F = reinterpret_cast<float*>(sm + tF);
  float* const H1 = reinterpret_cast<float*>(sm + tH1);
  float* const H2 = reinterpret_cast<float*>(sm + tH2);
  float* const D1 = reinterpret_cast<float*>(sm + tD1);
  float* const D2 = reinterpret_cast<float*>(sm + tD2);
  float* const DZ = reinterpret_cast<float*>(sm + tDZ);
  float* const red = reinterpret_cast<float*>(sm + tRed);
  float* const P = partial + (size_t)blockIdx.x * kPartStride;
  if (warp == 0) tc::tmemAlloc(&tbase, 64);
  if (tid == 0) tc::mbarInit(&bar, 1);
  // the inputs as bf16, 8 columns per thread
  {
    __align__(16) __nv_bfloat16 x[8];
    float4 a = make_float4(0.f, 0.f, 0.f, 0.f), b = a;
    if (valid) {
      const float4* xr = reinterpret_cast<const float4*>(X + (size_t)row * kIn + 8 * half);
      a = __ldg(xr);
      b = __ldg(xr + 1);
    }
    const float v[8] = {a.x, a.y, a.z, a.w, b.x, b.y, b.z, b.w};
#pragma unroll
    for (int e = 0; e < 8; ++e) x[e] = __float2bfloat16_rn(v[e]);
    *reinterpret_cast<uint4*>(sm + tA + tc::coreOffset(r, 8 * half, kIn)) = *reinterpret_cast<uint4*>(x);
  }
  const float target = valid ? T[row] : 0.f;
  // all of the above, the batch included, does not depend on the preceding
  // step; the weights do
  const uint32_t w0 = afterPrevious((uint32_t)tid);
  {
    const uint4* src = reinterpret_cast<const uint4*>(blob);
    uint4* dst = reinterpret_cast<uint4*>(sm + tW);
    // every load before the first store: one round trip to L2 (a loop took 2.7 us)
    constexpr uint32_t kEach = (bF32 / 16u + kStepThreads - 1u) / kStepThreads;
    uint4 v[kEach];
#pragma unroll
    for (uint32_t k = 0; k < kEach; ++k)
      if (w0 + k * kStepThreads < bF32 / 16u) v[k] = src[w0 + k * kStepThreads];
    const float* fs = reinterpret_cast<const float*>(blob + bF32);
    const float f0 = fs[w0], f1 = fs[4 * kHid];
#pragma unroll
    for (uint32_t k = 0; k < kEach; ++k)
      if (w0 + k * kStepThreads < bF32 / 16u) dst[w0 + k * kStepThreads] = v[k];
    F[w0] = f0;
    if (w0 == 0u) F[4 * kHid] = f1;
  }
  tc::fenceProxyAsync();
  tc::fenceBeforeSync();
  __syncthreads();
  tc::fenceAfterSync();
  const uint32_t tmem = tbase;
  const uint32_t tRow = tmem + ((uint32_t)((warp & 3) * 32) << 16) + (uint32_t)c0;
  const uint32_t aAddr = tc::smemAddr(sm + tA);
  constexpr uint32_t idesc = tc::idescBf16F32(kRows, kHid);
  uint32_t phase = 0;
  bool ok = true;  // this thread's waits have all come back
  // D = A B^T on the tensor cores; every thread has fenced and synchronised
  auto issue = [&](uint32_t wOffset, uint32_t K) {
    if (tid == 0 && ok) {
      const uint32_t wAddr = tc::smemAddr(sm + tW + wOffset), sbo = (K / 8) * 128;
      for (uint32_t ks = 0; ks < K / 16; ++ks)
        tc::mma(tmem, tc::smemDesc(aAddr + ks * 256, 128, sbo), tc::smemDesc(wAddr + ks * 256, 128, sbo), idesc,
                ks > 0);
      tc::commit(&bar);
    }
  };
  // When a wait expires, the error word says so, no further MMA is issued over
  // the one that may still run, and the later waits are not tried; no barrier
  // is skipped, and the CTA goes on to release its TMEM.
  auto await = [&]() {
    if (ok && !tc::mbarWait(&bar, phase, kSpin)) {
      ok = false;
      atomicOr(err, kErrMma);
    }
    phase ^= 1u;
    tc::fenceAfterSync();
  };
  auto ready = [&]() {  // A written, the accumulator read: the next MMA may start
    tc::fenceProxyAsync();
    tc::fenceBeforeSync();
    __syncthreads();
    if (tid == 0) tc::fenceAfterSync();
  };
  auto storeA8 = [&](int c, const float* v) {  // columns c .. c + 7 of this row as bf16
    __align__(16) __nv_bfloat16 h[8];
#pragma unroll
    for (int e = 0; e < 8; ++e) h[e] = __float2bfloat16_rn(v[e]);
    *reinterpret_cast<uint4*>(sm + tA + tc::coreOffset(r, c, kHid)) = *reinterpret_cast<uint4*>(h);
  };
  auto store4 = [&](float* buf, int c, float a, float b, float d, float e) {
    *reinterpret_cast<float4*>(buf + r * kLd + c) = make_float4(a, b, d, e);
  };

  // ---- forward, layers 1 and 2
#pragma unroll 1
  for (int layer = 0; layer < 2; ++layer) {
    issue(layer == 0 ? bW1 : bW2, layer == 0 ? kIn : kHid);
    await();
    float* const H = layer == 0 ? H1 : H2;
    float* const D = layer == 0 ? D1 : D2;
    const float* bias = F + layer * kHid + c0;
#pragma unroll
    for (int c = 0; c < 32; c += 16) {
      float z[16], d[16];
      tc::ld16(tRow + c, z);
#pragma unroll
      for (int e = 0; e < 16; ++e) {
        const float a = z[e] + bias[c + e];
        const float s = sigm(a);
        z[e] = __bfloat162float(__float2bfloat16_rn(a * s));
        d[e] = s * (1.f + a * (1.f - s));
      }
      storeA8(c0 + c, z);
      storeA8(c0 + c + 8, z + 8);
#pragma unroll
      for (int e = 0; e < 16; e += 4) {
        store4(H, c0 + c + e, z[e], z[e + 1], z[e + 2], z[e + 3]);
        store4(D, c0 + c + e, d[e], d[e + 1], d[e + 2], d[e + 3]);
      }
    }
    ready();
  }
  // ---- forward, layer 3 and the output; h3 and silu'(z3) stay in registers
  issue(bW3, kHid);
  await();
  float h3[32], dz[32];
  {
    const float* bias = F + 2 * kHid + c0;
    const float* w4 = F + 3 * kHid + c0;
#pragma unroll
    for (int c = 0; c < 32; c += 16) {
      float z[16];
      tc::ld16(tRow + c, z);
#pragma unroll
      for (int e = 0; e < 16; ++e) {
        const float a = z[e] + bias[c + e];
        const float s = sigm(a);
        h3[c + e] = a * s;
        dz[c + e] = s * (1.f + a * (1.f - s));
      }
    }
    // the output adds its 64 columns in order: the second half continues the
    // first half's sum
    auto output = [&](float y) {
#pragma unroll
      for (int c = 0; c < 32; ++c) y = __fmaf_rn(h3[c], w4[c], y);
      red[r] = y;
    };
    if (half == 0) output(F[4 * kHid]);
    __syncthreads();
    if (half == 1) output(red[r]);
  }
  tc::fenceBeforeSync();
  __syncthreads();
  const float e = red[r] - target;
  const float dy = valid ? 2.f * e / (float)rows : 0.f;
#pragma unroll
  for (int c = 0; c < 32; ++c) dz[c] = dy * F[3 * kHid + c0 + c] * dz[c];
  // gradients of w4 and b4 and the squared error, each over the rows in order
#pragma unroll
  for (int c = 0; c < 32; c += 4) store4(DZ, c0 + c, h3[c], h3[c + 1], h3[c + 2], h3[c + 3]);
  if (half == 0) {
    red[kRows + r] = dy;
    red[2 * kRows + r] = valid ? __fmul_rn(e, e) : 0.f;
  }
  __syncthreads();
  if (tid < kHid) {
    float acc = 0.f;
#pragma unroll 16
    for (int q = 0; q < kRows; ++q) acc = __fmaf_rn(red[kRows + q], DZ[q * kLd + tid], acc);
    P[oW4 + tid] = acc;
  } else if (tid == 64 || tid == 96) {
    const float* v = red + (tid == 64 ? kRows : 2 * kRows);
    float acc = 0.f;
#pragma unroll 16
    for (int q = 0; q < kRows; ++q) acc = __fadd_rn(acc, v[q]);
    if (tid == 64)
      P[oB4] = acc;
    else
      sqerr[blockIdx.x] = acc;
  }
  __syncthreads();  // DZ is free
  // ---- backward, layers 3 and 2: dz -> dW, db; the previous layer's dz
#pragma unroll 1
  for (int layer = 2; layer >= 1; --layer) {
#pragma unroll
    for (int c = 0; c < 32; c += 8) {
      storeA8(c0 + c, dz + c);
      store4(DZ, c0 + c, dz[c], dz[c + 1], dz[c + 2], dz[c + 3]);
      store4(DZ, c0 + c + 4, dz[c + 4], dz[c + 5], dz[c + 6], dz[c + 7]);
    }
    ready();
    issue(layer == 2 ? bW3T : bW2T, kHid);
    wgrad<kHid>(DZ, layer == 2 ? H2 : H1, P + (layer == 2 ? oW3 : oW2), P + (layer == 2 ? oB3 : oB2));
    await();
    const float* D = layer == 2 ? D2 : D1;
#pragma unroll
    for (int c = 0; c < 32; c += 16) {
      float g[16];
      tc::ld16(tRow + c, g);
#pragma unroll
      for (int q = 0; q < 16; q += 4) {
        const float4 d = *reinterpret_cast<const float4*>(D + r * kLd + c0 + c + q);
        dz[c + q] = g[q] * d.x;
        dz[c + q + 1] = g[q + 1] * d.y;
        dz[c + q + 2] = g[q + 2] * d.z;
        dz[c + q + 3] = g[q + 3] * d.w;
      }
    }
    tc::fenceBeforeSync();
    __syncthreads();  // DZ and H are free
  }
  // ---- layer 1: dW1 = dz1^T x (x as bf16, the network's input precision)
#pragma unroll
  for (int c = 0; c < 32; c += 4) store4(DZ, c0 + c, dz[c], dz[c + 1], dz[c + 2], dz[c + 3]);
  {
    float4 a = make_float4(0.f, 0.f, 0.f, 0.f), b = a;
    if (valid) {
      const float4* xr = reinterpret_cast<const float4*>(X + (size_t)row * kIn + 8 * half);
      a = __ldg(xr);
      b = __ldg(xr + 1);
    }
    auto rnd = [](float v) { return __bfloat162float(__float2bfloat16_rn(v)); };
    store4(H1, 8 * half, rnd(a.x), rnd(a.y), rnd(a.z), rnd(a.w));
    store4(H1, 8 * half + 4, rnd(b.x), rnd(b.y), rnd(b.z), rnd(b.w));
  }
  __syncthreads();  // DZ and x are written
  wgrad<kIn>(DZ, H1, P + oW1, P + oB1);
  tc::fenceBeforeSync();
  __syncthreads();
  tc::fenceAfterSync();
  if (warp == 0) tc::tmemDealloc(tmem, 64);
}

// The gradient, grad[p] = sum over CTAs of partial[cta][p] in order, and the
// mean squared error. With w: the Adam update of the parameter and its bf16
// copy in the blob follow in the same thread. A thread per parameter; the
// loads of 32 partials are in flight at once, their additions are a chain.
struct Adam {
  float *w, *m, *v;
  float lr, b1, b2, eps, c1, c2;
};
constexpr int kReduceParams = 64;
__global__ void __launch_bounds__(kReduceParams) k_mlp_reduce(const float* partial, uint32_t nparts,
                                                              const float* sqerr, uint32_t rows,
                                                              float* grad, float* loss,
                                                              Adam A, uint8_t* blob) {
  const uint32_t p = afterPreviousEager(blockIdx.x * kReduceParams + threadIdx.x);
  if (p < (uint32_t)kParams) {
    float gi = 0.f;
#pragma unroll 32
    for (uint32_t c = 0; c < nparts; ++c) gi = __fadd_rn(gi, partial[(size_t)c * kPartStride + p]);
    if (grad) grad[p] = gi;
    if (A.w) {
      const float mi = A.b1 * A.m[p] + (1.f - A.b1) * gi;
      const float vi = A.b2 * A.v[p] + (1.f - A.b2) * gi * gi;
      A.m[p] = mi;
      A.v[p] = vi;
      const float wi = A.w[p] - A.lr * (mi / A.c1) / (sqrtf(vi / A.c2) + A.eps);
      A.w[p] = wi;
      packParam(blob, (int)p, wi);
    }
  }
  if (blockIdx.x == gridDim.x - 1u && threadIdx.x == kReduceParams - 1) {
    float se = 0.f;
#pragma unroll 32
    for (uint32_t c = 0; c < nparts; ++c) se = __fadd_rn(se, sqerr[c]);
    *loss = se / (float)rows;
  }
}

}  // namespace

int mlp_param_count() { return kParams; }
size_t mlp_blob_bytes() { return kBlobBytes; }

size_t mlp_partial_floats(uint32_t rows) { return (size_t)((rows + kRows - 1) / kRows) * kPartStride; }

void mlp_pack(const float* dParams, void* dBlob, cudaStream_t st) {
  k_mlp_pack<<<(kParams + 255) / 256, 256, 0, st>>>(dParams, static_cast<uint8_t*>(dBlob));
}

cudaError_t mlp_forward(const float* dX, uint32_t rows, const void* dBlob, float* dY, int* dErr, cudaStream_t st,
                        bool skipZero) {
  static bool attr = false;
  if (!attr) {
    cudaError_t e = cudaFuncSetAttribute(k_mlp_fwd, cudaFuncAttributeMaxDynamicSharedMemorySize, kFwdSmem);
    if (e != cudaSuccess) return e;
    attr = true;
  }
  if (rows == 0) return cudaSuccess;
  const uint32_t ntiles = (rows + kRows - 1) / kRows;
  // 48 registers and 37 KB of shared memory: six CTAs per SM (384 TMEM columns)
  const uint32_t grid = ntiles < 152u * 6u ? ntiles : 152u * 6u;
  k_mlp_fwd<<<grid, kRows, kFwdSmem, st>>>(dX, rows, static_cast<const uint8_t*>(dBlob), dY, dErr, skipZero ? 1 : 0);
  return cudaGetLastError();
}

namespace {
cudaError_t stepKernel(const float* dX, const float* dT, uint32_t rows, const void* dBlob, float* dPartial, float* dSq,
                       int* dErr, cudaStream_t st) {
  cudaError_t e = cudaFuncSetAttribute(k_mlp_step, cudaFuncAttributeMaxDynamicSharedMemorySize, kStepSmem);
  if (e != cudaSuccess) return e;
  launchChained(k_mlp_step, (rows + kRows - 1) / kRows, kStepThreads, kStepSmem, st, dX, dT, rows,
                static_cast<const uint8_t*>(dBlob), dPartial, dSq, dErr);
  return cudaGetLastError();
}
void reduceKernel(const float* dPartial, const float* dSq, uint32_t rows, float* dGrad, float* dLoss, const Adam& adam,
                  uint8_t* blob, cudaStream_t st) {
  launchChained(k_mlp_reduce, (kParams + kReduceParams - 1) / kReduceParams, kReduceParams, 0, st, dPartial,
                (rows + kRows - 1) / kRows, dSq, rows, dGrad, dLoss, adam, blob);
}
}  // namespace

// The gradient (and mean squared error) on rows X, targets T. Scratch:
// dPartial [mlp_partial_floats(rows)], dSq [ceil(rows / 128)].
cudaError_t mlp_grad(const float* dX, const float* dT, uint32_t rows, const void* dBlob, float* dPartial, float* dSq,
                     float* dGrad, float* dLoss, int* dErr, cudaStream_t st) {
  if (rows == 0) return cudaSuccess;
  cudaError_t e = stepKernel(dX, dT, rows, dBlob, dPartial, dSq, dErr, st);
  if (e != cudaSuccess) return e;
  reduceKernel(dPartial, dSq, rows, dGrad, dLoss, Adam{}, nullptr, st);
  return cudaGetLastError();
}

// One Adam step on the parameters dW (moments dM, dV) and their packed copy.
cudaError_t mlp_train_step(const float* dX, const float* dT, uint32_t rows, float* dW, float* dM, float* dV,
                           void* dBlob, float* dPartial, float* dSq, float* dLoss, float lr, int step, int* dErr,
                           cudaStream_t st) {
  cudaError_t e = stepKernel(dX, dT, rows, dBlob, dPartial, dSq, dErr, st);
  if (e != cudaSuccess) return e;
  const float b1 = 0.9f, b2 = 0.999f;
  const float c1 = 1.f - powf(b1, (float)step), c2 = 1.f - powf(b2, (float)step);
  reduceKernel(dPartial, dSq, rows, nullptr, dLoss, Adam{dW, dM, dV, lr, b1, b2, 1e-8f, c1, c2},
               static_cast<uint8_t*>(dBlob), st);
  return cudaGetLastError();
}

}  // namespace xpbi
