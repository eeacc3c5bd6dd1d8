// BF16 tensor-core kernels of the learned corrector (tcgen05 MMA, FP32 accumulation in tensor
// memory).  This file holds a general GEMM and the training kernels; the fused per-particle inference
// kernel lives in corrector.cu.
//
// k_tc_gemm: D[M][N] = A[M][K] . B[N][K]^T, bf16 operands row-major in global memory, float32 D.
// A CTA of 128 threads owns a 128-row block of D (all N columns, N <= 256, in one TMEM allocation)
// and a K range; per 64-wide K chunk every thread copies 16-byte vectors of A and B into the K-major
// core-matrix layout of tc.cuh, one thread issues four K = 16 MMAs and commits them to an mbarrier,
// and the CTA waits (bounded) before the next chunk overwrites the tiles.  The epilogue reads the
// accumulator with tcgen05.ld (warp w owns TMEM lanes 32w..32w+31 = rows of D) and stores or, for
// split-K, adds it to D.
#include <cuda_bf16.h>
#include <cuda_runtime.h>

#include <algorithm>

#include "common.cuh"
#include "internal.h"
#include "tc.cuh"

namespace ffmpm {
namespace {

constexpr int kGemmThreads = 128;
constexpr int kKChunk = 64;
constexpr uint32_t kChunkSBO = (kKChunk / 8) * 128;  // 8-row groups of a 64-wide K chunk: 1 KB apart

template <int BN>
__global__ void __launch_bounds__(kGemmThreads) k_tc_gemm(const uint16_t* __restrict__ A, const uint16_t* __restrict__ B,
                                                          float* __restrict__ D, int M, int N, int K, int k_per_split,
                                                          int add_out, int32_t* status) {
  extern __shared__ __align__(1024) unsigned char smem[];
  unsigned char* sa = smem;                   // 128 x 64 bf16
  unsigned char* sb = smem + 128 * kKChunk * 2;  // BN x 64 bf16
  __shared__ uint64_t bar;
  __shared__ uint32_t tmem_base;
  __shared__ int s_fail;
  constexpr uint32_t kCols = BN < 32 ? 32 : BN;
  constexpr uint32_t kIdesc = tc::idesc_bf16_f32(128, BN);
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int m0 = blockIdx.x * 128;
  const int kbeg = blockIdx.y * k_per_split;
  const int kend = min(K, kbeg + k_per_split);
  if (warp == 0) tc::tmem_alloc(&tmem_base, kCols);
  if (tid == 0) {
    mbar_init(&bar, 1);
    fence_barrier_init();
    s_fail = 0;
  }
  tc::fence_before_sync();
  __syncthreads();
  tc::fence_after_sync();
  const uint32_t tmem = tmem_base;
  uint32_t phase = 0;
  bool issued = false;
  for (int k0 = kbeg; k0 < kend; k0 += kKChunk) {
    for (int v = tid; v < 128 * 8; v += kGemmThreads) {
      const int r = v >> 3, c = v & 7;
      const uint4 val = *reinterpret_cast<const uint4*>(A + (size_t)(m0 + r) * K + k0 + 8 * c);
      *reinterpret_cast<uint4*>(sa + tc::kmajor_offset(r, 8 * c, kChunkSBO)) = val;
    }
    for (int v = tid; v < BN * 8; v += kGemmThreads) {
      const int r = v >> 3, c = v & 7;
      uint4 val = make_uint4(0u, 0u, 0u, 0u);
      if (r < N) val = *reinterpret_cast<const uint4*>(B + (size_t)r * K + k0 + 8 * c);
      *reinterpret_cast<uint4*>(sb + tc::kmajor_offset(r, 8 * c, kChunkSBO)) = val;
    }
    fence_proxy_async_shared();  // generic-proxy smem writes -> visible to the tensor core
    tc::fence_before_sync();
    __syncthreads();
    tc::fence_after_sync();
    if (tid == 0) {
      const uint32_t a0 = tc::smem_addr(sa), b0 = tc::smem_addr(sb);
#pragma unroll
      for (int s = 0; s < kKChunk / 16; ++s)
        tc::mma_bf16(tmem, tc::make_desc(a0 + 256u * s, tc::kLBO, kChunkSBO),
                     tc::make_desc(b0 + 256u * s, tc::kLBO, kChunkSBO), kIdesc, issued || s > 0);
      tc::commit(&bar);
    }
    issued = true;
    if (!mbar_wait(&bar, phase)) s_fail = 1;
    phase ^= 1u;
    tc::fence_before_sync();
    __syncthreads();
    tc::fence_after_sync();
    if (s_fail) break;
  }
  if (s_fail) {
    if (tid == 0) {
      if (status) raise_status(status, FFMPM_STATUS_TIMEOUT);
      // the MMAs of the last commit may still be running: wait for them once more (bounded) before
      // their tensor memory is freed
      mbar_wait(&bar, phase ^ 1u);
    }
  } else if (issued) {
    const int row = m0 + 32 * warp + lane;
#pragma unroll 1
    for (int c0 = 0; c0 < BN; c0 += 16) {
      float v[16];
      tc::tmem_ld16(tc::taddr_of(tmem, 32u * warp, c0), v);
      if (row < M) {
#pragma unroll
        for (int j = 0; j < 16; ++j) {
          const int col = c0 + j;
          if (col < N) {
            if (add_out)
              atomicAdd(&D[(size_t)row * N + col], v[j]);
            else
              D[(size_t)row * N + col] = v[j];
          }
        }
      }
    }
  }
  tc::fence_before_sync();
  __syncthreads();
  if (warp == 0) tc::tmem_free(tmem, kCols);
}

template <int BN>
int launch_gemm(const uint16_t* A, const uint16_t* B, float* D, int M, int N, int K, int split, int32_t* status,
                cudaStream_t s) {
  const size_t smem = size_t(128 + BN) * kKChunk * 2;
  if (!allow_smem(reinterpret_cast<const void*>(k_tc_gemm<BN>), smem)) return FFMPM_ERR_CUDA;
  const int chunks = K / kKChunk;
  split = std::max(1, std::min(split, chunks));
  const int per = (chunks + split - 1) / split * kKChunk;
  const int gy = (K + per - 1) / per;
  dim3 grid(M / 128, gy);
  k_tc_gemm<BN><<<grid, kGemmThreads, smem, s>>>(A, B, D, M, N, K, per, gy > 1 ? 1 : 0, status);
  return cudaGetLastError() == cudaSuccess ? FFMPM_OK : FFMPM_ERR_CUDA;
}

// ---------------------------------------------------------------------------------------------
// Training: the activation, its derivative, and the launch shape of the elementwise kernels (Adam, packing).
constexpr int kEw = 256;

__device__ __forceinline__ float gelu_f(float z) { return 0.5f * z * (1.f + erff(z * 0.70710678118654752f)); }
// d/dz GELU(z) = Phi(z) + z phi(z)
__device__ __forceinline__ float gelu_grad(float z) {
  return 0.5f * (1.f + erff(z * 0.70710678118654752f)) + z * 0.3989422804014327f * expf(-0.5f * z * z);
}

// ---------------------------------------------------------------------------------------------
// Forward and backward of the whole network, a tile of 128 rows at a time.  A CTA has 256 threads:
// thread t works on row t & 127 (its TMEM lane) and on one half of a layer's 64 columns (t >> 7).
// 32,768 rows (GB300): 45 + 64 us, and 117 us for a whole training step; a launch for each GEMM and each
// elementwise part, with transposes written a 16-bit word at a time, took 777.  Bound by the chain of a
// tile's layers (an MMA, its commit, the activation), two CTAs (forward) or one (backward) per SM.
constexpr int kTrain = 256;
constexpr uint32_t kSbo64 = (64 / 8) * 128, kSbo128 = (128 / 8) * 128;

// Copy a bf16 row-major [rows][k] matrix (row stride k) into the K-major core-matrix layout.
__device__ __forceinline__ void stage_kmajor(unsigned char* dst, const uint16_t* src, int rows, int k, uint32_t sbo) {
  const int vecs = k / 8;
  for (int v = threadIdx.x; v < rows * vecs; v += blockDim.x) {
    const int r = v / vecs, c = v - r * vecs;
    *reinterpret_cast<uint4*>(dst + tc::kmajor_offset(r, 8 * c, sbo)) =
        *reinterpret_cast<const uint4*>(src + (size_t)r * k + 8 * c);
  }
}

// The transpose of a K-major tile [128 rows][cols] as rows of a bf16 matrix [cols][B]: out[c][r0 + r], two
// rows per 32-bit store, columns from `valid` on as zeros.
__device__ __forceinline__ void store_transposed(const unsigned char* tile, uint32_t sbo, int cols, int valid,
                                                 uint16_t* __restrict__ out, int B, int r0) {
  for (int i = threadIdx.x; i < cols * 64; i += blockDim.x) {
    const int c = i >> 6, r = 2 * (i & 63);
    uint32_t w = 0u;
    if (c < valid)
      w = uint32_t(*reinterpret_cast<const uint16_t*>(tile + tc::kmajor_offset(r, c, sbo))) |
          (uint32_t(*reinterpret_cast<const uint16_t*>(tile + tc::kmajor_offset(r + 1, c, sbo))) << 16);
    *reinterpret_cast<uint32_t*>(out + (size_t)c * B + r0 + r) = w;
  }
}

// D (+)= A . B^T over K = 16 ksteps, both operands K-major tiles.
__device__ __forceinline__ void mma_tile(uint32_t d, const unsigned char* A, uint32_t sboA, const unsigned char* B,
                                         uint32_t sboB, uint32_t idesc, int ksteps, bool accumulate) {
  const uint32_t a0 = tc::smem_addr(A), b0 = tc::smem_addr(B);
  for (int s = 0; s < ksteps; ++s)
    tc::mma_bf16(d, tc::make_desc(a0 + 256u * s, tc::kLBO, sboA), tc::make_desc(b0 + 256u * s, tc::kLBO, sboB), idesc,
                 accumulate || s > 0);
}

// Four floats at p, whole where the caller's arrays are 16-byte aligned (`vec`), else one by one.
__device__ __forceinline__ float4 load4(const float* p, bool vec) {
  return vec ? *reinterpret_cast<const float4*>(p) : make_float4(p[0], p[1], p[2], p[3]);
}
__device__ __forceinline__ void store4(float* p, float4 v, bool vec) {
  if (vec) {
    *reinterpret_cast<float4*>(p) = v;
  } else {
    p[0] = v.x;
    p[1] = v.y;
    p[2] = v.z;
    p[3] = v.w;
  }
}
__device__ __forceinline__ void add4(float* p, float4 v, bool vec) {
  if (vec) {
    atomicAdd(reinterpret_cast<float4*>(p), v);
  } else {
    atomicAdd(p, v.x);
    atomicAdd(p + 1, v.y);
    atomicAdd(p + 2, v.z);
    atomicAdd(p + 3, v.w);
  }
}

struct FwdSmem {
  static constexpr size_t w1 = 0, w2 = w1 + 64 * 128 * 2, w3 = w2 + 64 * 64 * 2, w4 = w3 + 64 * 64 * 2,
                          x = w4 + 16 * 64 * 2, h = x + 128 * 128 * 2, bias = h + 128 * 64 * 2,
                          total = bias + 3 * 64 * 4;
};

// Y = network(X) (before out_scale, without b4).  Keeps Z1..Z3 (with the biases), H1..H3 = gelu(Z) and the
// transposes Ht and Xt, as the ABI documents; the backward pass reads Y, Z and the transposes.  One CTA per 128 rows:
// the layers follow one another in shared and tensor memory (an MMA a layer), so that X is read once and
// everything is written once.
__global__ void __launch_bounds__(kTrain) k_mlp_forward(ffmpm_mlp_trainer t, const uint16_t* __restrict__ X, int B,
                                                        bool vec) {
  extern __shared__ __align__(1024) unsigned char smem[];
  unsigned char *sX = smem + FwdSmem::x, *sH = smem + FwdSmem::h;
  float* sbias = reinterpret_cast<float*>(smem + FwdSmem::bias);
  __shared__ uint64_t bar;
  __shared__ uint32_t tmem_base;
  __shared__ int s_fail;
  const int tid = threadIdx.x, warp = tid >> 5, row = tid & 127, c0 = 32 * (tid >> 7);
  const uint32_t lanes = 32u * (warp & 3);
  const int r0 = blockIdx.x * 128;
  stage_kmajor(sX, X + (size_t)r0 * FFMPM_MLP_IN, 128, FFMPM_MLP_IN, kSbo128);
  stage_kmajor(smem + FwdSmem::w1, t.W1, 64, 128, kSbo128);
  stage_kmajor(smem + FwdSmem::w2, t.W2, 64, 64, kSbo64);
  stage_kmajor(smem + FwdSmem::w3, t.W3, 64, 64, kSbo64);
  stage_kmajor(smem + FwdSmem::w4, t.W4, 16, 64, kSbo64);
  if (tid < 192) sbias[tid] = t.params[FFMPM_MLP_OFF_B1 + tid];  // b1, b2, b3 lie one after another
  if (warp == 0) tc::tmem_alloc(&tmem_base, 128);
  if (tid == 0) {
    mbar_init(&bar, 1);
    fence_barrier_init();
    s_fail = 0;
  }
  fence_proxy_async_shared();
  tc::fence_before_sync();
  __syncthreads();
  tc::fence_after_sync();
  const uint32_t tmem = tmem_base;
  uint32_t phase = 0;
  float* const Zs[3] = {t.Z1, t.Z2, t.Z3};
  uint16_t* const Hs[3] = {t.H1, t.H2, t.H3};
  uint16_t* const Hts[3] = {t.H1t, t.H2t, t.H3t};
#pragma unroll 1
  for (int layer = 0; layer < 4; ++layer) {
    if (tid == 0) {
      const size_t wo = layer == 0 ? FwdSmem::w1 : layer == 1 ? FwdSmem::w2 : layer == 2 ? FwdSmem::w3 : FwdSmem::w4;
      if (layer == 0)
        mma_tile(tmem, sX, kSbo128, smem + wo, kSbo128, tc::idesc_bf16_f32(128, 64), 8, false);
      else
        mma_tile(tmem + (layer == 3 ? 64u : 0u), sH, kSbo64, smem + wo, kSbo64,
                 layer == 3 ? tc::idesc_bf16_f32(128, 16) : tc::idesc_bf16_f32(128, 64), 4, false);
      tc::commit(&bar);
    }
    // while the tensor core works: the transpose of the layer's input
    if (layer == 0)
      store_transposed(sX, kSbo128, 128, FFMPM_MLP_FEATURES, t.Xt, B, r0);
    else
      store_transposed(sH, kSbo64, 64, 64, Hts[layer - 1], B, r0);
    if (!mbar_wait(&bar, phase)) s_fail = 1;
    phase ^= 1u;
    tc::fence_after_sync();
    __syncthreads();  // also: every thread has read sH
    if (s_fail) break;
    if (layer < 3) {
#pragma unroll 1
      for (int c = c0; c < c0 + 32; c += 16) {
        float a[16];
        tc::tmem_ld16(tc::taddr_of(tmem, lanes, c), a);
        uint32_t hw[8];
#pragma unroll
        for (int j = 0; j < 16; ++j) a[j] += sbias[64 * layer + c + j];
#pragma unroll
        for (int j = 0; j < 8; ++j)
          hw[j] = uint32_t(tc::bf16_bits(gelu_f(a[2 * j]))) | (uint32_t(tc::bf16_bits(gelu_f(a[2 * j + 1]))) << 16);
        const size_t at = (size_t)(r0 + row) * 64 + c;
#pragma unroll
        for (int j = 0; j < 4; ++j)
          store4(Zs[layer] + at + 4 * j, make_float4(a[4 * j], a[4 * j + 1], a[4 * j + 2], a[4 * j + 3]), vec);
        uint4* h = reinterpret_cast<uint4*>(Hs[layer] + at);
#pragma unroll
        for (int j = 0; j < 2; ++j) {
          const uint4 v = make_uint4(hw[4 * j], hw[4 * j + 1], hw[4 * j + 2], hw[4 * j + 3]);
          h[j] = v;
          *reinterpret_cast<uint4*>(sH + tc::kmajor_offset(row, c + 8 * j, kSbo64)) = v;
        }
      }
      fence_proxy_async_shared();
      tc::fence_before_sync();
      __syncthreads();
      tc::fence_after_sync();
    } else if (c0 == 0) {
      float y[16];
      tc::tmem_ld16(tc::taddr_of(tmem, lanes, 64), y);
#pragma unroll
      for (int j = 0; j < 4; ++j)
        store4(t.Y + (size_t)(r0 + row) * 16 + 4 * j, make_float4(y[4 * j], y[4 * j + 1], y[4 * j + 2], y[4 * j + 3]),
               vec);
    }
  }
  if (s_fail && tid == 0) {
    if (t.status) raise_status(t.status, FFMPM_STATUS_TIMEOUT);
    // the MMAs of the last commit may still be running: wait for them once more (bounded) before
    // their tensor memory is freed
    mbar_wait(&bar, phase ^ 1u);
  }
  tc::fence_before_sync();
  __syncthreads();
  if (warp == 0) tc::tmem_free(tmem, 128);
}

// Tensor-memory columns of the backward pass: the gradients of the four weight matrices (row = output
// unit) and the adjoint of a layer's input.
constexpr uint32_t kColW1 = 0, kColW2 = 128, kColW3 = 192, kColW4 = 256, kColDH = 320;
struct BwdSmem {
  static constexpr size_t w4t = 0, w3t = w4t + 64 * 64 * 2, w2t = w3t + 64 * 64 * 2,
                          g = w2t + 64 * 64 * 2,     // dY / dZ [128 rows][64]
                          gt = g + 128 * 64 * 2,     // its transpose [128: 64 used][128 rows]
                          it = gt + 128 * 128 * 2,   // transpose of the layer's input [up to 128][128 rows]
                          used = it + 128 * 128 * 2;
  // one CTA per SM: each holds all 512 tensor-memory columns
  static constexpr size_t total = used > 120 * 1024 ? used : 120 * 1024;
};

// Two neighbouring columns c (even), c + 1 of the thread's row into the transposed tile [c][row]: the lanes
// of two neighbouring rows swap a value, so that each stores one 32-bit word.
__device__ __forceinline__ void put_transposed2(unsigned char* tile, int c, int row, uint32_t lo, uint32_t hi) {
  const bool odd = row & 1;
  const uint32_t got = __shfl_xor_sync(0xffffffffu, odd ? lo : hi, 1);
  const uint32_t w = odd ? (got | (hi << 16)) : (lo | (got << 16));
  *reinterpret_cast<uint32_t*>(tile + tc::kmajor_offset(c + (odd ? 1 : 0), row & ~1, kSbo128)) = w;
}

// Sum over the warp's 32 rows of 32 columns: lane l returns the sum of column l.
__device__ __forceinline__ float column_sum(float (&v)[32]) {
  const int lane = threadIdx.x & 31;
#pragma unroll
  for (int o = 16; o >= 1; o >>= 1)
#pragma unroll
    for (int i = 0; i < o; ++i) {
      const bool up = lane & o;
      const float keep = up ? v[i + o] : v[i], send = up ? v[i] : v[i + o];
      v[i] = keep + __shfl_xor_sync(0xffffffffu, send, o);
    }
  return v[0];
}

// Loss and the gradient of every parameter (added to zeroed grads).  Per tile of 128 rows and layer, from
// the last to the first: g = dL/d(layer's output) in bf16, then on the tensor cores the adjoint of the
// layer's input, g . W, and the layer's weight gradient, g^T . input, whose accumulator stays in tensor
// memory over all the tiles of the CTA.
__global__ void __launch_bounds__(kTrain) k_mlp_backward(ffmpm_mlp_trainer t, const float* __restrict__ T,
                                                         const float* __restrict__ w, int B,
                                                         double* __restrict__ loss, bool vec) {
  extern __shared__ __align__(1024) unsigned char smem[];
  unsigned char *sG = smem + BwdSmem::g, *sGt = smem + BwdSmem::gt, *sIt = smem + BwdSmem::it;
  __shared__ uint64_t bar;
  __shared__ uint32_t tmem_base;
  __shared__ int s_fail;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, row = tid & 127, c0 = 32 * (tid >> 7);
  const uint32_t lanes = 32u * (warp & 3);
  stage_kmajor(smem + BwdSmem::w4t, t.W4t, 64, 64, kSbo64);
  stage_kmajor(smem + BwdSmem::w3t, t.W3t, 64, 64, kSbo64);
  stage_kmajor(smem + BwdSmem::w2t, t.W2t, 64, 64, kSbo64);
  for (int i = tid; i < 128 * 128 * 2 / 16; i += kTrain) reinterpret_cast<uint4*>(sGt)[i] = make_uint4(0u, 0u, 0u, 0u);
  if (warp == 0) tc::tmem_alloc(&tmem_base, 512);
  if (tid == 0) {
    mbar_init(&bar, 1);
    fence_barrier_init();
    s_fail = 0;
  }
  tc::fence_before_sync();
  __syncthreads();
  tc::fence_after_sync();
  const uint32_t tmem = tmem_base;
  uint32_t phase = 0;
  bool first = true;
  double l = 0.0;
  float db[4] = {0.f, 0.f, 0.f, 0.f};  // column c0 + lane of b1..b4, over the warp's rows
  const float* const Zs[3] = {t.Z1, t.Z2, t.Z3};
  const uint16_t* const ins[4] = {t.Xt, t.H1t, t.H2t, t.H3t};  // the layers' inputs, transposed [width][B]
  const float* const b4 = t.params + FFMPM_MLP_OFF_B4;
#pragma unroll 1
  for (int tile = blockIdx.x; tile * 128 < B; tile += gridDim.x) {
    const size_t r = (size_t)tile * 128 + row;
#pragma unroll 1
    for (int layer = 3; layer >= 0; --layer) {
      float g[32];  // dL/d(output of the layer before its activation), the thread's columns
      if (layer == 3) {
        const float invB = 1.f / float(B);
#pragma unroll
        for (int j = 0; j < 32; ++j) g[j] = 0.f;
        if (c0 == 0) {
#pragma unroll
          for (int j = 0; j < FFMPM_MLP_OUT; ++j) {
            const float e = t.Y[r * 16 + j] + b4[j] - T[r * FFMPM_MLP_OUT + j];
            l += double(w[j]) * double(e) * double(e);
            g[j] = 2.f * w[j] * e * invB;
          }
        }
      } else {
        const float* z = Zs[layer] + r * 64 + c0;
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          float a[16];
          tc::tmem_ld16(tc::taddr_of(tmem, lanes, kColDH + c0 + 16 * h), a);
#pragma unroll
          for (int j = 0; j < 4; ++j) {
            const float4 zz = load4(z + 16 * h + 4 * j, vec);
            g[16 * h + 4 * j] = a[4 * j] * gelu_grad(zz.x);
            g[16 * h + 4 * j + 1] = a[4 * j + 1] * gelu_grad(zz.y);
            g[16 * h + 4 * j + 2] = a[4 * j + 2] * gelu_grad(zz.z);
            g[16 * h + 4 * j + 3] = a[4 * j + 3] * gelu_grad(zz.w);
          }
        }
      }
      // g as the operand of g . W (layer > 0) and, transposed, of g^T . input
#pragma unroll
      for (int j = 0; j < 32; j += 8) {
        uint32_t q[4];
#pragma unroll
        for (int k = 0; k < 4; ++k) {
          const uint32_t lo = tc::bf16_bits(g[j + 2 * k]), hi = tc::bf16_bits(g[j + 2 * k + 1]);
          q[k] = lo | (hi << 16);
          put_transposed2(sGt, c0 + j + 2 * k, row, lo, hi);
        }
        if (layer > 0)
          *reinterpret_cast<uint4*>(sG + tc::kmajor_offset(row, c0 + j, kSbo64)) = make_uint4(q[0], q[1], q[2], q[3]);
      }
      // the layer's input: 128 columns of its transpose (rows 113.. of Xt are zero: those features take no
      // gradient)
      {
        const uint16_t* in = ins[layer] + (size_t)tile * 128;
        const int width = layer > 0 ? 64 : 128;
        for (int v = tid; v < width * 16; v += kTrain) {
          const int c = v >> 4, q = 8 * (v & 15);
          *reinterpret_cast<uint4*>(sIt + tc::kmajor_offset(c, q, kSbo128)) =
              *reinterpret_cast<const uint4*>(in + (size_t)c * B + q);
        }
      }
      db[layer] += column_sum(g);
      fence_proxy_async_shared();
      tc::fence_before_sync();
      __syncthreads();
      tc::fence_after_sync();
      if (tid == 0) {
        if (layer > 0) {
          const size_t wt = layer == 3 ? BwdSmem::w4t : layer == 2 ? BwdSmem::w3t : BwdSmem::w2t;
          mma_tile(tmem + kColDH, sG, kSbo64, smem + wt, kSbo64, tc::idesc_bf16_f32(128, 64), 4, false);
        }
        const uint32_t col = layer == 3 ? kColW4 : layer == 2 ? kColW3 : layer == 1 ? kColW2 : kColW1;
        mma_tile(tmem + col, sGt, kSbo128, sIt, kSbo128, tc::idesc_bf16_f32(128, layer > 0 ? 64 : 128), 8, !first);
        tc::commit(&bar);
      }
      if (!mbar_wait(&bar, phase)) s_fail = 1;
      phase ^= 1u;
      tc::fence_after_sync();
      __syncthreads();
      if (s_fail) break;
    }
    if (s_fail) break;
    first = false;
  }
  if (s_fail) {
    if (tid == 0) {
      if (t.status) raise_status(t.status, FFMPM_STATUS_TIMEOUT);
      mbar_wait(&bar, phase ^ 1u);
    }
  } else if (!first) {
    float* G = t.grads;
    // the weight gradients: row = lane of tensor memory (64 used, 12 for W4), the columns split over the halves
    const int out = row;
    const auto add = [&](uint32_t col, int cols, int off, int ld, int rows) {
#pragma unroll 1
      for (int c = (tid >> 7) * (cols / 2); c < ((tid >> 7) + 1) * (cols / 2); c += 16) {
        float a[16];
        tc::tmem_ld16(tc::taddr_of(tmem, lanes, col + c), a);
        if (out < rows) {
#pragma unroll
          for (int j = 0; j < 4; ++j)
            add4(G + off + (size_t)out * ld + c + 4 * j,
                 make_float4(a[4 * j], a[4 * j + 1], a[4 * j + 2], a[4 * j + 3]), vec);
        }
      }
    };
    add(kColW1, 128, FFMPM_MLP_OFF_W1, 128, 64);
    add(kColW2, 64, FFMPM_MLP_OFF_W2, 64, 64);
    add(kColW3, 64, FFMPM_MLP_OFF_W3, 64, 64);
    add(kColW4, 64, FFMPM_MLP_OFF_W4, 64, FFMPM_MLP_OUT);
    atomicAdd(&G[FFMPM_MLP_OFF_B1 + c0 + lane], db[0]);
    atomicAdd(&G[FFMPM_MLP_OFF_B2 + c0 + lane], db[1]);
    atomicAdd(&G[FFMPM_MLP_OFF_B3 + c0 + lane], db[2]);
    if (c0 == 0 && lane < FFMPM_MLP_OUT) atomicAdd(&G[FFMPM_MLP_OFF_B4 + lane], db[3]);
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) l += __shfl_xor_sync(0xffffffffu, l, o);
    if (lane == 0 && c0 == 0) atomicAdd(loss, l / double(B));
  }
  tc::fence_before_sync();
  __syncthreads();
  if (warp == 0) tc::tmem_free(tmem, 512);
}

__global__ void __launch_bounds__(kEw) k_adam(float* __restrict__ p, const float* __restrict__ g,
                                              float* __restrict__ m, float* __restrict__ v, int count, float lr,
                                              float b1, float b2, float eps, float c1, float c2) {
  const int i = blockIdx.x * kEw + threadIdx.x;
  if (i >= count) return;
  const float gi = g[i];
  const float mi = b1 * m[i] + (1.f - b1) * gi;
  const float vi = b2 * v[i] + (1.f - b2) * gi * gi;
  m[i] = mi;
  v[i] = vi;
  p[i] -= lr * (mi / c1) / (sqrtf(vi / c2) + eps);
}

// params -> bf16 W1 [64][128], W2/W3 [64][64], W4 [16][64] (rows >= 12 zero) and W2t/W3t/W4t [64][64].
__global__ void __launch_bounds__(kEw) k_pack(const float* __restrict__ P, uint16_t* W1, uint16_t* W2, uint16_t* W3,
                                              uint16_t* W4, uint16_t* W2t, uint16_t* W3t, uint16_t* W4t) {
  const int i = blockIdx.x * kEw + threadIdx.x;
  if (i < 64 * 128) W1[i] = tc::bf16_bits(P[FFMPM_MLP_OFF_W1 + i]);
  if (i < 64 * 64) {
    const int r = i >> 6, c = i & 63;
    W2[i] = tc::bf16_bits(P[FFMPM_MLP_OFF_W2 + i]);
    W3[i] = tc::bf16_bits(P[FFMPM_MLP_OFF_W3 + i]);
    W2t[c * 64 + r] = W2[i];
    W3t[c * 64 + r] = W3[i];
    // W4t[h][j] = W4[j][h] for the 12 outputs j, zero for j >= 12
    const float w4 = r < FFMPM_MLP_OUT ? P[FFMPM_MLP_OFF_W4 + r * 64 + c] : 0.f;
    W4t[c * 64 + r] = tc::bf16_bits(w4);
    if (r < 16) W4[r * 64 + c] = tc::bf16_bits(w4);
  }
}

int ew_grid(int64_t n) { return (int)((n + kEw - 1) / kEw); }

// Whether the float buffers that the training kernels access four floats at a time are 16-byte aligned (the
// bf16 ones have to be).
bool aligned16(const ffmpm_mlp_trainer& t) {
  return ((reinterpret_cast<uintptr_t>(t.Z1) | reinterpret_cast<uintptr_t>(t.Z2) | reinterpret_cast<uintptr_t>(t.Z3) |
           reinterpret_cast<uintptr_t>(t.Y) | reinterpret_cast<uintptr_t>(t.grads)) & 15) == 0;
}

}  // namespace
}  // namespace ffmpm

using namespace ffmpm;

extern "C" {

int ffmpm_tc_gemm_bf16(const uint16_t* A, const uint16_t* B, float* D, int32_t M, int32_t N, int32_t K,
                       int32_t split_k, int32_t* status, void* stream) {
  if (!A || !B || !D || M <= 0 || N <= 0 || K <= 0) return FFMPM_ERR_BADARG;
  if (M % 128 || N % 16 || N > 256 || K % kKChunk) return FFMPM_ERR_BADARG;
  if ((reinterpret_cast<uintptr_t>(A) | reinterpret_cast<uintptr_t>(B)) & 15) return FFMPM_ERR_BADARG;
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  const int split = std::max(1, (int)split_k);
  if (N <= 16) return launch_gemm<16>(A, B, D, M, N, K, split, status, s);
  if (N <= 32) return launch_gemm<32>(A, B, D, M, N, K, split, status, s);
  if (N <= 64) return launch_gemm<64>(A, B, D, M, N, K, split, status, s);
  if (N <= 128) return launch_gemm<128>(A, B, D, M, N, K, split, status, s);
  return launch_gemm<256>(A, B, D, M, N, K, split, status, s);
}

int ffmpm_mlp_train_forward(const ffmpm_mlp_trainer* t, const uint16_t* X, int32_t B, void* stream) {
  if (!t || !X || B <= 0 || B % 128 || B > t->max_batch || (reinterpret_cast<uintptr_t>(X) & 15)) return FFMPM_ERR_BADARG;
  if (!allow_smem(reinterpret_cast<const void*>(k_mlp_forward), FwdSmem::total)) return FFMPM_ERR_CUDA;
  k_mlp_forward<<<B / 128, kTrain, FwdSmem::total, static_cast<cudaStream_t>(stream)>>>(*t, X, B, aligned16(*t));
  return cudaGetLastError() == cudaSuccess ? FFMPM_OK : FFMPM_ERR_CUDA;
}

int ffmpm_mlp_train_backward(const ffmpm_mlp_trainer* t, const float* T, const float* w, int32_t B, double* loss,
                             void* stream) {
  if (!t || !T || !w || !loss || B <= 0 || B % 128 || B > t->max_batch) return FFMPM_ERR_BADARG;
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  if (!allow_smem(reinterpret_cast<const void*>(k_mlp_backward), BwdSmem::total)) return FFMPM_ERR_CUDA;
  cudaMemsetAsync(t->grads, 0, sizeof(float) * FFMPM_MLP_PARAMS, s);
  k_mlp_backward<<<std::min(B / 128, sm_count()), kTrain, BwdSmem::total, s>>>(*t, T, w, B, loss, aligned16(*t));
  return cudaGetLastError() == cudaSuccess ? FFMPM_OK : FFMPM_ERR_CUDA;
}

int ffmpm_mlp_train_update(const ffmpm_mlp_trainer* t, float lr, float beta1, float beta2, float eps, int32_t step,
                           void* stream) {
  if (!t || step < 1) return FFMPM_ERR_BADARG;
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  const float c1 = 1.f - powf(beta1, (float)step), c2 = 1.f - powf(beta2, (float)step);
  k_adam<<<ew_grid(FFMPM_MLP_PARAMS), kEw, 0, s>>>(t->params, t->grads, t->adam_m, t->adam_v, FFMPM_MLP_PARAMS, lr,
                                                  beta1, beta2, eps, c1, c2);
  k_pack<<<ew_grid(64 * 128), kEw, 0, s>>>(t->params, t->W1, t->W2, t->W3, t->W4, t->W2t, t->W3t, t->W4t);
  return cudaGetLastError() == cudaSuccess ? FFMPM_OK : FFMPM_ERR_CUDA;
}

}  // extern "C"
