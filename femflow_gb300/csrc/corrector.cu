// Learned-corrector G2P: the 3D G2P of a coarse substep (three_d/g2p.py:9-59) fused with a
// per-particle MLP that corrects its result, run on the 5th-generation tensor cores.
//
// A CTA of 512 threads is four warpgroups, each on a tile of 128 particles of its own (persistent over
// tiles; thread t of a group owns particle tile * 128 + t and TMEM lane t, i.e. row t of every MLP
// layer); they share the weights and hide one another's latencies.  Per tile:
//   1. the 27 node velocities of every particle come to shared memory a plane of nine nodes at a time:
//      a warp takes its 32 particles one after another, its lanes on the 27 floats of a plane (three runs
//      of nine), so that one asynchronous load instruction touches a few lines where a load per thread
//      and float touches 32.  Each thread then forms v', C', F' and x' as the plain G2P does (node
//      velocities taken relative to the stencil's centre node u) and its bf16 features in row t of the
//      K-major input tile, eight to a store:
//        [0, 9)   F' - I            [9, 18)  C' dt            [18, 21) (v' - u) dt / dx
//        [21,102) (v_i - u) dt / dx for the 27 nodes i
//        [102,104) mu k, lam k      [104,113) PF k (the stress of this step's P2G)      [113,128) 0
//      with k = dt^2 / (rho dx^2) (stiffness and stress in units of the step's own CFL number
//      squared), each multiplied by the network's per-feature input scale;
//   2. four MMA layers 128->64->64->64->16 (GELU between), bf16 operands, FP32 accumulators in
//      TMEM; after each layer every thread reads its own row back (tcgen05.ld), adds the bias,
//      applies GELU and writes the bf16 row of the next layer's operand;
//   3. outputs y[0,12) times the output scale: F' += y[0,9), v' += y[9,12) dx / dt, x' += dt * that.
// 1,048,576 particles of a random order on 128^3 (GB300): 337 us, from 580 with one tile of 128 threads a CTA,
// loads and feature stores one float and one bf16 at a time and erff; bound by instruction issue (GELU of
// 192 units a particle) and the gathers' latency.
// Weights (bf16, K-major) and biases stay in shared memory for the whole launch.  Modes: apply the
// network, export the features (no network), or both off (the plain coarse G2P through the same
// arithmetic).  Every mbarrier wait is bounded.
#include <cuda_bf16.h>
#include <cuda_runtime.h>

#include <algorithm>

#include "common.cuh"
#include "internal.h"
#include "mpm_kernels.cuh"
#include "tc.cuh"

namespace ffmpm {
namespace {

constexpr int kIn = FFMPM_MLP_IN;    // 128 inputs (FFMPM_MLP_FEATURES used)
constexpr int kHid = FFMPM_MLP_HIDDEN;
constexpr int kOutPad = 16;
constexpr int kOut = FFMPM_MLP_OUT;  // 12
constexpr uint32_t kSboIn = (kIn / 8) * 128;
constexpr uint32_t kSboHid = (kHid / 8) * 128;
constexpr int kGroups = 4;                  // warpgroups (tiles in flight) per CTA
constexpr int kThreadsC = 128 * kGroups;
constexpr uint32_t kTmemCols = 128;         // per group: [0, 64) hidden layers, [64, 80) output layer
constexpr int kPlane = 27;                  // floats of a plane of nine nodes

struct SmemLayout {
  static constexpr size_t w1 = 0;
  static constexpr size_t w2 = w1 + size_t(kHid) * kIn * 2;
  static constexpr size_t w3 = w2 + size_t(kHid) * kHid * 2;
  static constexpr size_t w4 = w3 + size_t(kHid) * kHid * 2;
  static constexpr size_t f = w4 + size_t(kOutPad) * kHid * 2;  // floats: b1 b2 b3 b4 in_scale out_scale
  static constexpr int nf = 3 * kHid + kOutPad + kIn + kOutPad;
  static constexpr size_t group = f + sizeof(float) * nf;  // per group: input tile, then a plane of velocities
  static constexpr size_t x_bytes = size_t(128) * kIn * 2;  // the hidden layers' tile lies over the input tile
  static constexpr size_t group_bytes = x_bytes + size_t(128) * kPlane * 4;
  static constexpr size_t total = group + kGroups * group_bytes;
};
static_assert(SmemLayout::group % 128 == 0 && SmemLayout::group_bytes % 128 == 0, "aligned tiles");
static_assert(SmemLayout::total <= 227 * 1024 - 1024, "one CTA per SM");

// GELU(z) = z Phi(z), with Phi(-a) = 2^p(-a) for a = |z| and GELU(z) = max(z, 0) - a Phi(-a).  p: degree-10
// polynomial fitted to log2 of the normal distribution function on [-6, 0] (reweighted least squares at
// Chebyshev points, largest error 3.6e-7).  Beyond |z| = 6 the second term stays at its value there, 6e-9, so
// that it neither grows with z nor makes a NaN of an infinity; a NaN stays one (max.NaN).  In float over [-8, 8]:
// largest absolute error 2.4e-7, rms 5.2e-8, and 1.2e-6 relative for |z| < 4; 0.5 z (1 + erff(z / sqrt 2)) has
// 4.5e-7, 6.8e-8 and (where 1 + erf cancels) 4.6e-4.  Two at a time: the polynomial runs on packed FMAs.
__device__ __forceinline__ uint64_t pack2(float a, float b) {
  uint64_t r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(a), "f"(b));
  return r;
}
__device__ __forceinline__ uint64_t fma2(uint64_t a, uint64_t b, uint64_t c) {
  uint64_t r;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
  return r;
}
__device__ __forceinline__ float max_nan(float a, float b) {
  float r;
  asm("max.NaN.f32 %0, %1, %2;" : "=f"(r) : "f"(a), "f"(b));
  return r;
}
__device__ __forceinline__ void gelu2(float z0, float z1, float& g0, float& g1) {
  constexpr float kP[11] = {-0.999999642f, 1.15111935f, -0.459117204f, 0.0527117103f, 0.0073000202f, 0.000260737259f,
                            -0.000164237936f, -4.52711574e-05f, -5.93813365e-06f, -4.14644262e-07f, -1.23162778e-08f};
  const float m0 = max_nan(-fabsf(z0), -6.f), m1 = max_nan(-fabsf(z1), -6.f);
  const uint64_t m = pack2(m0, m1);
  uint64_t p = pack2(kP[10], kP[10]);
#pragma unroll
  for (int i = 9; i >= 0; --i) p = fma2(p, m, pack2(kP[i], kP[i]));
  float p0, p1;
  asm("mov.b64 {%0, %1}, %2;" : "=f"(p0), "=f"(p1) : "l"(p));
  g0 = fmaf(m0, exp2f(p0), fmaxf(z0, 0.f));
  g1 = fmaf(m1, exp2f(p1), fmaxf(z1, 0.f));
}

__device__ __forceinline__ uint32_t bf16x2(float a, float b) {
  return uint32_t(tc::bf16_bits(a)) | (uint32_t(tc::bf16_bits(b)) << 16);
}

// Copy a bf16 row-major [rows][k] matrix into the K-major core-matrix layout.
__device__ __forceinline__ void stage_kmajor(unsigned char* dst, const uint16_t* src, int rows, int k, uint32_t sbo) {
  const int vecs = k / 8;
  for (int v = threadIdx.x; v < rows * vecs; v += blockDim.x) {
    const int r = v / vecs, c = v % vecs;
    *reinterpret_cast<uint4*>(dst + tc::kmajor_offset(r, 8 * c, sbo)) =
        *reinterpret_cast<const uint4*>(src + (size_t)r * k + 8 * c);
  }
}

// Eight consecutive features (from 8 c on) of row r as one 16-byte store, scaled.
__device__ __forceinline__ void put8(unsigned char* tile, int r, int c, const float (&f)[8], const float* s_in) {
  const float4 s0 = *reinterpret_cast<const float4*>(s_in + 8 * c), s1 = *reinterpret_cast<const float4*>(s_in + 8 * c + 4);
  *reinterpret_cast<uint4*>(tile + tc::kmajor_offset(r, 8 * c, kSboIn)) =
      make_uint4(bf16x2(f[0] * s0.x, f[1] * s0.y), bf16x2(f[2] * s0.z, f[3] * s0.w), bf16x2(f[4] * s1.x, f[5] * s1.y),
                 bf16x2(f[6] * s1.z, f[7] * s1.w));
}

__device__ __forceinline__ void group_sync(int g) { asm volatile("bar.sync %0, 128;" ::"r"(g + 1) : "memory"); }

// Order-preserving float -> int key (for atomicMin / atomicMax on signed floats).
__device__ __forceinline__ int float_key(float f) {
  const int i = __float_as_int(f);
  return i >= 0 ? i : i ^ 0x7FFFFFFF;
}

template <bool kApply, bool kExport>
__global__ void __launch_bounds__(kThreadsC, 1) k_corrector(KParams<float> kp, const float* __restrict__ gv,
                                                            PView<float> P, uint32_t n, ffmpm_mlp net,
                                                            uint16_t* __restrict__ feat_out,
                                                            int* __restrict__ det_keys, int32_t* status) {
  extern __shared__ __align__(1024) unsigned char smem[];
  float* const sbias = reinterpret_cast<float*>(smem + SmemLayout::f);  // b1, b2, b3
  float* const sb4 = sbias + 3 * kHid;
  float* const s_in = sb4 + kOutPad;
  float* const s_out = s_in + kIn;
  __shared__ uint64_t bars[kGroups];
  __shared__ uint32_t tmem_base;
  __shared__ int s_fail[kGroups];
  const int grp = threadIdx.x >> 7, tid = threadIdx.x & 127, lane = tid & 31;
  unsigned char* const sX = smem + SmemLayout::group + grp * SmemLayout::group_bytes;
  float* const sV = reinterpret_cast<float*>(sX + SmemLayout::x_bytes);  // [128][kPlane]
  float* const warpV = sV + (tid & ~31) * kPlane;

  for (int i = threadIdx.x; i < kIn; i += kThreadsC) s_in[i] = net.in_scale ? net.in_scale[i] : 1.f;
  if (kApply) {
    stage_kmajor(smem + SmemLayout::w1, net.W1, kHid, kIn, kSboIn);
    stage_kmajor(smem + SmemLayout::w2, net.W2, kHid, kHid, kSboHid);
    stage_kmajor(smem + SmemLayout::w3, net.W3, kHid, kHid, kSboHid);
    stage_kmajor(smem + SmemLayout::w4, net.W4, kOutPad, kHid, kSboHid);
    for (int i = threadIdx.x; i < kHid; i += kThreadsC) {
      sbias[i] = net.b1[i];
      sbias[kHid + i] = net.b2[i];
      sbias[2 * kHid + i] = net.b3[i];
    }
    for (int i = threadIdx.x; i < kOutPad; i += kThreadsC) {
      sb4[i] = net.b4[i];
      s_out[i] = net.out_scale[i];
    }
    if (threadIdx.x < 32) tc::tmem_alloc(&tmem_base, kGroups * kTmemCols);
    fence_proxy_async_shared();
  }
  if (threadIdx.x < kGroups) {
    mbar_init(&bars[threadIdx.x], 1);
    fence_barrier_init();
    s_fail[threadIdx.x] = 0;
  }
  tc::fence_before_sync();
  __syncthreads();
  tc::fence_after_sync();
  const uint32_t tmem = (kApply ? tmem_base : 0u) + grp * kTmemCols;
  uint64_t* const bar = &bars[grp];
  const uint32_t lane_base = 32u * (tid >> 5);
  uint32_t phase = 0;
  const float dt = kp.dt, inv_dx = kp.inv_dx;
  const float vs = dt * inv_dx;  // velocity -> cells per step
  const int R = kp.res + 1;
  const int64_t RR = (int64_t)R * R;
  float dmin = 3.4e38f, dmax = -3.4e38f;

  // neighbouring groups of a CTA take tiles a grid apart, so that few tiles spread over the SMs
  for (int64_t tile = blockIdx.x + (int64_t)gridDim.x * grp; tile * 128 < n; tile += (int64_t)gridDim.x * kGroups) {
    const uint32_t p = (uint32_t)(tile * 128 + tid);
    bool valid = p < n;
    float xo[3], Fo[9], Co[9], vo[3];
    float x[3], fx[3], w[3][3];
    int node = -1;
    if (valid) {
      int b[3];
      bool ok = true;
#pragma unroll
      for (int d = 0; d < 3; ++d) x[d] = P.x[P.at(p, d, 3)];
#pragma unroll
      for (int d = 0; d < 3; ++d) ok = ok && base_of(x[d], inv_dx, kp.res, b[d], fx[d]);
      if (!ok) {
        raise_status(status, FFMPM_STATUS_OOB);
        valid = false;
      } else {
        node = (int)node_index<3>(R, b);
#pragma unroll
        for (int d = 0; d < 3; ++d) {
          float ww[3];
          bspline(fx[d], ww);
          w[0][d] = ww[0];
          w[1][d] = ww[1];
          w[2][d] = ww[2];
        }
      }
    }
    float u[3] = {0.f, 0.f, 0.f}, v[3] = {0.f, 0.f, 0.f}, C[9] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
    if (valid) {
      const float* c = gv + 3 * (node + RR + R + 1);
#pragma unroll
      for (int d = 0; d < 3; ++d) u[d] = c[d];
    }
    float wzd[3];
#pragma unroll
    for (int k = 0; k < 3; ++k) wzd[k] = valid ? w[k][2] * (float(k) - fx[2]) : 0.f;
    float keep[6] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f};   // features of a chunk of eight that a later plane completes
    float first[3] = {0.f, 0.f, 0.f};                 // features 21..23, for the chunk 16..23
    const int sj = lane / 9;  // the lane's run of nine floats (27 lanes) and its place in it
    const int64_t soff = (int64_t)3 * sj * R + (lane - 9 * sj);
#pragma unroll
    for (int i = 0; i < 3; ++i) {
      __syncwarp();  // the previous plane (or tile) has been read
      for (int l = 0; l < 32; ++l) {
        const int nb = __shfl_sync(0xffffffffu, node, l);
        if (nb >= 0 && lane < kPlane)
          asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(smem_u32(warpV + l * kPlane + lane)),
                       "l"(gv + 3 * (nb + i * RR) + soff)
                       : "memory");
      }
      asm volatile("cp.async.wait_all;" ::: "memory");
      __syncwarp();
      if (valid) {
        const float* g = sV + tid * kPlane;
        float f[kPlane];
        float t0[3] = {0.f, 0.f, 0.f}, t1[3] = {0.f, 0.f, 0.f}, t2[3] = {0.f, 0.f, 0.f};
#pragma unroll
        for (int j = 0; j < 3; ++j) {
          float sa[3] = {0.f, 0.f, 0.f}, sb[3] = {0.f, 0.f, 0.f};
#pragma unroll
          for (int k = 0; k < 3; ++k)
#pragma unroll
            for (int r = 0; r < 3; ++r) {
              const float d = g[9 * j + 3 * k + r] - u[r];
              sa[r] += w[k][2] * d;
              sb[r] += wzd[k] * d;
              f[9 * j + 3 * k + r] = d * vs;
            }
          const float wy = w[j][1], wyd = wy * (float(j) - fx[1]);
#pragma unroll
          for (int r = 0; r < 3; ++r) {
            t0[r] += wy * sa[r];
            t1[r] += wyd * sa[r];
            t2[r] += wy * sb[r];
          }
        }
        const float wx = w[i][0], wxd = wx * (float(i) - fx[0]);
#pragma unroll
        for (int r = 0; r < 3; ++r) {
          v[r] += wx * t0[r];
          C[r * 3 + 0] += wxd * t0[r];
          C[r * 3 + 1] += wx * t1[r];
          C[r * 3 + 2] += wx * t2[r];
        }
        // features 21 + 27 i ...: whole chunks of eight go out, the ends wait for their neighbours
        float q[8];
        if (i == 0) {
#pragma unroll
          for (int e = 0; e < 3; ++e) first[e] = f[e];
#pragma unroll
          for (int c = 0; c < 3; ++c) {
#pragma unroll
            for (int e = 0; e < 8; ++e) q[e] = f[3 + 8 * c + e];
            put8(sX, tid, 3 + c, q, s_in);
          }
        } else if (i == 1) {
#pragma unroll
          for (int c = 0; c < 3; ++c) {
#pragma unroll
            for (int e = 0; e < 8; ++e) q[e] = f[8 * c + e];
            put8(sX, tid, 6 + c, q, s_in);
          }
#pragma unroll
          for (int e = 0; e < 3; ++e) keep[e] = f[24 + e];
        } else {
#pragma unroll
          for (int e = 0; e < 8; ++e) q[e] = e < 3 ? keep[e] : f[e - 3];
          put8(sX, tid, 9, q, s_in);
#pragma unroll
          for (int c = 0; c < 2; ++c) {
#pragma unroll
            for (int e = 0; e < 8; ++e) q[e] = f[5 + 8 * c + e];
            put8(sX, tid, 10 + c, q, s_in);
          }
#pragma unroll
          for (int e = 0; e < 6; ++e) keep[e] = f[21 + e];
        }
      }
    }
    if (valid) {
      float F[9];
#pragma unroll
      for (int i = 0; i < 9; ++i) F[i] = P.F[P.at(p, i, 9)];
      const float c4 = 4.f * inv_dx;
#pragma unroll
      for (int i = 0; i < 9; ++i) Co[i] = C[i] * c4;
#pragma unroll
      for (int d = 0; d < 3; ++d) vo[d] = u[d] + v[d];
#pragma unroll
      for (int r = 0; r < 3; ++r)
#pragma unroll
        for (int c = 0; c < 3; ++c)
          Fo[r * 3 + c] = F[r * 3 + c] + dt * (Co[r * 3 + 0] * F[0 * 3 + c] + Co[r * 3 + 1] * F[1 * 3 + c] +
                                               Co[r * 3 + 2] * F[2 * 3 + c]);
#pragma unroll
      for (int d = 0; d < 3; ++d) xo[d] = x[d] + dt * vo[d];
      // material and stress features 102..112 (from the pre-step F, as the P2G of this step)
      float m_, mu_, lam_, FmR[9];
      lame_of(kp, P, p, m_, mu_, lam_);
      const float kk = dt * dt * inv_dx * inv_dx * kp.volume / m_;
      if (!f_minus_r_small_strain3(F, FmR)) {
        float Rr[9];
        polar3<float>(F, Rr, nullptr);
#pragma unroll
        for (int i = 0; i < 9; ++i) FmR[i] = F[i] - Rr[i];
      }
      const float J = det3(F);
      const float sc = lam_ * (J - 1.f) * J;
      float pf[9];
#pragma unroll
      for (int a = 0; a < 3; ++a)
#pragma unroll
        for (int c = 0; c < 3; ++c) {
          float s = (a == c || kp.model != FFMPM_MODEL_FIXED_COROTATED) ? sc : 0.f;
#pragma unroll
          for (int e = 0; e < 3; ++e) s += 2.f * mu_ * FmR[a * 3 + e] * F[c * 3 + e];
          pf[a * 3 + c] = s * kk;
        }
      float h[24];  // features 0..23
#pragma unroll
      for (int i = 0; i < 9; ++i) {
        h[i] = Fo[i] - (i % 4 == 0 ? 1.f : 0.f);
        h[9 + i] = Co[i] * dt;
      }
#pragma unroll
      for (int d = 0; d < 3; ++d) {
        h[18 + d] = v[d] * vs;
        h[21 + d] = first[d];
      }
      float q[8];
#pragma unroll
      for (int c = 0; c < 3; ++c) {
#pragma unroll
        for (int e = 0; e < 8; ++e) q[e] = h[8 * c + e];
        put8(sX, tid, c, q, s_in);
      }
#pragma unroll
      for (int e = 0; e < 8; ++e) q[e] = e < 6 ? keep[e] : e == 6 ? mu_ * kk : lam_ * kk;
      put8(sX, tid, 12, q, s_in);
#pragma unroll
      for (int e = 0; e < 8; ++e) q[e] = pf[e];
      put8(sX, tid, 13, q, s_in);
      // 112 is the last feature; the padding is zero whatever its scales
      *reinterpret_cast<uint4*>(sX + tc::kmajor_offset(tid, 112, kSboIn)) =
          make_uint4(bf16x2(pf[8] * s_in[112], 0.f), 0u, 0u, 0u);
      *reinterpret_cast<uint4*>(sX + tc::kmajor_offset(tid, 120, kSboIn)) = make_uint4(0u, 0u, 0u, 0u);
    } else {
#pragma unroll
      for (int k = 0; k < kIn; k += 8)
        *reinterpret_cast<uint4*>(sX + tc::kmajor_offset(tid, k, kSboIn)) = make_uint4(0u, 0u, 0u, 0u);
    }
    if (kExport && valid) {
      uint4* dst = reinterpret_cast<uint4*>(feat_out + (size_t)p * kIn);
#pragma unroll
      for (int c = 0; c < kIn / 8; ++c) dst[c] = *reinterpret_cast<const uint4*>(sX + tc::kmajor_offset(tid, 8 * c, kSboIn));
    }
    if (kApply) {
      float y[16];
#pragma unroll 1
      for (int layer = 0; layer < 4; ++layer) {
        fence_proxy_async_shared();
        tc::fence_before_sync();
        group_sync(grp);
        tc::fence_after_sync();
        if (tid == 0) {
          // the hidden layers' tile lies where the input tile was: an MMA has read it before it is rewritten
          const unsigned char* B = smem + (layer == 0   ? SmemLayout::w1
                                           : layer == 1 ? SmemLayout::w2
                                           : layer == 2 ? SmemLayout::w3
                                                        : SmemLayout::w4);
          const int ksteps = (layer == 0 ? kIn : kHid) / 16;
          const uint32_t sbo = layer == 0 ? kSboIn : kSboHid;
          const uint32_t idesc = layer == 3 ? tc::idesc_bf16_f32(128, kOutPad) : tc::idesc_bf16_f32(128, kHid);
          const uint32_t d = tmem + (layer == 3 ? 64u : 0u);
          const uint32_t a0 = tc::smem_addr(sX), b0 = tc::smem_addr(B);
          for (int s = 0; s < ksteps; ++s)
            tc::mma_bf16(d, tc::make_desc(a0 + 256u * s, tc::kLBO, sbo), tc::make_desc(b0 + 256u * s, tc::kLBO, sbo),
                         idesc, s > 0);
          tc::commit(bar);
        }
        if (!mbar_wait(bar, phase)) s_fail[grp] = 1;
        phase ^= 1u;
        tc::fence_after_sync();
        group_sync(grp);
        if (s_fail[grp]) break;
        if (layer < 3) {
          const float* bias = sbias + kHid * layer;
#pragma unroll 1
          for (int c0 = 0; c0 < kHid; c0 += 16) {
            float a[16];
            tc::tmem_ld16(tc::taddr_of(tmem, lane_base, c0), a);
            uint32_t h[8];
#pragma unroll
            for (int j = 0; j < 8; ++j) {
              float g0, g1;
              gelu2(a[2 * j] + bias[c0 + 2 * j], a[2 * j + 1] + bias[c0 + 2 * j + 1], g0, g1);
              h[j] = bf16x2(g0, g1);
            }
#pragma unroll
            for (int j = 0; j < 2; ++j)
              *reinterpret_cast<uint4*>(sX + tc::kmajor_offset(tid, c0 + 8 * j, kSboHid)) =
                  make_uint4(h[4 * j], h[4 * j + 1], h[4 * j + 2], h[4 * j + 3]);
          }
        } else {
          tc::tmem_ld16(tc::taddr_of(tmem, lane_base, 64u), y);
        }
      }
      if (s_fail[grp]) break;
      if (valid) {
#pragma unroll
        for (int i = 0; i < 9; ++i) Fo[i] += (y[i] + sb4[i]) * s_out[i];
        const float inv_vs = 1.f / vs;
#pragma unroll
        for (int d = 0; d < 3; ++d) {
          const float dv = (y[9 + d] + sb4[9 + d]) * s_out[9 + d] * inv_vs;
          vo[d] += dv;
          xo[d] += dt * dv;
        }
      }
    }
    if (valid) {
#pragma unroll
      for (int d = 0; d < 3; ++d) {
        P.x[P.at(p, d, 3)] = xo[d];
        P.v[P.at(p, d, 3)] = vo[d];
      }
#pragma unroll
      for (int i = 0; i < 9; ++i) {
        P.F[P.at(p, i, 9)] = Fo[i];
        P.C[P.at(p, i, 9)] = Co[i];
      }
      const float J = det3(Fo);
      dmin = fminf(dmin, J);
      dmax = fmaxf(dmax, J);
    }
    // the next tile rewrites the group's tile: every thread is past this tile's MMAs and reads
    group_sync(grp);
  }
  if (s_fail[grp] && tid == 0) {
    raise_status(status, FFMPM_STATUS_TIMEOUT);
    // the MMAs of the last commit may still be running: wait for them once more (bounded) before
    // their tensor memory is freed
    mbar_wait(bar, phase ^ 1u);
  }
  if (det_keys) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      dmin = fminf(dmin, __shfl_xor_sync(0xffffffffu, dmin, o));
      dmax = fmaxf(dmax, __shfl_xor_sync(0xffffffffu, dmax, o));
    }
    if (lane == 0 && dmin <= dmax) {
      atomicMin(&det_keys[0], float_key(dmin));
      atomicMax(&det_keys[1], float_key(dmax));
    }
  }
  if (kApply) {
    tc::fence_before_sync();
    __syncthreads();
    if (threadIdx.x < 32) tc::tmem_free(tmem_base, kGroups * kTmemCols);
  }
}

template <bool A, bool E>
int launch_corrector(const ffmpm_params& p, const ffmpm_grid& g, ffmpm_particles& Pp, const ffmpm_mlp* net,
                     uint16_t* feat, int* det_keys, int32_t* status, cudaStream_t s) {
  auto kern = k_corrector<A, E>;
  const size_t smem = SmemLayout::total;
  if (!allow_smem(reinterpret_cast<const void*>(kern), smem)) return FFMPM_ERR_CUDA;
  const int64_t tiles = (Pp.n + 127) / 128;
  const int grid = (int)std::max<int64_t>(1, std::min<int64_t>(tiles, sm_count()));
  ffmpm_mlp nn{};
  if (net) nn = *net;
  kern<<<grid, kThreadsC, smem, s>>>(kparams<float>(p), static_cast<const float*>(g.velocity), pview<float>(Pp),
                                     (uint32_t)Pp.n, nn, feat, det_keys, status);
  return cudaGetLastError() == cudaSuccess ? FFMPM_OK : FFMPM_ERR_CUDA;
}

}  // namespace
}  // namespace ffmpm

using namespace ffmpm;

extern "C" {

int ffmpm_corrector_g2p(const ffmpm_params* p, const ffmpm_grid* grid, ffmpm_particles* P, const ffmpm_mlp* net,
                        uint16_t* features_out, int32_t* det_range, int32_t* status, void* stream) {
  if (!p || !grid || !grid->velocity || !P || P->n < 0 || P->n > int64_t(0x7FFFFFFF)) return FFMPM_ERR_BADARG;
  if (p->dim != 3 || p->real_bytes != 4) return FFMPM_ERR_UNSUPPORTED;
  if (P->stride != 0 && P->stride < P->n) return FFMPM_ERR_BADARG;
  if (P->n == 0) return FFMPM_OK;
  if (!P->x || !P->v || !P->F || !P->C) return FFMPM_ERR_BADARG;
  if (net && (!net->W1 || !net->W2 || !net->W3 || !net->W4 || !net->b1 || !net->b2 || !net->b3 || !net->b4 ||
              !net->out_scale))
    return FFMPM_ERR_BADARG;
  if (features_out && (reinterpret_cast<uintptr_t>(features_out) & 15)) return FFMPM_ERR_BADARG;
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  ffmpm_particles Q = *P;
  if (net && features_out) return launch_corrector<true, true>(*p, *grid, Q, net, features_out, det_range, status, s);
  if (net) return launch_corrector<true, false>(*p, *grid, Q, net, nullptr, det_range, status, s);
  if (features_out) return launch_corrector<false, true>(*p, *grid, Q, nullptr, features_out, det_range, status, s);
  return launch_corrector<false, false>(*p, *grid, Q, nullptr, nullptr, det_range, status, s);
}

}  // extern "C"
