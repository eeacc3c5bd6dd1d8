// Substep kernels that need no block sort: a warp takes 32 consecutive particles, whatever their
// order, and works on its own (no CTA barrier, no shared tile, no plan).
//
//   k_p2g_warp        stress + 3^d-node scatter (three_d/p2g.py:14-80, two_d/p2g.py:11-76)
//   k_grid_update_dense  momentum -> velocity at every node
//   k_g2p_range       gather, advect, F update (three_d/g2p.py:9-59, two_d/g2p.py:5-47)
//   k_grid_fold_user / k_grid_pack_user  between the workspace grid and a caller's grid arrays
#pragma once

#include "mpm_kernels.cuh"

namespace ffmpm {

// A particle's record as the run sums read it: [m, q (DIM), a = dx A (DIM^2, row-major), fx (DIM)] with
// q = m v - dx A fx; its contribution to stencil node o is w_o(fx) (q + a o, m).
template <int DIM>
struct RunRec {
  static constexpr int kFloats = 1 + 2 * DIM + DIM * DIM;  // 16 (3D) or 9 (2D)
  static constexpr int kPacked = DIM == 3 ? 16 : 12;       // whole Node4s: stride of a stream in memory
  // stride in shared memory: an odd number of Node4s, so that a warp's vector stores of one record
  // per lane and the reads of three records at a time fall on distinct banks
  static constexpr int kSmem = DIM == 3 ? 20 : 12;
};

template <int DIM, typename T>
__device__ __forceinline__ int run_record(const KParams<T>& kp, const P2GIn<DIM, T>& in, int R,
                                          T (&rec)[RunRec<DIM>::kPacked], int32_t* status, uint32_t* fallbacks,
                                          int (&base)[DIM]) {
  constexpr int DD = DIM * DIM, a0 = 1 + DIM;
  T fx[DIM];
  bool ok = true;
#pragma unroll
  for (int d = 0; d < DIM; ++d) ok = ok && base_of(in.x[d], kp.inv_dx, kp.res, base[d], fx[d]);
  if (!ok) {
    raise_status(status, FFMPM_STATUS_OOB);
    return -1;
  }
  const T e = (kp.model == FFMPM_MODEL_SNOW) ? ffexp(kp.hardening * (T(1) - in.jp)) : kp.hardening;
  T A[DD];
  affine_of<DIM, T>(kp, in.F, in.C, in.m, in.mu0 * e, in.lam0 * e, A, fallbacks);
  rec[0] = in.m;
#pragma unroll
  for (int r = 0; r < DIM; ++r) {
    T af = T(0);
#pragma unroll
    for (int c = 0; c < DIM; ++c) af += A[r * DIM + c] * fx[c];
    rec[1 + r] = in.v[r] * in.m - kp.dx * af;
  }
#pragma unroll
  for (int i = 0; i < DD; ++i) rec[a0 + i] = kp.dx * A[i];
#pragma unroll
  for (int d = 0; d < DIM; ++d) rec[a0 + DD + d] = fx[d];
#pragma unroll
  for (int i = RunRec<DIM>::kFloats; i < RunRec<DIM>::kPacked; ++i) rec[i] = T(0);
  return (int)node_index<DIM>(R, base);
}

// What a lane of a warp's run sums stands for.  The lanes form three groups of nine (five idle); each
// group sums a part of the particles of its own.  3D: a lane is a (j, k) pair and sums the three
// nodes along x; 2D: a lane is one of the nine nodes.
template <int DIM, typename T>
struct RunLane {
  static constexpr int NX = DIM == 3 ? 3 : 1;
  int grp, oa, ob;  // 3D: (j, k); 2D: (i, j)
  T ra, ka, ea, rb, kb, eb;  // w = k (f - r)^2 + e for the lane's two offsets
  __device__ __forceinline__ RunLane() {
    const int lane = threadIdx.x & 31;
    grp = lane / 9;
    const int jk = lane - grp * 9;
    oa = jk / 3;
    ob = jk - 3 * oa;
    ra = T(1.5) - T(0.5) * T(oa);
    rb = T(1.5) - T(0.5) * T(ob);
    ka = oa == 1 ? T(-1) : T(0.5);
    kb = ob == 1 ? T(-1) : T(0.5);
    ea = oa == 1 ? T(0.75) : T(0);
    eb = ob == 1 ? T(0.75) : T(0);
  }
};

// Sums of the records [l0, l1) of a list grouped by base node (stride kS reals, shared memory) in
// registers while the base node stays the same, then one vector reduction per node into A.  The
// bounds may differ from group to group.  The sums hold momenta as they are: taken relative to a velocity of the
// list, one light or fast particle would cost every node of the list its digits.
template <int DIM, typename T>
__device__ __forceinline__ void run_flush(Node4<T>* at, const T (&acc)[DIM == 3 ? 3 : 1][4], int64_t RR) {
#pragma unroll
  for (int i = 0; i < (DIM == 3 ? 3 : 1); ++i) atomic_add4(at + i * RR, acc[i][0], acc[i][1], acc[i][2], acc[i][3]);
}

// A group's sums under way.
template <int DIM, typename T>
struct RunSums {
  static constexpr int NX = RunLane<DIM, T>::NX;
  int cur = -1;  // base node of the run (none yet: negative)
  T acc[NX][4] = {};
  T kept[NX][4] = {};  // kSlide: what the cells before brought to the run's nodes (a sum of cells' sums)
  __device__ __forceinline__ void take_up() {
#pragma unroll
    for (int i = 0; i < NX; ++i)
#pragma unroll
      for (int r = 0; r < 4; ++r) {
        acc[i][r] += kept[i][r];
        kept[i][r] = T(0);
      }
  }
};

// One record's contribution to the lane's nodes.
template <int DIM, typename T>
__device__ __forceinline__ void run_add(T (&acc)[DIM == 3 ? 3 : 1][4], const T* rec, const RunLane<DIM, T>& ln) {
  constexpr int a0 = 1 + DIM, f0 = 1 + DIM + DIM * DIM, NV = RunRec<DIM>::kPacked / 4;
  T rv[4 * NV];
  const Node4<T>* src = reinterpret_cast<const Node4<T>*>(rec);
#pragma unroll
  for (int i = 0; i < NV; ++i) {
    const Node4<T> q4 = src[i];
    rv[4 * i] = q4.x;
    rv[4 * i + 1] = q4.y;
    rv[4 * i + 2] = q4.z;
    rv[4 * i + 3] = q4.w;
  }
  if constexpr (DIM == 3) {
    const T da = rv[f0 + 1] - ln.ra, db = rv[f0 + 2] - ln.rb;
    const T wjk = (ln.ka * da * da + ln.ea) * (ln.kb * db * db + ln.eb);
    T wx[3];
    bspline(rv[f0], wx);
    T b[3];
#pragma unroll
    for (int r = 0; r < 3; ++r)
      b[r] = rv[1 + r] + rv[a0 + 3 * r + 1] * T(ln.oa) + rv[a0 + 3 * r + 2] * T(ln.ob);
#pragma unroll
    for (int i = 0; i < 3; ++i) {
      const T wt = wx[i] * wjk;
#pragma unroll
      for (int r = 0; r < 3; ++r) acc[i][r] += wt * (b[r] + T(i) * rv[a0 + 3 * r]);
      acc[i][3] += wt * rv[0];
    }
  } else {
    const T da = rv[f0] - ln.ra, db = rv[f0 + 1] - ln.rb;
    const T wt = (ln.ka * da * da + ln.ea) * (ln.kb * db * db + ln.eb);
#pragma unroll
    for (int r = 0; r < 2; ++r)
      acc[0][r] += wt * (rv[1 + r] + rv[a0 + 2 * r] * T(ln.oa) + rv[a0 + 2 * r + 1] * T(ln.ob));
    acc[0][3] += wt * rv[0];
  }
}

// kSlide: keep the sums of shared nodes from cell to cell, which leaves a third of the reductions, so that a
// node is a sum of fewer parts; it costs 24 shuffles a cell (the resident solver, 16,384 particles: 668 us a
// call with it, 613 without).
template <int DIM, typename T, int kS, bool kSlide>
__device__ __forceinline__ void run_sums(RunSums<DIM, T>& rs, const T* recs, const int* nodes, int l0, int l1,
                                         const RunLane<DIM, T>& ln, Node4<T>* __restrict__ Al, int64_t RR) {
  constexpr int NX = RunLane<DIM, T>::NX;
  for (int l = l0; l < l1; ++l) {
    const int nd = nodes[l];
    if (nd != rs.cur) {
      if constexpr (kSlide) rs.take_up();
      if (kSlide && nd == rs.cur + 1 && rs.cur >= 0) {
        // the next cell along the grid's last axis shares two thirds of the nodes: the sums move one
        // lane down, and only those that no lane holds any more go to the grid
        const unsigned group = 0x1ffu << (9 * ln.grp);
#pragma unroll
        for (int i = 0; i < NX; ++i) {
          if (ln.ob == 0) atomic_add4(Al + rs.cur + i * RR, rs.acc[i][0], rs.acc[i][1], rs.acc[i][2], rs.acc[i][3]);
#pragma unroll
          for (int r = 0; r < 4; ++r) {
            const T t = __shfl_down_sync(group, rs.acc[i][r], 1);
            rs.kept[i][r] = ln.ob < 2 ? t : T(0);
          }
        }
      } else if (rs.cur >= 0) {
        run_flush<DIM, T>(Al + rs.cur, rs.acc, RR);
      }
#pragma unroll
      for (int i = 0; i < NX; ++i) rs.acc[i][0] = rs.acc[i][1] = rs.acc[i][2] = rs.acc[i][3] = T(0);
      rs.cur = nd;
    }
    run_add<DIM, T>(rs.acc, recs + (size_t)l * kS, ln);
  }
}

// The groups' last runs into A; groups that end in the same run (a cell of many particles) add their
// sums up first.  Every lane of the warp calls it.
template <int DIM, typename T>
__device__ __forceinline__ void run_end(RunSums<DIM, T>& rs, const RunLane<DIM, T>& ln, Node4<T>* __restrict__ Al,
                                        int64_t RR) {
  constexpr unsigned kFull = 0xffffffffu;
  constexpr int NX = RunLane<DIM, T>::NX;
  __syncwarp();
  const int c0 = __shfl_sync(kFull, rs.cur, 0), c1 = __shfl_sync(kFull, rs.cur, 9), c2 = __shfl_sync(kFull, rs.cur, 18);
  if (c1 >= 0 && (c0 == c1 || c1 == c2)) {
#pragma unroll
    for (int to = 1; to >= 0; --to) {
      const bool join = to == 1 ? c1 == c2 : c0 == c1;
#pragma unroll
      for (int i = 0; i < NX; ++i)
#pragma unroll
        for (int r = 0; r < 4; ++r) {
          const T t = __shfl_down_sync(kFull, rs.acc[i][r], 9);
          if (join && ln.grp == to) rs.acc[i][r] += t;
        }
      if (join && ln.grp == to + 1) rs.cur = -1;
    }
  }
  if (rs.cur >= 0) run_flush<DIM, T>(Al + rs.cur, rs.acc, RR);
}

// Scatter of one warp's 32 particles.  Every lane hands in its particle's record (`node`: linear index
// of its base node, negative for none); the records go to the warp's own shared memory grouped by base
// node (lanes with the same base node share all their stencil nodes), a third of the list to each of
// the three groups of lanes.  Particles in cell order so cost about one reduction per node and cell;
// particles in no order cost one per node each, three neighbouring lanes to 48 contiguous bytes.
template <int DIM, typename T>
struct alignas(16) WarpRecs {
  T rec[32][RunRec<DIM>::kSmem];
  int node[32];
};

// The grouping alone: `rec` of every lane with a particle into wr, grouped by node.  Returns how many.
template <int DIM, typename T>
__device__ __forceinline__ int warp_group(WarpRecs<DIM, T>& wr, const T (&rec)[RunRec<DIM>::kPacked], int node,
                                          unsigned vmask) {
  constexpr unsigned kFull = 0xffffffffu;
  const int lane = threadIdx.x & 31;
  const bool valid = node >= 0;
  // slot of the lane's record: the lanes of one base node together, groups in order of first lane
  const unsigned peers = __match_any_sync(kFull, node);
  const unsigned before = peers & lanemask_lt();
  const int mine = valid && before == 0u ? __popc(peers) : 0;
  int inc = mine;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const int t = __shfl_up_sync(kFull, inc, o);
    if (lane >= o) inc += t;
  }
  const int start = __shfl_sync(kFull, inc - mine, __ffs(peers) - 1);
  if (valid) {
    const int slot = start + __popc(before);
    Node4<T>* dst = reinterpret_cast<Node4<T>*>(wr.rec[slot]);
#pragma unroll
    for (int i = 0; i < RunRec<DIM>::kPacked / 4; ++i)
      dst[i] = Node4<T>{rec[4 * i], rec[4 * i + 1], rec[4 * i + 2], rec[4 * i + 3]};
    wr.node[slot] = node;
  }
  __syncwarp();
  return __popc(vmask);
}

template <int DIM, typename T>
__device__ __forceinline__ void warp_scatter(WarpRecs<DIM, T>& wr, const T (&rec)[RunRec<DIM>::kPacked], int node,
                                             const RunLane<DIM, T>& ln, Node4<T>* __restrict__ A, int R) {
  constexpr unsigned kFull = 0xffffffffu;
  const unsigned vmask = __ballot_sync(kFull, node >= 0);
  if (vmask == 0u) return;
  RunSums<DIM, T> rs;
  const int nv = warp_group<DIM, T>(wr, rec, node, vmask);
  const int per = (nv + 2) / 3;
  const int l0 = ln.grp * per;
  const int64_t RR = DIM == 3 ? (int64_t)R * R : 0;
  Node4<T>* const Al = A + (ln.oa * R + ln.ob);
  run_sums<DIM, T, RunRec<DIM>::kSmem, false>(rs, &wr.rec[0][0], wr.node, l0,
                                              ln.grp < 3 ? min(nv, l0 + per) : 0, ln, Al, RR);
  run_end<DIM, T>(rs, ln, Al, RR);
  __syncwarp();  // the records are rewritten by the warp's next particles
}

// Threads per CTA of the warp kernels: at most kWarpCta; small counts take smaller CTAs so that the
// particles spread over the SMs.
template <typename T>
constexpr int kWarpCta = sizeof(T) == 4 ? 256 : 128;

// P2G of particles [p0, p1) (through perm, when given) into the workspace grid A.  `may_give_up`: perm comes from
// the radix sort, whose bounded wait may have left it incomplete.
template <int DIM, typename T>
__global__ void __launch_bounds__(kWarpCta<T>, 2) k_p2g_warp(KParams<T> kp, Geom<DIM> g, PView<T> P,
                                                            const uint32_t* __restrict__ perm, bool may_give_up,
                                                            uint32_t p0, uint32_t p1, Node4<T>* __restrict__ A,
                                                            int32_t* status, uint32_t* fallbacks) {
  dep_wait();
  if (may_give_up && wait_gave_up(status)) return;
  extern __shared__ __align__(128) unsigned char smem_raw[];
  WarpRecs<DIM, T>& wr = reinterpret_cast<WarpRecs<DIM, T>*>(smem_raw)[threadIdx.x >> 5];
  const RunLane<DIM, T> ln;
  const int lane = threadIdx.x & 31;
  for (uint32_t s = p0 + blockIdx.x * blockDim.x + (threadIdx.x & ~31u); s < p1; s += gridDim.x * blockDim.x) {
    T rec[RunRec<DIM>::kPacked];
    int node = -1;
    if (s + lane < p1) {
      P2GIn<DIM, T> in;
      p2g_load<DIM, T>(kp, P, perm ? perm[s + lane] : s + lane, in);
      int base[DIM];
      node = run_record<DIM, T>(kp, in, g.R, rec, status, fallbacks, base);
    }
    warp_scatter<DIM, T>(wr, rec, node, ln, A, g.R);
  }
}

// ----------------------------------------------------------------------------------------------
// Particles in no order: a node then receives hundreds of contributions one at a time, and the sum loses what
// a sum over cells keeps.  So they are put in cell order first, by a counting sort whose counters are the grid's
// nodes:
//   k_cell_rank     each particle's rank among those of its base node (one atomic per warp and node)
//   k_cell_offsets  first slot of every occupied node: tiles of nodes take their slots from one
//                   counter, so the tiles may come in any order and no CTA waits on another
//   k_cell_records  stress and record of every particle, written to its slot
//   k_cell_sums     run sums over the records as they lie
// or, for double particles and few float ones, whose records cost more to write and to wait for than their
// particles to gather:
//   k_cell_perm     the particles' indices in their slots, for k_p2g_warp
// 1,048,576 particles of a random order on 128^3, component-major (GB300): 18 + 5 + 66 + 49 us, where
// the block sort and the chunked scatter through its permutation took 150 + 305 us (every component
// of a particle then came from a sector of its own).  k_cell_records is bound by its scattered 64-byte
// record writes and wants the warps that 80 registers allow (a coarse step of 552 us takes 540 with them),
// k_cell_sums by instruction issue.
constexpr int kCellTile = 4096;      // nodes per CTA of k_cell_offsets
constexpr uint32_t kNoRank = 0xffffffffu;

template <int DIM, typename T>
__device__ __forceinline__ int base_node(const KParams<T>& kp, const PView<T>& P, uint32_t p, int R) {
  int b[DIM];
  bool ok = true;
#pragma unroll
  for (int d = 0; d < DIM; ++d) {
    T fx;
    ok = ok && base_of(P.x[P.at(p, d, DIM)], kp.inv_dx, kp.res, b[d], fx);
  }
  return ok ? (int)node_index<DIM>(R, b) : -1;
}

template <int DIM, typename T>
__global__ void __launch_bounds__(kThreads) k_cell_rank(KParams<T> kp, int R, PView<T> P, uint32_t n,
                                                        uint32_t* __restrict__ count, uint32_t* __restrict__ rank,
                                                        int* __restrict__ node_of) {
  dep_wait();
  const uint32_t p = blockIdx.x * blockDim.x + threadIdx.x;
  const int node = p < n ? base_node<DIM, T>(kp, P, p, R) : -1;
  const unsigned peers = __match_any_sync(0xffffffffu, node);
  const unsigned before = peers & lanemask_lt();
  uint32_t first = 0;
  if (node >= 0 && before == 0u) first = atomicAdd(&count[node], (uint32_t)__popc(peers));
  first = __shfl_sync(0xffffffffu, first, __ffs(peers) - 1);
  if (p < n) {
    rank[p] = node >= 0 ? first + __popc(before) : kNoRank;
    if (node_of) node_of[p] = node;
  }
}

// count -> start (occupied nodes only); the counters go back to zero for the next call.
static __global__ void __launch_bounds__(kThreads) k_cell_offsets(uint32_t* __restrict__ count,
                                                                  uint32_t* __restrict__ start, WsHeader* hdr) {
  dep_wait();
  constexpr int kPer = kCellTile / kThreads;
  static_assert(kPer == 16, "four vectors per thread");
  __shared__ uint32_t warp_sum[kThreads / 32];
  __shared__ uint32_t s_base;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  uint4* c4 = reinterpret_cast<uint4*>(count + (size_t)blockIdx.x * kCellTile) + threadIdx.x * (kPer / 4);
  uint32_t c[kPer];
  uint32_t sum = 0, occ = 0;
#pragma unroll
  for (int i = 0; i < kPer / 4; ++i) {
    const uint4 v = c4[i];
    c[4 * i] = v.x;
    c[4 * i + 1] = v.y;
    c[4 * i + 2] = v.z;
    c[4 * i + 3] = v.w;
  }
#pragma unroll
  for (int i = 0; i < kPer; ++i) {
    sum += c[i];
    occ += c[i] ? 1u : 0u;
  }
  occ = __reduce_add_sync(0xffffffffu, occ);
  if (lane == 0 && occ) atomicAdd(&hdr->cell_occupied, occ);
  uint32_t inc = sum;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const uint32_t t = __shfl_up_sync(0xffffffffu, inc, o);
    if (lane >= o) inc += t;
  }
  if (lane == 31) warp_sum[warp] = inc;
  __syncthreads();
  uint32_t before = 0, total = 0;
#pragma unroll
  for (int w = 0; w < kThreads / 32; ++w) {
    before += w < warp ? warp_sum[w] : 0u;
    total += warp_sum[w];
  }
  if (threadIdx.x == 0) s_base = total ? atomicAdd(&hdr->cell_cursor, total) : 0u;
  __syncthreads();
  if (sum == 0) return;
  uint32_t at = s_base + before + inc - sum;
  uint32_t* st = start + (size_t)blockIdx.x * kCellTile + threadIdx.x * kPer;
#pragma unroll
  for (int i = 0; i < kPer; ++i) {
    if (c[i]) st[i] = at;
    at += c[i];
  }
#pragma unroll
  for (int i = 0; i < kPer / 4; ++i) c4[i] = make_uint4(0u, 0u, 0u, 0u);
}

template <int DIM, typename T>
__global__ void __launch_bounds__(kThreads, 3) k_cell_records(KParams<T> kp, int R, PView<T> P, uint32_t n,
                                                           const uint32_t* __restrict__ rank,
                                                           const uint32_t* __restrict__ start, T* __restrict__ recs,
                                                           int* __restrict__ nodes, int32_t* status,
                                                           uint32_t* fallbacks) {
  dep_wait();
  const uint32_t p = blockIdx.x * blockDim.x + threadIdx.x;
  if (p >= n) return;
  P2GIn<DIM, T> in;
  p2g_load<DIM, T>(kp, P, p, in);
  const uint32_t rk = rank[p];
  T rec[RunRec<DIM>::kPacked];
  int base[DIM];
  const int node = run_record<DIM, T>(kp, in, R, rec, status, fallbacks, base);
  if (node < 0) return;
  const uint32_t at = start[node] + rk;
  nodes[at] = node;
  Node4<T>* dst = reinterpret_cast<Node4<T>*>(recs + (size_t)at * RunRec<DIM>::kPacked);
#pragma unroll
  for (int i = 0; i < RunRec<DIM>::kPacked / 4; ++i)
    dst[i] = Node4<T>{rec[4 * i], rec[4 * i + 1], rec[4 * i + 2], rec[4 * i + 3]};
}

// The particles in cell order as a permutation; those outside the grid, which no cell counted, come last.
static __global__ void __launch_bounds__(kThreads) k_cell_perm(uint32_t n, const uint32_t* __restrict__ rank,
                                                               const int* __restrict__ node_of,
                                                               const uint32_t* __restrict__ start, WsHeader* hdr,
                                                               uint32_t* __restrict__ perm) {
  dep_wait();
  const uint32_t p = blockIdx.x * blockDim.x + threadIdx.x;
  if (p >= n) return;
  const int node = node_of[p];
  perm[node >= 0 ? start[node] + rank[p] : hdr->cell_cursor + atomicAdd(&hdr->cell_outside, 1u)] = p;
}

// A warp sums a stretch of consecutive records, 96 at a time: they come to shared memory by asynchronous copies,
// while the SM's other warps sum theirs.  A run that crosses the end of a stretch belongs to the stretch it
// begins in when it began within the last 32 records, up to 32 records past the end.
//   Cells of a few particles: each group of lanes takes a third of the 96 (a stretch each), and keeps the sums of
// shared nodes from cell to cell along the last axis (run_sums).
//   Fuller cells: a third would be one or two cells, and a node would receive nearly a part per cell, added in
// no order.  So the groups share each run, add up what they have of it, and the warp goes from cell to cell with
// the sums of shared nodes.  Float error of a corrected coarse step beside that of sums in block-sorted chunks
// of 512: 0.97 times at 31 particles a cell (1,048,576 particles, 128^3), 1.07 at 24 (100,000, 64^3), 1.10 at 95
// (400,000, 64^3), where thirds have 1.16, 1.24 and 1.32; as fast (541, 101 and 230 us, from 538, 103 and 238).
// At 9 particles a cell it is slower (50,000 on 64^3: 93 us, 88 with thirds), for little (1.04, 1.09).
template <int DIM, typename T>
struct alignas(16) WarpStage {
  static constexpr int kPitch = 33;  // slots per group: the groups' reads fall on distinct banks
  T rec[3 * kPitch][RunRec<DIM>::kSmem];
  int node[3 * kPitch];
};

// How far past `at` the run that crosses it goes, when it belongs to the records before `at`.
__device__ __forceinline__ int run_shift(const int* __restrict__ nodes, int at, int total) {
  const int lane = threadIdx.x & 31;
  const auto node = [&](int i) { return i >= 0 && i < total ? nodes[i] : -1; };
  const unsigned before = __ballot_sync(0xffffffffu, node(at - 32 + lane) != node(at - 33 + lane));
  const unsigned after = __ballot_sync(0xffffffffu, node(at + lane) != node(at + lane - 1));
  return !(after & 1u) && before ? (after ? __ffs(after) - 1 : 32) : 0;
}

constexpr int kFullCell = 14;  // particles a cell (mean) from which the groups share runs: two cells to a third

template <int DIM, typename T>
__global__ void __launch_bounds__(64) k_cell_sums(int R, const T* __restrict__ recs, const int* __restrict__ nodes,
                                                  const WsHeader* hdr, Node4<T>* __restrict__ A) {
  dep_wait();
  static_assert(sizeof(T) == 4, "16-byte copies of Node4<float>");
  constexpr int NV = RunRec<DIM>::kPacked / 4, kS = RunRec<DIM>::kSmem, kPitch = WarpStage<DIM, T>::kPitch;
  extern __shared__ __align__(128) unsigned char smem_raw[];
  WarpStage<DIM, T>& ws = reinterpret_cast<WarpStage<DIM, T>*>(smem_raw)[threadIdx.x >> 5];
  const RunLane<DIM, T> ln;
  const int lane = threadIdx.x & 31;
  const int total = (int)hdr->cell_cursor;
  if (total == 0) return;
  const int mean = total / (int)max(1u, hdr->cell_occupied);
  const bool full = mean >= kFullCell;
  const int stages = mean < 64 ? 1 : min(16, mean / 24);
  const int64_t s0 = (int64_t)(blockIdx.x * 2 + (threadIdx.x >> 5)) * 96 * stages;
  if (s0 >= total) return;
  const auto stretch_at = [&](int64_t at) {
    return at < total ? (int)at + run_shift(nodes, (int)at, total) : total;
  };
  // records [b, b + nr) to slots from `slot` on (every lane calls it)
  const auto fetch = [&](int slot, int b, int nr) {
    for (int q = lane; q < nr * NV; q += 32) {
      const int r = q / NV, c = q - r * NV;
      asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(smem_u32(&ws.rec[slot + r][4 * c])),
                   "l"(recs + (size_t)(b + r) * RunRec<DIM>::kPacked + 4 * c)
                   : "memory");
    }
    for (int r = lane; r < nr; r += 32) ws.node[slot + r] = nodes[b + r];
  };
  const int64_t RR = DIM == 3 ? (int64_t)R * R : 0;
  Node4<T>* const Al = A + (ln.oa * R + ln.ob);
  RunSums<DIM, T> rs;
  if (!full) {
    const int lo[4] = {stretch_at(s0), stretch_at(s0 + 32), stretch_at(s0 + 64), stretch_at(s0 + 96)};
    const int len = max(max(lo[1] - lo[0], lo[2] - lo[1]), lo[3] - lo[2]);
    const int my_len = ln.grp == 0 ? lo[1] - lo[0] : ln.grp == 1 ? lo[2] - lo[1] : ln.grp == 2 ? lo[3] - lo[2] : 0;
    for (int k = 0; k < len; k += 32) {
#pragma unroll
      for (int g = 0; g < 3; ++g) fetch(kPitch * g, lo[g] + k, min(32, lo[g + 1] - lo[g] - k));
      asm volatile("cp.async.wait_all;" ::: "memory");
      __syncwarp();
      const int l0 = kPitch * min(ln.grp, 2);
      run_sums<DIM, T, kS, true>(rs, &ws.rec[0][0], ws.node, l0, l0 + max(0, min(32, my_len - k)), ln, Al, RR);
      __syncwarp();
    }
    rs.take_up();
    run_end<DIM, T>(rs, ln, Al, RR);
    return;
  }
  constexpr unsigned kAll = 0xffffffffu;
  constexpr int NX = RunLane<DIM, T>::NX;
  const int hi = stretch_at(s0 + 96 * stages);
  for (int b = stretch_at(s0); b < hi; b += 96) {
    const int nr = min(96, hi - b);
    fetch(0, b, nr);
    asm volatile("cp.async.wait_all;" ::: "memory");
    __syncwarp();
    for (int l = 0; l < nr;) {
      // the run's end: the first of the next 32 records with another node, if any
      const int nd = ws.node[l];
      int e = l;
      unsigned other;
      do {
        const int i = e + lane;
        other = __ballot_sync(kAll, i >= nr || ws.node[min(i, nr - 1)] != nd);
        e += other ? __ffs(other) - 1 : 32;
      } while (!other);
      if (nd != rs.cur) {  // rs.acc: the first group's lanes hold the sums of the cells before
        const bool next = nd == rs.cur + 1 && rs.cur >= 0;
#pragma unroll
        for (int i = 0; i < NX; ++i) {
          if (ln.grp == 0 && rs.cur >= 0 && (!next || ln.ob == 0))
            atomic_add4(Al + rs.cur + i * RR, rs.acc[i][0], rs.acc[i][1], rs.acc[i][2], rs.acc[i][3]);
#pragma unroll
          for (int r = 0; r < 4; ++r) {
            const T t = __shfl_down_sync(kAll, rs.acc[i][r], 1);
            rs.acc[i][r] = next && ln.ob < 2 ? t : T(0);
          }
        }
        rs.cur = nd;
      }
      T part[NX][4] = {};
      const int per = (e - l + 2) / 3, l0 = l + ln.grp * per, l1 = ln.grp < 3 ? min(e, l0 + per) : 0;
      for (int q = l0; q < l1; ++q) run_add<DIM, T>(part, &ws.rec[q][0], ln);
      __syncwarp();
#pragma unroll
      for (int i = 0; i < NX; ++i)
#pragma unroll
        for (int r = 0; r < 4; ++r)
          rs.acc[i][r] += part[i][r] + (__shfl_down_sync(kAll, part[i][r], 9) + __shfl_down_sync(kAll, part[i][r], 18));
      l = e;
    }
    __syncwarp();
  }
  if (ln.grp == 0 && rs.cur >= 0) run_flush<DIM, T>(Al + rs.cur, rs.acc, RR);
}

// Grid update of every node (three_d/grid_op.py:5-47 / two_d/grid_op.py:5-24): momentum of A ->
// velocity in B, A re-zeroed.  B is written at every node: one whose sums are all zero has velocity zero, and
// particles do read it (without mass and stress at full weight; half a cell from their neighbours at weight
// zero, which an infinity left there by an earlier call would still spoil).  Writing it (450,000 particles on
// 128^3, four substeps: 840 us, 834 without) is cheaper than to read first whether it holds a value (854).
template <int DIM, typename T>
__global__ void __launch_bounds__(kThreads) k_grid_update_dense(KParams<T> kp, Geom<DIM> g, WsHeader* hdr,
                                                                Node4<T>* __restrict__ A, Node4<T>* __restrict__ B) {
  dep_wait();
  const int R = g.R;
  const int64_t nn = DIM == 3 ? (int64_t)R * R * R : (int64_t)R * R;
  if (blockIdx.x == 0 && threadIdx.x == 0) hdr->cell_cursor = hdr->cell_occupied = hdr->cell_outside = 0u;  // for the next call
  constexpr int U = 4;  // nodes of a thread in flight
  const int64_t stride = (int64_t)gridDim.x * blockDim.x;
  for (int64_t n0 = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; n0 < nn; n0 += U * stride) {
    Node4<T> a[U];
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const int64_t node = n0 + u * stride;
      a[u] = node < nn ? A[node] : Node4<T>{T(0), T(0), T(0), T(0)};
    }
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const int64_t node = n0 + u * stride;
      if (a[u].x == T(0) && a[u].y == T(0) && a[u].z == T(0) && a[u].w == T(0)) {
        if (node < nn) B[node] = Node4<T>{T(0), T(0), T(0), T(0)};
        continue;
      }
      int I[DIM];
      const uint32_t nu = (uint32_t)node;  // below 2^31: the sort keys bound the grid
      if constexpr (DIM == 3) {
        I[0] = (int)(nu / ((uint32_t)R * (uint32_t)R));
        I[1] = (int)((nu / (uint32_t)R) % (uint32_t)R);
        I[2] = (int)(nu % (uint32_t)R);
      } else {
        I[0] = (int)(nu / (uint32_t)R);
        I[1] = (int)(nu % (uint32_t)R);
      }
      T vel[3] = {a[u].x, a[u].y, a[u].z};
      grid_node<DIM, T>(kp, I, vel, a[u].w);
      B[node] = Node4<T>{vel[0], vel[1], vel[2], a[u].w};
      A[node] = Node4<T>{T(0), T(0), T(0), T(0)};
    }
  }
}

// G2P of particles [p0, p1) in place, every stencil gathered from the global velocity grid B.
template <int DIM, typename T>
__global__ void __launch_bounds__(kWarpCta<T>, sizeof(T) == 4 ? 3 : 1) k_g2p_range(KParams<T> kp, Geom<DIM> g, PView<T> P, uint32_t p0,
                                                           uint32_t p1, const Node4<T>* __restrict__ B,
                                                           int32_t* status) {
  dep_wait();
  G2PExtra ex{};
  ex.grid_global = B;
  int org[DIM];
#pragma unroll
  for (int d = 0; d < DIM; ++d) org[d] = -(1 << 24);  // no staged tile: every stencil is off-tile
  const bool need_jp = (DIM == 2) || kp.model == FFMPM_MODEL_SNOW;
  for (uint32_t p = p0 + blockIdx.x * blockDim.x + threadIdx.x; p < p1; p += gridDim.x * blockDim.x) {
    G2PIn<DIM, T> in;
    g2p_load<DIM, T>(P, p, need_jp, in);
    g2p_particle<DIM, T>(kp, g, P, P, p, p, org, nullptr, status, false, ex, in);
  }
}

// ----------------------------------------------------------------------------------------------
// Fused G2P + P2G of the resident solver: substep k's G2P and substep k+1's P2G in one pass over the
// particles.  The updated particle (x, v, C, F) goes straight from the gather into the next substep's
// record, so v and C never travel through memory between the two, and x and F are read once per
// substep.  A warp takes 32 particles of the solver's cell order: its gathers fall on the nodes of a few
// cells, its scatter is warp_scatter's (the particles that crossed a cell boundary since the last re-sort
// join the run of their new cell there).  The grid update visits the blocks the plan touches: a
// particle whose new stencil may leave them adds the blocks it covers to the list itself.
// Two cubes of 1,048,576 particles on 128^3 (GB300): 106 us a launch; chunks of 512 particles with a
// shared-memory tile for each side, an in-chunk counting sort and CTA barriers between the phases took
// 156.  16,384 particles on 64^3: 13 us a substep against 40 (512 one-warp batches instead of 32 chunks).
// Bound by instruction issue and the latency of the gathers.

// Add the blocks covered by the stencil at `base` to the touched list (each block once: `tmark` is
// nonzero for every listed block; 2 where the blocks of every stencil based in the block are listed).
template <int DIM>
__device__ __forceinline__ void mark_touched(const Geom<DIM>& g, const int base[DIM], uint32_t* tmark,
                                             uint32_t* touched, uint32_t* n_touched) {
  int lo[DIM], ext[DIM];
  int id = 0;
#pragma unroll
  for (int d = 0; d < DIM; ++d) {
    lo[d] = base[d] >> g.bs_shift;
    ext[d] = min((base[d] + 2) >> g.bs_shift, g.nb - 1) - lo[d];  // 0 or 1
    id = id * g.nb + lo[d];
  }
  if (__ldcg(&tmark[id]) == 2u) return;
  for (int o = 0; o < (1 << DIM); ++o) {
    int at = 0;
    bool ok = true;
#pragma unroll
    for (int d = 0; d < DIM; ++d) {
      const int od = (o >> (DIM - 1 - d)) & 1;
      ok = ok && od <= ext[d];
      at = at * g.nb + lo[d] + od;
    }
    if (ok && __ldcg(&tmark[at]) == 0u && atomicCAS(&tmark[at], 0u, 1u) == 0u)
      touched[atomicAdd(n_touched, 1u)] = (uint32_t)at;
  }
}

// kNext: G2P and the next substep's P2G; else the last substep's G2P alone (which writes v and C).
template <int DIM, typename T, bool kNext>
__global__ void __launch_bounds__(kWarpCta<T>, sizeof(T) == 4 ? 2 : 1) k_g2p_sorted(
    KParams<T> kp, Geom<DIM> g, PView<T> Pin, PView<T> Pout, const uint32_t* __restrict__ perm, uint32_t n,
    G2PExtra ex, Node4<T>* __restrict__ A, WsHeader* hdr, uint32_t* __restrict__ tmark,
    uint32_t* __restrict__ touched) {
  dep_wait();
  int32_t* const status = &hdr->status;
  if (perm && wait_gave_up(status)) return;
  extern __shared__ __align__(128) unsigned char smem_raw[];
  WarpRecs<DIM, T>& wr = reinterpret_cast<WarpRecs<DIM, T>*>(smem_raw)[kNext ? threadIdx.x >> 5 : 0];
  const RunLane<DIM, T> ln;
  const int lane = threadIdx.x & 31;
  int org[DIM];
#pragma unroll
  for (int d = 0; d < DIM; ++d) org[d] = -(1 << 24);  // no staged tile: every stencil is off-tile
  for (uint32_t s0 = blockIdx.x * blockDim.x + (threadIdx.x & ~31u); s0 < n; s0 += gridDim.x * blockDim.x) {
    const uint32_t s = s0 + lane;
    T rec[RunRec<DIM>::kPacked];
    int node = -1;
    if (s < n) {
      const uint32_t p = perm ? perm[s] : s;
      G2PIn<DIM, T> in;
      g2p_load<DIM, T>(Pin, p, true, in);
      P2GIn<DIM, T> nx;
      if (g2p_particle<DIM, T, kNext>(kp, g, Pin, Pout, p, s, org, nullptr, status, true, ex, in, &nx)) {
        if constexpr (kNext) {
          int base[DIM];
          node = run_record<DIM, T>(kp, nx, g.R, rec, status, &hdr->polar_fallbacks, base);
          if (node >= 0) mark_touched<DIM>(g, base, tmark, touched, &hdr->n_touched);
        }
      }
    }
    if constexpr (kNext) warp_scatter<DIM, T>(wr, rec, node, ln, A, g.R);
  }
}

// The sums of A (momentum xyz, mass) added into a caller's grid_velocity [nodes][DIM] and grid_mass
// [nodes]; A re-zeroed.  Atomically, as the block-sorted form adds: another stream may add other particles
// (over another workspace) to the same grid.
template <int DIM, typename T>
__global__ void __launch_bounds__(kThreads) k_grid_fold_user(int64_t nn, WsHeader* hdr, Node4<T>* __restrict__ A, T* __restrict__ gv,
                                                             T* __restrict__ gm) {
  dep_wait();
  if (blockIdx.x == 0 && threadIdx.x == 0) hdr->cell_cursor = hdr->cell_occupied = hdr->cell_outside = 0u;  // for the next call
  for (int64_t node = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; node < nn;
       node += (int64_t)gridDim.x * blockDim.x) {
    const Node4<T> a = A[node];
    if (a.x == T(0) && a.y == T(0) && a.z == T(0) && a.w == T(0)) continue;
    atomicAdd(&gv[node * DIM + 0], a.x);
    atomicAdd(&gv[node * DIM + 1], a.y);
    if constexpr (DIM == 3) atomicAdd(&gv[node * DIM + 2], a.z);
    atomicAdd(&gm[node], a.w);
    A[node] = Node4<T>{T(0), T(0), T(0), T(0)};
  }
}

// A caller's grid_velocity [nodes][DIM] into the workspace's B (one aligned vector per node).
template <int DIM, typename T>
__global__ void __launch_bounds__(kThreads) k_grid_pack_user(int64_t nn, const T* __restrict__ gv,
                                                             Node4<T>* __restrict__ B) {
  dep_wait();
  for (int64_t node = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; node < nn;
       node += (int64_t)gridDim.x * blockDim.x) {
    T v[3] = {gv[node * DIM + 0], gv[node * DIM + 1], T(0)};
    if constexpr (DIM == 3) v[2] = gv[node * DIM + 2];
    B[node] = Node4<T>{v[0], v[1], v[2], T(0)};
  }
}

}  // namespace ffmpm
