// extern "C" entry points of libfemflow_mpm.so (declared in include/femflow_mpm.h) and the host
// code that sequences the kernels of a substep on the caller's stream.
#include <cuda.h>
#include <cuda_runtime.h>
#include <cudaTypedefs.h>

#include <algorithm>
#include <cstddef>
#include <cstring>
#include <map>
#include <mutex>
#include <vector>

#include "common.cuh"
#include "device_once.h"
#include "internal.h"
#include "mpm_kernels.cuh"
#include "warp_kernels.cuh"

namespace ffmpm {

namespace {

size_t align_up(size_t v, size_t a) { return (v + a - 1) / a * a; }

// The Python mirror (_native.Params / Particles, ctypes) relies on these layouts; its test checks
// the same sizes.
static_assert(sizeof(ffmpm_params) == 504, "ffmpm_params layout");
static_assert(sizeof(ffmpm_particles) == 80, "ffmpm_particles layout");

int ilog2_ceil(int64_t v) {
  int b = 0;
  while ((int64_t(1) << b) < v) ++b;
  return b;
}

int default_block_size(int dim, bool det) {
  if (dim == 3) return det ? 4 : 8;
  return det ? 8 : 16;
}

bool valid_params(const ffmpm_params* p) {
  if (!p) return false;
  if (p->dim != 2 && p->dim != 3) return false;
  if (p->real_bytes != 4 && p->real_bytes != 8) return false;
  if (p->res < 3 || p->res > 4096) return false;
  if (p->model != FFMPM_MODEL_NEO_HOOKEAN && p->model != FFMPM_MODEL_SNOW && p->model != FFMPM_MODEL_FIXED_COROTATED)
    return false;
  if (p->wall_mode != FFMPM_WALLS_REFERENCE && p->wall_mode != FFMPM_WALLS_STICKY3) return false;
  if (p->block_size != 0 && (p->block_size < 2 || p->block_size > 16 || (p->block_size & (p->block_size - 1))))
    return false;
  if (p->n_planes < 0 || p->n_planes > FFMPM_MAX_PLANES) return false;
  if (p->plane_rule != FFMPM_PLANES_STICKY && p->plane_rule != FFMPM_PLANES_REFERENCE_LITERAL) return false;
  for (int q = 0; q < p->n_planes; ++q) {
    double ss = 0.0;
    for (int d = 0; d < 6; ++d)
      if (!std::isfinite(p->planes[q][d])) return false;
    for (int d = 0; d < p->dim; ++d) ss += p->planes[q][3 + d] * p->planes[q][3 + d];
    if (!(ss > 0.0)) return false;
  }
  return true;
}

// One substep (or one phase) on the caller's arrays without a block sort (warp_kernels.cuh): the
// default outside the deterministic mode and the P2G variants.  Its grid pass visits every node (9 us at 2.1 M
// nodes), so a grid that is large against the particle count keeps the sorted form, which visits the touched
// blocks only.  The line is on the safe side of where the two cross: four substeps of 20,000 particles take 536 us
// sorted and 478 unsorted on 192^3 (7.2 M nodes), 545 and 683 on 255^3; of 200,000 particles 979 and 636, 1,434 and
// 877.
bool unsorted(const ffmpm_params& p, const Layout& L) {
  return !p.deterministic && (p.variant & (kVariantP2GDirect | kVariantP2GLanes)) == 0 &&
         L.nnodes <= std::max<int64_t>(int64_t(1) << 22, 16 * L.n);
}

// How such an operation scatters particles that may lie in any order (warp_kernels.cuh), unless the caller keeps
// them near cell order (kVariantCellOrder).  As they come, a node sums its particles one after another, and the float
// error of a substep's C grows, beside that of the block sort, with the particles of a cell: 1.01 times for 2,048 in
// 3D at 4, 1.02 for 4,096 at 8, 1.04 for 2,000 in 2D at 6, 1.12 for 4,000 at 12, and 5 times for many at 30.  Small
// counts, whose cells hold few, are scattered so all the same: one launch does the work of four (2,048 particles,
// eight substeps: 333 us, 416 in cell order).
// Double particles, and no more float ones than kRecordsMin, are put in order as a permutation: records in cell
// order (float64 ones of 128 bytes) take three times as long (200,000 in 2D, four substeps: 2,590 us, 917 as a
// permutation and 1,154 as they come).
enum class ScatterForm { kAsTheyCome, kPermuted, kRecords };
constexpr int64_t kRecordsMin = 4096;
ScatterForm scatter_form(const ffmpm_params& p, const Layout& L) {
  if (p.deterministic || (p.variant & kVariantCellOrder) || L.n <= (p.dim == 3 ? 4096 : 2048) ||
      L.nnodes > std::max<int64_t>(int64_t(1) << 22, 16 * L.n))
    return ScatterForm::kAsTheyCome;
  return p.real_bytes == 8 || L.n <= kRecordsMin ? ScatterForm::kPermuted : ScatterForm::kRecords;
}

}  // namespace

bool make_layout(const ffmpm_params& p, int64_t n, Layout* L) {
  // below 2^30 particles: the radix sort's look-back words carry 30-bit counts
  if (!valid_params(&p) || n < 0 || n >= (int64_t(1) << 30)) return false;
  L->dim = p.dim;
  L->real_bytes = p.real_bytes;
  L->res = p.res;
  L->R = p.res + 1;
  L->bs = p.block_size ? p.block_size : default_block_size(p.dim, p.deterministic != 0);
  L->nb = (L->R + L->bs - 1) / L->bs;
  L->tile = L->bs + 2;
  L->nblocks = p.dim == 3 ? int64_t(L->nb) * L->nb * L->nb : int64_t(L->nb) * L->nb;
  L->nnodes = p.dim == 3 ? int64_t(L->R) * L->R * L->R : int64_t(L->R) * L->R;
  // keys order particles by block, then by cell inside the block, so that each P2G chunk spans few
  // cells (between re-sorts the P2G regroups each chunk by cell itself)
  L->cell_bits = p.dim * ilog2_ceil(L->bs);
  L->key_bits = ilog2_ceil(L->nblocks) + L->cell_bits;
  if (L->key_bits > 31) return false;
  L->passes = std::max(1, (L->key_bits + 7) / 8);
  if (L->passes > kMaxRadixPasses) return false;
  L->n = n;
  L->ntiles = std::max<int64_t>(1, (n + radix_tile(n) - 1) / radix_tile(n));
  L->max_chunks = (n + kChunk - 1) / kChunk + L->nblocks;
  const size_t node_bytes = size_t(4) * p.real_bytes;
  const int64_t tile_nodes = p.dim == 3 ? int64_t(L->tile) * L->tile * L->tile : int64_t(L->tile) * L->tile;
  size_t off = sizeof(WsHeader);
  auto take = [&](size_t bytes) {
    const size_t o = off;
    off = align_up(off + bytes, 256);
    return o;
  };
  L->off_block_count = take(sizeof(uint32_t) * L->nblocks);
  L->off_block_start = take(sizeof(uint32_t) * L->nblocks);
  L->off_block_cnt = take(sizeof(uint32_t) * L->nblocks);
  L->off_chunks = take(sizeof(int4) * L->max_chunks);
  L->off_touched = take(sizeof(uint32_t) * L->nblocks);
  L->off_tmark = take(sizeof(uint32_t) * L->nblocks);
  L->off_occupied = take(sizeof(int4) * L->nblocks);
  L->off_keys_next = take(sizeof(uint32_t) * std::max<int64_t>(n, 1));
  L->off_keys0 = take(sizeof(uint32_t) * std::max<int64_t>(n, 1));
  L->off_keys1 = take(sizeof(uint32_t) * std::max<int64_t>(n, 1));
  L->off_vals0 = take(sizeof(uint32_t) * std::max<int64_t>(n, 1));
  L->off_vals1 = take(sizeof(uint32_t) * std::max<int64_t>(n, 1));
  L->off_hist = take(sizeof(uint32_t) * radix_scratch_words(L->passes, L->ntiles));
  L->off_gridA = take(node_bytes * L->nnodes);
  L->off_gridB = take(node_bytes * L->nnodes);
  L->off_stage = take(p.deterministic ? node_bytes * tile_nodes * L->nblocks : 0);
  // the plan kernels' per-block prefixes (3 x nblocks) and per-CTA totals and offsets
  L->off_plan_pref = take(sizeof(uint32_t) * 3 * L->nblocks);
  L->off_plan_cta = take(2 * 16 * ((L->nblocks + kPlanCta - 1) / kPlanCta));
  // the counting sort by cell of the unsorted operations (warp_kernels.cuh): counters and first slots
  // per node, and the records in cell order
  const ScatterForm form = scatter_form(p, *L);
  if (form != ScatterForm::kAsTheyCome) {
    const size_t cells = align_up(size_t(L->nnodes), kCellTile);
    L->off_cell_count = take(sizeof(uint32_t) * cells);
    L->off_cell_start = take(sizeof(uint32_t) * cells);
  }
  if (form == ScatterForm::kRecords)
    L->off_recs = take(sizeof(float) * (p.dim == 3 ? RunRec<3>::kPacked : RunRec<2>::kPacked) * n);
  L->total = off;
  return true;
}

bool allow_smem(const void* kernel, size_t bytes) {
  static DeviceOnce once;
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess) return false;
  return once.run(dev, kernel, [&] {
    if (cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes) == cudaSuccess) return true;
    cudaGetLastError();
    return false;
  });
}

int sm_count() {
  static int cached = 0;
  if (!cached) {
    int dev = 0;
    cudaGetDevice(&dev);
    int v = 0;
    cudaDeviceGetAttribute(&v, cudaDevAttrMultiProcessorCount, dev);
    cached = v > 0 ? v : 148;
  }
  return cached;
}

namespace {

PFN_cuTensorMapEncodeTiled_v12000 encode_fn() {
  static PFN_cuTensorMapEncodeTiled_v12000 fn = nullptr;
  static std::once_flag once;
  std::call_once(once, [] {
    void* ptr = nullptr;
    cudaDriverEntryPointQueryResult q;
    if (cudaGetDriverEntryPointByVersion("cuTensorMapEncodeTiled", &ptr, 12000, cudaEnableDefault, &q) ==
            cudaSuccess &&
        q == cudaDriverEntryPointSuccess)
      fn = reinterpret_cast<PFN_cuTensorMapEncodeTiled_v12000>(ptr);
  });
  return fn;
}

// Tensor map of a dense grid of Node4 records: dims (4 components, R, R[, R]) innermost first.
bool encode_grid_map(CUtensorMap* map, void* base, const Layout& L) {
  auto fn = encode_fn();
  if (!fn) return false;
  const CUtensorMapDataType dt = L.real_bytes == 4 ? CU_TENSOR_MAP_DATA_TYPE_FLOAT32 : CU_TENSOR_MAP_DATA_TYPE_FLOAT64;
  const cuuint64_t eb = L.real_bytes;
  cuuint64_t dims[4] = {4, (cuuint64_t)L.R, (cuuint64_t)L.R, (cuuint64_t)L.R};
  cuuint64_t strides[3] = {4 * eb, 4 * eb * L.R, 4 * eb * L.R * L.R};  // bytes, dims 1..rank-1
  cuuint32_t box[4] = {4, (cuuint32_t)L.tile, (cuuint32_t)L.tile, (cuuint32_t)L.tile};
  cuuint32_t estr[4] = {1, 1, 1, 1};
  const cuuint32_t rank = L.dim == 3 ? 4 : 3;
  CUresult r = fn(map, dt, rank, base, dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
                  CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  return r == CUDA_SUCCESS;
}

template <int DIM>
Geom<DIM> geom(const Layout& L) {
  Geom<DIM> g;
  g.res = L.res;
  g.R = L.R;
  g.bs = L.bs;
  g.bs_shift = __builtin_ctz((unsigned)L.bs);
  g.nb = L.nb;
  g.nblocks = (int)L.nblocks;
  g.tile = L.tile;
  return g;
}

struct Ws {
  unsigned char* base;
  WsHeader* hdr;
  uint32_t *block_count, *block_start, *block_cnt, *touched, *tmark, *keys_next, *keys0, *keys1, *vals0, *vals1, *hist;
  int4 *chunks, *occupied;
  void *gridA, *gridB, *stage;
  uint32_t* plan_pref;
  Scan4 *cta_tot, *cta_off;
  uint32_t *cell_count, *cell_start;
  void* recs;
};

Ws bind(void* ws, const Layout& L) {
  Ws w;
  w.base = static_cast<unsigned char*>(ws);
  w.hdr = reinterpret_cast<WsHeader*>(w.base);
  w.block_count = reinterpret_cast<uint32_t*>(w.base + L.off_block_count);
  w.block_start = reinterpret_cast<uint32_t*>(w.base + L.off_block_start);
  w.block_cnt = reinterpret_cast<uint32_t*>(w.base + L.off_block_cnt);
  w.chunks = reinterpret_cast<int4*>(w.base + L.off_chunks);
  w.touched = reinterpret_cast<uint32_t*>(w.base + L.off_touched);
  w.tmark = reinterpret_cast<uint32_t*>(w.base + L.off_tmark);
  w.occupied = reinterpret_cast<int4*>(w.base + L.off_occupied);
  w.keys_next = reinterpret_cast<uint32_t*>(w.base + L.off_keys_next);
  w.keys0 = reinterpret_cast<uint32_t*>(w.base + L.off_keys0);
  w.keys1 = reinterpret_cast<uint32_t*>(w.base + L.off_keys1);
  w.vals0 = reinterpret_cast<uint32_t*>(w.base + L.off_vals0);
  w.vals1 = reinterpret_cast<uint32_t*>(w.base + L.off_vals1);
  w.hist = reinterpret_cast<uint32_t*>(w.base + L.off_hist);
  w.gridA = w.base + L.off_gridA;
  w.gridB = w.base + L.off_gridB;
  w.stage = w.base + L.off_stage;
  w.plan_pref = reinterpret_cast<uint32_t*>(w.base + L.off_plan_pref);
  w.cta_tot = reinterpret_cast<Scan4*>(w.base + L.off_plan_cta);
  w.cta_off = w.cta_tot + (L.nblocks + kPlanCta - 1) / kPlanCta;
  w.cell_count = reinterpret_cast<uint32_t*>(w.base + L.off_cell_count);
  w.cell_start = reinterpret_cast<uint32_t*>(w.base + L.off_cell_start);
  w.recs = w.base + L.off_recs;
  return w;
}

int check_launch() {
  const cudaError_t e = cudaGetLastError();
  return e == cudaSuccess ? FFMPM_OK : FFMPM_ERR_CUDA;
}

int work_grid(int64_t max_items, int per_sm) {
  const int64_t cap = int64_t(sm_count()) * per_sm;
  return (int)std::max<int64_t>(1, std::min<int64_t>(max_items, cap));
}

// Resident CTAs per SM of `kernel` at kThreads threads and `smem` dynamic bytes (cached), so the
// chunk-loop kernels launch exactly one wave.
template <typename F>
int resident_per_sm(F* kernel, size_t smem) {
  static std::mutex mu;
  static std::map<std::pair<const void*, size_t>, int> cache;
  std::lock_guard<std::mutex> lock(mu);
  const auto key = std::make_pair(reinterpret_cast<const void*>(kernel), smem);
  auto it = cache.find(key);
  if (it != cache.end()) return it->second;
  int nb = 0;
  if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&nb, kernel, kThreads, smem) != cudaSuccess || nb < 1) nb = 1;
  cache[key] = nb;
  return nb;
}

// Optional per-phase CUDA-event timer of the profiling entry point.
struct PhaseTimer {
  std::vector<cudaEvent_t> ev;     // pairs (start, stop)
  std::vector<int> phase;
  std::vector<int> launches;
  cudaStream_t s = nullptr;
  void begin(int ph) {
    cudaEvent_t e0, e1;
    cudaEventCreate(&e0);
    cudaEventCreate(&e1);
    cudaEventRecord(e0, s);
    ev.push_back(e0);
    ev.push_back(e1);
    phase.push_back(ph);
  }
  void end(int nlaunch) {
    cudaEventRecord(ev.back(), s);
    launches.push_back(nlaunch);
  }
  void collect(double* ms, int64_t* cnt) {
    cudaStreamSynchronize(s);
    for (size_t i = 0; i < phase.size(); ++i) {
      float t = 0.f;
      cudaEventElapsedTime(&t, ev[2 * i], ev[2 * i + 1]);
      ms[phase[i]] += t;
      cnt[phase[i]] += launches[i];
    }
    for (auto e : ev) cudaEventDestroy(e);
    ev.clear();
  }
};

// Substeps between re-sorts (ffmpm_params.variant bits 8..15; 0 or 1: every substep).  The
// deterministic mode always re-sorts (the CTA that sums a block needs every particle in that block).
int sort_every(const ffmpm_params& p) {
  const int k = (p.variant >> kVariantSortShift) & 0xFF;
  return (p.deterministic || k < 1) ? 1 : k;
}

// Start of a substep of a cadenced run: re-sort when the cadence says so or when the previous
// G2P saw a particle leave the neighbourhood its block's plan covers.
__global__ void k_sort_decide(WsHeader* h, int periodic) {
  h->sort_now = (periodic || h->far_stray) ? 1u : 0u;
  h->far_stray = 0u;
}

// keys -> sort -> plan.  Leaves the permutation pointer in *perm.  With `flag` (cadenced runs) the
// sort and the plan do their work only when the device word reads 1.  With `sym` (default: with a
// flag) the plan dilates the occupied blocks by +-1 so that it stays valid until the next re-sort.
template <int DIM, typename T>
void sort_and_plan(const ffmpm_params& p, const Layout& L, const Ws& w, const PView<T>& x, bool keys_ready,
                   const uint32_t** perm, cudaStream_t s, PhaseTimer* tm = nullptr, const uint32_t* flag = nullptr,
                   int sym = -1) {
  const KParams<T> kp = kparams<T>(p);
  const Geom<DIM> g = geom<DIM>(L);
  const uint32_t n = (uint32_t)L.n;
  if (!keys_ready) {
    if (tm) tm->begin(0);
    launch(false, k_keys<DIM, T>, (n + kThreads - 1) / kThreads, kThreads, 0, s, kp, g, x, n, L.cell_bits, w.keys_next,
                                                                       w.block_count, &w.hdr->status);
    if (tm) tm->end(1);
  }
  const uint32_t* ks = nullptr;
  if (tm) tm->begin(1);
  radix_sort(w.keys_next, n, L.passes, w.keys0, w.keys1, w.vals0, w.vals1, w.hist, radix_tile(L.n), &w.hdr->status, s,
             &ks, perm, flag, p.wait_limit, p.inject);
  if (tm) tm->end(1 + L.passes);
  if (tm) tm->begin(2);
  const int ncta = (int)((L.nblocks + kPlanCta - 1) / kPlanCta);
  launch(true, k_plan_local<DIM>, ncta, kPlanCta, 0, s, g, w.block_count, w.block_start, w.block_cnt, w.tmark, w.plan_pref,
                                              w.cta_tot, flag, sym >= 0 ? sym : (flag ? 1 : 0));
  launch(true, k_plan_offsets, 1, kPlanCta, 0, s, w.cta_tot, w.cta_off, ncta, w.hdr, flag);
  launch(true, k_plan_write<DIM>, ncta, kPlanCta, 0, s, g, w.block_count, w.block_start, w.block_cnt, w.tmark, w.plan_pref,
                                              w.cta_off, w.chunks, w.touched, w.occupied, flag);
  if (tm) tm->end(3);
}

template <int DIM, typename T>
size_t tile_smem(const Layout& L) {
  const int64_t tn = DIM == 3 ? int64_t(L.tile) * L.tile * L.tile : int64_t(L.tile) * L.tile;
  return size_t(tn) * 4 * sizeof(T);
}

// Dynamic shared memory every kernel may use (set_smem raises each kernel's limit to it).
constexpr size_t kMaxDynSmem = 200 * 1024;

// Dynamic shared memory of the cell-run P2G for this layout.
size_t cells_smem_bytes(const Layout& L) {
  if (L.real_bytes == 4)
    return L.dim == 3 ? tile_smem<3, float>(L) + cell_run_smem_bytes<3, float>(L.bs)
                      : tile_smem<2, float>(L) + cell_run_smem_bytes<2, float>(L.bs);
  return L.dim == 3 ? tile_smem<3, double>(L) + cell_run_smem_bytes<3, double>(L.bs)
                    : tile_smem<2, double>(L) + cell_run_smem_bytes<2, double>(L.bs);
}

template <typename F>
void set_smem(F* kernel, size_t bytes) {
  if (bytes > 48 * 1024) allow_smem(reinterpret_cast<const void*>(kernel), kMaxDynSmem);
}

template <int DIM, typename T, typename Sink>
void launch_p2g(const ffmpm_params& p, const Layout& L, const Ws& w, const PView<T>& P, const uint32_t* perm,
                const Sink& sink, cudaStream_t s, const uint32_t* flag = nullptr) {
  // plans kept over several substeps need the stray path of the cell-run kernel
  const bool direct = !flag && (p.variant & kVariantP2GDirect) != 0;
  const bool lanes = !flag && (p.variant & kVariantP2GLanes) != 0;
  if (!direct && !lanes) {
    // default: cell-run P2G (tile + per-particle records + cell ids + run starts)
    const size_t smem = tile_smem<DIM, T>(L) + cell_run_smem_bytes<DIM, T>(L.bs);
    auto kern = k_p2g_cells<DIM, T, Sink>;
    set_smem(kern, smem);
    kern<<<work_grid(L.max_chunks, resident_per_sm(kern, smem)), kThreads, smem, s>>>(
        kparams<T>(p), geom<DIM>(L), P, perm, w.chunks, w.hdr, sink, &w.hdr->status, &w.hdr->polar_fallbacks, flag);
    return;
  }
  const size_t smem = direct ? 0 : tile_smem<DIM, T>(L);
  auto kern = direct ? k_p2g<DIM, T, Sink, true> : k_p2g<DIM, T, Sink, false>;
  set_smem(kern, smem);
  kern<<<work_grid(L.max_chunks, resident_per_sm(kern, smem)), kThreads, smem, s>>>(
      kparams<T>(p), geom<DIM>(L), P, perm, w.chunks, w.hdr, sink, &w.hdr->status, &w.hdr->polar_fallbacks);
}

template <int DIM, typename T>
void launch_p2g_det(const ffmpm_params& p, const Layout& L, const Ws& w, const PView<T>& P, const uint32_t* perm,
                    cudaStream_t s) {
  const int tn = DIM == 3 ? L.tile * L.tile * L.tile : L.tile * L.tile;
  const size_t smem = p2g_det_smem_bytes<DIM, T>(tn);
  auto kern = k_p2g_det<DIM, T>;
  set_smem(kern, smem);
  cudaMemsetAsync(w.hdr->det_next, 0, sizeof(w.hdr->det_next), s);  // the CTAs' shared work counters
  kern<<<work_grid(L.nblocks, resident_per_sm(kern, smem)), kThreads, smem, s>>>(
      kparams<T>(p), geom<DIM>(L), P, perm, w.occupied, w.hdr, static_cast<Node4<T>*>(w.stage), &w.hdr->status,
      &w.hdr->polar_fallbacks, w.hdr->det_next);
}

template <int DIM, typename T>
void launch_grid_update_det(const ffmpm_params& p, const Layout& L, const Ws& w, cudaStream_t s, T* user_gv = nullptr,
                            T* user_gm = nullptr) {
  launch(true, k_grid_update_det<DIM, T>, work_grid(L.nblocks, 8), kThreads, 0, s, 
      kparams<T>(p), geom<DIM>(L), w.touched, w.block_cnt, w.hdr, static_cast<const Node4<T>*>(w.stage),
      static_cast<Node4<T>*>(w.gridB), user_gv, user_gm);
}

template <int DIM, typename T>
void launch_grid_update(const ffmpm_params& p, const Layout& L, const Ws& w, cudaStream_t s, bool dep = true) {
  launch(dep, k_grid_update<DIM, T>, work_grid(L.nblocks, 8), kThreads, 0, s, kparams<T>(p), geom<DIM>(L), w.touched, w.hdr,
         static_cast<Node4<T>*>(w.gridA), static_cast<Node4<T>*>(w.gridB));
}

template <int DIM, typename T, bool kTma, bool kSorted>
int launch_g2p(const ffmpm_params& p, const Layout& L, const Ws& w, const PView<T>& Pin, const PView<T>& Pout,
               const uint32_t* perm, const T* user_gv, const G2PExtra& ex, cudaStream_t s,
               const uint32_t* flag = nullptr) {
  alignas(64) CUtensorMap map;
  std::memset(&map, 0, sizeof(map));
  if (kTma && !encode_grid_map(&map, w.gridB, L)) return FFMPM_ERR_CUDA;
  const size_t smem = tile_smem<DIM, T>(L) + 128 + 16;  // + alignment pad + mbarrier
  auto kern = k_g2p<DIM, T, kTma, kSorted>;
  set_smem(kern, smem);
  kern<<<work_grid(L.max_chunks, resident_per_sm(kern, smem)), kThreads, smem, s>>>(
      kparams<T>(p), geom<DIM>(L), Pin, Pout, perm, w.chunks, w.hdr, map, user_gv, ex, &w.hdr->status, flag);
  return FFMPM_OK;
}

// Fused G2P + P2G in the sorted solver: the default outside the deterministic mode and the P2G
// variants, for runs of two or more substeps.  3D blocks of 16 nodes a side keep separate launches, as when the
// fused kernel's tiles of them did not fit (1,048,576 particles: 312 us a substep, 126 fused, 115 with blocks of 8).
bool fused(const ffmpm_params& p, const Layout& L, int nsteps) {
  return !p.deterministic && nsteps >= 2 &&
         (p.variant & (kVariantNoFuse | kVariantP2GDirect | kVariantP2GLanes)) == 0 && !(L.dim == 3 && L.bs > 8);
}

// ---------------------------------------------------------------------------- unsorted operations
// Launch shape of the warp kernels for `count` particles: whole CTAs while they fill the SMs, else
// CTAs of 64 threads, so that a small count spreads over more SMs.
template <typename T>
struct WarpShape {
  int threads, grid;
  WarpShape(int64_t count, int per_sm) {
    threads = kWarpCta<T>;
    while (threads > 64 && (count + threads - 1) / threads < sm_count()) threads /= 2;
    grid = work_grid((count + threads - 1) / threads, per_sm * (kWarpCta<T> / threads));
  }
};

template <int DIM, typename T>
void launch_p2g_warp(const ffmpm_params& p, const Layout& L, const Ws& w, const PView<T>& P, const uint32_t* perm,
                     int64_t p0, int64_t p1, cudaStream_t s, bool dep, bool may_give_up = false) {
  const WarpShape<T> sh(p1 - p0, 8);
  const size_t smem = sizeof(WarpRecs<DIM, T>) * (sh.threads / 32);
  launch(dep, k_p2g_warp<DIM, T>, sh.grid, sh.threads, smem, s, kparams<T>(p), geom<DIM>(L), P, perm,
                                                       may_give_up, (uint32_t)p0, (uint32_t)p1, static_cast<Node4<T>*>(w.gridA), &w.hdr->status,
                                                       &w.hdr->polar_fallbacks);
}

// G2P of a sorted run, with the next substep's P2G (kNext) or alone.
template <int DIM, typename T, bool kNext>
void launch_g2p_sorted(const ffmpm_params& p, const Layout& L, const Ws& w, const PView<T>& Pin, const PView<T>& Pout,
                       const uint32_t* perm, const G2PExtra& ex, cudaStream_t s) {
  const WarpShape<T> sh(L.n, 8);
  const size_t smem = kNext ? sizeof(WarpRecs<DIM, T>) * (sh.threads / 32) : 0;
  // plainly: set up early it takes registers from the grid update before it (16,384 particles: 613 us a
  // 40-substep call, 585 like this; 1M: 4,939 and 4,963)
  launch(false, k_g2p_sorted<DIM, T, kNext>, sh.grid, sh.threads, smem, s, kparams<T>(p), geom<DIM>(L), Pin, Pout, perm,
                                                                 (uint32_t)L.n, ex, static_cast<Node4<T>*>(w.gridA),
                                                                 w.hdr, w.tmark, w.touched);
}

// Half of an SM for the stages of k_cell_sums.  With what fills the SM (13 CTAs, 229 KB) the kernels that follow
// in the chain of dependent launches are left with the L1 of that split, and k_g2p_range takes twice its time:
// 480,000 particles on 96^3, two substeps: 574 us, 406 like this and 407 with 30.  A corrected coarse step of
// 1,048,576 particles, which launches its gather plainly: 532 us, 541 like this and 551 with 30; of 400,000 on 64^3:
// 243, 230 and 227.
constexpr int kSumsCarveout = 50;

// Scatter of the whole state into grid A, in the form that scatter_form names.
template <int DIM, typename T>
void scatter_unsorted(const ffmpm_params& p, const Layout& L, const Ws& w, const PView<T>& P, cudaStream_t s) {
  const ScatterForm form = scatter_form(p, L);
  if (form == ScatterForm::kAsTheyCome) {
    launch_p2g_warp<DIM, T>(p, L, w, P, nullptr, 0, L.n, s, false);
    return;
  }
  const KParams<T> kp = kparams<T>(p);
  const uint32_t n = (uint32_t)L.n;
  const unsigned pg = (n + kThreads - 1) / kThreads;
  uint32_t* rank = w.keys0;
  int* nodes = reinterpret_cast<int*>(w.vals0);  // by particle (kPermuted) or by slot (kRecords)
  const bool permuted = form == ScatterForm::kPermuted;
  launch(false, k_cell_rank<DIM, T>, pg, kThreads, 0, s, kp, L.R, P, n, w.cell_count, rank, permuted ? nodes : nullptr);
  launch(true, k_cell_offsets, (L.nnodes + kCellTile - 1) / kCellTile, kThreads, 0, s, w.cell_count, w.cell_start, w.hdr);
  if (permuted) {
    launch(true, k_cell_perm, pg, kThreads, 0, s, n, rank, nodes, w.cell_start, w.hdr, w.keys1);
    launch_p2g_warp<DIM, T>(p, L, w, P, w.keys1, 0, L.n, s, true);
    return;
  }
  if constexpr (sizeof(T) == 4) {
    T* recs = static_cast<T*>(w.recs);
    launch(true, k_cell_records<DIM, T>, pg, kThreads, 0, s, kp, L.R, P, n, rank, w.cell_start, recs, nodes, &w.hdr->status,
           &w.hdr->polar_fallbacks);
    launch_carved(kSumsCarveout, true, k_cell_sums<DIM, T>, (L.n + 191) / 192, 64, 2 * sizeof(WarpStage<DIM, T>), s, L.R,
                  recs, nodes, w.hdr, static_cast<Node4<T>*>(w.gridA));
  }
}

template <int DIM, typename T>
void launch_grid_update_dense(const ffmpm_params& p, const Layout& L, const Ws& w, cudaStream_t s, bool dep = true) {
  launch(dep, k_grid_update_dense<DIM, T>, work_grid((L.nnodes + 4 * kThreads - 1) / (4 * kThreads), 8), kThreads, 0, s, 
      kparams<T>(p), geom<DIM>(L), w.hdr, static_cast<Node4<T>*>(w.gridA), static_cast<Node4<T>*>(w.gridB));
}

template <int DIM, typename T>
void launch_g2p_range(const ffmpm_params& p, const Layout& L, const Ws& w, const PView<T>& P, int64_t p0, int64_t p1,
                      cudaStream_t s, bool dep = true) {
  const WarpShape<T> sh(p1 - p0, 8);
  launch(dep, k_g2p_range<DIM, T>, sh.grid, sh.threads, 0, s, kparams<T>(p), geom<DIM>(L), P, (uint32_t)p0, (uint32_t)p1,
                                                     static_cast<const Node4<T>*>(w.gridB), &w.hdr->status);
}

// ------------------------------------------------------------------------------------ operations
template <int DIM, typename T>
int op_substep(const ffmpm_params& p, const Layout& L, const Ws& w, ffmpm_particles* P, cudaStream_t s) {
  const PView<T> pv = pview<T>(*P);
  if (unsorted(p, L)) {
    scatter_unsorted<DIM, T>(p, L, w, pv, s);
    launch_grid_update_dense<DIM, T>(p, L, w, s);
    launch_g2p_range<DIM, T>(p, L, w, pv, 0, L.n, s);
    return check_launch();
  }
  const uint32_t* perm = nullptr;
  sort_and_plan<DIM, T>(p, L, w, pv, false, &perm, s);
  if (p.deterministic) {
    launch_p2g_det<DIM, T>(p, L, w, pv, perm, s);
    launch_grid_update_det<DIM, T>(p, L, w, s);
  } else {
    launch_p2g<DIM, T>(p, L, w, pv, perm, InternalSink<T>{static_cast<Node4<T>*>(w.gridA)}, s);
    launch_grid_update<DIM, T>(p, L, w, s);
  }
  G2PExtra ex{};
  int rc = launch_g2p<DIM, T, true, false>(p, L, w, pv, pv, perm, nullptr, ex, s);
  return rc != FFMPM_OK ? rc : check_launch();
}

// ----------------------------------------------------------------------------- host-array substep
// Copy streams and events of ffmpm_substep_host, one set per device, created by the first call on
// that device (with it current) and kept until the process exits.
// Four chunks: a fifth costs its copies and launches and hides less than that below a million particles
// (262,145: 442 us, 463 with five; 400,000: 576, 601; 800,000: 1,001, 1,031; 1,048,576: 1,322, 1,310).
constexpr int kHostChunks = 4;
struct HostPipe {
  cudaStream_t up = nullptr, down = nullptr;
  cudaEvent_t start = nullptr, gathered_all = nullptr, down_done = nullptr;
  cudaEvent_t landed[kHostChunks] = {}, gathered[kHostChunks] = {};
};

int host_pipe(HostPipe** out) {
  constexpr int kMaxDevices = 64;
  static std::mutex mu;
  static HostPipe pipes[kMaxDevices];
  static bool made[kMaxDevices] = {};
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= kMaxDevices) return FFMPM_ERR_CUDA;
  std::lock_guard<std::mutex> lock(mu);
  HostPipe& h = pipes[dev];
  if (!made[dev]) {
    bool ok = cudaStreamCreateWithFlags(&h.up, cudaStreamNonBlocking) == cudaSuccess &&
              cudaStreamCreateWithFlags(&h.down, cudaStreamNonBlocking) == cudaSuccess &&
              cudaEventCreateWithFlags(&h.start, cudaEventDisableTiming) == cudaSuccess &&
              cudaEventCreateWithFlags(&h.gathered_all, cudaEventDisableTiming) == cudaSuccess &&
              cudaEventCreateWithFlags(&h.down_done, cudaEventDisableTiming) == cudaSuccess;
    for (int k = 0; ok && k < kHostChunks; ++k)
      ok = cudaEventCreateWithFlags(&h.landed[k], cudaEventDisableTiming) == cudaSuccess &&
           cudaEventCreateWithFlags(&h.gathered[k], cudaEventDisableTiming) == cudaSuccess;
    if (!ok) return FFMPM_ERR_CUDA;
    made[dev] = true;
  }
  *out = &h;
  return FFMPM_OK;
}

// One substep on host arrays H through the device arrays D (same shapes, row-major).  Chunk k of
// every input array goes up on the upload stream and is scattered on `s` once it has landed; after
// the dense grid update, chunk k is gathered on `s` and its outputs go down on the download stream
// while chunk k + 1 is gathered.  `s` finally waits for the last download, so that the call is
// complete, host arrays included, once `s` has run.  (Kernels reading and writing mapped pinned
// host memory in place measured about 4x slower than this on a GB300: the copy engines, not SM
// loads and stores, reach the host link's rate here.)
template <int DIM, typename T>
int op_substep_host(const ffmpm_params& p, const Layout& L, const Ws& w, const ffmpm_particles* H,
                    ffmpm_particles* D, cudaStream_t s) {
  const int64_t n = H->n;
  HostPipe* hp = nullptr;
  int rc = host_pipe(&hp);
  if (rc != FFMPM_OK) return rc;
  const size_t rb = sizeof(T);
  struct Arr {
    void* h;
    void* d;
    size_t per;   // bytes per particle
    bool in;      // read by the substep
    bool out;     // written by the substep
    bool whole;   // one real per particle: sent up whole before the first chunk (fewer, larger copies)
  };
  // Jp is read and changed only in 2D and for snow (two_d/g2p.py:44-46, three_d/p2g.py:57-61,
  // three_d/g2p.py:48-58): elsewhere it is neither sent up nor sent back
  const bool jp_used = DIM == 2 || p.model == FFMPM_MODEL_SNOW;
  const Arr arrs[8] = {{H->x, D->x, DIM * rb, true, true, false},
                       {H->v, D->v, DIM * rb, true, true, false},
                       {H->F, D->F, DIM * DIM * rb, true, true, false},
                       {H->C, D->C, DIM * DIM * rb, true, true, false},
                       {H->Jp, D->Jp, rb, jp_used, jp_used, true},
                       {const_cast<void*>(H->mass), const_cast<void*>(D->mass), rb, true, false, true},
                       {const_cast<void*>(H->mu_0), const_cast<void*>(D->mu_0), rb, true, false, true},
                       {const_cast<void*>(H->lambda_0), const_cast<void*>(D->lambda_0), rb, true, false, true}};
  // copies of [a, b) of the chunked arrays (whole = false: the per-particle scalars over [0, n))
  auto copy = [&](bool down, int64_t a, int64_t b, cudaStream_t cs, bool whole = false) {
    for (const Arr& r : arrs) {
      if (!r.h || (down && !r.out) || (!down && (!r.in || r.whole != whole))) continue;
      unsigned char* hb = static_cast<unsigned char*>(r.h) + a * r.per;
      unsigned char* db = static_cast<unsigned char*>(r.d) + a * r.per;
      if (down)
        cudaMemcpyAsync(hb, db, (b - a) * r.per, cudaMemcpyDeviceToHost, cs);
      else
        cudaMemcpyAsync(db, hb, (b - a) * r.per, cudaMemcpyHostToDevice, cs);
    }
  };
  // the uploads start after the work already queued on the caller's stream
  cudaEventRecord(hp->start, s);
  cudaStreamWaitEvent(hp->up, hp->start, 0);
  if (p.deterministic) {
    // the fixed summation order needs the block-sorted path: whole arrays up, ffmpm_substep, down
    copy(false, 0, n, hp->up, true);
    copy(false, 0, n, hp->up);
    cudaEventRecord(hp->landed[0], hp->up);
    cudaStreamWaitEvent(s, hp->landed[0], 0);
    rc = op_substep<DIM, T>(p, L, w, D, s);
    if (rc != FFMPM_OK) return rc;
    copy(true, 0, n, s);
    return check_launch();
  }
  // Upload chunks shrink (sizes K, K-1, ..., 1) so that little scatter is left once the last one
  // has landed; gather/download chunks grow (1, 2, ..., K) so that the first download starts soon
  // after the grid update.
  const int K = (int)std::max<int64_t>(1, std::min<int64_t>(kHostChunks, (n + 65535) / 65536));
  const int64_t parts = int64_t(K) * (K + 1) / 2;
  auto up_lo = [&](int k) { return n * (int64_t(k) * (2 * K - k + 1) / 2) / parts; };
  auto lo = [&](int k) { return n * (int64_t(k) * (k + 1) / 2) / parts; };
  const PView<T> pv = pview<T>(*D);
  copy(false, 0, n, hp->up, true);
  for (int k = 0; k < K; ++k) {
    const int64_t a = up_lo(k), b = up_lo(k + 1);
    copy(false, a, b, hp->up);
    cudaEventRecord(hp->landed[k], hp->up);
    cudaStreamWaitEvent(s, hp->landed[k], 0);
    launch_p2g_warp<DIM, T>(p, L, w, pv, nullptr, a, b, s, false);
  }
  launch_grid_update_dense<DIM, T>(p, L, w, s, false);
  for (int k = 0; k < K; ++k) {
    const int64_t a = lo(k), b = lo(k + 1);
    launch_g2p_range<DIM, T>(p, L, w, pv, a, b, s, false);
    cudaEventRecord(hp->gathered[k], s);
    cudaStreamWaitEvent(hp->down, hp->gathered[k], 0);
    copy(true, a, b, hp->down);
  }
  cudaEventRecord(hp->down_done, hp->down);
  cudaStreamWaitEvent(s, hp->down_done, 0);
  return check_launch();
}

// Per-substep copies of the positions and ids (ffmpm_substeps_sorted_snapshots): after substep k
// the output buffer's x (dim components of n reals, in its sorted order) goes to x + k dim n and
// its ids to ids + k n, on the run's stream.
struct SnapOut {
  void* x;
  int32_t* ids;
};

template <int DIM, typename T>
void snapshot(const SnapOut* snap, int k, const PView<T>& out, const int32_t* ids_out, int64_t n, cudaStream_t s) {
  if (!snap) return;
  T* dst = static_cast<T*>(snap->x) + (size_t)k * DIM * n;
  if (out.soa == n) {
    cudaMemcpyAsync(dst, out.x, sizeof(T) * DIM * n, cudaMemcpyDeviceToDevice, s);
  } else {
    for (int d = 0; d < DIM; ++d)
      cudaMemcpyAsync(dst + (size_t)d * n, out.x + (size_t)d * out.soa, sizeof(T) * n, cudaMemcpyDeviceToDevice, s);
  }
  cudaMemcpyAsync(snap->ids + (size_t)k * n, ids_out, sizeof(int32_t) * n, cudaMemcpyDeviceToDevice, s);
}

// Substeps 0..n-1 with the fused kernel: P2G(0), then for k = 0..n-2: grid update(k), re-sort if
// due (k a multiple of the cadence), G2P(k) + P2G(k+1); then grid update(n-1) and G2P(n-1).  The
// state after every substep is in buffer a or b as in the unfused loop (x, F, Jp, ids, per-particle
// material), with v and C written by the last G2P only.  The grid update of substep k runs before
// the re-sort, on the touched blocks of the plan its P2G scattered under.  The re-sorts are
// scheduled on the host: the fused kernel adds the blocks a fast particle reaches to the touched
// list itself, so correctness does not wait for a re-sort, and substeps without one launch no
// sort or plan kernel at all.  Keys and the block histogram are written only by the fused launch
// that precedes a re-sort.
template <int DIM, typename T>
int op_substeps_fused(const ffmpm_params& p, const Layout& L, const Ws& w, PView<T> va, PView<T> vb, int32_t* ids_a,
                      int32_t* ids_b, int nsteps, cudaStream_t s, PhaseTimer* tm, const SnapOut* snap) {
  const int K = sort_every(p);
  const auto resorts = [&](int k) { return k >= 1 && k <= nsteps - 2 && k % K == 0; };
  const uint32_t* sorted_perm = nullptr;
  sort_and_plan<DIM, T>(p, L, w, va, false, &sorted_perm, s, tm, nullptr, 1);
  const uint32_t* perm = sorted_perm;  // the permutation the next P2G / G2P applies (null: none)
  if (tm) tm->begin(3);
  launch_p2g_warp<DIM, T>(p, L, w, va, perm, 0, L.n, s, true, true);
  if (tm) tm->end(1);
  for (int k = 0; k < nsteps; ++k) {
    const PView<T>& in = (k & 1) ? vb : va;
    const PView<T>& out = (k & 1) ? va : vb;
    const int32_t* ids_in = (k & 1) ? ids_b : ids_a;
    int32_t* ids_out = (k & 1) ? ids_a : ids_b;
    if (tm) tm->begin(4);
    launch_grid_update<DIM, T>(p, L, w, s, !snap);  // a snapshot's copies lie between
    if (tm) tm->end(1);
    if (k == nsteps - 1) {
      // k >= 1: the buffer is already in the order of the current plan
      G2PExtra ex{ids_in, ids_out, nullptr, nullptr, L.cell_bits, w.gridB, nullptr};
      if (tm) tm->begin(5);
      launch_g2p_sorted<DIM, T, false>(p, L, w, in, out, nullptr, ex, s);
      if (tm) tm->end(1);
      snapshot<DIM, T>(snap, k, out, ids_out, L.n, s);
      break;
    }
    if (k > 0) perm = nullptr;
    if (resorts(k)) sort_and_plan<DIM, T>(p, L, w, in, true, &perm, s, tm, nullptr, 1);
    const bool keys = resorts(k + 1);
    G2PExtra ex{ids_in, ids_out, keys ? w.keys_next : nullptr, keys ? w.block_count : nullptr, L.cell_bits, w.gridB,
                nullptr};
    if (tm) tm->begin(6);
    launch_g2p_sorted<DIM, T, true>(p, L, w, in, out, perm, ex, s);
    if (tm) tm->end(1);
    snapshot<DIM, T>(snap, k, out, ids_out, L.n, s);
  }
  return check_launch();
}

template <int DIM, typename T>
int op_substeps_sorted(const ffmpm_params& p, const Layout& L, const Ws& w, ffmpm_particles* a, ffmpm_particles* b,
                       int32_t* ids_a, int32_t* ids_b, int nsteps, cudaStream_t s, PhaseTimer* tm = nullptr,
                       const SnapOut* snap = nullptr) {
  PView<T> va = pview<T>(*a), vb = pview<T>(*b);
  if (fused(p, L, nsteps)) return op_substeps_fused<DIM, T>(p, L, w, va, vb, ids_a, ids_b, nsteps, s, tm, snap);
  const int K = sort_every(p);
  const uint32_t* flag = K > 1 ? &w.hdr->sort_now : nullptr;
  for (int k = 0; k < nsteps; ++k) {
    const PView<T>& in = (k & 1) ? vb : va;
    const PView<T>& out = (k & 1) ? va : vb;
    const int32_t* ids_in = (k & 1) ? ids_b : ids_a;
    int32_t* ids_out = (k & 1) ? ids_a : ids_b;
    const uint32_t* perm = nullptr;
    if (flag) k_sort_decide<<<1, 1, 0, s>>>(w.hdr, k % K == 0 ? 1 : 0);
    sort_and_plan<DIM, T>(p, L, w, in, k > 0, &perm, s, tm, flag);
    if (tm) tm->begin(3);
    if (p.deterministic)
      launch_p2g_det<DIM, T>(p, L, w, in, perm, s);
    else
      launch_p2g<DIM, T>(p, L, w, in, perm, InternalSink<T>{static_cast<Node4<T>*>(w.gridA)}, s, flag);
    if (tm) tm->end(1);
    if (tm) tm->begin(4);
    if (p.deterministic)
      launch_grid_update_det<DIM, T>(p, L, w, s);
    else
      launch_grid_update<DIM, T>(p, L, w, s);
    if (tm) tm->end(1);
    G2PExtra ex{ids_in, ids_out, w.keys_next, w.block_count, L.cell_bits, w.gridB, flag ? &w.hdr->far_stray : nullptr};
    if (tm) tm->begin(5);
    if (p.deterministic) {
      // by warps, not by chunks of the 4^3 blocks, a fifth of whose slots are empty (particle by particle the
      // same sums, bit for bit)
      launch_g2p_sorted<DIM, T, false>(p, L, w, in, out, perm, ex, s);
    } else {
      if (!flag) ex.grid_global = nullptr;
      const int rc = launch_g2p<DIM, T, true, true>(p, L, w, in, out, perm, nullptr, ex, s, flag);
      if (rc != FFMPM_OK) return rc;
    }
    if (tm) tm->end(1);
    snapshot<DIM, T>(snap, k, out, ids_out, L.n, s);
  }
  // The last G2P counted the blocks of the final state for a substep that will not run here:
  // clear the histogram so the workspace invariant (zero between calls) holds.
  cudaMemsetAsync(w.block_count, 0, sizeof(uint32_t) * L.nblocks, s);
  return check_launch();
}

template <int DIM, typename T>
int op_p2g(const ffmpm_params& p, const Layout& L, const Ws& w, const ffmpm_particles* P, ffmpm_grid* grid,
           cudaStream_t s) {
  const PView<T> pv = pview<T>(*P);
  if (unsorted(p, L)) {
    scatter_unsorted<DIM, T>(p, L, w, pv, s);
    launch(true, k_grid_fold_user<DIM, T>, work_grid((L.nnodes + kThreads - 1) / kThreads, 8), kThreads, 0, s, 
        L.nnodes, w.hdr, static_cast<Node4<T>*>(w.gridA), static_cast<T*>(grid->velocity),
        static_cast<T*>(grid->mass));
    return check_launch();
  }
  const uint32_t* perm = nullptr;
  sort_and_plan<DIM, T>(p, L, w, pv, false, &perm, s);
  if (p.deterministic) {
    launch_p2g_det<DIM, T>(p, L, w, pv, perm, s);
    launch_grid_update_det<DIM, T>(p, L, w, s, static_cast<T*>(grid->velocity), static_cast<T*>(grid->mass));
  } else {
    launch_p2g<DIM, T>(p, L, w, pv, perm,
                       UserSink<T, DIM>{static_cast<T*>(grid->velocity), static_cast<T*>(grid->mass)}, s);
  }
  return check_launch();
}

template <int DIM, typename T>
int op_g2p(const ffmpm_params& p, const Layout& L, const Ws& w, const ffmpm_grid* grid, ffmpm_particles* P,
           cudaStream_t s) {
  const PView<T> pv = pview<T>(*P);
  if (unsorted(p, L)) {
    launch(false, k_grid_pack_user<DIM, T>, work_grid((L.nnodes + kThreads - 1) / kThreads, 8), kThreads, 0, s, 
        L.nnodes, static_cast<const T*>(grid->velocity), static_cast<Node4<T>*>(w.gridB));
    launch_g2p_range<DIM, T>(p, L, w, pv, 0, L.n, s);
    return check_launch();
  }
  const uint32_t* perm = nullptr;
  sort_and_plan<DIM, T>(p, L, w, pv, false, &perm, s);
  G2PExtra ex{};
  int rc = launch_g2p<DIM, T, false, false>(p, L, w, pv, pv, perm, static_cast<const T*>(grid->velocity), ex, s);
  return rc != FFMPM_OK ? rc : check_launch();
}

template <int DIM, typename T>
int op_grid_op(const ffmpm_params& p, ffmpm_grid* grid, cudaStream_t s) {
  const int R = p.res + 1;
  const int64_t nn = DIM == 3 ? int64_t(R) * R * R : int64_t(R) * R;
  const int blocks = (int)std::min<int64_t>((nn + kThreads - 1) / kThreads, int64_t(sm_count()) * 16);
  k_grid_op_dense<DIM, T><<<std::max(blocks, 1), kThreads, 0, s>>>(kparams<T>(p), R, static_cast<T*>(grid->velocity),
                                                                   static_cast<const T*>(grid->mass));
  return check_launch();
}

template <int DIM, typename T>
int op_sort(const ffmpm_params& p, const Layout& L, const Ws& w, const void* x, uint32_t* keys_out,
            uint32_t* perm_out, cudaStream_t s) {
  const KParams<T> kp = kparams<T>(p);
  const Geom<DIM> g = geom<DIM>(L);
  const uint32_t n = (uint32_t)L.n;
  PView<T> xv{};
  xv.x = static_cast<T*>(const_cast<void*>(x));
  launch(false, k_keys<DIM, T>, (n + kThreads - 1) / kThreads, kThreads, 0, s, kp, g, xv, n, L.cell_bits, w.keys_next, nullptr,
                                                                     &w.hdr->status);
  const uint32_t *ks = nullptr, *perm = nullptr;
  radix_sort(w.keys_next, n, L.passes, w.keys0, w.keys1, w.vals0, w.vals1, w.hist, radix_tile(L.n), &w.hdr->status, s, &ks,
             &perm, nullptr, p.wait_limit, p.inject);
  if (keys_out) cudaMemcpyAsync(keys_out, ks, sizeof(uint32_t) * n, cudaMemcpyDeviceToDevice, s);
  if (perm_out) cudaMemcpyAsync(perm_out, perm, sizeof(uint32_t) * n, cudaMemcpyDeviceToDevice, s);
  return check_launch();
}

template <int DIM, typename T>
int op_diag(const ffmpm_params& p, const ffmpm_particles* P, double* out, cudaStream_t s) {
  k_diag_init<<<1, 32, 0, s>>>(out);
  const uint32_t n = (uint32_t)P->n;
  const int blocks = std::max(1, (int)std::min<int64_t>((n + kThreads - 1) / kThreads, int64_t(sm_count()) * 8));
  if (n > 0) k_diag<DIM, T><<<blocks, kThreads, 0, s>>>(kparams<T>(p), pview<T>(*P), n, out);
  return check_launch();
}

// Dispatch on (dim, precision).
template <template <int, typename> class Op, typename... Args>
int dispatch(const ffmpm_params& p, Args&&... args) {
  if (p.dim == 3) {
    if (p.real_bytes == 4) return Op<3, float>::run(p, args...);
    return Op<3, double>::run(p, args...);
  }
  if (p.real_bytes == 4) return Op<2, float>::run(p, args...);
  return Op<2, double>::run(p, args...);
}

#define FFMPM_OP(NAME, FN)                                          \
  template <int DIM, typename T>                                    \
  struct NAME {                                                     \
    template <typename... A>                                        \
    static int run(const ffmpm_params& p, A&&... a) {               \
      return FN<DIM, T>(p, a...);                                   \
    }                                                               \
  };
FFMPM_OP(SubstepOp, op_substep)
FFMPM_OP(SubstepHostOp, op_substep_host)
FFMPM_OP(SortedOp, op_substeps_sorted)
FFMPM_OP(ProfileOp, op_substeps_sorted)
FFMPM_OP(SnapshotOp, op_substeps_sorted)
FFMPM_OP(P2GOp, op_p2g)
FFMPM_OP(G2POp, op_g2p)
FFMPM_OP(GridOp, op_grid_op)
FFMPM_OP(SortOp, op_sort)
FFMPM_OP(DiagOp, op_diag)
#undef FFMPM_OP

bool particles_ok(const ffmpm_params& p, const ffmpm_particles* P, bool need_jp) {
  if (!P || P->n < 0) return false;
  if (P->stride != 0 && P->stride < P->n) return false;
  if (P->n == 0) return true;
  if (!P->x || !P->v || !P->F || !P->C) return false;
  if (need_jp && !P->Jp) return false;
  return true;
}

bool supported(const ffmpm_params& p) { return true; }

int prologue(const ffmpm_params* p, int64_t n, void* ws, size_t ws_bytes, Layout* L) {
  if (!p || !make_layout(*p, n, L)) return FFMPM_ERR_BADARG;
  if (!supported(*p)) return FFMPM_ERR_UNSUPPORTED;
  if (p->deterministic) {
    const int tn = p->dim == 3 ? L->tile * L->tile * L->tile : L->tile * L->tile;
    const size_t smem = p->real_bytes == 4 ? (p->dim == 3 ? p2g_det_smem_bytes<3, float>(tn) : p2g_det_smem_bytes<2, float>(tn))
                                           : (p->dim == 3 ? p2g_det_smem_bytes<3, double>(tn)
                                                          : p2g_det_smem_bytes<2, double>(tn));
    if (smem > kMaxDynSmem) return FFMPM_ERR_UNSUPPORTED;  // warp tiles + records must fit in shared memory
  } else if (cells_smem_bytes(*L) > kMaxDynSmem) {
    return FFMPM_ERR_UNSUPPORTED;  // the cell-run P2G's tile and records must fit in shared memory
  }
  if (!ws || ws_bytes < L->total || (reinterpret_cast<uintptr_t>(ws) & 255)) return FFMPM_ERR_WORKSPACE;
  return FFMPM_OK;
}

// Eight bytes of page-locked memory per host thread, for ffmpm_status_read: a copy into pageable memory
// goes through the driver's own staging and costs twice as much (a status read: 14 us, 9 with this).  Given
// back when the thread ends; null when it cannot be had.
struct StatusSlot {
  uint32_t* p = nullptr;
  StatusSlot() {
    const RelaxedCapture mode;
    if (cudaHostAlloc(reinterpret_cast<void**>(&p), 8, cudaHostAllocPortable) != cudaSuccess) {
      cudaGetLastError();
      p = nullptr;
    }
  }
  ~StatusSlot() {
    if (!p) return;
    const RelaxedCapture mode;
    cudaFreeHost(p);
  }

 private:
  // a thread's first read, and its end, may fall into another thread's stream capture, which page-locking and its
  // undoing would spoil
  struct RelaxedCapture {
    cudaStreamCaptureMode mode = cudaStreamCaptureModeRelaxed;
    RelaxedCapture() { cudaThreadExchangeStreamCaptureMode(&mode); }
    ~RelaxedCapture() { cudaThreadExchangeStreamCaptureMode(&mode); }
  };
};
uint32_t* status_slot() {
  static thread_local StatusSlot slot;
  return slot.p;
}

}  // namespace
}  // namespace ffmpm

using namespace ffmpm;

extern "C" {

const char* ffmpm_version(void) { return "femflow_gb300 mpm 0.1 (sm_103a)"; }

int ffmpm_workspace_size(const ffmpm_params* p, int64_t n, size_t* bytes) {
  Layout L;
  if (!p || !bytes || !make_layout(*p, n, &L)) return FFMPM_ERR_BADARG;
  *bytes = L.total;
  return FFMPM_OK;
}

int ffmpm_workspace_init(const ffmpm_params* p, int64_t n, void* ws, size_t ws_bytes, void* stream) {
  Layout L;
  if (!p || !make_layout(*p, n, &L)) return FFMPM_ERR_BADARG;
  if (!ws || ws_bytes < L.total) return FFMPM_ERR_WORKSPACE;
  cudaMemsetAsync(ws, 0, L.total, static_cast<cudaStream_t>(stream));
  return check_launch();
}

int ffmpm_status_read(void* ws, int32_t* status, uint32_t* polar_fallbacks, void* stream) {
  if (!ws) return FFMPM_ERR_WORKSPACE;
  static_assert(offsetof(WsHeader, status) == 0 && offsetof(WsHeader, polar_fallbacks) == 4, "first eight bytes");
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  uint32_t stack[2] = {0, 0};
  uint32_t* slot = status_slot();
  if (!slot) slot = stack;
  if (cudaMemcpyAsync(slot, ws, 8, cudaMemcpyDeviceToHost, s) != cudaSuccess) return FFMPM_ERR_CUDA;
  if (cudaStreamSynchronize(s) != cudaSuccess) return FFMPM_ERR_CUDA;
  if (status) *status = (int32_t)slot[0];
  if (polar_fallbacks) *polar_fallbacks = slot[1];
  return FFMPM_OK;
}

int ffmpm_status_clear(void* ws, void* stream) {
  if (!ws) return FFMPM_ERR_WORKSPACE;
  cudaMemsetAsync(ws, 0, 8, static_cast<cudaStream_t>(stream));  // status + polar_fallbacks
  return check_launch();
}

int ffmpm_substep(const ffmpm_params* p, ffmpm_particles* P, void* ws, size_t ws_bytes, void* stream) {
  Layout L;
  if (!P) return FFMPM_ERR_BADARG;
  int rc = prologue(p, P->n, ws, ws_bytes, &L);
  if (rc != FFMPM_OK) return rc;
  if (!particles_ok(*p, P, true)) return FFMPM_ERR_BADARG;
  if (P->n == 0) return FFMPM_OK;
  Ws w = bind(ws, L);
  return dispatch<SubstepOp>(*p, L, w, P, static_cast<cudaStream_t>(stream));
}

int ffmpm_substep_host(const ffmpm_params* p, const ffmpm_particles* host, ffmpm_particles* dev, void* ws,
                       size_t ws_bytes, void* stream) {
  Layout L;
  if (!host || !dev || host->n != dev->n || host->stride != 0 || dev->stride != 0) return FFMPM_ERR_BADARG;
  int rc = prologue(p, host->n, ws, ws_bytes, &L);
  if (rc != FFMPM_OK) return rc;
  if (!particles_ok(*p, host, true) || !particles_ok(*p, dev, true)) return FFMPM_ERR_BADARG;
  if ((host->mass && !dev->mass) || (host->mu_0 && !dev->mu_0) || (host->lambda_0 && !dev->lambda_0))
    return FFMPM_ERR_BADARG;
  if (host->n == 0) return FFMPM_OK;
  // the device arrays stand in for the host ones: material pointers the host leaves NULL stay NULL
  ffmpm_particles d = *dev;
  if (!host->mass) d.mass = nullptr;
  if (!host->mu_0) d.mu_0 = nullptr;
  if (!host->lambda_0) d.lambda_0 = nullptr;
  Ws w = bind(ws, L);
  return dispatch<SubstepHostOp>(*p, L, w, host, &d, static_cast<cudaStream_t>(stream));
}

int ffmpm_substeps_sorted(const ffmpm_params* p, ffmpm_particles* a, ffmpm_particles* b, int32_t* ids_a,
                          int32_t* ids_b, int32_t nsteps, void* ws, size_t ws_bytes, void* stream) {
  Layout L;
  if (!a || !b || nsteps < 0 || a->n != b->n) return FFMPM_ERR_BADARG;
  int rc = prologue(p, a->n, ws, ws_bytes, &L);
  if (rc != FFMPM_OK) return rc;
  if (!particles_ok(*p, a, true) || !particles_ok(*p, b, true)) return FFMPM_ERR_BADARG;
  if ((a->mass != nullptr) != (b->mass != nullptr) || (a->mu_0 != nullptr) != (b->mu_0 != nullptr) ||
      (a->lambda_0 != nullptr) != (b->lambda_0 != nullptr) || ((ids_a != nullptr) != (ids_b != nullptr)))
    return FFMPM_ERR_BADARG;
  if (a->n == 0 || nsteps == 0) return FFMPM_OK;
  Ws w = bind(ws, L);
  return dispatch<SortedOp>(*p, L, w, a, b, ids_a, ids_b, (int)nsteps, static_cast<cudaStream_t>(stream));
}

int ffmpm_substeps_sorted_snapshots(const ffmpm_params* p, ffmpm_particles* a, ffmpm_particles* b, int32_t* ids_a,
                                    int32_t* ids_b, int32_t nsteps, void* snap_x, int32_t* snap_ids, void* ws,
                                    size_t ws_bytes, void* stream) {
  Layout L;
  if (!a || !b || nsteps < 0 || a->n != b->n || !ids_a || !ids_b || !snap_x || !snap_ids) return FFMPM_ERR_BADARG;
  if (a->stride < a->n || b->stride < b->n) return FFMPM_ERR_BADARG;  // component-major buffers only
  int rc = prologue(p, a->n, ws, ws_bytes, &L);
  if (rc != FFMPM_OK) return rc;
  if (!particles_ok(*p, a, true) || !particles_ok(*p, b, true)) return FFMPM_ERR_BADARG;
  if ((a->mass != nullptr) != (b->mass != nullptr) || (a->mu_0 != nullptr) != (b->mu_0 != nullptr) ||
      (a->lambda_0 != nullptr) != (b->lambda_0 != nullptr))
    return FFMPM_ERR_BADARG;
  if (a->n == 0 || nsteps == 0) return FFMPM_OK;
  Ws w = bind(ws, L);
  const SnapOut snap{snap_x, snap_ids};
  return dispatch<SnapshotOp>(*p, L, w, a, b, ids_a, ids_b, (int)nsteps, static_cast<cudaStream_t>(stream),
                              static_cast<PhaseTimer*>(nullptr), &snap);
}

int ffmpm_profile_substeps(const ffmpm_params* p, ffmpm_particles* a, ffmpm_particles* b, int32_t* ids_a,
                           int32_t* ids_b, int32_t nsteps, void* ws, size_t ws_bytes, void* stream, double* phase_ms,
                           int64_t* phase_launches) {
  Layout L;
  if (!a || !b || nsteps < 0 || a->n != b->n || !phase_ms || !phase_launches) return FFMPM_ERR_BADARG;
  int rc = prologue(p, a->n, ws, ws_bytes, &L);
  if (rc != FFMPM_OK) return rc;
  if (!particles_ok(*p, a, true) || !particles_ok(*p, b, true)) return FFMPM_ERR_BADARG;
  if (a->n == 0 || nsteps == 0) return FFMPM_OK;
  Ws w = bind(ws, L);
  PhaseTimer tm;
  tm.s = static_cast<cudaStream_t>(stream);
  rc = dispatch<ProfileOp>(*p, L, w, a, b, ids_a, ids_b, (int)nsteps, tm.s, &tm);
  tm.collect(phase_ms, phase_launches);
  return rc;
}

int ffmpm_plan_info(const ffmpm_params* p, int64_t n, int64_t* info) {
  Layout L;
  if (!p || !info || !make_layout(*p, n, &L)) return FFMPM_ERR_BADARG;
  info[0] = L.bs;
  info[1] = L.nb;
  info[2] = L.nblocks;
  info[3] = L.key_bits;
  info[4] = L.passes;
  // digit histogram + one kernel per radix pass + 3 plan kernels + P2G + grid + G2P (+ the re-sort
  // decision of cadenced runs)
  info[5] = L.passes + 7 + (sort_every(*p) > 1 ? 1 : 0);
  info[6] = L.tile;
  info[7] = L.max_chunks;
  return FFMPM_OK;
}

int ffmpm_check_collision_points(const ffmpm_params* p, const double* points, const double* normals, int32_t n,
                                 void* grid_velocity, void* stream) {
  if (!p || n < 0 || (n > 0 && (!points || !normals || !grid_velocity))) return FFMPM_ERR_BADARG;
  if (!valid_params(p)) return FFMPM_ERR_BADARG;
  if (p->plane_rule != FFMPM_PLANES_STICKY && p->plane_rule != FFMPM_PLANES_REFERENCE_LITERAL) return FFMPM_ERR_BADARG;
  const int dim = p->dim;
  for (int i = 0; i < n * dim; ++i)
    if (!std::isfinite(points[i]) || !std::isfinite(normals[i])) return FFMPM_ERR_BADARG;
  for (int i = 0; i < n; ++i) {
    double ss = 0.0;
    for (int d = 0; d < dim; ++d) ss += normals[i * dim + d] * normals[i * dim + d];
    if (!(ss > 0.0)) return FFMPM_ERR_BADARG;  // the reference divides by |normal|
  }
  const int64_t R = p->res + 1;
  const int64_t nnodes = dim == 3 ? R * R * R : R * R;
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  // the planes go to the kernel in batches of FFMPM_MAX_PLANES (zeroing is idempotent, so the
  // batches compose like the reference's loop over planes)
  for (int b = 0; b < n; b += FFMPM_MAX_PLANES) {
    ffmpm_params q = *p;
    q.n_planes = std::min(n - b, FFMPM_MAX_PLANES);
    for (int i = 0; i < q.n_planes; ++i)
      for (int d = 0; d < 3; ++d) {
        q.planes[i][d] = d < dim ? points[(b + i) * dim + d] : 0.0;
        q.planes[i][3 + d] = d < dim ? normals[(b + i) * dim + d] : 0.0;
      }
    const int blocks = work_grid((nnodes + kThreads - 1) / kThreads, 8);
    if (p->real_bytes == 4) {
      if (dim == 3)
        k_collision_points<3, float><<<blocks, kThreads, 0, s>>>(kparams<float>(q), static_cast<float*>(grid_velocity), nnodes);
      else
        k_collision_points<2, float><<<blocks, kThreads, 0, s>>>(kparams<float>(q), static_cast<float*>(grid_velocity), nnodes);
    } else {
      if (dim == 3)
        k_collision_points<3, double><<<blocks, kThreads, 0, s>>>(kparams<double>(q), static_cast<double*>(grid_velocity), nnodes);
      else
        k_collision_points<2, double><<<blocks, kThreads, 0, s>>>(kparams<double>(q), static_cast<double*>(grid_velocity), nnodes);
    }
  }
  return check_launch();
}

int ffmpm_kernels_per_call(const ffmpm_params* p, int64_t n, int32_t nsteps, int64_t* count) {
  Layout L;
  if (!p || !count || nsteps < 0 || !make_layout(*p, n, &L)) return FFMPM_ERR_BADARG;
  const int64_t sort = 1 + L.passes + 3;  // digit histogram, one kernel per pass, three plan kernels
  if (n == 0 || nsteps == 0) {
    *count = 0;
  } else if (fused(*p, L, nsteps)) {
    // keys + sort + P2G; per substep k < n-1: grid update + fused kernel (+ sort when 1 <= k <= n-2
    // is a multiple of the cadence); the last substep: grid update + G2P
    *count = (1 + sort + 1) + int64_t(nsteps - 1) * 2 + int64_t((nsteps - 2) / sort_every(*p)) * sort + 2;
  } else {
    // per substep: (decide) + sort + P2G + grid update + G2P; keys once
    *count = int64_t(nsteps) * ((sort_every(*p) > 1 ? 1 : 0) + sort + 3) + 1;
  }
  return FFMPM_OK;
}

int ffmpm_p2g(const ffmpm_params* p, const ffmpm_particles* P, ffmpm_grid* grid, void* ws, size_t ws_bytes,
              void* stream) {
  Layout L;
  if (!P || !grid || !grid->velocity || !grid->mass) return FFMPM_ERR_BADARG;
  int rc = prologue(p, P->n, ws, ws_bytes, &L);
  if (rc != FFMPM_OK) return rc;
  if (!particles_ok(*p, P, p->model == FFMPM_MODEL_SNOW)) return FFMPM_ERR_BADARG;
  if (P->n == 0) return FFMPM_OK;
  Ws w = bind(ws, L);
  return dispatch<P2GOp>(*p, L, w, P, grid, static_cast<cudaStream_t>(stream));
}

int ffmpm_grid_op(const ffmpm_params* p, ffmpm_grid* grid, void* stream) {
  Layout L;
  if (!p || !make_layout(*p, 0, &L)) return FFMPM_ERR_BADARG;
  if (!grid || !grid->velocity || !grid->mass) return FFMPM_ERR_BADARG;
  return dispatch<GridOp>(*p, grid, static_cast<cudaStream_t>(stream));
}

int ffmpm_g2p(const ffmpm_params* p, const ffmpm_grid* grid, ffmpm_particles* P, void* ws, size_t ws_bytes,
              void* stream) {
  Layout L;
  if (!P || !grid || !grid->velocity) return FFMPM_ERR_BADARG;
  int rc = prologue(p, P->n, ws, ws_bytes, &L);
  if (rc != FFMPM_OK) return rc;
  if (!particles_ok(*p, P, p->dim == 2 || p->model == FFMPM_MODEL_SNOW)) return FFMPM_ERR_BADARG;
  if (P->n == 0) return FFMPM_OK;
  Ws w = bind(ws, L);
  return dispatch<G2POp>(*p, L, w, grid, P, static_cast<cudaStream_t>(stream));
}

int ffmpm_sort_by_block(const ffmpm_params* p, const void* x, int64_t n, uint32_t* keys_out, uint32_t* perm_out,
                        void* ws, size_t ws_bytes, void* stream) {
  Layout L;
  if (!p || !make_layout(*p, n, &L)) return FFMPM_ERR_BADARG;
  if (!ws || ws_bytes < L.total || (reinterpret_cast<uintptr_t>(ws) & 255)) return FFMPM_ERR_WORKSPACE;
  if (n == 0) return FFMPM_OK;
  if (!x) return FFMPM_ERR_BADARG;
  Ws w = bind(ws, L);
  return dispatch<SortOp>(*p, L, w, x, keys_out, perm_out, static_cast<cudaStream_t>(stream));
}

int ffmpm_diagnostics_fp64(const ffmpm_params* p, const ffmpm_particles* P, double* out, void* stream) {
  Layout L;
  if (!p || !make_layout(*p, 0, &L) || !P || !out) return FFMPM_ERR_BADARG;
  if (P->n > 0 && (!P->x || !P->v || !P->F)) return FFMPM_ERR_BADARG;
  return dispatch<DiagOp>(*p, P, out, static_cast<cudaStream_t>(stream));
}

}  // extern "C"
