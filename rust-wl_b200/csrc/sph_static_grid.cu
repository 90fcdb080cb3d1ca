// Neighbour-table build that allocates nothing: vxl_sph_build_grid_static.
//
// Some callers cannot allocate device memory while they run: an engine that reserves
// one fixed arena for all GPU work at start-up and forbids further cudaMalloc, or a
// per-frame plugin that must not call cudaMalloc/cudaFree because both can synchronise
// the device and stall the host's frame loop. This entry point serves them. The caller
// passes device buffers for the input positions and the output table; the working
// memory the sort needs (cell counts, per-particle cell and rank, the unordered
// placement and the scan partials) lives in one file-scope __device__ array of fixed
// size, which every GPU that loads this library holds until the process exits.
//
// The table is the one the handle-based path builds at the start of each substep
// (crates/vxl-phys-fluid/src/grid.rs:29-76 with the grid rule of
// crates/vxl-phys-core/src/grid.rs:34-50): items[] = particle indices grouped by cell,
// ascending index inside a cell; start[c]..start[c+1] = the slots of cell c.
#include <cstring>
#include <mutex>
#include <string>

#include "sph_device.cuh"
#include "vxl_sph.h"
#include "vxl_sph_internal.h"

using namespace vxl;

namespace {

constexpr uint32_t kStaticMaxParticles = 1u << 19;  // 524,288
constexpr uint32_t kStaticMaxCells = 1u << 19;      // 524,288
constexpr int kTile = 2048;
constexpr int kTileThreads = 256;
constexpr uint32_t kMaxTiles = (kStaticMaxCells + kTile - 1) / kTile;  // 256
constexpr uint32_t kBoxBlocks = 148 * 2;  // blocks of ks_box, each leaving one box
constexpr int kBoxThreads = 256;
constexpr int kWideThreads = 512;     // block of ks_canon_wide
constexpr uint32_t kWideRank = 2048;  // cells up to this size are ranked entry against entry
constexpr uint32_t kMaxWide = kStaticMaxParticles / (kWideRank + 1) + 1;  // larger cells there can be
constexpr uint32_t kWideSmemWords = (kStaticMaxParticles + 31) / 32;      // 64 KB: a bit per particle

constexpr size_t align256(size_t x) { return (x + 255) & ~size_t(255); }
constexpr size_t kCountsOff = 0;
constexpr size_t kRankOff = align256(kCountsOff + (size_t)(kStaticMaxCells + 1) * 4);
constexpr size_t kTmpOff = align256(kRankOff + (size_t)kStaticMaxParticles * 8);
constexpr size_t kPartialOff = align256(kTmpOff + (size_t)kStaticMaxParticles * 4);
constexpr size_t kGridOff = align256(kPartialOff + (size_t)kMaxTiles * 4);
constexpr size_t kCtlOff = align256(kGridOff + sizeof(GridBox));
constexpr size_t kScratchBytes = align256(kCtlOff + sizeof(uint32_t) * (3 + kMaxWide));
static_assert(kBoxBlocks * 6 <= kStaticMaxParticles, "the blocks' boxes use the placement's words");

// Control words at kCtlOff: blocks done in ks_box and in ks_scan_partial, cells above
// kWideRank, and their indices. The array starts zeroed; ks_keys, between their users, zeroes
// the three counts, so that whatever a call left in them lasts no longer than the next.
struct Ctl {
  uint32_t box_done, scan_done, nwide;
  uint32_t wide[kMaxWide];
};

// The working memory (about 8.4 MB). Host code must not pass this name to a kernel: on
// the host it is only a stand-in; the device address comes from cudaGetSymbolAddress.
static __device__ __align__(256) unsigned char g_grid_scratch[kScratchBytes];

std::mutex g_mu;
void* g_scratch_addr[128] = {};  // per device ordinal, resolved on the first call there

vxl_status fail(vxl_status s, const std::string& m) {
  vxl_set_last_error(m.c_str());  // read back through vxl_sph_last_error()
  return s;
}

// Bounding box and grid, and the counts zeroed (the array keeps the previous call's
// contents), in one launch: each block leaves the box of its particles, and whichever finishes
// last (an atomic count; nothing waits) reduces the blocks' boxes and applies the grid rule.
// Six global atomics per warp on one box took 13k turns per address at 430k particles.
__global__ void __launch_bounds__(kBoxThreads) ks_box(const float* __restrict__ xyz, uint32_t n, float h,
                                                      uint32_t max_bins, uint32_t* __restrict__ boxes, GridBox* g,
                                                      uint32_t* __restrict__ counts, Ctl* ctl) {
  __shared__ uint32_t s_box[6][kBoxThreads / 32];
  __shared__ bool last;
  const uint32_t step = gridDim.x * kBoxThreads;
  for (uint32_t c = blockIdx.x * kBoxThreads + threadIdx.x; c <= max_bins; c += step) counts[c] = 0u;
  uint32_t mn[3] = {~0u, ~0u, ~0u}, mx[3] = {0u, 0u, 0u};
  for (uint32_t i = blockIdx.x * kBoxThreads + threadIdx.x; i < n; i += step)
#pragma unroll
    for (int a = 0; a < 3; ++a) {
      const float v = xyz[3 * i + a];
      if (v == v) {  // NaN never wins
        mn[a] = min(mn[a], f2o(v));
        mx[a] = max(mx[a], f2o(v));
      }
    }
  auto reduce = [&]() {  // over the block, into thread a < 6's s_box[a][0]
    const uint32_t lane = threadIdx.x & 31, w = threadIdx.x >> 5;
#pragma unroll
    for (int a = 0; a < 3; ++a) {
      const uint32_t lo = __reduce_min_sync(0xffffffffu, mn[a]), hi = __reduce_max_sync(0xffffffffu, mx[a]);
      if (lane == 0) {
        s_box[a][w] = lo;
        s_box[3 + a][w] = hi;
      }
    }
    __syncthreads();
    if (threadIdx.x < 6) {
      uint32_t v = s_box[threadIdx.x][0];
      for (int k = 1; k < kBoxThreads / 32; ++k)
        v = threadIdx.x < 3 ? min(v, s_box[threadIdx.x][k]) : max(v, s_box[threadIdx.x][k]);
      s_box[threadIdx.x][0] = v;
    }
    __syncthreads();
  };
  reduce();
  if (threadIdx.x < 6) boxes[6 * blockIdx.x + threadIdx.x] = s_box[threadIdx.x][0];
  __threadfence();  // this block's box is visible before it counts itself done
  __syncthreads();
  if (threadIdx.x == 0) last = atomicAdd(&ctl->box_done, 1u) == gridDim.x - 1;
  __syncthreads();
  if (!last) return;
  __threadfence();
#pragma unroll
  for (int a = 0; a < 3; ++a) {
    mn[a] = ~0u;
    mx[a] = 0u;
  }
  for (uint32_t k = threadIdx.x; k < gridDim.x; k += kBoxThreads)
#pragma unroll
    for (int a = 0; a < 3; ++a) {
      mn[a] = min(mn[a], __ldcg(boxes + 6 * k + a));  // written by other blocks: skip L1
      mx[a] = max(mx[a], __ldcg(boxes + 6 * k + 3 + a));
    }
  __syncthreads();
  reduce();
  if (threadIdx.x == 0) {
    GridBox gb;
    grid_box(o2f(s_box[0][0]), o2f(s_box[1][0]), o2f(s_box[2][0]), o2f(s_box[3][0]), o2f(s_box[4][0]), o2f(s_box[5][0]),
             h, max_bins, gb);
    *g = gb;
  }
}

__global__ void ks_keys(const float* __restrict__ xyz, uint32_t n, const GridBox* __restrict__ gp,
                        uint32_t* __restrict__ counts, uint2* __restrict__ cellrank, Ctl* ctl) {
  const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i == 0) ctl->box_done = ctl->scan_done = ctl->nwide = 0u;
  const bool valid = i < n;
  uint32_t c = 0xffffffffu;
  if (valid) c = cell_index(*gp, xyz[3 * i], xyz[3 * i + 1], xyz[3 * i + 2]);
  const uint32_t active = __ballot_sync(0xffffffffu, valid);
  if (!valid) return;
  const uint32_t peers = __match_any_sync(active, c);
  const int lane = threadIdx.x & 31;
  const int leader = __ffs(peers) - 1;
  uint32_t base = 0;
  if (lane == leader) base = atomicAdd(&counts[c], (uint32_t)__popc(peers));
  base = __shfl_sync(peers, base, leader);
  cellrank[i] = make_uint2(c, base + __popc(peers & ((1u << lane) - 1u)));
}

// Per-tile sums of the counts, and in the block that finishes last their exclusive scan in
// place and the total.
__global__ void ks_scan_partial(const uint32_t* __restrict__ counts, const GridBox* __restrict__ gp,
                                uint32_t* __restrict__ partial, uint32_t* __restrict__ start, Ctl* ctl) {
  const uint32_t total = gp->total, base = blockIdx.x * kTile, ntiles = (total + kTile - 1) / kTile;
  if (base >= total) return;
  uint32_t sum = 0;
  for (uint32_t i = base + threadIdx.x; i < min(base + kTile, total); i += kTileThreads) sum += counts[i];
  sum = __reduce_add_sync(0xffffffffu, sum);
  __shared__ uint32_t ws[kTileThreads / 32];
  __shared__ bool last;
  if ((threadIdx.x & 31) == 0) ws[threadIdx.x >> 5] = sum;
  __syncthreads();
  if (threadIdx.x == 0) {
    uint32_t t = 0;
    for (int w = 0; w < kTileThreads / 32; ++w) t += ws[w];
    partial[blockIdx.x] = t;
    __threadfence();
    last = atomicAdd(&ctl->scan_done, 1u) == ntiles - 1;
  }
  __syncthreads();
  if (!last) return;
  __threadfence();
  static_assert(kTileThreads >= (int)kMaxTiles, "a thread per tile");
  const uint32_t t = threadIdx.x, lane = t & 31, w = t >> 5;
  const uint32_t v = t < ntiles ? __ldcg(partial + t) : 0u;
  uint32_t incl = v;
#pragma unroll
  for (int off = 1; off < 32; off <<= 1) {
    const uint32_t y = __shfl_up_sync(0xffffffffu, incl, off);
    if ((int)lane >= off) incl += y;
  }
  __syncthreads();
  if (lane == 31) ws[w] = incl;
  __syncthreads();
  for (uint32_t k = 0; k < w; ++k) incl += ws[k];
  if (t < ntiles) partial[t] = incl - v;
  if (t == kTileThreads - 1) start[total] = incl;
}

__global__ void ks_scan_final(const uint32_t* __restrict__ counts, const GridBox* __restrict__ gp,
                              const uint32_t* __restrict__ partial, uint32_t* __restrict__ start, Ctl* ctl) {
  const uint32_t total = gp->total, base = blockIdx.x * kTile;
  if (base >= total) return;
  constexpr int kPer = kTile / kTileThreads;
  uint32_t v[kPer], local = 0;
  const uint32_t i0 = base + threadIdx.x * kPer;
#pragma unroll
  for (int q = 0; q < kPer; ++q) {
    v[q] = (i0 + q) < total ? counts[i0 + q] : 0u;
    local += v[q];
  }
  uint32_t incl = local;
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
#pragma unroll
  for (int off = 1; off < 32; off <<= 1) {
    const uint32_t y = __shfl_up_sync(0xffffffffu, incl, off);
    if (lane >= off) incl += y;
  }
  __shared__ uint32_t ws[kTileThreads / 32];
  if (lane == 31) ws[wid] = incl;
  __syncthreads();
  uint32_t woff = 0;
  for (int w = 0; w < wid; ++w) woff += ws[w];
  uint32_t run = partial[blockIdx.x] + woff + incl - local;
#pragma unroll
  for (int q = 0; q < kPer; ++q) {
    if ((i0 + q) < total) start[i0 + q] = run;
    if (v[q] > kWideRank) {
      const uint32_t at = atomicAdd(&ctl->nwide, 1u);  // any order: a block each
      if (at < kMaxWide) ctl->wide[at] = i0 + q;
    }
    run += v[q];
  }
}

__global__ void ks_place(const uint2* __restrict__ cellrank, const uint32_t* __restrict__ start, uint32_t n,
                         uint32_t* __restrict__ tmp) {
  const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const uint2 cr = cellrank[i];
  tmp[start[cr.x] + cr.y] = i;
}

// The placed indices of each cell of at most kWideRank entries in ascending order, into
// items: a thread per entry ranks it against its cell's entries (the lanes of a cell read the
// same ones). A warp per cell, and a pass of blocks over all cells for those above 32 entries,
// took most of a call's 182 us at 430k particles; a call takes 76 now (62 -> 54 at 125: launches).
__global__ void __launch_bounds__(256) ks_canon(const uint32_t* __restrict__ tmp, const uint2* __restrict__ cellrank,
                                                const uint32_t* __restrict__ start, uint32_t n,
                                                uint32_t* __restrict__ items) {
  const uint32_t e = blockIdx.x * blockDim.x + threadIdx.x;
  if (e >= n) return;
  const uint32_t key = tmp[e], c = cellrank[key].x;
  const uint32_t b = start[c], end = start[c + 1];
  if (end - b > kWideRank) return;  // ks_canon_wide
  uint32_t dst = b, j = b;
  for (; j + 4 <= end; j += 4) {
    const uint32_t k0 = tmp[j], k1 = tmp[j + 1], k2 = tmp[j + 2], k3 = tmp[j + 3];
    dst += (k0 < key ? 1u : 0u) + (k1 < key ? 1u : 0u) + (k2 < key ? 1u : 0u) + (k3 < key ? 1u : 0u);
  }
  for (; j < end; ++j) dst += tmp[j] < key ? 1u : 0u;
  items[dst] = key;
}

// Cells above kWideRank entries, a block per cell in turn: the cell's indices are distinct
// values below n, so they are set in a bitmap of n bits in shared memory and read back in
// ascending order (n / 32 words scanned once, whatever the cell's size).
__global__ void __launch_bounds__(kWideThreads) ks_canon_wide(const uint32_t* __restrict__ tmp,
                                                              const uint32_t* __restrict__ start,
                                                              const Ctl* __restrict__ ctl, uint32_t n,
                                                              uint32_t* __restrict__ items) {
  extern __shared__ uint32_t sm[];  // kWideSmemWords
  __shared__ uint32_t s_warp[kWideThreads / 32];
  const uint32_t t = threadIdx.x, lane = t & 31, wid = t >> 5;
  for (uint32_t q = blockIdx.x; q < min(ctl->nwide, kMaxWide); q += gridDim.x) {
    const uint32_t c = ctl->wide[q], b = start[c], m = start[c + 1] - b;
    const uint32_t words = (n + 31) / 32;
    for (uint32_t w = t; w < words; w += kWideThreads) sm[w] = 0;
    __syncthreads();
    for (uint32_t e = t; e < m; e += kWideThreads) {
      const uint32_t v = tmp[b + e];
      atomicOr(&sm[v >> 5], 1u << (v & 31));
    }
    __syncthreads();
    // thread t owns words [w0, w1); exclusive scan of their set bits over the block
    const uint32_t per = (words + kWideThreads - 1) / kWideThreads;
    const uint32_t w0 = min(t * per, words), w1 = min(w0 + per, words);
    uint32_t cnt = 0;
    for (uint32_t w = w0; w < w1; ++w) cnt += __popc(sm[w]);
    uint32_t incl = cnt;
#pragma unroll
    for (int off = 1; off < 32; off <<= 1) {
      const uint32_t y = __shfl_up_sync(0xffffffffu, incl, off);
      if ((int)lane >= off) incl += y;
    }
    if (lane == 31) s_warp[wid] = incl;
    __syncthreads();
    uint32_t r = incl - cnt;
    for (uint32_t k = 0; k < wid; ++k) r += s_warp[k];
    for (uint32_t w = w0; w < w1; ++w) {
      uint32_t bits = sm[w];
      while (bits) {
        const uint32_t bit = (uint32_t)__ffs(bits) - 1u;
        bits &= bits - 1u;
        items[b + r++] = w * 32u + bit;
      }
    }
    __syncthreads();
  }
}

// Device address of the scratch array on the current device (resolved once per device).
vxl_status scratch_on(int dev, unsigned char** out) {
  if (dev < 0 || dev >= 128) return fail(VXL_INVALID_ARGUMENT, "device ordinal out of range");
  std::lock_guard<std::mutex> lk(g_mu);
  if (!g_scratch_addr[dev]) {
    void* p = nullptr;
    cudaError_t e = cudaGetSymbolAddress(&p, g_grid_scratch);
    if (e != cudaSuccess || !p)
      return fail(VXL_CUDA_ERROR, std::string("cudaGetSymbolAddress(scratch): ") + cudaGetErrorString(e));
    e = cudaFuncSetAttribute(ks_canon_wide, cudaFuncAttributeMaxDynamicSharedMemorySize,
                             (int)(kWideSmemWords * sizeof(uint32_t)));
    if (e != cudaSuccess)
      return fail(VXL_CUDA_ERROR, std::string("cudaFuncSetAttribute(ks_canon_wide): ") + cudaGetErrorString(e));
    g_scratch_addr[dev] = p;
  }
  *out = (unsigned char*)g_scratch_addr[dev];
  return VXL_OK;
}

}  // namespace

extern "C" vxl_status vxl_sph_build_grid_static(const float* d_pos_xyz, uint32_t n, float h, uint32_t max_bins,
                                                uint32_t* d_items, uint32_t* d_start, uint64_t start_cap,
                                                vxl_sph_grid_info* info, void* cuda_stream) {
  if (!d_pos_xyz || !d_items || !d_start || !info) return fail(VXL_NULL_POINTER, "NULL argument");
  if (info->hdr.size != sizeof(vxl_sph_grid_info) || info->hdr.version != VXL_SPH_ABI_VERSION)
    return fail(VXL_SIZE_MISMATCH, "grid_info header");
  if (n == 0 || n > kStaticMaxParticles)
    return fail(VXL_INVALID_ARGUMENT, "n must be in [1, " + std::to_string(kStaticMaxParticles) + "]");
  const uint32_t budget = max_bins ? max_bins : kStaticMaxCells;
  if (budget > kStaticMaxCells)
    return fail(VXL_INVALID_ARGUMENT, "max_bins above the static limit of " + std::to_string(kStaticMaxCells));
  if (start_cap < (uint64_t)budget + 1)
    return fail(VXL_SIZE_MISMATCH, "start must hold max_bins + 1 entries");
  int dev = -1;
  if (cudaGetDevice(&dev) != cudaSuccess) return fail(VXL_CUDA_ERROR, "cudaGetDevice failed");
  unsigned char* base = nullptr;
  vxl_status st = scratch_on(dev, &base);
  if (st != VXL_OK) return st;
  cudaStream_t s = (cudaStream_t)cuda_stream;
  uint32_t* counts = (uint32_t*)(base + kCountsOff);
  uint2* cellrank = (uint2*)(base + kRankOff);
  uint32_t* tmp = (uint32_t*)(base + kTmpOff);
  uint32_t* partial = (uint32_t*)(base + kPartialOff);
  GridBox* g = (GridBox*)(base + kGridOff);
  Ctl* ctl = (Ctl*)(base + kCtlOff);
  const uint32_t nblk = (n + 255) / 256, tiles = (budget + kTile - 1) / kTile;
  ks_box<<<kBoxBlocks, kBoxThreads, 0, s>>>(d_pos_xyz, n, h, budget, tmp, g, counts, ctl);
  ks_keys<<<nblk, 256, 0, s>>>(d_pos_xyz, n, g, counts, cellrank, ctl);
  ks_scan_partial<<<tiles, kTileThreads, 0, s>>>(counts, g, partial, d_start, ctl);
  ks_scan_final<<<tiles, kTileThreads, 0, s>>>(counts, g, partial, d_start, ctl);
  ks_place<<<nblk, 256, 0, s>>>(cellrank, d_start, n, tmp);
  ks_canon<<<nblk, 256, 0, s>>>(tmp, cellrank, d_start, n, d_items);
  ks_canon_wide<<<32, kWideThreads, kWideSmemWords * sizeof(uint32_t), s>>>(tmp, d_start, ctl, n, d_items);
  cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) return fail(VXL_CUDA_ERROR, std::string("grid build launch: ") + cudaGetErrorString(e));
  GridBox hg;
  e = cudaMemcpyAsync(&hg, g, sizeof(GridBox), cudaMemcpyDeviceToHost, s);
  if (e == cudaSuccess) e = cudaStreamSynchronize(s);
  if (e != cudaSuccess) return fail(VXL_CUDA_ERROR, std::string("grid build: ") + cudaGetErrorString(e));
  info->min[0] = hg.minx;
  info->min[1] = hg.miny;
  info->min[2] = hg.minz;
  info->inv = hg.inv;
  info->bin = hg.bin;
  info->dims[0] = hg.nx;
  info->dims[1] = hg.ny;
  info->dims[2] = hg.nz;
  info->total = hg.total;
  return VXL_OK;
}
