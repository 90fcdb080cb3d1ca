// Multi-scene WCSPH engine: the device kernels of one substep for any number of
// resident scenes (sm_100a). One scene is the plain drop-in; many scenes are the
// batched and served forms.
//
// Layout. All scenes share one pool of particle slots, packed without gaps in scene
// order: scene q owns slots [base_q, base_q + n_q) and its particles never leave that
// range. Per slot (structure of arrays):
//   pos[s]  float4 (x, y, z, m)   m = +particle mass for fluid, -pmass for boundary
//   vel[s]  float4 (vx, vy, vz, 0)
//   orig[s] global reference index (base_q + the particle's index in its scene);
//           slot_of[orig[s]] == s
// Each substep every scene gets its own grid (the reference's grid rule on its own
// AABB, crates/vxl-phys-core/src/grid.rs:34-50) and a range of a global cell space
// [cell_off_q, cell_off_q + cells_q), assigned in scene order. A particle's key is
// cell_off_q + its cell, so one counting sort over the global cells is a segmented sort
// that keeps each scene inside its slot range, and inside every cell the slots ascend by
// reference index: the reference's cells (crates/vxl-phys-fluid/src/grid.rs:29-76), but in
// z-major order (cell_slot; the reference's table has x outermost, which the export
// restores). Walking a scene's 27 cells in the reference's (dz, dy, dx) order visits
// neighbours in the order of UniformGrid::for_neighbors_in (grid.rs:115-155), so every
// per-particle sum matches the reference's CPU path bit for bit, and the three cells of a
// (dz, dy) row are one run of slots.
//
// Work list. The particle kernels run persistent blocks over a list of tiles
// (scene, first slot, count): a block takes the next tile from an atomic counter, so the
// scene of a tile is uniform and scenes of very different sizes balance across SMs.
//
// Substep: gridbox (per scene) -> cell offsets -> keys -> scan -> place -> canon ->
// filter words -> density + EOS (+ neighbour lists) -> force + XSPH + integrate -> boundary reactions ->
// per-span reduction.
#pragma once

#include "sph_device.cuh"

// Resident threads per SM the density and force passes are compiled for (register
// budget = 65536 / this). Force at 1280 / 1536 instead of 1024 (which does not spill) is 11% / 56%
// slower on the 1M dam break, 8% / 52% on the 10M one. Density at 768 is 20% slower than at 1024; at 1280 it was
// 1-2% faster with queues of 12 windows (kWalkQueue), but that has no room for longer ones.
#ifndef VXL_DENSITY_THREADS_PER_SM
#define VXL_DENSITY_THREADS_PER_SM 1024
#endif
#ifndef VXL_FORCE_THREADS_PER_SM
#define VXL_FORCE_THREADS_PER_SM 1024
#endif


namespace vxl {

constexpr uint32_t kErrCellCap = 1u << 3;  // the scenes' cells exceed the cell capacity
constexpr uint32_t kErrScanWait = 1u << 4;  // the scan's wait ran out (with kErrCellCap: the substep is skipped)

// Per-scene device record (one per scene of the engine). The fields up to `g` are
// written by the host (constants, substep dt, slot range); the rest by the kernels.
struct SceneDev {
  SphConst k;
  float dt, vmax, vmax2, pad0;
  uint32_t base;        // first slot
  uint32_t count;       // slots (fluid + boundary)
  uint32_t prov_first;  // the scene's providers in the engine's provider array
  uint32_t prov_count;  // 0: no provider walls
  GridBox g;            // this substep's grid
  uint32_t cell_off;    // first global cell this substep
  uint32_t cells;       // cells this substep
  uint32_t fbox[6];     // fluid AABB accumulator (ordered uint)
  uint32_t bbox[6];     // boundary AABB (fixed within a tick)
};

// Per-body pose of the device-side boundary rebuild.
struct BodyPoseDev {
  float px, py, pz;
  float qx, qy, qz, qw;
  float vx, vy, vz;
  float wx, wy, wz;
};

// A rigid body of the device-side coupling loop: pose and velocities (the BodyPoseDev
// fields, same names), mass properties, and the global index of the span whose reaction
// drives it (~0u: none).
struct RigidBodyDev {
  float px, py, pz;
  float qx, qy, qz, qw;
  float vx, vy, vz;
  float wx, wy, wz;
  float inv_mass, iix, iiy, iiz;
  uint32_t dynamic, span;
};

struct TileDev {
  uint32_t scene, first, count, pad;
};

// Body span (global reference indices [start, end)) and its reduction chunks.
struct SpanDev {
  uint32_t body;
  float ox, oy, oz;
  uint32_t start, end;
  uint32_t rigid;  // coupled rigid body whose position is the torque origin (~0u: use ox, oy, oz)
  uint32_t bfirst;  // the scene's first boundary particle (global reference index) ...
  uint32_t bword;   // ... and its word in the wet mask of k_e_bforce
};

struct LongSpan {  // a span above kReactExactSpan, summed by a block of its own
  uint32_t span;
};

// Spans of at most this many particles (bodies) are summed by one warp each; larger ones
// (tank walls) by one block each. Both add the terms in index order: the reference's sum,
// bit for bit.
constexpr uint32_t kReactExactSpan = 8192;
constexpr int kReactThreads = 512;                       // block of k_react_long: staging warps, the last one sums
constexpr uint32_t kReactBatch = kReactThreads - 32;     // terms a block stages per step
constexpr uint32_t kReactWords = 256;                    // mask words (8,192 particles) a block compacts at a time
constexpr float kReactArm = 1e18f;                       // arms below this keep every product with a zero force zero
constexpr int kReactSpanWarps = 2;                       // spans per block of k_react_spans (one warp each)

// Engine-wide control block.
constexpr int kWorkSlots = 16;  // persistent-kernel work counters per substep
struct EngineCtl {
  uint32_t cells;  // sum of the scenes' cells this substep
  uint32_t err;
  uint32_t slow_gathers;
  uint32_t epoch;    // substep counter: wet[c] == epoch marks cells holding fluid this substep
  uint32_t work[kWorkSlots];
};

// Work counter indices (zeroed at the start of every substep). The provider-wall passes
// keep their per-substep results in slots 4-6: pushed particles, "some pushed pair is
// closer than 0.2 h", "the separation moved a particle".
enum WorkId : int {
  kWorkDensity = 0, kWorkForce = 1, kWorkBforce = 2, kWorkScan = 3,
  kWorkPushed = 4, kWorkTrigger = 5, kWorkMoved = 6
};

// Provider walls (analytic ProviderColliders queried on the device). A plane of a FACES
// provider is (axis, d = plane coordinate, sign); of a CONVEX provider (n, d).
struct WallPlaneDev {
  float nx, ny, nz, d;
  uint32_t axis;
  float sign;
  uint32_t pad0, pad1;
};

// One side (mirror or projection) of the contact tables: ent[global reference index] =
// entry + 1 (0: no planes), entry e owning planes [start[e], start[e + 1]), each plane two
// float4 (contact point, outward normal).
struct ContactTableDev {
  const uint32_t* ent;
  const uint32_t* start;
  const float4* planes;
};

struct ProviderDev {
  uint32_t kind, first, count, has_bounds;
  float bminx, bminy, bminz, bmaxx, bmaxy, bmaxz;
  uint32_t pad0, pad1;
};

constexpr uint32_t kProviderFaces = 0u, kProviderConvex = 1u;
// A contact table (any ProviderColliders, gathered on the host once per tick, as the
// reference's GPU tier does: crates/vxl-phys-gpu/src/pipeline/walls.rs:143-215) is one more
// provider of the scene, after its analytic ones, queried by particle.
constexpr uint32_t kProviderTable = 2u;
constexpr uint32_t kMaxWallPlanes = 8;     // mirror planes per particle (fluid_density.rs:110)
constexpr uint32_t kPushedChunk = 4096;    // reference indices per block of the pushed-list passes

namespace {

constexpr int kScanTile = 2048;
constexpr int kScanThreads = 256;
constexpr int kBGatherCap = 64;
// Density walk: windows queued per thread. h-sized bins need 9 or 10 (a row each), 2h bins
// about 20. On the 10M dam break 12 / 14 / 22 are 10% / 6% / 2% slower than 18 (shorter queues are
// emptied more often, longer ones leave less L1), on the 1M one all are the same.
#ifndef VXL_WALK_QUEUE
#define VXL_WALK_QUEUE 18
#endif
constexpr uint32_t kWalkQueue = VXL_WALK_QUEUE;
constexpr uint32_t kListPrefetch = 4;  // force pass: list entries fetched into L2 this far ahead

// Block-level ordered-uint min/max of (x, y, z), one atomic per component into acc.
__device__ __forceinline__ void block_bbox_accumulate(uint32_t* acc, float x, float y, float z, bool valid) {
  uint32_t mn[3], mx[3];
  const float v[3] = {x, y, z};
#pragma unroll
  for (int a = 0; a < 3; ++a) {
    const bool ok = valid && (v[a] == v[a]);  // NaN never wins (Rust f32::min/max ignore NaN)
    mn[a] = ok ? f2o(v[a]) : 0xffffffffu;
    mx[a] = ok ? f2o(v[a]) : 0u;
  }
#pragma unroll
  for (int off = 16; off > 0; off >>= 1) {
#pragma unroll
    for (int a = 0; a < 3; ++a) {
      mn[a] = min(mn[a], __shfl_xor_sync(0xffffffffu, mn[a], off));
      mx[a] = max(mx[a], __shfl_xor_sync(0xffffffffu, mx[a], off));
    }
  }
  __shared__ uint32_t s_mn[3][32], s_mx[3][32];
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5, nw = (blockDim.x + 31) >> 5;
  if (lane == 0) {
#pragma unroll
    for (int a = 0; a < 3; ++a) {
      s_mn[a][wid] = mn[a];
      s_mx[a][wid] = mx[a];
    }
  }
  __syncthreads();
  if (wid == 0) {
#pragma unroll
    for (int a = 0; a < 3; ++a) {
      mn[a] = lane < nw ? s_mn[a][lane] : 0xffffffffu;
      mx[a] = lane < nw ? s_mx[a][lane] : 0u;
    }
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) {
#pragma unroll
      for (int a = 0; a < 3; ++a) {
        mn[a] = min(mn[a], __shfl_xor_sync(0xffffffffu, mn[a], off));
        mx[a] = max(mx[a], __shfl_xor_sync(0xffffffffu, mx[a], off));
      }
    }
    if (lane == 0) {
#pragma unroll
      for (int a = 0; a < 3; ++a) {
        if (mn[a] != 0xffffffffu) atomicMin(&acc[a], mn[a]);
        if (mx[a] != 0u) atomicMax(&acc[3 + a], mx[a]);
      }
    }
  }
  __syncthreads();
}

// Next tile of a persistent kernel (block-uniform); >= ntiles means done.
__device__ __forceinline__ uint32_t next_tile(uint32_t* counter) {
  __shared__ uint32_t s_tile;
  if (threadIdx.x == 0) s_tile = atomicAdd(counter, 1u);
  __syncthreads();
  const uint32_t t = s_tile;
  __syncthreads();
  return t;
}

// Tile scheduling of the particle passes. A grid of at least ntiles blocks runs one
// block per tile (the hardware block scheduler balances); a smaller grid is persistent
// and its blocks draw tiles from the atomic counter until the list is exhausted.
__device__ __forceinline__ uint32_t first_tile(uint32_t* counter, uint32_t ntiles) {
  return gridDim.x >= ntiles ? blockIdx.x : next_tile(counter);
}
__device__ __forceinline__ uint32_t following_tile(uint32_t* counter, uint32_t ntiles) {
  return gridDim.x >= ntiles ? ntiles : next_tile(counter);
}

// ---------------------------------------------------------------- set-up kernels

// Scatter one scene's host-order input (xyz triples, scene-local index) into its slots
// [base, base + n) in reference order.
__global__ void k_e_init_scene(const float* __restrict__ pin, const float* __restrict__ vin,
                               const float* __restrict__ pm, float4* __restrict__ pos, float4* __restrict__ vel,
                               uint32_t* __restrict__ orig, uint32_t* __restrict__ slot_of,
                               float4* __restrict__ bpos, uint32_t base, uint32_t n, uint32_t nf, float mass) {
  const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const float x = pin[3 * i], y = pin[3 * i + 1], z = pin[3 * i + 2];
  const bool fluid = i < nf;
  const uint32_t g = base + i;
  pos[g] = make_float4(x, y, z, fluid ? mass : -pm[i]);
  vel[g] = make_float4(vin[3 * i], vin[3 * i + 1], vin[3 * i + 2], 0.0f);
  orig[g] = g;
  slot_of[g] = g;
  if (!fluid) bpos[g] = make_float4(x, y, z, 0.0f);
}

// Overwrite one scene's positions/velocities (scene-local reference order input),
// keeping its current slot order.
__global__ void k_e_write_scene(const float* __restrict__ pin, const float* __restrict__ vin,
                                float4* __restrict__ pos, float4* __restrict__ vel,
                                const uint32_t* __restrict__ orig, float4* __restrict__ bpos, uint32_t base,
                                uint32_t n, uint32_t nf) {
  const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const uint32_t s = base + i;
  const uint32_t o = orig[s] - base;
  if (pin) {
    float4 p = pos[s];
    p.x = pin[3 * o];
    p.y = pin[3 * o + 1];
    p.z = pin[3 * o + 2];
    pos[s] = p;
    if (o >= nf) bpos[base + o] = make_float4(p.x, p.y, p.z, 0.0f);
  }
  if (vin) vel[s] = make_float4(vin[3 * o], vin[3 * o + 1], vin[3 * o + 2], 0.0f);
}

// Boundary segment re-upload of one scene (crates/vxl-phys-gpu/src/pipeline/coupling.rs:
// 20-50): boundary particle k of the scene sits in slot slot_of[base + nf + k].
__global__ void k_e_upload_boundary(const float* __restrict__ pin, const float* __restrict__ vin,
                                    float4* __restrict__ pos, float4* __restrict__ vel,
                                    const uint32_t* __restrict__ slot_of, float4* __restrict__ bpos,
                                    uint32_t* __restrict__ bbox_acc, uint32_t base, uint32_t nf, uint32_t nb) {
  const uint32_t q = blockIdx.x * blockDim.x + threadIdx.x;
  const bool valid = q < nb;
  float x = 0, y = 0, z = 0;
  if (valid) {
    const uint32_t g = base + nf + q;
    const uint32_t s = slot_of[g];
    x = pin[3 * q];
    y = pin[3 * q + 1];
    z = pin[3 * q + 2];
    float4 p = pos[s];
    p.x = x;
    p.y = y;
    p.z = z;
    pos[s] = p;
    vel[s] = make_float4(vin[3 * q], vin[3 * q + 1], vin[3 * q + 2], 0.0f);
    bpos[g] = make_float4(x, y, z, 0.0f);
  }
  block_bbox_accumulate(bbox_acc, x, y, z, valid);
}

// AABBs of one scene's fluid (pos.w > 0) and boundary (pos.w < 0) slots into its (emptied)
// accumulators.
__global__ void k_e_bbox(const float4* __restrict__ pos, uint32_t base, uint32_t n, SceneDev* __restrict__ S) {
  const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
  float4 p = make_float4(0, 0, 0, 0);
  if (i < n) p = pos[base + i];
  if (__syncthreads_or(p.w > 0.0f)) block_bbox_accumulate(S->fbox, p.x, p.y, p.z, p.w > 0.0f);
  if (__syncthreads_or(p.w < 0.0f)) block_bbox_accumulate(S->bbox, p.x, p.y, p.z, p.w < 0.0f);
}

__global__ void k_e_box_empty(SceneDev* __restrict__ S, int fluid, int boundary) {
  const uint32_t a = threadIdx.x;
  if (a < 6 && fluid) S->fbox[a] = a < 3 ? 0xffffffffu : 0u;
  if (a < 6 && boundary) S->bbox[a] = a < 3 ? 0xffffffffu : 0u;
}

// set_boundary_particles on the device (crates/vxl-phys-fluid/src/fluid_step.rs:13-53): for
// boundary particle k of a scene (reference order), with body-frame lattice point L and
// its body's pose, world position p = body.pos + rotate(q, L) (Quat::rotate_vec3:
// t = 2 (q.xyz x L); L + q.xyz x t + w t) and velocity v = linvel + angvel x (p - body.pos),
// in f32 in the reference's operation order. Written at the particle's current slot and in
// reference order (bpos); the boundary AABB is re-accumulated. The class/mass word is kept.
__device__ __forceinline__ void cross3(float ax, float ay, float az, float bx, float by, float bz, float& cx,
                                       float& cy, float& cz) {
  cx = ay * bz - az * by;
  cy = az * bx - ax * bz;
  cz = ax * by - ay * bx;
}

template <class Pose>
__global__ void k_e_body_rebuild(const float4* __restrict__ blocal, const Pose* __restrict__ poses,
                                 float4* __restrict__ pos, float4* __restrict__ vel,
                                 const uint32_t* __restrict__ slot_of, float4* __restrict__ bpos,
                                 uint32_t* __restrict__ bbox_acc, uint32_t base, uint32_t nf, uint32_t nb) {
  const uint32_t q = blockIdx.x * blockDim.x + threadIdx.x;
  const bool valid = q < nb;
  float x = 0, y = 0, z = 0;
  if (valid) {
    const uint32_t g = base + nf + q;
    const float4 L = blocal[g];
    const Pose P = poses[__float_as_uint(L.w)];
    float tx, ty, tz;
    cross3(P.qx, P.qy, P.qz, L.x, L.y, L.z, tx, ty, tz);
    tx = tx * 2.0f;
    ty = ty * 2.0f;
    tz = tz * 2.0f;
    float ux, uy, uz;
    cross3(P.qx, P.qy, P.qz, tx, ty, tz, ux, uy, uz);
    const float rx = (L.x + ux) + tx * P.qw;
    const float ry = (L.y + uy) + ty * P.qw;
    const float rz = (L.z + uz) + tz * P.qw;
    x = P.px + rx;
    y = P.py + ry;
    z = P.pz + rz;
    float ax, ay, az;
    cross3(P.wx, P.wy, P.wz, x - P.px, y - P.py, z - P.pz, ax, ay, az);
    const uint32_t s = slot_of[g];
    float4 p = pos[s];
    p.x = x;
    p.y = y;
    p.z = z;
    pos[s] = p;
    vel[s] = make_float4(P.vx + ax, P.vy + ay, P.vz + az, 0.0f);
    bpos[g] = make_float4(x, y, z, 0.0f);
  }
  block_bbox_accumulate(bbox_acc, x, y, z, valid);
}

// Move whole scenes to new bases (the served form's repack): slot ranges are copied into
// the second buffer set, reference indices shifted by the move. from_base/to_base/count
// per moved scene; one block row per scene (blockIdx.y).
__global__ void k_e_move(const float4* __restrict__ pos_in, const float4* __restrict__ vel_in,
                         const uint32_t* __restrict__ orig_in, const float4* __restrict__ bpos_in,
                         float4* __restrict__ pos_out, float4* __restrict__ vel_out, uint32_t* __restrict__ orig_out,
                         float4* __restrict__ bpos_out, const uint4* __restrict__ moves) {
  const uint4 m = moves[blockIdx.y];  // from, to, count, -
  for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < m.z; i += gridDim.x * blockDim.x) {
    pos_out[m.y + i] = pos_in[m.x + i];
    vel_out[m.y + i] = vel_in[m.x + i];
    orig_out[m.y + i] = orig_in[m.x + i] - m.x + m.y;
    bpos_out[m.y + i] = bpos_in[m.x + i];
  }
}

__global__ void k_e_slot_of(const uint32_t* __restrict__ orig, uint32_t* __restrict__ slot_of, uint32_t n) {
  const uint32_t s = blockIdx.x * blockDim.x + threadIdx.x;
  if (s < n) slot_of[orig[s]] = s;
}

// ---------------------------------------------------------------- substep kernels

// Grid boxes and cell offsets (one block, any scene count): each scene's grid for this
// substep (crates/vxl-phys-fluid/src/grid.rs:37-44 -> crates/vxl-phys-core/src/grid.rs:34-50)
// from its AABB accumulators, which are then reset for the force pass's epilogue; then an
// exclusive scan of the scenes' cell counts;
// flags the substep when the total exceeds the cell capacity (every later kernel then
// returns without touching memory).
// A warp for up to 32 scenes, kCelloffThreads threads for more.
constexpr uint32_t kCelloffThreads = 1024;
__global__ void __launch_bounds__(kCelloffThreads) k_e_celloff(SceneDev* __restrict__ sc, uint32_t nscenes,
                                                               EngineCtl* ctl, uint32_t cell_cap) {
  __shared__ uint32_t ws[32];
  const uint32_t lane = threadIdx.x & 31, w = threadIdx.x >> 5, warps = blockDim.x >> 5;
  unsigned long long carry = 0;  // the same in every thread
  if (threadIdx.x < kWorkSlots) ctl->work[threadIdx.x] = 0;  // work counters of this substep
  if (threadIdx.x == 0) ctl->epoch = ctl->epoch + 1u;
  for (uint32_t b0 = 0; b0 < nscenes; b0 += blockDim.x) {
    const uint32_t q = b0 + threadIdx.x;
    uint32_t v = 0;
    if (q < nscenes) {
      // this substep's grid from the AABB accumulators (the reference's rule on all of the
      // scene's particles, crates/vxl-phys-core/src/grid.rs:34-50); reset the fluid one
      SceneDev& s = sc[q];
      float lo[3], hi[3];
      for (int a = 0; a < 3; ++a) {
        lo[a] = fminf(o2f(s.fbox[a]), o2f(s.bbox[a]));
        hi[a] = fmaxf(o2f(s.fbox[3 + a]), o2f(s.bbox[3 + a]));
      }
      GridBox g;
      if (!grid_box(lo[0], lo[1], lo[2], hi[0], hi[1], hi[2], s.k.h, s.k.max_bins, g))
        atomicOr(&ctl->err, kErrGridLoop);
      s.g = g;
      s.cells = g.total;
      for (int a = 0; a < 3; ++a) {
        s.fbox[a] = 0xffffffffu;
        s.fbox[3 + a] = 0u;
      }
      v = g.total;
    }
    // exclusive scan of the scenes' cells (at most 2^21 each: a block's sum fits 32 bits)
    uint32_t incl = v;
#pragma unroll
    for (int off = 1; off < 32; off <<= 1) {
      const uint32_t y = __shfl_up_sync(0xffffffffu, incl, off);
      if ((int)lane >= off) incl += y;
    }
    if (lane == 31) ws[w] = incl;
    __syncthreads();
    uint32_t before = 0, total = 0;
    for (uint32_t k = 0; k < warps; ++k) {
      if (k < w) before += ws[k];
      total += ws[k];
    }
    const unsigned long long ex = carry + before + (incl - v);
    if (q < nscenes) sc[q].cell_off = ex > 0xffffffffull ? 0xffffffffu : (uint32_t)ex;
    carry += total;
    __syncthreads();
  }
  if (threadIdx.x == 0) {
    if (carry > (unsigned long long)cell_cap) {
      atomicOr(&ctl->err, kErrCellCap);
      ctl->cells = 0;
    } else {
      ctl->cells = (uint32_t)carry;
    }
  }
}

// Cell key + arrival rank per slot (tiles, one block per tile in turn). Lanes with equal
// keys share one atomic (warp-aggregated); the rank is only a placement ticket — canon
// makes the final order deterministic. Cells holding a fluid particle get wet[c] = epoch.
__global__ void k_e_keys(const float4* __restrict__ pos, const SceneDev* __restrict__ sc,
                         const TileDev* __restrict__ tiles, uint32_t ntiles, const EngineCtl* __restrict__ ctl,
                         uint32_t* __restrict__ counts, uint2* __restrict__ cellrank, uint32_t* __restrict__ wet) {
  if (ctl->err & kErrCellCap) return;
  const uint32_t epoch = ctl->epoch;
  for (uint32_t t = blockIdx.x; t < ntiles; t += gridDim.x) {
    const TileDev td = tiles[t];
    const GridBox g = sc[td.scene].g;
    const uint32_t off = sc[td.scene].cell_off;
    for (uint32_t b0 = 0; b0 < td.count; b0 += blockDim.x) {
      const uint32_t i = b0 + threadIdx.x;
      const bool valid = i < td.count;
      uint32_t c = 0xffffffffu;
      if (valid) {
        const float4 p = pos[td.first + i];
        c = off + cell_slot(g, p.x, p.y, p.z);
        if (p.w > 0.0f) wet[c] = epoch;
      }
      const uint32_t active = __ballot_sync(0xffffffffu, valid);
      if (valid) {
        const uint32_t peers = __match_any_sync(active, c);
        const int lane = threadIdx.x & 31;
        const int leader = __ffs(peers) - 1;
        uint32_t base = 0;
        if (lane == leader) base = atomicAdd(&counts[c], (uint32_t)__popc(peers));
        base = __shfl_sync(peers, base, leader);
        cellrank[td.first + i] = make_uint2(c, base + __popc(peers & ((1u << lane) - 1u)));
      }
    }
  }
}

// Exclusive scan of the counts into start, in one pass; the counts are zeroed for the next
// substep. Blocks draw tiles of kScanTile cells in order from an atomic counter; a tile's block publishes
// the tile's sum, then looks back over its predecessors, 32 at a time, adding sums until it meets
// one whose whole prefix is known, and publishes its own. A published word is (epoch, kind,
// value) in 64 bits, so words of earlier substeps read as unpublished. Every tile looked at
// was drawn earlier by a block that publishes without waiting, so the wait ends; it has a limit
// all the same (`wait` looks at a group of predecessors), after which the substep is flagged like a
// cell overflow: the block goes on with a prefix of its own making, so that every tile is drawn and its
// counts zeroed, and the later kernels touch nothing. In two launches (tile sums, then tiles) the scan took 8 us of a
// small scene's substep: with the cell offsets 17 us of a 33k-particle substep, 11 in one; at
// 10M particles 20 us either way.
constexpr uint32_t kScanSum = 1u, kScanPrefix = 2u;
__global__ void __launch_bounds__(kScanThreads) k_e_scan(uint32_t* __restrict__ counts, EngineCtl* ctl,
                                                         unsigned long long* state, uint32_t* __restrict__ start,
                                                         uint32_t wait) {
  if (__syncthreads_or((ctl->err & kErrCellCap) != 0u)) return;  // a whole block: another may flag its wait meanwhile
  const uint32_t total = ctl->cells;
  const uint32_t ntiles = (total + kScanTile - 1) / kScanTile;
  const uint32_t tag = ctl->epoch << 2;  // upper half of this substep's words: tag | kind
  constexpr int kPer = kScanTile / kScanThreads;
  __shared__ uint32_t ws[kScanThreads / 32], s_prefix;
  const uint32_t lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  volatile unsigned long long* vs = state;
  if (total == 0) {
    if (blockIdx.x == 0 && threadIdx.x == 0) start[0] = 0u;
    return;
  }
  for (uint32_t tile = next_tile(&ctl->work[kWorkScan]); tile < ntiles; tile = next_tile(&ctl->work[kWorkScan])) {
    const uint32_t i0 = tile * kScanTile + threadIdx.x * kPer;
    uint32_t v[kPer], local = 0;
#pragma unroll
    for (int q = 0; q < kPer; ++q) {
      v[q] = (i0 + q) < total ? counts[i0 + q] : 0u;
      local += v[q];
    }
    uint32_t incl = local;
#pragma unroll
    for (int off = 1; off < 32; off <<= 1) {
      const uint32_t y = __shfl_up_sync(0xffffffffu, incl, off);
      if ((int)lane >= off) incl += y;
    }
    if (lane == 31) ws[w] = incl;
    __syncthreads();
    uint32_t before = 0, sum = 0;
    for (uint32_t k = 0; k < kScanThreads / 32; ++k) {
      if (k < w) before += ws[k];
      sum += ws[k];
    }
    if (w == 0) {
      if (lane == 0)
        vs[tile] = ((unsigned long long)(tag | (tile == 0 ? kScanPrefix : kScanSum)) << 32) | sum;
      uint32_t prefix = 0;
      for (uint32_t at = tile; at > 0;) {  // look back over tiles at - 32 .. at - 1, lane 0 the nearest
        const bool in = lane < at;
        uint32_t kind = in ? 0u : kScanPrefix, val = 0;  // before the first tile: a known prefix of 0
        for (uint32_t tries = 0; !__all_sync(0xffffffffu, kind != 0u); ++tries) {
          if (tries == wait) {
            if (kind == 0u) {
              atomicOr(&ctl->err, kErrCellCap | kErrScanWait);
              kind = kScanPrefix;
            }
          } else if (kind == 0u) {
            const unsigned long long word = vs[at - 1 - lane];
            if ((uint32_t)(word >> 34) == tag >> 2) {
              kind = (uint32_t)(word >> 32) & 3u;
              val = (uint32_t)word;
            }
          }
        }
        const uint32_t known = __ballot_sync(0xffffffffu, kind == kScanPrefix);
        const uint32_t last = known ? (uint32_t)__ffs(known) - 1u : 31u;  // add up to the nearest known prefix
        prefix += __reduce_add_sync(0xffffffffu, lane <= last ? val : 0u);
        at = known ? 0u : at - 32u;
      }
      if (lane == 0) {
        if (tile) vs[tile] = ((unsigned long long)(tag | kScanPrefix) << 32) | (prefix + sum);
        s_prefix = prefix;
      }
    }
    __syncthreads();
    uint32_t run = s_prefix + before + incl - local;
#pragma unroll
    for (int q = 0; q < kPer; ++q) {
      if ((i0 + q) < total) {
        start[i0 + q] = run;
        counts[i0 + q] = 0u;
      }
      run += v[q];
    }
    if (tile == ntiles - 1 && threadIdx.x == kScanThreads - 1) start[total] = run;
  }
}

// Place each slot's (reference index, old slot) and its cell at start[cell] + rank (tiles).
__global__ void k_e_place(const uint2* __restrict__ cellrank, const uint32_t* __restrict__ start,
                          const uint32_t* __restrict__ orig, const TileDev* __restrict__ tiles, uint32_t ntiles,
                          const EngineCtl* __restrict__ ctl, uint2* __restrict__ items, uint32_t* __restrict__ icell) {
  if (ctl->err & kErrCellCap) return;
  for (uint32_t t = blockIdx.x; t < ntiles; t += gridDim.x) {
    const TileDev td = tiles[t];
    for (uint32_t i = threadIdx.x; i < td.count; i += blockDim.x) {
      const uint32_t s = td.first + i;
      const uint2 cr = cellrank[s];
      const uint32_t e = start[cr.x] + cr.y;
      items[e] = make_uint2(orig[s], s);
      icell[e] = cr.x;
    }
  }
}

// Order the placed entries of each cell by reference index (grid.rs:56-62) and gather
// position and velocity into the sorted buffer. A thread per entry, which ranks it against
// its cell's entries (the lanes of a cell read the same ones) while its gathers are in
// flight: the work spreads evenly whatever the cells hold. With a warp per 32 cells a
// pool's few crowded rows of cells were left to a few hundred warps: 1.4M pool at doubled bins 185 -> 54
// us, 10M dam break 501 -> 258, 1M 62 -> 25, 16k 20 -> 7.5.
__global__ void __launch_bounds__(256) k_e_canon(const uint2* __restrict__ items, const uint32_t* __restrict__ icell,
                                                 const uint32_t* __restrict__ start, uint32_t n,
                                                 const EngineCtl* __restrict__ ctl, const float4* __restrict__ pos_in,
                                                 const float4* __restrict__ vel_in, float4* __restrict__ pos_out,
                                                 float4* __restrict__ vel_out, uint32_t* __restrict__ orig,
                                                 uint32_t* __restrict__ slot_of) {
  const uint32_t e = blockIdx.x * blockDim.x + threadIdx.x;
  if (e >= n || (ctl->err & kErrCellCap)) return;
  const uint2 it = items[e];
  const uint32_t c = icell[e];
  const float4 p = pos_in[it.y], v = vel_in[it.y];
  const uint32_t b = start[c], end = start[c + 1];
  uint32_t dst = b;
  uint32_t j = b;
  for (; j + 4 <= end; j += 4) {
    const uint32_t k0 = items[j].x, k1 = items[j + 1].x, k2 = items[j + 2].x, k3 = items[j + 3].x;
    dst += (k0 < it.x ? 1u : 0u) + (k1 < it.x ? 1u : 0u) + (k2 < it.x ? 1u : 0u) + (k3 < it.x ? 1u : 0u);
  }
  for (; j < end; ++j) dst += items[j].x < it.x ? 1u : 0u;
  pos_out[dst] = p;
  vel_out[dst] = v;
  orig[dst] = it.x;
  slot_of[it.x] = dst;
}

// Squared gaps from a particle at p in cell c to the faces of that cell, per axis (0 where p
// lies beyond the face), and the squared reach: a neighbouring cell whose gaps sum above it
// holds no particle with r2 <= h2. The margin bin / 1024 on h is far above the f32 rounding of
// cell faces and bin assignment.
struct CellGaps {
  float xl, xr, yl, yr, zl, zr, reach2;
};

__device__ __forceinline__ CellGaps cell_gaps(const GridBox& g, float px, float py, float pz, uint32_t cx, uint32_t cy,
                                              uint32_t cz, float h) {
  const float lx = g.minx + (float)cx * g.bin, ly = g.miny + (float)cy * g.bin, lz = g.minz + (float)cz * g.bin;
  const float xl = fmaxf(px - lx, 0.0f), xr = fmaxf(lx + g.bin - px, 0.0f);
  const float yl = fmaxf(py - ly, 0.0f), yr = fmaxf(ly + g.bin - py, 0.0f);
  const float zl = fmaxf(pz - lz, 0.0f), zr = fmaxf(lz + g.bin - pz, 0.0f);
  const float reach = h + g.bin * (1.0f / 1024.0f);
  return CellGaps{xl * xl, xr * xr, yl * yl, yr * yr, zl * zl, zr * zr, reach * reach};
}

// Slots [j0, j1) of the row of cells at offset (dy, dz) from cell (cx, cy, cz): those of its up
// to three cells in the grid that lie within reach. Empty when none does. `start` is the
// scene's slice of the cell table.
__device__ __forceinline__ bool cell_row(const GridBox& g, const uint32_t* __restrict__ start, const CellGaps& w,
                                         uint32_t cx, uint32_t cy, uint32_t cz, int dy, int dz, uint32_t& j0,
                                         uint32_t& j1) {
  const int z = (int)cz + dz, y = (int)cy + dy;
  const float gap = (dz < 0 ? w.zl : (dz > 0 ? w.zr : 0.0f)) + (dy < 0 ? w.yl : (dy > 0 ? w.yr : 0.0f));
  if (z < 0 || z >= (int)g.nz || y < 0 || y >= (int)g.ny || gap > w.reach2) return false;
  const uint32_t c = ((uint32_t)z * g.ny + (uint32_t)y) * g.nx + cx;
  j0 = start[c - (cx > 0 && !(gap + w.xl > w.reach2) ? 1u : 0u)];
  j1 = start[c + (cx + 1 < g.nx && !(gap + w.xr > w.reach2) ? 2u : 1u)];
  return j0 < j1;
}

// Walk the 27 cells around position p (cell (cx, cy, cz)) in the reference order (dz outer,
// dy, dx inner; crates/vxl-phys-fluid/src/grid.rs:123-153), calling f(j) for every slot j in
// them, the particle's own among them, except cells farther than h from p (skipping them
// changes neither the set nor the order of accepted neighbours).
template <class F>
__device__ __forceinline__ void walk27(const GridBox& g, const uint32_t* __restrict__ start, float px, float py,
                                       float pz, uint32_t cx, uint32_t cy, uint32_t cz, float h, F&& f) {
  const CellGaps w = cell_gaps(g, px, py, pz, cx, cy, cz, h);
#pragma unroll 1
  for (int dz = -1; dz <= 1; ++dz)
#pragma unroll 1
    for (int dy = -1; dy <= 1; ++dy) {
      uint32_t j, j1;
      if (cell_row(g, start, w, cx, cy, cz, dy, dz, j, j1))
        for (; j < j1; ++j) f(j);
    }
}

// Compact neighbour-list entries, 16 bits. Every neighbour of a particle in cell (cx, cy, cz) lies
// in one of the nine rows (dy, dz) of its 27 cells, each a run of slots from the first slot of cell
// (max(cx - 1, 0), cy + dy, cz + dz); the rows of one z-plane dz follow one another. In most scenes
// an entry is (dz + 1) << 14 | the slot's distance from the first slot of its plane's first row,
// which spans two x rows of the grid: three bases decode it. Where two rows hold more than 14 bits
// (scenes long in x; k_e_groups finds them) it is (dz + 1) << 14 | (dy + 1) << 12 | the distance from the first slot
// of its own row, whose three cells hold 192 particles at rest at 2h bins; its base is loaded from
// the cell table. A neighbour whose distance has more bits makes its list unusable (bit 31 of the
// count): the consumers then walk the cells again. Tick of four substeps, 1.9M particles 1,200
// long at 2h bins: 4.6 ms by rows (force 0.44 ms a substep), 16.4 with a z-plane's entries only (3.37).
// A scene that could do with planes pays for loading the bases: a sixth of the force pass, a twentieth of
// the density pass. By rows for every scene, with the nine bases in shared memory, density is 4% and
// force 3% slower at all sizes, by the L1 cache they take.
constexpr uint32_t kListBad = 0x80000000u;
constexpr uint32_t kListOffBits = 14, kListRowBits = 12;
constexpr uint32_t kListOffMask = (1u << kListOffBits) - 1u, kListRowMask = (1u << kListRowBits) - 1u;

struct ListPlanes {
  uint32_t b0, b1, b2;  // first slot of plane cz - 1 (= b1 at the grid's edge), cz, cz + 1 (~0u if none)
};

__device__ __forceinline__ ListPlanes list_planes(const GridBox& g, const uint32_t* __restrict__ cst, uint32_t cx,
                                                  uint32_t cy, uint32_t cz) {
  const uint32_t xy = (cy > 0 ? cy - 1 : 0) * g.nx + (cx > 0 ? cx - 1 : 0), nxy = g.nx * g.ny;
  ListPlanes lp;
  lp.b1 = cst[cz * nxy + xy];
  lp.b0 = cz > 0 ? cst[(cz - 1) * nxy + xy] : lp.b1;
  lp.b2 = cz + 1 < g.nz ? cst[(cz + 1) * nxy + xy] : 0xffffffffu;
  return lp;
}

__device__ __forceinline__ uint32_t list_decode(const ListPlanes& lp, uint32_t e) {
  const uint32_t pl = e >> kListOffBits;
  return (pl == 0u ? lp.b0 : (pl == 1u ? lp.b1 : lp.b2)) + (e & kListOffMask);
}

// First slots of the rows, 4 (dz + 1) + dy + 1, those that lie in the grid.
struct ListRows {
  const uint32_t* first;  // of row 0
  uint32_t nx, nxy;
  __device__ __forceinline__ uint32_t operator()(uint32_t r) const { return first[(r >> 2) * nxy + (r & 3u) * nx]; }
  __device__ __forceinline__ uint32_t slot(uint32_t e) const { return (*this)(e >> kListRowBits) + (e & kListRowMask); }
};

__device__ __forceinline__ ListRows list_rows(const GridBox& g, const uint32_t* __restrict__ cst, uint32_t cx, uint32_t cy,
                                              uint32_t cz) {
  const int nx = (int)g.nx, nxy = (int)(g.nx * g.ny);
  return ListRows{cst + (((int)cz - 1) * nxy + ((int)cy - 1) * nx + (int)(cx > 0 ? cx - 1 : 0)), g.nx, g.nx * g.ny};
}

// walk27 through the candidate filter (sph_device.cuh): the same rows in the same order and in
// each row the same slots in ascending order, except the slot `self` and those the filter
// shows to lie farther than h. words holds the slots' filter words for the particle's residue
// (padded by 32 past the last slot), tested eight per step; what is left comes out a window at a
// time, push(m, base, dy, dz): bit 31 - t of m (not 0) is slot base + t of row (dy, dz);
// the first is found by one leading-zero count (find-first-set is two instructions of the
// 16-lane unit: 7% of the density pass on the 1M dam break).
// Called by whole warps (`active`: this lane walks); row() follows each row, converged.
// A candidate costs a dp4a and a funnel shift (39 pairs per clock and SM) instead of a 16-byte
// gather and eight float operations; what binds the walk is its work per row, which is why
// the rows are runs of slots and the words are kept per residue: with one frame's words per
// cell, 27 cells and a window each, the pass takes 10% (2h bins) to 45% (h-sized bins) longer. Density
// pass with the cells one by one, every candidate gathered and tested exactly, and now: 0.475 -> 0.254 ms on the
// 1M dam break (h-sized bins), 0.84 -> 0.53 ms on a 1.4M pool and 5.5 -> 3.45 ms on the 10M one (2h bins).
template <class P, class R>
__device__ __forceinline__ void walk27_q(const GridBox& g, const uint32_t* __restrict__ start,
                                         const uint32_t* __restrict__ words, float px, float py, float pz, uint32_t cx,
                                         uint32_t cy, uint32_t cz, float h, uint32_t self, bool active, P&& push,
                                         R&& row) {
  const CellGaps w = cell_gaps(g, px, py, pz, cx, cy, cz, h);
  const int ax = axis_sub(g.minx, px, g.inv, cx) - 32, ay = axis_sub(g.miny, py, g.inv, cy) - 32,
            az = axis_sub(g.minz, pz, g.inv, cz) - 32;
  const uint32_t Mx = (uint32_t)(-ax & 255) | (kSubNorm << 24);
  const int Tx = (int)g.reach_q - ax * ax;
#pragma unroll 1
  for (int dz = -1; dz <= 1; ++dz)
#pragma unroll 1
    for (int dy = -1; dy <= 1; ++dy) {
      uint32_t j0, j1;
      if (active && cell_row(g, start, w, cx, cy, cz, dy, dz, j0, j1)) {
        const int my = (int)kSubUnits * dy - ay, mz = (int)kSubUnits * dz - az;
        const int M = (int)(Mx | ((uint32_t)(my & 255) << 8) | ((uint32_t)(mz & 255) << 16));
        const int over = -((Tx - (my * my + mz * mz)) >> 1) - 1;  // kept: word . M + over < 0
        uint32_t low = ~0u >> (j0 & 3u);
        for (uint32_t base = j0 & ~3u; base < j1; base += 32) {
          // eight words at a time, each sign bit shifted in from below
          uint32_t m = 0;
          const int4* wp = reinterpret_cast<const int4*>(words + base);
          const uint32_t octets = (min(j1 - base, 32u) + 7u) / 8u;
          const int4* const we = wp + 2 * octets;
          do {
            const int4 wa = wp[0], wb = wp[1];
            wp += 2;
            m = __funnelshift_l((uint32_t)__dp4a(wa.x, M, over), m, 1);
            m = __funnelshift_l((uint32_t)__dp4a(wa.y, M, over), m, 1);
            m = __funnelshift_l((uint32_t)__dp4a(wa.z, M, over), m, 1);
            m = __funnelshift_l((uint32_t)__dp4a(wa.w, M, over), m, 1);
            m = __funnelshift_l((uint32_t)__dp4a(wb.x, M, over), m, 1);
            m = __funnelshift_l((uint32_t)__dp4a(wb.y, M, over), m, 1);
            m = __funnelshift_l((uint32_t)__dp4a(wb.z, M, over), m, 1);
            m = __funnelshift_l((uint32_t)__dp4a(wb.w, M, over), m, 1);
          } while (wp != we);
          m = m << (32u - 8u * octets) & low;
          low = ~0u;
          if (j1 - base < 32u) m &= ~(~0u >> (j1 - base));
          if (dz == 0 && dy == 0 && self - base < 32u) m &= ~(0x80000000u >> (self - base));
          if (m) push(m, base, dy, dz);
        }
      }
      row();
    }
}

// ---------------------------------------------------------------- filter words and walk order
//
// k_e_groups writes every slot's candidate-filter words from its sorted position, and for
// scenes whose cell budget doubled the bins to 2h or more the order in which the density
// pass takes the slots: each chunk of a tile (up to kGroupChunk slots) by octant of the
// cell (the half along x, y and z; a stable counting sort into order[]). At 2h bins a
// particle reaches the cells on its own octant's side only, so a warp whose lanes share one
// octant walks one set of cells. Octants follow one another in Gray-code order (0 1 3 2 6
// 7 5 4), so a warp that straddles two octants walks the union of two sets that differ along
// one axis only (12 cells instead of 8; up to 27 for octants apart in all three). A chunk
// holds 8 octant runs, 7 boundaries over kGroupChunk / 32 warps; chunks of 512 slots (tiles
// of 512) let fewer warps straddle, but cost the grouping pass about as much as they save.
//
// It also finds the scenes whose lists go by rows (g.rows, zero before): the first slot of every eighth chunk
// looks up how many slots its own plane's entries span, and a span near the 14 bits marks the scene.
// That is often enough: spans change little from cell to cell, a list that fails all the same is
// walked again, and 512 slots less than the limit leave room for that. A slot of every warp cost 0.05 ms of the
// 10M dam break's substep. (By the fluid's length and rest density a tank with splashes at both ends is full.)
#ifndef VXL_GROUP_CHUNK
#define VXL_GROUP_CHUNK 256
#endif
constexpr uint32_t kGroupChunk = VXL_GROUP_CHUNK;  // slots per chunk = threads per block
static_assert(kGroupChunk % 128 == 0 && kGroupChunk <= 1024, "chunk: 128..1024 slots, whole warps");

__device__ __forceinline__ uint32_t octant_rank(uint32_t oct) { return oct ^ (oct >> 1) ^ (oct >> 2); }

// 1,280 threads per SM (48 registers): with 54 the pass is 10% slower.
__global__ void __launch_bounds__(kGroupChunk, 1280 / kGroupChunk) k_e_groups(
    const float4* __restrict__ pos, const SceneDev* __restrict__ sc, const TileDev* __restrict__ tiles, uint32_t ntiles,
    const EngineCtl* __restrict__ ctl, uint32_t* __restrict__ order, uint32_t* __restrict__ words, uint32_t wstride,
    const uint32_t* __restrict__ start, SceneDev* mark) {
  if (ctl->err & kErrCellCap) return;
  constexpr uint32_t kW = kGroupChunk / 32;  // warps
  constexpr uint32_t kV = 8 * kW / 32;       // (rank, warp) counts per lane of the scan
  __shared__ uint32_t s_cnt[8 * kW];         // [octant rank][warp]: slots per octant in each warp
  const uint32_t lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  const uint32_t lt = (1u << lane) - 1u;
  // the block's chunks one after another, each one's positions loaded while the previous
  // one is sorted
  uint32_t t = blockIdx.x, c1 = 0;
  uint32_t turn = blockIdx.x;  // chunks of this block, counted from its index: the blocks' eighths differ
  TileDev tn = t < ntiles ? tiles[t] : TileDev{};
  float4 pn = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
  if (t < ntiles && threadIdx.x < tn.count) pn = pos[tn.first + threadIdx.x];
  while (t < ntiles) {  // uniform over the block
    const TileDev td = tn;
    const uint32_t c0 = c1;
    const float4 p = pn;
    c1 += kGroupChunk;
    if (c1 >= tn.count) {
      t += gridDim.x;
      c1 = 0;
      if (t < ntiles) tn = tiles[t];
    }
    if (t < ntiles && c1 + threadIdx.x < tn.count) pn = pos[tn.first + c1 + threadIdx.x];
    const GridBox g = sc[td.scene].g;
    const bool half = g.bin >= 2.0f * sc[td.scene].k.h;  // uniform over the block
    const float hb = g.bin * 0.5f;
    const uint32_t i = threadIdx.x;
    const bool valid = i < min(kGroupChunk, td.count - c0);
    ++turn;
    uint32_t oct = 0;
    if (valid) {
      uint32_t cx, cy, cz;
      bin_of(g, p.x, p.y, p.z, cx, cy, cz);
      const int bx = axis_sub(g.minx, p.x, g.inv, cx), by = axis_sub(g.miny, p.y, g.inv, cy) - 32,
                bz = axis_sub(g.minz, p.z, g.inv, cz) - 32;
      uint32_t side = (cx + 1) % 3;  // (cx - p + 1) mod 3, p = 0, 1, 2
#pragma unroll
      for (uint32_t q = 0; q < 3; ++q) {
        words[(size_t)q * wstride + td.first + c0 + i] = sub_word((int)(kSubUnits * side) + bx - 96, by, bz);
        side = side ? side - 1 : 2;
      }
      if (start && i == 0 && (turn & 7u) == 0) {
        const uint32_t* row = start + sc[td.scene].cell_off + cz * g.ny * g.nx;
        const uint32_t first = row[(cy > 0 ? cy - 1 : 0) * g.nx + (cx > 0 ? cx - 1 : 0)];
        const uint32_t end = row[min(cy + 1, g.ny - 1u) * g.nx + min(cx + 1, g.nx - 1u) + 1];
        if (end - first > kListOffMask - 512u) mark[td.scene].g.rows = 1u;  // any number of writers, one value; not read here
      }
      if (half)
        oct = (p.x >= g.minx + (float)cx * g.bin + hb ? 1u : 0u) | (p.y >= g.miny + (float)cy * g.bin + hb ? 2u : 0u) |
              (p.z >= g.minz + (float)cz * g.bin + hb ? 4u : 0u);
    }
    if (!half) continue;
    const uint32_t key = octant_rank(oct);
    uint32_t rank = 0;
#pragma unroll
    for (uint32_t o = 0; o < 8; ++o) {
      const uint32_t b = __ballot_sync(0xffffffffu, valid && key == o);
      if (lane == 0) s_cnt[o * kW + w] = __popc(b);
      if (valid && key == o) rank = __popc(b & lt);
    }
    __syncthreads();
    if (w == 0) {  // exclusive scan of the 8 * kW counts in (rank, warp) order
      uint32_t v[kV], tot = 0;
#pragma unroll
      for (uint32_t k = 0; k < kV; ++k) {
        v[k] = s_cnt[lane * kV + k];
        tot += v[k];
      }
      uint32_t incl = tot;
#pragma unroll
      for (int off = 1; off < 32; off <<= 1) {
        const uint32_t u = __shfl_up_sync(0xffffffffu, incl, off);
        if ((int)lane >= off) incl += u;
      }
      uint32_t ex = incl - tot;
#pragma unroll
      for (uint32_t k = 0; k < kV; ++k) {
        s_cnt[lane * kV + k] = ex;
        ex += v[k];
      }
    }
    __syncthreads();
    if (valid) order[td.first + c0 + s_cnt[key * kW + w] + rank] = td.first + c0 + i;
    __syncthreads();
  }
}

// ---------------------------------------------------------------- provider walls
// ProviderColliders::bounds prefilter of the fluid passes: skip the provider when p lies
// outside its bounds expanded by m (fluid_density.rs:90-101, fluid_boundary.rs:60-71).
__device__ __forceinline__ bool provider_outside(const ProviderDev& pr, float x, float y, float z, float m) {
  return pr.has_bounds && (x < pr.bminx - m || x > pr.bmaxx + m || y < pr.bminy - m || y > pr.bmaxy + m ||
                           z < pr.bminz - m || z > pr.bmaxz + m);
}

// contacts_point(p, probe) of one provider, calling emit(point xyz, outward normal xyz) for
// each contact in the provider's order. FACES: every face with (p[axis] - plane) * sign <=
// 2 probe, at p with that coordinate set to the plane (crates/vxl-phys-fluid/src/tests.rs:
// 81-110). CONVEX: the decisive plane (largest n.p - d) when -(n.p - d) >= -probe, at
// p - n (n.p - d) (crates/vxl-phys-terrain/src/plane_set.rs:60-76, 166-181).
// TABLE: the particle's planes of the table side in use, in their table order.
template <class F>
__device__ __forceinline__ void provider_contacts(const ProviderDev& pr, const WallPlaneDev* __restrict__ pl,
                                                  const ContactTableDev& ct, uint32_t gref, float px, float py,
                                                  float pz, float probe, F&& emit) {
  if (pr.kind == kProviderTable) {
    const uint32_t e = ct.ent ? ct.ent[gref] : 0u;
    if (!e) return;
    for (uint32_t k = ct.start[e - 1], k1 = ct.start[e]; k < k1; ++k) {
      const float4 a = ct.planes[2 * k], n = ct.planes[2 * k + 1];
      emit(a.x, a.y, a.z, n.x, n.y, n.z);
    }
    return;
  }
  if (pr.kind == kProviderFaces) {
    for (uint32_t k = pr.first; k < pr.first + pr.count; ++k) {
      const WallPlaneDev f = pl[k];
      const float comp = f.axis == 0u ? px : (f.axis == 1u ? py : pz);
      const float sdf = (comp - f.d) * f.sign;
      if (sdf > 2.0f * probe) continue;
      float cx = px, cy = py, cz = pz, nx = 0.0f, ny = 0.0f, nz = 0.0f;
      if (f.axis == 0u) {
        cx = f.d;
        nx = f.sign;
      } else if (f.axis == 1u) {
        cy = f.d;
        ny = f.sign;
      } else {
        cz = f.d;
        nz = f.sign;
      }
      emit(cx, cy, cz, nx, ny, nz);
    }
    return;
  }
  if (pr.count == 0u) return;
  float best = -INFINITY;
  uint32_t kb = pr.first;
  for (uint32_t k = pr.first; k < pr.first + pr.count; ++k) {
    const WallPlaneDev q = pl[k];
    const float sd = (q.nx * px + q.ny * py + q.nz * pz) - q.d;
    if (sd > best) {
      best = sd;
      kb = k;
    }
  }
  if (-best < -probe) return;
  const WallPlaneDev q = pl[kb];
  const float t = (q.nx * px + q.ny * py + q.nz * pz) - q.d;
  emit(px - q.nx * t, py - q.ny * t, pz - q.nz * t, q.nx, q.ny, q.nz);
}

// Density (poly6 with self term) + Tait EOS, persistent over tiles, one thread per slot.
// Fluid: rho = mass * (w0 + sum_fluid W) + sum_boundary pmass_j W
// (crates/vxl-phys-fluid/src/fluid_density.rs:24-51); boundary: rho = pmass_i w0 +
// sum_fluid pmass_j W (fluid_density.rs:59-69). Writes (rho, p / rho^2) for the force
// pass (the reference recomputes press/(rho*rho) per pair: same value). Also records, in
// walk order, the slots of the neighbours that contributed (all for fluid, fluid ones for
// boundary particles): nbr[k * stride + s], k < cap, with the full count in nbr_n[s]
// (a count above cap sends the consumers back to walking the cells).
// kWalls: scenes with provider walls add, for a fluid particle, after each neighbour's term
// its mirror ghosts in the particle's provider planes (0 < sdf < h, at most 8; ghost
// g = pj - 2 ((pj - point).n) n with pj = pi - d, W(|pi - g|) if within h), in the
// reference's order (wall_planes_in and the ghost loop, fluid_density.rs:25-47, 76-118).
template <int kBlock, bool kWalls = false>
__global__ void __launch_bounds__(kBlock, VXL_DENSITY_THREADS_PER_SM / kBlock) k_e_density(
    const float4* __restrict__ pos, const uint32_t* __restrict__ start, const SceneDev* __restrict__ sc,
    const TileDev* __restrict__ tiles, uint32_t ntiles, EngineCtl* ctl, const uint32_t* __restrict__ words,
    uint32_t wstride, float2* __restrict__ rc, float* __restrict__ press_out, uint16_t* __restrict__ nbr,
    uint32_t* __restrict__ nbr_n, uint32_t cap, uint32_t stride, const uint32_t* __restrict__ wet,
    const uint32_t* __restrict__ order, const ProviderDev* __restrict__ prov = nullptr,
    const WallPlaneDev* __restrict__ wplanes = nullptr, const uint32_t* __restrict__ orig = nullptr,
    ContactTableDev ctm = ContactTableDev{nullptr, nullptr, nullptr}) {
  if (ctl->err & kErrCellCap) return;
  // Windows of kept candidates (mask, first slot | plane << 30; by rows first slot / 4 << 4 | row),
  // a column per thread: the walk queues them and the warp takes the exact tests from the queue
  // together, so that its lanes, whose windows hold different counts, run one loop of about equal
  // length instead of waiting for one another in every window.
  __shared__ uint2 s_win[kWalkQueue][kBlock];
  // First slots of the particle's list planes (list_planes): read once a window, and three
  // registers less in both loops (7% of the pass on the 1M dam break, 3% on the 10M one).
  __shared__ uint32_t s_plane[3][kBlock];
  for (uint32_t t = first_tile(&ctl->work[kWorkDensity], ntiles); t < ntiles; t = following_tile(&ctl->work[kWorkDensity], ntiles)) {
    const TileDev td = tiles[t];
    const SceneDev& S = sc[td.scene];
    const GridBox g = S.g;
    const SphConst& k = S.k;
    const uint32_t* cst = start + S.cell_off;
    const float h = k.h, h2 = k.h2, k6 = k.k6, w0 = k.w0, mass = k.mass;
    const bool ordered = g.bin >= 2.0f * h;  // uniform over the tile: octant order (k_e_groups)
    const uint32_t epoch = ctl->epoch;
    auto tile = [&](auto by_rows) {
      constexpr bool kRows = decltype(by_rows)::value;
      for (uint32_t i0 = threadIdx.x & ~31u; i0 < td.count; i0 += kBlock) {  // whole warps (lanes past the tile idle)
        const uint32_t i = i0 + (threadIdx.x & 31u);
        const bool valid = i < td.count;
        const uint32_t s = valid ? (ordered ? order[td.first + i] : td.first + i) : td.first;
        const float4 pi = pos[s];
        const bool fluid_i = pi.w > 0.0f;
        uint32_t cx, cy, cz;
        bin_of(g, pi.x, pi.y, pi.z, cx, cy, cz);
        float sum = fluid_i ? w0 : 0.0f;
        float sum_b = 0.0f;
        uint32_t cnt = 0, bad = 0;
        uint16_t* wp = nbr + s;  // next list entry: nbr[cnt * stride + s]
        if constexpr (!kRows) {
          const ListPlanes lp = list_planes(g, cst, cx, cy, cz);
          s_plane[0][threadIdx.x] = lp.b0;
          s_plane[1][threadIdx.x] = lp.b1;
          s_plane[2][threadIdx.x] = lp.b2;
        }
        uint32_t kadd = 0;  // list entry of slot j in the window being taken: j + kadd
        float wpt[kWalls ? 3 * kMaxWallPlanes : 1], wn[kWalls ? 3 * kMaxWallPlanes : 1];
        uint32_t np = 0;
        if (kWalls && fluid_i) {
          for (uint32_t q = S.prov_first; q < S.prov_first + S.prov_count; ++q) {
            const ProviderDev pr = prov[q];
            if (provider_outside(pr, pi.x, pi.y, pi.z, h)) continue;
            provider_contacts(pr, wplanes, ctm, orig ? orig[s] : 0u, pi.x, pi.y, pi.z, h,
                              [&](float cx_, float cy_, float cz_, float nx_, float ny_, float nz_) {
                                const float sdf = (pi.x - cx_) * nx_ + (pi.y - cy_) * ny_ + (pi.z - cz_) * nz_;
                                if (sdf > 0.0f && sdf < h && np < kMaxWallPlanes) {
                                  wpt[3 * np] = cx_;
                                  wpt[3 * np + 1] = cy_;
                                  wpt[3 * np + 2] = cz_;
                                  wn[3 * np] = nx_;
                                  wn[3 * np + 1] = ny_;
                                  wn[3 * np + 2] = nz_;
                                  ++np;
                                }
                              });
          }
        }
        auto visit = [&](uint32_t j, const float4& pj) {  // j != s (the walk leaves it out)
          const float dx = pi.x - pj.x, dy = pi.y - pj.y, dz = pi.z - pj.z;
          const float r2 = dx * dx + dy * dy + dz * dz;
          if (r2 <= h2) {
            const float tt = h2 - r2;
            const float w = k6 * tt * tt * tt;
            bool rec = true;
            if (fluid_i) {
              if (pj.w > 0.0f) sum += w;
              else sum_b += (-pj.w) * w;
              for (uint32_t q = 0; q < np; ++q) {
                const float qx = pi.x - dx, qy = pi.y - dy, qz = pi.z - dz;  // pj = pi - d
                const float dn = (qx - wpt[3 * q]) * wn[3 * q] + (qy - wpt[3 * q + 1]) * wn[3 * q + 1] +
                                 (qz - wpt[3 * q + 2]) * wn[3 * q + 2];
                const float t2 = 2.0f * dn;
                const float ex = pi.x - (qx - wn[3 * q] * t2), ey = pi.y - (qy - wn[3 * q + 1] * t2),
                            ez = pi.z - (qz - wn[3 * q + 2] * t2);
                const float rg2 = ex * ex + ey * ey + ez * ez;
                if (rg2 <= h2) {
                  const float tg = h2 - rg2;
                  sum += k6 * tg * tg * tg;
                }
              }
            } else if (pj.w > 0.0f) {
              sum += pj.w * w;
            } else {
              rec = false;
            }
            if (rec) {
              if (cnt < cap) {
                __stcs(wp, (unsigned short)(j + kadd));  // streaming store: the list is read once, by the force pass
                wp += stride;
              }
              ++cnt;
            }
          }
        };
        // A boundary particle sums fluid neighbours only: with no fluid particle in its 27
        // cells (none marked wet this substep) its walk would accept nothing.
        bool dry = false;
        if (!fluid_i && valid) {
          const uint32_t* wc = wet + S.cell_off;
          dry = true;
          for (int dz = -1; dz <= 1; ++dz) {
            const int z = (int)cz + dz;
            if (z < 0 || z >= (int)g.nz) continue;
            for (int dy = -1; dy <= 1; ++dy) {
              const int y = (int)cy + dy;
              if (y < 0 || y >= (int)g.ny) continue;
              for (int dx = -1; dx <= 1; ++dx) {
                const int x = (int)cx + dx;
                if (x < 0 || x >= (int)g.nx) continue;
                if (wc[((uint32_t)z * g.ny + (uint32_t)y) * g.nx + (uint32_t)x] == epoch) dry = false;
              }
            }
          }
        }
        // Without provider walls: the same test and sums as `visit`.
        auto visit1 = [&](uint32_t j, const float4& pj) {
          const float ddx = pi.x - pj.x, ddy = pi.y - pj.y, ddz = pi.z - pj.z;
          const float r2 = ddx * ddx + ddy * ddy + ddz * ddz;
          if (r2 <= h2) {
            const float tt = h2 - r2;
            const float w = k6 * tt * tt * tt;
            // the neighbour's class selected, not branched on (the same sums: an unselected
            // term is not added)
            const bool fj = pj.w > 0.0f;
            const float tf = fluid_i ? w : pj.w * w;
            const float tb = (-pj.w) * w;
            sum = fj ? sum + tf : sum;
            sum_b = (fluid_i && !fj) ? sum_b + tb : sum_b;
            if (fj || fluid_i) {
              if (cnt < cap) {
                __stcs(wp, (unsigned short)(j + kadd));  // streaming store: read once, by the force pass
                wp += stride;
              }
              ++cnt;
            }
          }
        };
        // Take the queued windows, the next candidate's position loaded while the current one is
        // tested. The list entry of a window's slot j is j + ka; a last slot (kept or not) whose
        // distance has too many bits marks the list unusable.
        uint32_t nq = 0;
        const uint32_t full = kWalkQueue - (ordered ? 6u : 2u);  // a row adds one window or two, at 2h bins four to six
        auto drain = [&]() {
          uint32_t m = 0, base = 0, ka = 0, k = 0;
          auto next = [&]() -> uint32_t {
            if (m == 0u) {
              if (k == nq) return ~0u;
              const uint2 win = s_win[k][threadIdx.x];
              ++k;
              m = win.x;
              if constexpr (kRows) {
                base = win.y >> 2 & ~3u;
                const uint32_t r = win.y & 15u;
                const uint32_t first = list_rows(g, cst, cx, cy, cz)(r);
                bad |= base + 31u - first > kListRowMask ? 1u : 0u;
                ka = (r << kListRowBits) - first;
              } else {
                base = win.y & 0x3fffffffu;
                const uint32_t pl = win.y >> 30;
                ka = (pl << kListOffBits) - s_plane[pl][threadIdx.x];
              }
            }
            const uint32_t t = (uint32_t)__clz((int)m);
            m &= ~(0x80000000u >> t);
            return base + t;
          };
          uint32_t j = next();
          float4 pj = j != ~0u ? pos[j] : pi;
          while (j != ~0u) {
            kadd = ka;
            const uint32_t jn = next();
            const float4 pn = jn != ~0u ? pos[jn] : pj;
            if constexpr (kWalls) visit(j, pj);
            else visit1(j, pj);
            j = jn;
            pj = pn;
          }
          nq = 0;
        };
        walk27_q(
            g, cst, words + (size_t)(cx % 3) * wstride, pi.x, pi.y, pi.z, cx, cy, cz, h, s, valid && !dry,
            [&](uint32_t m, uint32_t base, int dy, int dz) {
              if (nq == kWalkQueue) drain();  // a crowded row
              if constexpr (kRows) {
                s_win[nq++][threadIdx.x] = make_uint2(m, base << 2 | (uint32_t)(4 * dz + dy + 5));  // base is a multiple of 4
              } else {
                const uint32_t pl = (uint32_t)(dz + 1);
                bad |= base + 31u - s_plane[pl][threadIdx.x] > kListOffMask ? 1u : 0u;
                s_win[nq++][threadIdx.x] = make_uint2(m, base | (pl << 30));
              }
            },
            [&]() {
              if (__any_sync(0xffffffffu, nq > full)) drain();
            });
        drain();
        if (!valid) continue;
        nbr_n[s] = cnt | (bad ? kListBad : 0u);
        const float rho = fluid_i ? (mass * sum + sum_b) : ((-pi.w) * w0 + sum);
        const float p = tait(k, rho);
        rc[s] = make_float2(rho, p / (rho * rho));
        if (press_out) press_out[s] = p;
      }
    };
    if (__builtin_expect(g.rows == 0u, 1)) tile(std::false_type{});  // uniform over the block
    else tile(std::true_type{});
  }
}

// Terms of one neighbour pair of the force pass (fluid_force.rs:165-214): the pressure and
// viscosity scales of d = pi - pj, whether the viscosity applies (approaching pairs only), and the XSPH
// scale of vj - vi.
struct PairTerms {
  float q, q2, f;
  bool take;
};

__device__ __forceinline__ PairTerms force_pair(const SphConst& k, bool safe, float dx, float dy, float dz, float r2,
                                                float rho_i, float ci2, const float4& vi, float rho_j, float cj2,
                                                float mj, const float4& vj) {
  const float r = sqrtf(r2);
  const float tt = k.h - r;
  const float sp = k.ks * tt * tt;
  const float coef = mj * sp * (ci2 + cj2);
  const float denom = fmaxf(r, 1e-9f);
  const float vx = vi.x - vj.x, vy = vi.y - vj.y, vz = vi.z - vj.z;
  const float vdn = -(vx * dx + vy * dy + vz * dz);
  PairTerms o;
  o.take = vdn > 0.0f;
  const float vdh = o.take ? vdn * k.h : 0.0f;
  const float dmu = r2 + k.h001, sum = rho_i + rho_j;
  const float t2 = k.h2 - r2;
  const float w = k.k6 * t2 * t2 * t2;
  // the viscosity is computed for every pair and selected, so the warp does not diverge
  // around it (the sums are the same)
  const float ysum = recip_rn(sum), yden = recip_rn(denom);
  const float mu = quot_rn(vdh, dmu, recip_rn(dmu));
  const float c = mj * quot_rn(k.alpha_c * mu, 0.5f * sum, 2.0f * ysum) * sp;
  o.q = quot_rn(coef, denom, yden);
  o.q2 = quot_rn(c, denom, yden);
  o.f = quot_rn(mj * 2.0f, sum, ysum) * w;
  if (!(safe && pair_safe(sum, mj, coef, vdh, c, denom, dmu))) {
    o.q = coef / denom;
    o.q2 = mj * (k.alpha_c * (vdn * k.h / dmu) / (0.5f * sum)) * sp / denom;
    o.f = mj * 2.0f / sum * w;
  }
  return o;
}

// Semi-implicit Euler with the CFL clamp (fluid_step.rs:112-123).
__device__ __forceinline__ void integrate_slot(const SphConst& k, float dt, float vmax, float vmax2, const float4& pi,
                                               const float4& vi, float ax, float ay, float az, float xx, float xy,
                                               float xz, float4& p, float4& v) {
  const float eps = k.eps;
  float ux = vi.x + ax * dt + xx * eps;
  float uy = vi.y + ay * dt + xy * eps;
  float uz = vi.z + az * dt + xz * eps;
  const float s2 = ux * ux + uy * uy + uz * uz;
  if (s2 > vmax2) {
    const float scl = vmax / sqrtf(s2);
    ux = ux * scl;
    uy = uy * scl;
    uz = uz * scl;
  }
  p = make_float4(pi.x + ux * dt, pi.y + uy * dt, pi.z + uz * dt, pi.w);
  v = make_float4(ux, uy, uz, 0.0f);
}

// Force (gravity + spiky pressure + Monaghan viscosity + XSPH, fluid_force.rs:165-214)
// fused with integration (semi-implicit Euler + CFL clamp, fluid_step.rs:112-123) for
// fluid slots; boundary slots are copied unchanged (kinematic within the tick).
// Neighbours come from the density pass's list (same walk order, so the same sums); a
// particle whose list overflowed walks the 27 cells again. Reads the sorted buffer and
// writes the integrated state to (pos_out, vel_out) in the same slot order; accumulates
// each tile's fluid AABB into its scene's accumulator for the next grid box.
template <int kBlock>
__global__ void __launch_bounds__(kBlock, VXL_FORCE_THREADS_PER_SM / kBlock) k_e_force(
    const float4* __restrict__ pos, const float4* __restrict__ vel, const float2* __restrict__ rc,
    const uint32_t* __restrict__ start, const uint16_t* __restrict__ nbr, const uint32_t* __restrict__ nbr_n,
    uint32_t cap, uint32_t stride, SceneDev* __restrict__ sc, const TileDev* __restrict__ tiles, uint32_t ntiles,
    EngineCtl* ctl, float4* __restrict__ pos_out, float4* __restrict__ vel_out, float4* __restrict__ acc_out,
    float4* __restrict__ xsph_out) {
  if (ctl->err & kErrCellCap) return;
  for (uint32_t t = first_tile(&ctl->work[kWorkForce], ntiles); t < ntiles; t = following_tile(&ctl->work[kWorkForce], ntiles)) {
    const TileDev td = tiles[t];
    SceneDev& S = sc[td.scene];
    const SphConst& k = S.k;
    const float dt = S.dt, vmax = S.vmax, vmax2 = S.vmax2;
    const bool safe = scene_safe(k.h, k.alpha_c);
    for (uint32_t b0 = 0; b0 < td.count; b0 += kBlock) {
      const uint32_t i = b0 + threadIdx.x;
      const bool valid = i < td.count;
      float nx = 0, ny = 0, nz = 0;
      bool fluid_i = false;
      if (valid) {
        const uint32_t s = td.first + i;
        const float4 pi = pos[s];
        const float4 vi = vel[s];
        fluid_i = pi.w > 0.0f;
        if (!fluid_i) {
          pos_out[s] = pi;
          vel_out[s] = vi;
        } else {
          const float2 rci = rc[s];
          const float rho_i = rci.x, ci2 = rci.y;
          const float h = k.h, h2 = k.h2;
          float ax = k.gx, ay = k.gy, az = k.gz;
          float xx = 0.0f, xy = 0.0f, xz = 0.0f;
          auto pair = [&](uint32_t j, const float4& pj, float dx, float dy, float dz, float r2) {
            const float2 rcj = rc[j];
            const float4 vj = vel[j];
            const PairTerms o = force_pair(k, safe, dx, dy, dz, r2, rho_i, ci2, vi, rcj.x, rcj.y, fabsf(pj.w), vj);
            ax = ax + dx * o.q;
            ay = ay + dy * o.q;
            az = az + dz * o.q;
            ax = o.take ? ax + dx * o.q2 : ax;
            ay = o.take ? ay + dy * o.q2 : ay;
            az = o.take ? az + dz * o.q2 : az;
            xx = xx + (vj.x - vi.x) * o.f;
            xy = xy + (vj.y - vi.y) * o.f;
            xz = xz + (vj.z - vi.z) * o.f;
          };
          const uint32_t cnt = nbr_n[s];
          const GridBox g = S.g;
          uint32_t cx, cy, cz;
          bin_of(g, pi.x, pi.y, pi.z, cx, cy, cz);
          if (cnt <= cap && !g.rows) {
            // the next list entry is loaded one neighbour ahead, so each iteration waits on
            // one dependent gather (pos/vel/rc of j) instead of two (measured: 6-8% faster),
            // and the one kListPrefetch ahead is fetched into L2 (the list is not L2-resident)
            const ListPlanes lp = list_planes(g, start + S.cell_off, cx, cy, cz);
            const uint16_t* np = nbr + s;
            uint32_t en = cnt ? *np : 0u;
            for (uint32_t q = 0; q < cnt; ++q) {
              const uint32_t j = list_decode(lp, en);
              np += stride;
              if (q + kListPrefetch < cnt)  // the entry kListPrefetch ahead into L2
                asm volatile("prefetch.global.L2 [%0];" ::"l"(np + (size_t)(kListPrefetch - 1) * stride));
              if (q + 1 < cnt) en = *np;
              const float4 pj = pos[j];
              const float dx = pi.x - pj.x, dy = pi.y - pj.y, dz = pi.z - pj.z;
              pair(j, pj, dx, dy, dz, dx * dx + dy * dy + dz * dz);
            }
          } else if (cnt <= cap) {  // by rows: the next neighbour's slot is formed one ahead
            const uint16_t* np = nbr + s;
            // (the cell formed anew per entry: with a ListRows kept in registers the loop above, which most
            // scenes take, is compiled 4% slower, 2.41 vs 2.32 ms on the 10M dam break)
            auto slot = [&](uint32_t e) {
              const uint32_t r = e >> kListRowBits, z = cz + (r >> 2) - 1u, y = cy + (r & 3u) - 1u;
              return start[S.cell_off + (z * g.ny + y) * g.nx + (cx > 0 ? cx - 1 : 0)] + (e & kListRowMask);
            };
            uint32_t jn = cnt ? slot(*np) : s;
            for (uint32_t q = 0; q < cnt; ++q) {
              const uint32_t j = jn;
              np += stride;
              if (q + kListPrefetch < cnt)
                asm volatile("prefetch.global.L2 [%0];" ::"l"(np + (size_t)(kListPrefetch - 1) * stride));
              if (q + 1 < cnt) jn = slot(*np);
              const float4 pj = pos[j];
              const float dx = pi.x - pj.x, dy = pi.y - pj.y, dz = pi.z - pj.z;
              pair(j, pj, dx, dy, dz, dx * dx + dy * dy + dz * dz);
            }
          } else {
            walk27(g, start + S.cell_off, pi.x, pi.y, pi.z, cx, cy, cz, h, [&](uint32_t j) {
              if (j == s) return;
              const float4 pj = pos[j];
              const float dx = pi.x - pj.x, dy = pi.y - pj.y, dz = pi.z - pj.z;
              const float r2 = dx * dx + dy * dy + dz * dz;
              if (r2 <= h2) pair(j, pj, dx, dy, dz, r2);
            });
          }
          if (acc_out) {
            acc_out[s] = make_float4(ax, ay, az, 0.0f);
            xsph_out[s] = make_float4(xx, xy, xz, 0.0f);
          }
          float4 p, v;
          integrate_slot(k, dt, vmax, vmax2, pi, vi, ax, ay, az, xx, xy, xz, p, v);
          nx = p.x;
          ny = p.y;
          nz = p.z;
          pos_out[s] = p;
          vel_out[s] = v;
        }
      }
      // scenes with provider walls take their fluid AABB after the projection pass
      if (S.prov_count == 0u) block_bbox_accumulate(S.fbox, nx, ny, nz, valid && fluid_i);
    }
  }
}

// ---------------------------------------------------------------- small scenes: several lanes per particle
//
// With few particles on the GPU the passes are bound by the length of one particle's chain
// (rows, candidates, pairs one after another, each a gather and a few dozen dependent
// instructions), not by the number of instructions. The team kernels give a particle T lanes
// (8 or 4): they test its candidates and form its pairs' terms T at a time and put the terms in shared memory, from which one lane per component adds them in the walk's order,
// so every sum is the one-lane kernels' sum, bit for bit. Terms that are not taken are
// stored as the neutral element of the addition (-0: x + -0 = x for every x). 2.7k particles,
// per substep: density 34 -> 16 us, force 26 -> 12, boundary forces 16 -> 11; 33k: 36 -> 26, 30 -> 19,
// 26 -> 22. Where the lines lie: team_lanes.
constexpr uint32_t kTeams = 32;     // particles per block
constexpr uint32_t kTeamList = 64;  // candidates held per particle (pitch + T: the teams of a warp on different banks)

template <uint32_t T>
__global__ void __launch_bounds__(kTeams * T) k_e_density_team(
    const float4* __restrict__ pos, const uint32_t* __restrict__ start, const SceneDev* __restrict__ sc,
    const TileDev* __restrict__ tiles, uint32_t subs, const EngineCtl* __restrict__ ctl,
    const uint32_t* __restrict__ words, uint32_t wstride, float2* __restrict__ rc, float* __restrict__ press_out,
    uint16_t* __restrict__ nbr, uint32_t* __restrict__ nbr_n, uint32_t cap, uint32_t stride,
    const uint32_t* __restrict__ wet) {
  if (ctl->err & kErrCellCap) return;
  constexpr uint32_t kMask = (1u << T) - 1u;
  __shared__ uint32_t s_list[kTeams][kTeamList + T];
  __shared__ __align__(16) float s_fluid[kTeams][kTeamList + T], s_bound[kTeams][kTeamList + T];
  const TileDev td = tiles[blockIdx.x / subs];
  const uint32_t first = blockIdx.x % subs * kTeams;  // this block's particles within the tile
  if (first >= td.count) return;
  const uint32_t team = threadIdx.x / T, l = threadIdx.x % T, shift = threadIdx.x & (32u - T);
  const bool valid = first + team < td.count;
  const uint32_t s = td.first + (valid ? first + team : 0u);
  const SceneDev& S = sc[td.scene];
  const GridBox g = S.g;
  const SphConst& k = S.k;
  const uint32_t* cst = start + S.cell_off;
  const float h2 = k.h2, k6 = k.k6;
  const float4 pi = pos[s];
  const bool fluid_i = pi.w > 0.0f;
  uint32_t cx, cy, cz;
  bin_of(g, pi.x, pi.y, pi.z, cx, cy, cz);
  const ListPlanes lp = list_planes(g, cst, cx, cy, cz);
  bool active = valid;
  if (!fluid_i) {  // a boundary particle with no fluid in its 27 cells has nothing to sum
    const uint32_t* wc = wet + S.cell_off;
    const uint32_t epoch = ctl->epoch;
    active = false;
    for (uint32_t r = l; r < 9; r += T) {
      const int z = (int)cz + (int)(r / 3) - 1, y = (int)cy + (int)(r % 3) - 1;
      if (z < 0 || z >= (int)g.nz || y < 0 || y >= (int)g.ny) continue;
      const uint32_t c = ((uint32_t)z * g.ny + (uint32_t)y) * g.nx + cx;
      active |= wc[c] == epoch || (cx > 0 && wc[c - 1] == epoch) || (cx + 1 < g.nx && wc[c + 1] == epoch);
    }
  }
  active = ((__ballot_sync(0xffffffffu, active) >> shift) & kMask) != 0u && valid;
  // the particle's rows, row r in lane r mod T (and the ninth in every lane), all loads in flight together
  const CellGaps w = cell_gaps(g, pi.x, pi.y, pi.z, cx, cy, cz, k.h);
  uint32_t ja[8 / T], jb[8 / T], ja8 = 0, jb8 = 0;
#pragma unroll
  for (uint32_t v = 0; v < 8 / T; ++v) {
    const int r = (int)(l + v * T);
    if (!active || !cell_row(g, cst, w, cx, cy, cz, r % 3 - 1, r / 3 - 1, ja[v], jb[v])) ja[v] = jb[v] = 0;
  }
  if (!active || !cell_row(g, cst, w, cx, cy, cz, 1, 1, ja8, jb8)) ja8 = jb8 = 0;
  const int ax = axis_sub(g.minx, pi.x, g.inv, cx) - 32, ay = axis_sub(g.miny, pi.y, g.inv, cy) - 32,
            az = axis_sub(g.minz, pi.z, g.inv, cz) - 32;
  const uint32_t* wd = words + (size_t)(cx % 3) * wstride;
  const uint32_t below = (1u << l) - 1u;
  float sum = l == 0 && fluid_i ? k.w0 : 0.0f;  // lane 0: fluid terms, lane 1: boundary terms
  uint32_t cnt = 0, bad = 0, n = 0;              // recorded neighbours, candidates held
  auto drain = [&]() {
    __syncwarp();
    const uint32_t most = __reduce_max_sync(0xffffffffu, n);
    for (uint32_t q = l; q - l < most; q += T) {  // whole rounds: the same trips in every lane
      const bool on = q < n;
      const uint32_t j = on ? s_list[team][q] : s;
      const float4 pj = pos[j];
      const float dx = pi.x - pj.x, dy = pi.y - pj.y, dz = pi.z - pj.z;
      const float r2 = dx * dx + dy * dy + dz * dz;
      const float tt = h2 - r2;
      const float wv = k6 * tt * tt * tt;
      const bool near = on && r2 <= h2, fj = pj.w > 0.0f;
      s_fluid[team][q] = near && fj ? (fluid_i ? wv : pj.w * wv) : -0.0f;
      s_bound[team][q] = near && fluid_i && !fj ? (-pj.w) * wv : -0.0f;
      const bool rec = near && (fj || fluid_i);
      const uint32_t taken = (__ballot_sync(0xffffffffu, rec) >> shift) & kMask;
      if (rec) {
        const uint32_t at = cnt + (uint32_t)__popc(taken & below);
        const uint32_t pl = (j >= lp.b1 ? 1u : 0u) + (j >= lp.b2 ? 1u : 0u);
        const uint32_t off = j - (pl == 0u ? lp.b0 : (pl == 1u ? lp.b1 : lp.b2));
        bad |= off > kListOffMask ? 1u : 0u;
        if (at < cap) nbr[(size_t)at * stride + s] = (unsigned short)((pl << kListOffBits) + off);
      }
      cnt += (uint32_t)__popc(taken);
    }
    __syncwarp();
    if (l < 2) {
      const float* t = l == 0 ? s_fluid[team] : s_bound[team];
      for (uint32_t q = 0; q < most; q += 4) {  // entries past n hold the neutral element
        const float4 a = *reinterpret_cast<const float4*>(t + q);
        sum = sum + a.x;
        sum = sum + a.y;
        sum = sum + a.z;
        sum = sum + a.w;
      }
    }
    __syncwarp();
    n = 0;
  };
#pragma unroll 1
  for (uint32_t r = 0; r < 9; ++r) {
    uint32_t j0 = ja8, j1 = jb8;
#pragma unroll
    for (uint32_t v = 0; v < 8 / T; ++v) {
      const uint32_t a0 = __shfl_sync(0xffffffffu, ja[v], (int)(r % T), T);
      const uint32_t a1 = __shfl_sync(0xffffffffu, jb[v], (int)(r % T), T);
      if (r / T == v) {
        j0 = a0;
        j1 = a1;
      }
    }
    const int my = (int)kSubUnits * ((int)(r % 3) - 1) - ay, mz = (int)kSubUnits * ((int)(r / 3) - 1) - az;
    const int M = (int)((uint32_t)(-ax & 255) | ((uint32_t)(my & 255) << 8) | ((uint32_t)(mz & 255) << 16) |
                        (kSubNorm << 24));
    const int over = -(((int)g.reach_q - (ax * ax + my * my + mz * mz)) >> 1) - 1;  // kept: word . M + over < 0
    for (uint32_t base = j0 & ~3u; __any_sync(0xffffffffu, base < j1); base += 4 * T) {
      const uint32_t o = base + 4 * l;  // this lane's four slots
      uint32_t m = 0;
      if (o < j1) {
        const int4 v = *reinterpret_cast<const int4*>(wd + o);
        m = ((uint32_t)__dp4a(v.x, M, over) >> 31) | ((uint32_t)__dp4a(v.y, M, over) >> 31 << 1) |
            ((uint32_t)__dp4a(v.z, M, over) >> 31 << 2) | ((uint32_t)__dp4a(v.w, M, over) >> 31 << 3);
        if (o < j0) m &= 15u << (j0 - o);
        if (j1 - o < 4u) m &= (1u << (j1 - o)) - 1u;
        if (s - o < 4u) m &= ~(1u << (s - o));
      }
      uint32_t incl = (uint32_t)__popc(m);
#pragma unroll
      for (int d = 1; d < (int)T; d <<= 1) {
        const uint32_t y = __shfl_up_sync(0xffffffffu, incl, d, T);
        if ((int)l >= d) incl += y;
      }
      const uint32_t total = __shfl_sync(0xffffffffu, incl, T - 1, T);
      if (__any_sync(0xffffffffu, n + total > kTeamList)) drain();
      uint32_t at = n + incl - (uint32_t)__popc(m);
#pragma unroll
      for (uint32_t t = 0; t < 4; ++t)
        if ((m >> t) & 1u) s_list[team][at++] = o + t;
      n += total;
    }
  }
  drain();
  const float sf = __shfl_sync(0xffffffffu, sum, 0, T), sb = __shfl_sync(0xffffffffu, sum, 1, T);
  const bool any_bad = ((__ballot_sync(0xffffffffu, bad != 0u) >> shift) & kMask) != 0u;
  if (l == 0 && valid) {
    nbr_n[s] = cnt | (any_bad ? kListBad : 0u);
    const float rho = fluid_i ? (k.mass * sf + sb) : ((-pi.w) * k.w0 + sf);
    const float p = tait(k, rho);
    rc[s] = make_float2(rho, p / (rho * rho));
    if (press_out) press_out[s] = p;
  }
}

template <uint32_t T>
__global__ void __launch_bounds__(kTeams * T) k_e_force_team(
    const float4* __restrict__ pos, const float4* __restrict__ vel, const float2* __restrict__ rc,
    const uint32_t* __restrict__ start, const uint16_t* __restrict__ nbr, const uint32_t* __restrict__ nbr_n,
    uint32_t cap, uint32_t stride, SceneDev* __restrict__ sc, const TileDev* __restrict__ tiles, uint32_t subs,
    const EngineCtl* __restrict__ ctl, float4* __restrict__ pos_out, float4* __restrict__ vel_out,
    float4* __restrict__ acc_out, float4* __restrict__ xsph_out) {
  if (ctl->err & kErrCellCap) return;
  // a team's terms: pressure xyz, viscosity xyz, XSPH xyz of T pairs (9 T words a team: the
  // teams of a warp fall on different banks)
  __shared__ __align__(16) float s_term[kTeams][9][T];
  const TileDev td = tiles[blockIdx.x / subs];
  const uint32_t first = blockIdx.x % subs * kTeams;
  if (first >= td.count) return;
  const uint32_t team = threadIdx.x / T, l = threadIdx.x % T;
  const bool valid = first + team < td.count;
  const uint32_t s = td.first + (valid ? first + team : 0u);
  SceneDev& S = sc[td.scene];
  const SphConst& k = S.k;
  const GridBox g = S.g;
  const uint32_t* cst = start + S.cell_off;
  const bool safe = scene_safe(k.h, k.alpha_c);
  const float4 pi = pos[s], vi = vel[s];
  const float2 rci = rc[s];
  const bool fluid_i = valid && pi.w > 0.0f;
  if (valid && !fluid_i && l == 0) {
    pos_out[s] = pi;
    vel_out[s] = vi;
  }
  const uint32_t cnt = fluid_i ? nbr_n[s] : 0u;
  const bool listed = cnt <= cap;
  uint32_t cx, cy, cz;
  bin_of(g, pi.x, pi.y, pi.z, cx, cy, cz);
  // lane a < 3: acceleration and XSPH component a
  float acc = l == 0 ? k.gx : (l == 1 ? k.gy : k.gz), xs = 0.0f;
  auto round = [&](bool on, const float4& pj, const float4& vj, const float2& rcj) {
    const float dx = pi.x - pj.x, dy = pi.y - pj.y, dz = pi.z - pj.z;
    const PairTerms o = force_pair(k, safe, dx, dy, dz, dx * dx + dy * dy + dz * dz, rci.x, rci.y, vi, rcj.x, rcj.y,
                                   fabsf(pj.w), vj);
    const bool visc = on && o.take;
    s_term[team][0][l] = on ? dx * o.q : -0.0f;
    s_term[team][1][l] = on ? dy * o.q : -0.0f;
    s_term[team][2][l] = on ? dz * o.q : -0.0f;
    s_term[team][3][l] = visc ? dx * o.q2 : -0.0f;
    s_term[team][4][l] = visc ? dy * o.q2 : -0.0f;
    s_term[team][5][l] = visc ? dz * o.q2 : -0.0f;
    s_term[team][6][l] = on ? (vj.x - vi.x) * o.f : -0.0f;
    s_term[team][7][l] = on ? (vj.y - vi.y) * o.f : -0.0f;
    s_term[team][8][l] = on ? (vj.z - vi.z) * o.f : -0.0f;
    __syncwarp();
    if (l < 3) {
#pragma unroll
      for (uint32_t q = 0; q < T; q += 4) {
        const float4 a = *reinterpret_cast<const float4*>(&s_term[team][l][q]),
                     b = *reinterpret_cast<const float4*>(&s_term[team][l + 3][q]),
                     c = *reinterpret_cast<const float4*>(&s_term[team][l + 6][q]);
        acc = acc + a.x;
        acc = acc + b.x;
        acc = acc + a.y;
        acc = acc + b.y;
        acc = acc + a.z;
        acc = acc + b.z;
        acc = acc + a.w;
        acc = acc + b.w;
        xs = xs + c.x;
        xs = xs + c.y;
        xs = xs + c.z;
        xs = xs + c.w;
      }
    }
    __syncwarp();
  };
  {  // the recorded list, T neighbours a round, the next round's loaded beside the current one's terms
    const uint32_t n = listed ? cnt : 0u;
    const uint32_t most = __reduce_max_sync(0xffffffffu, n);
    const ListPlanes lp = list_planes(g, cst, cx, cy, cz);
    uint32_t j = l < n ? list_decode(lp, nbr[(size_t)l * stride + s]) : s;
    float4 pj = pos[j], vj = vel[j];
    float2 rcj = rc[j];
    uint32_t jn = l + T < n ? list_decode(lp, nbr[(size_t)(l + T) * stride + s]) : s;
    for (uint32_t q = l; q - l < most; q += T) {
      const float4 pc = pj, vc = vj;
      const float2 rcc = rcj;
      pj = pos[jn];
      vj = vel[jn];
      rcj = rc[jn];
      jn = q + 2 * T < n ? list_decode(lp, nbr[(size_t)(q + 2 * T) * stride + s]) : s;
      round(q < n, pc, vc, rcc);
    }
  }
  if (__any_sync(0xffffffffu, !listed)) {  // longer or unusable lists: the cells again, T slots at a time
    const CellGaps w = cell_gaps(g, pi.x, pi.y, pi.z, cx, cy, cz, k.h);
#pragma unroll 1
    for (int r = 0; r < 9; ++r) {
      uint32_t j0 = 0, j1 = 0;
      if (listed || !cell_row(g, cst, w, cx, cy, cz, r % 3 - 1, r / 3 - 1, j0, j1)) j0 = j1 = 0;
      const uint32_t most = __reduce_max_sync(0xffffffffu, j1 - j0);
      for (uint32_t q = 0; q < most; q += T) {
        const uint32_t j = j0 + q + l;
        const bool in = j < j1 && j != s;
        const float4 pj = in ? pos[j] : pi;
        const float dx = pi.x - pj.x, dy = pi.y - pj.y, dz = pi.z - pj.z;
        const bool on = in && dx * dx + dy * dy + dz * dz <= k.h2;
        if (__any_sync(0xffffffffu, on)) round(on, pj, on ? vel[j] : vi, on ? rc[j] : rci);
      }
    }
  }
  const float ax = __shfl_sync(0xffffffffu, acc, 0, T), ay = __shfl_sync(0xffffffffu, acc, 1, T),
              az = __shfl_sync(0xffffffffu, acc, 2, T), xx = __shfl_sync(0xffffffffu, xs, 0, T),
              xy = __shfl_sync(0xffffffffu, xs, 1, T), xz = __shfl_sync(0xffffffffu, xs, 2, T);
  float4 p = make_float4(0.0f, 0.0f, 0.0f, 0.0f), v;
  if (fluid_i && l == 0) {
    if (acc_out) {
      acc_out[s] = make_float4(ax, ay, az, 0.0f);
      xsph_out[s] = make_float4(xx, xy, xz, 0.0f);
    }
    integrate_slot(k, S.dt, S.vmax, S.vmax2, pi, vi, ax, ay, az, xx, xy, xz, p, v);
    pos_out[s] = p;
    vel_out[s] = v;
  }
  // scenes with provider walls take their fluid AABB after the projection pass
  if (S.prov_count == 0u) block_bbox_accumulate(S.fbox, p.x, p.y, p.z, fluid_i && l == 0);
}

// ---------------------------------------------------------------- provider walls after integration
// boundary_pass (crates/vxl-phys-fluid/src/fluid_boundary.rs:45-101) on the integrated state of
// the scenes with providers, one thread per fluid slot: for each contact of each provider at the
// integrated position pi (probe = skin = 0.15 h) with penetration pen = -(pi - point).n > 0, the
// particle moves by n min(pen + skin, h) and loses its inward normal velocity; the normal sum of a
// pushed particle is kept for the separation, by reference index (pflag, pnsum; w = scene).
// The scene's fluid AABB for the next grid is accumulated here, from the projected positions.
__global__ void k_e_wall_project(float4* __restrict__ pos, float4* __restrict__ vel, SceneDev* __restrict__ sc,
                                 const TileDev* __restrict__ tiles, uint32_t ntiles, const EngineCtl* __restrict__ ctl,
                                 const ProviderDev* __restrict__ prov, const WallPlaneDev* __restrict__ wplanes,
                                 const uint32_t* __restrict__ orig, uint32_t* __restrict__ pflag,
                                 float4* __restrict__ pnsum, ContactTableDev ctp) {
  if (ctl->err & kErrCellCap) return;
  for (uint32_t t = blockIdx.x; t < ntiles; t += gridDim.x) {
    const TileDev td = tiles[t];
    SceneDev& S = sc[td.scene];
    if (S.prov_count == 0u) continue;  // uniform over the block
    const float h = S.k.h, skin = 0.15f * h;  // fluid_access.rs:47
    for (uint32_t b0 = 0; b0 < td.count; b0 += blockDim.x) {
      const uint32_t i = b0 + threadIdx.x;
      const bool valid = i < td.count;
      float x = 0.0f, y = 0.0f, z = 0.0f;
      bool fluid = false;
      if (valid) {
        const uint32_t sl = td.first + i;
        const float4 p = pos[sl];
        fluid = p.w > 0.0f;
        x = p.x;
        y = p.y;
        z = p.z;
        if (fluid) {
          const float4 v = vel[sl];
          float vx = v.x, vy = v.y, vz = v.z, nsx = 0.0f, nsy = 0.0f, nsz = 0.0f;
          bool hit = false;
          for (uint32_t q = S.prov_first; q < S.prov_first + S.prov_count; ++q) {
            const ProviderDev pr = prov[q];
            if (provider_outside(pr, p.x, p.y, p.z, h)) continue;
            provider_contacts(pr, wplanes, ctp, orig[sl], p.x, p.y, p.z, skin,
                              [&](float cx, float cy, float cz, float nx, float ny, float nz) {
                                const float sdf = (p.x - cx) * nx + (p.y - cy) * ny + (p.z - cz) * nz;
                                const float pen = -sdf;
                                if (pen <= 0.0f) return;
                                const float m = fminf(pen + skin, h);
                                x = x + nx * m;
                                y = y + ny * m;
                                z = z + nz * m;
                                nsx = nsx + nx;
                                nsy = nsy + ny;
                                nsz = nsz + nz;
                                hit = true;
                                const float vn = vx * nx + vy * ny + vz * nz;
                                if (vn < 0.0f) {
                                  vx = vx - nx * vn;
                                  vy = vy - ny * vn;
                                  vz = vz - nz * vn;
                                }
                              });
          }
          pos[sl] = make_float4(x, y, z, p.w);
          vel[sl] = make_float4(vx, vy, vz, v.w);
          const uint32_t o = orig[sl];
          pflag[o] = hit ? 1u : 0u;
          if (hit) pnsum[o] = make_float4(nsx, nsy, nsz, __uint_as_float(td.scene));
        }
      }
      block_bbox_accumulate(S.fbox, x, y, z, valid && fluid);
    }
  }
}

// The pushed particles in ascending reference index (plist), in two passes over chunks of
// kPushedChunk indices: per-chunk counts, then each chunk's entries at its offset. The last
// chunk stores the total in ctl->work[kWorkPushed].
__device__ __forceinline__ uint32_t block_sum(uint32_t v, uint32_t* sh) {
  for (int off = 16; off > 0; off >>= 1) v += __shfl_xor_sync(0xffffffffu, v, off);
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5, nw = (blockDim.x + 31) >> 5;
  __syncthreads();
  if (lane == 0) sh[wid] = v;
  __syncthreads();
  uint32_t tot = 0;
  for (int w = 0; w < nw; ++w) tot += sh[w];
  return tot;
}

__global__ void k_e_pushed_count(const uint32_t* __restrict__ pflag, uint32_t n, const EngineCtl* __restrict__ ctl,
                                 uint32_t* __restrict__ blk) {
  if (ctl->err & kErrCellCap) return;
  __shared__ uint32_t sh[32];
  const uint32_t base = blockIdx.x * kPushedChunk;
  uint32_t c = 0;
  for (uint32_t k = threadIdx.x; k < kPushedChunk; k += blockDim.x) {
    const uint32_t o = base + k;
    if (o < n && pflag[o]) ++c;
  }
  c = block_sum(c, sh);
  if (threadIdx.x == 0) blk[blockIdx.x] = c;
}

__global__ void k_e_pushed_emit(const uint32_t* __restrict__ pflag, uint32_t n, const uint32_t* __restrict__ blk,
                                EngineCtl* __restrict__ ctl, uint32_t* __restrict__ plist,
                                const float4* __restrict__ pos, const float4* __restrict__ pnsum,
                                const uint32_t* __restrict__ slot_of, float4* __restrict__ ppos) {
  if (ctl->err & kErrCellCap) return;
  __shared__ uint32_t sh[32], wtot[32];
  uint32_t part = 0;
  for (uint32_t k = threadIdx.x; k < blockIdx.x; k += blockDim.x) part += blk[k];
  uint32_t off = block_sum(part, sh);
  const uint32_t base = blockIdx.x * kPushedChunk;
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5, nw = (blockDim.x + 31) >> 5;
  for (uint32_t r0 = 0; r0 < kPushedChunk; r0 += blockDim.x) {
    const uint32_t o = base + r0 + threadIdx.x;
    const bool f = o < n && pflag[o] != 0u;
    const uint32_t bal = __ballot_sync(0xffffffffu, f);
    __syncthreads();
    if (lane == 0) wtot[wid] = __popc(bal);
    __syncthreads();
    uint32_t before = 0, total = 0;
    for (int w = 0; w < nw; ++w) {
      if (w < wid) before += wtot[w];
      total += wtot[w];
    }
    if (f) {
      const uint32_t at = off + before + __popc(bal & ((1u << lane) - 1u));
      plist[at] = o;
      const float4 p = pos[slot_of[o]];
      ppos[at] = make_float4(p.x, p.y, p.z, pnsum[o].w);
    }
    off += total;
  }
  if (blockIdx.x == gridDim.x - 1 && threadIdx.x == 0) ctl->work[kWorkPushed] = off;
}

// First position in the ascending list a[0, n) whose value is >= key.
__device__ __forceinline__ uint32_t lower_bound_u32(const uint32_t* __restrict__ a, uint32_t n, uint32_t key) {
  uint32_t lo = 0, hi = n;
  while (lo < hi) {
    const uint32_t mid = (lo + hi) >> 1;
    if (a[mid] < key) lo = mid + 1;
    else hi = mid;
  }
  return lo;
}

// separate_coincident (fluid_boundary.rs:103-128) moves a pushed particle only if some
// earlier pushed particle of its scene lies closer than r_min = 0.2 h. If no pair is that
// close at the projected positions, nothing moves (by induction over the sequential loop):
// this pass decides whether the sequential pass must run. The pairs of a scene go over the GPU
// as pairs of tiles of kCheckTile pushed particles (gathered with their scene by k_e_pushed_emit):
// a thread holds one particle of the later tile (a row) and tests it against an earlier tile in
// shared memory. blockIdx.y takes rows, up and down in turn so that long and short ones mix;
// blockIdx.x takes tiles back from the row's own and stops at the first that ends in an earlier
// scene: the list ascends by scene, so a batch of scenes costs the sum of their pairs, not the
// pairs of all (wall kernels of a substep of 64 scenes with 2,048 pushed particles each: 91 us,
// 1.33 ms with all pairs; of one scene 65 us either way). 4 or 16 columns are within 10% of 8. One
// thread per particle and gathers through plist and slot_of was P dependent loads long (0.15 ms
// of a 65k-particle tank's 0.31 ms substep).
constexpr uint32_t kCheckTile = 128;
constexpr uint32_t kCheckRows = 148, kCheckCols = 8;  // grid: (cols, rows), so that a few rows still spread over the SMs
__global__ void __launch_bounds__(kCheckTile) k_e_separate_check(const SceneDev* __restrict__ sc,
                                                                 const uint32_t* __restrict__ plist,
                                                                 const float4* __restrict__ pnsum,
                                                                 const float4* __restrict__ ppos,
                                                                 EngineCtl* __restrict__ ctl) {
  if (ctl->err & kErrCellCap) return;
  __shared__ float4 tile[kCheckTile];
  __shared__ uint32_t found;
  const uint32_t P = ctl->work[kWorkPushed], nt = (P + kCheckTile - 1) / kCheckTile;
  for (uint32_t turn = 0; turn * kCheckRows < nt; ++turn) {
    const uint32_t row = turn * kCheckRows + ((turn & 1u) ? kCheckRows - 1u - blockIdx.y : blockIdx.y);
    if (row >= nt || blockIdx.x > row) continue;
    auto load = [&](uint32_t back) {
      const uint32_t b = (row - back) * kCheckTile + threadIdx.x;
      return b < P ? ppos[b] : make_float4(0.0f, 0.0f, 0.0f, 0.0f);
    };
    float4 next = load(blockIdx.x);  // in flight beside the row's own loads, the following ones beside the tests
    const uint32_t a = row * kCheckTile + threadIdx.x;
    const uint32_t earliest = __float_as_uint(ppos[row * kCheckTile].w);  // scene of the row's first particle
    bool moves = false;
    float4 pa = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
    float rm2 = 0.0f;
    if (a < P) {
      const float4 na = pnsum[plist[a]];
      moves = !(sqrtf(na.x * na.x + na.y * na.y + na.z * na.z) <= 1e-9f);
      pa = ppos[a];
      const float r_min = 0.2f * sc[__float_as_uint(pa.w)].k.h;
      rm2 = r_min * r_min;
    }
    for (uint32_t back = blockIdx.x; back <= row; back += kCheckCols) {
      __syncthreads();
      tile[threadIdx.x] = next;
      if (threadIdx.x == 0) found = *(volatile const uint32_t*)&ctl->work[kWorkTrigger];
      __syncthreads();
      if (found) return;
      if (back && __float_as_uint(tile[kCheckTile - 1].w) < earliest) break;  // (a tile before the row's own is full)
      if (back + kCheckCols <= row) next = load(back + kCheckCols);
      if (moves) {
        const uint32_t q = __float_as_uint(pa.w);
        bool close = false;
        const uint32_t n = back ? kCheckTile : threadIdx.x;  // of its own tile, the earlier ones
#pragma unroll 8
        for (uint32_t t = 0; t < n; ++t) {
          const float4 pb = tile[t];
          const float dx = pa.x - pb.x, dy = pa.y - pb.y, dz = pa.z - pb.z;
          close |= dx * dx + dy * dy + dz * dz < rm2 && __float_as_uint(pb.w) == q;
        }
        if (close) atomicOr(&ctl->work[kWorkTrigger], 1u);
      }
    }
  }
}

// The sequential separation itself, one block, only when the check found a close pair: for
// each pushed particle a in order (normal sum n_a, |n_a| > 1e-9), for each earlier pushed b of
// its scene in order, with the current (already separated) positions: if |pa - pb|^2 < r_min^2,
// pa += n_a / |n_a| (r_min - |pa - pb|). The block tests a window of b in parallel against the
// current pa and applies the first hit, then resumes after it. If anything moved, the AABB
// accumulators of the scenes with providers are reset for k_e_wall_rebox.
__global__ void __launch_bounds__(1024) k_e_separate(float4* __restrict__ pos, SceneDev* __restrict__ sc,
                                                     uint32_t nscenes, const uint32_t* __restrict__ plist,
                                                     const float4* __restrict__ pnsum,
                                                     const uint32_t* __restrict__ slot_of, EngineCtl* __restrict__ ctl) {
  if ((ctl->err & kErrCellCap) || !ctl->work[kWorkTrigger]) return;
  const uint32_t P = ctl->work[kWorkPushed];
  __shared__ float4 pa_s;
  __shared__ uint32_t first;
  bool moved = false;  // thread 0
  for (uint32_t a = 0; a < P; ++a) {
    const uint32_t oa = plist[a];
    const float4 na = pnsum[oa];
    const float nl = sqrtf(na.x * na.x + na.y * na.y + na.z * na.z);
    if (nl <= 1e-9f) continue;  // uniform over the block
    const uint32_t q = __float_as_uint(na.w);
    const float r_min = 0.2f * sc[q].k.h;
    const float rm2 = r_min * r_min;
    const float inv = 1.0f / nl;
    const float dirx = na.x * inv, diry = na.y * inv, dirz = na.z * inv;
    const uint32_t sa = slot_of[oa];
    if (threadIdx.x == 0) pa_s = pos[sa];
    __syncthreads();
    uint32_t b0 = lower_bound_u32(plist, a, sc[q].base);  // the scene's first pushed particle
    while (b0 < a) {
      if (threadIdx.x == 0) first = 0xffffffffu;
      __syncthreads();
      const float4 cur = pa_s;
      const uint32_t b = b0 + threadIdx.x;
      if (b < a) {
        const float4 pb = pos[slot_of[plist[b]]];
        const float dx = cur.x - pb.x, dy = cur.y - pb.y, dz = cur.z - pb.z;
        if (dx * dx + dy * dy + dz * dz < rm2) atomicMin(&first, b);
      }
      __syncthreads();
      const uint32_t f = first;
      if (f == 0xffffffffu) {
        b0 += blockDim.x;
      } else {
        if (threadIdx.x == 0) {
          const float4 pb = pos[slot_of[plist[f]]];
          const float dx = cur.x - pb.x, dy = cur.y - pb.y, dz = cur.z - pb.z;
          const float r = sqrtf(dx * dx + dy * dy + dz * dz);
          const float m = r_min - r;
          pa_s = make_float4(cur.x + dirx * m, cur.y + diry * m, cur.z + dirz * m, cur.w);
          moved = true;
        }
        b0 = f + 1;
      }
      __syncthreads();
    }
    if (threadIdx.x == 0) pos[sa] = pa_s;
    __syncthreads();
  }
  if (threadIdx.x == 0 && moved) {
    ctl->work[kWorkMoved] = 1u;
    for (uint32_t q = 0; q < nscenes; ++q)
      if (sc[q].prov_count) {
        for (int c = 0; c < 3; ++c) {
          sc[q].fbox[c] = 0xffffffffu;
          sc[q].fbox[3 + c] = 0u;
        }
      }
  }
}

// After a separation that moved particles: the fluid AABB of the scenes with providers again,
// from the final positions.
__global__ void k_e_wall_rebox(const float4* __restrict__ pos, SceneDev* __restrict__ sc,
                               const TileDev* __restrict__ tiles, uint32_t ntiles, const EngineCtl* __restrict__ ctl) {
  if ((ctl->err & kErrCellCap) || !ctl->work[kWorkMoved]) return;
  for (uint32_t t = blockIdx.x; t < ntiles; t += gridDim.x) {
    const TileDev td = tiles[t];
    SceneDev& S = sc[td.scene];
    if (S.prov_count == 0u) continue;
    for (uint32_t b0 = 0; b0 < td.count; b0 += blockDim.x) {
      const uint32_t i = b0 + threadIdx.x;
      const bool valid = i < td.count;
      float4 p = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
      if (valid) p = pos[td.first + i];
      block_bbox_accumulate(S.fbox, p.x, p.y, p.z, valid && p.w > 0.0f);
    }
  }
}

// Pair term of the boundary reaction for fluid i on boundary j, from i's side of the
// reference loop (crates/vxl-phys-fluid/src/fluid_force.rs:182-207): returns
// q = m_i (coef + cv) / denom, with d = p_i - p_j; the caller applies bforce -= d * q.
__device__ __forceinline__ float bforce_pair(const SphConst& k, bool safe, float r2, float dx, float dy, float dz,
                                             float rho_i, float ci2, float mi, float4 vi, float rho_j, float cj2,
                                             float mj, float4 vj) {
  const float r = sqrtf(r2);
  const float t = k.h - r;
  const float sp = k.ks * t * t;
  const float coef = mj * sp * (ci2 + cj2);
  const float denom = fmaxf(r, 1e-9f);
  const float vx = vi.x - vj.x, vy = vi.y - vj.y, vz = vi.z - vj.z;
  const float vdn = -(vx * dx + vy * dy + vz * dz);
  const float vdh = vdn > 0.0f ? vdn * k.h : 0.0f;
  const float dmu = r2 + k.h001, sum = rho_i + rho_j;
  const float mu = quot_rn(vdh, dmu, recip_rn(dmu));
  const float cv = mj * quot_rn(k.alpha_c * mu, 0.5f * sum, 2.0f * recip_rn(sum)) * sp;
  const float num = mi * (coef + (vdn > 0.0f ? cv : 0.0f));
  if (safe && pair_safe(sum, mj, num, vdh, cv, denom, dmu)) return quot_rn(num, denom, recip_rn(denom));
  float ce = 0.0f;
  if (vdn > 0.0f) ce = mj * (k.alpha_c * (vdn * k.h / dmu) / (0.5f * sum)) * sp;
  return mi * (coef + ce) / denom;
}

// Whether a boundary particle's terms count in its span's sums: without force it adds only
// zeros, unless its arm is not a small finite number.
__device__ __forceinline__ bool bforce_wet(float bx, float by, float bz, const float4& p) {
  const bool arm = fabsf(p.x) < kReactArm && fabsf(p.y) < kReactArm && fabsf(p.z) < kReactArm;  // false for NaN
  return !(bx == 0.0f && by == 0.0f && bz == 0.0f) || !arm;
}

// Reaction on each boundary particle j: the reference accumulates bforce[j] -= F_ij over
// fluid i in ascending reference index (the outer loop of force_pass_serial). Here the
// boundary particle takes its fluid neighbours (recorded by the density pass, or found by
// walking the 27 cells when that list overflowed), orders them by reference index and sums
// in that order, so the result is the same sum. Runs over boundary tiles in reference
// order (every lane a boundary particle; slot_of finds its sorted slot); output by global
// reference index.
__global__ void __launch_bounds__(128) k_e_bforce(
    const float4* __restrict__ pos, const float4* __restrict__ vel, const float2* __restrict__ rc,
    const uint32_t* __restrict__ start, const uint32_t* __restrict__ orig, const uint16_t* __restrict__ nbr,
    const uint32_t* __restrict__ nbr_n, uint32_t cap, uint32_t stride, const SceneDev* __restrict__ sc,
    const uint32_t* __restrict__ slot_of, const TileDev* __restrict__ btiles, uint32_t ntiles, EngineCtl* ctl,
    float4* __restrict__ bforce, uint32_t* __restrict__ bwet) {
  if (ctl->err & kErrCellCap) return;
  for (uint32_t t = first_tile(&ctl->work[kWorkBforce], ntiles); t < ntiles; t = following_tile(&ctl->work[kWorkBforce], ntiles)) {
    const TileDev td = btiles[t];
    const SceneDev& S = sc[td.scene];
    const SphConst& k = S.k;
    const GridBox g = S.g;
    const uint32_t* cst = start + S.cell_off;
    const float h2 = k.h2;
    const bool safe = scene_safe(k.h, k.alpha_c);
    // a tile is at most one particle per thread (kBoundaryTile)
    const uint32_t i = threadIdx.x;
    bool wet = false;
    if (i < td.count) {
      const uint32_t o = td.first + i;  // global reference index of a boundary particle
      const uint32_t s = slot_of[o];
      const float4 pj = pos[s];
      const float4 vj = vel[s];
      const float2 rcj = rc[s];
      const float mj = -pj.w;
      uint32_t cx, cy, cz;
      bin_of(g, pj.x, pj.y, pj.z, cx, cy, cz);
      // insertion-sort buffer: only entries [0, n) are ever read (not zero-filled: that
      // cost 64 local stores per particle)
      uint32_t key[kBGatherCap];
      uint32_t slot[kBGatherCap];
      int n = 0;
      bool overflow = false;
      auto insert = [&](uint32_t ii) {
        if (n < kBGatherCap) {
          const uint32_t o = orig[ii];
          int q = n++;
          for (; q > 0; --q) {
            const uint32_t kq = key[q - 1];
            if (kq <= o) break;
            key[q] = kq;
            slot[q] = slot[q - 1];
          }
          key[q] = o;
          slot[q] = ii;
        } else {
          overflow = true;
        }
      };
      const uint32_t cnt = nbr_n[s];
      if (cnt <= cap && g.rows) {
        const ListRows rows = list_rows(g, cst, cx, cy, cz);
        for (uint32_t q = 0; q < cnt; ++q) insert(rows.slot(nbr[(size_t)q * stride + s]));
      } else if (cnt <= cap) {
        const ListPlanes lp = list_planes(g, cst, cx, cy, cz);
        for (uint32_t q = 0; q < cnt; ++q) insert(list_decode(lp, nbr[(size_t)q * stride + s]));
      } else {
        walk27(g, cst, pj.x, pj.y, pj.z, cx, cy, cz, k.h, [&](uint32_t ii) {
          const float4 p = pos[ii];
          if (!(p.w > 0.0f)) return;
          const float dx = p.x - pj.x, dy = p.y - pj.y, dz = p.z - pj.z;
          if (!(dx * dx + dy * dy + dz * dz <= h2)) return;
          insert(ii);
        });
      }
      float bx = 0.0f, by = 0.0f, bz = 0.0f;
      auto apply = [&](uint32_t ii) {
        const float4 p = pos[ii];
        const float dx = p.x - pj.x, dy = p.y - pj.y, dz = p.z - pj.z;
        const float r2 = dx * dx + dy * dy + dz * dz;
        const float2 rci = rc[ii];
        const float q = bforce_pair(k, safe, r2, dx, dy, dz, rci.x, rci.y, p.w, vel[ii], rcj.x, rcj.y, mj, vj);
        bx = bx - dx * q;
        by = by - dy * q;
        bz = bz - dz * q;
      };
      if (!overflow) {
        for (int q = 0; q < n; ++q) apply(slot[q]);
      } else {
        // Slow path: fluid neighbours in ascending reference index by repeated minimum
        // search (O(neighbours x candidates)); counted in ctl->slow_gathers.
        atomicAdd(&ctl->slow_gathers, 1u);
        uint32_t last = 0;
        bool first = true;
        for (;;) {
          uint32_t best = 0xffffffffu, best_slot = 0;
          walk27(g, cst, pj.x, pj.y, pj.z, cx, cy, cz, k.h, [&](uint32_t ii) {
            const float4 p = pos[ii];
            if (!(p.w > 0.0f)) return;
            const uint32_t o = orig[ii];
            if (!first && o <= last) return;
            if (o >= best) return;
            const float dx = p.x - pj.x, dy = p.y - pj.y, dz = p.z - pj.z;
            if (!(dx * dx + dy * dy + dz * dz <= h2)) return;
            best = o;
            best_slot = ii;
          });
          if (best == 0xffffffffu) break;
          apply(best_slot);
          last = best;
          first = false;
        }
      }
      bforce[o] = make_float4(bx, by, bz, 0.0f);
      wet = bforce_wet(bx, by, bz, pj);
    }
    const uint32_t wm = __ballot_sync(0xffffffffu, wet);
    if ((threadIdx.x & 31) == 0) bwet[4 * t + (threadIdx.x >> 5)] = wm;
  }
}

// The same with T lanes per boundary particle (see the small-scene kernels above): the
// neighbours' reference indices are ranked against one another in shared memory instead of
// inserted one by one, and the pairs' terms formed T at a time and subtracted in order by a lane per
// component (x - 0 = x: the neutral term). A block is 32 consecutive boundary particles, a
// word of the wet mask. kRows: some scene's list entries may go by rows (seven registers more, 1.2 us of a
// small handle's 55 us substep).
template <uint32_t T, bool kRows>
__global__ void __launch_bounds__(kTeams * T) k_e_bforce_team(
    const float4* __restrict__ pos, const float4* __restrict__ vel, const float2* __restrict__ rc,
    const uint32_t* __restrict__ start, const uint32_t* __restrict__ orig, const uint16_t* __restrict__ nbr,
    const uint32_t* __restrict__ nbr_n, uint32_t cap, uint32_t stride, const SceneDev* __restrict__ sc,
    const uint32_t* __restrict__ slot_of, const TileDev* __restrict__ btiles, EngineCtl* ctl,
    float4* __restrict__ bforce, uint32_t* __restrict__ bwet) {
  if (ctl->err & kErrCellCap) return;
  static_assert(kBGatherCap <= (int)kTeamList, "a team's list holds the gathered neighbours");
  constexpr uint32_t kMask = (1u << T) - 1u;
  __shared__ uint32_t s_key[kTeams][kTeamList + T], s_slot[kTeams][kTeamList + T], s_sorted[kTeams][kTeamList + T];
  __shared__ __align__(16) float s_term[kTeams][3][T];
  __shared__ uint32_t s_wet;
  const uint32_t t = blockIdx.x / 4, first = blockIdx.x % 4 * kTeams;  // a boundary tile is 128 particles
  const TileDev td = btiles[t];
  const uint32_t team = threadIdx.x / T, l = threadIdx.x % T, shift = threadIdx.x & (32u - T);
  if (threadIdx.x == 0) s_wet = 0u;
  __syncthreads();
  const bool valid = first + team < td.count;
  const SceneDev& S = sc[td.scene];
  const SphConst& k = S.k;
  const GridBox g = S.g;
  const uint32_t* cst = start + S.cell_off;
  const bool safe = scene_safe(k.h, k.alpha_c);
  const uint32_t o = td.first + (valid ? first + team : 0u);
  const uint32_t s = slot_of[o];
  const float4 pj = pos[s], vj = vel[s];
  const float2 rcj = rc[s];
  const float mj = -pj.w;
  uint32_t cx, cy, cz;
  bin_of(g, pj.x, pj.y, pj.z, cx, cy, cz);
  const uint32_t cnt = valid ? nbr_n[s] : 0u;
  const bool listed = cnt <= cap;
  uint32_t n = listed ? cnt : 0u;
  bool overflow = false;
  if (listed) {
    auto gather = [&](auto&& slot) {
      for (uint32_t q = l; q < n; q += T) {
        const uint32_t ii = slot(nbr[(size_t)q * stride + s]);
        s_slot[team][q] = ii;
        s_key[team][q] = orig[ii];
      }
    };
    if (kRows && g.rows) {
      const ListRows rows = list_rows(g, cst, cx, cy, cz);
      gather([&](uint32_t e) { return rows.slot(e); });
    } else {
      const ListPlanes lp = list_planes(g, cst, cx, cy, cz);
      gather([&](uint32_t e) { return list_decode(lp, e); });
    }
  }
  const CellGaps w = cell_gaps(g, pj.x, pj.y, pj.z, cx, cy, cz, k.h);
  if (__any_sync(0xffffffffu, !listed)) {  // longer or unusable lists: the cells again, T slots at a time
#pragma unroll 1
    for (int r = 0; r < 9; ++r) {
      uint32_t j0 = 0, j1 = 0;
      if (listed || !cell_row(g, cst, w, cx, cy, cz, r % 3 - 1, r / 3 - 1, j0, j1)) j0 = j1 = 0;
      const uint32_t most = __reduce_max_sync(0xffffffffu, j1 - j0);
      for (uint32_t q = 0; q < most; q += T) {
        const uint32_t ii = j0 + q + l;
        bool on = false;
        if (ii < j1) {
          const float4 p = pos[ii];
          const float dx = p.x - pj.x, dy = p.y - pj.y, dz = p.z - pj.z;
          on = p.w > 0.0f && dx * dx + dy * dy + dz * dz <= k.h2;
        }
        const uint32_t taken = (__ballot_sync(0xffffffffu, on) >> shift) & kMask;
        const uint32_t at = n + (uint32_t)__popc(taken & ((1u << l) - 1u));
        if (on && at < (uint32_t)kBGatherCap) {
          s_slot[team][at] = ii;
          s_key[team][at] = orig[ii];
        }
        n += (uint32_t)__popc(taken);
      }
    }
    overflow = n > (uint32_t)kBGatherCap;
    if (overflow) n = 0;
  }
  __syncwarp();
  for (uint32_t q = l; q < n; q += T) {
    const uint32_t key = s_key[team][q];
    uint32_t rank = 0;
    for (uint32_t m = 0; m < n; ++m) rank += s_key[team][m] < key ? 1u : 0u;
    s_sorted[team][rank] = s_slot[team][q];
  }
  __syncwarp();
  float b = 0.0f;  // lane a < 3: component a
  auto pair_q = [&](uint32_t ii, float& dx, float& dy, float& dz) {
    const float4 p = pos[ii];
    dx = p.x - pj.x;
    dy = p.y - pj.y;
    dz = p.z - pj.z;
    const float2 rci = rc[ii];
    return bforce_pair(k, safe, dx * dx + dy * dy + dz * dz, dx, dy, dz, rci.x, rci.y, p.w, vel[ii], rcj.x, rcj.y, mj, vj);
  };
  const uint32_t most = __reduce_max_sync(0xffffffffu, n);
  for (uint32_t q = l; q - l < most; q += T) {
    float dx = 0.0f, dy = 0.0f, dz = 0.0f, qq = 0.0f;
    if (q < n) qq = pair_q(s_sorted[team][q], dx, dy, dz);
    s_term[team][0][l] = q < n ? dx * qq : 0.0f;
    s_term[team][1][l] = q < n ? dy * qq : 0.0f;
    s_term[team][2][l] = q < n ? dz * qq : 0.0f;
    __syncwarp();
    if (l < 3) {
#pragma unroll
      for (uint32_t c = 0; c < T; c += 4) {
        const float4 x = *reinterpret_cast<const float4*>(&s_term[team][l][c]);
        b = b - x.x;
        b = b - x.y;
        b = b - x.z;
        b = b - x.w;
      }
    }
    __syncwarp();
  }
  if (__any_sync(0xffffffffu, overflow)) {
    // more fluid neighbours than the list holds: in ascending reference index by repeated
    // minimum search, the team's lanes over the candidates; counted in ctl->slow_gathers
    if (overflow && l == 0) atomicAdd(&ctl->slow_gathers, 1u);
    uint32_t last = 0;
    bool begun = false, more = overflow;
    while (__any_sync(0xffffffffu, more)) {
      unsigned long long best = ~0ull;  // reference index, slot
      if (more) {
#pragma unroll 1
        for (int r = 0; r < 9; ++r) {
          uint32_t j0, j1;
          if (!cell_row(g, cst, w, cx, cy, cz, r % 3 - 1, r / 3 - 1, j0, j1)) continue;
          for (uint32_t ii = j0 + l; ii < j1; ii += T) {
            const float4 p = pos[ii];
            if (!(p.w > 0.0f)) continue;
            const uint32_t oi = orig[ii];
            if (begun && oi <= last) continue;
            const float dx = p.x - pj.x, dy = p.y - pj.y, dz = p.z - pj.z;
            if (!(dx * dx + dy * dy + dz * dz <= k.h2)) continue;
            best = min(best, ((unsigned long long)oi << 32) | ii);
          }
        }
      }
#pragma unroll
      for (int d = 1; d < (int)T; d <<= 1) best = min(best, __shfl_xor_sync(0xffffffffu, best, d, T));
      more = more && best != ~0ull;
      if (more) {
        float dx, dy, dz;
        const float qq = pair_q((uint32_t)best, dx, dy, dz);
        b = b - (l == 0 ? dx : (l == 1 ? dy : dz)) * qq;
        last = (uint32_t)(best >> 32);
        begun = true;
      }
    }
  }
  const float bx = __shfl_sync(0xffffffffu, b, 0, T), by = __shfl_sync(0xffffffffu, b, 1, T),
              bz = __shfl_sync(0xffffffffu, b, 2, T);
  if (valid && l == 0) {
    bforce[o] = make_float4(bx, by, bz, 0.0f);
    if (bforce_wet(bx, by, bz, pj)) atomicOr(&s_wet, 1u << team);
  }
  __syncthreads();
  if (threadIdx.x == 0) bwet[blockIdx.x] = s_wet;
}

// Per-span force and torque about the body origin (fluid_boundary.rs:10-28), added to
// the tick accumulator in index order (the reference's sum, bit for bit): six independent
// sequential sums, so what bounds a span is the number of its terms times the latency of one
// addition. Particles that no fluid touches (the outer faces of walls, dry floors: most of a
// tank) have zero terms, and adding a zero of either sign changes no sum that began at +0;
// k_e_bforce marks the others in a bit mask over each scene's boundary particles (bwet), and
// the kernels compact the marked ones of a span, in order, before they load and add them.
// Spans of at most kReactExactSpan particles (bodies) take a warp each: lane a (a < 6) adds
// component a of 32 terms while the next 32 are being loaded. Larger spans (tank walls) take
// a block each, whose last warp adds one batch while the others stage the next. Span ranges
// are global reference indices. The walls of a 1.4M-particle pool (floor of 245k particles,
// 27k wet): 1.76 -> 0.30 ms per substep, which had been longer than the rest of the substep;
// bodies and walls of a 33k-particle tank 87 -> 34 us.

// Torque origin of a span: its coupled rigid body's position, or the origin it was given.
__device__ __forceinline__ void span_origin(const SpanDev& sp, const RigidBodyDev* __restrict__ rb, float& ox,
                                            float& oy, float& oz) {
  if (sp.rigid != ~0u && rb) {
    ox = rb[sp.rigid].px;
    oy = rb[sp.rigid].py;
    oz = rb[sp.rigid].pz;
  } else {
    ox = sp.ox;
    oy = sp.oy;
    oz = sp.oz;
  }
}

// The wet particles of 32 consecutive boundary particles, those of word w of the span's scene
// (its particles bfirst + 32 (w - bword) ..), cut to the span. With an arm that is not a small
// finite number every term counts (0 * inf is not 0).
__device__ __forceinline__ uint32_t span_word(const SpanDev& sp, bool all, const uint32_t* __restrict__ bwet, uint32_t rel) {
  const uint32_t lo = sp.start - sp.bfirst, hi = sp.end - sp.bfirst;  // rel: first particle of the word, < hi
  uint32_t m = all ? 0xffffffffu : bwet[sp.bword + (rel >> 5)];
  if (rel < lo) m &= ~0u << (lo - rel);
  if (hi - rel < 32u) m &= (1u << (hi - rel)) - 1u;
  return m;
}

__device__ __forceinline__ bool span_arm_unsafe(const SpanDev& sp) {
  return !(fabsf(sp.ox) < kReactArm && fabsf(sp.oy) < kReactArm && fabsf(sp.oz) < kReactArm);
}

// Force and torque terms of one particle.
__device__ __forceinline__ void span_terms(const float4& fk, const float4& p, const SpanDev& sp, float* t, uint32_t stride) {
  const float rx = p.x - sp.ox, ry = p.y - sp.oy, rz = p.z - sp.oz;
  t[0] = fk.x;
  t[stride] = fk.y;
  t[2 * stride] = fk.z;
  t[3 * stride] = ry * fk.z - rz * fk.y;
  t[4 * stride] = rz * fk.x - rx * fk.z;
  t[5 * stride] = rx * fk.y - ry * fk.x;
}

__global__ void __launch_bounds__(kReactThreads) k_react_long(const float4* __restrict__ bforce,
                                                              const float4* __restrict__ bpos,
                                                              const uint32_t* __restrict__ bwet,
                                                              const SpanDev* __restrict__ spans,
                                                              const LongSpan* __restrict__ longs,
                                                              const RigidBodyDev* __restrict__ rb,
                                                              const EngineCtl* __restrict__ ctl,
                                                              float* __restrict__ breact) {
  if (ctl->err & kErrCellCap) return;
  __shared__ __align__(16) float terms[2][6][kReactBatch];
  __shared__ uint16_t s_idx[32 * kReactWords];  // wet particles of the words at hand, from the first word's first
  __shared__ uint32_t s_warp[kReactWords / 32];
  constexpr uint32_t kSum = kReactThreads / 32 - 1;  // the summing warp
  const uint32_t lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  const uint32_t span = longs[blockIdx.x].span;
  SpanDev sp = spans[span];
  span_origin(sp, rb, sp.ox, sp.oy, sp.oz);
  const bool all = span_arm_unsafe(sp);
  const uint32_t hi = sp.end - sp.bfirst;
  float f = 0.0f;  // lane a < 6 of the summing warp: component a (force xyz, torque xyz)
  for (uint32_t rel0 = (sp.start - sp.bfirst) & ~31u; rel0 < hi; rel0 += 32 * kReactWords) {
    // compact the wet particles of the next kReactWords words
    uint32_t m = 0, incl = 0;
    if (threadIdx.x < kReactWords) {
      const uint32_t rel = rel0 + 32 * threadIdx.x;
      if (rel < hi) m = span_word(sp, all, bwet, rel);
      incl = (uint32_t)__popc(m);
#pragma unroll
      for (int off = 1; off < 32; off <<= 1) {
        const uint32_t y = __shfl_up_sync(0xffffffffu, incl, off);
        if ((int)lane >= off) incl += y;
      }
      if (lane == 31) s_warp[w] = incl;
    }
    __syncthreads();
    uint32_t total = 0, at = incl - (uint32_t)__popc(m);
    for (uint32_t k = 0; k < kReactWords / 32; ++k) {
      if (k < w) at += s_warp[k];
      total += s_warp[k];
    }
    while (m) {
      s_idx[at++] = (uint16_t)(32 * threadIdx.x + (uint32_t)(__ffs(m) - 1));
      m &= m - 1u;
    }
    __syncthreads();
    const uint32_t first = sp.bfirst + rel0;
    for (uint32_t b0 = 0, buf = 0; b0 < total + kReactBatch; b0 += kReactBatch, buf ^= 1u) {
      if (w != kSum) {
        if (b0 + threadIdx.x < total) {
          const uint32_t kk = first + s_idx[b0 + threadIdx.x];
          span_terms(bforce[kk], bpos[kk], sp, &terms[buf][0][threadIdx.x], kReactBatch);
        }
      } else if (b0 && lane < 6) {  // the batch staged in the previous step
        const uint32_t nb = min(kReactBatch, total - (b0 - kReactBatch));
        const float* tt = terms[buf ^ 1u][lane];
        uint32_t t = 0;
        for (; t + 16 <= nb; t += 16) {  // 16 terms loaded together, then added one by one
          float v[16];
#pragma unroll
          for (int i = 0; i < 16; i += 4) {
            const float4 q = *reinterpret_cast<const float4*>(tt + t + i);
            v[i] = q.x;
            v[i + 1] = q.y;
            v[i + 2] = q.z;
            v[i + 3] = q.w;
          }
#pragma unroll
          for (int i = 0; i < 16; ++i) f = f + v[i];
        }
        for (; t < nb; ++t) f = f + tt[t];
      }
      __syncthreads();
    }
  }
  if (w == kSum && lane < 6) breact[6 * span + lane] = breact[6 * span + lane] + f;
}

// Spans of at most kReactExactSpan particles, one warp each (the others: k_react_long).
__global__ void k_react_spans(const float4* __restrict__ bforce, const float4* __restrict__ bpos,
                              const uint32_t* __restrict__ bwet, const SpanDev* __restrict__ spans,
                              const RigidBodyDev* __restrict__ rb, const EngineCtl* __restrict__ ctl,
                              float* __restrict__ breact, uint32_t nspans) {
  if (ctl->err & kErrCellCap) return;
  __shared__ float terms[kReactSpanWarps][6][33];
  __shared__ uint16_t s_idx[kReactSpanWarps][1024];
  const uint32_t w = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const uint32_t q = blockIdx.x * kReactSpanWarps + w;
  if (q >= nspans) return;  // uniform over the warp
  SpanDev sp = spans[q];
  span_origin(sp, rb, sp.ox, sp.oy, sp.oz);
  if (sp.end - sp.start > kReactExactSpan) return;  // uniform over the warp
  const bool all = span_arm_unsafe(sp);
  const uint32_t hi = sp.end - sp.bfirst;
  float f = 0.0f;  // lane a < 6: component a (force xyz, torque xyz)
  for (uint32_t rel0 = (sp.start - sp.bfirst) & ~31u; rel0 < hi; rel0 += 1024) {
    uint32_t m = rel0 + 32 * lane < hi ? span_word(sp, all, bwet, rel0 + 32 * lane) : 0u;
    uint32_t incl = (uint32_t)__popc(m);
#pragma unroll
    for (int off = 1; off < 32; off <<= 1) {
      const uint32_t y = __shfl_up_sync(0xffffffffu, incl, off);
      if ((int)lane >= off) incl += y;
    }
    uint32_t at = incl - (uint32_t)__popc(m);
    const uint32_t total = __shfl_sync(0xffffffffu, incl, 31);
    while (m) {
      s_idx[w][at++] = (uint16_t)(32 * lane + (uint32_t)(__ffs(m) - 1));
      m &= m - 1u;
    }
    __syncwarp();
    const uint32_t first = sp.bfirst + rel0;
    float4 fk = make_float4(0.0f, 0.0f, 0.0f, 0.0f), p = fk;
    if (lane < total) {
      fk = bforce[first + s_idx[w][lane]];
      p = bpos[first + s_idx[w][lane]];
    }
    for (uint32_t b0 = 0; b0 < total; b0 += 32) {
      if (b0 + lane < total) span_terms(fk, p, sp, &terms[w][0][lane], 33);
      __syncwarp();
      if (b0 + 32 + lane < total) {  // the next batch's loads run beside the sums
        fk = bforce[first + s_idx[w][b0 + 32 + lane]];
        p = bpos[first + s_idx[w][b0 + 32 + lane]];
      }
      if (lane < 6) {
        const uint32_t nb = min(32u, total - b0);
        if (nb == 32u) {  // the batch's terms loaded together, then added one by one
          float v[32];
#pragma unroll
          for (int i = 0; i < 32; ++i) v[i] = terms[w][lane][i];
#pragma unroll
          for (int i = 0; i < 32; ++i) f = f + v[i];
        } else {
          for (uint32_t t = 0; t < nb; ++t) f = f + terms[w][lane][t];
        }
      }
      __syncwarp();
    }
  }
  if (lane < 6) breact[6 * q + lane] = breact[6 * q + lane] + f;
}

// Rigid substeps of the coupling loop without contacts, one thread per body, f32 in the
// reference's order: per substep the gravity field adds g * (1 / inv_mass)
// (crates/vxl-phys-field/src/lib.rs:22-31) and the fluid reaction pass adds the tick-averaged
// reaction of the body's span (crates/vxl-phys/src/world_step.rs:235-255); then
// Integrator::integrate_velocities with gravity ZERO (v += (0 + F inv_m) dt; w += I_world^-1 tau
// dt with I_world^-1 = R diag(I^-1) R^T, crates/vxl-phys-core/src/body.rs:172-176; whole-vector
// speed clamps) and integrate_positions (x += v dt; q = normalize(q + dt/2 (0, w) q),
// crates/vxl-phys-core/src/math.rs:216-252), crates/vxl-phys-integrate/src/lib.rs:18-60.
// `with_reaction` is 0 before the first fluid tick of the loop (no reaction yet).
__device__ __forceinline__ void rigid_world_inv_inertia(const RigidBodyDev& b, float lx, float ly, float lz,
                                                        float& ox, float& oy, float& oz) {
  const float xx = b.qx * b.qx, yy = b.qy * b.qy, zz = b.qz * b.qz;
  const float xy = b.qx * b.qy, xz = b.qx * b.qz, yz = b.qy * b.qz;
  const float wx = b.qw * b.qx, wy = b.qw * b.qy, wz = b.qw * b.qz;
  const float m00 = 1.0f - 2.0f * (yy + zz), m01 = 2.0f * (xy - wz), m02 = 2.0f * (xz + wy);
  const float m10 = 2.0f * (xy + wz), m11 = 1.0f - 2.0f * (xx + zz), m12 = 2.0f * (yz - wx);
  const float m20 = 2.0f * (xz - wy), m21 = 2.0f * (yz + wx), m22 = 1.0f - 2.0f * (xx + yy);
  const float tx = m00 * lx + m10 * ly + m20 * lz;
  const float ty = m01 * lx + m11 * ly + m21 * lz;
  const float tz = m02 * lx + m12 * ly + m22 * lz;
  const float vx = tx * b.iix, vy = ty * b.iiy, vz = tz * b.iiz;
  ox = m00 * vx + m01 * vy + m02 * vz;
  oy = m10 * vx + m11 * vy + m12 * vz;
  oz = m20 * vx + m21 * vy + m22 * vz;
}

__global__ void k_rigid_step(RigidBodyDev* __restrict__ bodies, uint32_t n, const float* __restrict__ breact,
                             int with_reaction, float gx, float gy, float gz, float dt, uint32_t substeps,
                             float max_linear, float max_angular) {
  const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  RigidBodyDev b = bodies[i];
  if (!b.dynamic) return;
  float rf[6] = {0, 0, 0, 0, 0, 0};
  if (with_reaction && b.span != ~0u)
    for (int a = 0; a < 6; ++a) rf[a] = breact[6 * b.span + a];
  const float hd = 0.5f * dt;
  for (uint32_t k = 0; k < substeps; ++k) {
    const float mass = 1.0f / b.inv_mass;
    float fx = 0.0f + gx * mass, fy = 0.0f + gy * mass, fz = 0.0f + gz * mass;
    fx = fx + rf[0];
    fy = fy + rf[1];
    fz = fz + rf[2];
    const float tqx = 0.0f + rf[3], tqy = 0.0f + rf[4], tqz = 0.0f + rf[5];
    b.vx = b.vx + (0.0f + fx * b.inv_mass) * dt;
    b.vy = b.vy + (0.0f + fy * b.inv_mass) * dt;
    b.vz = b.vz + (0.0f + fz * b.inv_mass) * dt;
    float ax, ay, az;
    rigid_world_inv_inertia(b, tqx, tqy, tqz, ax, ay, az);
    b.wx = b.wx + ax * dt;
    b.wy = b.wy + ay * dt;
    b.wz = b.wz + az * dt;
    const float sp = sqrtf(b.vx * b.vx + b.vy * b.vy + b.vz * b.vz);
    if (sp > max_linear) {
      const float s = max_linear / sp;
      b.vx = b.vx * s;
      b.vy = b.vy * s;
      b.vz = b.vz * s;
    }
    const float ws = sqrtf(b.wx * b.wx + b.wy * b.wy + b.wz * b.wz);
    if (ws > max_angular) {
      const float s = max_angular / ws;
      b.wx = b.wx * s;
      b.wy = b.wy * s;
      b.wz = b.wz * s;
    }
    b.px = b.px + b.vx * dt;
    b.py = b.py + b.vy * dt;
    b.pz = b.pz + b.vz * dt;
    // dq = (w, 0) * q (Hamilton), then q + dq dt/2, normalized
    const float dqx = 0.0f * b.qx + b.wx * b.qw + b.wy * b.qz - b.wz * b.qy;
    const float dqy = 0.0f * b.qy - b.wx * b.qz + b.wy * b.qw + b.wz * b.qx;
    const float dqz = 0.0f * b.qz + b.wx * b.qy - b.wy * b.qx + b.wz * b.qw;
    const float dqw = 0.0f * b.qw - b.wx * b.qx - b.wy * b.qy - b.wz * b.qz;
    const float nx = b.qx + dqx * hd, ny = b.qy + dqy * hd, nz = b.qz + dqz * hd, nw = b.qw + dqw * hd;
    const float len2 = nx * nx + ny * ny + nz * nz + nw * nw;
    if (len2 > 1e-16f) {
      const float inv = 1.0f / sqrtf(len2);
      b.qx = nx * inv;
      b.qy = ny * inv;
      b.qz = nz * inv;
      b.qw = nw * inv;
    } else {
      b.qx = 0.0f;
      b.qy = 0.0f;
      b.qz = 0.0f;
      b.qw = 1.0f;
    }
  }
  bodies[i] = b;
}

// Tick average (fluid_step.rs:84-88): e *= 1 / substeps.
__global__ void k_scale(float* __restrict__ breact, uint32_t n, float inv) {
  const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) breact[i] = breact[i] * inv;
}

// ---------------------------------------------------------------- export kernels

// One scene's state in its reference order (scene-local index).
__global__ void k_e_read_scene(const float4* __restrict__ pos, const float4* __restrict__ vel,
                               const uint32_t* __restrict__ orig, float* __restrict__ pout, float* __restrict__ vout,
                               uint32_t base, uint32_t n) {
  const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const uint32_t s = base + i;
  const uint32_t o = orig[s] - base;
  if (pout) {
    const float4 p = pos[s];
    pout[3 * o] = p.x;
    pout[3 * o + 1] = p.y;
    pout[3 * o + 2] = p.z;
  }
  if (vout) {
    const float4 v = vel[s];
    vout[3 * o] = v.x;
    vout[3 * o + 1] = v.y;
    vout[3 * o + 2] = v.z;
  }
}

__global__ void k_e_read_fields(const float2* __restrict__ rc, const float* __restrict__ press,
                                const float4* __restrict__ acc, const float4* __restrict__ xsph,
                                const uint32_t* __restrict__ orig, float* __restrict__ dout, float* __restrict__ pout,
                                float* __restrict__ aout, float* __restrict__ xout, uint32_t base, uint32_t n, uint32_t nf) {
  const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const uint32_t s = base + i;
  const uint32_t o = orig[s] - base;
  if (dout) dout[o] = rc[s].x;
  if (pout) pout[o] = press[s];
  if (aout) {
    const float4 a = o < nf ? acc[s] : make_float4(0.0f, 0.0f, 0.0f, 0.0f);  // the force pass records fluid slots only
    aout[3 * o] = a.x;
    aout[3 * o + 1] = a.y;
    aout[3 * o + 2] = a.z;
  }
  if (xout) {
    const float4 x = o < nf ? xsph[s] : make_float4(0.0f, 0.0f, 0.0f, 0.0f);
    xout[3 * o] = x.x;
    xout[3 * o + 1] = x.y;
    xout[3 * o + 2] = x.z;
  }
}

// One scene's table in the reference's cell order (x outermost, z innermost), from the
// engine's (z outermost): per reference cell its count, then, with the exclusive scan of the
// counts in ref_start, each cell's particles (scene-local index) and each particle's cell.
__device__ __forceinline__ uint32_t engine_cell(const GridBox& g, uint32_t c) {
  const uint32_t z = c % g.nz, xy = c / g.nz, y = xy % g.ny, x = xy / g.ny;
  return (z * g.ny + y) * g.nx + x;
}

constexpr uint32_t kExportTile = 512;
constexpr int kExportThreads = 256;

// Reference cells of one tile: their counts, and the tile's sum.
__global__ void __launch_bounds__(kExportThreads) k_e_export_counts(const uint32_t* __restrict__ start,
                                                                    const SceneDev* __restrict__ sc, uint32_t scene,
                                                                    uint32_t* __restrict__ ref_start,
                                                                    uint32_t* __restrict__ sums) {
  __shared__ uint32_t sh[32];
  const SceneDev& S = sc[scene];
  uint32_t sum = 0;
  for (uint32_t k = threadIdx.x; k < kExportTile; k += kExportThreads) {
    const uint32_t c = blockIdx.x * kExportTile + k;
    if (c > S.cells) break;
    const uint32_t e = S.cell_off + (c < S.cells ? engine_cell(S.g, c) : 0u);
    const uint32_t n = c < S.cells ? start[e + 1] - start[e] : 0u;
    ref_start[c] = n;
    sum += n;
  }
  sum = block_sum(sum, sh);
  if (threadIdx.x == 0) sums[blockIdx.x] = sum;
}

// The tile's exclusive scan in place, from the sums of the tiles before it, and its cells'
// particles. Tiles of 512 spread a small scene's cells over the SMs: 33k particles in 9k cells, a
// call of 0.117 ms (0.14 with tiles of 2,048); 1.1M cells 0.60 ms, 1.86 when one block scanned them all.
__global__ void __launch_bounds__(kExportThreads) k_e_export_table(const uint32_t* __restrict__ start,
                                                                   const uint32_t* __restrict__ orig,
                                                                   const SceneDev* __restrict__ sc, uint32_t scene,
                                                                   uint32_t* __restrict__ ref_start,
                                                                   const uint32_t* __restrict__ sums,
                                                                   uint32_t* __restrict__ items, uint32_t* __restrict__ bins) {
  constexpr uint32_t kPer = kExportTile / kExportThreads;
  __shared__ uint32_t sh[32], s_at[kExportTile];
  const SceneDev& S = sc[scene];
  uint32_t part = 0;
  for (uint32_t k = threadIdx.x; k < blockIdx.x; k += kExportThreads) part += sums[k];
  uint32_t run = block_sum(part, sh);
  const uint32_t c0 = blockIdx.x * kExportTile, last = min(kExportTile, S.cells + 1u - c0);  // cells of the tile, one past the last too
  for (uint32_t k = threadIdx.x; k < last; k += kExportThreads) s_at[k] = ref_start[c0 + k];
  __syncthreads();
  uint32_t v[kPer], local = 0;
#pragma unroll
  for (uint32_t q = 0; q < kPer; ++q) {
    const uint32_t k = threadIdx.x * kPer + q;
    v[q] = k < last ? s_at[k] : 0u;
    local += v[q];
  }
  const uint32_t lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  uint32_t incl = local;
#pragma unroll
  for (int off = 1; off < 32; off <<= 1) {
    const uint32_t y = __shfl_up_sync(0xffffffffu, incl, off);
    if ((int)lane >= off) incl += y;
  }
  if (lane == 31) sh[w] = incl;
  __syncthreads();
  for (uint32_t k = 0; k < w; ++k) run += sh[k];
  run += incl - local;
#pragma unroll
  for (uint32_t q = 0; q < kPer; ++q) {
    const uint32_t k = threadIdx.x * kPer + q;
    if (k < last) s_at[k] = run;
    run += v[q];
  }
  __syncthreads();
  for (uint32_t k = threadIdx.x; k < last; k += kExportThreads) {
    const uint32_t c = c0 + k;
    uint32_t at = s_at[k];
    ref_start[c] = at;
    if (c == S.cells || (!items && !bins)) continue;
    const uint32_t e = S.cell_off + engine_cell(S.g, c);
    for (uint32_t q = start[e]; q < start[e + 1]; ++q) {
      const uint32_t o = orig[q] - S.base;
      if (items) items[at] = o;
      if (bins) bins[o] = c;
      ++at;
    }
  }
}

// Contact table entries by global reference index: ent[ids[e]] = e + 1 (ent zeroed before).
__global__ void k_e_ctab_scatter(const uint32_t* __restrict__ ids, uint32_t n, uint32_t* __restrict__ ent) {
  const uint32_t e = blockIdx.x * blockDim.x + threadIdx.x;
  if (e < n) ent[ids[e]] = e + 1u;
}

// Neighbour-list export of one scene (last substep): the list count of each slot in the
// scene's reference order.
__global__ void k_e_export_nbr_counts(const uint32_t* __restrict__ nbr_n, const uint32_t* __restrict__ orig,
                                      uint32_t base, uint32_t n, uint32_t* __restrict__ out) {
  const uint32_t t = blockIdx.x * blockDim.x + threadIdx.x;
  if (t < n) out[orig[base + t] - base] = nbr_n[base + t] & ~kListBad;
}

// The entries of each slot's list, in its walk order, as scene-local reference indices,
// at offsets[reference index]: the recorded list, or for a list longer than the cap the
// same neighbours walked again from the sorted positions and cell table of that substep
// (the walk the force pass and the boundary gather fall back to).
__global__ void k_e_export_nbr_entries(const float4* __restrict__ pos, const uint32_t* __restrict__ start,
                                       const SceneDev* __restrict__ sc, uint32_t q, const uint32_t* __restrict__ orig,
                                       const uint16_t* __restrict__ nbr, const uint32_t* __restrict__ nbr_n,
                                       uint32_t cap, uint32_t stride, const unsigned long long* __restrict__ offsets,
                                       uint32_t* __restrict__ out) {
  const SceneDev& S = sc[q];
  const uint32_t t = blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= S.count) return;
  const uint32_t s = S.base + t;
  const uint32_t base = S.base;
  unsigned long long o = offsets[orig[s] - base];
  const uint32_t c = nbr_n[s];
  const GridBox g = S.g;
  const float4 pi = pos[s];
  uint32_t cx, cy, cz;
  bin_of(g, pi.x, pi.y, pi.z, cx, cy, cz);
  if (c <= cap) {
    const uint32_t* cst = start + S.cell_off;
    const ListPlanes lp = list_planes(g, cst, cx, cy, cz);
    const ListRows rows = list_rows(g, cst, cx, cy, cz);
    for (uint32_t k = 0; k < c; ++k) {
      const uint32_t e = nbr[(size_t)k * stride + s];
      out[o + k] = orig[g.rows ? rows.slot(e) : list_decode(lp, e)] - base;
    }
    return;
  }
  const bool fluid_i = pi.w > 0.0f;
  const float h2 = S.k.h2;
  walk27(g, start + S.cell_off, pi.x, pi.y, pi.z, cx, cy, cz, S.k.h, [&](uint32_t j) {
    if (j == s) return;
    const float4 pj = pos[j];
    const float dx = pi.x - pj.x, dy = pi.y - pj.y, dz = pi.z - pj.z;
    const float r2 = dx * dx + dy * dy + dz * dz;
    if (r2 <= h2 && (fluid_i || pj.w > 0.0f)) out[o++] = orig[j] - base;
  });
}

}  // namespace
}  // namespace vxl
