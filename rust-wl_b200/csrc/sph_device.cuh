// Device-side building blocks of the WCSPH step for sm_100a.
//
// Arithmetic contract: this file is compiled with -fmad=false (no FMA contraction),
// IEEE division and square root (-prec-div=true -prec-sqrt=true) and no flush to zero,
// and every expression keeps the reference's evaluation order, so results are
// bit-identical to the reference's Rust f32 CPU path
// (crates/vxl-phys-fluid/src/fluid_density.rs, fluid_force.rs, fluid_step.rs).
#pragma once

#include <cstdint>
#include <cuda_runtime.h>

namespace vxl {

constexpr uint32_t kGridDimMax = 1u << 14;   // crates/vxl-phys-core/src/grid.rs:8
constexpr uint32_t kErrGridLoop = 1u << 0;    // grid-box doubling loop did not settle

// Grid box of one substep: crates/vxl-phys-core/src/grid.rs:34-50 (min, bin, dims)
// plus inv = 1 / bin (crates/vxl-phys-fluid/src/grid.rs:50).
struct GridBox {
  float minx, miny, minz, inv;
  float bin;
  uint32_t nx, ny, nz;
  uint32_t total;
  uint32_t reach_q;  // candidate filter: the squared reach in cell units of 1/64 bin (sub_word below)
  uint32_t rows;     // neighbour-list entries by rows (k_e_groups)
  uint32_t pad;
};

// Constants of one scene, computed on the host exactly as FluidSystem::new does
// (crates/vxl-phys-fluid/src/fluid_access.rs:8-13).
struct SphConst {
  float h, h2, k6, ks, w0, b_tait, mass, rho0;
  float gamma, eps, alpha_c, h001;  // h001 = 0.01 * h2 (fluid_force.rs:197)
  float gx, gy, gz;
  uint32_t clamp_p, gamma7;
  uint32_t n_fluid, n_total, max_bins;
};

// Ordered-uint encoding of floats: monotone, so atomicMin/atomicMax on the code give
// exact float min/max independent of order.
__device__ __forceinline__ uint32_t f2o(float f) {
  uint32_t u = __float_as_uint(f);
  return (u & 0x80000000u) ? ~u : (u | 0x80000000u);
}
__device__ __forceinline__ float o2f(uint32_t o) {
  uint32_t u = (o & 0x80000000u) ? (o & 0x7fffffffu) : ~o;
  return __uint_as_float(u);
}

// `((v - o) * inv).floor().max(0.0) as u32).min(n - 1)`: crates/vxl-phys-fluid/src/grid.rs:79-100.
__device__ __forceinline__ uint32_t axis_bin(float o, float v, float inv, uint32_t n) {
  float f = fmaxf(floorf((v - o) * inv), 0.0f);
  uint32_t b = (f >= 4294967296.0f) ? 0xffffffffu : (uint32_t)f;
  return min(b, n - 1u);
}

__device__ __forceinline__ void bin_of(const GridBox& g, float x, float y, float z, uint32_t& cx,
                                       uint32_t& cy, uint32_t& cz) {
  cx = axis_bin(g.minx, x, g.inv, g.nx);
  cy = axis_bin(g.miny, y, g.inv, g.ny);
  cz = axis_bin(g.minz, z, g.inv, g.nz);
}

__device__ __forceinline__ uint32_t cell_index(const GridBox& g, float x, float y, float z) {
  uint32_t cx, cy, cz;
  bin_of(g, x, y, z, cx, cy, cz);
  uint32_t idx = (cx * g.ny + cy) * g.nz + cz;
  return min(idx, g.total - 1u);
}

// Cell of the engine's own table: z outermost, x innermost. The neighbour walk takes its 27
// cells in (dz, dy, dx) order, so in this order the three cells of a (dz, dy) row are one
// run of slots, in walk order. (The reference's table has x outermost; the export converts.)
__device__ __forceinline__ uint32_t cell_slot(const GridBox& g, float x, float y, float z) {
  uint32_t cx, cy, cz;
  bin_of(g, x, y, z, cx, cy, cz);
  return min((cz * g.ny + cy) * g.nx + cx, g.total - 1u);
}

// Candidate filter of the density walk. A slot's position inside its cell, in 1/64 of a bin
// (0..63 per axis), is kept in three 32-bit words, one for each residue p of an observer's x
// cell modulo 3: seen from there the slot's cell is the left, middle or right one of a row, so
// word p holds b = (64 ((cx - p + 1) mod 3) + x - 96, y - 32, z - 32) as signed bytes and
// floor(|b|^2 / 90) in byte 3 (|b|^2 <= 11264: at most 125). A particle at sub-cell position q
// in a cell of residue p sees the whole row at offset (dy, dz) from A = (q.x - 32, q.y - 64 dy
// - 32, q.z - 64 dz - 32), and |b - A|^2 = 2 (|b|^2 / 2 - A.b) + |A|^2: with M = (-A, 45) as signed
// bytes, one four-way byte dot product per candidate, word . M <= |b|^2 / 2 - A.b, decides
// |b - A|^2 <= T conservatively. A slot the filter drops is farther than sqrt(T); one it keeps is
// tested exactly. T = (64 h / bin + 1.75 + 4.2e-5 n)^2, n the longest axis in cells: flooring
// two positions moves their difference by less than 1 per axis (sqrt(3) = 1.733 in all), and the
// f32 rounding of (v - o) * inv (three roundings) by at most 64 n 3 2^-24 = 1.15e-5 n per axis
// and particle (2 sqrt(3) times that in all); the rest covers the rounding of r2 and of T's own
// terms. Positions outside the grid's cells are clamped into the last one, which never moves
// two particles apart, so the filter stays conservative there.
constexpr uint32_t kSubUnits = 64;
constexpr uint32_t kSubNorm = 45;  // |b|^2 / 2 is kept in multiples of this

__device__ __forceinline__ int axis_sub(float o, float v, float inv, uint32_t c) {
  const float f = (v - o) * inv * (float)kSubUnits - (float)c * (float)kSubUnits;  // power-of-two scaling: exact
  return (int)fminf(fmaxf(f, 0.0f), (float)(kSubUnits - 1));
}

__device__ __forceinline__ uint32_t sub_word(int bx, int by, int bz) {
  const uint32_t norm = (uint32_t)(bx * bx + by * by + bz * bz) / (2 * kSubNorm);
  return (uint32_t)(bx & 255) | ((uint32_t)(by & 255) << 8) | ((uint32_t)(bz & 255) << 16) | (norm << 24);
}

// IEEE quotients by a shared reciprocal. An IEEE single division costs about 36 issue slots
// on sm_100a (3.5 results per clock and SM), and a neighbour pair of the force pass has five, by
// three different denominators. With y = RN(1 / b), q = RN(a y) and the residual r = a - b q
// exact in an FMA, RN(q + r y) is the correctly rounded a / b (P. Markstein, Computation of
// elementary functions on the IBM RISC System/6000 processor, IBM J. Res. Dev. 34, 1990; also
// Muller et al., Handbook of Floating-Point Arithmetic, division by Newton-Raphson), so a
// denominator's reciprocal is formed once and each quotient by it takes three instructions. One
// Newton step from an approximation within 1 ulp (the documented bound of rcp.approx; from within 1.5
// ulp 19 significands come out wrong) rounds 1 / b correctly unless b's significand is all ones. Where a's
// significand lies below b's, q is only within 1.5 ulp and the theorem does not apply as it stands; but
// the step can then round wrongly only quotients within 4 parts in 2^48 b of a rounding midpoint, and
// tests/c/quotients.cu tries all of those for every b, and every reciprocal, on the device. The
// all-ones case and operands whose quotient or residual could leave the normal range are the caller's
// to keep out (scene_safe, pair_safe).
__device__ __forceinline__ float recip_rn(float b) {
  float y;
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(b));
  return __fmaf_rn(y, __fmaf_rn(-b, y, 1.0f), y);
}

__device__ __forceinline__ float quot_rn(float a, float b, float y) {
  const float q = a * y;
  return __fmaf_rn(__fmaf_rn(-b, q, a), y, q);
}

// Scene constants with which pair_safe keeps every quotient of a pair normal: r2 + h001 lies
// in [2^-27, 2^21], a distance no smaller than 1e-9 in [2^-30, 2^10], and alpha_c scales by
// at most 2^10 either way.
__device__ __forceinline__ bool scene_safe(float h, float alpha_c) {
  return h >= 0x1p-10f && h <= 0x1p10f && (alpha_c == 0.0f || (alpha_c >= 0x1p-10f && alpha_c <= 0x1p10f));
}

// The pair's numerators are 0 or in [2^-40, 2^40] (sum, the density sum, and mj are positive),
// and no denominator's significand is all ones. NaN and infinity fail.
__device__ __forceinline__ bool pair_safe(float sum, float mj, float coef, float vdh, float c, float denom, float dmu) {
  constexpr uint32_t kLo = 0x2b800000u, kHi = 0x53800000u, kFrac = 0x7fffffu;  // 2^-40, 2^40
  const uint32_t s = __float_as_uint(sum), m = __float_as_uint(mj), p = __float_as_uint(fabsf(coef)),
                 v = __float_as_uint(vdh), a = __float_as_uint(c);
  const uint32_t hi = max(max(max(s, m), max(p, v)), a);
  const uint32_t lo = min(min(min(s, m), min(p - 1u, v - 1u)), a - 1u);  // 0 - 1 passes
  const uint32_t frac = min(min(~s & kFrac, ~__float_as_uint(denom) & kFrac), ~__float_as_uint(dmu) & kFrac);
  return hi <= kHi && lo >= kLo && frac != 0u;
}

// Tait EOS with the free-surface clamp: crates/vxl-phys-fluid/src/fluid_force.rs:11-29.
__device__ __forceinline__ float tait(const SphConst& k, float rho) {
  float q = rho / k.rho0;
  float p;
  if (k.gamma7) {
    float q2 = q * q;
    float q4 = q2 * q2;
    p = k.b_tait * (q * q2 * q4 - 1.0f);
  } else {
    p = k.b_tait * (powf(q, k.gamma) - 1.0f);
  }
  if (k.clamp_p && p < 0.0f) p = 0.0f;
  return p;
}

// crates/vxl-phys-core/src/grid.rs:34-50 on the device (same f32 operations).
__device__ inline bool grid_box(float lox, float loy, float loz, float hix, float hiy, float hiz, float h,
                                uint32_t max_bins, GridBox& g) {
  float bin = fmaxf(h, 1e-6f);
  float ext[3] = {hix - lox, hiy - loy, hiz - loz};
  uint32_t dims[3] = {1, 1, 1};
  bool ok = false;
  for (int it = 0; it < 512; ++it) {
    for (int a = 0; a < 3; ++a) {
      float f = floorf(ext[a] / bin);
      unsigned long long d;
      if (!(f > 0.0f)) d = 0ull;
      else if (f >= 18446744073709551616.0f) d = ~0ull;
      else d = (unsigned long long)f;
      d += 1ull;  // wraps like the reference's release build
      if (d < 1ull) d = 1ull;
      if (d > kGridDimMax) d = kGridDimMax;
      dims[a] = (uint32_t)d;
    }
    if ((unsigned long long)dims[0] * dims[1] * dims[2] <= (unsigned long long)max_bins) {
      ok = true;
      break;
    }
    bin *= 2.0f;
  }
  g.minx = lox;
  g.miny = loy;
  g.minz = loz;
  g.bin = bin;
  g.inv = 1.0f / bin;
  g.nx = dims[0];
  g.ny = dims[1];
  g.nz = dims[2];
  g.total = dims[0] * dims[1] * dims[2];
  const float reach = (float)kSubUnits * (h / bin) + (1.75f + 4.2e-5f * (float)max(dims[0], max(dims[1], dims[2])));
  g.reach_q = (uint32_t)ceilf(reach * reach);
  g.rows = 0;
  return ok;
}

}  // namespace vxl
