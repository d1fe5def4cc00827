// cpm_sweep_common.cuh — device pieces shared by the sweep kernels
// (cpm_sweep.cuh, cpm_cluster.cu): lane masks, source coordinates and
// chemotaxis, the deltas of the double-buffered cell tables, the constraint
// and Metropolis arithmetic.
#pragma once

#include <cstdint>

#include "cpm_device.cuh"

namespace gpucpm {
namespace {

constexpr unsigned kFull = 0xffffffffu;

__device__ __forceinline__ unsigned lanemask_lt() {
  unsigned m;
  asm("mov.u32 %0, %%lanemask_lt;" : "=r"(m));
  return m;
}

// Chemotaxis: unit copy direction (target minus source) dotted with the
// field at the source site, every step rounded as written (the oracle
// repeats it).  As in the reference, the direction is the raw difference of
// the wrapped coordinates in 2D (src/kernels2d.cu:302-309) and the nearest
// image in 3D (src/kernels3d.cu:275-299).  F: the replica's field, `sites`
// values per component.
__device__ __forceinline__ int wrap_coord(int v, int n) {
  return v < 0 ? v + n : (v >= n ? v - n : v);
}

// Coordinates of the source of an attempt: neighbour `kdir` (in (dz, dy, dx)
// order, the target itself left out) of the target (x, y, z), wrapped.
template <int NDIM>
__device__ __forceinline__ void source_coords(int kdir, int x, int y, int z, int nx, int ny,
                                              int nz, int& sx, int& sy, int& sz) {
  int ox, oy, oz;
  if (NDIM == 2) {
    const int m = kdir + (kdir >= 4);
    oz = 0;
    oy = m / 3 - 1;
    ox = m % 3 - 1;
  } else {
    const int m = kdir + (kdir >= 13);
    oz = m / 9 - 1;
    oy = (m / 3) % 3 - 1;
    ox = m % 3 - 1;
  }
  sx = wrap_coord(x + ox, nx);
  sy = wrap_coord(y + oy, ny);
  sz = NDIM == 3 ? wrap_coord(z + oz, nz) : 0;
}

// Unit copy direction (target minus source) of neighbour kdir: the raw
// difference of the wrapped coordinates in 2D (src/kernels2d.cu:302-309),
// the nearest image in 3D (src/kernels3d.cu:275-299); FP32, rounded as
// written (the oracle repeats it).  Also returns the source coordinates.
template <int NDIM>
__device__ __forceinline__ void unit_dir(int kdir, int x, int y, int z, int nx, int ny, int nz,
                                         float& ux, float& uy, float& uz, int& sx, int& sy,
                                         int& sz) {
  source_coords<NDIM>(kdir, x, y, z, nx, ny, nz, sx, sy, sz);
  int dx = x - sx, dy = y - sy, dz = z - sz;
  if (NDIM == 3) {
    if (dx > nx / 2) dx -= nx;
    if (dx < -(nx / 2)) dx += nx;
    if (dy > ny / 2) dy -= ny;
    if (dy < -(ny / 2)) dy += ny;
    if (dz > nz / 2) dz -= nz;
    if (dz < -(nz / 2)) dz += nz;
  }
  const float fx = (float)dx, fy = (float)dy, fz = (float)dz;
  float s2 = __fmul_rn(fx, fx);
  s2 = __fmaf_rn(fy, fy, s2);
  if (NDIM == 3) s2 = __fmaf_rn(fz, fz, s2);
  const float len = __fsqrt_rn(s2);
  ux = __fdiv_rn(fx, len);
  uy = __fdiv_rn(fy, len);
  uz = NDIM == 3 ? __fdiv_rn(fz, len) : 0.0f;
}

template <int NDIM>
__device__ __forceinline__ float chemo_dot(const float* F, long long sites, int x, int y,
                                           int z, int kdir, int nx, int ny, int nz) {
  float ux, uy, uz;
  int sx, sy, sz;
  unit_dir<NDIM>(kdir, x, y, z, nx, ny, nz, ux, uy, uz, sx, sy, sz);
  const long long site = ((long long)sz * ny + sy) * nx + sx;
  float c = __fmul_rn(ux, __ldg(F + site));
  c = __fmaf_rn(uy, __ldg(F + sites + site), c);
  if (NDIM == 3) c = __fmaf_rn(uz, __ldg(F + 2 * sites + site), c);
  return c;
}

// Per-phase view of the double-buffered tables.
template <int NDIM>
struct PhaseTables {
  const unsigned long long* rap;  // read copy (tables at phase start)
  const long long* rcs;
  unsigned long long* wap;        // other copy: receives this phase's deltas
  long long* wcs;
  unsigned long long* dap;        // this phase's deltas (replayed next phase)
  long long* dcs;
};

// One accepted copy's change of one table row: added to the other table
// copy and to the phase delta table.  Reductions only (no value comes
// back), so the accepting warp does not wait on L2.  The row goes on the
// block's dirty list separately (warp-aggregated, duplicates allowed).
template <int NDIM>
__device__ __forceinline__ void add_delta(const PhaseTables<NDIM>& pt,
                                          long long row, int darea, int dperim,
                                          const long long* img, long long sign) {
  const unsigned long long pd = pack_delta(darea, dperim);
  atomicAdd(pt.wap + row, pd);
  atomicAdd(pt.dap + row, pd);
#pragma unroll
  for (int k = 0; k < NDIM; ++k) {
    const unsigned long long v = (unsigned long long)(sign * img[k]);
    atomicAdd(reinterpret_cast<unsigned long long*>(pt.wcs + row * NDIM + k), v);
    atomicAdd(reinterpret_cast<unsigned long long*>(pt.dcs + row * NDIM + k), v);
  }
}

// A type's constraint parameters, one 16-byte shared-memory load.
struct alignas(16) TypeParams {
  float lam_area;
  int tgt_area;
  float lam_perim;
  int tgt_perim;
};
// Words per row of the shared-memory adhesion matrix: entry (a, b) lies in
// bank 5 a + b, so that up to five types never meet in one.
constexpr int kJPitch = 37;

// The integers that the constraints multiply: dp (2 (P - P*) + dp) for a
// perimeter that changes by dp, 1 +- 2 (A - A*) for an area that changes by
// +-1 (`sign`), each rounded once to FP32.  Where the tables and targets are
// below 2^21 (kSmallTable) all factors are exact in FP32 and so is the rounding
// of their product; otherwise in 64 bits.
constexpr unsigned kSmallTable = 1u << 21;
__device__ __forceinline__ void constraint_terms_small(int area, int perim, int dp, int sign,
                                                       const TypeParams& p, float& qp,
                                                       float& qa) {
  qp = __fmul_rn((float)dp, (float)(2 * (perim - p.tgt_perim) + dp));
  qa = (float)(1 + sign * 2 * (area - p.tgt_area));
}
__device__ __forceinline__ void constraint_terms_wide(int area, int perim, int dp, int sign,
                                                      const TypeParams& p, float& qp,
                                                      float& qa) {
  qp = __ll2float_rn((long long)dp * (2LL * ((long long)perim - p.tgt_perim) + dp));
  qa = __ll2float_rn(1 + sign * 2LL * ((long long)area - p.tgt_area));
}

// Metropolis test.  `draw`: the attempt's random word; ex receives
// exp(-dH/T) where 0 <= dH and T > 0.
__device__ __forceinline__ bool metropolis(float dH, float T, uint32_t draw, float& ex) {
  if (dH < 0.0f) return true;
  if (!(T > 0.0f)) return false;
  ex = exp_neg(__fdiv_rn(-dH, T));
  return __fmul_rn(__uint2float_rn((draw >> 8) | 1u), 0x1p-24f) < ex;
}

// Paired evaluation: an attempt on two neighbouring lanes, the even one
// (side 0) with the source cell's values, the odd one (side 1) with the
// target cell's.  Each sums its own configuration's adhesion e (side 0 the
// new one's, side 1 the old one's) and its own constraint integers; the
// energy is put together on both in the order of the one-lane form:
// adhesion, chemotaxis (and what else `extra` holds), perimeter of source
// and target, area of source and target.  Where a phase is the chain of one
// warp through its attempts this halves what a lane does one after the
// other.  `mask`: the lanes that call, pairs complete.
__device__ __forceinline__ float pair_energy(unsigned mask, int side, bool has_s, bool has_t,
                                             float e, float extra, float qp, float qa,
                                             const TypeParams& p, bool perim_on) {
  const float e2 = __shfl_xor_sync(mask, e, 1);
  const float qp2 = __shfl_xor_sync(mask, qp, 1), qa2 = __shfl_xor_sync(mask, qa, 1);
  const float lp2 = __shfl_xor_sync(mask, p.lam_perim, 1);
  const float la2 = __shfl_xor_sync(mask, p.lam_area, 1);
  float dH = __fsub_rn(side ? e2 : e, side ? e : e2);
  dH = __fadd_rn(extra, dH);
  if (perim_on) {
    const float ds = __fmaf_rn(side ? lp2 : p.lam_perim, side ? qp2 : qp, dH);
    dH = has_s ? ds : dH;
    const float dt = __fmaf_rn(side ? p.lam_perim : lp2, side ? qp : qp2, dH);
    dH = has_t ? dt : dH;
  }
  const float ds = __fmaf_rn(side ? la2 : p.lam_area, side ? qa2 : qa, dH);
  dH = has_s ? ds : dH;
  const float dt = __fmaf_rn(side ? p.lam_area : la2, side ? qa : qa2, dH);
  return has_t ? dt : dH;
}

}  // namespace
}  // namespace gpucpm
