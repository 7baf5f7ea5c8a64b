// pip_ghosts.cuh -- ghost images of an updated cell (PIPbnd after the stage: x faces first,
// then y faces, Boundary_rot.f90:54-125 order, so a corner ghost carries both sign flips).
#pragma once

#include "pip_kernels.cuh"

namespace pip {

// Only cells within 2*margin of a boundary can be a ghost source.
template <int NDIM>
__device__ __forceinline__ bool near_boundary(const KParams &p, int gi, int gj) {
  return gi < 2 * p.m0 || gi >= p.ix - 2 * p.m0 ||
         (NDIM == 2 && (gj < 2 * p.m1 || gj >= p.jx - 2 * p.m1));
}

// Calls put(offset in the plane, flips) for every ghost image of cell (gi, gj); bit n of
// flips: plane n changes sign there.  Each lane walks the set bits of its own source masks,
// so the lanes of a warp write their first images together, then their second ones; the
// caller keeps the cell's planes in registers.  Measured on a 64x64 grid, cycles from a corner
// tile's update to its last store: 9000 when each plane was read back from the state and
// every candidate tested in turn, 8000 with the planes in registers, 1000 with the masks.
template <int NDIM, typename F>
__device__ __forceinline__ void ghost_images(const KParams &p, int gi, int gj, F put) {
  unsigned mx = 0u, my = 0u;      // bit s*kMaxMargin + l: ghost layer l of side s copies the cell
#pragma unroll
  for (int s = 0; s < 2; ++s)
#pragma unroll
    for (int l = 0; l < kMaxMargin; ++l) {
      if (p.gx[s][l] == gi) mx |= 1u << (s * kMaxMargin + l);
      if (NDIM == 2 && p.gy[s][l] == gj) my |= 1u << (s * kMaxMargin + l);
    }
  int a = -1;
  for (;;) {
    const int sx = a >= kMaxMargin ? 1 : 0, lx = a - sx * kMaxMargin;
    const int tx = a < 0 ? gi : sx ? p.ix - p.m0 + lx : lx;
    const unsigned fx = a < 0 ? 0u : sx ? p.flipx[1] : p.flipx[0];
    int b = -1;
    for (unsigned rest = my;;) {
      if (a >= 0 || b >= 0) {
        const int sy = b >= kMaxMargin ? 1 : 0, ly = b - sy * kMaxMargin;
        const int ty = b < 0 ? gj : sy ? p.jx - p.m1 + ly : ly;
        const unsigned fy = b < 0 ? 0u : sy ? p.flipy[1] : p.flipy[0];
        put((long long)ty * p.ix + tx, fx ^ fy);
      }
      if (NDIM == 1 || !rest) break;
      b = __ffs(rest) - 1;
      rest &= rest - 1u;
    }
    if (!mx) break;
    a = __ffs(mx) - 1;
    mx &= mx - 1u;
  }
}

// v with its sign changed where bit n of flips is set.
__device__ __forceinline__ double flipped(double v, unsigned flips, int n) {
  return __hiloint2double(__double2hiint(v) ^ (int)((flips >> n) << 31), __double2loint(v));
}
__device__ __forceinline__ float flipped(float v, unsigned flips, int n) {
  return __int_as_float(__float_as_int(v) ^ (int)((flips >> n) << 31));
}

}  // namespace pip
