// Receiver gather, adjoint-source injection and boundary-shell save/restore
// in the stencil kernels' epilogues (the reference runs them as separate
// kernels every step: recording and res_injection, utilities.cu:481-507;
// from_bnd / to_bnd, utilities.cu:323-420 with Boundary.cu:59-138).
//
// Shell: the points of the reference's 5-cell boundary shell inside
// [2, n-3]^3 are stored per step as [9][npts] in (z, x, y) order.  A row
// (z, x) of the grid holds no shell point, one run of points y in
// [ya0, yb1], or two runs [ya0, ya1] and [yb0, yb1] (ShellMap), so a thread
// finds its cell's shell index in O(1) from one row entry that is uniform
// over its warp.  Receivers: a per-plane map of unique receiver cells
// (RecArgs::plane, RecArgs::map).
#pragma once
#include "efwi_common.cuh"
#include "efwi_kernels.h"
#include "efwi_vec.cuh"

namespace efwi {

constexpr int SHELL_SPLIT = 1 << 30;

// Shell point index of a cell at y whose row entry is `row`, or -1.
__host__ __device__ __forceinline__ int shell_index(const ShellMap &s, int row, int y) {
  if (row < 0) return -1;
  const int base = row & ~SHELL_SPLIT;
  if (!(row & SHELL_SPLIT)) return (y >= s.ya0 && y <= s.yb1) ? base + y - s.ya0 : -1;
  if (y >= s.ya0 && y <= s.ya1) return base + y - s.ya0;
  if (y >= s.yb0 && y <= s.yb1) return base + (s.ya1 - s.ya0 + 1) + y - s.yb0;
  return -1;
}

// Shell point indices of the four cells of a vector in a row with entry
// `row` (-1: none, or a cell that the thread does not update); true when
// there is one.
__device__ __forceinline__ bool shell_cells(const ShellMap &s, int row, const VecCell &c,
                                            int k[VEC]) {
  bool any = false;
#pragma unroll
  for (int e = 0; e < VEC; ++e) {
    k[e] = c.act[e] ? shell_index(s, row, c.y + e) : -1;
    any = any || k[e] >= 0;
  }
  return any;
}

// Map of the receiver cells in plane z of the shot, or -1.
__device__ __forceinline__ int receiver_map(const RecArgs &r, int nz, int shot, int z) {
  return r.plane ? r.plane[shot * nz + z] : -1;
}
// The map's entries at the four cells of vector c.
__device__ __forceinline__ const float *receiver_row(const RecArgs &r, int map, const Geo &g,
                                                     const VecCell &c) {
  return reinterpret_cast<const float *>(r.map + (long long)map * r.nxpy + c.x * g.sx + c.y);
}

// f(r) for the receivers r on a cell with map entry u, in their order.
template <class F>
__device__ __forceinline__ void receivers_of(const RecArgs &rec, int u, F f) {
  int k = 0, end = 1;
  if (u >= 0) { k = rec.uptr[u]; end = rec.uptr[u + 1]; }
#pragma unroll 1
  for (; k < end; ++k) f(u >= 0 ? rec.rec[k] : -2 - u);
}

// recording (utilities.cu:481-495) of the components wanted (x, y, z) at a
// receiver cell of the shot (map entry u) at sample it.
__device__ __forceinline__ void record_cell(const RecArgs &rec, float *traces_tm, int it, int shot,
                                            int u, bool x, float vx, bool y, float vy, bool z,
                                            float vz) {
  const int nr = rec.nrec[shot];
  float *t = traces_tm + rec.trace_off[shot] + (long long)it * 3 * nr;
  receivers_of(rec, u, [&](int r) {
    if (x) t[r] = vx;
    if (y) t[nr + r] = vy;
    if (z) t[2 * nr + r] = vz;
  });
}

// res_injection (utilities.cu:497-507) at a receiver cell of shot 0 (map
// entry u): the receivers on the cell are added one after the other in
// receiver order.
__device__ __forceinline__ void inject_cell(const RecArgs &rec, const float *res_tm, int it, int u,
                                            float &vz, float &vx, float &vy) {
  const int nr = rec.nrec[0];
  const float *t = res_tm + rec.trace_off[0] + (long long)it * 3 * nr;
  receivers_of(rec, u, [&](int r) {
    vx += t[r];
    vy += t[nr + r];
    vz += t[2 * nr + r];
  });
}

}  // namespace efwi
