// Four-cell vectors of the direct stencil kernels (efwi_fwd_vec.cu,
// efwi_rev_vec.cu, efwi_exact_vec.cu).
//
// A thread owns the four cells y .. y+3 (y a multiple of 4, so every row
// access is one aligned 16-byte load: the pitch is a multiple of 4) of one row
// (z, x).  Its y neighbours are the tail of the vector before and the head of
// the vector after it; its x and z neighbours are the same vector of other
// rows.  Nothing is shared between threads inside a launch: neighbours come
// through L1 and L2, and every load of a thread is independent of the others.
#pragma once
#include "efwi_common.cuh"

namespace efwi {

constexpr int VEC = 4;

// CTA of the stencil kernels: 8 vectors (32 cells along y: one 128-byte line
// per row) x 4 rows x 4 planes.  A CTA's rows and planes share their halo
// through L1, and 128 threads keep the waves small.  On the 152^3 grid 16
// vectors x 2 rows x 4 planes ran 12 % slower, 2-row or 2-plane CTAs 1-8 %,
// 256-thread ones 3-6 %.
//
// A kernel has several outputs.  With enough CTAs a thread forms them one after
// the other; on small grids (vec_split) PARTS warps of a CTA share one plane's
// outputs, a part to each, and the latency of a launch drops to that of the
// longest part.
constexpr int VEC_TY = 8, VEC_TX = 4, VEC_TZ = 4, VEC_THREADS = VEC_TY * VEC_TX * VEC_TZ;
// planes and threads of a CTA whose vectors have PARTS threads
constexpr int vec_tz(int parts) { return parts > 1 ? 1 : VEC_TZ; }
constexpr int vec_threads(int parts) { return VEC_TY * VEC_TX * vec_tz(parts) * parts; }
__device__ __forceinline__ int vec_thread() {
  return (threadIdx.z * VEC_TX + threadIdx.y) * VEC_TY + threadIdx.x;
}

struct Row {
  float v[VEC];
  __device__ __forceinline__ float operator[](int e) const { return v[e]; }
};

__device__ __forceinline__ Row ld_row(const float *p) {
  const float4 t = *reinterpret_cast<const float4 *>(p);
  return Row{{t.x, t.y, t.z, t.w}};
}
__device__ __forceinline__ void st_row(float *p, const Row &r) {
  *reinterpret_cast<float4 *>(p) = make_float4(r.v[0], r.v[1], r.v[2], r.v[3]);
}

// Asks for the thread's row of a field that a later part of the kernel reads:
// into L2, so that the part waits for L2 and not for DRAM.  One lane per
// 128-byte line.
__device__ __forceinline__ void prefetch_row(const float *p) {
  if (threadIdx.x == 0) asm volatile("prefetch.global.L2 [%0];" ::"l"(p));
}

// Cells y-2 .. y+5 of a row around the vector c at y: (e, k) is cell y+e+k.
struct Span {
  float v[VEC + 4];
  __device__ __forceinline__ float operator()(int e, int k) const { return v[e + k + 2]; }
};

// The thread's place in its launch.
struct VecCell {
  int z, x, y;        // first of the four cells
  int i;              // its linear index
  bool lo, hi;        // a vector lies before / after it in the row
  bool act[VEC];      // cells of [2, ny-3]
};

__device__ __forceinline__ VecCell vec_cell(const Geo &g, int z, int x, int y, int pitch) {
  VecCell c;
  c.z = z; c.x = x; c.y = y;
  c.i = (z * g.nx + x) * pitch + y;
  c.lo = y > 0;
  c.hi = y + VEC < pitch;
#pragma unroll
  for (int e = 0; e < VEC; ++e) c.act[e] = y + e >= 2 && y + e <= g.ny - 3;
  return c;
}
__device__ __forceinline__ VecCell vec_cell(const Geo &g, int z, int x, int y) {
  return vec_cell(g, z, x, y, g.sx);
}

// The vector m at p with its neighbours; cells outside the row (only ever
// next to inactive cells) read as zero.
__device__ __forceinline__ Span ld_span(const float *p, const Row &m, const VecCell &c) {
  float2 l = make_float2(0.f, 0.f), r = make_float2(0.f, 0.f);
  if (c.lo) l = *reinterpret_cast<const float2 *>(p - 2);
  if (c.hi) r = *reinterpret_cast<const float2 *>(p + VEC);
  return Span{{l.x, l.y, m.v[0], m.v[1], m.v[2], m.v[3], r.x, r.y}};
}

// The C-PML work of a thread.  A slab row along y (z and x slabs) has ny
// cells, a y slab row 2 np.  VA: ny and np are multiples of 4, so that every
// vector lies in or out of a slab as a whole and its four memory variables
// are one aligned 16-byte vector; otherwise they are single cells, of which
// those that the thread's cells do not own are not touched.  The two cases
// are separate kernels: the single-cell code would more than double the
// instructions that a vector-aligned grid has to fetch past.
inline bool psi_vectors(const Geo &g) { return ((g.ny | g.np) & 3) == 0; }

template <bool VA>
struct Pml {
  bool zs, xs;
  bool ys[VEC], yany;
  int kz, kx, ky;
};

// `v` selects the velocity update's slabs (quirk Q2: x and y start one cell
// later on the high side).
template <bool VA>
__device__ __forceinline__ Pml<VA> pml_of(const Geo &g, const VecCell &c, bool v) {
  Pml<VA> p;
  p.zs = slab_s(c.z, g.nz, g.np);
  p.xs = v ? slab_v(c.x, g.nx, g.np) : slab_s(c.x, g.nx, g.np);
  p.kz = p.zs ? psi_z_idx(g, c.z, c.x, c.y) : 0;
  p.kx = p.xs ? psi_x_idx(g, c.z, c.x, c.y) : 0;
  p.yany = c.y < g.np || c.y + VEC > g.ny - g.np;
  // index of cell y (VA; single cells: of cell y on the low side)
  p.ky = (c.z * g.nx + c.x) * (2 * g.np) + c.y;
  if (VA && c.y >= g.np) p.ky -= g.ny - 2 * g.np;
#pragma unroll
  for (int e = 0; e < VEC; ++e) {
    const int y = c.y + e;
    p.ys[e] = c.act[e] && (v ? slab_v(y, g.ny, g.np) : slab_s(y, g.ny, g.np));
  }
  return p;
}

// Four cells at offset k of a z or x slab.
template <bool VA>
__device__ __forceinline__ Row ld_psi(const float *p, int k, const VecCell &c) {
  if (VA) return ld_row(p + k);
  Row r;
#pragma unroll
  for (int e = 0; e < VEC; ++e) r.v[e] = c.act[e] ? p[k + e] : 0.f;
  return r;
}
template <bool VA>
__device__ __forceinline__ void st_psi(float *p, int k, const Row &r, const VecCell &c) {
  if (VA) { st_row(p + k, r); return; }
#pragma unroll
  for (int e = 0; e < VEC; ++e)
    if (c.act[e]) p[k + e] = r.v[e];
}
// The same of memory variable `slot` of an axis with slabs of `slab` cells.  Its
// offset passes 2^31 cells on large grids; whole vectors are counted in 32 bits.
template <bool VA>
__device__ __forceinline__ Row ld_psi(const float *p, int slot, long long slab, int k,
                                      const VecCell &c) {
  if (VA)
    return ld_row(p + (size_t)(slot * ((unsigned)slab / VEC) + (unsigned)k / VEC) * VEC);
  return ld_psi<VA>(p + slot * slab, k, c);
}
// Four cells of a y slab.
template <bool VA>
__device__ __forceinline__ int psi_y_cell(const Geo &g, const Pml<VA> &m, const VecCell &c, int e) {
  return m.ky + e - (c.y + e < g.np ? 0 : g.ny - 2 * g.np);
}
template <bool VA>
__device__ __forceinline__ Row ld_psi_y(const float *p, const Geo &g, const Pml<VA> &m,
                                        const VecCell &c) {
  if (VA) return ld_row(p + m.ky);
  Row r;
#pragma unroll
  for (int e = 0; e < VEC; ++e) r.v[e] = m.ys[e] ? p[psi_y_cell(g, m, c, e)] : 0.f;
  return r;
}
template <bool VA>
__device__ __forceinline__ Row ld_psi_y(const float *p, int slot, const Geo &g, const Pml<VA> &m,
                                        const VecCell &c) {
  if (VA) return ld_psi<VA>(p, slot, g.slab_y, m.ky, c);
  return ld_psi_y(p + slot * g.slab_y, g, m, c);
}
template <bool VA>
__device__ __forceinline__ void st_psi_y(float *p, const Row &r, const Pml<VA> &m, const Geo &g,
                                         const VecCell &c) {
  if (VA) { st_row(p + m.ky, r); return; }
#pragma unroll
  for (int e = 0; e < VEC; ++e)
    if (m.ys[e]) p[psi_y_cell(g, m, c, e)] = r.v[e];
}

// Coefficient row `which` of the y profile at the thread's cells.
template <bool VA>
__device__ __forceinline__ Row coef_y(const Geo &g, const VecCell &c, int which) {
  const float *p = g.cy + which * g.ny + c.y;
  if (VA) return ld_row(p);
  Row r;
#pragma unroll
  for (int e = 0; e < VEC; ++e) r.v[e] = c.y + e < g.ny ? p[e] : 0.f;
  return r;
}
__device__ __forceinline__ Row fill(float v) { return Row{{v, v, v, v}}; }

// prefetch_row of the memory variables s0 .. s0 + N - 1 at the thread's row.
template <int N, bool VA>
__device__ __forceinline__ void prefetch_psi(const Geo &g, const Psi &ps, const Pml<VA> &m,
                                             const VecCell &c, int s0) {
  if (!g.far) return;
  const bool ys = c.y < g.np || c.y + VEC * VEC_TY > g.ny - g.np;  // of lane 0: the CTA's row
#pragma unroll
  for (int k = 0; k < N; ++k) {
    if (m.zs) prefetch_row(ps.z + (s0 + k) * g.slab_z + m.kz);
    if (m.xs) prefetch_row(ps.x + (s0 + k) * g.slab_x + m.kx);
    if (ys) prefetch_row(ps.y + (s0 + k) * g.slab_y + (c.z * g.nx + c.x) * (2 * g.np));
  }
}

// m = b m + a d,  d = d / K + m  of one cell.
__device__ __forceinline__ void pml_step(float Ki, float a, float b, float &m, float &d) {
  m = __fmaf_rn(a, d, __fmul_rn(b, m));
  d = d * Ki + m;
}

// Derivative d of the z axis (x: the same): `r` holds the memory variables,
// loaded before the derivative's operands so that the latencies overlap;
// cf: the axis's coefficient rows of n at the thread's cell.
template <bool VA>
__device__ __forceinline__ void pml_row(float *p, int k, Row &r, const VecCell &c, const float *cf,
                                        int n, float d[VEC]) {
  const float Ki = cf[CK * n], a = cf[CA * n], b = cf[CB * n];
#pragma unroll
  for (int e = 0; e < VEC; ++e) {
    float m = r.v[e];
    pml_step(Ki, a, b, m, d[e]);
    if (c.act[e]) r.v[e] = m;
  }
  st_psi<VA>(p, k, r, c);
}

// Derivative d of the y axis (half: coefficients at half points).
template <bool VA>
__device__ __forceinline__ void pml_row_y(float *p, Row &r, const Geo &g, const Pml<VA> &m,
                                          const VecCell &c, int half, float d[VEC]) {
  const Row Ki = coef_y<VA>(g, c, 3 * half + CK), a = coef_y<VA>(g, c, 3 * half + CA),
            b = coef_y<VA>(g, c, 3 * half + CB);
#pragma unroll
  for (int e = 0; e < VEC; ++e)
    if (m.ys[e]) pml_step(Ki[e], a[e], b[e], r.v[e], d[e]);
  st_psi_y(p, r, m, g, c);
}

// ---- adjoint side: the memory variables of one axis at the stencil's four
// points, negated and transposed differences (zero outside the slab, where
// the reference's full-grid arrays are never written).
template <bool VA>
struct PsiGather {
  const Geo &g;
  const VecCell &c;
  const Pml<VA> &m;
  __device__ __forceinline__ Row x(const float *p, int xn) const {
    return slab_s(xn, g.nx, g.np) ? ld_psi<VA>(p, psi_x_idx(g, c.z, xn, c.y), c) : Row{};
  }
  __device__ __forceinline__ Row z(const float *p, int zn) const {
    return slab_s(zn, g.nz, g.np) ? ld_psi<VA>(p, psi_z_idx(g, zn, c.x, c.y), c) : Row{};
  }
  __device__ __forceinline__ Span y(const float *p) const {
    Span s{};
    if (VA) {
      const Row r = ld_row(p + m.ky);
      float2 l = make_float2(0.f, 0.f), h = make_float2(0.f, 0.f);
      if (c.y > 0 && slab_s(c.y - 1, g.ny, g.np)) l = *reinterpret_cast<const float2 *>(p + m.ky - 2);
      if (c.y + VEC < g.ny && slab_s(c.y + VEC, g.ny, g.np))
        h = *reinterpret_cast<const float2 *>(p + m.ky + VEC);
      return Span{{l.x, l.y, r.v[0], r.v[1], r.v[2], r.v[3], h.x, h.y}};
    }
    const float *row = p + (c.z * g.nx + c.x) * (2 * g.np);
#pragma unroll
    for (int k = 0; k < VEC + 4; ++k) {
      const int yn = c.y + k - 2;
      if (yn >= 0 && yn < g.ny && slab_s(yn, g.ny, g.np)) s.v[k] = row[slab_c(yn, g.ny, g.np)];
    }
    return s;
  }
  __device__ __forceinline__ Row dpx(const float *p) const {
    const Row a = x(p, c.x - 1), b = x(p, c.x), d = x(p, c.x + 1), h = x(p, c.x + 2);
    Row r;
#pragma unroll
    for (int e = 0; e < VEC; ++e) r.v[e] = __fmul_rn(-dplus(a[e], b[e], d[e], h[e]), g.idx);
    return r;
  }
  __device__ __forceinline__ Row dmx(const float *p) const {
    const Row a = x(p, c.x - 2), b = x(p, c.x - 1), d = x(p, c.x), h = x(p, c.x + 1);
    Row r;
#pragma unroll
    for (int e = 0; e < VEC; ++e) r.v[e] = __fmul_rn(-dminus(a[e], b[e], d[e], h[e]), g.idx);
    return r;
  }
  __device__ __forceinline__ Row dpz(const float *p) const {
    const Row a = z(p, c.z - 1), b = z(p, c.z), d = z(p, c.z + 1), h = z(p, c.z + 2);
    Row r;
#pragma unroll
    for (int e = 0; e < VEC; ++e) r.v[e] = __fmul_rn(-dplus(a[e], b[e], d[e], h[e]), g.idz);
    return r;
  }
  __device__ __forceinline__ Row dmz(const float *p) const {
    const Row a = z(p, c.z - 2), b = z(p, c.z - 1), d = z(p, c.z), h = z(p, c.z + 1);
    Row r;
#pragma unroll
    for (int e = 0; e < VEC; ++e) r.v[e] = __fmul_rn(-dminus(a[e], b[e], d[e], h[e]), g.idz);
    return r;
  }
  __device__ __forceinline__ Row dpy(const float *p) const {
    const Span s = y(p);
    Row r;
#pragma unroll
    for (int e = 0; e < VEC; ++e) r.v[e] = __fmul_rn(-dplus(s(e, -1), s(e, 0), s(e, 1), s(e, 2)), g.idy);
    return r;
  }
  __device__ __forceinline__ Row dmy(const float *p) const {
    const Span s = y(p);
    Row r;
#pragma unroll
    for (int e = 0; e < VEC; ++e) r.v[e] = __fmul_rn(-dminus(s(e, -2), s(e, -1), s(e, 0), s(e, 1)), g.idy);
    return r;
  }
};

// Memory-variable update m = b m + add dt of a z or x slab row, or of a y slab
// row with the coefficients b of its cells.  OLD: the product with the old
// value is the one that the sum's rounding takes in.
template <bool VA, bool OLD = false>
__device__ __forceinline__ void mem_row(float *p, int k, const VecCell &c, float b,
                                        const Row &add, float dt) {
  Row r = ld_psi<VA>(p, k, c);
#pragma unroll
  for (int e = 0; e < VEC; ++e)
    if (c.act[e])
      r.v[e] = OLD ? __fmaf_rn(b, r[e], __fmul_rn(add[e], dt)) : __fmaf_rn(add[e], dt, __fmul_rn(b, r[e]));
  st_psi<VA>(p, k, r, c);
}
template <bool VA>
__device__ __forceinline__ void mem_row_y(float *p, const Geo &g, const Pml<VA> &m,
                                          const VecCell &c, const Row &b, const Row &add,
                                          float dt) {
  Row r = ld_psi_y(p, g, m, c);
#pragma unroll
  for (int e = 0; e < VEC; ++e)
    if (m.ys[e]) r.v[e] = __fmaf_rn(add[e], dt, __fmul_rn(b[e], r[e]));
  st_psi_y(p, r, m, g, c);
}

// Rows that a thread needs at its own cell only, brought to shared memory by
// asynchronous 16-byte copies that it issues before its first neighbour load
// and reads back after the differences: the bytes in flight cost no
// registers, and as every thread reads only what it copied itself there is
// no barrier.  `slot` is row-major over the CTA's threads (conflict-free).
template <int THREADS>
struct Stash {
  float4 *slot;  // [rows][THREADS], already at the thread's column
  __device__ __forceinline__ void fetch(int r, const float *p) {
    const uint32_t dst = (uint32_t)__cvta_generic_to_shared(slot + r * THREADS);
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst), "l"(p) : "memory");
  }
  __device__ __forceinline__ void wait() { asm volatile("cp.async.wait_all;" ::: "memory"); }
  __device__ __forceinline__ Row get(int r) const {
    const float4 t = slot[r * THREADS];
    return Row{{t.x, t.y, t.z, t.w}};
  }
};

// Grid over the cells [2, n-3]^3 (y: vectors up to the one of cell ny-3) of S
// shots.
inline dim3 vec_grid(const Geo &g, int S = 1, int parts = 1) {
  const int TZ = vec_tz(parts);
  const int nv = (g.ny - 3) / VEC + 1, nzb = (g.nz - 4 + TZ - 1) / TZ;
  return dim3((nv + VEC_TY - 1) / VEC_TY, (g.nx - 4 + VEC_TX - 1) / VEC_TX, (unsigned)(S * nzb));
}
// The forward kernels split their outputs over warps where the unsplit grid
// would leave SMs short of one wave (5 CTAs of 148 SMs): launches then take one
// thread's chain of loads, which the split shortens.  Of an isolated launch,
// unsplit and split (us, ~6 of them the measurement): 26 x 30 x 28 K_S 10.5 /
// 8.4; 84^3 (1200 CTAs) 22.6 / 18.5, but 45.1 / 48.2 ms for the whole gradient
// there, whose launches overlap; 152^3 72 / 98 and 56 / 58: a split vector's
// rows are loaded by several warps.
constexpr int VEC_SPLIT_CTAS = 148 * 5;
inline bool vec_split(const Geo &g, int S) {
  const dim3 n = vec_grid(g, S);
  return (long long)n.x * n.y * n.z < VEC_SPLIT_CTAS;
}
inline bool vec_fits(const Geo &g, int S) {
  return (g.nx - 4 + VEC_TX - 1) / VEC_TX <= 65535 &&
         (long long)S * ((g.nz - 4 + VEC_TZ - 1) / VEC_TZ) <= 65535;
}

// Launch of a stencil kernel.  `chained`: it may begin while the kernel before
// it in the stream drains (programmatic dependent launch).  Then what the
// kernel reads before vec_begin() must not be written by the kernel right
// before it; kernels further back are complete, since that one is past its own
// vec_begin().  Such reads are the rows of the fields that the kernel itself
// updates, the model and the images.
template <class... P, class... T>
inline void vec_launch(void (*kernel)(P...), dim3 grid, int tz, bool chained, cudaStream_t st,
                       T... args) {
  cudaLaunchAttribute at{};
  at.id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at.val.programmaticStreamSerializationAllowed = 1;
  cudaLaunchConfig_t cf{};
  cf.gridDim = grid;
  cf.blockDim = dim3(VEC_TY, VEC_TX, tz);
  cf.stream = st;
  cf.attrs = &at;
  cf.numAttrs = chained ? 1 : 0;
  cudaLaunchKernelEx(&cf, kernel, static_cast<P>(args)...);
}
// Waits until the kernels before this one are complete and their writes
// visible, then lets the next kernel's CTAs start (once all of this grid's
// have come here or left).
__device__ __forceinline__ void vec_begin() {
  asm volatile("griddepcontrol.wait;" ::: "memory");
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
}

}  // namespace efwi
