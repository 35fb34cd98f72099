// Exact discrete adjoint of the forward time step, one thread per four cells
// (efwi_vec.cuh); the same transposes and images as efwi_exact.cu, whose
// notation is used here: G = coefficient x adjoint of an output, Q = G outside
// the slab and G / K + a (L + G) in it, the adjoint field gathers -D-transposed
// Q of its neighbours.
//
// A CTA (8 vectors x 4 rows x 4 planes) forms the Q of its cells and of their
// halo once into shared memory -- z-axis terms with two planes on each side,
// x-axis terms with two rows, y-axis terms with a vector -- and after a barrier
// every thread gathers from there.  Forming the neighbours' Q in every thread
// from global memory instead takes 66 row loads per thread where this takes 24
// and thrashes L1: 105 / 91 us per launch (stress / velocity stage) at 120^3.
//
// A vector has two threads.  Latency bounds the kernel (a third of the DRAM and
// L2 rates), and the images need nothing of the Q: the second half of the
// warps forms them while the first takes the Q's items, 32 at a time, then
// helps with what is left; after the barrier the halves share the outputs.
#include "efwi_common.cuh"
#include "efwi_exact.h"
#include "efwi_vec.cuh"

namespace efwi {
namespace {

// Q of the CTA's terms.  z rows are planes z0-2 .. z0+5 of the CTA's x rows, x
// rows are x0-2 .. x0+5 of its planes, y rows have a vector on each side.
constexpr int QZ = VEC_TZ + 4, QX = VEC_TX + 4, QY = VEC_TY + 2;
struct QTile {
  float4 z[3][QZ][VEC_TX][VEC_TY];
  float4 x[3][VEC_TZ][QX][VEC_TY];
  float4 y[3][VEC_TZ][VEC_TX][QY];
  int next;  // item of the first phase that no warp has taken yet
};
// Work of the first phase: the CTA's rows (QY vectors each, the outer two for
// the y terms only), the z halo's rows, the x halo's.
constexpr int kItemsC = VEC_TZ * VEC_TX * QY, kItemsZ = 4 * VEC_TX * VEC_TY,
              kItemsX = 4 * VEC_TZ * VEC_TY, kItems = kItemsC + kItemsZ + kItemsX;
static_assert(kItemsC % 32 == 0 && kItemsZ % 32 == 0 && kItemsX % 32 == 0, "one kind per warp");
constexpr int EX_THREADS = 2 * VEC_THREADS;  // two threads per vector

__device__ __forceinline__ float4 to4(const Row &r) {
  return make_float4(r.v[0], r.v[1], r.v[2], r.v[3]);
}
__device__ __forceinline__ Row row4(const float4 &t) { return Row{{t.x, t.y, t.z, t.w}}; }

// A term's place: slot, coefficients at half points, source row, target.
struct Term {
  int slot, half;
};

// Q of four cells of a z or x slab row (cf: coefficient rows of n at the row's
// plane), and, for rows that the CTA owns, the memory variables after the
// stage, b (L + G).
template <bool VA, bool OWN>
__device__ __forceinline__ Row q_slab(const float *in, float *out, int k, const VecCell &c,
                                      const float *cf, int n, int half, const Row &G) {
  const float K = cf[(3 * half + CK) * n], a = cf[(3 * half + CA) * n];
  const Row L = ld_psi<VA>(in, k, c);
  Row q;
#pragma unroll
  for (int e = 0; e < VEC; ++e) q.v[e] = c.act[e] ? qpml(G[e], true, L[e], K, a) : 0.f;
  if (OWN) {
    const float b = cf[(3 * half + CB) * n];
    Row r;
#pragma unroll
    for (int e = 0; e < VEC; ++e) r.v[e] = c.act[e] ? b * (L[e] + G[e]) : 0.f;
    st_psi<VA>(out, k, r, c);
  }
  return q;
}
template <bool VA>
__device__ __forceinline__ Row q_slab_y(const float *in, float *out, const Geo &g,
                                        const Pml<VA> &m, const VecCell &c, int half, bool own,
                                        const Row &G) {
  const Row K = coef_y<VA>(g, c, 3 * half + CK), a = coef_y<VA>(g, c, 3 * half + CA);
  const Row L = ld_psi_y(in, g, m, c);
  Row q;
#pragma unroll
  for (int e = 0; e < VEC; ++e) q.v[e] = m.ys[e] ? qpml(G[e], true, L[e], K[e], a[e]) : G[e];
  if (own) {
    const Row b = coef_y<VA>(g, c, 3 * half + CB);
    Row r;
#pragma unroll
    for (int e = 0; e < VEC; ++e) r.v[e] = m.ys[e] ? b[e] * (L[e] + G[e]) : 0.f;
    st_psi_y(out, r, m, g, c);
  }
  return q;
}
// G at the cells that the forward step updates, zero elsewhere (adjoint
// sources may lie outside them).
__device__ __forceinline__ Row masked(const Row &G, const VecCell &c) {
  Row q;
#pragma unroll
  for (int e = 0; e < VEC; ++e) q.v[e] = c.act[e] ? G[e] : 0.f;
  return q;
}

// First phase.  `load(i)` gives the three G of each axis at the vector at
// linear index i: Gs::z, Gs::x, Gs::y (x and z halos use their own three
// only).  V: the velocity stage's slabs.
struct Gs {
  Row z[3], x[3], y[3];
};
template <bool VA, bool V, class Load>
__device__ __forceinline__ void fill_q(QTile &q, const Geo &g, const Psi &lin, const Psi &lout,
                                       int x0, int y0, int z0, const Term tz[3], const Term tx[3],
                                       const Term ty[3], const Load &load) {
  const int lane = vec_thread() & 31;
  for (;;) {
    // 32 items for the warp (the kinds' counts are multiples of 32)
    int it = lane == 0 ? atomicAdd(&q.next, 32) : 0;
    it = __shfl_sync(0xffffffffu, it, 0) + lane;
    if (it >= kItems) break;
    // the item's row and vector relative to the CTA
    int dz, dx, v, kind;
    if (it < kItemsC) {
      const int r = it / QY;
      kind = 0; v = it - r * QY - 1; dz = r / VEC_TX; dx = r % VEC_TX;
    } else if (it < kItemsC + kItemsZ) {
      const int k = it - kItemsC, r = k / VEC_TY, h = r / VEC_TX;
      kind = 1; v = k % VEC_TY; dx = r % VEC_TX; dz = h < 2 ? h - 2 : h + VEC_TZ - 2;
    } else {
      const int k = it - kItemsC - kItemsZ, r = k / VEC_TY, h = r % 4;
      kind = 2; v = k % VEC_TY; dz = r / 4; dx = h < 2 ? h - 2 : h + VEC_TX - 2;
    }
    const int z = z0 + dz, x = x0 + dx, y = y0 + VEC * v;
    const bool in = z >= 2 && z <= g.nz - 3 && x >= 2 && x <= g.nx - 3 && y >= 0 && y <= g.ny - 3;
    const VecCell c = vec_cell(g, z, x, y);
    Gs G{};
    if (in) load(c.i, kind, G);
    const bool own = kind == 0 && v >= 0 && v < VEC_TY;
    if (kind == 1 || own) {
      const bool s = in && slab_s(z, g.nz, g.np);
#pragma unroll
      for (int k = 0; k < 3; ++k) {
        Row r = masked(G.z[k], c);
        const float *p = lin.z + tz[k].slot * g.slab_z;
        float *o = lout.z + tz[k].slot * g.slab_z;
        if (s && kind == 1)
          r = q_slab<VA, false>(p, o, psi_z_idx(g, z, x, y), c, g.cz + z, g.nz, tz[k].half, G.z[k]);
        else if (s)
          r = q_slab<VA, true>(p, o, psi_z_idx(g, z, x, y), c, g.cz + z, g.nz, tz[k].half, G.z[k]);
        q.z[k][dz + 2][dx][v] = to4(r);
      }
    }
    if (kind == 2 || own) {
      const bool s = in && (V ? slab_v(x, g.nx, g.np) : slab_s(x, g.nx, g.np));
#pragma unroll
      for (int k = 0; k < 3; ++k) {
        Row r = masked(G.x[k], c);
        const float *p = lin.x + tx[k].slot * g.slab_x;
        float *o = lout.x + tx[k].slot * g.slab_x;
        if (s && kind == 2)
          r = q_slab<VA, false>(p, o, psi_x_idx(g, z, x, y), c, g.cx + x, g.nx, tx[k].half, G.x[k]);
        else if (s)
          r = q_slab<VA, true>(p, o, psi_x_idx(g, z, x, y), c, g.cx + x, g.nx, tx[k].half, G.x[k]);
        q.x[k][dz][dx + 2][v] = to4(r);
      }
    }
    if (kind == 0) {
      const Pml<VA> m = pml_of<VA>(g, c, V);
      const bool s = in && m.yany;
#pragma unroll
      for (int k = 0; k < 3; ++k) {
        Row r = G.y[k];
        if (s)
          r = q_slab_y(lin.y + ty[k].slot * g.slab_y, lout.y + ty[k].slot * g.slab_y, g, m, c,
                       ty[k].half, own, G.y[k]);
        q.y[k][dz][dx][v + 1] = to4(masked(r, c));
      }
    }
  }
}

// Second phase: differences of the staged Q at the thread's cells.
struct QGather {
  const QTile &q;
  const Geo &g;
  const int tz;
  __device__ __forceinline__ Row z(int k, int d) const {
    return row4(q.z[k][tz + 2 + d][threadIdx.y][threadIdx.x]);
  }
  __device__ __forceinline__ Row x(int k, int d) const {
    return row4(q.x[k][tz][threadIdx.y + 2 + d][threadIdx.x]);
  }
  __device__ __forceinline__ Span y(int k) const {
    const float4 *p = &q.y[k][tz][threadIdx.y][threadIdx.x + 1];
    const float4 l = p[-1], m = p[0], h = p[1];
    return Span{{l.z, l.w, m.x, m.y, m.z, m.w, h.x, h.y}};
  }
  // d -= (D+ or D-) / h along an axis
  __device__ __forceinline__ void zp(Row &d, int k) const {
    const Row a = z(k, -1), b = z(k, 0), h = z(k, 1), l = z(k, 2);
#pragma unroll
    for (int e = 0; e < VEC; ++e) d.v[e] -= dplus(a[e], b[e], h[e], l[e]) * g.idz;
  }
  __device__ __forceinline__ void zm(Row &d, int k) const {
    const Row a = z(k, -2), b = z(k, -1), h = z(k, 0), l = z(k, 1);
#pragma unroll
    for (int e = 0; e < VEC; ++e) d.v[e] -= dminus(a[e], b[e], h[e], l[e]) * g.idz;
  }
  __device__ __forceinline__ void xp(Row &d, int k) const {
    const Row a = x(k, -1), b = x(k, 0), h = x(k, 1), l = x(k, 2);
#pragma unroll
    for (int e = 0; e < VEC; ++e) d.v[e] -= dplus(a[e], b[e], h[e], l[e]) * g.idx;
  }
  __device__ __forceinline__ void xm(Row &d, int k) const {
    const Row a = x(k, -2), b = x(k, -1), h = x(k, 0), l = x(k, 1);
#pragma unroll
    for (int e = 0; e < VEC; ++e) d.v[e] -= dminus(a[e], b[e], h[e], l[e]) * g.idx;
  }
  __device__ __forceinline__ void yp(Row &d, int k) const {
    const Span w = y(k);
#pragma unroll
    for (int e = 0; e < VEC; ++e) d.v[e] -= dplus(w(e, -1), w(e, 0), w(e, 1), w(e, 2)) * g.idy;
  }
  __device__ __forceinline__ void ym(Row &d, int k) const {
    const Span w = y(k);
#pragma unroll
    for (int e = 0; e < VEC; ++e) d.v[e] -= dminus(w(e, -2), w(e, -1), w(e, 0), w(e, 1)) * g.idy;
  }
};

// Forward differences of the images, times 1/h.
__device__ __forceinline__ Row diff_p(const float *q, int s, float ih) {
  const Row a = ld_row(q - s), b = ld_row(q), d = ld_row(q + s), h = ld_row(q + 2 * s);
  Row r;
#pragma unroll
  for (int e = 0; e < VEC; ++e) r.v[e] = dplus(a[e], b[e], d[e], h[e]) * ih;
  return r;
}
__device__ __forceinline__ Row diff_m(const float *q, int s, float ih) {
  const Row a = ld_row(q - 2 * s), b = ld_row(q - s), d = ld_row(q), h = ld_row(q + s);
  Row r;
#pragma unroll
  for (int e = 0; e < VEC; ++e) r.v[e] = dminus(a[e], b[e], d[e], h[e]) * ih;
  return r;
}
__device__ __forceinline__ Row diff_py(const float *q, const VecCell &c, float ih) {
  const Row b = ld_row(q);
  const Span w = ld_span(q, b, c);
  Row r;
#pragma unroll
  for (int e = 0; e < VEC; ++e) r.v[e] = dplus(w(e, -1), b[e], w(e, 1), w(e, 2)) * ih;
  return r;
}
__device__ __forceinline__ Row diff_my(const float *q, const VecCell &c, float ih) {
  const Row b = ld_row(q);
  const Span w = ld_span(q, b, c);
  Row r;
#pragma unroll
  for (int e = 0; e < VEC; ++e) r.v[e] = dminus(w(e, -2), w(e, -1), b[e], w(e, 1)) * ih;
  return r;
}

}  // namespace

template <bool VA, int MINB>
__global__ void __launch_bounds__(EX_THREADS, MINB) k_adj_stress_vec(ExactArgs A) {
  const Geo &g = A.g;
  __shared__ QTile q;
  const int z0 = 2 + blockIdx.z * VEC_TZ, x0 = 2 + blockIdx.y * VEC_TX,
            y0 = VEC * blockIdx.x * VEC_TY;
  const int tz = threadIdx.z % VEC_TZ, part = threadIdx.z / VEC_TZ;
  const int z = z0 + tz, x = x0 + threadIdx.y, y = y0 + VEC * threadIdx.x;
  const int nz = g.nz, nx = g.nx;
  const float dt = g.dt, idz = g.idz, idx = g.idx, idy = g.idy;
  if (threadIdx.x + threadIdx.y + threadIdx.z == 0) q.next = 0;
  __syncthreads();
  vec_begin();
  const bool in = z <= nz - 3 && x <= nx - 3 && y <= g.ny - 3;
  const VecCell c = vec_cell(g, z, x, y);
  const int i = c.i;
  if (g.far && part == 0 && in)  // read after the barrier
    for (const float *p : {A.a.vz, A.a.vx, A.a.vy}) prefetch_row(p + i);
  if (part == 1 && in && A.g0) {
    const Pml<VA> m = pml_of<VA>(g, c, false);
    const float *azz = A.a.szz + i, *axx = A.a.sxx + i, *ayy = A.a.syy + i;
    const float *axz = A.a.sxz + i, *axy = A.a.sxy + i, *ayz = A.a.syz + i;
    // ---- images from the forward velocities of the same step: the modified
    // derivatives d / K + (b psi + a d)
    auto mod = [&](Row &d, float Ki, float a, float b, const Row &p) {
#pragma unroll
      for (int e = 0; e < VEC; ++e) d.v[e] = d[e] * Ki + (b * p[e] + a * d[e]);
    };
    auto mod_z = [&](Row &d, int slot, int half) {
      if (!m.zs) return;
      const float *cf = g.cz + 3 * half * nz + z;
      mod(d, cf[CK * nz], cf[CA * nz], cf[CB * nz], ld_psi<VA>(A.ps.z, slot, g.slab_z, m.kz, c));
    };
    auto mod_x = [&](Row &d, int slot, int half) {
      if (!m.xs) return;
      const float *cf = g.cx + 3 * half * nx + x;
      mod(d, cf[CK * nx], cf[CA * nx], cf[CB * nx], ld_psi<VA>(A.ps.x, slot, g.slab_x, m.kx, c));
    };
    auto mod_y = [&](Row &d, int slot, int half) {
      if (!m.yany) return;
      const Row K = coef_y<VA>(g, c, 3 * half + CK), a = coef_y<VA>(g, c, 3 * half + CA),
                b = coef_y<VA>(g, c, 3 * half + CB), p = ld_psi_y(A.ps.y, slot, g, m, c);
#pragma unroll
      for (int e = 0; e < VEC; ++e)
        if (m.ys[e]) d.v[e] = d[e] * K[e] + (b[e] * p[e] + a[e] * d[e]);
    };
    const VecCell cf = vec_cell(g, z, x, y, A.pitch_f);  // in the forward state
    const int fx = A.pitch_f, fz = nx * fx;
    const float *vz = A.f.vz + cf.i, *vx = A.f.vx + cf.i, *vy = A.f.vy + cf.i;
    Row gm;
    {
      Row ez = diff_m(vz, fz, idz), ex = diff_m(vx, fx, idx), ey = diff_my(vy, cf, idy);
      mod_z(ez, PSI_VA, 0);
      mod_x(ex, PSI_VA, 0);
      mod_y(ey, PSI_VA, 0);
      const Row pz = ld_row(azz), px = ld_row(axx), py = ld_row(ayy);
      Row gl = ld_row(A.g0 + i);
#pragma unroll
      for (int e = 0; e < VEC; ++e) {
        if (c.act[e]) gl.v[e] += (pz[e] + px[e] + py[e]) * (ez[e] + ex[e] + ey[e]) * dt;
        gm.v[e] = 2.0f * (pz[e] * ez[e] + px[e] * ex[e] + py[e] * ey[e]);
      }
      st_row(A.g0 + i, gl);
    }
    auto share = [&](const float *s, const Row &d0, const Row &d1) {
      const Row p = ld_row(s);
#pragma unroll
      for (int e = 0; e < VEC; ++e) gm.v[e] += p[e] * (d0[e] + d1[e]);
    };
    {
      Row d0 = diff_p(vx, fz, idz), d1 = diff_p(vz, fx, idx);
      mod_z(d0, PSI_VB1, 1);
      mod_x(d1, PSI_VB1, 1);
      share(axz, d0, d1);
    }
    {
      Row d0 = diff_py(vx, cf, idy), d1 = diff_p(vy, fx, idx);
      mod_y(d0, PSI_VB2, 1);
      mod_x(d1, PSI_VB2, 1);
      share(axy, d0, d1);
    }
    {
      Row d0 = diff_p(vy, fz, idz), d1 = diff_py(vz, cf, idy);
      mod_z(d0, PSI_VB2, 1);
      mod_y(d1, PSI_VB1, 1);
      share(ayz, d0, d1);
    }
    Row g1 = ld_row(A.g1 + i);
#pragma unroll
    for (int e = 0; e < VEC; ++e)
      if (c.act[e]) g1.v[e] += gm[e] * dt;
    st_row(A.g1 + i, g1);
  }
  {
    // z: vz <- ez, vx <- xz, vy <- yz; x: vx <- ex, vz <- xz, vy <- xy;
    // y: vy <- ey, vz <- yz, vx <- xy
    constexpr Term t[3] = {{PSI_VA, 0}, {PSI_VB1, 1}, {PSI_VB2, 1}};
    fill_q<VA, false>(q, g, A.lin, A.lout, x0, y0, z0, t, t, t, [&](int i, int kind, Gs &G) {
      const Row l = ld_row(A.lam + i), u = ld_row(A.mu + i);
      const Row zz = ld_row(A.a.szz + i), xx = ld_row(A.a.sxx + i), yy = ld_row(A.a.syy + i);
      Row xz{}, xy{}, yz{};
      xz = ld_row(A.a.sxz + i);
      if (kind != 1) xy = ld_row(A.a.sxy + i);
      if (kind != 2) yz = ld_row(A.a.syz + i);
#pragma unroll
      for (int e = 0; e < VEC; ++e) {
        const float l2u = l[e] + 2.0f * u[e];
        G.z[0].v[e] = (l2u * zz[e] + l[e] * (xx[e] + yy[e])) * dt;
        G.x[0].v[e] = (l2u * xx[e] + l[e] * (zz[e] + yy[e])) * dt;
        G.y[0].v[e] = (l2u * yy[e] + l[e] * (zz[e] + xx[e])) * dt;
        G.z[1].v[e] = G.x[1].v[e] = u[e] * xz[e] * dt;
        G.x[2].v[e] = G.y[2].v[e] = u[e] * xy[e] * dt;
        G.z[2].v[e] = G.y[1].v[e] = u[e] * yz[e] * dt;
      }
    });
  }
  __syncthreads();
  if (!in) return;
  const QGather Q{q, g, tz};
  auto finish = [&](float *dst, const Row &d) {
    Row n = ld_row(dst);
#pragma unroll
    for (int e = 0; e < VEC; ++e)
      if (c.act[e]) n.v[e] += d[e];
    st_row(dst, n);
  };
  if (part == 0) {
    {
      Row d{};
      Q.zp(d, 0); Q.xm(d, 1); Q.ym(d, 1);
      finish(A.a.vz + i, d);
    }
  } else {
    {
      Row d{};
      Q.xp(d, 0); Q.zm(d, 1); Q.ym(d, 2);
      finish(A.a.vx + i, d);
    }
    {
      Row d{};
      Q.yp(d, 0); Q.xm(d, 2); Q.zm(d, 2);
      finish(A.a.vy + i, d);
    }
  }
}

template <bool VA, int MINB>
__global__ void __launch_bounds__(EX_THREADS, MINB) k_adj_velocity_vec(ExactArgs A) {
  const Geo &g = A.g;
  __shared__ QTile q;
  const int z0 = 2 + blockIdx.z * VEC_TZ, x0 = 2 + blockIdx.y * VEC_TX,
            y0 = VEC * blockIdx.x * VEC_TY;
  const int tz = threadIdx.z % VEC_TZ, part = threadIdx.z / VEC_TZ;
  const int z = z0 + tz, x = x0 + threadIdx.y, y = y0 + VEC * threadIdx.x;
  const int nz = g.nz, nx = g.nx;
  const float dt = g.dt, idz = g.idz, idx = g.idx, idy = g.idy;
  if (threadIdx.x + threadIdx.y + threadIdx.z == 0) q.next = 0;
  __syncthreads();
  vec_begin();
  const bool in = z <= nz - 3 && x <= nx - 3 && y <= g.ny - 3;
  const VecCell c = vec_cell(g, z, x, y);
  const int i = c.i;
  if (g.far && part == 0 && in)  // read after the barrier
    for (const float *p : {A.a.szz, A.a.sxx, A.a.syy, A.a.sxz, A.a.sxy, A.a.syz}) prefetch_row(p + i);
  if (part == 1 && in && A.g0) {
    const Pml<VA> m = pml_of<VA>(g, c, true);
    const float *avz = A.a.vz + i, *avx = A.a.vx + i, *avy = A.a.vy + i;
    // ---- buoyancy image from the forward stresses of the same step: modified
    // derivatives d / K + psi (the memory variables are the step's new ones)
    auto mod_z = [&](Row &d, int slot, int half) {
      if (!m.zs) return;
      const float Ki = g.cz[(3 * half + CK) * nz + z];
      const Row p = ld_psi<VA>(A.ps.z, slot, g.slab_z, m.kz, c);
#pragma unroll
      for (int e = 0; e < VEC; ++e) d.v[e] = d[e] * Ki + p[e];
    };
    auto mod_x = [&](Row &d, int slot, int half) {
      if (!m.xs) return;
      const float Ki = g.cx[(3 * half + CK) * nx + x];
      const Row p = ld_psi<VA>(A.ps.x, slot, g.slab_x, m.kx, c);
#pragma unroll
      for (int e = 0; e < VEC; ++e) d.v[e] = d[e] * Ki + p[e];
    };
    auto mod_y = [&](Row &d, int slot, int half) {
      if (!m.yany) return;
      const Row K = coef_y<VA>(g, c, 3 * half + CK), p = ld_psi_y(A.ps.y, slot, g, m, c);
#pragma unroll
      for (int e = 0; e < VEC; ++e)
        if (m.ys[e]) d.v[e] = d[e] * K[e] + p[e];
    };
    const VecCell cf = vec_cell(g, z, x, y, A.pitch_f);  // in the forward state
    const int fx = A.pitch_f, fz = nx * fx;
    const float *szz = A.f.szz + cf.i, *sxx = A.f.sxx + cf.i, *syy = A.f.syy + cf.i;
    const float *sxz = A.f.sxz + cf.i, *sxy = A.f.sxy + cf.i, *syz = A.f.syz + cf.i;
    Row im;
    {
      Row d0 = diff_p(szz, fz, idz), d1 = diff_m(sxz, fx, idx), d2 = diff_my(syz, cf, idy);
      mod_z(d0, PSI_SAA, 1);
      mod_x(d1, PSI_SAB1, 0);
      mod_y(d2, PSI_SAB1, 0);
      const Row v = ld_row(avz);
#pragma unroll
      for (int e = 0; e < VEC; ++e) im.v[e] = v[e] * (d0[e] + d1[e] + d2[e]);
    }
    {
      Row d0 = diff_m(sxz, fz, idz), d1 = diff_p(sxx, fx, idx), d2 = diff_my(sxy, cf, idy);
      mod_z(d0, PSI_SAB1, 0);
      mod_x(d1, PSI_SAA, 1);
      mod_y(d2, PSI_SAB2, 0);
      const Row v = ld_row(avx);
#pragma unroll
      for (int e = 0; e < VEC; ++e) im.v[e] += v[e] * (d0[e] + d1[e] + d2[e]);
    }
    {
      Row d0 = diff_m(syz, fz, idz), d1, d2 = diff_py(syy, cf, idy);
      const Row s0 = ld_row(sxy), s1 = ld_row(sxy - fx), s2 = ld_row(sxy - 2 * fx);
#pragma unroll
      for (int e = 0; e < VEC; ++e) d1.v[e] = dquirk(s2[e], s1[e], s0[e]) * idx;
      mod_z(d0, PSI_SAB2, 0);
      mod_x(d1, PSI_SAB2, 0);
      mod_y(d2, PSI_SAA, 1);
      const Row v = ld_row(avy);
#pragma unroll
      for (int e = 0; e < VEC; ++e) im.v[e] += v[e] * (d0[e] + d1[e] + d2[e]);
    }
    Row g0 = ld_row(A.g0 + i);
#pragma unroll
    for (int e = 0; e < VEC; ++e)
      if (c.act[e]) g0.v[e] += im[e] * dt;
    st_row(A.g0 + i, g0);
  }
  {
    // in the order vz, vx, vy: the stresses szz, sxz, syz (z), sxz, sxx, sxy
    // (x) and syz, sxy, syy (y) that each reads
    constexpr Term tz[3] = {{PSI_SAA, 1}, {PSI_SAB1, 0}, {PSI_SAB2, 0}};
    constexpr Term tx[3] = {{PSI_SAB1, 0}, {PSI_SAA, 1}, {PSI_SAB2, 0}};
    constexpr Term ty[3] = {{PSI_SAB1, 0}, {PSI_SAB2, 0}, {PSI_SAA, 1}};
    fill_q<VA, true>(q, g, A.lin, A.lout, x0, y0, z0, tz, tx, ty, [&](int i, int, Gs &G) {
      const Row b = ld_row(A.buoy + i), vz = ld_row(A.a.vz + i), vx = ld_row(A.a.vx + i),
                vy = ld_row(A.a.vy + i);
#pragma unroll
      for (int e = 0; e < VEC; ++e) {
        const float s = b[e] * dt;
        G.z[0].v[e] = G.x[0].v[e] = G.y[0].v[e] = vz[e] * s;
        G.z[1].v[e] = G.x[1].v[e] = G.y[1].v[e] = vx[e] * s;
        G.z[2].v[e] = G.x[2].v[e] = G.y[2].v[e] = vy[e] * s;
      }
    });
  }
  __syncthreads();
  if (!in) return;
  const QGather Q{q, g, tz};
  auto finish = [&](float *dst, const Row &d) {
    Row n = ld_row(dst);
#pragma unroll
    for (int e = 0; e < VEC; ++e)
      if (c.act[e]) n.v[e] += d[e];
    st_row(dst, n);
  };
  if (part == 0) {
    {
      Row d{};
      Q.zm(d, 0);
      finish(A.a.szz + i, d);
    }
    {
      Row d{};
      Q.xm(d, 1);
      finish(A.a.sxx + i, d);
    }
    {
      Row d{};
      Q.xp(d, 0); Q.zp(d, 1);
      finish(A.a.sxz + i, d);
    }
  } else {
    {
      Row d{};
      Q.ym(d, 2);
      finish(A.a.syy + i, d);
    }
    {
      Row d{};
      Q.yp(d, 0); Q.zp(d, 2);
      finish(A.a.syz + i, d);
    }
    {  // sxy, with the transpose of the quirk-Q1 difference
      Row d{};
      Q.yp(d, 1);
      const Row q0 = Q.x(2, 0), q1 = Q.x(2, 1), q2 = Q.x(2, 2);
  #pragma unroll
      for (int e = 0; e < VEC; ++e) d.v[e] += dq_t(q0[e], q1[e], q2[e]) * idx;
      finish(A.a.sxy + i, d);
    }
  }
}

// Resident CTAs per SM (33 KB of shared memory each).  At 120^3 (us, event
// overhead of 6 in all) the stress stage takes 82 / 72 / 72 and the velocity
// stage 82 / 72 / 66 with 3 / 4 / 5 CTAs; with one thread per vector for both
// kinds of work, 6 CTAs of 128 threads, 87 and 80.  The single-cell memory
// variables need more than the 48 registers of 5 CTAs.
void launch_adj_stress_vec(cudaStream_t st, const ExactArgs &A) {
  auto k = psi_vectors(A.g) ? k_adj_stress_vec<true, 4> : k_adj_stress_vec<false, 4>;
  vec_launch(k, vec_grid(A.g), 2 * VEC_TZ, true, st, A);
}

void launch_adj_velocity_vec(cudaStream_t st, const ExactArgs &A) {
  auto k = psi_vectors(A.g) ? k_adj_velocity_vec<true, 5> : k_adj_velocity_vec<false, 4>;
  vec_launch(k, vec_grid(A.g), 2 * VEC_TZ, true, st, A);
}

}  // namespace efwi
