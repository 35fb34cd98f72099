// Reverse sweep of the reference gradient, one thread per four cells
// (efwi_vec.cuh); the same arithmetic and fusion as efwi_rev.cu (K1 =
// velocity(rev) + velocity_adj, K2 = add_source(sub) + stress(rev) +
// stress_adj).  Restated reference kernels: velocity.cu:102-131,
// stress.cu:103-135, velocity_adj.cu:59-144, stress_adj.cu:52-142.
//
// Fused epilogues (efwi_fuse.cuh): K1 restores the reverse velocities at
// the boundary-shell points (to_bnd of the velocities) and adds the adjoint
// source at the receiver cells to the adjoint velocities (res_injection);
// K2 restores the reverse stresses at the shell points.
//
// As in the forward kernels every output is formed on its own, from rows that
// L1 serves again, so that few values are live.
#include "efwi_common.cuh"
#include "efwi_fuse.cuh"
#include "efwi_kernels.h"
#include "efwi_vec.cuh"

namespace efwi {

namespace {

// Differences of four cells times 1/h; q: the thread's cell, s: the axis's
// stride.  p / py: forward difference (y: along the vector), m / my:
// backward; np, nm, npy, nmy: negated, the adjoint's.
struct Diff {
  const VecCell &c;
#define EFWI_DIFF(NAME, SIGN)                                                                     \
  __device__ __forceinline__ Row NAME##p(const float *q, int s, float ih) const {                 \
    const Row a = ld_row(q - s), b = ld_row(q), d = ld_row(q + s), h = ld_row(q + 2 * s);         \
    Row r;                                                                                        \
    _Pragma("unroll") for (int e = 0; e < VEC; ++e) r.v[e] = __fmul_rn(SIGN dplus(a[e], b[e], d[e], h[e]), ih); \
    return r;                                                                                     \
  }                                                                                               \
  __device__ __forceinline__ Row NAME##m(const float *q, int s, float ih) const {                 \
    const Row a = ld_row(q - 2 * s), b = ld_row(q - s), d = ld_row(q), h = ld_row(q + s);         \
    Row r;                                                                                        \
    _Pragma("unroll") for (int e = 0; e < VEC; ++e) r.v[e] = __fmul_rn(SIGN dminus(a[e], b[e], d[e], h[e]), ih); \
    return r;                                                                                     \
  }                                                                                               \
  __device__ __forceinline__ Row NAME##py(const float *q, float ih) const {                       \
    const Row b = ld_row(q);                                                                      \
    const Span w = ld_span(q, b, c);                                                              \
    Row r;                                                                                        \
    _Pragma("unroll") for (int e = 0; e < VEC; ++e)                                               \
      r.v[e] = __fmul_rn(SIGN dplus(w(e, -1), b[e], w(e, 1), w(e, 2)), ih);                                 \
    return r;                                                                                     \
  }                                                                                               \
  __device__ __forceinline__ Row NAME##my(const float *q, float ih) const {                       \
    const Row b = ld_row(q);                                                                      \
    const Span w = ld_span(q, b, c);                                                              \
    Row r;                                                                                        \
    _Pragma("unroll") for (int e = 0; e < VEC; ++e)                                               \
      r.v[e] = __fmul_rn(SIGN dminus(w(e, -2), w(e, -1), b[e], w(e, 1)), ih);                               \
    return r;                                                                                     \
  }
  EFWI_DIFF(, )
  EFWI_DIFF(n, -)
#undef EFWI_DIFF
};

// Cells of the vector inside [np, n-1-np]^3, where the reverse update runs.
__device__ __forceinline__ bool inner_cells(const Geo &g, const VecCell &c, bool in[VEC]) {
  const bool zx = c.z >= g.np && c.z <= g.nz - 1 - g.np && c.x >= g.np && c.x <= g.nx - 1 - g.np;
  bool any = false;
#pragma unroll
  for (int e = 0; e < VEC; ++e) {
    in[e] = zx && c.act[e] && c.y + e >= g.np && c.y + e <= g.ny - 1 - g.np;
    any = any || in[e];
  }
  return any;
}

}  // namespace

template <bool VA, int MINB>
__global__ void __launch_bounds__(VEC_THREADS, MINB)
k_rev_velocity_vec(Geo g, Fields f, Fields a, Psi ps, const float *__restrict__ lam,
                   const float *__restrict__ mu, const float *__restrict__ buoy, float *grho,
                   int do_rev, int do_adj, ShellMap shell, RecFuse inj) {
  const int z = 2 + blockIdx.z * VEC_TZ + threadIdx.z;
  const int x = 2 + blockIdx.y * VEC_TX + threadIdx.y;
  const int y = VEC * (blockIdx.x * VEC_TY + threadIdx.x);
  const int nz = g.nz, nx = g.nx, ny = g.ny;
  if (z > nz - 3 || x > nx - 3 || y > ny - 3) return;
  const VecCell c = vec_cell(g, z, x, y);
  const Diff D{c};
  const int i = c.i, sz = (int)g.sz, sx = g.sx;
  const float dt = g.dt, idz = g.idz, idx = g.idx, idy = g.idy;
  __shared__ float4 stash[10 * VEC_THREADS];
  Stash<VEC_THREADS> own{stash + vec_thread()};
  enum { VZ, VX, VY, AVZ, AVX, AVY, BU, LA, MU, GR };
  own.fetch(AVZ, a.vz + i); own.fetch(AVX, a.vx + i); own.fetch(AVY, a.vy + i);
  own.fetch(BU, buoy + i);
  if (do_adj) { own.fetch(LA, lam + i); own.fetch(MU, mu + i); }
  const Pml<VA> m = pml_of<VA>(g, c, false);
  if (do_adj && g.far)
    for (const float *p : {a.szz, a.sxx, a.syy, a.sxz, a.sxy, a.syz}) prefetch_row(p + i);
  bool in[VEC];
  const bool any_in = do_rev && inner_cells(g, c, in);
  if (any_in && g.far)
    for (const float *p : {f.sxx, f.sxy, f.syy}) prefetch_row(p + i);
  // to_bnd: the shell points take the stored velocities of the step
  int sk[VEC] = {-1, -1, -1, -1};
  bool any_sk = false;
  if (do_rev && shell.rows) {
    const int srow = shell.rows[z * nx + x];
    if (srow >= 0) any_sk = shell_cells(shell, srow, c, sk);
  }
  const int rmap = do_adj ? receiver_map(inj.a, nz, 0, z) : -1;
  if (any_in || any_sk) {
    own.fetch(VZ, f.vz + i); own.fetch(VX, f.vx + i); own.fetch(VY, f.vy + i);
    if (any_in) own.fetch(GR, grho + i);
  }
  vec_begin();  // up to here: nothing that the stress kernel writes
  if (any_in || any_sk) {
    Row gi{};
    // reverse update of one velocity and its share of the rho image (img3)
    auto reverse = [&](int r, int ra, int q, float *dst, const Row &d) {
      Row n = own.get(r);
      const Row b = own.get(BU), av = own.get(ra);
#pragma unroll
      for (int e = 0; e < VEC; ++e) {
        const float nb2 = -(b[e] * b[e]);
        if (any_in && in[e]) {
          n.v[e] = undo(n[e], d[e], b[e], dt);
          const float p = __fmul_rn(__fmul_rn(av[e], d[e]), dt);
          gi.v[e] = r == VZ ? p : r == VX ? __fmaf_rn(gi[e], nb2, __fmul_rn(p, nb2))
                                          : __fmaf_rn(p, nb2, gi[e]);
        }
        if (sk[e] >= 0) n.v[e] = shell.store[(size_t)q * shell.npts + sk[e]];
      }
      st_row(dst, n);
    };
    Row d{};
    if (any_in) {
      const Row d0 = D.p(f.szz + i, sz, 1.f), d1 = D.m(f.sxz + i, sx, 1.f), d2 = D.my(f.syz + i, 1.f);
#pragma unroll
      for (int e = 0; e < VEC; ++e) d.v[e] = sum3d(d0[e], idz, d1[e], idx, d2[e], idy);
    }
    own.wait();
    reverse(VZ, AVZ, 6, f.vz + i, d);
    if (any_in) {
      const Row d0 = D.m(f.sxz + i, sz, 1.f), d1 = D.p(f.sxx + i, sx, 1.f), d2 = D.my(f.sxy + i, 1.f);
#pragma unroll
      for (int e = 0; e < VEC; ++e) d.v[e] = sum3d(d0[e], idz, d1[e], idx, d2[e], idy);
    }
    reverse(VX, AVX, 7, f.vx + i, d);
    if (any_in) {
      const Row d0 = D.m(f.syz + i, sz, 1.f), d2 = D.py(f.syy + i, 1.f);
      const Row m0 = ld_row(f.sxy + i), m1 = ld_row(f.sxy + i - sx), m2 = ld_row(f.sxy + i - 2 * sx);
#pragma unroll
      for (int e = 0; e < VEC; ++e)
        d.v[e] = sum3d(d0[e], idz, dquirk(m2[e], m1[e], m0[e]), idx, d2[e], idy);
    }
    reverse(VY, AVY, 8, f.vy + i, d);
    if (any_in) {
      Row gr = own.get(GR);
#pragma unroll
      for (int e = 0; e < VEC; ++e)
        if (in[e]) gr.v[e] = __fadd_rn(gr[e], -gi[e]);
      st_row(grho + i, gr);
    }
  }
  if (!do_adj) { own.wait(); return; }

  const PsiGather<VA> G{g, c, m};
  float *pz = ps.z, *px = ps.x, *py = ps.y;
  const long long lz = g.slab_z, lx = g.slab_x, ly = g.slab_y;
  auto cfz = [&](int k, float out) { return m.zs ? g.cz[k * nz + z] : out; };
  auto cfx = [&](int k, float out) { return m.xs ? g.cx[k * nx + x] : out; };
  auto cfy = [&](int k, float out) { return m.yany ? coef_y<VA>(g, c, k) : fill(out); };
  // the memory variables that one new adjoint velocity feeds
  auto feed = [&](const Row &v, const Row &b, int slx, int bx, int slz, int bz, int sly) {
    Row add;
#pragma unroll
    for (int e = 0; e < VEC; ++e) add.v[e] = __fmul_rn(b[e], v[e]);
    if (m.xs && slx == PSI_SAB1)
      mem_row<VA, true>(px + slx * lx, m.kx, c, g.cx[bx * nx + x], add, dt);
    if (m.xs && slx != PSI_SAB1) mem_row<VA>(px + slx * lx, m.kx, c, g.cx[bx * nx + x], add, dt);
    if (m.zs) mem_row<VA>(pz + slz * lz, m.kz, c, g.cz[bz * nz + z], add, dt);
    if (m.yany) mem_row_y(py + sly * ly, g, m, c, coef_y<VA>(g, c, CB), add, dt);
  };
  Row nax, naz, nay;
  own.wait();
  {  // adjoint vx
    Row acc;
    {
      const Row s0 = D.np(a.szz + i, sx, idx), s1 = D.np(a.sxx + i, sx, idx), s2 = D.np(a.syy + i, sx, idx);
      const Row t0 = D.nm(a.sxz + i, sz, idz), t1 = D.nmy(a.sxy + i, idy);
      const float K = cfx(CK, 1.f), Kz = cfz(CKH, 1.f);
      const Row Ky = cfy(CKH, 1.f), l = own.get(LA), u = own.get(MU);
#pragma unroll
      for (int e = 0; e < VEC; ++e) {
        const float l2u = l[e] + 2.0f * u[e];
        acc.v[e] = add4(0.f, l2u, s1[e], K, dt);
        acc.v[e] = add4(acc[e], l[e], s0[e], K, dt);
        acc.v[e] = add4(acc[e], l[e], s2[e], K, dt);
        acc.v[e] = add4(acc[e], u[e], Kz, t0[e], dt);
        acc.v[e] = add4(acc[e], u[e], Ky[e], t1[e], dt);
      }
    }
    auto gather = [&](float k, const Row &q) {
#pragma unroll
      for (int e = 0; e < VEC; ++e) acc.v[e] = __fmaf_rn(k, q[e], acc[e]);
    };
    if (m.xs) gather(cfx(CA, 0.f), G.dpx(px + PSI_VA * lx));
    if (m.zs) gather(cfz(CAH, 0.f), G.dmz(pz + PSI_VB1 * lz));
    if (m.yany) {
      const Row k = coef_y<VA>(g, c, CAH), q = G.dmy(py + PSI_VB2 * ly);
#pragma unroll
      for (int e = 0; e < VEC; ++e)
        if (m.ys[e]) acc.v[e] = __fmaf_rn(k[e], q[e], acc[e]);
    }
    const Row o = own.get(AVX), b = own.get(BU);
#pragma unroll
    for (int e = 0; e < VEC; ++e) nax.v[e] = c.act[e] ? __fadd_rn(o[e], acc[e]) : o[e];
    feed(nax, b, PSI_SAA, CBH, PSI_SAB1, CB, PSI_SAB2);
  }
  {  // adjoint vz
    Row acc;
    {
      const Row s0 = D.np(a.szz + i, sz, idz), s1 = D.np(a.sxx + i, sz, idz), s2 = D.np(a.syy + i, sz, idz);
      const Row t0 = D.nm(a.sxz + i, sx, idx), t1 = D.nmy(a.syz + i, idy);
      const float K = cfz(CK, 1.f), Kx = cfx(CKH, 1.f);
      const Row Ky = cfy(CKH, 1.f), l = own.get(LA), u = own.get(MU);
#pragma unroll
      for (int e = 0; e < VEC; ++e) {
        const float l2u = l[e] + 2.0f * u[e];
        acc.v[e] = add4(0.f, l2u, s0[e], K, dt);
        acc.v[e] = add4(acc[e], l[e], s1[e], K, dt);
        acc.v[e] = add4(acc[e], l[e], s2[e], K, dt);
        acc.v[e] = add4(acc[e], u[e], Ky[e], t1[e], dt);
        acc.v[e] = add4(acc[e], u[e], Kx, t0[e], dt);
      }
    }
    auto gather = [&](float k, const Row &q) {
#pragma unroll
      for (int e = 0; e < VEC; ++e) acc.v[e] = __fmaf_rn(k, q[e], acc[e]);
    };
    if (m.zs) gather(cfz(CA, 0.f), G.dpz(pz + PSI_VA * lz));
    if (m.yany) {
      const Row k = coef_y<VA>(g, c, CAH), q = G.dmy(py + PSI_VB1 * ly);
#pragma unroll
      for (int e = 0; e < VEC; ++e)
        if (m.ys[e]) acc.v[e] = __fmaf_rn(k[e], q[e], acc[e]);
    }
    if (m.xs) gather(cfx(CAH, 0.f), G.dmx(px + PSI_VB1 * lx));
    const Row o = own.get(AVZ), b = own.get(BU);
#pragma unroll
    for (int e = 0; e < VEC; ++e) naz.v[e] = c.act[e] ? __fadd_rn(o[e], acc[e]) : o[e];
    feed(naz, b, PSI_SAB1, CB, PSI_SAA, CBH, PSI_SAB1);
  }
  {  // adjoint vy
    Row acc;
    {
      const Row s0 = D.npy(a.szz + i, idy), s1 = D.npy(a.sxx + i, idy), s2 = D.npy(a.syy + i, idy);
      const Row t0 = D.nm(a.sxy + i, sx, idx), t1 = D.nm(a.syz + i, sz, idz);
      const float Kx = cfx(CKH, 1.f), Kz = cfz(CKH, 1.f);
      const Row K = cfy(CK, 1.f), l = own.get(LA), u = own.get(MU);
#pragma unroll
      for (int e = 0; e < VEC; ++e) {
        const float l2u = l[e] + 2.0f * u[e];
        acc.v[e] = add4(0.f, l[e], s1[e], K[e], dt);
        acc.v[e] = add4(acc[e], l2u, s2[e], K[e], dt);
        acc.v[e] = add4(acc[e], l[e], s0[e], K[e], dt);
        acc.v[e] = add4(acc[e], u[e], Kx, t0[e], dt);
        acc.v[e] = add4(acc[e], u[e], Kz, t1[e], dt);
      }
    }
    auto gather = [&](float k, const Row &q) {
#pragma unroll
      for (int e = 0; e < VEC; ++e) acc.v[e] = __fmaf_rn(k, q[e], acc[e]);
    };
    if (m.yany) {
      const Row k = coef_y<VA>(g, c, CA), q = G.dpy(py + PSI_VA * ly);
#pragma unroll
      for (int e = 0; e < VEC; ++e)
        if (m.ys[e]) acc.v[e] = __fmaf_rn(k[e], q[e], acc[e]);
    }
    if (m.xs) gather(cfx(CAH, 0.f), G.dmx(px + PSI_VB2 * lx));
    if (m.zs) gather(cfz(CAH, 0.f), G.dmz(pz + PSI_VB2 * lz));
    const Row o = own.get(AVY), b = own.get(BU);
#pragma unroll
    for (int e = 0; e < VEC; ++e) nay.v[e] = c.act[e] ? __fadd_rn(o[e], acc[e]) : o[e];
    feed(nay, b, PSI_SAB2, CB, PSI_SAB2, CBH, PSI_SAA);
  }
  if (rmap >= 0) {  // res_injection after the adjoint update
    const Row entry = ld_row(receiver_row(inj.a, rmap, g, c));
#pragma unroll
    for (int e = 0; e < VEC; ++e) {
      const int u = __float_as_int(entry[e]);
      if (c.act[e] && u != -1)
        inject_cell(inj.a, inj.tm, inj.it, u, naz.v[e], nax.v[e], nay.v[e]);
    }
  }
  st_row(a.vx + i, nax); st_row(a.vz + i, naz); st_row(a.vy + i, nay);
}

template <bool VA, int MINB>
__global__ void __launch_bounds__(VEC_THREADS, MINB)
k_rev_stress_vec(Geo g, Fields f, Fields a, Psi ps, const float *__restrict__ lam,
                 const float *__restrict__ mu, const float *__restrict__ buoy, float *glam,
                 float *gmu, int do_rev, int do_adj, SrcArgs src, ShellMap shell) {
  const int z = 2 + blockIdx.z * VEC_TZ + threadIdx.z;
  const int x = 2 + blockIdx.y * VEC_TX + threadIdx.y;
  const int y = VEC * (blockIdx.x * VEC_TY + threadIdx.x);
  const int nz = g.nz, nx = g.nx, ny = g.ny;
  if (z > nz - 3 || x > nx - 3 || y > ny - 3) return;
  const VecCell c = vec_cell(g, z, x, y);
  const Diff D{c};
  const int i = c.i, sz = (int)g.sz, sx = g.sx;
  const float dt = g.dt, idz = g.idz, idx = g.idx, idy = g.idy;
  __shared__ float4 stash[17 * VEC_THREADS];
  Stash<VEC_THREADS> own{stash + vec_thread()};
  enum { SZZ, SXX, SYY, SXZ, SXY, SYZ, AZZ, AXX, AYY, AXZ, AXY, AYZ, LA, MU, BU, GL, GM };
  own.fetch(LA, lam + i); own.fetch(MU, mu + i);
  own.fetch(AZZ, a.szz + i); own.fetch(AXX, a.sxx + i); own.fetch(AYY, a.syy + i);
  own.fetch(AXZ, a.sxz + i); own.fetch(AXY, a.sxy + i); own.fetch(AYZ, a.syz + i);
  const Pml<VA> m = pml_of<VA>(g, c, false);
  if (do_adj && g.far)
    for (const float *p : {a.vz, a.vx, a.vy}) prefetch_row(p + i);
  bool in[VEC];
  const bool any_in = do_rev && inner_cells(g, c, in);
  // to_bnd: the shell points take the stored stresses of the step
  int sk[VEC] = {-1, -1, -1, -1};
  bool any_sk = false;
  if (do_rev && shell.rows) {
    const int srow = shell.rows[z * nx + x];
    if (srow >= 0) any_sk = shell_cells(shell, srow, c, sk);
  }
  const long long hit = (do_rev && src.cell) ? src.cell[0] - i : -1;
  const bool any_hit = hit >= 0 && hit < VEC;
  const bool any_rev = any_in || any_sk || any_hit;
  if (any_rev) {
    own.fetch(SZZ, f.szz + i); own.fetch(SXX, f.sxx + i); own.fetch(SYY, f.syy + i);
    own.fetch(SXZ, f.sxz + i); own.fetch(SXY, f.sxy + i); own.fetch(SYZ, f.syz + i);
    if (any_in) { own.fetch(GL, glam + i); own.fetch(GM, gmu + i); }
  }
  if (do_adj) own.fetch(BU, buoy + i);
  vec_begin();  // up to here: nothing that the velocity kernel writes
  if (any_rev) {
    auto restore = [&](int q, Row &n) {
      if (!any_sk) return;
#pragma unroll
      for (int e = 0; e < VEC; ++e)
        if (sk[e] >= 0) n.v[e] = shell.store[(size_t)q * shell.npts + sk[e]];
    };
    Row gm{};
    {
      Row ezz{}, exx{}, eyy{};
      if (any_in) {
        ezz = D.m(f.vz + i, sz, idz);
        exx = D.m(f.vx + i, sx, idx);
        eyy = D.my(f.vy + i, idy);
      }
      own.wait();
      Row szz = own.get(SZZ), sxx = own.get(SXX), syy = own.get(SYY);
      if (any_hit) {
        const float src_amp = src.stf ? src.stf[src.it] : 0.f;
        const double am = 2250000.0 * (double)src_amp * (double)dt;
#pragma unroll
        for (int e = 0; e < VEC; ++e) {
          if (hit != e) continue;
          szz.v[e] = (float)((double)szz[e] - am);
          sxx.v[e] = (float)((double)sxx[e] - am);
          syy.v[e] = (float)((double)syy[e] - am);
        }
      }
      if (any_in) {
        const Row l = own.get(LA), u = own.get(MU);
        const Row azz = own.get(AZZ), axx = own.get(AXX), ayy = own.get(AYY);
        Row gl = own.get(GL);
#pragma unroll
        for (int e = 0; e < VEC; ++e) {
          if (!in[e]) continue;
          const float le = l[e], l2u = le + 2.0f * u[e];
          szz.v[e] = __fmaf_rn(-dot3(l2u, ezz[e], le, exx[e], le, eyy[e]), dt, szz[e]);
          sxx.v[e] = __fmaf_rn(-dot3(le, ezz[e], l2u, exx[e], le, eyy[e]), dt, sxx[e]);
          syy.v[e] = __fmaf_rn(-dot3(le, ezz[e], le, exx[e], l2u, eyy[e]), dt, syy[e]);
          gl.v[e] = undo(gl[e], sum3(azz[e], axx[e], ayy[e]), sum3(ezz[e], exx[e], eyy[e]), dt);
          gm.v[e] = dot3(2.0f * azz[e], ezz[e], 2.0f * axx[e], exx[e], 2.0f * ayy[e], eyy[e]);
        }
        st_row(glam + i, gl);
      }
      restore(0, szz); restore(2, sxx); restore(3, syy);
      st_row(f.szz + i, szz); st_row(f.sxx + i, sxx); st_row(f.syy + i, syy);
    }
    if (any_in || any_sk) {
      // one shear stress from its two derivatives, and its share of the mu image
      auto shear = [&](int r, int ra, int q, float *dst, const Row &d0, float i0, const Row &d1,
                       float i1) {
        Row n = own.get(r);
        const Row u = own.get(MU), as = own.get(ra);
#pragma unroll
        for (int e = 0; e < VEC; ++e) {
          if (!any_in || !in[e]) continue;
          const float s = sum2d(d0[e], i0, d1[e], i1);
          n.v[e] = undo(n[e], s, u[e], dt);
          gm.v[e] = __fmaf_rn(as[e], s, gm[e]);
        }
        restore(q, n);
        st_row(dst, n);
      };
      Row d0{}, d1{};
      if (any_in) { d0 = D.p(f.vx + i, sz, 1.f); d1 = D.p(f.vz + i, sx, 1.f); }
      shear(SXZ, AXZ, 1, f.sxz + i, d0, idz, d1, idx);
      if (any_in) { d0 = D.p(f.vy + i, sz, 1.f); d1 = D.py(f.vz + i, 1.f); }
      shear(SYZ, AYZ, 5, f.syz + i, d0, idz, d1, idy);
      if (any_in) { d0 = D.py(f.vx + i, 1.f); d1 = D.p(f.vy + i, sx, 1.f); }
      shear(SXY, AXY, 4, f.sxy + i, d0, idy, d1, idx);
      if (any_in) {
        Row gr = own.get(GM);
#pragma unroll
        for (int e = 0; e < VEC; ++e)
          if (in[e]) gr.v[e] = __fmaf_rn(-gm[e], dt, gr[e]);
        st_row(gmu + i, gr);
      }
    }
  }
  if (!do_adj) { own.wait(); return; }

  const PsiGather<VA> G{g, c, m};
  float *pz = ps.z, *px = ps.x, *py = ps.y;
  const long long lz = g.slab_z, lx = g.slab_x, ly = g.slab_y;
  auto cfz = [&](int k, float out) { return m.zs ? g.cz[k * nz + z] : out; };
  auto cfx = [&](int k, float out) { return m.xs ? g.cx[k * nx + x] : out; };
  auto cfy = [&](int k, float out) { return m.yany ? coef_y<VA>(g, c, k) : fill(out); };
  own.wait();
  auto scaled = [&](const Row &s) {  // s * mu, what a shear stress feeds
    const Row u = own.get(MU);
    Row r;
#pragma unroll
    for (int e = 0; e < VEC; ++e) r.v[e] = __fmul_rn(s[e], u[e]);
    return r;
  };
  auto add_k = [&](Row &acc, float k, const Row &q) {
#pragma unroll
    for (int e = 0; e < VEC; ++e) acc.v[e] = __fmaf_rn(k, q[e], acc[e]);
  };
  auto add_y = [&](Row &acc, int which, const Row &q) {
    const Row k = coef_y<VA>(g, c, which);
#pragma unroll
    for (int e = 0; e < VEC; ++e)
      if (m.ys[e]) acc.v[e] = __fmaf_rn(k[e], q[e], acc[e]);
  };
  auto finish = [&](int r, float *dst, const Row &acc) {  // old + acc at active cells
    Row s = own.get(r);
#pragma unroll
    for (int e = 0; e < VEC; ++e)
      if (c.act[e]) s.v[e] = __fadd_rn(s[e], acc[e]);
    st_row(dst, s);
    return s;
  };
  {  // sxz
    const Row d0 = D.np(a.vz + i, sx, idx), d1 = D.np(a.vx + i, sz, idz);
    const float K0 = cfx(CK, 1.f), K1 = cfz(CK, 1.f);
    const Row b = own.get(BU);
    Row acc;
#pragma unroll
    for (int e = 0; e < VEC; ++e) {
      acc.v[e] = add4(0.f, d0[e], K0, b[e], dt);
      acc.v[e] = add4(acc[e], d1[e], K1, b[e], dt);
    }
    if (m.xs) add_k(acc, cfx(CA, 0.f), G.dpx(px + PSI_SAB1 * lx));
    if (m.zs) add_k(acc, cfz(CA, 0.f), G.dpz(pz + PSI_SAB1 * lz));
    const Row s = finish(AXZ, a.sxz + i, acc);
    if (m.xs) mem_row<VA>(px + PSI_VB1 * lx, m.kx, c, g.cx[CBH * nx + x], scaled(s), dt);
    if (m.zs) mem_row<VA>(pz + PSI_VB1 * lz, m.kz, c, g.cz[CBH * nz + z], scaled(s), dt);
  }
  {  // sxy
    const Row d0 = D.np(a.vy + i, sx, idx), d1 = D.npy(a.vx + i, idy);
    const float K0 = cfx(CK, 1.f);
    const Row K1 = cfy(CK, 1.f), b = own.get(BU);
    Row acc;
#pragma unroll
    for (int e = 0; e < VEC; ++e) {
      acc.v[e] = add4(0.f, d1[e], K1[e], b[e], dt);
      acc.v[e] = add4(acc[e], d0[e], K0, b[e], dt);
    }
    if (m.xs) add_k(acc, cfx(CA, 0.f), G.dpx(px + PSI_SAB2 * lx));
    if (m.yany) add_y(acc, CA, G.dpy(py + PSI_SAB2 * ly));
    const Row s = finish(AXY, a.sxy + i, acc);
    if (m.yany) mem_row_y(py + PSI_VB2 * ly, g, m, c, coef_y<VA>(g, c, CBH), scaled(s), dt);
    if (m.xs) mem_row<VA>(px + PSI_VB2 * lx, m.kx, c, g.cx[CBH * nx + x], scaled(s), dt);
  }
  {  // syz
    const Row d0 = D.npy(a.vz + i, idy), d1 = D.np(a.vy + i, sz, idz);
    const float K1 = cfz(CK, 1.f);
    const Row K0 = cfy(CK, 1.f), b = own.get(BU);
    Row acc;
#pragma unroll
    for (int e = 0; e < VEC; ++e) {
      acc.v[e] = add4(0.f, d0[e], K0[e], b[e], dt);
      acc.v[e] = add4(acc[e], d1[e], K1, b[e], dt);
    }
    if (m.yany) add_y(acc, CA, G.dpy(py + PSI_SAB1 * ly));
    if (m.zs) add_k(acc, cfz(CA, 0.f), G.dpz(pz + PSI_SAB2 * lz));
    const Row s = finish(AYZ, a.syz + i, acc);
    if (m.yany) mem_row_y(py + PSI_VB1 * ly, g, m, c, coef_y<VA>(g, c, CBH), scaled(s), dt);
    if (m.zs) mem_row<VA>(pz + PSI_VB2 * lz, m.kz, c, g.cz[CBH * nz + z], scaled(s), dt);
  }
  {  // normal stresses
    const Row b = own.get(BU);
    // own + b d Kh dt + a_h (difference of the axis's memory variable)
    auto normal = [&](int r, float *dst, const Row &d, const Row &K, int ax) {
      Row s = own.get(r), q{}, k = fill(0.f);
      const Row old = s;
      if (ax == 0 && m.zs) { q = G.dmz(pz + PSI_SAA * lz); k = fill(cfz(CAH, 0.f)); }
      if (ax == 1 && m.xs) { q = G.dmx(px + PSI_SAA * lx); k = fill(cfx(CAH, 0.f)); }
      if (ax == 2 && m.yany) { q = G.dmy(py + PSI_SAA * ly); k = coef_y<VA>(g, c, CAH); }
      const bool slab = ax == 0 ? m.zs : ax == 1 ? m.xs : m.yany;
#pragma unroll
      for (int e = 0; e < VEC; ++e) {
        s.v[e] = add4(s[e], b[e], d[e], K[e], dt);
        if (slab && (ax != 2 || m.ys[e])) s.v[e] = __fmaf_rn(k[e], q[e], s[e]);
        if (!c.act[e]) s.v[e] = old[e];
      }
      st_row(dst, s);
      return s;
    };
    const Row sxx = normal(AXX, a.sxx + i, D.nm(a.vx + i, sx, idx), fill(cfx(CKH, 1.f)), 1);
    const Row szz = normal(AZZ, a.szz + i, D.nm(a.vz + i, sz, idz), fill(cfz(CKH, 1.f)), 0);
    const Row syy = normal(AYY, a.syy + i, D.nmy(a.vy + i, idy), cfy(CKH, 1.f), 2);
    if (m.xs || m.zs || m.yany) {
      const Row l = own.get(LA), u = own.get(MU);
      Row l2;
#pragma unroll
      for (int e = 0; e < VEC; ++e) l2.v[e] = l[e] + 2.0f * u[e];
      // b m + (cz szz + cx sxx + cy syy) dt
      auto feed = [&](float *p, int k, float bz, const Row &cz, const Row &cx,
                      const Row &cy) {
        Row r = ld_psi<VA>(p, k, c);
#pragma unroll
        for (int e = 0; e < VEC; ++e)
          if (c.act[e])
            r.v[e] = add3(add3(add3(__fmul_rn(bz, r[e]), cz[e], szz[e], dt), cx[e],
                               sxx[e], dt), cy[e], syy[e], dt);
        st_psi<VA>(p, k, r, c);
      };
      if (m.xs) feed(px + PSI_VA * lx, m.kx, g.cx[CB * nx + x], l, l2, l);
      if (m.zs) feed(pz + PSI_VA * lz, m.kz, g.cz[CB * nz + z], l2, l, l);
      if (m.yany) {
        float *p = py + PSI_VA * ly;
        const Row bz = coef_y<VA>(g, c, CB);
        Row r = ld_psi_y(p, g, m, c);
#pragma unroll
        for (int e = 0; e < VEC; ++e)
          if (m.ys[e])
            r.v[e] = add3(add3(add3(__fmul_rn(bz[e], r[e]), l[e], szz[e], dt), l[e],
                               sxx[e], dt), l2[e], syy[e], dt);
        st_psi_y(p, r, m, g, c);
      }
    }
  }
}

// K1 6 and K2 5 resident CTAs per SM (80 and 93 registers).  At 152^3 K1 takes
// 150 / 144 / 137 us with 4 / 5 / 6 CTAs, K2 138 / 139 / 152; with the own rows
// fetched ahead of the kernel before, both 130 (271 and 289 in z-marching
// kernels on bulk copies).  Latency bounds them: DRAM at 0.5 of the copy
// bandwidth, L1's data pipe 55-60 % busy at a hit rate of 47 %, 20-24 warps per
// SM.  More warps do not help: the reverse and the adjoint half on different
// warps, 32 per SM, take 170 and 149.
void launch_rev_velocity_vec(cudaStream_t st, const Geo &g, const Fields &f, const Fields &a,
                             const Psi &ps, const float *lam, const float *mu, const float *buoy,
                             float *grho, int do_rev, int do_adj, const ShellMap &shell,
                             const RecFuse &inj, bool after_stress) {
  if (psi_vectors(g))
    vec_launch(k_rev_velocity_vec<true, 6>, vec_grid(g), VEC_TZ, after_stress, st, g, f, a, ps, lam, mu, buoy, grho, do_rev, do_adj, shell, inj);
  else
    vec_launch(k_rev_velocity_vec<false, 6>, vec_grid(g), VEC_TZ, after_stress, st, g, f, a, ps, lam, mu, buoy, grho, do_rev, do_adj, shell, inj);
}

void launch_rev_stress_vec(cudaStream_t st, const Geo &g, const Fields &f, const Fields &a,
                           const Psi &ps, const float *lam, const float *mu, const float *buoy,
                           float *glam, float *gmu, int do_rev, int do_adj, const SrcArgs &src,
                           const ShellMap &shell, bool after_velocity) {
  if (psi_vectors(g))
    vec_launch(k_rev_stress_vec<true, 5>, vec_grid(g), VEC_TZ, after_velocity, st, g, f, a, ps, lam, mu, buoy, glam, gmu, do_rev, do_adj, src, shell);
  else
    vec_launch(k_rev_stress_vec<false, 5>, vec_grid(g), VEC_TZ, after_velocity, st, g, f, a, ps, lam, mu, buoy, glam, gmu, do_rev, do_adj, src, shell);
}

}  // namespace efwi
