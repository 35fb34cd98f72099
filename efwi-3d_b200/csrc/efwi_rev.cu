// Reverse sweep of the reference gradient (mode "reference").
//
// One reverse time step of the reference (libCUFD.cu:532-612) is
//   velocity(rev) -> restore v shell -> add_source(sub) -> stress(rev)
//   -> restore sigma shell -> velocity_adj -> res_injection -> stress_adj.
// Here it runs as two fused kernels plus the shell restores:
//   K1 = velocity(rev) [interior, rho imaging]   + velocity_adj [2, n-3]
//   K2 = add_source(sub) + stress(rev) [interior, lambda/mu imaging]
//        + stress_adj [2, n-3]
// The reorderings are exact: velocity_adj reads only adjoint stresses and
// stress-type adjoint memory variables, which stress(rev) does not touch;
// the rho image reads the adjoint velocity before velocity_adj updates it,
// and the lambda/mu image reads the adjoint stress before stress_adj
// updates it, as in the reference's sequential order.
//
// Restated kernels: velocity.cu:102-131, stress.cu:103-135,
// velocity_adj.cu:59-144, stress_adj.cu:52-142.  The adjoint memory
// variables reuse the forward slab buffers (the reference re-zeroes and
// reuses its 18 full-grid arrays, libCUFD.cu:481-498).
#include "efwi_common.cuh"
#include "efwi_kernels.h"

namespace efwi {

namespace {

// -D+ / -D- of slab memory variables at neighbours, zero outside the slab.
__device__ __forceinline__ float nxp(const Geo &g, const float *p, int z, int x, int y) {
  return -dplus(psi_x_get(g, p, z, x - 1, y), psi_x_get(g, p, z, x, y),
                psi_x_get(g, p, z, x + 1, y), psi_x_get(g, p, z, x + 2, y));
}
__device__ __forceinline__ float nxm(const Geo &g, const float *p, int z, int x, int y) {
  return -dminus(psi_x_get(g, p, z, x - 2, y), psi_x_get(g, p, z, x - 1, y),
                 psi_x_get(g, p, z, x, y), psi_x_get(g, p, z, x + 1, y));
}
__device__ __forceinline__ float nyp(const Geo &g, const float *p, int z, int x, int y) {
  return -dplus(psi_y_get(g, p, z, x, y - 1), psi_y_get(g, p, z, x, y),
                psi_y_get(g, p, z, x, y + 1), psi_y_get(g, p, z, x, y + 2));
}
__device__ __forceinline__ float nym(const Geo &g, const float *p, int z, int x, int y) {
  return -dminus(psi_y_get(g, p, z, x, y - 2), psi_y_get(g, p, z, x, y - 1),
                 psi_y_get(g, p, z, x, y), psi_y_get(g, p, z, x, y + 1));
}
__device__ __forceinline__ float nzp(const Geo &g, const float *p, int z, int x, int y) {
  return -dplus(psi_z_get(g, p, z - 1, x, y), psi_z_get(g, p, z, x, y),
                psi_z_get(g, p, z + 1, x, y), psi_z_get(g, p, z + 2, x, y));
}
__device__ __forceinline__ float nzm(const Geo &g, const float *p, int z, int x, int y) {
  return -dminus(psi_z_get(g, p, z - 2, x, y), psi_z_get(g, p, z - 1, x, y),
                 psi_z_get(g, p, z, x, y), psi_z_get(g, p, z + 1, x, y));
}

struct Coef {
  float K, a, b, Kh, ah, bh;
};
__device__ __forceinline__ Coef coef(const float *c, int n, int i) {
  Coef r;
  r.K = c[CK * n + i]; r.a = c[CA * n + i]; r.b = c[CB * n + i];
  r.Kh = c[CKH * n + i]; r.ah = c[CAH * n + i]; r.bh = c[CBH * n + i];
  return r;
}

}  // namespace

template <int BX>
__global__ void __launch_bounds__(32 * BX)
k_rev_velocity(Geo g, Fields f, Fields a, Psi ps, const float *__restrict__ lam,
               const float *__restrict__ mu, const float *__restrict__ buoy, float *grho,
               int zchunk, int nzc, int do_rev, int do_adj) {
  const int y = blockIdx.x * 32 + threadIdx.x;
  const int x = blockIdx.y * BX + threadIdx.y;
  const int zc = blockIdx.z % nzc;
  const int z0 = max(zc * zchunk, 2);
  const int z1 = min(zc * zchunk + zchunk, g.nz - 2);
  if (x < 2 || x > g.nx - 3 || y < 2 || y > g.ny - 3 || z0 >= z1) return;

  const int np = g.np, nz = g.nz, nx = g.nx, ny = g.ny;
  const long long sz = g.sz;
  const int sx = g.sx;
  const float dt = g.dt, idz = g.idz, idx = g.idx, idy = g.idy;
  const bool xin = x >= np && x <= nx - 1 - np, yin = y >= np && y <= ny - 1 - np;
  const bool xs = slab_s(x, nx, np), ys = slab_s(y, ny, np);
  const Coef cx = coef(g.cx, nx, x), cy = coef(g.cy, ny, y);

  const float *__restrict__ szz = f.szz;
  const float *__restrict__ sxx = f.sxx;
  const float *__restrict__ syy = f.syy;
  const float *__restrict__ sxz = f.sxz;
  const float *__restrict__ sxy = f.sxy;
  const float *__restrict__ syz = f.syz;
  const float *__restrict__ aszz = a.szz;
  const float *__restrict__ asxx = a.sxx;
  const float *__restrict__ asyy = a.syy;
  const float *__restrict__ asxz = a.sxz;
  const float *__restrict__ asxy = a.sxy;
  const float *__restrict__ asyz = a.syz;
  const float *psz = ps.z, *psx = ps.x, *psy = ps.y;
  float *pz = ps.z, *px = ps.x, *py = ps.y;

  for (int z = z0; z < z1; ++z) {
    const long long i = ((long long)z * nx + x) * sx + y;
    const float b = buoy[i];
    const float avz0 = a.vz[i], avx0 = a.vx[i], avy0 = a.vy[i];
    if (do_rev && xin && yin && z >= np && z <= nz - 1 - np) {
      const float dz_ = sum3d(dplus(szz[i - sz], szz[i], szz[i + sz], szz[i + 2 * sz]), idz,
                             dminus(sxz[i - 2 * sx], sxz[i - sx], sxz[i], sxz[i + sx]), idx,
                             dminus(syz[i - 2], syz[i - 1], syz[i], syz[i + 1]), idy);
      const float dx_ = sum3d(dminus(sxz[i - 2 * sz], sxz[i - sz], sxz[i], sxz[i + sz]), idz,
                             dplus(sxx[i - sx], sxx[i], sxx[i + sx], sxx[i + 2 * sx]), idx,
                             dminus(sxy[i - 2], sxy[i - 1], sxy[i], sxy[i + 1]), idy);
      const float dy_ = sum3d(dminus(syz[i - 2 * sz], syz[i - sz], syz[i], syz[i + sz]), idz,
                             dquirk(sxy[i - 2 * sx], sxy[i - sx], sxy[i]), idx,
                             dplus(syy[i - 1], syy[i], syy[i + 1], syy[i + 2]), idy);
      f.vz[i] = undo(f.vz[i], dz_, b, dt);
      f.vx[i] = undo(f.vx[i], dx_, b, dt);
      f.vy[i] = undo(f.vy[i], dy_, b, dt);
      const float nb2 = -(b * b);
      grho[i] = __fadd_rn(grho[i], -img3(avz0, dz_, avx0, dx_, avy0, dy_, dt, nb2));
    }
    if (!do_adj) continue;
    const bool zs = slab_s(z, nz, np);
    const Coef cz = coef(g.cz, nz, z);
    const float l = lam[i], u = mu[i], l2u = l + 2.0f * u;
    // ---- adjoint vx
    {
      const float dszz_dx = __fmul_rn(-dplus(aszz[i - sx], aszz[i], aszz[i + sx], aszz[i + 2 * sx]), idx);
      const float dsxx_dx = __fmul_rn(-dplus(asxx[i - sx], asxx[i], asxx[i + sx], asxx[i + 2 * sx]), idx);
      const float dsyy_dx = __fmul_rn(-dplus(asyy[i - sx], asyy[i], asyy[i + sx], asyy[i + 2 * sx]), idx);
      const float dsxz_dz = __fmul_rn(-dminus(asxz[i - 2 * sz], asxz[i - sz], asxz[i], asxz[i + sz]), idz);
      const float dsxy_dy = __fmul_rn(-dminus(asxy[i - 2], asxy[i - 1], asxy[i], asxy[i + 1]), idy);
      float acc = 0.f;
      acc = add4(acc, l2u, dsxx_dx, cx.K, dt);
      acc = add4(acc, l, dszz_dx, cx.K, dt);
      acc = add4(acc, l, dsyy_dx, cx.K, dt);
      acc = add4(acc, u, cz.Kh, dsxz_dz, dt);
      acc = add4(acc, u, cy.Kh, dsxy_dy, dt);
      if (xs) acc = __fmaf_rn(cx.a, __fmul_rn(nxp(g, psx + PSI_VA * g.slab_x, z, x, y), idx), acc);
      if (zs) acc = __fmaf_rn(cz.ah, __fmul_rn(nzm(g, psz + PSI_VB1 * g.slab_z, z, x, y), idz), acc);
      if (ys) acc = __fmaf_rn(cy.ah, __fmul_rn(nym(g, psy + PSI_VB2 * g.slab_y, z, x, y), idy), acc);
      const float v = __fadd_rn(avx0, acc);
      a.vx[i] = v;
      if (xs) { const long long k = PSI_SAA * g.slab_x + psi_x_idx(g, z, x, y); px[k] = add3(__fmul_rn(cx.bh, px[k]), b, v, dt); }
      if (zs) { const long long k = PSI_SAB1 * g.slab_z + psi_z_idx(g, z, x, y); pz[k] = add3(__fmul_rn(cz.b, pz[k]), b, v, dt); }
      if (ys) { const long long k = PSI_SAB2 * g.slab_y + psi_y_idx(g, z, x, y); py[k] = add3(__fmul_rn(cy.b, py[k]), b, v, dt); }
    }
    // ---- adjoint vz
    {
      const float dszz_dz = __fmul_rn(-dplus(aszz[i - sz], aszz[i], aszz[i + sz], aszz[i + 2 * sz]), idz);
      const float dsxx_dz = __fmul_rn(-dplus(asxx[i - sz], asxx[i], asxx[i + sz], asxx[i + 2 * sz]), idz);
      const float dsyy_dz = __fmul_rn(-dplus(asyy[i - sz], asyy[i], asyy[i + sz], asyy[i + 2 * sz]), idz);
      const float dsxz_dx = __fmul_rn(-dminus(asxz[i - 2 * sx], asxz[i - sx], asxz[i], asxz[i + sx]), idx);
      const float dsyz_dy = __fmul_rn(-dminus(asyz[i - 2], asyz[i - 1], asyz[i], asyz[i + 1]), idy);
      float acc = 0.f;
      acc = add4(acc, l2u, dszz_dz, cz.K, dt);
      acc = add4(acc, l, dsxx_dz, cz.K, dt);
      acc = add4(acc, l, dsyy_dz, cz.K, dt);
      acc = add4(acc, u, cy.Kh, dsyz_dy, dt);
      acc = add4(acc, u, cx.Kh, dsxz_dx, dt);
      if (zs) acc = __fmaf_rn(cz.a, __fmul_rn(nzp(g, psz + PSI_VA * g.slab_z, z, x, y), idz), acc);
      if (ys) acc = __fmaf_rn(cy.ah, __fmul_rn(nym(g, psy + PSI_VB1 * g.slab_y, z, x, y), idy), acc);
      if (xs) acc = __fmaf_rn(cx.ah, __fmul_rn(nxm(g, psx + PSI_VB1 * g.slab_x, z, x, y), idx), acc);
      const float v = __fadd_rn(avz0, acc);
      a.vz[i] = v;
      if (xs) { const long long k = PSI_SAB1 * g.slab_x + psi_x_idx(g, z, x, y); px[k] = __fmaf_rn(cx.b, px[k], __fmul_rn(__fmul_rn(b, v), dt)); }
      if (zs) { const long long k = PSI_SAA * g.slab_z + psi_z_idx(g, z, x, y); pz[k] = add3(__fmul_rn(cz.bh, pz[k]), b, v, dt); }
      if (ys) { const long long k = PSI_SAB1 * g.slab_y + psi_y_idx(g, z, x, y); py[k] = add3(__fmul_rn(cy.b, py[k]), b, v, dt); }
    }
    // ---- adjoint vy
    {
      const float dsyy_dy = __fmul_rn(-dplus(asyy[i - 1], asyy[i], asyy[i + 1], asyy[i + 2]), idy);
      const float dsxx_dy = __fmul_rn(-dplus(asxx[i - 1], asxx[i], asxx[i + 1], asxx[i + 2]), idy);
      const float dszz_dy = __fmul_rn(-dplus(aszz[i - 1], aszz[i], aszz[i + 1], aszz[i + 2]), idy);
      const float dsxy_dx = __fmul_rn(-dminus(asxy[i - 2 * sx], asxy[i - sx], asxy[i], asxy[i + sx]), idx);
      const float dsyz_dz = __fmul_rn(-dminus(asyz[i - 2 * sz], asyz[i - sz], asyz[i], asyz[i + sz]), idz);
      float acc = 0.f;
      acc = add4(acc, l, dsxx_dy, cy.K, dt);
      acc = add4(acc, l2u, dsyy_dy, cy.K, dt);
      acc = add4(acc, l, dszz_dy, cy.K, dt);
      acc = add4(acc, u, cx.Kh, dsxy_dx, dt);
      acc = add4(acc, u, cz.Kh, dsyz_dz, dt);
      if (ys) acc = __fmaf_rn(cy.a, __fmul_rn(nyp(g, psy + PSI_VA * g.slab_y, z, x, y), idy), acc);
      if (xs) acc = __fmaf_rn(cx.ah, __fmul_rn(nxm(g, psx + PSI_VB2 * g.slab_x, z, x, y), idx), acc);
      if (zs) acc = __fmaf_rn(cz.ah, __fmul_rn(nzm(g, psz + PSI_VB2 * g.slab_z, z, x, y), idz), acc);
      const float v = __fadd_rn(avy0, acc);
      a.vy[i] = v;
      if (xs) { const long long k = PSI_SAB2 * g.slab_x + psi_x_idx(g, z, x, y); px[k] = add3(__fmul_rn(cx.b, px[k]), b, v, dt); }
      if (zs) { const long long k = PSI_SAB2 * g.slab_z + psi_z_idx(g, z, x, y); pz[k] = add3(__fmul_rn(cz.bh, pz[k]), b, v, dt); }
      if (ys) { const long long k = PSI_SAA * g.slab_y + psi_y_idx(g, z, x, y); py[k] = add3(__fmul_rn(cy.b, py[k]), b, v, dt); }
    }
  }
}

template <int BX>
__global__ void __launch_bounds__(32 * BX)
k_rev_stress(Geo g, Fields f, Fields a, Psi ps, const float *__restrict__ lam,
             const float *__restrict__ mu, const float *__restrict__ buoy, float *glam,
             float *gmu, int zchunk, int nzc, int do_rev, int do_adj, SrcArgs src) {
  const int y = blockIdx.x * 32 + threadIdx.x;
  const int x = blockIdx.y * BX + threadIdx.y;
  const int zc = blockIdx.z % nzc;
  const int z0 = max(zc * zchunk, 2);
  const int z1 = min(zc * zchunk + zchunk, g.nz - 2);
  if (x < 2 || x > g.nx - 3 || y < 2 || y > g.ny - 3 || z0 >= z1) return;

  const int np = g.np, nz = g.nz, nx = g.nx, ny = g.ny;
  const long long sz = g.sz;
  const int sx = g.sx;
  const float dt = g.dt, idz = g.idz, idx = g.idx, idy = g.idy;
  const bool xin = x >= np && x <= nx - 1 - np, yin = y >= np && y <= ny - 1 - np;
  const bool xs = slab_s(x, nx, np), ys = slab_s(y, ny, np);
  const Coef cx = coef(g.cx, nx, x), cy = coef(g.cy, ny, y);
  const long long src_cell = (do_rev && src.cell) ? src.cell[0] : -1;
  const float src_amp = (do_rev && src.stf) ? src.stf[src.it] : 0.f;

  const float *__restrict__ vz = f.vz;
  const float *__restrict__ vx = f.vx;
  const float *__restrict__ vy = f.vy;
  const float *__restrict__ avz = a.vz;
  const float *__restrict__ avx = a.vx;
  const float *__restrict__ avy = a.vy;
  const float *psz = ps.z, *psx = ps.x, *psy = ps.y;
  float *pz = ps.z, *px = ps.x, *py = ps.y;

  for (int z = z0; z < z1; ++z) {
    const long long i = ((long long)z * nx + x) * sx + y;
    const float l = lam[i], u = mu[i], l2u = l + 2.0f * u;
    const float azz0 = a.szz[i], axx0 = a.sxx[i], ayy0 = a.syy[i];
    const float axz0 = a.sxz[i], axy0 = a.sxy[i], ayz0 = a.syz[i];
    if (do_rev) {
      float szz = f.szz[i], sxx = f.sxx[i], syy = f.syy[i];
      if (i == src_cell) {
        const double am = 2250000.0 * (double)src_amp * (double)dt;
        szz = (float)((double)szz - am);
        sxx = (float)((double)sxx - am);
        syy = (float)((double)syy - am);
      }
      if (xin && yin && z >= np && z <= nz - 1 - np) {
        const float ezz = __fmul_rn(dminus(vz[i - 2 * sz], vz[i - sz], vz[i], vz[i + sz]), idz);
        const float exx = __fmul_rn(dminus(vx[i - 2 * sx], vx[i - sx], vx[i], vx[i + sx]), idx);
        const float eyy = __fmul_rn(dminus(vy[i - 2], vy[i - 1], vy[i], vy[i + 1]), idy);
        szz = __fmaf_rn(-dot3(l2u, ezz, l, exx, l, eyy), dt, szz);
        sxx = __fmaf_rn(-dot3(l, ezz, l2u, exx, l, eyy), dt, sxx);
        syy = __fmaf_rn(-dot3(l, ezz, l, exx, l2u, eyy), dt, syy);
        const float exz = sum2d(dplus(vx[i - sz], vx[i], vx[i + sz], vx[i + 2 * sz]), idz,
                                dplus(vz[i - sx], vz[i], vz[i + sx], vz[i + 2 * sx]), idx);
        const float exy = sum2d(dplus(vx[i - 1], vx[i], vx[i + 1], vx[i + 2]), idy,
                                dplus(vy[i - sx], vy[i], vy[i + sx], vy[i + 2 * sx]), idx);
        const float eyz = sum2d(dplus(vy[i - sz], vy[i], vy[i + sz], vy[i + 2 * sz]), idz,
                                dplus(vz[i - 1], vz[i], vz[i + 1], vz[i + 2]), idy);
        f.sxz[i] = undo(f.sxz[i], exz, u, dt);
        f.sxy[i] = undo(f.sxy[i], exy, u, dt);
        f.syz[i] = undo(f.syz[i], eyz, u, dt);
        glam[i] = undo(glam[i], sum3(azz0, axx0, ayy0), sum3(ezz, exx, eyy), dt);
        float gm = dot3(2.0f * azz0, ezz, 2.0f * axx0, exx, 2.0f * ayy0, eyy);
        gm = __fmaf_rn(axz0, exz, gm);
        gm = __fmaf_rn(ayz0, eyz, gm);
        gm = __fmaf_rn(axy0, exy, gm);
        gmu[i] = __fmaf_rn(-gm, dt, gmu[i]);
      }
      f.szz[i] = szz; f.sxx[i] = sxx; f.syy[i] = syy;
    }
    if (!do_adj) continue;
    const bool zs = slab_s(z, nz, np);
    const Coef cz = coef(g.cz, nz, z);
    const float b = buoy[i];
    // ---- sxz
    {
      const float dvz_dx = __fmul_rn(-dplus(avz[i - sx], avz[i], avz[i + sx], avz[i + 2 * sx]), idx);
      const float dvx_dz = __fmul_rn(-dplus(avx[i - sz], avx[i], avx[i + sz], avx[i + 2 * sz]), idz);
      float acc = 0.f;
      acc = add4(acc, dvz_dx, cx.K, b, dt);
      acc = add4(acc, dvx_dz, cz.K, b, dt);
      if (xs) acc = __fmaf_rn(cx.a, __fmul_rn(nxp(g, psx + PSI_SAB1 * g.slab_x, z, x, y), idx), acc);
      if (zs) acc = __fmaf_rn(cz.a, __fmul_rn(nzp(g, psz + PSI_SAB1 * g.slab_z, z, x, y), idz), acc);
      const float s = __fadd_rn(axz0, acc);
      a.sxz[i] = s;
      if (xs) { const long long k = PSI_VB1 * g.slab_x + psi_x_idx(g, z, x, y); px[k] = add3(__fmul_rn(cx.bh, px[k]), s, u, dt); }
      if (zs) { const long long k = PSI_VB1 * g.slab_z + psi_z_idx(g, z, x, y); pz[k] = add3(__fmul_rn(cz.bh, pz[k]), s, u, dt); }
    }
    // ---- sxy
    {
      const float dvy_dx = __fmul_rn(-dplus(avy[i - sx], avy[i], avy[i + sx], avy[i + 2 * sx]), idx);
      const float dvx_dy = __fmul_rn(-dplus(avx[i - 1], avx[i], avx[i + 1], avx[i + 2]), idy);
      float acc = 0.f;
      acc = add4(acc, dvx_dy, cy.K, b, dt);
      acc = add4(acc, dvy_dx, cx.K, b, dt);
      if (xs) acc = __fmaf_rn(cx.a, __fmul_rn(nxp(g, psx + PSI_SAB2 * g.slab_x, z, x, y), idx), acc);
      if (ys) acc = __fmaf_rn(cy.a, __fmul_rn(nyp(g, psy + PSI_SAB2 * g.slab_y, z, x, y), idy), acc);
      const float s = __fadd_rn(axy0, acc);
      a.sxy[i] = s;
      if (ys) { const long long k = PSI_VB2 * g.slab_y + psi_y_idx(g, z, x, y); py[k] = add3(__fmul_rn(cy.bh, py[k]), s, u, dt); }
      if (xs) { const long long k = PSI_VB2 * g.slab_x + psi_x_idx(g, z, x, y); px[k] = add3(__fmul_rn(cx.bh, px[k]), s, u, dt); }
    }
    // ---- syz
    {
      const float dvz_dy = __fmul_rn(-dplus(avz[i - 1], avz[i], avz[i + 1], avz[i + 2]), idy);
      const float dvy_dz = __fmul_rn(-dplus(avy[i - sz], avy[i], avy[i + sz], avy[i + 2 * sz]), idz);
      float acc = 0.f;
      acc = add4(acc, dvz_dy, cy.K, b, dt);
      acc = add4(acc, dvy_dz, cz.K, b, dt);
      if (ys) acc = __fmaf_rn(cy.a, __fmul_rn(nyp(g, psy + PSI_SAB1 * g.slab_y, z, x, y), idy), acc);
      if (zs) acc = __fmaf_rn(cz.a, __fmul_rn(nzp(g, psz + PSI_SAB2 * g.slab_z, z, x, y), idz), acc);
      const float s = __fadd_rn(ayz0, acc);
      a.syz[i] = s;
      if (ys) { const long long k = PSI_VB1 * g.slab_y + psi_y_idx(g, z, x, y); py[k] = add3(__fmul_rn(cy.bh, py[k]), s, u, dt); }
      if (zs) { const long long k = PSI_VB2 * g.slab_z + psi_z_idx(g, z, x, y); pz[k] = add3(__fmul_rn(cz.bh, pz[k]), s, u, dt); }
    }
    // ---- normal stresses
    {
      const float dvx_dx = __fmul_rn(-dminus(avx[i - 2 * sx], avx[i - sx], avx[i], avx[i + sx]), idx);
      const float dvz_dz = __fmul_rn(-dminus(avz[i - 2 * sz], avz[i - sz], avz[i], avz[i + sz]), idz);
      const float dvy_dy = __fmul_rn(-dminus(avy[i - 2], avy[i - 1], avy[i], avy[i + 1]), idy);
      float sxx = add4(axx0, b, dvx_dx, cx.Kh, dt);
      float szz = add4(azz0, b, dvz_dz, cz.Kh, dt);
      float syy = add4(ayy0, b, dvy_dy, cy.Kh, dt);
      if (xs) sxx = __fmaf_rn(cx.ah, __fmul_rn(nxm(g, psx + PSI_SAA * g.slab_x, z, x, y), idx), sxx);
      if (zs) szz = __fmaf_rn(cz.ah, __fmul_rn(nzm(g, psz + PSI_SAA * g.slab_z, z, x, y), idz), szz);
      if (ys) syy = __fmaf_rn(cy.ah, __fmul_rn(nym(g, psy + PSI_SAA * g.slab_y, z, x, y), idy), syy);
      a.sxx[i] = sxx; a.szz[i] = szz; a.syy[i] = syy;
      if (xs) { const long long k = PSI_VA * g.slab_x + psi_x_idx(g, z, x, y); px[k] = add3(add3(add3(__fmul_rn(cx.b, px[k]), l, szz, dt), l2u, sxx, dt), l, syy, dt); }
      if (zs) { const long long k = PSI_VA * g.slab_z + psi_z_idx(g, z, x, y); pz[k] = add3(add3(add3(__fmul_rn(cz.b, pz[k]), l2u, szz, dt), l, sxx, dt), l, syy, dt); }
      if (ys) { const long long k = PSI_VA * g.slab_y + psi_y_idx(g, z, x, y); py[k] = add3(add3(add3(__fmul_rn(cy.b, py[k]), l, szz, dt), l, sxx, dt), l2u, syy, dt); }
    }
  }
}

void launch_rev_velocity(int bx, dim3 grid, cudaStream_t st, const Geo &g, const Fields &f,
                         const Fields &a, const Psi &ps, const float *lam, const float *mu,
                         const float *buoy, float *grho, int zchunk, int nzc, int do_rev,
                         int do_adj) {
  if (bx == 8)
    k_rev_velocity<8><<<grid, dim3(32, 8), 0, st>>>(g, f, a, ps, lam, mu, buoy, grho, zchunk,
                                                   nzc, do_rev, do_adj);
  else
    k_rev_velocity<4><<<grid, dim3(32, 4), 0, st>>>(g, f, a, ps, lam, mu, buoy, grho, zchunk,
                                                   nzc, do_rev, do_adj);
}

void launch_rev_stress(int bx, dim3 grid, cudaStream_t st, const Geo &g, const Fields &f,
                       const Fields &a, const Psi &ps, const float *lam, const float *mu,
                       const float *buoy, float *glam, float *gmu, int zchunk, int nzc,
                       int do_rev, int do_adj, const SrcArgs &src) {
  if (bx == 8)
    k_rev_stress<8><<<grid, dim3(32, 8), 0, st>>>(g, f, a, ps, lam, mu, buoy, glam, gmu, zchunk,
                                                 nzc, do_rev, do_adj, src);
  else
    k_rev_stress<4><<<grid, dim3(32, 4), 0, st>>>(g, f, a, ps, lam, mu, buoy, glam, gmu, zchunk,
                                                 nzc, do_rev, do_adj, src);
}

}  // namespace efwi
