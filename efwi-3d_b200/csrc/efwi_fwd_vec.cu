// Forward half-steps, one thread per four cells (efwi_vec.cuh); the same
// arithmetic as efwi_fwd.cu.
//
// K_S  stress update + C-PML (slabs only) + point-source injection
//      (restates stress.cu:36-97 and add_source, utilities.cu:442-479)
// K_V  velocity update + C-PML (slabs only) + receiver gather
//      (restates velocity.cu:35-96, quirks Q1 and Q2 kept)
//
// Fused epilogues (efwi_fuse.cuh): K_S stores the step's starting state at
// the boundary-shell points (gradient sweeps, from_bnd); K_V records the
// receivers (recording).
#include "efwi_common.cuh"
#include "efwi_fuse.cuh"
#include "efwi_kernels.h"
#include "efwi_vec.cuh"

namespace efwi {

enum { VEC_STEP, VEC_STEP_TO, VEC_ILLUM };  // what a launch does besides the step

// The thread's vector in volume q of the state that a step writes.
__device__ __forceinline__ float *step_to(const StepTo &to, const Geo &g, int q, int z, int x, int y) {
  const long long n = (long long)g.nz * g.nx * to.pitch_out;
  return to.out + q * n + (z * g.nx + x) * to.pitch_out + y;
}

// Both kernels form one output (K_S: the normal stresses together) at a time,
// each from its own differences, so that few values are live: registers, not
// bandwidth, hold these kernels' occupancy down, and the rows read again for
// the next output come from L1.  PARTS > 1: the outputs lie on different warps
// instead (vec_split); a memory variable belongs to one derivative and so to one
// part, and the shell's copy of an output is taken by the part that updates it.
//
// VEC_STEP_TO: the results go to another state (exact gradient: a checkpoint),
// zero where no step writes, at the cost of no copy.  A checkpoint's rows have
// no padding to whole lines.  A kernel of its own: with the offsets in every
// launch, 26 x 30 x 28 and 84^3 ran 3-4 % slower.
//
// VEC_ILLUM: the kernels add the step's share of the source illumination (the diagonal
// pseudo-Hessian of k_illumination, efwi_exact.cu), whose derivatives they have
// in registers, to the shot's own sums.  Two more rows in and out for K_S and
// one for K_V take the place of a pass that reads the nine fields again with
// their neighbours: 80^3, four shots, 78 us a step in all; 329 with the pass,
// whose own 246 were one thread's chain over the shots and eight planes.
template <bool VA, int PARTS, int MINB, int MODE = VEC_STEP>
__global__ void __launch_bounds__(vec_threads(PARTS), MINB)
k_stress_fwd_vec(Geo g, Fields f, Psi ps, const float *__restrict__ lam,
                 const float *__restrict__ mu, int nzb, SrcArgs src, ShellMap shell, IllumSum il, StepTo to) {
  constexpr bool IL = MODE == VEC_ILLUM;
  static_assert(!IL || PARTS == 1, "the sums need all outputs in one thread");
  const long long tp = MODE == VEC_STEP_TO ? to.psi : 0;
  const int shot = blockIdx.z / nzb;
  constexpr int TZ = vec_tz(PARTS), T = vec_threads(PARTS);
  const int part = PARTS > 1 ? threadIdx.z / TZ : 0;
  const int z = 2 + (blockIdx.z - shot * nzb) * TZ + threadIdx.z % TZ;
  const int x = 2 + blockIdx.y * VEC_TX + threadIdx.y;
  const int y = VEC * (blockIdx.x * VEC_TY + threadIdx.x);
  const int nz = g.nz, nx = g.nx, ny = g.ny;
  if (z > nz - 3 || x > nx - 3 || y > ny - 3) return;
  const VecCell c = vec_cell(g, z, x, y);
  const VecCell r = MODE == VEC_STEP_TO ? vec_cell(g, z, x, y, to.pitch_in) : c;  // in the state read
  const long long so = (long long)shot * g.N + r.i;
  const float *__restrict__ vz = f.vz + so;
  const float *__restrict__ vx = f.vx + so;
  const float *__restrict__ vy = f.vy + so;
  const int sx = MODE == VEC_STEP_TO ? to.pitch_in : g.sx;
  const int sz = MODE == VEC_STEP_TO ? nx * sx : (int)g.sz;
  const float dt = g.dt, idz = g.idz, idx = g.idx, idy = g.idy;
  float *szz = f.szz + so, *sxx = f.sxx + so, *syy = f.syy + so;
  float *sxz = f.sxz + so, *sxy = f.sxy + so, *syz = f.syz + so;
  // where output volume q (in the order of Fields) of a field at p goes
  auto dest = [&](float *p, int q) {
    return MODE == VEC_STEP_TO ? step_to(to, g, q, z, x, y) : p;
  };
  __shared__ float4 stash[(IL ? 10 : 8) * T];
  Stash<T> own{stash + vec_thread()};
  // outputs of the thread: 0 the normal stresses, 1 sxz, 2 sxy, 3 syz
  auto mine = [&](int k) { return PARTS == 1 || part == k; };
  if (mine(0)) {
    own.fetch(0, szz); own.fetch(1, sxx); own.fetch(2, syy); own.fetch(6, lam + c.i);
  }
  if (mine(1)) own.fetch(3, sxz);
  if (mine(2)) own.fetch(4, sxy);
  if (mine(3)) own.fetch(5, syz);
  own.fetch(7, mu + c.i);
  float am[VEC] = {};  // IL: squared strains of hm
  if (IL) {
    own.fetch(8, il.of(shot, 0) + c.i);
    own.fetch(9, il.of(shot, 1) + c.i);
  }

  const Pml<VA> m = pml_of<VA>(g, c, false);
  prefetch_psi<3>(g, Psi{ps.z + (long long)shot * 6 * g.slab_z, ps.x + (long long)shot * 6 * g.slab_x,
                         ps.y + (long long)shot * 6 * g.slab_y}, m, c, PSI_VA);
  float *pz = ps.z + (long long)shot * 6 * g.slab_z;
  float *px = ps.x + (long long)shot * 6 * g.slab_x;
  float *py = ps.y + (long long)shot * 6 * g.slab_y;
  vec_begin();  // up to here: nothing that the velocity kernel writes
  if (shell.rows) {  // from_bnd: the state at the start of the step
    const int srow = shell.rows[z * nx + x];
    int sk[VEC];
    if (srow >= 0 && shell_cells(shell, srow, c, sk)) {
      auto keep = [&](int q, const float *p) {
        const Row r = ld_row(p);
        float *st = shell.store + (size_t)q * shell.npts;
#pragma unroll
        for (int e = 0; e < VEC; ++e)
          if (sk[e] >= 0) st[sk[e]] = r[e];
      };
      if (mine(0)) { keep(0, szz); keep(2, sxx); keep(3, syy); }
      if (mine(1)) { keep(1, sxz); keep(6, vz); }
      if (mine(2)) { keep(4, sxy); keep(7, vx); }
      if (mine(3)) { keep(5, syz); keep(8, vy); }
    }
  }
  // memory variables `slot` of one axis, and their derivative's update (half:
  // the coefficients at half points)
  auto ld_z = [&](int slot) { return m.zs ? ld_psi<VA>(pz + slot * g.slab_z, m.kz, c) : Row{}; };
  auto ld_x = [&](int slot) { return m.xs ? ld_psi<VA>(px + slot * g.slab_x, m.kx, c) : Row{}; };
  auto ld_y = [&](int slot) { return m.yany ? ld_psi_y(py + slot * g.slab_y, g, m, c) : Row{}; };
  auto pml_z = [&](int slot, int half, Row &r, float d[VEC]) {
    if (m.zs) pml_row<VA>(pz + slot * g.slab_z + tp, m.kz, r, c, g.cz + 3 * half * nz + z, nz, d);
  };
  auto pml_x = [&](int slot, int half, Row &r, float d[VEC]) {
    if (m.xs) pml_row<VA>(px + slot * g.slab_x + tp, m.kx, r, c, g.cx + 3 * half * nx + x, nx, d);
  };
  auto pml_y = [&](int slot, int half, Row &r, float d[VEC]) {
    if (m.yany) pml_row_y(py + slot * g.slab_y + tp, r, g, m, c, half, d);
  };

  if (mine(0)) {  // normal stresses
    Row qz = ld_z(PSI_VA), qx = ld_x(PSI_VA), qy = ld_y(PSI_VA);
    float ezz[VEC], exx[VEC], eyy[VEC];
    const Row z0 = ld_row(vz), x0 = ld_row(vx), y0 = ld_row(vy);
    {
      const Row a = ld_row(vz - 2 * sz), b = ld_row(vz - sz), d = ld_row(vz + sz);
#pragma unroll
      for (int e = 0; e < VEC; ++e) ezz[e] = dminus(a[e], b[e], z0[e], d[e]) * idz;
    }
    {
      const Row a = ld_row(vx - 2 * sx), b = ld_row(vx - sx), d = ld_row(vx + sx);
#pragma unroll
      for (int e = 0; e < VEC; ++e) exx[e] = dminus(a[e], b[e], x0[e], d[e]) * idx;
    }
    {
      const Span w = ld_span(vy, y0, r);
#pragma unroll
      for (int e = 0; e < VEC; ++e) eyy[e] = dminus(w(e, -2), w(e, -1), y0[e], w(e, 1)) * idy;
    }
    pml_z(PSI_VA, 0, qz, ezz);
    pml_x(PSI_VA, 0, qx, exx);
    pml_y(PSI_VA, 0, qy, eyy);
    own.wait();
    const Row l = own.get(6), u = own.get(7);
    Row nzz = own.get(0), nxx = own.get(1), nyy = own.get(2);
#pragma unroll
    for (int e = 0; e < VEC; ++e) {
      if (!c.act[e]) continue;
      const float le = l[e], ue = u[e], l2u = le + 2.0f * ue;
      nzz.v[e] += (l2u * ezz[e] + le * exx[e] + le * eyy[e]) * dt;
      nxx.v[e] += (le * ezz[e] + l2u * exx[e] + le * eyy[e]) * dt;
      nyy.v[e] += (le * ezz[e] + le * exx[e] + l2u * eyy[e]) * dt;
    }
    if (IL) {
      Row hl = own.get(8);
#pragma unroll
      for (int e = 0; e < VEC; ++e) {
        const float div = ezz[e] + exx[e] + eyy[e];
        if (c.act[e]) hl.v[e] += 3.0f * div * div * (dt * dt);
        am[e] = 4.0f * (ezz[e] * ezz[e] + exx[e] * exx[e] + eyy[e] * eyy[e]);
      }
      st_row(il.of(shot, 0) + c.i, hl);
    }
    const long long hit = src.cell ? src.cell[shot] - c.i : -1;
    if (hit >= 0 && hit < VEC) {
      // add_source follows the stress kernel; amplitude formed in double
      // from pow(1500, 2) (utilities.cu:450-461).
      const int sit = src.it_dev ? *src.it_dev : src.it;
      const float src_amp = src.stf ? src.stf[(long long)shot * src.nt + sit] : 0.f;
      const double a = 2250000.0 * (double)src_amp * (double)dt;
#pragma unroll
      for (int e = 0; e < VEC; ++e) {
        if (hit != e) continue;
        nzz.v[e] = (float)((double)nzz[e] + a);
        nxx.v[e] = (float)((double)nxx[e] + a);
        nyy.v[e] = (float)((double)nyy[e] + a);
      }
    }
    st_row(dest(szz, 3), nzz); st_row(dest(sxx, 4), nxx); st_row(dest(syy, 5), nyy);
  }
  // one shear stress from its two derivatives
  auto shear = [&](int k, float *dst, const float d0[VEC], const float d1[VEC]) {
    if (PARTS > 1) own.wait();
    Row n = own.get(k);
    const Row u = own.get(7);
#pragma unroll
    for (int e = 0; e < VEC; ++e)
      if (c.act[e]) n.v[e] += u[e] * (d0[e] + d1[e]) * dt;
    if (IL) {
#pragma unroll
      for (int e = 0; e < VEC; ++e) am[e] += (d0[e] + d1[e]) * (d0[e] + d1[e]);
    }
    st_row(dst, n);
  };
  if (mine(1)) {  // sxz
    Row qz = ld_z(PSI_VB1), qx = ld_x(PSI_VB1);
    float dvx_dz[VEC], dvz_dx[VEC];
    {
      const Row a = ld_row(vx - sz), m = ld_row(vx), b = ld_row(vx + sz), d = ld_row(vx + 2 * sz);
#pragma unroll
      for (int e = 0; e < VEC; ++e) dvx_dz[e] = dplus(a[e], m[e], b[e], d[e]) * idz;
    }
    {
      const Row a = ld_row(vz - sx), m = ld_row(vz), b = ld_row(vz + sx), d = ld_row(vz + 2 * sx);
#pragma unroll
      for (int e = 0; e < VEC; ++e) dvz_dx[e] = dplus(a[e], m[e], b[e], d[e]) * idx;
    }
    pml_z(PSI_VB1, 1, qz, dvx_dz);
    pml_x(PSI_VB1, 1, qx, dvz_dx);
    shear(3, dest(sxz, 6), dvx_dz, dvz_dx);
  }
  if (mine(2)) {  // sxy
    Row qx = ld_x(PSI_VB2), qy = ld_y(PSI_VB2);
    float dvx_dy[VEC], dvy_dx[VEC];
    {
      const Row m = ld_row(vx);
      const Span w = ld_span(vx, m, r);
#pragma unroll
      for (int e = 0; e < VEC; ++e) dvx_dy[e] = dplus(w(e, -1), m[e], w(e, 1), w(e, 2)) * idy;
    }
    {
      const Row a = ld_row(vy - sx), m = ld_row(vy), b = ld_row(vy + sx), d = ld_row(vy + 2 * sx);
#pragma unroll
      for (int e = 0; e < VEC; ++e) dvy_dx[e] = dplus(a[e], m[e], b[e], d[e]) * idx;
    }
    pml_x(PSI_VB2, 1, qx, dvy_dx);
    pml_y(PSI_VB2, 1, qy, dvx_dy);
    shear(4, dest(sxy, 7), dvx_dy, dvy_dx);
  }
  if (mine(3)) {  // syz
    Row qz = ld_z(PSI_VB2), qy = ld_y(PSI_VB1);
    float dvy_dz[VEC], dvz_dy[VEC];
    {
      const Row a = ld_row(vy - sz), m = ld_row(vy), b = ld_row(vy + sz), d = ld_row(vy + 2 * sz);
#pragma unroll
      for (int e = 0; e < VEC; ++e) dvy_dz[e] = dplus(a[e], m[e], b[e], d[e]) * idz;
    }
    {
      const Row m = ld_row(vz);
      const Span w = ld_span(vz, m, r);
#pragma unroll
      for (int e = 0; e < VEC; ++e) dvz_dy[e] = dplus(w(e, -1), m[e], w(e, 1), w(e, 2)) * idy;
    }
    pml_z(PSI_VB2, 1, qz, dvy_dz);
    pml_y(PSI_VB1, 1, qy, dvz_dy);
    shear(5, dest(syz, 8), dvy_dz, dvz_dy);
  }
  if (IL) {
    Row hm = own.get(9);
#pragma unroll
    for (int e = 0; e < VEC; ++e)
      if (c.act[e]) hm.v[e] += am[e] * (dt * dt);
    st_row(il.of(shot, 1) + c.i, hm);
  }
}

template <bool VA, int PARTS, int MINB, int MODE = VEC_STEP>
__global__ void __launch_bounds__(vec_threads(PARTS), MINB)
k_velocity_fwd_vec(Geo g, Fields f, Psi ps, const float *__restrict__ buoy, int nzb, RecFuse rec,
                   IllumSum il, StepTo to) {
  constexpr bool IL = MODE == VEC_ILLUM;
  static_assert(!IL || PARTS == 1, "the sums need all outputs in one thread");
  const long long tp = MODE == VEC_STEP_TO ? to.psi : 0;
  const int shot = blockIdx.z / nzb;
  constexpr int TZ = vec_tz(PARTS), T = vec_threads(PARTS);
  const int part = PARTS > 1 ? threadIdx.z / TZ : 0;
  const int z = 2 + (blockIdx.z - shot * nzb) * TZ + threadIdx.z % TZ;
  const int x = 2 + blockIdx.y * VEC_TX + threadIdx.y;
  const int y = VEC * (blockIdx.x * VEC_TY + threadIdx.x);
  const int nz = g.nz, nx = g.nx, ny = g.ny;
  if (z > nz - 3 || x > nx - 3 || y > ny - 3) return;
  const VecCell c = vec_cell(g, z, x, y);
  // in the stresses: its K_S's output
  const VecCell r = MODE == VEC_STEP_TO ? vec_cell(g, z, x, y, to.pitch_out) : c;
  const long long so = (long long)shot * g.N + r.i;
  const float *__restrict__ szz = f.szz + so;
  const float *__restrict__ sxx = f.sxx + so;
  const float *__restrict__ syy = f.syy + so;
  const float *__restrict__ sxz = f.sxz + so;
  const float *__restrict__ sxy = f.sxy + so;
  const float *__restrict__ syz = f.syz + so;
  const int sx = MODE == VEC_STEP_TO ? to.pitch_out : g.sx;
  const int sz = MODE == VEC_STEP_TO ? nx * sx : (int)g.sz;
  const float idz = g.idz, idx = g.idx, idy = g.idy, dt = g.dt;
  const long long vo = MODE == VEC_STEP_TO ? (z * nx + x) * to.pitch_in + y : so;
  float *vz = f.vz + vo, *vx = f.vx + vo, *vy = f.vy + vo;
  auto dest = [&](float *p, int q) {
    return MODE == VEC_STEP_TO ? step_to(to, g, q, z, x, y) : p;
  };
  __shared__ float4 stash[(IL || PARTS > 1 ? 5 : 4) * T];
  Stash<T> own{stash + vec_thread()};
  // outputs of the thread: 0 vz, 1 vx, 2 vy
  auto mine = [&](int k) { return PARTS == 1 || part == k; };
  if (mine(0)) own.fetch(0, vz);
  if (mine(1)) own.fetch(1, vx);
  if (mine(2)) own.fetch(2, vy);
  own.fetch(3, buoy + c.i);
  float ab[VEC] = {};  // IL: squared stress divergence of hb
  if (IL) own.fetch(4, il.of(shot, 2) + c.i);
  if (g.far)
    for (const float *p : {sxx, sxy, syy}) prefetch_row(p);
  const int rmap = receiver_map(rec.a, nz, shot, z);  // early: the latency overlaps
  if (PARTS > 1 && rmap >= 0) own.fetch(4, receiver_row(rec.a, rmap, g, c));

  const Pml<VA> m = pml_of<VA>(g, c, true);
  prefetch_psi<3>(g, Psi{ps.z + (long long)shot * 6 * g.slab_z, ps.x + (long long)shot * 6 * g.slab_x,
                         ps.y + (long long)shot * 6 * g.slab_y}, m, c, PSI_SAA);
  float *pz = ps.z + (long long)shot * 6 * g.slab_z;
  float *px = ps.x + (long long)shot * 6 * g.slab_x;
  float *py = ps.y + (long long)shot * 6 * g.slab_y;
  vec_begin();  // up to here: nothing that the stress kernel writes
  // memory variables `slot` of one axis, and their derivative's update (half:
  // the coefficients at half points)
  auto ld_z = [&](int slot) { return m.zs ? ld_psi<VA>(pz + slot * g.slab_z, m.kz, c) : Row{}; };
  auto ld_x = [&](int slot) { return m.xs ? ld_psi<VA>(px + slot * g.slab_x, m.kx, c) : Row{}; };
  auto ld_y = [&](int slot) { return m.yany ? ld_psi_y(py + slot * g.slab_y, g, m, c) : Row{}; };
  auto pml_z = [&](int slot, int half, Row &r, float d[VEC]) {
    if (m.zs) pml_row<VA>(pz + slot * g.slab_z + tp, m.kz, r, c, g.cz + 3 * half * nz + z, nz, d);
  };
  auto pml_x = [&](int slot, int half, Row &r, float d[VEC]) {
    if (m.xs) pml_row<VA>(px + slot * g.slab_x + tp, m.kx, r, c, g.cx + 3 * half * nx + x, nx, d);
  };
  auto pml_y = [&](int slot, int half, Row &r, float d[VEC]) {
    if (m.yany) pml_row_y(py + slot * g.slab_y + tp, r, g, m, c, half, d);
  };

  // one velocity from its three derivatives
  auto update = [&](int k, const float d0[VEC], const float d1[VEC], const float d2[VEC]) {
    if (PARTS > 1) own.wait();
    Row n = own.get(k);
    const Row b = own.get(3);
#pragma unroll
    for (int e = 0; e < VEC; ++e)
      if (c.act[e]) n.v[e] += (d0[e] + d1[e] + d2[e]) * b[e] * dt;
    if (IL) {
#pragma unroll
      for (int e = 0; e < VEC; ++e)
        ab[e] += (d0[e] + d1[e] + d2[e]) * (d0[e] + d1[e] + d2[e]);
    }
    return n;
  };
  Row nvz{}, nvx{}, nvy{};
  if (mine(0)) {  // vz
    Row qz = ld_z(PSI_SAA), qx = ld_x(PSI_SAB1), qy = ld_y(PSI_SAB1);
    float dszz_dz[VEC], dsxz_dx[VEC], dsyz_dy[VEC];
    {
      const Row a = ld_row(szz - sz), b = ld_row(szz), d = ld_row(szz + sz),
                h = ld_row(szz + 2 * sz);
#pragma unroll
      for (int e = 0; e < VEC; ++e) dszz_dz[e] = dplus(a[e], b[e], d[e], h[e]) * idz;
    }
    {
      const Row a = ld_row(sxz - 2 * sx), b = ld_row(sxz - sx), m = ld_row(sxz),
                d = ld_row(sxz + sx);
#pragma unroll
      for (int e = 0; e < VEC; ++e) dsxz_dx[e] = dminus(a[e], b[e], m[e], d[e]) * idx;
    }
    {
      const Row m = ld_row(syz);
      const Span w = ld_span(syz, m, r);
#pragma unroll
      for (int e = 0; e < VEC; ++e) dsyz_dy[e] = dminus(w(e, -2), w(e, -1), m[e], w(e, 1)) * idy;
    }
    pml_z(PSI_SAA, 1, qz, dszz_dz);
    pml_x(PSI_SAB1, 0, qx, dsxz_dx);
    pml_y(PSI_SAB1, 0, qy, dsyz_dy);
    own.wait();
    nvz = update(0, dszz_dz, dsxz_dx, dsyz_dy);
    st_row(dest(vz, 0), nvz);
  }
  if (mine(1)) {  // vx
    Row qz = ld_z(PSI_SAB1), qx = ld_x(PSI_SAA), qy = ld_y(PSI_SAB2);
    float dsxz_dz[VEC], dsxx_dx[VEC], dsxy_dy[VEC];
    {
      const Row h = ld_row(sxz - 2 * sz), k = ld_row(sxz - sz), m = ld_row(sxz),
                l = ld_row(sxz + sz);
#pragma unroll
      for (int e = 0; e < VEC; ++e) dsxz_dz[e] = dminus(h[e], k[e], m[e], l[e]) * idz;
    }
    {
      const Row a = ld_row(sxx - sx), m = ld_row(sxx), b = ld_row(sxx + sx),
                d = ld_row(sxx + 2 * sx);
#pragma unroll
      for (int e = 0; e < VEC; ++e) dsxx_dx[e] = dplus(a[e], m[e], b[e], d[e]) * idx;
    }
    {
      const Row m = ld_row(sxy);
      const Span w = ld_span(sxy, m, r);
#pragma unroll
      for (int e = 0; e < VEC; ++e) dsxy_dy[e] = dminus(w(e, -2), w(e, -1), m[e], w(e, 1)) * idy;
    }
    pml_z(PSI_SAB1, 0, qz, dsxz_dz);
    pml_x(PSI_SAA, 1, qx, dsxx_dx);
    pml_y(PSI_SAB2, 0, qy, dsxy_dy);
    nvx = update(1, dsxz_dz, dsxx_dx, dsxy_dy);
    st_row(dest(vx, 1), nvx);
  }
  if (mine(2)) {  // vy
    Row qz = ld_z(PSI_SAB2), qx = ld_x(PSI_SAB2), qy = ld_y(PSI_SAA);
    float dsyz_dz[VEC], dsxy_dx[VEC], dsyy_dy[VEC];
    {
      const Row h = ld_row(syz - 2 * sz), k = ld_row(syz - sz), m = ld_row(syz),
                l = ld_row(syz + sz);
#pragma unroll
      for (int e = 0; e < VEC; ++e) dsyz_dz[e] = dminus(h[e], k[e], m[e], l[e]) * idz;
    }
    {
      const Row m = ld_row(sxy), a = ld_row(sxy - sx), b = ld_row(sxy - 2 * sx);
      // Quirk Q1 (velocity.cu:79): c2 * (sxy[i-1] - sxy[i-2]) along x.
#pragma unroll
      for (int e = 0; e < VEC; ++e)
        dsxy_dx[e] = (EFWI_C1 * (m[e] - a[e]) - EFWI_C2 * (a[e] - b[e])) * idx;
    }
    {
      const Row m = ld_row(syy);
      const Span w = ld_span(syy, m, r);
#pragma unroll
      for (int e = 0; e < VEC; ++e) dsyy_dy[e] = dplus(w(e, -1), m[e], w(e, 1), w(e, 2)) * idy;
    }
    pml_z(PSI_SAB2, 0, qz, dsyz_dz);
    pml_x(PSI_SAB2, 0, qx, dsxy_dx);
    pml_y(PSI_SAA, 1, qy, dsyy_dy);
    nvy = update(2, dsyz_dz, dsxy_dx, dsyy_dy);
    st_row(dest(vy, 2), nvy);
  }
  if (IL) {
    Row hb = own.get(4);
#pragma unroll
    for (int e = 0; e < VEC; ++e)
      if (c.act[e]) hb.v[e] += ab[e] * (dt * dt);
    st_row(il.of(shot, 2) + c.i, hb);
  }
  if (rmap >= 0) {
    // fetched ahead where a launch is one thread's chain of loads; elsewhere
    // that only costs (84^3 misfit + 2 %)
    const Row entry = PARTS > 1 ? own.get(4) : ld_row(receiver_row(rec.a, rmap, g, c));
#pragma unroll
    for (int e = 0; e < VEC; ++e) {
      const int u = __float_as_int(entry[e]);
      if (c.act[e] && u != -1)
        record_cell(rec.a, rec.tm, rec.it, shot, u, mine(1), nvx[e], mine(2), nvy[e], mine(0), nvz[e]);
    }
  }
}

// Registers decide the resident CTAs per SM: K_S 6 (80 registers), K_V 5 (96).
// At 152^3, one shot of a gradient (microseconds, event overhead of 6 in all):
// K_S 94 / 82 / 79 / 89 and K_V 68 / 64 / 62 / 68 with 4 / 5 / 6 / 7 CTAs; K_V
// with 6 is no faster where a launch has few waves (75 x 109 x 91).  With the
// own rows fetched ahead of the kernel before, K_S takes 72 and K_V 55 (126 and
// 91 in z-marching kernels on bulk copies); four shots 203 and 181 (408, 280),
// 0.84 and 0.77 of the copy bandwidth: DRAM bounds batches, the tail of each
// launch and the loads' latency single shots.
void launch_stress_fwd_vec(int S, cudaStream_t st, const Geo &g, const Fields &f, const Psi &ps,
                           const float *lam, const float *mu, const SrcArgs &src,
                           const ShellMap &shell, const IllumSum &il, const StepTo &to, bool after_velocity) {
  const int mode = il.first ? VEC_ILLUM : to.out ? VEC_STEP_TO : VEC_STEP;
  const int parts = mode == VEC_STEP && vec_split(g, S) ? 4 : 1;
  const dim3 grid = vec_grid(g, S, parts);
  const int nzb = grid.z / S;
  const bool va = psi_vectors(g);
  auto k = mode == VEC_ILLUM ? (va ? k_stress_fwd_vec<true, 1, 5, VEC_ILLUM> : k_stress_fwd_vec<false, 1, 5, VEC_ILLUM>)
           : mode == VEC_STEP_TO ? (va ? k_stress_fwd_vec<true, 1, 6, VEC_STEP_TO> : k_stress_fwd_vec<false, 1, 6, VEC_STEP_TO>)
           : parts > 1 ? (va ? k_stress_fwd_vec<true, 4, 8> : k_stress_fwd_vec<false, 4, 8>)
                       : (va ? k_stress_fwd_vec<true, 1, 6> : k_stress_fwd_vec<false, 1, 6>);
  vec_launch(k, grid, vec_tz(parts) * parts, after_velocity, st, g, f, ps, lam, mu, nzb, src, shell, il, to);
}

void launch_velocity_fwd_vec(int S, cudaStream_t st, const Geo &g, const Fields &f, const Psi &ps,
                             const float *buoy, const RecFuse &rec, const IllumSum &il, const StepTo &to) {
  const int mode = il.first ? VEC_ILLUM : to.out ? VEC_STEP_TO : VEC_STEP;
  const int parts = mode == VEC_STEP && vec_split(g, S) ? 3 : 1;
  const dim3 grid = vec_grid(g, S, parts);
  const int nzb = grid.z / S;
  const bool va = psi_vectors(g);
  auto k = mode == VEC_ILLUM ? (va ? k_velocity_fwd_vec<true, 1, 5, VEC_ILLUM> : k_velocity_fwd_vec<false, 1, 5, VEC_ILLUM>)
           : mode == VEC_STEP_TO ? (va ? k_velocity_fwd_vec<true, 1, 5, VEC_STEP_TO> : k_velocity_fwd_vec<false, 1, 5, VEC_STEP_TO>)
           : parts > 1 ? (va ? k_velocity_fwd_vec<true, 3, 8> : k_velocity_fwd_vec<false, 3, 8>)
                       : (va ? k_velocity_fwd_vec<true, 1, 5> : k_velocity_fwd_vec<false, 1, 5>);
  vec_launch(k, grid, vec_tz(parts) * parts, true, st, g, f, ps, buoy, nzb, rec, il, to);
}

}  // namespace efwi
