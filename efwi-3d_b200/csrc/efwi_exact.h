// Exact discrete adjoint kernels (efwi_exact.cu).
#pragma once
#include "efwi_common.cuh"
#include "efwi_kernels.h"

namespace efwi {

// Adjoint of one C-PML-modified derivative (see efwi_exact.cu).
__device__ __forceinline__ float qpml(float G, bool slab, float L, float kinv, float a) {
  return slab ? G * kinv + a * (L + G) : G;
}

// Transpose of the quirk-Q1 difference over the rows x, x+1, x+2.
__device__ __forceinline__ float dq_t(float p0, float p1, float p2) {
  return EFWI_C1 * p0 - (EFWI_C1 + EFWI_C2) * p1 + EFWI_C2 * p2;
}


struct ExactArgs {
  Geo g;
  Fields f;        // forward state S_k (read), rows of
  int pitch_f;     // this pitch (the one-cell kernels: the grid's)
  Psi ps;          // forward memory variables of S_k (read)
  Fields a;        // adjoint fields (updated in place)
  Psi lin, lout;   // adjoint memory variables: read from lin, written to lout
  const float *lam, *mu, *buoy;
  float *g0, *g1;  // images: stress stage (lambda, mu); velocity stage (buoyancy, unused)
};

// Transpose of the stress stage of step k (+ lambda/mu images), then of the
// velocity stage of step k-1 (+ buoyancy image); the grid is
// (ceil(ny/32), ceil(nx/bx), ceil(nz/zchunk)) with 32 x bx threads, bx 4 or 8.
void launch_adj_stress_exact(int bx, dim3 grid, cudaStream_t st, const ExactArgs &A, int zchunk,
                             int nzc);
void launch_adj_velocity_exact(int bx, dim3 grid, cudaStream_t st, const ExactArgs &A, int zchunk,
                               int nzc);
// One thread per four cells (efwi_exact_vec.cu).
void launch_adj_stress_vec(cudaStream_t st, const ExactArgs &A);
void launch_adj_velocity_vec(cudaStream_t st, const ExactArgs &A);

__global__ void k_buoy_to_rho(const float *gB, const float *buoy, float *grho, int nz, int nx,
                              int ny, int py);
__global__ void k_stf_gradient(Fields a, const long long *src_cell, const float *w2, float *out,
                               int k, float scale);
__global__ void k_state_convert(Geo g, float *full, Fields f, Psi ps, int to_engine);
__global__ void k_illum_reduce(IllumSum il, int S, long long n);
__global__ void k_illumination(Geo g, Fields f, Psi ps, int S, const float *buoy, int do_stress,
                               float *hl, float *hm, float *hb);
__global__ void k_buoy_to_rho_sq(float *hb, const float *buoy, int nz, int nx, int ny, int py);

}  // namespace efwi
