// 3-D convolutions of the learned gradient preconditioner on BF16 tensor
// cores with FP32 accumulation (no reference counterpart).
//
// Layer: 3x3x3 kernel, stride 1, zero padding 1, 16 input and 16 output
// channels (narrower inputs and outputs are zero-padded to 16 by the
// caller).  Layouts:
//   activations  [D][H][W][16] bf16 (channels last: one voxel = 32 bytes)
//   weights      [27][16 co][16 ci] bf16, tap t = (dz+1)*9 + (dy+1)*3 + (dx+1)
//   bias         [16] f32
// Voxels outside the volume read as zero.  With W'[t][a][b] = W[26-t][b][a]
// the forward convolution also computes the gradient of the input (the
// transposed convolution).
//
// Kernels (efwi_conv3d_set_kernel / efwi_conv3d_set_wgrad_kernel choose):
//   k_conv3d_fwd_zm   forward on tcgen05.mma (the default): tiles of 8 x 16
//                     voxels march through z, one MMA per (dy, dx) for the
//                     three dz, accumulators in tensor memory, input planes
//                     staged by bulk tensor copies
//   k_conv3d_fwd_tc2  per tile of 128 voxels one MMA per tap, input tiles
//                     staged by bulk tensor copies
//   k_conv3d_fwd_ws   the same, warp-specialised (copy + MMA warp, four
//                     epilogue warps)
//   k_conv3d_fwd_tc   the same MMAs, tiles staged by plain loads
//   k_conv3d_fwd      forward on mma.sync.m16n8k16: per output row of 16
//                     voxels one warp, A fragments by ldmatrix
//   k_conv3d_wgrad_tc dW[t][co][ci] = sum_u dy[u - off_t][co] x[u][ci] on
//                     tcgen05.mma (the default): the (dy, dz) of the taps
//                     stacked on the MMA's rows, the dx on its columns,
//                     K = voxels
//   k_conv3d_wgrad    the same on mma.sync: one warp per tap
// Both weight gradients leave per-CTA partial sums that k_reduce_partials
// adds in a fixed order.
#include <cuda.h>
#include <cudaTypedefs.h>
#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <stdint.h>

#include <algorithm>
#include <atomic>

#include "efwi_tma.cuh"

namespace efwi {
namespace {

__device__ __forceinline__ void mma_bf16_16816(float c[4], const uint32_t a[4], uint32_t b0,
                                               uint32_t b1) {
  asm volatile(
      "mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 "
      "{%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, {%0, %1, %2, %3};\n"
      : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
      : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}

__device__ __forceinline__ uint32_t ld32(const __nv_bfloat16 *p) {
  return *reinterpret_cast<const uint32_t *>(p);
}
__device__ __forceinline__ uint32_t ld16(const __nv_bfloat16 *p) {
  return (uint32_t)(*reinterpret_cast<const unsigned short *>(p));
}

constexpr int kC = 16;              // channels
constexpr int kRowsFwd = 8;   // warps per CTA of k_conv3d_fwd: one y row each
constexpr int kTileX = 16;    // voxels per warp row
constexpr int kVoxPitch = 48; // bytes per staged voxel (32 of data): ldmatrix rows hit
                              // distinct banks
constexpr int kTileVox = 3 * (kRowsFwd + 2) * (kTileX + 2);

__device__ __forceinline__ void ldmatrix_x4(uint32_t a[4], uint32_t addr) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0, %1, %2, %3}, [%4];\n"
               : "=r"(a[0]), "=r"(a[1]), "=r"(a[2]), "=r"(a[3])
               : "r"(addr));
}

// A CTA computes the voxels (z, y0 .. y0+7, x0 .. x0+15).  Its input with a
// 1-voxel halo (3 x 10 x 18 voxels) is staged in shared memory once; each
// warp then takes, per tap, the 16 x 16 A fragment of its row with one
// ldmatrix.x4 (matrices: voxels 0-7 / 8-15 x channels 0-7 / 8-15, which is
// the register order of the mma A operand).
__global__ void __launch_bounds__(32 * kRowsFwd)
k_conv3d_fwd(const __nv_bfloat16 *__restrict__ x, const __nv_bfloat16 *__restrict__ w,
             const float *__restrict__ bias, int D, int H, int W, int relu,
             __nv_bfloat16 *__restrict__ yb, float *__restrict__ yf) {
  __shared__ __align__(16) uint32_t sw[27 * kC * kC / 2];  // [t][co][ci pair]
  __shared__ __align__(16) unsigned char sx[kTileVox * kVoxPitch];
  const int tid = threadIdx.x;
  const int x0 = blockIdx.x * kTileX, y0 = blockIdx.y * kRowsFwd, z = blockIdx.z;
  // w and yb may lie on 2-byte boundaries (the tcgen05 forms' unaligned calls
  // come here)
  const bool w4 = ((uintptr_t)w & 3) == 0, y4 = ((uintptr_t)yb & 3) == 0;
  for (int k = tid; k < 27 * kC * kC / 2; k += blockDim.x)
    sw[k] = w4 ? ld32(w + 2 * k) : ld16(w + 2 * k) | (ld16(w + 2 * k + 1) << 16);
  for (int c = tid; c < 2 * kTileVox; c += blockDim.x) {
    const int v = c >> 1, h = c & 1;
    const int xx = v % (kTileX + 2), t = v / (kTileX + 2);
    const int yy = t % (kRowsFwd + 2), zz = t / (kRowsFwd + 2);
    const int gz = z - 1 + zz, gy = y0 - 1 + yy, gx = x0 - 1 + xx;
    uint4 val = make_uint4(0u, 0u, 0u, 0u);
    if (gz >= 0 && gz < D && gy >= 0 && gy < H && gx >= 0 && gx < W)
      val = *reinterpret_cast<const uint4 *>(x + (((long long)gz * H + gy) * W + gx) * kC + h * 8);
    *reinterpret_cast<uint4 *>(sx + v * kVoxPitch + h * 16) = val;
  }
  __syncthreads();
  const int lane = tid & 31, warp = tid >> 5;
  const int y = y0 + warp;
  if (y >= H) return;  // no barrier follows
  const int g = lane >> 2, q = lane & 3;
  const uint32_t sxa = (uint32_t)__cvta_generic_to_shared(sx);
  const int lrow = ((lane >> 3) & 1) * 8 + (lane & 7);  // voxel of this lane's ldmatrix row
  const int lcol = (lane >> 4) * 16;                      // channel half (bytes)

  float c[2][4] = {{0.f, 0.f, 0.f, 0.f}, {0.f, 0.f, 0.f, 0.f}};
#pragma unroll
  for (int dz = 0; dz < 3; ++dz) {
#pragma unroll
    for (int dy = 0; dy < 3; ++dy) {
#pragma unroll
      for (int dx = 0; dx < 3; ++dx) {
        const int t = dz * 9 + dy * 3 + dx;
        const int v0 = (dz * (kRowsFwd + 2) + warp + dy) * (kTileX + 2) + dx;
        uint32_t a[4];
        ldmatrix_x4(a, sxa + (uint32_t)((v0 + lrow) * kVoxPitch + lcol));
#pragma unroll
        for (int nt = 0; nt < 2; ++nt) {
          const uint32_t *wb = sw + (t * kC + nt * 8 + g) * (kC / 2);
          mma_bf16_16816(c[nt], a, wb[q], wb[q + 4]);
        }
      }
    }
  }
  // epilogue: c[nt][0..1] -> voxel x0+g, channels nt*8 + 2q, +1; [2..3] -> voxel x0+g+8
#pragma unroll
  for (int nt = 0; nt < 2; ++nt) {
    const int co = nt * 8 + 2 * q;
    const float b0 = bias ? bias[co] : 0.f, b1 = bias ? bias[co + 1] : 0.f;
#pragma unroll
    for (int hh = 0; hh < 2; ++hh) {
      const int xv = x0 + g + 8 * hh;
      if (xv >= W) continue;
      float o0 = c[nt][2 * hh] + b0, o1 = c[nt][2 * hh + 1] + b1;
      if (relu) { o0 = fmaxf(o0, 0.f); o1 = fmaxf(o1, 0.f); }
      const long long off = (((long long)z * H + y) * W + xv) * kC + co;
      if (yb && y4) {
        *reinterpret_cast<__nv_bfloat162 *>(yb + off) = __floats2bfloat162_rn(o0, o1);
      } else if (yb) {
        yb[off] = __float2bfloat16_rn(o0);
        yb[off + 1] = __float2bfloat16_rn(o1);
      }
      if (yf) { yf[off] = o0; yf[off + 1] = o1; }
    }
  }
}

// One CTA of 27 warps (warp t = tap t) sums dW over a contiguous range of
// voxel rows; partial[cta][t][co][ci].
__global__ void __launch_bounds__(27 * 32)
k_conv3d_wgrad(const __nv_bfloat16 *__restrict__ x, const __nv_bfloat16 *__restrict__ dy,
               int D, int H, int W, float *__restrict__ partial) {
  const int lane = threadIdx.x & 31, t = threadIdx.x >> 5;
  const int g = lane >> 2, q = lane & 3;
  const int dz = t / 9 - 1, dyy = (t / 3) % 3 - 1, dx = t % 3 - 1;
  const int nxc = (W + 15) >> 4;
  const long long units = (long long)D * H * nxc;
  const long long u0 = units * blockIdx.x / gridDim.x, u1 = units * (blockIdx.x + 1) / gridDim.x;
  float c[2][4] = {{0.f, 0.f, 0.f, 0.f}, {0.f, 0.f, 0.f, 0.f}};
  for (long long u = u0; u < u1; ++u) {
    const int xc = (int)(u % nxc);
    const long long zy = u / nxc;
    const int y = (int)(zy % H), z = (int)(zy / H);
    const int zz = z + dz, yy = y + dyy;
    if (zz < 0 || zz >= D || yy < 0 || yy >= H) continue;
    const int x0 = xc * 16;
    const __nv_bfloat16 *grow = dy + ((long long)z * H + y) * W * kC;
    const __nv_bfloat16 *xrow = x + ((long long)zz * H + yy) * W * kC;
    // A (co x voxel): register r holds voxels (2q, 2q+1) (+8 for r = 2, 3)
    // of channel g (r = 0, 2) or g + 8 (r = 1, 3).
    const int va = x0 + 2 * q, vb = va + 8;
    uint32_t a[4];
    {
      const bool a0 = va < W, a1 = va + 1 < W, b0 = vb < W, b1 = vb + 1 < W;
      const uint32_t p00 = a0 ? ld16(grow + va * kC + g) : 0u, p01 = a1 ? ld16(grow + (va + 1) * kC + g) : 0u;
      const uint32_t p10 = a0 ? ld16(grow + va * kC + g + 8) : 0u, p11 = a1 ? ld16(grow + (va + 1) * kC + g + 8) : 0u;
      const uint32_t p20 = b0 ? ld16(grow + vb * kC + g) : 0u, p21 = b1 ? ld16(grow + (vb + 1) * kC + g) : 0u;
      const uint32_t p30 = b0 ? ld16(grow + vb * kC + g + 8) : 0u, p31 = b1 ? ld16(grow + (vb + 1) * kC + g + 8) : 0u;
      a[0] = p00 | (p01 << 16);
      a[1] = p10 | (p11 << 16);
      a[2] = p20 | (p21 << 16);
      a[3] = p30 | (p31 << 16);
    }
    // B (voxel x ci): voxels 2q, 2q+1 (b0) and 2q+8, 2q+9 (b1), shifted by dx
    const int sa = va + dx, sb = vb + dx;
    const bool s0 = sa >= 0 && sa < W && va < W, s1 = sa + 1 >= 0 && sa + 1 < W && va + 1 < W;
    const bool s2 = sb >= 0 && sb < W && vb < W, s3 = sb + 1 >= 0 && sb + 1 < W && vb + 1 < W;
#pragma unroll
    for (int nt = 0; nt < 2; ++nt) {
      const int ci = nt * 8 + g;
      const uint32_t e0 = s0 ? ld16(xrow + sa * kC + ci) : 0u, e1 = s1 ? ld16(xrow + (sa + 1) * kC + ci) : 0u;
      const uint32_t e2 = s2 ? ld16(xrow + sb * kC + ci) : 0u, e3 = s3 ? ld16(xrow + (sb + 1) * kC + ci) : 0u;
      mma_bf16_16816(c[nt], a, e0 | (e1 << 16), e2 | (e3 << 16));
    }
  }
  // C (co x ci): c[nt][0..1] -> co g, ci nt*8 + 2q, +1; [2..3] -> co g + 8
  float *out = partial + ((long long)blockIdx.x * 27 + t) * kC * kC;
#pragma unroll
  for (int nt = 0; nt < 2; ++nt) {
    const int ci = nt * 8 + 2 * q;
    out[g * kC + ci] = c[nt][0];
    out[g * kC + ci + 1] = c[nt][1];
    out[(g + 8) * kC + ci] = c[nt][2];
    out[(g + 8) * kC + ci + 1] = c[nt][3];
  }
}

// out[i] = sum over the CTAs' partial sums, in a fixed order: warp w of a CTA
// adds the partials w, w + 32, ... of 32 outputs (one 128-byte line each), the
// warps' sums are added in warp order.  Latency bounds it: one thread per
// output, reading all partials one after the other, took 40 us for 592 of
// them; 8 warps 9 us for 296, 32 warps 5.
constexpr int kRedWarps = 32;
struct Partials {
  const float *p;  // [parts][n]
  int parts, n;
  float *out;
};
// Blocks [0, ceil(a.n / 32)) reduce a, the rest b.
__global__ void __launch_bounds__(32 * kRedWarps) k_reduce_partials(Partials a, Partials b) {
  __shared__ float sum[kRedWarps][32];
  const int na = (a.n + 31) / 32;
  const bool second = (int)blockIdx.x >= na;
  const Partials r = second ? b : a;
  const int i = ((int)blockIdx.x - (second ? na : 0)) * 32 + threadIdx.x, w = threadIdx.y;
  float s = 0.f;
  if (i < r.n) {
#pragma unroll 8
    for (int p = w; p < r.parts; p += kRedWarps) s += r.p[(long long)p * r.n + i];
  }
  sum[w][threadIdx.x] = s;
  __syncthreads();
  if (w == 0 && i < r.n) {
#pragma unroll
    for (int k = 1; k < kRedWarps; ++k) s += sum[k][threadIdx.x];
    r.out[i] = s;
  }
}

// What the backward pass of a layer needs before its two convolutions, in one
// pass over the volume: the gradient behind the ReLU, g = gy * (y > 0) in
// float32 (rounded to BF16 into `dy`), per-CTA sums of g over the voxels (the
// bias gradient) and the weights of the transposed convolution,
// wt[t][a][b] = w[26-t][b][a].  A thread takes 8 channels of a voxel, the same
// half for all its voxels (an even number of threads).
constexpr int kPrepThreads = 256;
template <class T>
__device__ __forceinline__ void ld8(const T *p, float v[8]);
template <>
__device__ __forceinline__ void ld8(const __nv_bfloat16 *p, float v[8]) {
  const uint4 r = *reinterpret_cast<const uint4 *>(p);
  const uint32_t u[4] = {r.x, r.y, r.z, r.w};
#pragma unroll
  for (int k = 0; k < 4; ++k) {
    v[2 * k] = __uint_as_float(u[k] << 16);
    v[2 * k + 1] = __uint_as_float(u[k] & 0xffff0000u);
  }
}
template <>
__device__ __forceinline__ void ld8(const float *p, float v[8]) {
  const float4 a = *reinterpret_cast<const float4 *>(p), b = *reinterpret_cast<const float4 *>(p + 4);
  v[0] = a.x; v[1] = a.y; v[2] = a.z; v[3] = a.w;
  v[4] = b.x; v[5] = b.y; v[6] = b.z; v[7] = b.w;
}
// A gradient of channel 0 alone, [voxel] f32: the others are zero.
struct Head {
  float v;
};
template <class T>
__device__ __forceinline__ void ld8_at(const T *p, long long i, float v[8]) {
  ld8(p + 8 * i, v);
}
template <>
__device__ __forceinline__ void ld8_at(const Head *p, long long i, float v[8]) {
#pragma unroll
  for (int q = 0; q < 8; ++q) v[q] = 0.f;
  if ((i & 1) == 0) v[0] = p[i >> 1].v;
}
template <class TG, class TY>
__global__ void __launch_bounds__(kPrepThreads)
k_conv3d_grad_prep(const TG *__restrict__ gy, const TY *__restrict__ y, long long nhalf,
                   __nv_bfloat16 *__restrict__ dy, float *__restrict__ dbp,
                   const __nv_bfloat16 *__restrict__ w, __nv_bfloat16 *__restrict__ wt) {
  __shared__ float red[kPrepThreads][9];
  const int tid = threadIdx.x;
  if (wt)
    for (int k = blockIdx.x * kPrepThreads + tid; k < 27 * kC * kC; k += gridDim.x * kPrepThreads) {
      const int t = k / (kC * kC), a = k / kC % kC, b = k % kC;
      wt[k] = w[((26 - t) * kC + b) * kC + a];
    }
  float s[8];
#pragma unroll
  for (int q = 0; q < 8; ++q) s[q] = 0.f;
  for (long long i = blockIdx.x * (long long)kPrepThreads + tid; i < nhalf;
       i += (long long)gridDim.x * kPrepThreads) {
    float g[8];
    ld8_at(gy, i, g);
    if (y) {
      float v[8];
      ld8(y + 8 * i, v);
#pragma unroll
      for (int q = 0; q < 8; ++q) g[q] *= v[q] > 0.f ? 1.f : 0.f;
    }
#pragma unroll
    for (int q = 0; q < 8; ++q) s[q] += g[q];
    if (dy) {
      uint32_t pk[4];
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        const __nv_bfloat162 b2 = __floats2bfloat162_rn(g[2 * q], g[2 * q + 1]);
        pk[q] = *reinterpret_cast<const uint32_t *>(&b2);
      }
      *reinterpret_cast<uint4 *>(dy + 8 * i) = make_uint4(pk[0], pk[1], pk[2], pk[3]);
    }
  }
#pragma unroll
  for (int q = 0; q < 8; ++q) red[tid][q] = s[q];
  __syncthreads();
  for (int n = kPrepThreads / 2; n >= 2; n >>= 1) {  // even strides keep the channel half
    if (tid < n)
#pragma unroll
      for (int q = 0; q < 8; ++q) red[tid][q] += red[tid + n][q];
    __syncthreads();
  }
  if (tid < kC) dbp[(long long)blockIdx.x * kC + tid] = red[tid >> 3][tid & 7];
}


// ------------------------------------------------------------- tcgen05 form
// The forward convolution on the 5th-generation tensor cores: per tile of
// 128 voxels (8 x by 16 y at one z) and tap t, D[128 voxels][16 co] +=
// A_t[128][16 ci] B_t[16 ci][16 co] with one tcgen05.mma.kind::f16 (M 128,
// N 16, K 16; BF16 operands from shared memory, FP32 accumulator in TMEM).
// The CTA's input tile with its 1-voxel halo (3 x 18 x 10 voxels) is staged
// as two planes of 16-byte chunks (channels 0-7, channels 8-15), x fastest,
// so that A_t is the canonical K-major, non-swizzled operand at a shifted
// base: core matrices of 8 rows (8 consecutive x) x 16 bytes, the 16 rows
// of the tile one staged row apart (SBO = 10 x 16 B), the two K halves one
// plane apart (LBO).  B_t is staged the same way ([t][half][co][8 ci]).  One
// thread issues the 27 MMAs and commits them to an mbarrier; each warp then
// reads its 32 TMEM lanes (32 voxels x 16 fp32 columns) with tcgen05.ld.
// CTAs are persistent (the weights are staged once per CTA) and hold 32 TMEM
// columns each, allocated on entry and freed on exit.
constexpr int kTcX = 8, kTcY = 16;                   // tile: 128 voxels
constexpr int kTcSX = kTcX + 2, kTcSY = kTcY + 2;    // staged with the halo
constexpr int kTcVox = 3 * kTcSY * kTcSX;            // 540 staged voxels
constexpr int kTcPlane = kTcVox * 16;                // bytes of one channel-half plane
constexpr int kTcWBytes = 27 * 2 * kC * 16;          // staged weights
constexpr int kTcSmem = 2 * kTcPlane + kTcWBytes;

// Shared-memory matrix descriptor of tcgen05.mma: start address, leading
// (K) and stride (M/N) byte offsets, descriptor version 1, no swizzle.
__device__ __forceinline__ uint64_t tc_desc(uint32_t saddr, uint32_t lbo, uint32_t sbo) {
  return (uint64_t)((saddr >> 4) & 0x3FFFu) | ((uint64_t)((lbo >> 4) & 0x3FFFu) << 16) |
         ((uint64_t)((sbo >> 4) & 0x3FFFu) << 32) | (1ull << 46);
}

// Instruction descriptor of kind::f16: FP32 accumulator, BF16 A and B, both
// K-major, N = 16, M = 128.
constexpr uint32_t kTcIdesc = (1u << 4) | (1u << 7) | (1u << 10) | ((16u >> 3) << 17) |
                              ((128u >> 4) << 24);

__device__ __forceinline__ void tc_mma(uint32_t d, uint64_t a, uint64_t b, uint32_t acc) {
  asm volatile(
      "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}\n" ::"r"(d),
      "l"(a), "l"(b), "r"(kTcIdesc), "r"(acc));
}

__device__ __forceinline__ void tc_commit(uint64_t *bar) {
  asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(
                   smem_u32(bar))
               : "memory");
}

__device__ __forceinline__ void tc_ld16(uint32_t taddr, float v[16]) {
  uint32_t r[16];
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, "
      "%11, %12, %13, %14, %15}, [%16];"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]),
        "=r"(r[7]), "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]),
        "=r"(r[14]), "=r"(r[15])
      : "r"(taddr));
  asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
  for (int k = 0; k < 16; ++k) v[k] = __uint_as_float(r[k]);
}

__device__ int g_conv_status;  // EFWI_STATUS_TIMEOUT after a wait that ran out

// The 27 MMAs of one tile into the accumulator at TMEM address d: the
// descriptors of tap t are the tap-0 ones with the start address moved by
// the tap's offset (the 14-bit start field cannot carry: shared addresses
// stay below 256 KB), so the unrolled loop issues one add per operand.
__device__ __forceinline__ void tc_tile_mmas(uint32_t d, uint32_t sxa, uint32_t plane_bytes,
                                             uint32_t swa) {
  const uint64_t a0 = tc_desc(sxa, plane_bytes, kTcSX * 16);
  const uint64_t b0 = tc_desc(swa, kC * 16, 8 * 16);
#pragma unroll
  for (int t = 0; t < 27; ++t) {
    const int dz = t / 9, dy = (t / 3) % 3, dx = t % 3;
    const uint64_t ao = (uint64_t)((dz * kTcSY + dy) * kTcSX + dx);  // 16-byte units
    const uint64_t bo = (uint64_t)(t * 2 * kC);                      // 16-byte units
    tc_mma(d, a0 + ao, b0 + bo, t > 0 ? 1u : 0u);
  }
}

__global__ void __launch_bounds__(128)
k_conv3d_fwd_tc(const __nv_bfloat16 *__restrict__ x, const __nv_bfloat16 *__restrict__ w,
                const float *__restrict__ bias, int D, int H, int W, int relu,
                __nv_bfloat16 *__restrict__ yb, float *__restrict__ yf) {
  extern __shared__ __align__(128) unsigned char smem[];
  __shared__ __align__(8) uint64_t bar;
  __shared__ uint32_t tmem_slot;
  unsigned char *sx = smem;                     // [half][z][y][x] x 16 B
  unsigned char *swt = smem + 2 * kTcPlane;     // [t][half][co] x 16 B
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  for (int k = tid; k < 27 * 2 * kC; k += blockDim.x) {
    const int t = k / (2 * kC), r = k % (2 * kC), h = r / kC, co = r % kC;
    *reinterpret_cast<uint4 *>(swt + ((t * 2 + h) * kC + co) * 16) =
        *reinterpret_cast<const uint4 *>(w + (t * kC + co) * kC + h * 8);
  }
  if (warp == 0) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], 32;" ::"r"(
                     smem_u32(&tmem_slot))
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  if (tid == 0) {
    mbar_init(&bar, 1);
    fence_mbar_init();
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  const uint32_t tmem = tmem_slot;
  const uint32_t sxa = smem_u32(sx), swa = smem_u32(swt);
  float bv[16];
#pragma unroll
  for (int k = 0; k < 16; ++k) bv[k] = bias ? bias[k] : 0.f;
  const int ntx = (W + kTcX - 1) / kTcX, nty = (H + kTcY - 1) / kTcY;
  const long long ntiles = (long long)ntx * nty * D;
  int phase = 0;
  bool ok = true;
  for (long long tile = blockIdx.x; tile < ntiles && ok; tile += gridDim.x) {
    const int tx = (int)(tile % ntx);
    const long long r = tile / ntx;
    const int ty = (int)(r % nty), z = (int)(r / nty);
    const int x0 = tx * kTcX, y0 = ty * kTcY;
    for (int c = tid; c < 2 * kTcVox; c += blockDim.x) {
      const int v = c >> 1, h = c & 1;
      const int xx = v % kTcSX, t2 = v / kTcSX;
      const int yy = t2 % kTcSY, zz = t2 / kTcSY;
      const int gz = z - 1 + zz, gy = y0 - 1 + yy, gx = x0 - 1 + xx;
      uint4 val = make_uint4(0u, 0u, 0u, 0u);
      if (gz >= 0 && gz < D && gy >= 0 && gy < H && gx >= 0 && gx < W)
        val = *reinterpret_cast<const uint4 *>(x + (((long long)gz * H + gy) * W + gx) * kC + h * 8);
      *reinterpret_cast<uint4 *>(sx + h * kTcPlane + v * 16) = val;
    }
    // the staged tile (generic-proxy writes) is read by the tensor cores
    fence_proxy_async_smem();
    __syncthreads();
    if (tid == 0) {
      asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
      tc_tile_mmas(tmem, sxa, kTcPlane, swa);
      tc_commit(&bar);
    }
    // every thread decides on the same value: tcgen05.ld is warp-collective
    const bool got = __syncthreads_and(mbar_wait_bounded(&bar, (uint32_t)phase));
    phase ^= 1;
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    if (got) {
      float v[16];
      tc_ld16(tmem + ((uint32_t)(warp * 32) << 16), v);
      const int m = warp * 32 + lane;
      const int xv = x0 + (m & 7), yv = y0 + (m >> 3);
      if (xv < W && yv < H) {
        const long long off = (((long long)z * H + yv) * W + xv) * kC;
        float o[16];
#pragma unroll
        for (int k = 0; k < 16; ++k) {
          o[k] = v[k] + bv[k];
          if (relu) o[k] = fmaxf(o[k], 0.f);
        }
        if (yb) {
          uint32_t pk[8];
#pragma unroll
          for (int k = 0; k < 8; ++k) {
            const __nv_bfloat162 b2 = __floats2bfloat162_rn(o[2 * k], o[2 * k + 1]);
            pk[k] = *reinterpret_cast<const uint32_t *>(&b2);
          }
          uint4 *dst = reinterpret_cast<uint4 *>(yb + off);
          dst[0] = make_uint4(pk[0], pk[1], pk[2], pk[3]);
          dst[1] = make_uint4(pk[4], pk[5], pk[6], pk[7]);
        }
        if (yf) {
          float4 *dst = reinterpret_cast<float4 *>(yf + off);
#pragma unroll
          for (int k = 0; k < 4; ++k) dst[k] = make_float4(o[4 * k], o[4 * k + 1], o[4 * k + 2], o[4 * k + 3]);
        }
      }
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();  // TMEM and the staged tile are free again
    ok = got;
  }
  if (!ok && tid == 0) {
    atomicExch(&g_conv_status, EFWI_STATUS_TIMEOUT);
    mbar_wait_bounded(&bar, (uint32_t)(phase ^ 1));  // the MMAs still in flight, bounded
  }
  __syncthreads();
  if (warp == 0)
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, 32;" ::"r"(tmem) : "memory");
}


// The same tile and MMAs with the input staged by bulk tensor copies and
// the work software-pipelined: while the warps drain tile j's accumulator,
// the tensor cores already work on tile j+1 (two accumulators of 16 TMEM
// columns, used in turn) and the copy engine fills stages ahead: the copies of
// tile j+2 are issued right after tile j+1's MMAs, into the third stage (it
// last held tile j-1, whose MMAs completed in the previous iteration).  The tensor map views x as [D][H][W][2 halves][8
// channels]; a box of 8 x 1 x 10 x 18 x 3 is one channel-half plane of the
// staged tile in exactly the layout above (zeros outside the volume), so
// each stage takes two copies.  Half planes start 128-byte aligned.
constexpr int kTc2Plane = (kTcPlane + 127) / 128 * 128;  // 8704
constexpr int kTc2Stage = 2 * kTc2Plane;
constexpr int kTc2Copy = 2 * kTcPlane;  // bytes the two copies deliver
template <int NS>
constexpr int tc2_smem() { return NS * kTc2Stage + kTcWBytes + 128; }  // + alignment slack

__device__ __forceinline__ void tma_load_5d(void *dst, const CUtensorMap *map, uint64_t *bar,
                                            int c0, int c1, int c2, int c3, int c4) {
  asm volatile(
      "cp.async.bulk.tensor.5d.shared::cluster.global.tile.mbarrier::complete_tx::bytes"
      " [%0], [%1, {%2, %3, %4, %5, %6}], [%7];" ::"r"(smem_u32(dst)),
      "l"(reinterpret_cast<uint64_t>(map)), "r"(c0), "r"(c1), "r"(c2), "r"(c3), "r"(c4),
      "r"(smem_u32(bar))
      : "memory");
}

__global__ void __launch_bounds__(128)
k_conv3d_fwd_tc2(const __grid_constant__ CUtensorMap xmap, const __nv_bfloat16 *__restrict__ w,
                 const float *__restrict__ bias, int D, int H, int W, int relu,
                 __nv_bfloat16 *__restrict__ yb, float *__restrict__ yf) {
  constexpr int NS = 3;  // stages
  extern __shared__ unsigned char smem_raw[];
  __shared__ __align__(8) uint64_t full[NS];  // stage filled (copies landed)
  __shared__ __align__(8) uint64_t done[2];   // accumulator b complete
  __shared__ uint32_t tmem_slot;
  __shared__ int s_abort;
  unsigned char *smem = smem_raw + ((128u - (smem_u32(smem_raw) & 127u)) & 127u);
  unsigned char *swt = smem + NS * kTc2Stage;  // [t][half][co] x 16 B
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int ntx = (W + kTcX - 1) / kTcX, nty = (H + kTcY - 1) / kTcY;
  const long long ntiles = (long long)ntx * nty * D;
  // tiles of this CTA: blockIdx.x + j * gridDim.x, j < nj
  const long long nj =
      (long long)blockIdx.x < ntiles ? (ntiles - blockIdx.x + gridDim.x - 1) / gridDim.x : 0;
  auto tile_origin = [&](long long j, int &x0, int &y0, int &z) {
    const long long tile = blockIdx.x + j * gridDim.x;
    x0 = (int)(tile % ntx) * kTcX;
    const long long r = tile / ntx;
    y0 = (int)(r % nty) * kTcY;
    z = (int)(r / nty);
  };
  const uint32_t swa = smem_u32(swt);
  uint32_t tmem = 0;
  // thread 0: copies of tile j into stage j % NS
  auto issue = [&](long long j) {
    int x0, y0, z;
    tile_origin(j, x0, y0, z);
    const int s = (int)(j % NS);
    mbar_arrive_expect_tx(&full[s], kTc2Copy);
    unsigned char *dst = smem + s * kTc2Stage;
    tma_load_5d(dst, &xmap, &full[s], 0, 0, x0 - 1, y0 - 1, z - 1);
    tma_load_5d(dst + kTc2Plane, &xmap, &full[s], 0, 1, x0 - 1, y0 - 1, z - 1);
  };
  // thread 0: the 27 MMAs of tile j into accumulator j & 1, once its stage landed
  auto mma = [&](long long j) -> bool {
    const int s = (int)(j % NS);
    if (!mbar_wait_bounded(&full[s], (uint32_t)((j / NS) & 1))) return false;
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    tc_tile_mmas(tmem + (uint32_t)((j & 1) * kC), smem_u32(smem + s * kTc2Stage), kTc2Plane, swa);
    tc_commit(&done[j & 1]);
    return true;
  };
  long long n_tma = 0, n_mma = 0;  // thread 0: tiles whose copies / MMAs were issued
  if (tid == 0) {
    for (int s = 0; s < NS; ++s) mbar_init(&full[s], 1);
    mbar_init(&done[0], 1);
    mbar_init(&done[1], 1);
    fence_mbar_init();
    s_abort = 0;
    for (; n_tma < 2 && n_tma < nj; ++n_tma) issue(n_tma);
  }
  for (int k = tid; k < 27 * 2 * kC; k += blockDim.x) {
    const int t = k / (2 * kC), r = k % (2 * kC), h = r / kC, co = r % kC;
    *reinterpret_cast<uint4 *>(swt + ((t * 2 + h) * kC + co) * 16) =
        *reinterpret_cast<const uint4 *>(w + (t * kC + co) * kC + h * 8);
  }
  float bv[16];
#pragma unroll
  for (int q = 0; q < 16; ++q) bv[q] = bias ? bias[q] : 0.f;
  if (warp == 0) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], 32;" ::"r"(
                     smem_u32(&tmem_slot))
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  fence_proxy_async_smem();  // the staged weights are read by the tensor cores
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  tmem = tmem_slot;
  if (tid == 0 && nj > 0) {
    if (mma(0)) n_mma = 1;
    else s_abort = 1;
  }
  __syncthreads();
  bool ok = !s_abort;
  for (long long j = 0; j < nj && ok; ++j) {
    if (tid == 0 && !s_abort) {
      // accumulator (j+1)&1 was drained in iteration j-1
      if (j + 1 < nj) {
        if (mma(j + 1)) n_mma = j + 2;
        else s_abort = 1;
      }
      if (!s_abort && j + 2 < nj) {
        issue(j + 2);
        n_tma = j + 3;
      }
    }
    // every thread takes the same branch: tcgen05.ld is warp-collective
    const bool got =
        __syncthreads_and(mbar_wait_bounded(&done[j & 1], (uint32_t)((j >> 1) & 1)));
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    if (got) {
      int x0, y0, z;
      tile_origin(j, x0, y0, z);
      float v[16];
      tc_ld16(tmem + ((uint32_t)(warp * 32) << 16) + (uint32_t)((j & 1) * kC), v);
      const int m = warp * 32 + lane;
      const int xv = x0 + (m & 7), yv = y0 + (m >> 3);
      if (xv < W && yv < H) {
        const long long off = (((long long)z * H + yv) * W + xv) * kC;
        float o[16];
#pragma unroll
        for (int q = 0; q < 16; ++q) {
          o[q] = v[q] + bv[q];
          if (relu) o[q] = fmaxf(o[q], 0.f);
        }
        if (yb) {
          uint32_t pk[8];
#pragma unroll
          for (int q = 0; q < 8; ++q) {
            const __nv_bfloat162 b2 = __floats2bfloat162_rn(o[2 * q], o[2 * q + 1]);
            pk[q] = *reinterpret_cast<const uint32_t *>(&b2);
          }
          uint4 *dst = reinterpret_cast<uint4 *>(yb + off);
          dst[0] = make_uint4(pk[0], pk[1], pk[2], pk[3]);
          dst[1] = make_uint4(pk[4], pk[5], pk[6], pk[7]);
        }
        if (yf) {
          float4 *dst = reinterpret_cast<float4 *>(yf + off);
#pragma unroll
          for (int q = 0; q < 4; ++q)
            dst[q] = make_float4(o[4 * q], o[4 * q + 1], o[4 * q + 2], o[4 * q + 3]);
        }
      }
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();  // accumulator j & 1 is free again; s_abort is published
    ok = got && !s_abort;
  }
  if (!ok && tid == 0) {
    atomicExch(&g_conv_status, EFWI_STATUS_TIMEOUT);
    // bounded waits for what may still be in flight: the copies of tiles
    // whose MMAs were never issued, and the last MMAs issued
    for (long long j = n_mma; j < n_tma; ++j)
      mbar_wait_bounded(&full[j % NS], (uint32_t)((j / NS) & 1));
    if (n_mma > 0) mbar_wait_bounded(&done[(n_mma - 1) & 1], (uint32_t)(((n_mma - 1) >> 1) & 1));
  }
  __syncthreads();
  if (warp == 0)
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, 32;" ::"r"(tmem) : "memory");
}


// z-marching form (the default).  What bounds the forms above is the operand
// path: every input voxel is read 27 times, for an MMA of N = 16.  Here a CTA
// marches the 8 x 16 tile through z, one staged input plane z' at a time, and
// one MMA per (dy, dx) multiplies it with the weights of all three dz at once:
// N = 48 = (output planes z'-1, z', z'+1) x 16 channels, so that a voxel is
// read 9 times.  Output plane p accumulates in TMEM columns 16 (p mod 3); the
// weights of one (dy, dx) lie in blocks of 16 rows in the dz order 2 1 0 2 1,
// of which an MMA takes three from block (1 - z') mod 3.  After plane z' the
// tile of plane z'-1 is complete: the warps read it, set its columns to zero
// for plane z'+2 and hand over to the next MMAs before they store.  A plane's
// sums see the taps in the same order as in the forms above (the same bits).
// What bounds it now is the tensor cores' reads of shared memory (44 of the
// SM's cycles per MMA: 25 us of the 39 at 128^3) and, with few tiles in flight,
// the chain from one plane's MMAs over its drain to the next plane's.  So a CTA
// has four tiles of four warps each that share the weights and nothing else
// (a barrier of their own per tile): 70 KB of shared memory, two CTAs or eight
// tiles per SM, all 512 TMEM columns.  One tile per CTA fits six times: 49 /
// 118 us at 128^3 / 192^3, 41 at 93 x 117 x 141; two per CTA 40 / 108, 36; four
// 39 / 106, 33; a third stage changes nothing.
constexpr int kZmStages = 2;
constexpr int kZmPlane = kTcSY * kTcSX * 32;                     // a staged plane
constexpr int kZmStage = (kZmPlane + 255) / 256 * 256;
constexpr int kZmWTap = 2 * 5 * kC * 16;                         // weights of one (dy, dx)
constexpr int kZmWBytes = 9 * kZmWTap;
constexpr int kZmTiles = 4;                                      // tiles of a CTA
constexpr int kZmSmem = kZmTiles * kZmStages * kZmStage + kZmWBytes + 256;  // + alignment slack

// kind::f16, FP32 accumulator, BF16 K-major operands, N = 48, M = 128.
constexpr uint32_t kZmIdesc = (1u << 4) | (1u << 7) | (1u << 10) | ((48u >> 3) << 17) |
                              ((128u >> 4) << 24);

__device__ __forceinline__ void tc_mma_idesc(uint32_t d, uint64_t a, uint64_t b, uint32_t idesc,
                                             uint32_t acc) {
  asm volatile(
      "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}\n" ::"r"(d),
      "l"(a), "l"(b), "r"(idesc), "r"(acc));
}

// Operand staged with the 32-byte swizzle of the bulk copies.  The pattern
// lies on 256-byte boundaries of shared memory, so an operand may start at
// any row of 32 bytes.
__device__ __forceinline__ uint64_t tc_desc_sw32(uint32_t saddr, uint32_t lbo, uint32_t sbo) {
  return tc_desc(saddr, lbo, sbo) | (6ull << 61);
}

__device__ __forceinline__ void tma_load_4d(void *dst, const CUtensorMap *map, uint64_t *bar,
                                            int c0, int c1, int c2, int c3) {
  asm volatile(
      "cp.async.bulk.tensor.4d.shared::cluster.global.tile.mbarrier::complete_tx::bytes"
      " [%0], [%1, {%2, %3, %4, %5}], [%6];" ::"r"(smem_u32(dst)),
      "l"(reinterpret_cast<uint64_t>(map)), "r"(c0), "r"(c1), "r"(c2), "r"(c3),
      "r"(smem_u32(bar))
      : "memory");
}

// Zeros in 16 TMEM columns of the warp's 32 lanes.
__device__ __forceinline__ void tc_zero16(uint32_t taddr) {
  asm volatile(
      "tcgen05.st.sync.aligned.32x32b.x16.b32 [%0], {%1, %1, %1, %1, %1, %1, %1, %1, %1, %1, "
      "%1, %1, %1, %1, %1, %1};" ::"r"(taddr),
      "r"(0)
      : "memory");
  asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
}

// Barriers of a tile's four warps; sync_and returns whether `ok` held for all
// their threads.  The warps leave them converged, as tcgen05.ld and .st need.
__device__ __forceinline__ void sync_128(int id) {
  __syncwarp();
  asm volatile("bar.sync %0, 128;" ::"r"(id) : "memory");
}
__device__ __forceinline__ bool sync_and(int id, bool ok) {
  int r;
  __syncwarp();
  asm volatile(
      "{\n\t.reg .pred p, q;\n\tsetp.ne.b32 p, %1, 0;\n\t"
      "bar.red.and.pred q, %2, 128, p;\n\tselp.b32 %0, 1, 0, q;\n\t}\n"
      : "=r"(r)
      : "r"((int)ok), "r"(id)
      : "memory");
  return r != 0;
}

__global__ void __launch_bounds__(128 * kZmTiles)
k_conv3d_fwd_zm(const __grid_constant__ CUtensorMap xmap, const __nv_bfloat16 *__restrict__ w,
                const float *__restrict__ bias, int D, int H, int W, int zlen, int units,
                int relu, __nv_bfloat16 *__restrict__ yb, float *__restrict__ yf,
                float *__restrict__ y0c) {
  extern __shared__ unsigned char smem_raw[];
  __shared__ __align__(8) uint64_t s_full[kZmTiles][kZmStages], s_done[kZmTiles];
  __shared__ uint32_t tmem_slot;
  __shared__ int s_abort_of[kZmTiles];
  unsigned char *smem = smem_raw + ((256u - (smem_u32(smem_raw) & 255u)) & 255u);
  // weights [dy][dx][half][5 dz blocks][co] x 16 B
  unsigned char *swt = smem + kZmTiles * kZmStages * kZmStage;
  const int tile = __shfl_sync(0xffffffffu, (int)(threadIdx.x >> 7), 0);
  const int tid = threadIdx.x & 127, warp = tid >> 5, lane = tid & 31;
  smem += tile * kZmStages * kZmStage;
  uint64_t *full = s_full[tile], &done = s_done[tile];
  int &s_abort = s_abort_of[tile];
  const int unit = (int)blockIdx.x * kZmTiles + tile;
  const int ntx = (W + kTcX - 1) / kTcX, nty = (H + kTcY - 1) / kTcY;
  const int x0 = unit % ntx * kTcX;
  const int rest = unit / ntx;
  const int y0 = rest % nty * kTcY, zb = rest / nty * zlen, ze = min(zb + zlen, D);
  const int nj = unit < units ? ze - zb + 2 : 0;  // input planes zb-1 .. ze
  auto issue = [&](int j) {    // thread 0: input plane zb-1+j into stage j % kZmStages
    const int s = j % kZmStages;
    mbar_arrive_expect_tx(&full[s], kZmPlane);
    tma_load_4d(smem + s * kZmStage, &xmap, &full[s], 0, x0 - 1, y0 - 1, zb - 1 + j);
  };
  int n_tma = 0;
  if (tid == 0) {
    for (int s = 0; s < kZmStages; ++s) mbar_init(&full[s], 1);
    mbar_init(&done, 1);
    fence_mbar_init();
    s_abort = 0;
    for (; n_tma < kZmStages && n_tma < nj; ++n_tma) issue(n_tma);
  }
  for (int k = threadIdx.x; k < 9 * 2 * 5 * kC; k += blockDim.x) {
    const int co = k % kC, b = k / kC % 5, h = k / (kC * 5) % 2, t = k / (kC * 10);
    const int dz = (5 - b) % 3;  // blocks in the order 2 1 0 2 1
    *reinterpret_cast<uint4 *>(swt + k * 16) =
        *reinterpret_cast<const uint4 *>(w + ((dz * 9 + t) * kC + co) * kC + h * 8);
  }
  if (threadIdx.x < 32) {  // one allocation: the permit is the CTA's
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(
                     smem_u32(&tmem_slot)),
                 "n"(64 * kZmTiles)
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  fence_proxy_async_smem();  // the staged weights are read by the tensor cores
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  const uint32_t tmem = tmem_slot + (uint32_t)(64 * tile),
                 tlane = tmem + ((uint32_t)(warp * 32) << 16);
  const uint32_t swa = smem_u32(swt);
  for (int s = 0; s < 3; ++s) tc_zero16(tlane + (uint32_t)(s * kC));
  float bv[16];
#pragma unroll
  for (int q = 0; q < 16; ++q) bv[q] = bias ? bias[q] : 0.f;
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();

  const int m = warp * 32 + lane;
  const int xv = x0 + (m & 7), yv = y0 + (m >> 3);
  const bool inside = xv < W && yv < H;
  int n_mma = 0;
  // thread 0: the nine MMAs of input plane j, once its stage landed
  auto mma = [&](int j) {
    const int s = j % kZmStages, z = zb - 1 + j;
    if (!mbar_wait_bounded(&full[s], (uint32_t)((j / kZmStages) & 1))) { s_abort = 1; return; }
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    const int b0 = ((1 - z) % 3 + 3) % 3;  // first weight block
    const uint64_t a = tc_desc_sw32(smem_u32(smem + s * kZmStage), 16, kTcSX * 32);
    const uint64_t b = tc_desc(swa + (uint32_t)(b0 * kC * 16), 5 * kC * 16, 8 * 16);
#pragma unroll
    for (int t = 0; t < 9; ++t)
      tc_mma_idesc(tmem, a + (uint64_t)(2 * ((t / 3) * kTcSX + t % 3)), b + (uint64_t)(t * (kZmWTap / 16)),
                   kZmIdesc, 1u);
    tc_commit(&done);
    n_mma = j + 1;
  };
  if (tid == 0 && nj > 0) mma(0);
  bool ok = true;
  for (int j = 0; j < nj; ++j) {
    // every thread takes the same branch: tcgen05.ld is warp-collective
    ok = sync_and(tile + 1, !s_abort && mbar_wait_bounded(&done, (uint32_t)(j & 1)));
    if (!ok) break;
    if (tid == 0 && n_tma < nj) { issue(n_tma); ++n_tma; }  // into plane j's stage
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    const int p = zb - 2 + j;  // the plane that is complete
    const uint32_t col = tlane + (uint32_t)((p + 3) % 3 * kC);
    float v[16];
    tc_ld16(col, v);
    if (j + 1 < nj) {
      tc_zero16(col);
      asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
      sync_128(tile + 1);
      if (tid == 0) mma(j + 1);
    }
    if (p >= zb && inside) {
      const long long off = (((long long)p * H + yv) * W + xv) * kC;
      float o[16];
#pragma unroll
      for (int q = 0; q < 16; ++q) {
        o[q] = v[q] + bv[q];
        if (relu) o[q] = fmaxf(o[q], 0.f);
      }
      if (y0c) y0c[((long long)p * H + yv) * W + xv] = o[0];
      if (yb) {
        uint32_t pk[8];
#pragma unroll
        for (int q = 0; q < 8; ++q) {
          const __nv_bfloat162 b2 = __floats2bfloat162_rn(o[2 * q], o[2 * q + 1]);
          pk[q] = *reinterpret_cast<const uint32_t *>(&b2);
        }
        uint4 *dst = reinterpret_cast<uint4 *>(yb + off);
        dst[0] = make_uint4(pk[0], pk[1], pk[2], pk[3]);
        dst[1] = make_uint4(pk[4], pk[5], pk[6], pk[7]);
      }
      if (yf) {
        float4 *dst = reinterpret_cast<float4 *>(yf + off);
#pragma unroll
        for (int q = 0; q < 4; ++q)
          dst[q] = make_float4(o[4 * q], o[4 * q + 1], o[4 * q + 2], o[4 * q + 3]);
      }
    }
  }
  if (!ok && tid == 0) {
    atomicExch(&g_conv_status, EFWI_STATUS_TIMEOUT);
    // bounded waits for what may still be in flight: the copies of planes
    // whose MMAs were never issued, and the last MMAs issued
    for (int j = n_mma; j < n_tma; ++j)
      mbar_wait_bounded(&full[j % kZmStages], (uint32_t)((j / kZmStages) & 1));
    if (n_mma > 0) mbar_wait_bounded(&done, (uint32_t)((n_mma - 1) & 1));
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  if (threadIdx.x < 32)
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem_slot),
                 "n"(64 * kZmTiles)
                 : "memory");
}


// Warp-specialised form of the copy-staged kernel: warp 0 (one elected
// thread) fills NS stages with bulk tensor copies and issues each tile's 27
// MMAs into one of two accumulators; warps 1-4 drain the accumulators
// (warp w reads TMEM lanes 32 (w % 4) .. + 31, so the four cover the 128
// rows).  The roles meet only at mbarriers -- stage full (copies landed),
// stage empty (its MMAs completed, committed by the MMA thread), accumulator
// full (committed) and accumulator empty (one arrival per epilogue warp
// after its tcgen05.ld) -- so no warp waits for the CTA at a barrier per
// tile.  Every wait is bounded: a role that gives up sets the status flag
// and a shared abort word that the other roles test once per tile; before
// TMEM is freed, thread 0 waits (bounded) for the copies and MMAs it issued.
constexpr int kWsThreads = 160;

__device__ __forceinline__ void mbar_arrive1(uint64_t *bar) {
  asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_u32(bar)) : "memory");
}

template <int NS>
__global__ void __launch_bounds__(kWsThreads)
k_conv3d_fwd_ws(const __grid_constant__ CUtensorMap xmap, const __nv_bfloat16 *__restrict__ w,
                const float *__restrict__ bias, int D, int H, int W, int relu,
                __nv_bfloat16 *__restrict__ yb, float *__restrict__ yf) {
  static_assert(NS >= 2 && NS <= 4, "two to four stages");
  extern __shared__ unsigned char smem_raw[];
  __shared__ __align__(8) uint64_t full[NS], empty[NS], tfull[2], tempty[2];
  __shared__ uint32_t tmem_slot;
  __shared__ volatile int s_abort;
  unsigned char *smem = smem_raw + ((128u - (smem_u32(smem_raw) & 127u)) & 127u);
  unsigned char *swt = smem + NS * kTc2Stage;  // [t][half][co] x 16 B
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int ntx = (W + kTcX - 1) / kTcX, nty = (H + kTcY - 1) / kTcY;
  const long long ntiles = (long long)ntx * nty * D;
  const long long nj =
      (long long)blockIdx.x < ntiles ? (ntiles - blockIdx.x + gridDim.x - 1) / gridDim.x : 0;
  auto tile_origin = [&](long long j, int &x0, int &y0, int &z) {
    const long long tile = blockIdx.x + j * gridDim.x;
    x0 = (int)(tile % ntx) * kTcX;
    const long long r = tile / ntx;
    y0 = (int)(r % nty) * kTcY;
    z = (int)(r / nty);
  };
  auto give_up = [&]() {
    s_abort = 1;
    atomicExch(&g_conv_status, EFWI_STATUS_TIMEOUT);
  };
  auto issue = [&](long long j) {  // thread 0: copies of tile j into stage j % NS
    int x0, y0, z;
    tile_origin(j, x0, y0, z);
    const int s = (int)(j % NS);
    mbar_arrive_expect_tx(&full[s], kTc2Copy);
    unsigned char *dst = smem + s * kTc2Stage;
    tma_load_5d(dst, &xmap, &full[s], 0, 0, x0 - 1, y0 - 1, z - 1);
    tma_load_5d(dst + kTc2Plane, &xmap, &full[s], 0, 1, x0 - 1, y0 - 1, z - 1);
  };
  long long jt = 0, jm = 0;  // thread 0: tiles whose copies / MMAs were issued
  if (tid == 0) {
    for (int s = 0; s < NS; ++s) {
      mbar_init(&full[s], 1);
      mbar_init(&empty[s], 1);
    }
    for (int b = 0; b < 2; ++b) {
      mbar_init(&tfull[b], 1);
      mbar_init(&tempty[b], 4);
    }
    fence_mbar_init();
    s_abort = 0;
    for (; jt < NS && jt < nj; ++jt) issue(jt);
  }
  for (int k = tid; k < 27 * 2 * kC; k += blockDim.x) {
    const int t = k / (2 * kC), r = k % (2 * kC), h = r / kC, co = r % kC;
    *reinterpret_cast<uint4 *>(swt + ((t * 2 + h) * kC + co) * 16) =
        *reinterpret_cast<const uint4 *>(w + (t * kC + co) * kC + h * 8);
  }
  if (warp == 0) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], 32;" ::"r"(
                     smem_u32(&tmem_slot))
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  fence_proxy_async_smem();  // the staged weights are read by the tensor cores
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  const uint32_t tmem = tmem_slot;
  const uint32_t swa = smem_u32(swt);

  if (warp == 0) {
    if (lane == 0) {  // copies and MMAs
      for (long long j = 0; j < nj; ++j) {
        if (s_abort) break;
        const int s = (int)(j % NS), b = (int)(j & 1);
        if (!mbar_wait_bounded(&full[s], (uint32_t)((j / NS) & 1))) { give_up(); break; }
        if (j >= 2 && !mbar_wait_bounded(&tempty[b], (uint32_t)(((j - 2) >> 1) & 1))) {
          give_up();
          break;
        }
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        tc_tile_mmas(tmem + (uint32_t)(b * kC), smem_u32(smem + s * kTc2Stage), kTc2Plane, swa);
        tc_commit(&tfull[b]);
        tc_commit(&empty[s]);
        jm = j + 1;
        // refill the stage of tile j-1 (its MMAs were issued one tile ago)
        if (j >= 1 && jt < nj) {
          const long long jp = j - 1;
          if (!mbar_wait_bounded(&empty[jp % NS], (uint32_t)((jp / NS) & 1))) { give_up(); break; }
          issue(jt);
          ++jt;
        }
      }
    }
  } else if (warp <= 4) {  // epilogue: TMEM lanes 32 (warp % 4) .. + 31
    const int q = warp & 3;
    float bv[16];
#pragma unroll
    for (int k = 0; k < 16; ++k) bv[k] = bias ? bias[k] : 0.f;
    for (long long j = 0; j < nj; ++j) {
      if (s_abort) break;
      const int b = (int)(j & 1);
      bool ok = mbar_wait_bounded(&tfull[b], (uint32_t)((j >> 1) & 1));
      ok = __all_sync(0xffffffffu, ok);  // tcgen05.ld is warp-collective
      if (!ok) {
        if (lane == 0) give_up();
        break;
      }
      asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
      float v[16];
      tc_ld16(tmem + ((uint32_t)(q * 32) << 16) + (uint32_t)(b * kC), v);
      asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
      __syncwarp();
      if (lane == 0) mbar_arrive1(&tempty[b]);
      int x0, y0, z;
      tile_origin(j, x0, y0, z);
      const int m = q * 32 + lane;
      const int xv = x0 + (m & 7), yv = y0 + (m >> 3);
      if (xv < W && yv < H) {
        const long long off = (((long long)z * H + yv) * W + xv) * kC;
        float o[16];
#pragma unroll
        for (int k = 0; k < 16; ++k) {
          o[k] = v[k] + bv[k];
          if (relu) o[k] = fmaxf(o[k], 0.f);
        }
        if (yb) {
          uint32_t pk[8];
#pragma unroll
          for (int k = 0; k < 8; ++k) {
            const __nv_bfloat162 b2 = __floats2bfloat162_rn(o[2 * k], o[2 * k + 1]);
            pk[k] = *reinterpret_cast<const uint32_t *>(&b2);
          }
          uint4 *dst = reinterpret_cast<uint4 *>(yb + off);
          dst[0] = make_uint4(pk[0], pk[1], pk[2], pk[3]);
          dst[1] = make_uint4(pk[4], pk[5], pk[6], pk[7]);
        }
        if (yf) {
          float4 *dst = reinterpret_cast<float4 *>(yf + off);
#pragma unroll
          for (int k = 0; k < 4; ++k)
            dst[k] = make_float4(o[4 * k], o[4 * k + 1], o[4 * k + 2], o[4 * k + 3]);
        }
      }
    }
  }
  __syncthreads();
  if (tid == 0) {
    // bounded waits for what thread 0 issued and nobody consumed: copies of
    // tiles whose MMAs were never issued, and the last MMAs (their commit)
    for (long long j = jm; j < jt; ++j) mbar_wait_bounded(&full[j % NS], (uint32_t)((j / NS) & 1));
    if (jm > 0) mbar_wait_bounded(&empty[(jm - 1) % NS], (uint32_t)(((jm - 1) / NS) & 1));
  }
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  __syncthreads();
  if (warp == 0)
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, 32;" ::"r"(tmem) : "memory");
}
// Weight gradient on tcgen05: dW[t][co][ci] = sum_w dy[w - dx][co]
// x[w + (dy, dz)][ci], the y and z shifts of a tap on x and its x shift on dy.
// K runs over voxels w, so both operands are "MN-major": a voxel's 16
// channels are contiguous, as in memory, and bulk tensor copies bring them
// to shared memory without a transposition (32-byte swizzle: rows of one
// voxel, blocks of 8 voxels of 256 bytes).
// A unit is 8 (x) x 16 (y) x 2 (z) voxels.  x is staged as [y 18][z 4][8 x],
// so the blocks of the taps (dy, dz) of one voxel row follow one another:
// block 4 dy' + dz' (dy' = dy + 1, dz' = dz + 1), the fourth of each four
// unused.  One MMA with M = 128 takes blocks 0-7, a second blocks 8-15 (of
// which 8-10 are taps).  dy is staged as [z][y][10 x]: the three x shifts are
// operands that start one voxel (32 bytes) apart, so that N = 48 = (2 - dx',
// co).  K = 16: two voxel rows.
// Two accumulators of 48 TMEM columns sum over a group of kWgGroup units;
// four warps then add them to sums in registers while the next group runs in
// a second pair: the tensor cores' accumulation truncates, so its error grows
// with the number of MMAs added in one go (at 93 x 117 x 141 the sums are
// 6e-6 off when a CTA's units stay in TMEM to the end).  The CTA's 27 x 16
// x 16 sums go to partial[cta] for the fixed-order reduction.  One thread of a
// fifth warp runs the copies (three stages) and the MMAs; every wait is
// bounded, and on a timeout the CTA sets the status flag and writes NaN
// partial sums.
constexpr int kWgX = 8, kWgY = 16, kWgZ = 2;          // voxels of a unit
constexpr int kWgZs = kWgZ + 2;                       // staged x planes
constexpr int kWgABytes = (kWgY + 2) * kWgZs * 256;   // staged x
constexpr int kWgGX = kWgX + 2;                       // staged dy: x with the shifts
constexpr int kWgCopied = kWgABytes + kWgZ * kWgY * kWgGX * 32;  // bytes of a stage
constexpr int kWgStage = (kWgCopied + 255) / 256 * 256;
constexpr int kWgStages = 3;
constexpr int kWgSmem = kWgStages * kWgStage + 1024;  // + alignment slack
constexpr int kWgThreads = 160;
constexpr int kWgGroup = 4;   // units per accumulator hand-over
constexpr int kWgCol2 = 64;  // first TMEM column of the second accumulator
// the second MMA of a unit's last rows reads past the staged x, into dy
static_assert(((kWgY - 2 + 1) * kWgZs + kWgZ - 1 + 16) * 256 <= kWgCopied, "in the stage");

// Both operands MN-major, N = 48, M = 128.
constexpr uint32_t kWgIdesc = (1u << 4) | (1u << 7) | (1u << 10) | (1u << 15) | (1u << 16) |
                              ((48u >> 3) << 17) | ((128u >> 4) << 24);

__global__ void __launch_bounds__(kWgThreads)
k_conv3d_wgrad_tc(const __grid_constant__ CUtensorMap xmap, const __grid_constant__ CUtensorMap gmap,
                  int D, int H, int W, float *__restrict__ partial) {
  extern __shared__ unsigned char smem_raw[];
  __shared__ __align__(8) uint64_t full[kWgStages], done[kWgStages], tfull[2], tempty[2];
  __shared__ uint32_t tmem_slot;
  __shared__ volatile int s_abort;
  unsigned char *smem = smem_raw + ((1024u - (smem_u32(smem_raw) & 1023u)) & 1023u);
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int nxw = (W + kWgX - 1) / kWgX, nyb = (H + kWgY - 1) / kWgY;
  const long long nunits = (long long)nxw * nyb * ((D + kWgZ - 1) / kWgZ);
  const long long nj =
      (long long)blockIdx.x < nunits ? (nunits - blockIdx.x + gridDim.x - 1) / gridDim.x : 0;
  const long long ng = (nj + kWgGroup - 1) / kWgGroup;
  if (warp == 0) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], 256;" ::"r"(
                     smem_u32(&tmem_slot))
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  if (tid == 0) {
    for (int s = 0; s < kWgStages; ++s) {
      mbar_init(&full[s], 1);
      mbar_init(&done[s], 1);
    }
    for (int b = 0; b < 2; ++b) {
      mbar_init(&tfull[b], 1);
      mbar_init(&tempty[b], 4);
    }
    fence_mbar_init();
    s_abort = 0;
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  const uint32_t tmem = tmem_slot;
  auto give_up = [&]() {
    s_abort = 1;
    atomicExch(&g_conv_status, EFWI_STATUS_TIMEOUT);
  };
  float sum[6][16];  // [2 accumulators x 3 shifts][co] of this thread's row
#pragma unroll
  for (int k = 0; k < 6; ++k)
#pragma unroll
    for (int q = 0; q < 16; ++q) sum[k][q] = 0.f;
  if (warp == 4) {
    if (lane == 0) {
      auto issue = [&](long long j) {
        const long long unit = blockIdx.x + j * gridDim.x;
        const int x0 = (int)(unit % nxw) * kWgX;
        const long long r = unit / nxw;
        const int y0 = (int)(r % nyb) * kWgY, z0 = (int)(r / nyb) * kWgZ;
        const int s = (int)(j % kWgStages);
        unsigned char *dst = smem + s * kWgStage;
        mbar_arrive_expect_tx(&full[s], kWgCopied);
        tma_load_4d(dst, &xmap, &full[s], 0, x0, z0 - 1, y0 - 1);
        tma_load_4d(dst + kWgABytes, &gmap, &full[s], 0, x0 - 1, y0, z0);
      };
      long long nt = 0, nm = 0;  // units whose copies / MMAs were issued
      for (; nt < kWgStages && nt < nj; ++nt) issue(nt);
      for (long long j = 0; j < nj && !s_abort; ++j) {
        const int s = (int)(j % kWgStages);
        const long long grp = j / kWgGroup;
        const int b = (int)(grp & 1);
        const bool first = j % kWgGroup == 0;
        // the accumulators of group grp - 2 have been drained
        if (first && grp >= 2 && !mbar_wait_bounded(&tempty[b], (uint32_t)(((grp - 2) >> 1) & 1))) {
          give_up();
          break;
        }
        if (!mbar_wait_bounded(&full[s], (uint32_t)((j / kWgStages) & 1))) { give_up(); break; }
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        const uint32_t a0 = smem_u32(smem + s * kWgStage), b0 = a0 + kWgABytes;
        const uint32_t acc0 = tmem + (uint32_t)(2 * kWgCol2 * b);
#pragma unroll 1
        for (int z = 0; z < kWgZ; ++z) {
          const uint64_t ad = tc_desc_sw32(a0 + z * 256, 256, kWgZs * 256);
          const uint64_t bd = tc_desc_sw32(b0 + z * kWgY * kWgGX * 32, 32, kWgGX * 32);
#pragma unroll
          for (int r = 0; r < kWgY; r += 2) {
            const uint32_t acc = (!first || z > 0 || r > 0) ? 1u : 0u;
            const uint64_t da = ad + (uint64_t)(r * kWgZs * 16), db = bd + (uint64_t)(r * kWgGX * 2);
            tc_mma_idesc(acc0, da, db, kWgIdesc, acc);
            tc_mma_idesc(acc0 + kWgCol2, da + 8 * 16, db, kWgIdesc, acc);
          }
        }
        tc_commit(&done[s]);
        if (j % kWgGroup == kWgGroup - 1 || j + 1 == nj) tc_commit(&tfull[b]);
        nm = j + 1;
        if (j >= 1 && nt < nj) {  // refill the stage of unit j-1 once its MMAs are done
          const long long p = j - 1;
          if (!mbar_wait_bounded(&done[p % kWgStages], (uint32_t)((p / kWgStages) & 1))) {
            give_up();
            break;
          }
          issue(nt);
          ++nt;
        }
      }
      // what is still in flight, bounded: copies that no MMA waited for, and
      // the last unit's MMAs (whose commit covers all before it)
      for (long long j = nm; j < nt; ++j)
        mbar_wait_bounded(&full[j % kWgStages], (uint32_t)((j / kWgStages) & 1));
      if (nm > 0 &&
          !mbar_wait_bounded(&done[(nm - 1) % kWgStages], (uint32_t)(((nm - 1) / kWgStages) & 1)))
        give_up();
    }
  } else {
    for (long long grp = 0; grp < ng && !s_abort; ++grp) {
      const int b = (int)(grp & 1);
      bool ok = mbar_wait_bounded(&tfull[b], (uint32_t)((grp >> 1) & 1));
      ok = __all_sync(0xffffffffu, ok);  // tcgen05.ld is warp-collective
      if (!ok) {
        if (lane == 0) give_up();
        break;
      }
      asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
      const uint32_t t0 = tmem + ((uint32_t)(warp * 32) << 16) + (uint32_t)(2 * kWgCol2 * b);
#pragma unroll
      for (int k = 0; k < 6; ++k) {
        float v[16];
        tc_ld16(t0 + (uint32_t)(kWgCol2 * (k / 3) + 16 * (k % 3)), v);
#pragma unroll
        for (int q = 0; q < 16; ++q) sum[k][q] += v[q];
      }
      asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
      __syncwarp();
      if (lane == 0) mbar_arrive1(&tempty[b]);
    }
  }
  __syncthreads();
  // accumulator k / 3, row (block, ci), column (2 - dx', co): tap block 8 (k/3) + row / 16
  if (warp < 4) {
    const bool ok = !s_abort;
    float *out = partial + (long long)blockIdx.x * 27 * kC * kC;
    const float nan = __int_as_float(0x7fc00000);
    const int row = warp * 32 + lane, ci = row & 15;
#pragma unroll
    for (int k = 0; k < 6; ++k) {
      const int blk = 8 * (k / 3) + (row >> 4), dyp = blk >> 2, dzp = blk & 3;
      if (dyp > 2 || dzp > 2) continue;
      float *o = out + (long long)(dzp * 9 + dyp * 3 + 2 - k % 3) * kC * kC + ci;
#pragma unroll
      for (int q = 0; q < 16; ++q) o[q * kC] = ok ? sum[k][q] : nan;
    }
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  if (warp == 0)
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, 256;" ::"r"(tmem) : "memory");
}

// out[v] = channels [v][16] of feats [c][v], zeros from c on.
__global__ void __launch_bounds__(256)
k_channels_last(const float *__restrict__ feats, int c, long long vox, __nv_bfloat16 *__restrict__ out) {
  for (long long v = blockIdx.x * 256LL + threadIdx.x; v < vox; v += gridDim.x * 256LL) {
    uint32_t pk[8];
#pragma unroll
    for (int q = 0; q < 8; ++q) {
      const float a = 2 * q < c ? feats[(2 * q) * vox + v] : 0.f;
      const float b = 2 * q + 1 < c ? feats[(2 * q + 1) * vox + v] : 0.f;
      const __nv_bfloat162 b2 = __floats2bfloat162_rn(a, b);
      pk[q] = *reinterpret_cast<const uint32_t *>(&b2);
    }
    uint4 *dst = reinterpret_cast<uint4 *>(out + v * kC);
    dst[0] = make_uint4(pk[0], pk[1], pk[2], pk[3]);
    dst[1] = make_uint4(pk[4], pk[5], pk[6], pk[7]);
  }
}
}  // namespace
}  // namespace efwi

using namespace efwi;

namespace {
// 0: mma.sync; 1: tcgen05, one MMA per tap, tile staged by loads; 2: tcgen05,
// z-marching; 3: as 1 with the tiles staged by bulk tensor copies three stages
// deep; 4 / 5: as 3, warp-specialised (copy + MMA warp, four epilogue warps),
// two / three stages
std::atomic<int> g_conv_kernel{2};
std::atomic<unsigned long long> g_tc_smem_set{0}, g_tc2_smem_set{0}, g_tc3_smem_set{0},
    g_ws2_smem_set{0}, g_ws3_smem_set{0};
int g_sm_count[64] = {0};
std::atomic<PFN_cuTensorMapEncodeTiled_v12000> g_conv_encode{nullptr};

PFN_cuTensorMapEncodeTiled_v12000 conv_encoder() {
  PFN_cuTensorMapEncodeTiled_v12000 f = g_conv_encode.load();
  if (f) return f;
  void *fn = nullptr;
  cudaDriverEntryPointQueryResult q;
  if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &fn, cudaEnableDefault, &q) !=
          cudaSuccess ||
      q != cudaDriverEntryPointSuccess || !fn)
    return nullptr;
  f = (PFN_cuTensorMapEncodeTiled_v12000)fn;
  g_conv_encode.store(f);
  return f;
}

// x [D][H][W][16] bf16 as a 5-D tensor (8 channels, 2 halves, W, H, D) with
// boxes of one channel half over the 10 x 18 x 3 staged voxels.
bool conv_map(CUtensorMap *m, const void *x, int D, int H, int W) {
  PFN_cuTensorMapEncodeTiled_v12000 enc = conv_encoder();
  if (!enc) return false;
  cuuint64_t dims[5] = {8, 2, (cuuint64_t)W, (cuuint64_t)H, (cuuint64_t)D};
  cuuint64_t strides[4] = {16, 32, 32ull * W, 32ull * W * H};
  cuuint32_t box[5] = {8, 1, (cuuint32_t)kTcSX, (cuuint32_t)kTcSY, 3};
  cuuint32_t es[5] = {1, 1, 1, 1, 1};
  return enc(m, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 5, const_cast<void *>(x), dims, strides, box,
             es, CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_NONE,
             CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

// x with boxes of one plane of 10 x 18 voxels of 32 bytes.
bool plane_map(CUtensorMap *m, const void *x, int D, int H, int W) {
  PFN_cuTensorMapEncodeTiled_v12000 enc = conv_encoder();
  if (!enc) return false;
  const cuuint64_t w = W, h = H, d = D;
  cuuint64_t dims[4] = {kC, w, h, d}, strides[3] = {32, 32 * w, 32 * w * h};
  cuuint32_t box[4] = {kC, kTcSX, kTcSY, 1}, es[4] = {1, 1, 1, 1};
  return enc(m, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 4, const_cast<void *>(x), dims, strides, box, es,
             CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_32B,
             CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

// Maps of the weight gradient, a voxel's 32 bytes innermost: x with boxes of
// 8 x, 4 z, 18 y (in that order in shared memory), dy of 10 x, 16 y, 2 z.
bool wgrad_maps(CUtensorMap *xm, CUtensorMap *gm, const void *x, const void *dy, int D, int H,
                int W) {
  PFN_cuTensorMapEncodeTiled_v12000 enc = conv_encoder();
  if (!enc) return false;
  const cuuint64_t w = W, h = H, d = D;
  cuuint64_t xd[4] = {kC, w, d, h}, xs[3] = {32, 32 * w * h, 32 * w};
  cuuint64_t gd[4] = {kC, w, h, d}, gs[3] = {32, 32 * w, 32 * w * h};
  cuuint32_t xb[4] = {kC, kWgX, kWgZs, kWgY + 2}, gb[4] = {kC, kWgGX, kWgY, kWgZ};
  cuuint32_t es[4] = {1, 1, 1, 1};
  auto one = [&](CUtensorMap *m, const void *p, cuuint64_t *dims, cuuint64_t *str, cuuint32_t *box) {
    return enc(m, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 4, const_cast<void *>(p), dims, str, box, es,
               CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_32B,
               CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
  };
  return one(xm, x, xd, xs, xb) && one(gm, dy, gd, gs, gb);
}

// SM count of the current device.
bool conv_sms(int *out) {
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess) return false;
  int &sms = g_sm_count[dev & 63];
  if (!sms && cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess)
    return false;
  *out = sms;
  return true;
}
}  // namespace

extern "C" int efwi_conv3d_set_kernel(int form) {
  if (form < 0 || form > 5) return 1;
  g_conv_kernel.store(form);
  return 0;
}

extern "C" int efwi_conv3d_status(int *timed_out, void *stream) {
  if (!timed_out) return 1;
  int v = 0, zero = 0;
  cudaStream_t st = (cudaStream_t)stream;
  if (cudaMemcpyFromSymbolAsync(&v, g_conv_status, sizeof(int), 0, cudaMemcpyDeviceToHost, st) !=
          cudaSuccess ||
      cudaMemcpyToSymbolAsync(g_conv_status, &zero, sizeof(int), 0, cudaMemcpyHostToDevice, st) !=
          cudaSuccess ||
      cudaStreamSynchronize(st) != cudaSuccess)
    return 2;
  *timed_out = v != 0;
  return 0;
}

namespace {
// The z-marching form; y0c: channel 0 alone, [D][H][W] f32.
int zm_launch(const CUtensorMap &map, const void *w, const float *bias, int D, int H, int W,
              int relu, void *y_bf16, float *y_f32, float *y0c, cudaStream_t st) {
  int sms = 0;
  if (!conv_sms(&sms)) return 2;
  // planes per tile: the fewest steps (waves of 8 tiles per SM times the planes
  // that a tile reads)
  const long long cols = (long long)((W + kTcX - 1) / kTcX) * ((H + kTcY - 1) / kTcY);
  const long long slots = 8LL * sms;
  long long best = -1;
  int zlen = D;
  for (int n = 1; n <= D; ++n) {
    const int len = (D + n - 1) / n;
    const long long ctas = cols * ((D + len - 1) / len);
    const long long steps = ((ctas + slots - 1) / slots) * (len + 2);
    if (best < 0 || steps < best) { best = steps; zlen = len; }
    if (ctas > 8 * slots) break;
  }
  const long long units = cols * ((D + zlen - 1) / zlen), ctas = (units + kZmTiles - 1) / kZmTiles;
  if (units > 0x7fffffffLL - kZmTiles) return 1;
  set_smem_once(k_conv3d_fwd_zm, kZmSmem, g_tc2_smem_set);
  k_conv3d_fwd_zm<<<(unsigned)ctas, 128 * kZmTiles, kZmSmem, st>>>(map, (const __nv_bfloat16 *)w, bias, D, H,
                                                        W, zlen, (int)units, relu, (__nv_bfloat16 *)y_bf16,
                                                        y_f32, y0c);
  return 0;
}

}  // namespace

extern "C" int efwi_channels_last(const float *feats, int c, long long voxels, void *out,
                                  void *stream) {
  if (!feats || !out || c < 1 || c > kC || voxels < 1 || ((uintptr_t)out & 15) != 0) return 1;
  const int blocks = (int)std::min<long long>((voxels + 255) / 256, 16384);
  k_channels_last<<<blocks, 256, 0, (cudaStream_t)stream>>>(feats, c, voxels, (__nv_bfloat16 *)out);
  return cudaGetLastError() == cudaSuccess ? 0 : 2;
}

extern "C" int efwi_conv3d_forward_head(const void *x, const void *w, const float *bias, int D,
                                        int H, int W, int relu, float *y, void *stream) {
  if (!x || !w || !y || D < 1 || H < 1 || W < 1 || D > 65535) return 1;
  if ((((uintptr_t)x | (uintptr_t)w) & 15) != 0) return 1;
  if (g_conv_kernel.load() != 2) return 3;
  CUtensorMap map;
  if (!plane_map(&map, x, D, H, W)) return 2;
  const int rc = zm_launch(map, w, bias, D, H, W, relu, nullptr, nullptr, y, (cudaStream_t)stream);
  if (rc) return rc;
  return cudaGetLastError() == cudaSuccess ? 0 : 2;
}

extern "C" int efwi_conv3d_forward(const void *x, const void *w, const float *bias, int D, int H,
                                   int W, int relu, void *y_bf16, float *y_f32, void *stream) {
  if (!x || !w || D < 1 || H < 1 || W < 1 || D > 65535 || (!y_bf16 && !y_f32)) return 1;
  if (((uintptr_t)x & 15) != 0) return 1;  // staged with 16-byte loads
  cudaStream_t st = (cudaStream_t)stream;
  const int form = g_conv_kernel.load();
  if (form != 0 && ((uintptr_t)w & 15) == 0 && ((uintptr_t)y_bf16 & 15) == 0 &&
      ((uintptr_t)y_f32 & 15) == 0) {
    int sms = 0;
    if (!conv_sms(&sms)) return 2;
    const long long tiles = (long long)((W + kTcX - 1) / kTcX) * ((H + kTcY - 1) / kTcY) * D;
    if (form >= 2) {
      CUtensorMap map;
      if (!(form == 2 ? plane_map(&map, x, D, H, W) : conv_map(&map, x, D, H, W))) return 2;
      if (form >= 4) {  // warp-specialised: two stages at 4 CTAs per SM, or three at 3
        const __nv_bfloat16 *wb = (const __nv_bfloat16 *)w;
        if (form == 4) {
          set_smem_once(k_conv3d_fwd_ws<2>, tc2_smem<2>(), g_ws2_smem_set);
          const int blocks = (int)std::min<long long>(tiles, 4LL * sms);
          k_conv3d_fwd_ws<2><<<blocks, kWsThreads, tc2_smem<2>(), st>>>(
              map, wb, bias, D, H, W, relu, (__nv_bfloat16 *)y_bf16, y_f32);
        } else {
          set_smem_once(k_conv3d_fwd_ws<3>, tc2_smem<3>(), g_ws3_smem_set);
          const int blocks = (int)std::min<long long>(tiles, 3LL * sms);
          k_conv3d_fwd_ws<3><<<blocks, kWsThreads, tc2_smem<3>(), st>>>(
              map, wb, bias, D, H, W, relu, (__nv_bfloat16 *)y_bf16, y_f32);
        }
      } else if (form == 2) {
        const int rc = zm_launch(map, w, bias, D, H, W, relu, y_bf16, y_f32, nullptr, st);
        if (rc) return rc;
      } else {  // three stages, 66 KB: 3 CTAs per SM
        set_smem_once(k_conv3d_fwd_tc2, tc2_smem<3>(), g_tc3_smem_set);
        const int blocks = (int)std::min<long long>(tiles, 3LL * sms);
        k_conv3d_fwd_tc2<<<blocks, 128, tc2_smem<3>(), st>>>(
            map, (const __nv_bfloat16 *)w, bias, D, H, W, relu, (__nv_bfloat16 *)y_bf16, y_f32);
      }
    } else {
      set_smem_once(k_conv3d_fwd_tc, kTcSmem, g_tc_smem_set);
      const int blocks = (int)std::min<long long>(tiles, 6LL * sms);
      k_conv3d_fwd_tc<<<blocks, 128, kTcSmem, st>>>((const __nv_bfloat16 *)x,
                                                    (const __nv_bfloat16 *)w, bias, D, H, W, relu,
                                                    (__nv_bfloat16 *)y_bf16, y_f32);
    }
    return cudaGetLastError() == cudaSuccess ? 0 : 2;
  }
  const dim3 grid((W + kTileX - 1) / kTileX, (H + kRowsFwd - 1) / kRowsFwd, D);
  k_conv3d_fwd<<<grid, 32 * kRowsFwd, 0, st>>>(
      (const __nv_bfloat16 *)x, (const __nv_bfloat16 *)w, bias, D, H, W, relu,
      (__nv_bfloat16 *)y_bf16, y_f32);
  return cudaGetLastError() == cudaSuccess ? 0 : 2;
}

namespace {
std::atomic<int> g_wgrad_kernel{1};  // 1: tcgen05, 0: mma.sync
std::atomic<unsigned long long> g_wg_smem_set{0};
}  // namespace

extern "C" int efwi_conv3d_set_wgrad_kernel(int tcgen05) {
  g_wgrad_kernel.store(tcgen05 ? 1 : 0);
  return 0;
}

namespace {
// Partial sums of the weight gradient; *parts: how many were written.
int wgrad_partials(const void *x, const void *dy, int D, int H, int W, float *partial, int nparts,
                   int *parts, cudaStream_t st) {
  *parts = nparts;
  // the bulk copies need 16-byte aligned volumes; others take mma.sync
  if (g_wgrad_kernel.load() == 1 && ((uintptr_t)x & 15) == 0 && ((uintptr_t)dy & 15) == 0) {
    int sms = 0;
    if (!conv_sms(&sms)) return 2;
    CUtensorMap xmap, gmap;
    if (!wgrad_maps(&xmap, &gmap, x, dy, D, H, W)) return 2;
    set_smem_once(k_conv3d_wgrad_tc, kWgSmem, g_wg_smem_set);
    // two resident CTAs per SM (87 KB of shared memory, half of TMEM each)
    const long long units = (long long)((W + kWgX - 1) / kWgX) * ((H + kWgY - 1) / kWgY) *
                            ((D + kWgZ - 1) / kWgZ);
    *parts = (int)std::min<long long>(std::min<long long>(nparts, 2LL * sms), units);
    k_conv3d_wgrad_tc<<<*parts, kWgThreads, kWgSmem, st>>>(xmap, gmap, D, H, W, partial);
  } else {
    k_conv3d_wgrad<<<nparts, 27 * 32, 0, st>>>((const __nv_bfloat16 *)x,
                                               (const __nv_bfloat16 *)dy, D, H, W, partial);
  }
  return 0;
}

void reduce_partials(const Partials &a, const Partials &b, cudaStream_t st) {
  k_reduce_partials<<<(a.n + 31) / 32 + (b.n + 31) / 32, dim3(32, kRedWarps), 0, st>>>(a, b);
}
}  // namespace

extern "C" int efwi_conv3d_wgrad(const void *x, const void *dy, int D, int H, int W,
                                 float *partial, int nparts, float *dw, void *stream) {
  if (!x || !dy || !partial || !dw || D < 1 || H < 1 || W < 1 || nparts < 1) return 1;
  cudaStream_t st = (cudaStream_t)stream;
  int parts = 0;
  const int rc = wgrad_partials(x, dy, D, H, W, partial, nparts, &parts, st);
  if (rc) return rc;
  reduce_partials({partial, parts, 27 * kC * kC, dw}, {nullptr, 0, 0, nullptr}, st);
  return cudaGetLastError() == cudaSuccess ? 0 : 2;
}

extern "C" long long efwi_conv3d_backward_scratch(int D, int H, int W, int nparts, int gy_f32,
                                                  int relu) {
  if (D < 1 || H < 1 || W < 1 || nparts < 1) return -1;
  const long long vox = (long long)D * H * W;
  const bool own = gy_f32 || relu;  // a BF16 copy of the gradient is written
  return (own ? vox * kC * 2 : 0) + 27LL * kC * kC * 2 + (27LL * kC * kC + kC) * 4 * nparts;
}

extern "C" int efwi_conv3d_backward(const void *x, const void *w, const void *gy, int gy_f32,
                                    const void *y, int y_f32, int D, int H, int W, void *scratch,
                                    int nparts, void *dx, float *dw, float *db, void *stream) {
  if (!x || !w || !gy || !scratch || !dw || !db || D < 1 || H < 1 || W < 1 || nparts < 1) return 1;
  if (gy_f32 < 0 || gy_f32 > 2 || (gy_f32 == 2 && y)) return 1;
  if ((((uintptr_t)x | (uintptr_t)gy | (uintptr_t)y | (uintptr_t)scratch | (uintptr_t)dx) & 15) != 0)
    return 1;
  cudaStream_t st = (cudaStream_t)stream;
  const long long vox = (long long)D * H * W;
  const bool own = gy_f32 || y;
  char *p = (char *)scratch;
  __nv_bfloat16 *dyb = own ? (__nv_bfloat16 *)p : nullptr;
  if (own) p += vox * kC * 2;
  __nv_bfloat16 *wt = (__nv_bfloat16 *)p;
  p += 27 * kC * kC * 2;
  float *dbp = (float *)p, *partial = dbp + (long long)kC * nparts;
  const int blocks = (int)std::min<long long>(nparts, (2 * vox + kPrepThreads - 1) / kPrepThreads);
  const __nv_bfloat16 *wb = (const __nv_bfloat16 *)w;
  auto prep = [&](auto g, auto yy) {
    k_conv3d_grad_prep<<<blocks, kPrepThreads, 0, st>>>(g, yy, 2 * vox, dyb, dbp, wb,
                                                        dx ? wt : nullptr);
  };
  const __nv_bfloat16 *gb = (const __nv_bfloat16 *)gy, *ybf = (const __nv_bfloat16 *)y;
  const float *gf = (const float *)gy, *yf = (const float *)y;
  if (gy_f32 == 2) prep((const Head *)gy, ybf);
  else if (gy_f32 && y_f32) prep(gf, yf);
  else if (gy_f32) prep(gf, ybf);
  else if (y_f32) prep(gb, yf);
  else prep(gb, ybf);
  const void *dy = own ? (const void *)dyb : gy;
  if (dx) {
    const int rc = efwi_conv3d_forward(dy, wt, nullptr, D, H, W, 0, dx, nullptr, stream);
    if (rc) return rc;
  }
  int parts = 0;
  const int rc = wgrad_partials(x, dy, D, H, W, partial, nparts, &parts, st);
  if (rc) return rc;
  reduce_partials({partial, parts, 27 * kC * kC, dw}, {dbp, blocks, kC, db}, st);
  return cudaGetLastError() == cudaSuccess ? 0 : 2;
}
