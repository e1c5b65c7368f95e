// BF16 tensor-core kernels of the warm-start surrogate (a 3-D convolutional U-Net
// that predicts velocity and pressure from geometry features).
//
// Activations are channels-last (N, D, H, W, C) BF16; weights are
// [27 taps][C_out][C_in] BF16 (C_in fastest) with FP32 master copies; every
// product accumulates in FP32 on the tensor cores (mma.sync m16n8k16 .bf16).
// A 3x3x3 convolution is an implicit GEMM: rows = output voxels, columns = output
// channels, reduction = 27 * C_in (C_in a multiple of 16, so a 16-wide reduction
// chunk never straddles two taps).
#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <stdint.h>

#include <algorithm>
#include <cmath>

#include "../../include/hemelb_gb300_nn.h"
#include "overlap.cuh"
#include "sm_count.h"

namespace {

__device__ __forceinline__ void mma_bf16(float* c, const uint32_t* a, const uint32_t* b) {
  asm volatile(
      "mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, "
      "{%0,%1,%2,%3};\n"
      : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
      : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b[0]), "r"(b[1]));
}

__device__ __forceinline__ uint32_t ld2(const __nv_bfloat16* p) {
  return *reinterpret_cast<const uint32_t*>(p);
}

__device__ __forceinline__ uint32_t pack2(__nv_bfloat16 lo, __nv_bfloat16 hi) {
  return (uint32_t)__bfloat16_as_ushort(lo) | ((uint32_t)__bfloat16_as_ushort(hi) << 16);
}

struct Vox {
  int n, z, y, x;
};
__device__ __forceinline__ Vox unflat(int64_t m, int D, int H, int W) {
  Vox v;
  v.x = (int)(m % W);
  m /= W;
  v.y = (int)(m % H);
  m /= H;
  v.z = (int)(m % D);
  v.n = (int)(m / D);
  return v;
}

// ---------------------------------------------------------------------------
// Convolution (stride 1, zero padding 1, or a 1x1x1 "taps == 1" convolution).
// out[m, co] = act( sum_{tap, ci} in[m + off(tap), ci] * w[tap][co][ci] + bias[co] )
// One warp: 16 output voxels x (8 * NT) output channels.  flip: use tap 26 - t
// (the data-gradient convolution runs the flipped, transposed kernel).
// ---------------------------------------------------------------------------
template <int NT>
__global__ void __launch_bounds__(128) k_conv3d(const __nv_bfloat16* __restrict__ in, int Cin,
                                                 const __nv_bfloat16* __restrict__ w,
                                                 const float* __restrict__ bias,
                                                 __nv_bfloat16* __restrict__ out, float* __restrict__ out_f32,
                                                 int Cout, int N, int D, int H, int W, int taps,
                                                 int relu) {
  const int lane = threadIdx.x & 31;
  const int warp = (blockIdx.x * 4) + (threadIdx.x >> 5);
  const int64_t M = (int64_t)N * D * H * W;
  const int64_t m0 = (int64_t)warp * 16;
  const int co0 = blockIdx.y * 8 * NT;
  if (m0 >= M) return;
  const int g = lane >> 2, t = lane & 3;
  float acc[NT][4];
#pragma unroll
  for (int j = 0; j < NT; ++j) acc[j][0] = acc[j][1] = acc[j][2] = acc[j][3] = 0.f;
  // the two output voxels whose A rows this lane loads
  const int64_t ma = m0 + g, mb = m0 + g + 8;
  const Vox va = unflat(ma < M ? ma : 0, D, H, W), vb = unflat(mb < M ? mb : 0, D, H, W);
  const int chunks = Cin / 16;
  for (int tap = 0; tap < taps; ++tap) {
    int dz = 0, dy = 0, dx = 0;
    if (taps == 27) {
      dz = tap / 9 - 1;
      dy = (tap / 3) % 3 - 1;
      dx = tap % 3 - 1;
    }
    const int za = va.z + dz, ya = va.y + dy, xa = va.x + dx;
    const int zb = vb.z + dz, yb = vb.y + dy, xb = vb.x + dx;
    const bool oka = ma < M && za >= 0 && za < D && ya >= 0 && ya < H && xa >= 0 && xa < W;
    const bool okb = mb < M && zb >= 0 && zb < D && yb >= 0 && yb < H && xb >= 0 && xb < W;
    const __nv_bfloat16* pa = in + ((((int64_t)va.n * D + za) * H + ya) * W + xa) * Cin;
    const __nv_bfloat16* pb = in + ((((int64_t)vb.n * D + zb) * H + yb) * W + xb) * Cin;
    const __nv_bfloat16* wt = w + (int64_t)tap * Cout * Cin;
    for (int c = 0; c < chunks; ++c) {
      const int ci = c * 16 + t * 2;
      uint32_t a[4];
      a[0] = oka ? ld2(pa + ci) : 0u;
      a[1] = okb ? ld2(pb + ci) : 0u;
      a[2] = oka ? ld2(pa + ci + 8) : 0u;
      a[3] = okb ? ld2(pb + ci + 8) : 0u;
#pragma unroll
      for (int j = 0; j < NT; ++j) {
        const int co = co0 + j * 8 + g;
        uint32_t b[2];
        if (co < Cout) {
          b[0] = ld2(wt + (int64_t)co * Cin + ci);
          b[1] = ld2(wt + (int64_t)co * Cin + ci + 8);
        } else {
          b[0] = b[1] = 0u;
        }
        mma_bf16(acc[j], a, b);
      }
    }
  }
  // epilogue: rows g and g+8, columns 2t and 2t+1 of each 8-wide tile
#pragma unroll
  for (int j = 0; j < NT; ++j) {
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      const int64_t m = m0 + g + 8 * h;
      if (m >= M) continue;
#pragma unroll
      for (int e = 0; e < 2; ++e) {
        const int co = co0 + j * 8 + 2 * t + e;
        if (co >= Cout) continue;
        float v = acc[j][2 * h + e] + (bias ? bias[co] : 0.f);
        if (relu && v < 0.f) v = 0.f;
        out[m * Cout + co] = __float2bfloat16_rn(v);
        if (out_f32) out_f32[m * Cout + co] = v;
      }
    }
  }
}

// Weight gradient: dw[tap][co][ci] += sum_m dy[m, co] * x[m + off(tap), ci] over a
// slice of voxels; one warp = one (tap, 16 co, 8 ci) tile; FP32 atomics join slices.
__global__ void __launch_bounds__(128) k_conv3d_wgrad(const __nv_bfloat16* __restrict__ x, int Cin,
                                                       const __nv_bfloat16* __restrict__ dy, int Cout,
                                                       float* __restrict__ dw, int N, int D, int H,
                                                       int W, int taps, int64_t slice) {
  const int lane = threadIdx.x & 31;
  const int g = lane >> 2, t = lane & 3;
  const int tiles_co = (Cout + 15) / 16, tiles_ci = Cin / 8;
  const int64_t tile = (int64_t)blockIdx.x * 4 + (threadIdx.x >> 5);
  const int64_t ntile = (int64_t)taps * tiles_co * tiles_ci;
  if (tile >= ntile) return;
  const int tap = (int)(tile / (tiles_co * tiles_ci));
  const int co0 = (int)((tile / tiles_ci) % tiles_co) * 16;
  const int ci0 = (int)(tile % tiles_ci) * 8;
  int dz = 0, dy_ = 0, dx = 0;
  if (taps == 27) {
    dz = tap / 9 - 1;
    dy_ = (tap / 3) % 3 - 1;
    dx = tap % 3 - 1;
  }
  const int64_t M = (int64_t)N * D * H * W;
  const int64_t mbeg = (int64_t)blockIdx.y * slice, mend = mbeg + slice < M ? mbeg + slice : M;
  float acc[4] = {0.f, 0.f, 0.f, 0.f};
  const __nv_bfloat16 zero = __float2bfloat16_rn(0.f);
  for (int64_t m = mbeg; m < mend; m += 16) {
    // A (16 co x 16 m): rows co0+g / co0+g+8, columns m+2t, m+2t+1, m+2t+8, m+2t+9
    // B (16 m x 8 ci): rows m+2t, m+2t+1, m+2t+8, m+2t+9, column ci0+g
    uint32_t a[4], b[2];
    __nv_bfloat16 av[8], bv[4];
    const int64_t mm[4] = {m + 2 * t, m + 2 * t + 1, m + 2 * t + 8, m + 2 * t + 9};
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      const bool in_m = mm[k] < mend;
      const int coa = co0 + g, cob = co0 + g + 8;
      av[2 * k] = (in_m && coa < Cout) ? dy[mm[k] * Cout + coa] : zero;
      av[2 * k + 1] = (in_m && cob < Cout) ? dy[mm[k] * Cout + cob] : zero;
      __nv_bfloat16 xv = zero;
      if (in_m) {
        Vox v = unflat(mm[k], D, H, W);
        const int z = v.z + dz, y = v.y + dy_, xx = v.x + dx;
        if (z >= 0 && z < D && y >= 0 && y < H && xx >= 0 && xx < W)
          xv = x[((((int64_t)v.n * D + z) * H + y) * W + xx) * Cin + ci0 + g];
      }
      bv[k] = xv;
    }
    a[0] = pack2(av[0], av[2]);  // row g: m+2t, m+2t+1
    a[1] = pack2(av[1], av[3]);  // row g+8
    a[2] = pack2(av[4], av[6]);  // row g: m+2t+8, m+2t+9
    a[3] = pack2(av[5], av[7]);
    b[0] = pack2(bv[0], bv[1]);
    b[1] = pack2(bv[2], bv[3]);
    mma_bf16(acc, a, b);
  }
  // D rows = co (g, g+8), columns = ci (2t, 2t+1)
#pragma unroll
  for (int h = 0; h < 2; ++h)
#pragma unroll
    for (int e = 0; e < 2; ++e) {
      const int co = co0 + g + 8 * h, ci = ci0 + 2 * t + e;
      if (co < Cout) atomicAdd(dw + ((int64_t)tap * Cout + co) * Cin + ci, acc[2 * h + e]);
    }
}

// ---------------------------------------------------------------------------
// Weight gradient of a 3x3x3 convolution, tiled through shared memory.
// A CTA owns a (16 C_out) x (16 NCI C_in) block of dW for all 27 taps and runs
// over a range of 4x4x8 voxel bricks: per brick it stages dY (128 voxels x 16 co)
// and X on the brick plus a one-voxel halo (6x6x10 voxels x 16 NCI ci) with
// cp.async (zero fill outside the volume), then each of the 8 warps accumulates
// its taps (warp, warp + 8, warp + 16, warp + 24) as
//   dW[tap] += dY^T (16 co x 16 voxels) * X_shifted (16 voxels x 8 ci)
// on mma.sync with both operands read by ldmatrix.trans (rows of 16 bytes; the
// row pitches of 48/80 bytes put the 8 rows of one ldmatrix in distinct banks).
// The FP32 accumulators are added to dW once per CTA (red.global.add).
// ---------------------------------------------------------------------------
constexpr int kBZ = 4, kBY = 4, kBX = 8, kBV = kBZ * kBY * kBX;  // brick
constexpr int kHZ = kBZ + 2, kHY = kBY + 2, kHX = kBX + 2, kHV = kHZ * kHY * kHX;

__device__ __forceinline__ void cp_async16(void* smem, const void* gmem, bool ok) {
  const unsigned s = (unsigned)__cvta_generic_to_shared(smem);
  const int sz = ok ? 16 : 0;
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;\n" ::"r"(s), "l"(gmem), "r"(sz));
}
__device__ __forceinline__ void cp_async_wait_all() {
  asm volatile("cp.async.commit_group;\ncp.async.wait_group 0;\n" ::: "memory");
}
__device__ __forceinline__ void ldsm_x4_trans(uint32_t* r, const void* smem) {
  const unsigned s = (unsigned)__cvta_generic_to_shared(smem);
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0,%1,%2,%3}, [%4];\n"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3])
               : "r"(s));
}
__device__ __forceinline__ void red_add(float* p, float v) {
  asm volatile("red.global.add.f32 [%0], %1;\n" ::"l"(p), "f"(v) : "memory");
}

template <int NCI>
__global__ void __launch_bounds__(256) k_wgrad_brick(const __nv_bfloat16* __restrict__ x, int Cin,
                                                      const __nv_bfloat16* __restrict__ dy, int Cout,
                                                      float* __restrict__ dw, int D, int H, int W, int nbz,
                                                      int nby, int nbx, int64_t nbricks, int bricks_per_cta) {
  constexpr int CIB = 16 * NCI, XS = CIB + 8, DS = 16 + 8, NTILE = 2 * NCI;
  __shared__ __align__(16) __nv_bfloat16 Xs[kHV * XS];
  __shared__ __align__(16) __nv_bfloat16 Ds[kBV * DS];
  const int co0 = blockIdx.y * 16, ci0 = blockIdx.z * CIB;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int q = lane >> 3, rr = lane & 7;
  float acc[4][NTILE][4];
#pragma unroll
  for (int j = 0; j < 4; ++j)
#pragma unroll
    for (int nt = 0; nt < NTILE; ++nt) acc[j][nt][0] = acc[j][nt][1] = acc[j][nt][2] = acc[j][nt][3] = 0.f;
  const int64_t b0 = (int64_t)blockIdx.x * bricks_per_cta;
  const int64_t b1 = b0 + bricks_per_cta < nbricks ? b0 + bricks_per_cta : nbricks;
  for (int64_t b = b0; b < b1; ++b) {
    const int bx = (int)(b % nbx);
    int64_t r = b / nbx;
    const int by = (int)(r % nby);
    r /= nby;
    const int bz = (int)(r % nbz);
    const int n = (int)(r / nbz);
    const int z0 = bz * kBZ, y0 = by * kBY, x0 = bx * kBX;
    for (int c = threadIdx.x; c < kBV * 2; c += 256) {
      const int v = c >> 1, part = c & 1;
      const int z = z0 + v / (kBY * kBX), y = y0 + (v / kBX) % kBY, xx = x0 + v % kBX;
      const bool ok = z < D && y < H && xx < W;
      const __nv_bfloat16* src = ok ? dy + ((((int64_t)n * D + z) * H + y) * W + xx) * Cout + co0 + part * 8 : dy;
      cp_async16(&Ds[v * DS + part * 8], src, ok);
    }
    for (int c = threadIdx.x; c < kHV * NTILE; c += 256) {
      const int h = c / NTILE, part = c % NTILE;
      const int z = z0 + h / (kHY * kHX) - 1, y = y0 + (h / kHX) % kHY - 1, xx = x0 + h % kHX - 1;
      const bool ok = z >= 0 && z < D && y >= 0 && y < H && xx >= 0 && xx < W;
      const __nv_bfloat16* src = ok ? x + ((((int64_t)n * D + z) * H + y) * W + xx) * Cin + ci0 + part * 8 : x;
      cp_async16(&Xs[h * XS + part * 8], src, ok);
    }
    cp_async_wait_all();
    __syncthreads();
#pragma unroll 1
    for (int s = 0; s < kBV / 16; ++s) {
      uint32_t a[4];
      ldsm_x4_trans(a, &Ds[(16 * s + rr + ((q >> 1) << 3)) * DS + (q & 1) * 8]);
      // the voxel whose X row this lane addresses for the B operand
      const int vb = 16 * s + rr + ((q & 1) << 3);
      const int vz = vb / (kBY * kBX), vy = (vb / kBX) % kBY, vx = vb % kBX;
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const int tap = warp + 8 * j;
        if (tap < 27) {
          const int h = ((vz + tap / 9) * kHY + (vy + (tap / 3) % 3)) * kHX + (vx + tap % 3);
#pragma unroll
          for (int nt = 0; nt < NTILE; nt += 2) {
            uint32_t bf[4];
            ldsm_x4_trans(bf, &Xs[h * XS + (nt + (q >> 1)) * 8]);
            mma_bf16(acc[j][nt], a, bf);
            mma_bf16(acc[j][nt + 1], a, bf + 2);
          }
        }
      }
    }
    __syncthreads();
  }
  const int g = lane >> 2, t = lane & 3;
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    const int tap = warp + 8 * j;
    if (tap < 27) {
#pragma unroll
      for (int nt = 0; nt < NTILE; ++nt)
#pragma unroll
        for (int hh = 0; hh < 2; ++hh)
#pragma unroll
          for (int e = 0; e < 2; ++e)
            red_add(dw + ((int64_t)tap * Cout + co0 + g + 8 * hh) * Cin + ci0 + nt * 8 + 2 * t + e,
                    acc[j][nt][2 * hh + e]);
    }
  }
}

// ---------------------------------------------------------------------------
// 3x3x3 convolution tiled through shared memory.  A CTA computes one 4x4x8 voxel
// brick (8 warps x 16 voxels) for 16 NCO output channels.  For each 16-channel
// slice of the input it stages X on the brick plus halo (6x6x10 voxels) with
// cp.async (zero fill outside the volume), and for each plane of 9 taps the
// weights W[tap][co][ci] of that slice; the warps then accumulate
//   out (16 voxels x 8 co) += X_shifted (16 voxels x 16 ci) * W[tap]^T (16 ci x 8 co)
// with A read by ldmatrix from the halo rows of the shifted voxels and B by
// ldmatrix from the weight rows.  Epilogue: bias, optional ReLU, BF16 (and FP32).
// ---------------------------------------------------------------------------
template <int NCO>
__global__ void __launch_bounds__(256) k_conv_brick(const __nv_bfloat16* __restrict__ in, int Cin,
                                                     const __nv_bfloat16* __restrict__ w,
                                                     const float* __restrict__ bias,
                                                     __nv_bfloat16* __restrict__ out, float* __restrict__ out_f32,
                                                     int Cout, int D, int H, int W, int nbz, int nby, int nbx,
                                                     int relu) {
  constexpr int COB = 16 * NCO, NTILE = 2 * NCO, XS = 24, WS = 24;
  __shared__ __align__(16) __nv_bfloat16 Xs[kHV * XS];
  __shared__ __align__(16) __nv_bfloat16 Ws[9 * COB * WS];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int q = lane >> 3, rr = lane & 7;
  const int co0 = blockIdx.y * COB;
  int64_t r = blockIdx.x;
  const int bx = (int)(r % nbx);
  r /= nbx;
  const int by = (int)(r % nby);
  r /= nby;
  const int bz = (int)(r % nbz);
  const int n = (int)(r / nbz);
  const int z0 = bz * kBZ, y0 = by * kBY, x0 = bx * kBX;
  float acc[NTILE][4];
#pragma unroll
  for (int nt = 0; nt < NTILE; ++nt) acc[nt][0] = acc[nt][1] = acc[nt][2] = acc[nt][3] = 0.f;
  // this lane's A row: voxel 16 warp + rr + 8 (q & 1) of the brick, channel half q >> 1
  const int va = 16 * warp + rr + ((q & 1) << 3);
  const int az = va / (kBY * kBX), ay = (va / kBX) % kBY, ax = va % kBX;
  for (int ci0 = 0; ci0 < Cin; ci0 += 16) {
    for (int c = threadIdx.x; c < kHV * 2; c += 256) {
      const int h = c >> 1, part = c & 1;
      const int z = z0 + h / (kHY * kHX) - 1, y = y0 + (h / kHX) % kHY - 1, xx = x0 + h % kHX - 1;
      const bool ok = z >= 0 && z < D && y >= 0 && y < H && xx >= 0 && xx < W;
      const __nv_bfloat16* src = ok ? in + ((((int64_t)n * D + z) * H + y) * W + xx) * Cin + ci0 + part * 8 : in;
      cp_async16(&Xs[h * XS + part * 8], src, ok);
    }
#pragma unroll 1
    for (int plane = 0; plane < 3; ++plane) {
      for (int c = threadIdx.x; c < 9 * COB * 2; c += 256) {
        const int row = c >> 1, part = c & 1;  // row = tap-in-plane * COB + co
        const int tp = row / COB, co = row % COB;
        const __nv_bfloat16* src = w + ((int64_t)(plane * 9 + tp) * Cout + co0 + co) * Cin + ci0 + part * 8;
        cp_async16(&Ws[row * WS + part * 8], src, true);
      }
      cp_async_wait_all();
      __syncthreads();
#pragma unroll
      for (int tp = 0; tp < 9; ++tp) {
        const int h = ((az + plane) * kHY + (ay + tp / 3)) * kHX + (ax + tp % 3);
        uint32_t a[4];
        {
          const unsigned sa = (unsigned)__cvta_generic_to_shared(&Xs[h * XS + (q >> 1) * 8]);
          asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0,%1,%2,%3}, [%4];\n"
                       : "=r"(a[0]), "=r"(a[1]), "=r"(a[2]), "=r"(a[3])
                       : "r"(sa));
        }
#pragma unroll
        for (int nt = 0; nt < NTILE; nt += 2) {
          uint32_t b[4];
          const unsigned sb =
              (unsigned)__cvta_generic_to_shared(&Ws[(tp * COB + (nt + (q >> 1)) * 8 + rr) * WS + (q & 1) * 8]);
          asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0,%1,%2,%3}, [%4];\n"
                       : "=r"(b[0]), "=r"(b[1]), "=r"(b[2]), "=r"(b[3])
                       : "r"(sb));
          mma_bf16(acc[nt], a, b);
          mma_bf16(acc[nt + 1], a, b + 2);
        }
      }
      __syncthreads();
    }
  }
  // epilogue: rows g and g + 8 of the warp's 16 voxels, columns 2t, 2t + 1 of each tile
  const int g = lane >> 2, t = lane & 3;
#pragma unroll
  for (int hh = 0; hh < 2; ++hh) {
    const int v = 16 * warp + g + 8 * hh;
    const int z = z0 + v / (kBY * kBX), y = y0 + (v / kBX) % kBY, xx = x0 + v % kBX;
    if (z >= D || y >= H || xx >= W) continue;
    const int64_t m = (((int64_t)n * D + z) * H + y) * W + xx;
#pragma unroll
    for (int nt = 0; nt < NTILE; ++nt)
#pragma unroll
      for (int e = 0; e < 2; ++e) {
        const int co = co0 + nt * 8 + 2 * t + e;
        float vv = acc[nt][2 * hh + e] + (bias ? bias[co] : 0.f);
        if (relu && vv < 0.f) vv = 0.f;
        out[m * Cout + co] = __float2bfloat16_rn(vv);
        if (out_f32) out_f32[m * Cout + co] = vv;
      }
  }
}

// Flipped, transposed weights for the data-gradient convolution:
// wt[taps - 1 - tap][ci][co] = w[tap][co][ci], 32 x 32 channels of a tap by a CTA through
// shared memory, so that both sides are 64-byte runs (192 -> 192 channels, 27 taps, 2 MB:
// 12.4 us with a thread per value, whose stores lay C_out values apart, 4.5 now).
__global__ void __launch_bounds__(256) k_flip_transpose(const __nv_bfloat16* w, __nv_bfloat16* wt, int Cout, int Cin,
                                                        int taps) {
  __shared__ __nv_bfloat16 tile[32][34];
  wait_for_previous();
  const unsigned nci = (unsigned)(Cin + 31) / 32, nco = (unsigned)(Cout + 31) / 32, q = blockIdx.x / nci;
  const int ci0 = (int)(blockIdx.x - q * nci) * 32, co0 = (int)(q % nco) * 32, tap = (int)(q / nco);
  const int a = threadIdx.x & 31, b = threadIdx.x >> 5;
  const __nv_bfloat16* src = w + (int64_t)tap * Cout * Cin;
  __nv_bfloat16* dst = wt + (int64_t)(taps - 1 - tap) * Cout * Cin;
#pragma unroll
  for (int k = b; k < 32; k += 8)
    if (co0 + k < Cout && ci0 + a < Cin) tile[k][a] = src[(int64_t)(co0 + k) * Cin + ci0 + a];
  __syncthreads();
#pragma unroll
  for (int k = b; k < 32; k += 8)
    if (ci0 + k < Cin && co0 + a < Cout) dst[(int64_t)(ci0 + k) * Cout + co0 + a] = tile[a][k];
}

// ReLU gradient in place: dy *= (y > 0)
__global__ void k_relu_bwd(__nv_bfloat16* __restrict__ dy, const __nv_bfloat16* __restrict__ y, int64_t n) {
  const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n && !(__bfloat162float(y[i]) > 0.f)) dy[i] = __float2bfloat16_rn(0.f);
}

// Bias gradient: db[c] += sum_m dy[m, c]
__global__ void k_bias_grad(const __nv_bfloat16* __restrict__ dy, float* __restrict__ db, int64_t M, int C) {
  const int c = blockIdx.y;
  float s = 0.f;
  for (int64_t m = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; m < M; m += (int64_t)gridDim.x * blockDim.x)
    s += __bfloat162float(dy[m * C + c]);
  for (int o = 16; o > 0; o >>= 1) s += __shfl_down_sync(0xffffffffu, s, o);
  if ((threadIdx.x & 31) == 0) atomicAdd(db + c, s);
}

// 2x average pooling (channels last) and its gradient
__global__ void k_pool2(const __nv_bfloat16* __restrict__ x, __nv_bfloat16* __restrict__ y, int N, int D,
                        int H, int W, int C) {
  const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  const int d = D / 2, h = H / 2, w = W / 2;
  const int64_t n = (int64_t)N * d * h * w * C;
  if (i >= n) return;
  const int c = (int)(i % C);
  Vox v = unflat(i / C, d, h, w);
  float s = 0.f;
  for (int a = 0; a < 2; ++a)
    for (int b = 0; b < 2; ++b)
      for (int e = 0; e < 2; ++e)
        s += __bfloat162float(x[((((int64_t)v.n * D + 2 * v.z + a) * H + 2 * v.y + b) * W + 2 * v.x + e) * C + c]);
  y[i] = __float2bfloat16_rn(0.125f * s);
}
__global__ void k_pool2_bwd(const __nv_bfloat16* __restrict__ dy, __nv_bfloat16* __restrict__ dx, int N,
                            int D, int H, int W, int C) {
  const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  const int64_t n = (int64_t)N * D * H * W * C;
  if (i >= n) return;
  const int c = (int)(i % C);
  Vox v = unflat(i / C, D, H, W);
  dx[i] = __float2bfloat16_rn(
      0.125f * __bfloat162float(dy[((((int64_t)v.n * (D / 2) + v.z / 2) * (H / 2) + v.y / 2) * (W / 2) + v.x / 2) * C + c]));
}
// nearest 2x upsampling and its gradient (sum over the 8 copies)
__global__ void k_up2(const __nv_bfloat16* __restrict__ x, __nv_bfloat16* __restrict__ y, int N, int D,
                      int H, int W, int C) {  // D, H, W: output (fine) sizes
  const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  const int64_t n = (int64_t)N * D * H * W * C;
  if (i >= n) return;
  const int c = (int)(i % C);
  Vox v = unflat(i / C, D, H, W);
  y[i] = x[((((int64_t)v.n * (D / 2) + v.z / 2) * (H / 2) + v.y / 2) * (W / 2) + v.x / 2) * C + c];
}
__global__ void k_up2_bwd(const __nv_bfloat16* __restrict__ dy, __nv_bfloat16* __restrict__ dx, int N, int D,
                          int H, int W, int C) {  // D, H, W: coarse sizes
  const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  const int64_t n = (int64_t)N * D * H * W * C;
  if (i >= n) return;
  const int c = (int)(i % C);
  Vox v = unflat(i / C, D, H, W);
  float s = 0.f;
  for (int a = 0; a < 2; ++a)
    for (int b = 0; b < 2; ++b)
      for (int e = 0; e < 2; ++e)
        s += __bfloat162float(dy[((((int64_t)v.n * 2 * D + 2 * v.z + a) * 2 * H + 2 * v.y + b) * 2 * W + 2 * v.x + e) * C + c]);
  dx[i] = __float2bfloat16_rn(s);
}
// channel concatenation y = [a | b] and its split
__global__ void k_concat(const __nv_bfloat16* __restrict__ a, int Ca, const __nv_bfloat16* __restrict__ b,
                         int Cb, __nv_bfloat16* __restrict__ y, int64_t M) {
  const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  const int C = Ca + Cb;
  if (i >= M * C) return;
  const int64_t m = i / C;
  const int c = (int)(i % C);
  y[i] = c < Ca ? a[m * Ca + c] : b[m * Cb + (c - Ca)];
}
__global__ void k_split(const __nv_bfloat16* __restrict__ y, __nv_bfloat16* __restrict__ da, int Ca,
                        __nv_bfloat16* __restrict__ db, int Cb, int64_t M, int accumulate_b) {
  const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  const int C = Ca + Cb;
  if (i >= M * C) return;
  const int64_t m = i / C;
  const int c = (int)(i % C);
  if (c < Ca) {
    da[m * Ca + c] = y[i];
  } else {
    const int64_t j = m * Cb + (c - Ca);
    db[j] = accumulate_b ? __float2bfloat16_rn(__bfloat162float(db[j]) + __bfloat162float(y[i])) : y[i];
  }
}
// in-place add: a += b
__global__ void k_add(__nv_bfloat16* __restrict__ a, const __nv_bfloat16* __restrict__ b, int64_t n) {
  const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) a[i] = __float2bfloat16_rn(__bfloat162float(a[i]) + __bfloat162float(b[i]));
}
// masked mean-squared error over voxels with mask > 0; returns loss sum in *loss
// and dy = 2 (pred - target) mask / count
__global__ void k_mse(const float* __restrict__ pred, const float* __restrict__ target,
                      const float* __restrict__ mask, __nv_bfloat16* __restrict__ dpred, float* __restrict__ loss,
                      int64_t M, int C, float inv_count) {
  const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  float l = 0.f;
  if (i < M * C) {
    const float mk = mask[i / C];
    const float d = (pred[i] - target[i]) * mk;
    l = d * d;
    dpred[i] = __float2bfloat16_rn(2.f * d * inv_count);
  }
  for (int o = 16; o > 0; o >>= 1) l += __shfl_down_sync(0xffffffffu, l, o);
  if ((threadIdx.x & 31) == 0) atomicAdd(loss, l);
}
// Adam on FP32 master weights, refreshing the BF16 copies: up to kAdamTensors tensors in
// a launch, 1,024 values of one tensor by a CTA.  A network has two tensors a layer, most
// of them small: one launch a tensor took 110 us for a step of the U-Net (30 tensors, 3.2M
// values) beside the gaps between them, this takes 15.
constexpr int kAdamTensors = 32, kAdamBlock = 1024;
struct AdamList {
  float* w[kAdamTensors];
  __nv_bfloat16* wb[kAdamTensors];
  const float* g[kAdamTensors];
  float* m[kAdamTensors];
  float* v[kAdamTensors];
  int64_t n[kAdamTensors];
  uint32_t first[kAdamTensors + 1];  // CTA each tensor starts at; the end
  int count;
};
__global__ void __launch_bounds__(256) k_adam(const __grid_constant__ AdamList a, float lr, float b1, float b2, float eps,
                                              float c1, float c2) {
  int t = 0;
  while (t + 1 < a.count && blockIdx.x >= a.first[t + 1]) ++t;
  const int64_t i0 = (int64_t)(blockIdx.x - a.first[t]) * kAdamBlock + threadIdx.x;
  float *w = a.w[t], *m = a.m[t], *v = a.v[t];
  const float* g = a.g[t];
  __nv_bfloat16* wb = a.wb[t];
  const int64_t n = a.n[t];
  wait_for_previous();
  float gi[4], mi[4], vi[4], wi[4];
#pragma unroll
  for (int k = 0; k < 4; ++k) {
    const int64_t i = i0 + k * 256;
    if (i < n) {
      gi[k] = g[i];
      mi[k] = m[i];
      vi[k] = v[i];
      wi[k] = w[i];
    }
  }
#pragma unroll
  for (int k = 0; k < 4; ++k) {
    const int64_t i = i0 + k * 256;
    if (i >= n) break;
    // fused as the compiler fused them in a kernel of one tensor: the same bits
    const float mn = __fmaf_rn(1.f - b1, gi[k], b1 * mi[k]);
    const float vn = __fmaf_rn((1.f - b2) * gi[k], gi[k], b2 * vi[k]);
    m[i] = mn;
    v[i] = vn;
    const float wn = wi[k] - lr * (mn * c1) / (sqrtf(vn * c2) + eps);
    w[i] = wn;
    if (wb) wb[i] = __float2bfloat16_rn(wn);
  }
}
__global__ void k_f32_to_bf16(const float* __restrict__ x, __nv_bfloat16* __restrict__ y, int64_t n) {
  const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) y[i] = __float2bfloat16_rn(x[i]);
}

// ---------------------------------------------------------------------------
// The channels-last element-wise passes in vectors of 8 channels (16 bytes).  Each is
// bound by HBM, so each reads and writes its tensors once, in 16-byte accesses, with
// 32-bit index arithmetic; what follows a pass directly in the network is fused into
// it (ReLU mask and bias sum, upsampling and concatenation, their gradients, pooling
// gradient and the sum into the skip's gradient).  The scalar kernels above take what
// these do not: channel counts that are no multiple of 8, buffers that are not
// 16-byte aligned, odd sizes, 2^31 vectors or more.  Values are the scalar kernels'
// bit for bit (same order of additions, same roundings); sums over voxels (bias,
// loss) run in FP32 per thread, per CTA, then one atomic per CTA and channel.
// A training step of the network at batch 4, 96^3 voxels, all levels, scalar -> vector
// (us): ReLU mask and bias sums 1457 + 2842 -> 318; upsampling and concatenation
// 1272 + 1116 -> 123; their gradients 214 + 1027 -> 111; loss 2872 (one atomic per
// warp on one word) -> 83 (6.9 TB/s); pooling gradient and sum 486 + 218 -> 50.
// These kernels, the Adam update, the flipped weights and the tcgen05 kernels are
// overlapped launches: each starts, up to its wait, while the last CTAs before it run,
// which took 1.9 us off each of a training step's 148 launches (90 since).  They let their
// successor in at their exit: CTAs let in earlier sit beside the running ones and end up
// unevenly on the SMs (training step 4580 us with ordinary launches, 4500 let in at the
// start, 4305 at the exit; prediction 448, 409, 399).
// ---------------------------------------------------------------------------
struct V8 {
  float v[8];
};
__device__ __forceinline__ V8 unpack8(uint4 u) {
  V8 r;
  const uint32_t w[4] = {u.x, u.y, u.z, u.w};
#pragma unroll
  for (int k = 0; k < 4; ++k) {
    r.v[2 * k] = __uint_as_float(w[k] << 16);
    r.v[2 * k + 1] = __uint_as_float(w[k] & 0xffff0000u);
  }
  return r;
}
__device__ __forceinline__ uint4 pack8(const V8& a) {
  uint32_t w[4];
#pragma unroll
  for (int k = 0; k < 4; ++k) {
    const __nv_bfloat162 h = __floats2bfloat162_rn(a.v[2 * k], a.v[2 * k + 1]);
    w[k] = *reinterpret_cast<const uint32_t*>(&h);
  }
  return make_uint4(w[0], w[1], w[2], w[3]);
}
// d where y > 0, else +0
__device__ __forceinline__ uint32_t mask_positive(uint32_t d, uint32_t y) {
  const __nv_bfloat162 z = __floats2bfloat162_rn(0.f, 0.f);
  return d & __hgt2_mask(*reinterpret_cast<const __nv_bfloat162*>(&y), z);
}

// dy *= (y > 0) in place (y not null) and db[c] += sum_m dy[m, c] (db not null).  A
// thread keeps one group of 8 channels (G groups) and walks the voxels; four rows in
// flight per thread.
__global__ void __launch_bounds__(256) k_relu_bias_v8(uint4* dy, const uint4* y,
                                                      float* db, uint32_t M, uint32_t G) {
  wait_for_previous();
  __shared__ float sh[256 * 8];
  const uint32_t rows = 256u / G, r = threadIdx.x / G, g = threadIdx.x - r * G;
  float acc[8];
#pragma unroll
  for (int k = 0; k < 8; ++k) acc[k] = 0.f;
  const uint32_t step = gridDim.x * rows;
  if (r < rows) {
    for (uint32_t m = blockIdx.x * rows + r; m < M; m += 4 * step) {
      uint4 d[4], yy[4];
#pragma unroll
      for (int u = 0; u < 4; ++u) {
        const uint32_t mu = m + u * step;
        d[u] = mu < M ? dy[(size_t)mu * G + g] : make_uint4(0u, 0u, 0u, 0u);
        if (y) yy[u] = mu < M ? *(y + (size_t)mu * G + g) : make_uint4(0u, 0u, 0u, 0u);
      }
#pragma unroll
      for (int u = 0; u < 4; ++u) {
        const uint32_t mu = m + u * step;
        if (y) {
          d[u].x = mask_positive(d[u].x, yy[u].x);
          d[u].y = mask_positive(d[u].y, yy[u].y);
          d[u].z = mask_positive(d[u].z, yy[u].z);
          d[u].w = mask_positive(d[u].w, yy[u].w);
          if (mu < M) dy[(size_t)mu * G + g] = d[u];
        }
        const V8 v = unpack8(d[u]);
#pragma unroll
        for (int k = 0; k < 8; ++k) acc[k] += v.v[k];
      }
    }
  }
  if (!db) return;
#pragma unroll
  for (int k = 0; k < 8; ++k) sh[threadIdx.x * 8 + k] = acc[k];
  __syncthreads();
  // rows of a channel in a fixed order, then one atomic
  for (uint32_t c = threadIdx.x; c < 8 * G; c += 256) {
    float s = 0.f;
    for (uint32_t q = 0; q < rows; ++q) s += sh[q * G * 8 + c];
    atomicAdd(db + c, s);
  }
}

// One thread per coarse voxel and 8 channels: its 8 fine voxels.  Sizes are fine.
struct Fine {
  uint32_t first, zs, ys;  // first fine voxel, strides of z and y in voxels
};
__device__ __forceinline__ Fine fine_of(uint32_t cv, uint32_t D, uint32_t H, uint32_t W) {
  const uint32_t w = W / 2, h = H / 2, d = D / 2;
  const uint32_t x = cv % w, t = cv / w, y = t % h, q = t / h, z = q % d, n = q / d;
  return Fine{((n * D + 2 * z) * H + 2 * y) * W + 2 * x, H * W, W};
}
__device__ __forceinline__ uint32_t fine_at(const Fine& f, int k) {  // k = 4 z + 2 y + x
  return f.first + (k >> 2) * f.zs + ((k >> 1) & 1) * f.ys + (k & 1);
}

__global__ void __launch_bounds__(256) k_pool2_v8(const uint4* x, uint4* y, uint32_t nv,
                                                  uint32_t G, uint32_t D, uint32_t H, uint32_t W) {
  wait_for_previous();
  const uint32_t i = blockIdx.x * 256 + threadIdx.x;
  if (i >= nv) return;
  const uint32_t cv = i / G, g = i - cv * G;
  const Fine f = fine_of(cv, D, H, W);
  uint4 u[8];
#pragma unroll
  for (int k = 0; k < 8; ++k) u[k] = *(x + (size_t)fine_at(f, k) * G + g);
  V8 s = {};
#pragma unroll
  for (int k = 0; k < 8; ++k) {
    const V8 v = unpack8(u[k]);
#pragma unroll
    for (int c = 0; c < 8; ++c) s.v[c] += v.v[c];
  }
#pragma unroll
  for (int c = 0; c < 8; ++c) s.v[c] *= 0.125f;
  y[i] = pack8(s);
}
// dx = dy / 8 spread over the 8 fine voxels (acc null), or acc += that (rounded to
// BF16 first, as the two passes round)
__global__ void __launch_bounds__(256) k_pool2_bwd_v8(const uint4* dy, uint4* dx,
                                                      uint32_t nv, uint32_t G, uint32_t D, uint32_t H, uint32_t W,
                                                      int add) {
  wait_for_previous();
  const uint32_t i = blockIdx.x * 256 + threadIdx.x;
  if (i >= nv) return;
  const uint32_t cv = i / G, g = i - cv * G;
  const Fine f = fine_of(cv, D, H, W);
  V8 v = unpack8(*(dy + i));
#pragma unroll
  for (int c = 0; c < 8; ++c) v.v[c] *= 0.125f;
  const uint4 q = pack8(v);
  if (!add) {
#pragma unroll
    for (int k = 0; k < 8; ++k) dx[(size_t)fine_at(f, k) * G + g] = q;
    return;
  }
  const V8 t = unpack8(q);
  uint4 u[8];
#pragma unroll
  for (int k = 0; k < 8; ++k) u[k] = dx[(size_t)fine_at(f, k) * G + g];
#pragma unroll
  for (int k = 0; k < 8; ++k) {
    V8 b = unpack8(u[k]);
#pragma unroll
    for (int c = 0; c < 8; ++c) b.v[c] += t.v[c];
    dx[(size_t)fine_at(f, k) * G + g] = pack8(b);
  }
}
// y (fine, Ga + Gb groups a voxel) = [x of the coarse voxel | skip]
__global__ void __launch_bounds__(256) k_up2_concat_v8(const uint4* x, uint32_t Ga,
                                                       const uint4* skip, uint32_t Gb,
                                                       uint4* y, uint32_t nv, uint32_t D, uint32_t H,
                                                       uint32_t W) {
  wait_for_previous();
  const uint32_t i = blockIdx.x * 256 + threadIdx.x, G = Ga + Gb;
  if (i >= nv) return;
  const uint32_t cv = i / G, g = i - cv * G;
  const Fine f = fine_of(cv, D, H, W);
  if (g < Ga) {
    const uint4 v = *(x + (size_t)cv * Ga + g);
#pragma unroll
    for (int k = 0; k < 8; ++k) y[(size_t)fine_at(f, k) * G + g] = v;
  } else {
    uint4 v[8];
#pragma unroll
    for (int k = 0; k < 8; ++k) v[k] = *(skip + (size_t)fine_at(f, k) * Gb + (g - Ga));
#pragma unroll
    for (int k = 0; k < 8; ++k) y[(size_t)fine_at(f, k) * G + g] = v[k];
  }
}
// its gradient: dx (coarse) = sum of the 8 fine values, dskip = the other channels
__global__ void __launch_bounds__(256) k_up2_split_v8(const uint4* dy, uint4* dx,
                                                      uint32_t Ga, uint4* dskip, uint32_t Gb,
                                                      uint32_t nv, uint32_t D, uint32_t H, uint32_t W) {
  wait_for_previous();
  const uint32_t i = blockIdx.x * 256 + threadIdx.x, G = Ga + Gb;
  if (i >= nv) return;
  const uint32_t cv = i / G, g = i - cv * G;
  const Fine f = fine_of(cv, D, H, W);
  uint4 u[8];
#pragma unroll
  for (int k = 0; k < 8; ++k) u[k] = *(dy + (size_t)fine_at(f, k) * G + g);
  if (g < Ga) {
    V8 s = {};
#pragma unroll
    for (int k = 0; k < 8; ++k) {
      const V8 v = unpack8(u[k]);
#pragma unroll
      for (int c = 0; c < 8; ++c) s.v[c] += v.v[c];
    }
    dx[(size_t)cv * Ga + g] = pack8(s);
  } else {
#pragma unroll
    for (int k = 0; k < 8; ++k) dskip[(size_t)fine_at(f, k) * Gb + (g - Ga)] = u[k];
  }
}

// Masked squared error, 4 values of one voxel per vector (C a multiple of 4)
__global__ void __launch_bounds__(256) k_mse_v4(const float4* pred, const float4* target,
                                                const float* mask, uint2* dpred,
                                                float* loss, uint32_t nv, uint32_t G, float inv_count) {
  wait_for_previous();
  __shared__ float sh[8];
  float l = 0.f;
  const uint32_t step = gridDim.x * 256;
  for (uint32_t i0 = blockIdx.x * 256 + threadIdx.x; i0 < nv; i0 += 4 * step) {
    float4 p[4], t[4];
    float mk[4];
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      const uint32_t i = i0 + u * step;
      const bool ok = i < nv;
      p[u] = ok ? *(pred + i) : make_float4(0.f, 0.f, 0.f, 0.f);
      t[u] = ok ? *(target + i) : make_float4(0.f, 0.f, 0.f, 0.f);
      mk[u] = ok ? *(mask + i / G) : 0.f;
    }
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      const uint32_t i = i0 + u * step;
      if (i >= nv) break;
      const float a = (p[u].x - t[u].x) * mk[u], b = (p[u].y - t[u].y) * mk[u], c = (p[u].z - t[u].z) * mk[u],
                  d = (p[u].w - t[u].w) * mk[u];
      l += (a * a + b * b) + (c * c + d * d);
      const __nv_bfloat162 lo = __floats2bfloat162_rn(2.f * a * inv_count, 2.f * b * inv_count);
      const __nv_bfloat162 hi = __floats2bfloat162_rn(2.f * c * inv_count, 2.f * d * inv_count);
      dpred[i] = make_uint2(*reinterpret_cast<const uint32_t*>(&lo), *reinterpret_cast<const uint32_t*>(&hi));
    }
  }
  for (int o = 16; o > 0; o >>= 1) l += __shfl_down_sync(0xffffffffu, l, o);
  if ((threadIdx.x & 31) == 0) sh[threadIdx.x >> 5] = l;
  __syncthreads();
  if (threadIdx.x == 0) {
#pragma unroll
    for (int k = 1; k < 8; ++k) l += sh[k];
    atomicAdd(loss, l);
  }
}

inline bool aligned16(const void* a, const void* b = nullptr, const void* c = nullptr) {
  return ((reinterpret_cast<uintptr_t>(a) | reinterpret_cast<uintptr_t>(b) | reinterpret_cast<uintptr_t>(c)) & 15u) ==
         0;
}
// vectors of 8 channels, 32-bit indices
inline bool vec8(int64_t elems, int64_t c) { return c > 0 && c % 8 == 0 && elems > 0 && elems / 8 < 0x7fff0000ll; }
inline bool even3(int32_t d, int32_t h, int32_t w) { return d % 2 == 0 && h % 2 == 0 && w % 2 == 0; }

// ReLU mask and bias sum in one pass: 8 CTAs of 256 threads a SM, at least
// four rows a thread.  False: not a shape of the vector kernel.
inline bool relu_bias(void* dy, const void* y, float* db, int64_t m, int32_t c, cudaStream_t st) {
  if (!vec8(m * c, c) || c > 2048 || m >= 0x7fff0000ll || !aligned16(dy, y)) return false;
  const uint32_t G = (uint32_t)c / 8, rows = 256 / G;
  const int64_t want = (m + 4 * rows - 1) / (4 * rows);
  launch_overlapped(k_relu_bias_v8, (unsigned)std::min<int64_t>(want, 8 * hlbg::sm_count()), 256, 0, st, (uint4*)dy, (const uint4*)y, db,
                    (uint32_t)m, G);
  return true;
}

inline unsigned blocks(int64_t n, int t = 256) { return (unsigned)((n + t - 1) / t); }

// Modelled microseconds of k_wgrad_brick, bpc bricks a CTA, for nbricks bricks of `shares`
// channel blocks (as wgrad_tc_time): rounds of two CTAs an SM, which slow each other down,
// and the additions to dw by their number and by the CTAs that meet at an address.
inline double wgrad_mma_time(int cin, int cout, int nci, int64_t bpc, int64_t nbricks, int shares, int sms) {
  const double gx = (double)((nbricks + bpc - 1) / bpc), ctas = gx * shares, per = ctas / (2.0 * sms);
  const double rounds = per > 2 ? per : std::max(1.0, std::ceil(per)), resident = std::min(2.0, std::max(1.0, ctas / sms));
  const double chain = rounds * ((double)bpc * (nci == 2 ? 1.5 : 0.93) * (1 + 2.4 * (resident - 1)) + (nci == 2 ? 1.5 : 0.2));
  const double adds = gx * 27e-6 * cin * cout * 2.0, meet = 0.061 * gx;
  return 3.5 + std::sqrt(std::sqrt(chain * chain * chain * chain + adds * adds * adds * adds + meet * meet * meet * meet));
}

int check_launch() { return cudaGetLastError() == cudaSuccess ? 0 : 3; }

}  // namespace

extern "C" {

// hlbg_nn_conv3d_wgrad_tc where its modelled time is within `limit` microseconds
// (nn_tc.cu; 1x1x1 has no model), else 1.
int hlbg_nn_wgrad_tc_within(const void* x, int32_t cin, const void* dy, int32_t cout, float* dw, int32_t n, int32_t d,
                            int32_t h, int32_t wd, int32_t taps, void* stream, double limit);

int hlbg_nn_conv3d(const void* in, int32_t cin, const void* w, const float* bias, void* out, float* out_f32,
                   int32_t cout, int32_t n, int32_t d, int32_t h, int32_t wd, int32_t taps, int32_t relu,
                   void* stream) {
  if (!in || !w || !out || cin <= 0 || cin % 16 || cout <= 0 || (taps != 27 && taps != 1)) return 1;
  const int64_t M = (int64_t)n * d * h * wd;
  cudaStream_t st = (cudaStream_t)stream;
  if (taps == 27 && cout % 16 == 0) {
    const int nbz = (d + kBZ - 1) / kBZ, nby = (h + kBY - 1) / kBY, nbx = (wd + kBX - 1) / kBX;
    const int64_t nbricks = (int64_t)n * nbz * nby * nbx;
    auto I = (const __nv_bfloat16*)in;
    auto Wt = (const __nv_bfloat16*)w;
    auto O = (__nv_bfloat16*)out;
    if (cout % 64 == 0) {
      dim3 grid((unsigned)nbricks, (unsigned)(cout / 64));
      k_conv_brick<4><<<grid, 256, 0, st>>>(I, cin, Wt, bias, O, out_f32, cout, d, h, wd, nbz, nby, nbx, relu);
    } else if (cout % 32 == 0) {
      dim3 grid((unsigned)nbricks, (unsigned)(cout / 32));
      k_conv_brick<2><<<grid, 256, 0, st>>>(I, cin, Wt, bias, O, out_f32, cout, d, h, wd, nbz, nby, nbx, relu);
    } else {
      dim3 grid((unsigned)nbricks, (unsigned)(cout / 16));
      k_conv_brick<1><<<grid, 256, 0, st>>>(I, cin, Wt, bias, O, out_f32, cout, d, h, wd, nbz, nby, nbx, relu);
    }
    return check_launch();
  }
  const int warps = (int)((M + 15) / 16);
  dim3 grid((unsigned)((warps + 3) / 4), 1);
  auto I = (const __nv_bfloat16*)in;
  auto Wt = (const __nv_bfloat16*)w;
  auto O = (__nv_bfloat16*)out;
  if (cout % 32 == 0) {
    grid.y = cout / 32;
    k_conv3d<4><<<grid, 128, 0, st>>>(I, cin, Wt, bias, O, out_f32, cout, n, d, h, wd, taps, relu);
  } else {
    grid.y = (cout + 7) / 8;
    k_conv3d<1><<<grid, 128, 0, st>>>(I, cin, Wt, bias, O, out_f32, cout, n, d, h, wd, taps, relu);
  }
  return check_launch();
}

int hlbg_nn_conv3d_wgrad(const void* x, int32_t cin, const void* dy, int32_t cout, float* dw, int32_t n,
                         int32_t d, int32_t h, int32_t wd, int32_t taps, void* stream) {
  if (!x || !dy || !dw || cin % 8 || cout <= 0) return 1;
  const bool by16 = cin % 16 == 0 && cout % 16 == 0;
  const int nbz = (d + kBZ - 1) / kBZ, nby = (h + kBY - 1) / kBY, nbx = (wd + kBX - 1) / kBX;
  const int64_t nbricks = (int64_t)n * nbz * nby * nbx;
  const int nci = cin % 32 == 0 ? 2 : 1;
  const int gy = cout / 16, gz = cin / (16 * nci);
  // about four waves of 2 CTAs per SM
  const int sms = hlbg::sm_count();
  const int64_t bpc = std::max<int64_t>(1, (nbricks * gy * gz + 8 * sms - 1) / (8 * sms));
  // The tcgen05 kernel where it is the faster one.  1x1x1: from 17 voxels on (us, mma.sync /
  // tcgen05, 96 -> 96: 8 voxels 2.7 / 3.5, 27 5.2 / 3.5, 4,096 436 / 4).  3x3x3: by the
  // modelled times (96 -> 96: 96 x 3 x 3 voxels 17.0 / 25.0, 24^3 50 / 25).
  const int64_t M = (int64_t)n * d * h * wd;
  if (by16 && aligned16(x, dy, dw) && (taps == 27 || M > 16)) {
    const double limit = taps == 27 ? wgrad_mma_time(cin, cout, nci, bpc, nbricks, gy * gz, sms) : 0.0;
    const int rc = hlbg_nn_wgrad_tc_within(x, cin, dy, cout, dw, n, d, h, wd, taps, stream, limit);
    if (rc != 1) return rc;
  }
  if (taps == 27 && by16) {
    dim3 grid((unsigned)((nbricks + bpc - 1) / bpc), (unsigned)gy, (unsigned)gz);
    auto X = (const __nv_bfloat16*)x;
    auto DY = (const __nv_bfloat16*)dy;
    if (nci == 2)
      k_wgrad_brick<2><<<grid, 256, 0, (cudaStream_t)stream>>>(X, cin, DY, cout, dw, d, h, wd, nbz, nby, nbx,
                                                                nbricks, (int)bpc);
    else
      k_wgrad_brick<1><<<grid, 256, 0, (cudaStream_t)stream>>>(X, cin, DY, cout, dw, d, h, wd, nbz, nby, nbx,
                                                                nbricks, (int)bpc);
    return check_launch();
  }
  const int64_t ntile = (int64_t)taps * ((cout + 15) / 16) * (cin / 8);
  const int64_t slice = 4096;
  dim3 grid((unsigned)((ntile + 3) / 4), (unsigned)((M + slice - 1) / slice));
  k_conv3d_wgrad<<<grid, 128, 0, (cudaStream_t)stream>>>((const __nv_bfloat16*)x, cin, (const __nv_bfloat16*)dy,
                                                        cout, dw, n, d, h, wd, taps, slice);
  return check_launch();
}

int hlbg_nn_flip_transpose(const void* w, void* wt, int32_t cout, int32_t cin, int32_t taps, void* stream) {
  const int64_t tiles = (int64_t)((cin + 31) / 32) * ((cout + 31) / 32) * taps;
  launch_overlapped(k_flip_transpose, (unsigned)tiles, 256, 0, (cudaStream_t)stream, (const __nv_bfloat16*)w, (__nv_bfloat16*)wt,
                    cout, cin, taps);
  return check_launch();
}

int hlbg_nn_relu_bwd(void* dy, const void* y, int64_t n, void* stream) {
  // From 2^18 values on in vectors (us, scalar / vector: 31,104 values 1.1 / 1.3, 110,592
  // 1.2 / 1.3, 331,776 1.4 / 1.4, 663,552 2.2 / 1.5)
  if (n >= 1 << 18 && n % 8 == 0 && relu_bias(dy, y, nullptr, n / 8, 8, (cudaStream_t)stream)) return check_launch();
  k_relu_bwd<<<blocks(n), 256, 0, (cudaStream_t)stream>>>((__nv_bfloat16*)dy, (const __nv_bfloat16*)y, n);
  return check_launch();
}

int hlbg_nn_bias_grad(const void* dy, float* db, int64_t m, int32_t c, void* stream) {
  // A small tensor of few channels is done in the scalar kernel before a CTA of the vector
  // kernel has added its rows, 256 for 8 channels (us, scalar / vector: 8 channels, 216
  // voxels 1.4 / 2.3, 1,728 1.8 / 2.5, 6,912 3.6 / 2.3; 16 channels, 216 1.5 / 1.8, 1,728
  // 2.1 / 1.7; 24 channels, 216 1.3 / 1.5; 48 the same in both).
  const bool small = c < 48 && m <= (c <= 8 ? 2048 : 512);
  if (!small && relu_bias(const_cast<void*>(dy), nullptr, db, m, c, (cudaStream_t)stream)) return check_launch();  // reads dy
  dim3 grid((unsigned)std::min<int64_t>((m + 255) / 256, 512), (unsigned)c);
  k_bias_grad<<<grid, 256, 0, (cudaStream_t)stream>>>((const __nv_bfloat16*)dy, db, m, c);
  return check_launch();
}

int hlbg_nn_relu_bias_bwd(void* dy, const void* y, float* db, int64_t m, int32_t c, void* stream) {
  if (relu_bias(dy, y, db, m, c, (cudaStream_t)stream)) return check_launch();
  const int rc = hlbg_nn_relu_bwd(dy, y, m * c, stream);
  return rc ? rc : hlbg_nn_bias_grad(dy, db, m, c, stream);
}

int hlbg_nn_pool2(const void* x, void* y, int32_t n, int32_t d, int32_t h, int32_t w, int32_t c, int32_t backward,
                  void* stream) {
  cudaStream_t st = (cudaStream_t)stream;
  const int64_t fine = (int64_t)n * d * h * w * c;
  if (vec8(fine, c) && even3(d, h, w) && aligned16(x, y)) {
    const uint32_t nv = (uint32_t)(fine / 64);
    if (!backward)
      launch_overlapped(k_pool2_v8, blocks(nv), 256, 0, st, (const uint4*)x, (uint4*)y, nv, c / 8, d, h, w);
    else
      launch_overlapped(k_pool2_bwd_v8, blocks(nv), 256, 0, st, (const uint4*)x, (uint4*)y, nv, c / 8, d, h, w, 0);
    return check_launch();
  }
  if (!backward) {
    const int64_t cnt = (int64_t)n * (d / 2) * (h / 2) * (w / 2) * c;
    k_pool2<<<blocks(cnt), 256, 0, st>>>((const __nv_bfloat16*)x, (__nv_bfloat16*)y, n, d, h, w, c);
  } else {  // x = dy (coarse), y = dx (fine); d, h, w fine sizes
    const int64_t cnt = (int64_t)n * d * h * w * c;
    k_pool2_bwd<<<blocks(cnt), 256, 0, st>>>((const __nv_bfloat16*)x, (__nv_bfloat16*)y, n, d, h, w, c);
  }
  return check_launch();
}

int hlbg_nn_up2(const void* x, void* y, int32_t n, int32_t d, int32_t h, int32_t w, int32_t c, int32_t backward,
                void* stream) {
  cudaStream_t st = (cudaStream_t)stream;
  const int64_t cnt = (int64_t)n * d * h * w * c;
  if (!backward && vec8(cnt, c) && even3(d, h, w) && aligned16(x, y)) {
    const uint32_t nv = (uint32_t)(cnt / 64);
    launch_overlapped(k_up2_concat_v8, blocks(nv), 256, 0, st, (const uint4*)x, c / 8, (const uint4*)nullptr, 0,
                      (uint4*)y, nv, d, h, w);
    return check_launch();
  }
  if (backward && vec8(8 * cnt, c) && aligned16(x, y)) {
    const uint32_t nv = (uint32_t)(cnt / 8);
    launch_overlapped(k_up2_split_v8, blocks(nv), 256, 0, st, (const uint4*)x, (uint4*)y, c / 8, (uint4*)nullptr, 0, nv,
                      2 * d, 2 * h, 2 * w);
    return check_launch();
  }
  if (!backward)  // d, h, w fine sizes
    k_up2<<<blocks(cnt), 256, 0, st>>>((const __nv_bfloat16*)x, (__nv_bfloat16*)y, n, d, h, w, c);
  else  // x = dy (fine), y = dx (coarse); d, h, w coarse sizes
    k_up2_bwd<<<blocks(cnt), 256, 0, st>>>((const __nv_bfloat16*)x, (__nv_bfloat16*)y, n, d, h, w, c);
  return check_launch();
}

int hlbg_nn_concat(const void* a, int32_t ca, const void* b, int32_t cb, void* y, int64_t m, void* stream) {
  k_concat<<<blocks(m * (ca + cb)), 256, 0, (cudaStream_t)stream>>>((const __nv_bfloat16*)a, ca,
                                                                      (const __nv_bfloat16*)b, cb,
                                                                      (__nv_bfloat16*)y, m);
  return check_launch();
}

int hlbg_nn_split(const void* y, void* da, int32_t ca, void* db, int32_t cb, int64_t m, int32_t accumulate_b,
                  void* stream) {
  k_split<<<blocks(m * (ca + cb)), 256, 0, (cudaStream_t)stream>>>((const __nv_bfloat16*)y, (__nv_bfloat16*)da,
                                                                     ca, (__nv_bfloat16*)db, cb, m, accumulate_b);
  return check_launch();
}

int hlbg_nn_up2_concat(const void* x, int32_t ca, const void* skip, int32_t cb, void* y, int32_t n, int32_t d,
                       int32_t h, int32_t w, void* stream) {
  const int64_t cnt = (int64_t)n * d * h * w * (ca + cb);
  if (ca <= 0 || cb <= 0 || ca % 8 || cb % 8 || !vec8(cnt, ca + cb) || !even3(d, h, w) || !aligned16(x, skip, y)) return 1;
  const uint32_t nv = (uint32_t)(cnt / 64);
  launch_overlapped(k_up2_concat_v8, blocks(nv), 256, 0, (cudaStream_t)stream, (const uint4*)x, ca / 8,
                    (const uint4*)skip, cb / 8, (uint4*)y, nv, d, h, w);
  return check_launch();
}

int hlbg_nn_up2_split(const void* dy, void* dx, int32_t ca, void* dskip, int32_t cb, int32_t n, int32_t d, int32_t h,
                      int32_t w, void* stream) {
  const int64_t cnt = (int64_t)n * d * h * w * (ca + cb);
  if (ca <= 0 || cb <= 0 || ca % 8 || cb % 8 || !vec8(cnt, ca + cb) || !even3(d, h, w) || !aligned16(dy, dx, dskip)) return 1;
  const uint32_t nv = (uint32_t)(cnt / 64);
  launch_overlapped(k_up2_split_v8, blocks(nv), 256, 0, (cudaStream_t)stream, (const uint4*)dy, (uint4*)dx, ca / 8,
                    (uint4*)dskip, cb / 8, nv, d, h, w);
  return check_launch();
}

int hlbg_nn_pool2_bwd_add(const void* dy, void* acc, int32_t n, int32_t d, int32_t h, int32_t w, int32_t c,
                          void* stream) {
  const int64_t cnt = (int64_t)n * d * h * w * c;
  if (!vec8(cnt, c) || !even3(d, h, w) || !aligned16(dy, acc)) return 1;
  const uint32_t nv = (uint32_t)(cnt / 64);
  launch_overlapped(k_pool2_bwd_v8, blocks(nv), 256, 0, (cudaStream_t)stream, (const uint4*)dy, (uint4*)acc, nv, c / 8, d,
                    h, w, 1);
  return check_launch();
}

int hlbg_nn_add(void* a, const void* b, int64_t n, void* stream) {
  k_add<<<blocks(n), 256, 0, (cudaStream_t)stream>>>((__nv_bfloat16*)a, (const __nv_bfloat16*)b, n);
  return check_launch();
}

int hlbg_nn_mse(const float* pred, const float* target, const float* mask, void* dpred, float* loss, int64_t m,
                int32_t c, float inv_count, void* stream) {
  if (c > 0 && c % 4 == 0 && m > 0 && m * c / 4 < 0x7fff0000ll && aligned16(pred, target, dpred)) {
    const uint32_t nv = (uint32_t)(m * c / 4);
    const unsigned g = std::min(blocks((nv + 3) / 4), 8u * hlbg::sm_count());  // 8 CTAs a SM; one atomic per CTA
    launch_overlapped(k_mse_v4, g, 256, 0, (cudaStream_t)stream, (const float4*)pred, (const float4*)target, mask,
                      (uint2*)dpred, loss, nv, c / 4, inv_count);
    return check_launch();
  }
  k_mse<<<blocks(m * c), 256, 0, (cudaStream_t)stream>>>(pred, target, mask, (__nv_bfloat16*)dpred, loss, m, c,
                                                         inv_count);
  return check_launch();
}

int hlbg_nn_adam_list(float* const* w, void* const* wb, const float* const* g, float* const* m, float* const* v,
                      const int64_t* n, int32_t count, float lr, float b1, float b2, float eps, int32_t step,
                      void* stream) {
  if (count < 0 || (count > 0 && (!w || !wb || !g || !m || !v || !n))) return 1;
  const float c1 = 1.f / (1.f - powf(b1, (float)step)), c2 = 1.f / (1.f - powf(b2, (float)step));
  AdamList a;
  a.count = 0;
  a.first[0] = 0;
  for (int32_t i = 0; i < count; ++i) {
    const int64_t ctas = (n[i] + kAdamBlock - 1) / kAdamBlock;
    if (n[i] < 0 || ctas > 0x3fffffff) return 1;
    if (ctas > 0) {
      const int k = a.count++;
      a.w[k] = w[i];
      a.wb[k] = static_cast<__nv_bfloat16*>(wb[i]);
      a.g[k] = g[i];
      a.m[k] = m[i];
      a.v[k] = v[i];
      a.n[k] = n[i];
      a.first[k + 1] = a.first[k] + (uint32_t)ctas;
    }
    if (a.count == 0 || (a.count < kAdamTensors && i + 1 < count && a.first[a.count] < 0x3fffffffu)) continue;
    launch_overlapped(k_adam, a.first[a.count], 256, 0, (cudaStream_t)stream, a, lr, b1, b2, eps, c1, c2);
    a.count = 0;
  }
  return check_launch();
}

int hlbg_nn_adam(float* w, void* wb, const float* g, float* m, float* v, int64_t n, float lr, float b1, float b2,
                 float eps, int32_t step, void* stream) {
  if (n <= 0) return 3;  // as a launch of no threads
  return hlbg_nn_adam_list(&w, &wb, &g, &m, &v, &n, 1, lr, b1, b2, eps, step, stream);
}

int hlbg_nn_to_bf16(const float* x, void* y, int64_t n, void* stream) {
  k_f32_to_bf16<<<blocks(n), 256, 0, (cudaStream_t)stream>>>(x, (__nv_bfloat16*)y, n);
  return check_launch();
}

}  // extern "C"
