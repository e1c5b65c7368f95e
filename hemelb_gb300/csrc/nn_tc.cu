// 3x3x3 convolution of the warm-start surrogate on the fifth-generation tensor
// cores: tcgen05.mma with the accumulators in tensor memory (TMEM), operands staged
// in shared memory by TMA (cp.async.bulk.tensor), completion tracked on mbarriers.
//
// Implicit GEMM, z-stacked.  One CTA computes a column of 8 (x) x 16 (y) x bz (z)
// voxels for `ct` output channels: one FP32 accumulator of ct TMEM columns per plane.
// The reduction runs over C_in in slices of 16 channels (K = 16 of an MMA) and, within
// a slice, over the bz + 2 input planes and the nine (dy, dx) taps:
//  * an input plane q feeds the output planes q + 1, q, q - 1 through the taps dz = 0,
//    1, 2.  Their accumulators are neighbours in TMEM (planes in descending order) and
//    the weights of the three dz are neighbours in shared memory, so one MMA of
//    N = 3 ct does the three taps: the A operand, whose read from shared memory (4 KB,
//    32 cycles) bounds an MMA of N < 128, is read once instead of three times;
//  * a TMA load brings an input plane with its halo -- 10 x 18 voxels, up to 64
//    channels, positions outside the volume (and channels past C_in) read as zeros,
//    which is the convolution's zero padding -- as rows of 32, 64 or 128 bytes in the
//    swizzle of that width.  The swizzle is a function of the shared-memory address, so
//    a tap (dy, dx) is a start address in the tile and a 16-channel slice another, with
//    8-row groups (8 consecutive x) one halo row of 10 voxels apart.  TMA moves about
//    one row a cycle whatever its width: with two loads of 8 channels (16-byte rows) per
//    slice it took 365 cycles a plane and slice, more than the nine MMAs;
//  * per slice, three TMA loads (one per dy) bring the 27 taps' weights, rows of 32
//    bytes in the 32-byte swizzle, ordered dx, dz, output channel; two buffers.
// Per output value the products are added in the order slice, dz, dy, dx, whatever the
// tile: the same order, and the same bits, as k_conv_brick (mma.sync); so the planes of
// a load stay in shared memory until their last slice is done.  The accumulators start
// as zeros.  Only MMAs of one accumulator range and shape are ordered by the hardware,
// so the MMAs of a plane wait for those of the plane before to complete unless the column
// is one plane high; a CTA therefore works on one to four such columns, each with a warp
// of its own, and several CTAs share an SM where TMEM and shared memory allow, to keep
// the pipe busy.
// CTAs are persistent.  One thread loads planes, one weights; the MMA warps run in uniform
// control flow, their lane 0 issues and returns each buffer with tcgen05.commit; four warps
// read the accumulators from TMEM (TMEM lanes 32w..32w+31: the rows y = 4w..4w+3 of the
// tile), add the bias, apply the ReLU, store BF16 (and optionally FP32) channels-last and
// clear the accumulators again.  Each of these runs ahead of the next, into the next tile:
// with one tile a CTA the first loads (4,000 cycles), the MMAs (12,000) and the epilogue
// (7,000) of a 16-channel tile ran one after the other, on all SMs at once.  The tile
// (ct, bz, cols) and the number of sets of accumulators are chosen per call by conv_plan.
// An MMA costs an SM max(N / 2, 36 + N / 5) cycles (measured, M = 128, K = 16, any
// layout), so stacking dz also lifts the pipe's use from 21 % (N = 16) to 55 %.  What
// bounds it now: that pipe at 16 channels (four columns an SM, 1,640 of 1,900 cycles a
// round), elsewhere the issue, 65 to 80 cycles an MMA.
// Measured at batch 4, C_in -> C_out at voxels (us; with one MMA per tap and plane, tiles
// of 8 x 16 x 2, one tile a CTA, 16-byte rows; z-stacked, issued from a branch of one lane
// and every plane waited for; now): 16 -> 16 at 96^3 208, 79, 74; 64 -> 16 568, 258, 241;
// 16 -> 64 412, 226, 171; 48 -> 48 at 48^3 89, 65, 52; 144 -> 48 214, 147, 115; 48 -> 144
// 226, 172, 135; 96 -> 96 at 24^3 44, 41, 29; 288 -> 96 103, 84, 65; 96 -> 288 309
// (mma.sync), 100, 77; 192 -> 192 at 12^3 95 (mma.sync), 34, 26; 1x1x1 16 -> 16 at 96^3,
// batch 1, 28 (planes loaded with a halo), 14.
//
// Every wait is bounded: a wait that gives up sets g_tc_err (read back by
// hlbg_nn_tc_error), the CTA waits (bounded) for the copies it issued, frees its
// TMEM and returns.  Tensor maps cover this GPU's own memory only (no multicast).
#include <cuda.h>
#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <cudaTypedefs.h>
#include <stdint.h>

#include <algorithm>
#include <atomic>
#include <cmath>
#include <mutex>

#include "../../include/hemelb_gb300_nn.h"
#include "overlap.cuh"
#include "sm_count.h"

namespace {

constexpr int kM = 128;            // rows of one MMA: an 8 x 16 plane of voxels
// Input plane of a tile: with its halo in x and y for 3x3x3 (full), without for 1x1x1.
__host__ __device__ constexpr int plane_x(bool full) { return full ? 10 : 8; }
__host__ __device__ constexpr int plane_y(bool full) { return full ? 18 : 16; }
__host__ __device__ constexpr int plane_rows(bool full) { return plane_x(full) * plane_y(full); }
constexpr int kMaxAStages = 40;
// Bytes of a plane's stage for rows of `span` bytes: whole swizzle atoms of 8 rows.
__host__ __device__ constexpr int stage_bytes(int span, bool full) {
  return (plane_rows(full) * span + 8 * span - 1) / (8 * span) * (8 * span);
}
constexpr int64_t kWaitLimit = 1ll << 22;    // polls before a wait gives up

__device__ int g_tc_err;

__device__ __forceinline__ uint32_t smem_u32(const void* p) {
  return (uint32_t)__cvta_generic_to_shared(p);
}

__device__ __forceinline__ void mbar_init(uint32_t bar, uint32_t count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(bar), "r"(count) : "memory");
}

__device__ __forceinline__ void mbar_expect_tx(uint32_t bar, uint32_t bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(bytes) : "memory");
}

__device__ __forceinline__ bool mbar_wait(uint32_t bar, uint32_t parity) {
  for (int64_t it = 0; it < kWaitLimit; ++it) {
    uint32_t done;
    asm volatile(
        "{\n .reg .pred p;\n mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n"
        " selp.u32 %0, 1, 0, p;\n}\n"
        : "=r"(done)
        : "r"(bar), "r"(parity)
        : "memory");
    if (done) return true;
  }
  return false;
}

// The same by a whole warp, one answer for all its lanes.
__device__ __forceinline__ bool warp_wait(uint32_t bar, uint32_t parity) {
  return __all_sync(0xffffffffu, mbar_wait(bar, parity));
}

// 32 bytes to a 32-byte aligned address: one whole sector.
__device__ __forceinline__ void store32(void* p, const uint32_t* v) {
  asm volatile("st.global.v8.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8};" ::"l"(p), "r"(v[0]), "r"(v[1]), "r"(v[2]),
               "r"(v[3]), "r"(v[4]), "r"(v[5]), "r"(v[6]), "r"(v[7])
               : "memory");
}

__device__ __forceinline__ void tma_load_5d(uint32_t dst, const CUtensorMap* map, uint32_t bar, int c0, int c1,
                                            int c2, int c3, int c4) {
  asm volatile(
      "cp.async.bulk.tensor.5d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4, %5, %6, "
      "%7}], [%2];" ::"r"(dst),
      "l"(reinterpret_cast<uint64_t>(map)), "r"(bar), "r"(c0), "r"(c1), "r"(c2), "r"(c3), "r"(c4)
      : "memory");
}

__device__ __forceinline__ void tma_load_4d(uint32_t dst, const CUtensorMap* map, uint32_t bar, int c0, int c1,
                                            int c2, int c3) {
  asm volatile(
      "cp.async.bulk.tensor.4d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4, %5, %6}], "
      "[%2];" ::"r"(dst),
      "l"(reinterpret_cast<uint64_t>(map)), "r"(bar), "r"(c0), "r"(c1), "r"(c2), "r"(c3)
      : "memory");
}

// Shared-memory matrix descriptor of a K-major tile of rows of `span` bytes (32, 64 or
// 128) in the swizzle of that width (the layout TMA writes): start address, bytes
// between 8-row groups, leading offset unused (1 by convention), the descriptor version
// of tcgen05 (1), layout code 6, 4 or 2.
__device__ __forceinline__ uint64_t desc_swizzled(uint32_t saddr, uint32_t span, uint32_t group) {
  uint64_t d = 0;
  d |= (uint64_t)((saddr >> 4) & 0x3FFFu);
  d |= (uint64_t)1u << 16;
  d |= (uint64_t)((group >> 4) & 0x3FFFu) << 32;
  d |= (uint64_t)1u << 46;
  d |= (uint64_t)(span == 32u ? 6u : (span == 64u ? 4u : 2u)) << 61;
  return d;
}

// Instruction descriptor of kind::f16: FP32 accumulator, BF16 A and B, both
// K-major, N = n, M = 128.
__device__ __forceinline__ uint32_t idesc_bf16(int n) {
  return (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(n >> 3) << 17) | ((uint32_t)(kM >> 4) << 24);
}

// D += A B by the lane where `on` (one of the warp), the descriptors given as their words.
// Predicated, not branched on: a warp whose control flow and values are uniform keeps the
// operands in uniform registers, where the instruction wants them; from a branch that one
// lane takes each operand is moved there first (nine MMAs 800 cycles, this way 600).
__device__ __forceinline__ void umma_bf16(uint32_t on, uint32_t tmem_d, uint32_t a_hi, uint32_t a_lo, uint32_t b_hi,
                                          uint32_t b_lo, uint32_t idesc) {
  asm volatile(
      "{\n .reg .b64 a, b;\n .reg .pred p;\n setp.ne.b32 p, %6, 0;\n mov.b64 a, {%2, %1};\n mov.b64 b, {%4, %3};\n"
      " @p tcgen05.mma.cta_group::1.kind::f16 [%0], a, b, %5, 1;\n}\n" ::"r"(tmem_d),
      "r"(a_hi), "r"(a_lo), "r"(b_hi), "r"(b_lo), "r"(idesc), "r"(on));
}

__device__ __forceinline__ void umma_commit(uint32_t on, uint32_t bar) {
  asm volatile(
      "{\n .reg .pred p;\n setp.ne.b32 p, %1, 0;\n"
      " @p tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];\n}\n" ::"r"(bar),
      "r"(on)
      : "memory");
}

__device__ __forceinline__ void tmem_zero16(uint32_t taddr) {
  asm volatile("tcgen05.st.sync.aligned.32x32b.x16.b32 [%0], {%1, %1, %1, %1, %1, %1, %1, %1, %1, %1, %1, %1, %1, %1, %1, %1};" ::"r"(
                   taddr),
               "r"(0u)
               : "memory");
}

__device__ __forceinline__ void tmem_ld16(uint32_t taddr, uint32_t* r) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, "
      "%15}, [%16];"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
        "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
      : "r"(taddr));
}  // valid after tcgen05.wait::ld

// SPAN: bytes of a row of an input plane, 32, 64 or 128 (16, 32 or 64 channels).  FULL:
// 3x3x3, else 1x1x1.
struct TcParams {
  int Cin, Cout, D, H, W, relu;
  int ct, bz, cols;      // output channels, planes of a column, columns (consecutive in z) of a tile
  int nbx, nby, nbz;     // tiles along x, y, z
  int tiles;             // nbx nby nbz N
  int a_stages;          // input planes in the ring (<= kMaxAStages; at least one load's of a tile)
  int b_buffers;         // weight buffers: 2, or 1 for one slice (loaded once)
  int t_buffers;         // sets of accumulators: 1 or 2
  int wide;              // the outputs start on 32-byte boundaries: whole-sector stores
  uint32_t b_bytes;      // bytes of one (slice) weight buffer: taps x ct x 32
  uint32_t ncols;        // TMEM columns allocated (a power of two >= 32 and >= t_buffers cols bz ct)
  const float* bias;     // [C_out] or null
  __nv_bfloat16* out;    // [voxels][C_out]
  float* out_f32;        // [voxels][C_out] or null
};

// One spatial tile: 8 x 16 voxels by cols columns of bz planes (fewer at the volume's
// end: whole columns, then one of `rem` planes).
struct TileAt {
  int n, x0, y0, z0, depth, whole, rem;
  __device__ __forceinline__ TileAt(const TcParams& p, int t) {
    x0 = t % p.nbx * 8;
    t /= p.nbx;
    y0 = t % p.nby * 16;
    t /= p.nby;
    z0 = t % p.nbz * p.bz * p.cols;
    n = t / p.nbz;
    depth = min(p.bz * p.cols, p.D - z0);
    whole = depth / p.bz;
    rem = depth - whole * p.bz;
  }
  // output planes of column c; columns that read an input plane q of theirs; input planes
  __device__ __forceinline__ int planes(const TcParams& p, int c) const { return c < whole ? p.bz : (c == whole ? rem : 0); }
  __device__ __forceinline__ int readers(int q, int halo) const { return whole + (rem > 0 && q < rem + 2 * halo ? 1 : 0); }
  __device__ __forceinline__ int inputs(const TcParams& p, int halo) const {
    return whole * (p.bz + 2 * halo) + (rem > 0 ? rem + 2 * halo : 0);
  }
  __device__ __forceinline__ int most(const TcParams& p, int halo) const { return (whole > 0 ? p.bz : rem) + 2 * halo; }
};

// Warps 0 and 1: loads; 2, 3 and 8, 9: MMAs of columns 0, 1 and 2, 3; 4-7: epilogue.
constexpr int kMaxCols = 4;
constexpr int kBatch = 2;  // steps of the epilogue read at once
constexpr int conv_threads(int cols) { return cols > 2 ? 320 : 256; }

template <uint32_t SPAN, bool FULL>
__global__ void __launch_bounds__(320, 2) k_conv3d_tc(const __grid_constant__ CUtensorMap tin,
                                                      const __grid_constant__ CUtensorMap tw, TcParams p) {
  extern __shared__ uint8_t smem_raw[];
  __shared__ __align__(16) float bias_sh[256];
  __shared__ __align__(8) uint64_t bars[2 * kMaxAStages + 8 + kMaxCols];
  __shared__ uint32_t tmem_slot;
  uint8_t* base = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  // [input plane stages | weight buffers]
  constexpr uint32_t stage = (uint32_t)stage_bytes(SPAN, FULL);
  constexpr int kHX = plane_x(FULL), kRows = plane_rows(FULL);
  const uint32_t a_base = smem_u32(base), b_base = a_base + ((p.a_stages * stage + 1023u) & ~1023u);
  const uint32_t afull0 = smem_u32(bars), aempty0 = afull0 + 8 * kMaxAStages, bfull0 = aempty0 + 8 * kMaxAStages,
                 bempty0 = bfull0 + 16, tfull0 = bempty0 + 16, tempty0 = tfull0 + 16, col0 = tempty0 + 16;
  // the warp's number from lane 0: the compiler then knows it is the same in all lanes
  const int warp = __shfl_sync(0xffffffffu, (int)threadIdx.x >> 5, 0), lane = threadIdx.x & 31;
  const int co0 = blockIdx.y * p.ct;
  constexpr int halo = FULL ? 1 : 0;  // input planes below and above a column
  constexpr int per_load = SPAN / 32;
  const int kslices = p.Cin / 16;
  const int loads = (kslices + per_load - 1) / per_load;
  const int AS = p.a_stages, BB = p.b_buffers, TB = p.t_buffers;
  const int set = p.cols * p.bz * p.ct;  // columns of one set of accumulators

  if (threadIdx.x == 32) {
    asm volatile("prefetch.tensormap [%0];" ::"l"(reinterpret_cast<uint64_t>(&tin)) : "memory");
    asm volatile("prefetch.tensormap [%0];" ::"l"(reinterpret_cast<uint64_t>(&tw)) : "memory");
  }
  if (threadIdx.x == 0) {
    for (int s = 0; s < AS; ++s) {
      mbar_init(afull0 + 8 * s, 1);
      mbar_init(aempty0 + 8 * s, 1);
    }
    for (int s = 0; s < 2; ++s) {
      mbar_init(bfull0 + 8 * s, 1);
      mbar_init(bempty0 + 8 * s, p.cols);
      mbar_init(tfull0 + 8 * s, p.cols);
      mbar_init(tempty0 + 8 * s, 4);
    }
    for (int c = 0; c < kMaxCols; ++c) mbar_init(col0 + 8 * c, 1);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == 2) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&tmem_slot)),
                 "r"(p.ncols)
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  // the loads wait for the kernel before this one, and with them all that depends on them
  if (warp < 2 || (warp >= 4 && warp < 8)) wait_for_previous();
  if (warp >= 4 && warp < 8)
    for (int c = threadIdx.x - 128; c < p.ct; c += 128) bias_sh[c] = p.bias ? p.bias[co0 + c] : 0.f;
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  const uint32_t tmem = __shfl_sync(0xffffffffu, tmem_slot, 0);

  if (warp == 0) {
    // ---- input planes, one thread: per load plane by plane, the columns in turn ----
    if (lane == 0) {
      int i = 0, s = 0;
      uint32_t ph = 1u;
      bool ok = true;
      for (int t = blockIdx.x; t < p.tiles && ok; t += gridDim.x) {
        const TileAt at(p, t);
        const int most = at.most(p, halo);
        for (int k = 0; k < loads && ok; ++k)
          for (int q = 0; q < most && ok; ++q) {
            const int n = at.readers(q, halo);
            for (int c = 0; c < n; ++c) {
              ok = mbar_wait(aempty0 + 8 * s, ph);
              if (!ok) break;
              mbar_expect_tx(afull0 + 8 * s, kRows * SPAN);
              tma_load_5d(a_base + s * stage, &tin, afull0 + 8 * s, k * per_load * 16, at.x0 - halo, at.y0 - halo,
                          at.z0 + c * p.bz - halo + q, at.n);
              ++i;
              if (++s == AS) {
                s = 0;
                ph ^= 1u;
              }
            }
          }
      }
      if (!ok) {
        atomicExch(&g_tc_err, 1);
        // the copies in flight land before the CTA's shared memory goes away
        for (int j = i > AS ? i - AS : 0; j < i; ++j) mbar_wait(afull0 + 8 * (j % AS), (uint32_t)(j / AS) & 1u);
      }
    }
    __syncwarp();
  } else if (warp == 1) {
    // ---- weights, one thread: every slice of every tile; a lone slice once ----
    if (lane == 0) {
      const int mine = (p.tiles - (int)blockIdx.x + (int)gridDim.x - 1) / (int)gridDim.x;
      const int total = kslices == 1 ? 1 : mine * kslices;
      const uint32_t row = (uint32_t)p.ct * 32u;  // one tap
      int i = 0;
      for (; i < total; ++i) {
        const int s = i % BB, ks = i % kslices;
        if (!mbar_wait(bempty0 + 8 * s, ((uint32_t)(i / BB) & 1u) ^ 1u)) break;
        const uint32_t sb = b_base + s * p.b_bytes;
        mbar_expect_tx(bfull0 + 8 * s, p.b_bytes);
        if (FULL) {
          for (int dy = 0; dy < 3; ++dy) tma_load_4d(sb + dy * 9 * row, &tw, bfull0 + 8 * s, ks * 16, co0, 0, dy * 3);
        } else {
          tma_load_4d(sb, &tw, bfull0 + 8 * s, ks * 16, co0, 0, 0);
        }
      }
      if (i < total) {
        atomicExch(&g_tc_err, 1);
        for (int j = i > BB ? i - BB : 0; j < i; ++j) mbar_wait(bfull0 + 8 * (j % BB), (uint32_t)(j / BB) & 1u);
      }
    }
    __syncwarp();
  } else if (warp < 4 || warp >= 8) {
    // ---- MMAs of one column, one warp, issued by its lane 0.  Block h of the column's
    // accumulators is its output plane planes - 1 - h.  The warp's own instructions count (a
    // plane's 9 MMAs take the tensor pipe 350 to 500 cycles, their issue 600), hence a warp
    // per column; stage numbers and phases run along instead of being divided out, and of a
    // descriptor only the low word is added to (its bits 0-13 are the address in 16 bytes). ----
    const int c = warp < 4 ? warp - 2 : warp - 6;
    if (c < p.cols) {
      const uint32_t leader = lane == 0 ? 1u : 0u;
      constexpr uint32_t kVox = SPAN >> 4, kRow = kHX * kVox;
      // consecutive planes of one accumulator are in order anyway; those of accumulators
      // apart need no order (one slice: each gets one MMA)
      const bool ordered = p.bz == 1 || (!FULL && kslices == 1);
      const int per = 256 / p.ct;                       // planes one MMA covers at most
      const uint32_t tap = (uint32_t)(p.ct * 2);        // one tap's rows of weights
      const uint32_t cols1 = (uint32_t)(p.ct >> 3) << 17;  // instruction descriptor: one plane's columns
      const uint32_t idesc0 = idesc_bf16(0);
      const uint64_t a_desc = desc_swizzled(a_base, SPAN, kHX * SPAN), b_desc = desc_swizzled(b_base, 32u, 256u);
      const uint32_t a_hi = (uint32_t)(a_desc >> 32), b_hi = (uint32_t)(b_desc >> 32);
      const uint32_t a_lo0 = (uint32_t)a_desc, b_lo0 = (uint32_t)b_desc;
      const uint32_t col = col0 + 8 * c;
      uint32_t turn = 1u;  // phase of the column's barrier that was armed last
      bool moved = false;
      int first = 0, tc = 0, sbuf = 0, tb = 0;
      uint32_t first_ph = 0u, b_ph = 0u, t_ph = 0u;
      bool ok = true;
      for (int t = blockIdx.x; t < p.tiles && ok; t += gridDim.x, ++tc) {
        const TileAt at(p, t);
        const int nz = at.planes(p, c), reads = nz > 0 ? nz + 2 * halo : 0, inputs = at.inputs(p, halo);
        ok = warp_wait(tempty0 + 8 * tb, t_ph);  // this set is zeroed
        const uint32_t acc = tmem + (uint32_t)(tb * set + c * p.bz * p.ct);
        for (int left = kslices; left > 0 && ok; left -= per_load) {
          const int slices = min(left, per_load);
          for (int sl = 0; sl < slices && ok; ++sl) {
            if (kslices > 1 || tc == 0) ok = warp_wait(bfull0 + 8 * sbuf, b_ph);
            const uint32_t b_lo = b_lo0 + (uint32_t)sbuf * (p.b_bytes >> 4);
            int s = first + c;
            uint32_t ph = first_ph;
            if (s >= AS) {
              s -= AS;
              ph ^= 1u;
            }
            for (int q = 0; q < reads && ok; ++q) {
              if (sl == 0) ok = warp_wait(afull0 + 8 * s, ph);
              // the column's previous plane (one outstanding at most: a parity tells no more)
              if (moved && !ordered) ok = ok && warp_wait(col, turn);
              if (!ok) break;
              asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
              // output planes hi, hi - 1, ..., lo through dz = q - hi, ... (1x1x1: plane q),
              // at most `per` planes an MMA
              const int hi = min(q, nz - 1), lo = FULL ? max(q - 2, 0) : q;
              const uint32_t a_lo = a_lo0 + (uint32_t)s * (stage >> 4) + 2u * (uint32_t)sl;
              uint32_t dst = acc + (uint32_t)((nz - 1 - hi) * p.ct);
              uint32_t bd = b_lo + (FULL ? (uint32_t)(q - hi) * tap : 0u);
              for (int n = hi - lo + 1; n > 0; n -= per) {
                const int m = min(per, n);
                const uint32_t idesc = idesc0 + (uint32_t)m * cols1;
                if (FULL) {
                  uint32_t bk = bd;
#pragma unroll
                  for (int k = 0; k < 9; ++k, bk += 3 * tap)
                    umma_bf16(leader, dst, a_hi, a_lo + (k / 3) * kRow + (k % 3) * kVox, b_hi, bk, idesc);
                } else {
                  umma_bf16(leader, dst, a_hi, a_lo, b_hi, bd, idesc);
                }
                dst += (uint32_t)(m * p.ct);
                bd += (uint32_t)m * tap;
              }
              if (!ordered) umma_commit(leader, col);
              if (sl == slices - 1) umma_commit(leader, aempty0 + 8 * s);
              moved = true;
              turn ^= 1u;
              s += at.readers(q, halo);
              if (s >= AS) {
                s -= AS;
                ph ^= 1u;
              }
            }
            if (kslices > 1) {
              umma_commit(leader, bempty0 + 8 * sbuf);
              if (++sbuf == BB) {
                sbuf = 0;
                b_ph ^= 1u;
              }
            }
          }
          first += inputs;
          if (first >= AS) {
            first -= AS;
            first_ph ^= 1u;
          }
        }
        umma_commit(leader, tfull0 + 8 * tb);  // arrives once every MMA this thread issued has completed
        if (++tb == TB) {
          tb = 0;
          t_ph ^= 1u;
        }
      }
      if (!ok && lane == 0) atomicExch(&g_tc_err, 1);
    }
    __syncwarp();
  } else {
    // ---- epilogue: TMEM lane = voxel row of a plane (x = row % 8, y = row / 8) ----
    const uint32_t mine = tmem + ((uint32_t)((warp - 4) * 32) << 16);
    auto release = [&](int tb) {  // the set is zeros again
      asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
      asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
      __syncwarp();
      if (lane == 0)
        asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(tempty0 + 8 * tb) : "memory");
      __syncwarp();
    };
    for (int tb = 0; tb < TB; ++tb) {
      for (int c = 0; c < set; c += 16) tmem_zero16(mine + (uint32_t)(tb * set + c));
      release(tb);
    }
    const int r0 = (warp - 4) * 32 + lane, chunks = p.ct / 16;
    const int64_t plane = (int64_t)p.H * p.W * p.Cout;
    int tc = 0;
    for (int t = blockIdx.x; t < p.tiles; t += gridDim.x, ++tc) {
      const TileAt at(p, t);
      const int tb = tc % TB;
      if (!warp_wait(tfull0 + 8 * tb, (uint32_t)(tc / TB) & 1u)) {
        if (lane == 0) atomicExch(&g_tc_err, 1);
        break;
      }
      asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
      const int x = at.x0 + (r0 & 7), y = at.y0 + (r0 >> 3);
      const bool inside = x < p.W && y < p.H;
      const int64_t at0 = ((((int64_t)at.n * p.D + at.z0) * p.H + y) * p.W + x) * p.Cout + co0;
      const bool again = t + (int)gridDim.x * TB < p.tiles;  // the set is used again
      // kBatch steps of one output plane and 16 channels at a time: their accumulators are
      // read together (a read takes hundreds of cycles while the tensor pipe is busy), and
      // cleared before anything is stored, the tile's last ones released
      int left = at.depth * chunks, pz = 0, ch = 0, c = 0, cz = 0;
      while (left > 0) {
        uint32_t r[kBatch][16];
        uint32_t from[kBatch];
        int to[kBatch], ch16[kBatch];
        const int m = min(left, kBatch);
        left -= m;
#pragma unroll
        for (int j = 0; j < kBatch; ++j) {
          if (j < m) {
            const int nz = c < at.whole ? p.bz : at.rem;
            from[j] = mine + (uint32_t)(tb * set + (c * p.bz + nz - 1 - cz) * p.ct + ch * 16);
            to[j] = pz;
            ch16[j] = ch * 16;
            tmem_ld16(from[j], r[j]);
            if (++ch == chunks) {
              ch = 0;
              ++pz;
              if (++cz == nz) {
                cz = 0;
                ++c;
              }
            }
          }
        }
        asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
        for (int j = 0; j < kBatch; ++j)
#pragma unroll
          for (int i = 0; i < 16; ++i) asm volatile("" : "+r"(r[j][i]));  // the values are there from here on
        if (again) {
#pragma unroll
          for (int j = 0; j < kBatch; ++j)
            if (j < m) tmem_zero16(from[j]);
          if (left == 0) release(tb);
        }
        if (inside) {
#pragma unroll
          for (int j = 0; j < kBatch; ++j) {
            if (j >= m) break;
            uint32_t* cur = r[j];
            const int64_t o = at0 + to[j] * plane + ch16[j];
            float v[16];
#pragma unroll
            for (int i = 0; i < 4; ++i) {
              const float4 bv = *reinterpret_cast<const float4*>(bias_sh + ch16[j] + 4 * i);
              v[4 * i] = __uint_as_float(cur[4 * i]) + bv.x;
              v[4 * i + 1] = __uint_as_float(cur[4 * i + 1]) + bv.y;
              v[4 * i + 2] = __uint_as_float(cur[4 * i + 2]) + bv.z;
              v[4 * i + 3] = __uint_as_float(cur[4 * i + 3]) + bv.w;
            }
            if (p.relu) {
#pragma unroll
              for (int i = 0; i < 16; ++i) v[i] = fmaxf(v[i], 0.f);
            }
            uint32_t packed[8];
#pragma unroll
            for (int i = 0; i < 8; ++i) {
              const __nv_bfloat162 h = __floats2bfloat162_rn(v[2 * i], v[2 * i + 1]);
              packed[i] = *reinterpret_cast<const uint32_t*>(&h);
            }
            __nv_bfloat16* dst = p.out + o;
            if (p.wide) {
              store32(dst, packed);
            } else {
              reinterpret_cast<uint4*>(dst)[0] = make_uint4(packed[0], packed[1], packed[2], packed[3]);
              reinterpret_cast<uint4*>(dst)[1] = make_uint4(packed[4], packed[5], packed[6], packed[7]);
            }
            if (p.out_f32) {
              float* df = p.out_f32 + o;
              if (p.wide) {
                store32(df, reinterpret_cast<const uint32_t*>(v));
                store32(df + 8, reinterpret_cast<const uint32_t*>(v + 8));
              } else {
#pragma unroll
                for (int i = 0; i < 4; ++i)
                  reinterpret_cast<float4*>(df)[i] = make_float4(v[4 * i], v[4 * i + 1], v[4 * i + 2], v[4 * i + 3]);
              }
            }
          }
        }
        __syncwarp();  // tcgen05.ld is warp-collective: every lane, converged
      }
    }
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  if (warp == 2) {
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(p.ncols) : "memory");
  }
}

PFN_cuTensorMapEncodeTiled_v12000 encode_fn() {
  static PFN_cuTensorMapEncodeTiled_v12000 fn = nullptr;
  static std::once_flag once;
  std::call_once(once, [] {
    void* ptr = nullptr;
    cudaDriverEntryPointQueryResult q;
    if (cudaGetDriverEntryPointByVersion("cuTensorMapEncodeTiled", &ptr, 12000, cudaEnableDefault, &q) ==
            cudaSuccess &&
        q == cudaDriverEntryPointSuccess)
      fn = reinterpret_cast<PFN_cuTensorMapEncodeTiled_v12000>(ptr);
  });
  return fn;
}

// Shared memory of an SM, what a CTA reserves and has as static arrays, and the most a
// CTA may ask for on top of these.
constexpr int kSmemSm = 233472, kSmemFixed = 1024 + 2048, kSmemDyn = 232448 - 2048;

// Tile of a convolution (see TcParams) and the shared memory that goes with it.
struct Plan {
  int ct, bz, cols, span, tb, tmem, per_sm, a_stages, b_buffers, smem;
};

// Modelled cycles of an MMA of n columns on an SM's tensor pipe (in a kernel of nothing
// but MMAs 36 + n / 5).
double mma_cost(int n) { return std::max(n / 2.0, 40.2 + 0.145 * n); }

// Whether a tile fits, with per_sm CTAs on an SM: tb sets of accumulators within 512
// TMEM columns, and within an equal share of shared memory (which is also requested, so
// that no more CTAs come) the planes of one load and the weight buffers.
bool conv_fit(int cin, int taps, int ct, int bz, int cols, int span, int tb, int per_sm, Plan& pl) {
  int tmem = 32;
  while (tmem < tb * cols * bz * ct) tmem *= 2;
  if (per_sm * tmem > 512) return false;
  const int smem = std::min(kSmemSm / per_sm - kSmemFixed, kSmemDyn);
  const int slices = cin / 16, bufs = slices > 1 ? 2 : 1, weights = bufs * taps * ct * 32;
  const int planes = cols * (bz + (taps == 27 ? 2 : 0)), loads = (slices * 32 + span - 1) / span;
  const int room = (smem - 2 * 1024 - weights) / stage_bytes(span, taps == 27);  // both regions start 1024-aligned
  const int stages = std::min({room, kMaxAStages, 2 * planes * loads});
  if (stages < planes) return false;
  pl = Plan{ct, bz, cols, span, tb, tmem, per_sm, stages, bufs, smem};
  return true;
}

// Modelled cycles of the whole convolution.  A column's planes take their MMAs on the
// tensor pipe or, if that is longer, their issue (kIssue an MMA), and waits: kTurn for the
// plane before where one has to be waited for, kLoad for a plane's load.  The columns that
// share an SM overlap (a 4-norm between one's time and the pipe's).  A CTA's tile is that
// and, with one set of accumulators, its epilogue (kStep per plane and 16 channels); the
// SM's TMA rows (kRow each) and bytes (loads and stores, kBytes a cycle) bound it from
// below.  The constants are a fit to every plan of 37 layers (some 8,000 timings): the
// plans it takes are 1 % slower than the best ones in the mean, 9 % at worst.
double conv_time(int cin, int cout, int n, int d, int h, int wd, int taps, int sms, const Plan& pl) {
  constexpr double kIssue = 77.7, kTurn = 132.0, kLoad = 123.0, kLaunch = 11700.0, kStep = 258.0, kRow = 1.1,
                   kBytes = 27.0;
  const int slices = cin / 16, planes = pl.bz + (taps == 27 ? 2 : 0), per = 256 / pl.ct, k = taps == 27 ? 9 : 1;
  const int loads = (slices * 32 + pl.span - 1) / pl.span;
  const int columns = (d + pl.bz - 1) / pl.bz, ny = cout / pl.ct;
  const int64_t tiles = (int64_t)n * ((wd + 7) / 8) * ((h + 15) / 16) * ((columns + pl.cols - 1) / pl.cols);
  const int64_t ctas = std::min<int64_t>(tiles, std::max(1, sms * pl.per_sm / ny)) * ny;
  const double resident = std::max(1.0, std::min((double)pl.per_sm, (double)ctas / sms));
  const double tiles_per_cta = std::ceil((double)(tiles * ny) / (double)ctas);
  double mma = 0, issue = 0;  // a column's planes, one slice
  for (int q = 0; q < planes; ++q) {
    const int first = taps == 27 ? std::max(q - 2, 0) : q, end = taps == 27 ? std::min(q, pl.bz - 1) : q;
    for (int m = end - first + 1; m > 0; m -= per) {
      mma += k * mma_cost(std::min(m, per) * pl.ct);
      issue += k * kIssue;
    }
  }
  const bool ordered = pl.bz == 1 || (taps == 1 && slices == 1);
  const double chain = std::max(mma, issue) + planes * ((ordered ? 0.0 : kTurn) + kLoad * loads / slices);
  const double pipe = resident * pl.cols * mma;
  const double turns = slices * std::sqrt(std::sqrt(chain * chain * chain * chain + pipe * pipe * pipe * pipe));
  const double weights = slices > 1 ? (double)slices * taps * pl.ct : 0.0;  // rows
  const double rows = (double)pl.cols * planes * loads * plane_rows(taps == 27) + weights;
  const double bytes = (double)pl.cols * planes * plane_rows(taps == 27) * cin * 2 + weights * 32 +
                       (double)pl.cols * pl.bz * pl.ct * 256;
  const double epi = kStep * pl.cols * pl.bz * pl.ct / 16;
  const double tile =
      std::max({pl.tb > 1 ? std::max(turns, epi) : turns + epi, resident * rows * kRow, resident * bytes / kBytes});
  return tiles_per_cta * tile + kLaunch + epi;
}

// The tile with the smallest modelled time: output channels a multiple of 16 that
// divides C_out (at most 256), every useful column height, one to four columns, one
// or two sets of accumulators, rows as wide as the channels allow or narrower (fewer bytes a plane).
bool conv_plan(int cin, int cout, int n, int d, int h, int wd, int taps, int sms, Plan& best) {
  double best_t = 0;
  bool found = false;
  for (int ct = 16; ct <= std::min(cout, 256); ct += 16) {
    if (cout % ct) continue;
    for (int bz = 1; bz <= std::min(d, 32) && bz * ct <= 512; ++bz) {
      const int columns = (d + bz - 1) / bz;
      if (bz > 1 && columns == (d + bz - 2) / (bz - 1)) continue;  // as many columns with fewer planes
      for (int cols = 1; cols <= std::min(kMaxCols, columns); ++cols)
        for (int span = 128; span >= 32; span /= 2) {  // of equal plans the one with fewer loads
          if (span > 32 && (taps == 1 || span >= cin * 4)) continue;
          for (int tb = 2; tb >= 1; --tb)
            for (int per_sm = 3; per_sm >= 1; --per_sm) {
              Plan pl;
              if (!conv_fit(cin, taps, ct, bz, cols, span, tb, per_sm, pl)) continue;
              const double t = conv_time(cin, cout, n, d, h, wd, taps, sms, pl);
              if (!found || t < best_t) {
                found = true;
                best_t = t;
                best = pl;
              }
            }
        }
    }
  }
  return found;
}

// conv_plan takes 10 to 40 us of host time, so each thread keeps the plans of the last
// shapes it asked for (a fixed table, by the shape and the SMs).
bool planned(int cin, int cout, int n, int d, int h, int wd, int taps, int sms, Plan& pl) {
  struct Entry {
    int shape[8];
    Plan plan;
  };
  static thread_local Entry table[64] = {};
  const int shape[8] = {cin, cout, n, d, h, wd, taps, sms};
  uint32_t hash = 0;
  for (int v : shape) hash = hash * 2654435761u + (uint32_t)v;
  Entry& e = table[hash >> 26];
  if (!std::equal(shape, shape + 8, e.shape)) {  // a zeroed entry has no valid shape
    Plan found;
    if (!conv_plan(cin, cout, n, d, h, wd, taps, sms, found)) return false;
    std::copy(shape, shape + 8, e.shape);
    e.plan = found;
  }
  pl = e.plan;
  return true;
}

#include "nn_wgrad_tc.cuh"

}  // namespace

extern "C" {

int hlbg_nn_conv3d_tc(const void* in, int32_t cin, const void* w, const float* bias, void* out, float* out_f32,
                      int32_t cout, int32_t n, int32_t d, int32_t h, int32_t wd, int32_t taps, int32_t relu,
                      void* stream) {
  if (!in || !w || !out || cin <= 0 || cin % 16 || cout < 16 || cout % 16 || n <= 0 || d <= 0 ||
      h <= 0 || wd <= 0 || (taps != 27 && taps != 1))
    return 1;
  // TMA: 16-byte aligned base addresses; the output is stored in 16-byte vectors
  if ((reinterpret_cast<uintptr_t>(in) | reinterpret_cast<uintptr_t>(w) | reinterpret_cast<uintptr_t>(out) |
       reinterpret_cast<uintptr_t>(out_f32)) & 15u)
    return 1;
  auto enc = encode_fn();
  if (!enc) return 3;
  const int sms = hlbg::sm_count();
  Plan pl;
  if (!planned(cin, cout, n, d, h, wd, taps, sms, pl)) return 1;
  CUtensorMap tin, tw;
  {
    const cuuint64_t dims[5] = {(cuuint64_t)cin, (cuuint64_t)wd, (cuuint64_t)h, (cuuint64_t)d, (cuuint64_t)n};
    const cuuint64_t strides[4] = {(cuuint64_t)cin * 2, (cuuint64_t)cin * 2 * wd, (cuuint64_t)cin * 2 * wd * h,
                                   (cuuint64_t)cin * 2 * wd * h * d};
    const cuuint32_t box[5] = {(cuuint32_t)(pl.span / 2), (cuuint32_t)plane_x(taps == 27), (cuuint32_t)plane_y(taps == 27), 1, 1};
    const CUtensorMapSwizzle swizzle = pl.span == 32 ? CU_TENSOR_MAP_SWIZZLE_32B
                                                     : (pl.span == 64 ? CU_TENSOR_MAP_SWIZZLE_64B : CU_TENSOR_MAP_SWIZZLE_128B);
    const cuuint32_t es[5] = {1, 1, 1, 1, 1};
    if (enc(&tin, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 5, const_cast<void*>(in), dims, strides, box, es,
            CU_TENSOR_MAP_INTERLEAVE_NONE, swizzle, CU_TENSOR_MAP_L2_PROMOTION_L2_128B,
            CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) != CUDA_SUCCESS)
      return 3;
  }
  {
    // w[(dz * 9 + dy * 3 + dx)][co][ci] seen as [dy * 3 + dx][dz][co][ci]
    const bool full = taps == 27;
    const cuuint64_t tap = (cuuint64_t)cin * 2 * cout;
    const cuuint64_t dims[4] = {(cuuint64_t)cin, (cuuint64_t)cout, full ? 3u : 1u, full ? 9u : 1u};
    const cuuint64_t strides[3] = {(cuuint64_t)cin * 2, full ? 9 * tap : tap, tap};
    const cuuint32_t box[4] = {16, (cuuint32_t)pl.ct, full ? 3u : 1u, full ? 3u : 1u};
    const cuuint32_t es[4] = {1, 1, 1, 1};
    if (enc(&tw, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 4, const_cast<void*>(w), dims, strides, box, es,
            CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_32B, CU_TENSOR_MAP_L2_PROMOTION_L2_128B,
            CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) != CUDA_SUCCESS)
      return 3;
  }
  TcParams p{};
  p.Cin = cin;
  p.Cout = cout;
  p.D = d;
  p.H = h;
  p.W = wd;
  p.relu = relu;
  p.ct = pl.ct;
  p.bz = pl.bz;
  p.cols = pl.cols;
  p.nbx = (wd + 7) / 8;
  p.nby = (h + 15) / 16;
  p.nbz = (d + pl.bz * pl.cols - 1) / (pl.bz * pl.cols);
  const int64_t tiles = (int64_t)n * p.nbz * p.nby * p.nbx;
  if (tiles > 0x3fffffff) return 1;
  p.tiles = (int)tiles;
  p.a_stages = pl.a_stages;
  p.b_buffers = pl.b_buffers;
  p.t_buffers = pl.tb;
  p.b_bytes = (uint32_t)(taps * pl.ct * 32);
  p.ncols = (uint32_t)pl.tmem;
  p.bias = bias;
  p.out = static_cast<__nv_bfloat16*>(out);
  p.out_f32 = out_f32;
  p.wide = ((reinterpret_cast<uintptr_t>(out) | reinterpret_cast<uintptr_t>(out_f32)) & 31u) == 0;
  const auto kernel = taps == 1 ? k_conv3d_tc<32, false>
                      : pl.span == 32 ? k_conv3d_tc<32, true>
                                      : (pl.span == 64 ? k_conv3d_tc<64, true> : k_conv3d_tc<128, true>);
  // the opt-in shared-memory limit is a per-device attribute of each kernel
  static std::atomic<bool> configured[64];
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return 3;
  if (!configured[dev].load()) {
    for (auto k : {k_conv3d_tc<32, false>, k_conv3d_tc<32, true>, k_conv3d_tc<64, true>, k_conv3d_tc<128, true>})
      if (cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, kSmemDyn) != cudaSuccess) return 3;
    configured[dev].store(true);
  }
  // persistent CTAs, as many as the SMs hold, over the tiles of each block of output channels
  const int ny = cout / pl.ct;
  const unsigned gx = (unsigned)std::min<int64_t>(tiles, std::max(1, sms * pl.per_sm / ny));
  launch_overlapped(kernel, dim3(gx, (unsigned)ny), conv_threads(pl.cols), pl.smem, static_cast<cudaStream_t>(stream),
                    tin, tw, p);
  return cudaGetLastError() == cudaSuccess ? 0 : 3;
}

int hlbg_nn_conv3d_wgrad_tc(const void* x, int32_t cin, const void* dy, int32_t cout, float* dw, int32_t n, int32_t d,
                            int32_t h, int32_t wd, int32_t taps, void* stream) {
  return wgrad_tc(x, cin, dy, cout, dw, n, d, h, wd, taps, static_cast<cudaStream_t>(stream), INFINITY);
}

// (nn_kernels.cu)
__attribute__((visibility("hidden"))) int hlbg_nn_wgrad_tc_within(const void* x, int32_t cin, const void* dy, int32_t cout,
                                                                  float* dw, int32_t n, int32_t d, int32_t h, int32_t wd,
                                                                  int32_t taps, void* stream, double limit) {
  return wgrad_tc(x, cin, dy, cout, dw, n, d, h, wd, taps, static_cast<cudaStream_t>(stream), limit);
}

int hlbg_nn_tc_error(int32_t reset) {
  int e = 0;
  if (cudaMemcpyFromSymbol(&e, g_tc_err, sizeof(int)) != cudaSuccess) return -1;
  if (reset && e) {
    const int zero = 0;
    cudaMemcpyToSymbol(g_tc_err, &zero, sizeof(int));
  }
  return e;
}

}  // extern "C"
