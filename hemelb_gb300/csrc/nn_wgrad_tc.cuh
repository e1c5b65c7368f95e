// Weight gradient of the warm-start surrogate's 3x3x3 (or 1x1x1) convolution on the
// fifth-generation tensor cores (included by nn_tc.cu, whose helpers it uses):
//   dw[tap][co][ci] += sum over voxels m of dy[m, co] x[m + off(tap), ci].
//
// A GEMM whose reduction runs over the voxels: both operands have their channels
// contiguous and the voxels as K, the MN-major form of tcgen05, which takes the tiles
// as TMA loads them (rows of 16, 32 or 64 channels in the swizzle of that width).  One
// operand (A, 128 rows of the accumulator) is dy or x, the other (B, its columns) the
// other one; a tile is 8 (x) x 16 (y) voxels of one plane, K = 16 two of its rows.
// Channel counts are small, so the taps fill the MMA:
//  * A's rows beyond its channels are the same tile shifted in x: the distance between
//    row groups of the operand descriptor is one voxel.  16 channels give 8 groups, 32
//    give 4 (3 shifts each, one MMA), 33 to 64 give 2 (two MMAs); with more channels the
//    two groups are channels and the three shifts are three MMAs;
//  * B's column groups are its tile shifted in y by 0, 1, 2 rows: N = 3 x 16, 32 or 64;
//  * the plane of B, z - 1, z or z + 1, is the tap's dz: all three by one CTA (ZG = 3)
//    where the accumulators fit, else one CTA each.
// So 16 -> 16 channels take one MMA of N = 48 per dz and K step: 8.6 cycles a voxel where
// the mma.sync kernel takes 22.  A's tile has a halo in x, B's in y, and B's planes reach
// one beyond A's; TMA's zeros outside the volume are the convolution's padding, and every
// pair of voxels meets exactly once.
//
// A unit of work is a run of at most `steps` K steps for one block of A's channels, one
// of B's and one dz group, into one set of accumulators, added to dw at its end (red of
// 16 bytes).  `steps` is the run the mma.sync kernel sums on its tensor cores before its
// FP32 additions to dw, so the rounding of the sums does not grow.  CTAs are persistent:
// one thread loads, one warp issues MMAs (all of one accumulator and shape are ordered), four
// warps add the finished set to dw while the other set fills.  Waits are bounded as in
// the convolution.
// Measured at batch 4 (us; mma.sync, issued from a branch of one lane, now; the tensor
// pipe's share in cycles is half to two thirds of it, the rest the issue): 16 -> 16 at
// 96^3 272, 162, 139; 64 -> 16 887, 285, 246; 48 -> 48 at 48^3 299, 88, 84; 144 -> 48 865,
// 222, 215; 288 -> 96 at 24^3 376, 141, 122; 192 -> 192 at 12^3 101, 48, 44; 1x1x1,
// 16 -> 16 at 96^3 556, 69, 54.
#pragma once

struct WgParams {
  int Ca, Cb;            // channels of A's and of B's tensor
  int a_is_dy;           // A is dy and B is x, or the other way round
  int D, H, W;
  int nbx, nby;
  int tiles;             // 8 x 16 tiles of all planes: n nby nbx D, z fastest
  int run;               // tiles of a unit
  int runs;              // units per block
  int na, nb, nzg;       // blocks of A's channels, of B's, dz groups
  int groups;            // MMAs per K step and dz: shifts of A left (1, 2 or 3)
  int stages_a, stages_b;
  int sets;              // sets of accumulators: 1 or 2
  uint32_t ncols;
  int Cout, Cin;
  float* dw;
};

// Bytes of a tile of rows of w channels: A with its halo in x (two channel groups when
// WA = 128), B with its halo in y.
__host__ __device__ constexpr int wg_a_bytes(int wa) { return (wa == 128 ? 2 : 1) * 16 * 10 * (wa == 128 ? 64 : wa) * 2; }
__host__ __device__ constexpr int wg_b_bytes(int wb) { return 18 * 8 * wb * 2; }

// MN-major operand of rows (voxels) of `span` bytes in the swizzle of that width:
// `group` bytes between groups of span / 2 channels, `k8` bytes between groups of 8 voxels.
__device__ __forceinline__ uint64_t desc_mn(uint32_t saddr, uint32_t span, uint32_t group, uint32_t k8) {
  uint64_t d = 0;
  d |= (uint64_t)((saddr >> 4) & 0x3FFFu);
  d |= (uint64_t)((group >> 4) & 0x3FFFu) << 16;
  d |= (uint64_t)((k8 >> 4) & 0x3FFFu) << 32;
  d |= (uint64_t)1u << 46;
  d |= (uint64_t)(span == 32u ? 6u : (span == 64u ? 4u : 2u)) << 61;
  return d;
}

__device__ __forceinline__ void umma_first(uint32_t on, uint32_t tmem_d, uint32_t a_hi, uint32_t a_lo, uint32_t b_hi,
                                           uint32_t b_lo, uint32_t idesc) {
  asm volatile(
      "{\n .reg .b64 a, b;\n .reg .pred p;\n setp.ne.b32 p, %6, 0;\n mov.b64 a, {%2, %1};\n mov.b64 b, {%4, %3};\n"
      " @p tcgen05.mma.cta_group::1.kind::f16 [%0], a, b, %5, 0;\n}\n" ::"r"(tmem_d),
      "r"(a_hi), "r"(a_lo), "r"(b_hi), "r"(b_lo), "r"(idesc), "r"(on));
}

__device__ __forceinline__ void red4(float* p, float a, float b, float c, float d) {
  asm volatile("red.global.add.v4.f32 [%0], {%1, %2, %3, %4};" ::"l"(p), "f"(a), "f"(b), "f"(c), "f"(d) : "memory");
}
__device__ __forceinline__ void red1(float* p, float a) {
  asm volatile("red.global.add.f32 [%0], %1;" ::"l"(p), "f"(a) : "memory");
}

// Where a unit starts: its blocks, dz group and first tile.
struct WgUnit {
  int ba, bb, zg, first, count;
  __device__ __forceinline__ WgUnit(const WgParams& p, int u) {
    const int blocks = p.na * p.nb * p.nzg, r = u / blocks;
    int k = u - r * blocks;
    zg = k % p.nzg;
    k /= p.nzg;
    bb = k % p.nb;
    ba = k / p.nb;
    first = r * p.run;
    count = min(p.run, p.tiles - first);
  }
};

constexpr int kWgThreads = 256;  // warp 0: loads; 1: MMAs; 4-7: epilogue
constexpr int kWgMaxStages = 16;

// WA: channels of A's row group (16, 32, 64; 128: two groups of 64), WB: of B's.  ZG: dz of
// a unit (3 or 1).  FULL: 3x3x3, else 1x1x1 (ZG = 1).
template <int WA, int WB, int ZG, bool FULL>
__global__ void __launch_bounds__(kWgThreads, 2) k_wgrad_tc(const __grid_constant__ CUtensorMap ta,
                                                            const __grid_constant__ CUtensorMap tb, WgParams p) {
  extern __shared__ uint8_t smem_raw[];
  __shared__ __align__(8) uint64_t bars[4 * kWgMaxStages + 4];
  __shared__ uint32_t tmem_slot;
  uint8_t* base = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  constexpr int RA = WA == 128 ? 64 : WA;  // channels of a row
  constexpr uint32_t kSpanA = RA * 2, kSpanB = WB * 2, kABytes = wg_a_bytes(WA), kBBytes = wg_b_bytes(WB);
  constexpr int N = FULL ? 3 * WB : WB;
  // [B stages | A stages | slack: A's row groups that are no shift of use read past a tile]
  const uint32_t b_base = smem_u32(base), a_base = b_base + (((uint32_t)p.stages_b * kBBytes + 1023u) & ~1023u);
  const uint32_t afull0 = smem_u32(bars), aempty0 = afull0 + 8 * kWgMaxStages, bfull0 = aempty0 + 8 * kWgMaxStages,
                 bempty0 = bfull0 + 8 * kWgMaxStages, tfull0 = bempty0 + 8 * kWgMaxStages, tempty0 = tfull0 + 16;
  const int warp = __shfl_sync(0xffffffffu, (int)threadIdx.x >> 5, 0), lane = threadIdx.x & 31;  // uniform, also to the compiler
  const int units = p.runs * p.na * p.nb * p.nzg;
  const int set = ZG * p.groups * N;  // columns of a set of accumulators

  if (threadIdx.x == 32) {
    asm volatile("prefetch.tensormap [%0];" ::"l"(reinterpret_cast<uint64_t>(&ta)) : "memory");
    asm volatile("prefetch.tensormap [%0];" ::"l"(reinterpret_cast<uint64_t>(&tb)) : "memory");
  }
  if (threadIdx.x == 0) {
    for (int s = 0; s < p.stages_a; ++s) {
      mbar_init(afull0 + 8 * s, 1);
      mbar_init(aempty0 + 8 * s, 1);
    }
    for (int s = 0; s < p.stages_b; ++s) {
      mbar_init(bfull0 + 8 * s, 1);
      mbar_init(bempty0 + 8 * s, 1);
    }
    for (int s = 0; s < 2; ++s) {
      mbar_init(tfull0 + 8 * s, 1);
      mbar_init(tempty0 + 8 * s, 4);
    }
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == 2) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&tmem_slot)),
                 "r"(p.ncols)
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  const uint32_t tmem = __shfl_sync(0xffffffffu, tmem_slot, 0);

  if (warp == 0) wait_for_previous();  // the loads, and with them all that depends on them
  if (warp == 0) {
    // ---- loads, one thread: per tile A's plane and the planes of B that are not there ----
    if (lane == 0) {
      int sa = 0, sb = 0, na = 0, nb = 0;
      uint32_t pa = 1u, pb = 1u;
      bool ok = true;
      auto load_b = [&](const WgUnit& w, int x0, int y0, int z, int n) {
        if (!mbar_wait(bempty0 + 8 * sb, pb)) return false;
        mbar_expect_tx(bfull0 + 8 * sb, kBBytes);
        tma_load_5d(b_base + sb * kBBytes, &tb, bfull0 + 8 * sb, w.bb * WB, x0, y0 - 1, z, n);
        ++nb;
        if (++sb == p.stages_b) {
          sb = 0;
          pb ^= 1u;
        }
        return true;
      };
      for (int u = blockIdx.x; u < units && ok; u += gridDim.x) {
        const WgUnit w(p, u);
        int z = w.first % p.D, c = w.first / p.D;
        bool fresh = true;
        for (int k = 0; k < w.count && ok; ++k) {
          const int x0 = c % p.nbx * 8, y0 = c / p.nbx % p.nby * 16, n = c / p.nbx / p.nby;
          if (ZG == 1) {
            ok = load_b(w, x0, y0, FULL ? z + w.zg - 1 : z, n);
          } else {
            for (int e = fresh ? 0 : 2; e < 3 && ok; ++e) ok = load_b(w, x0, y0, z + e - 1, n);
          }
          if (!ok) break;
          ok = mbar_wait(aempty0 + 8 * sa, pa);
          if (!ok) break;
          mbar_expect_tx(afull0 + 8 * sa, kABytes);
          const uint32_t dst = a_base + sa * kABytes;
          tma_load_5d(dst, &ta, afull0 + 8 * sa, w.ba * WA, x0 - 1, y0, z, n);
          if (WA == 128) tma_load_5d(dst + kABytes / 2, &ta, afull0 + 8 * sa, w.ba * WA + 64, x0 - 1, y0, z, n);
          ++na;
          if (++sa == p.stages_a) {
            sa = 0;
            pa ^= 1u;
          }
          fresh = false;
          if (++z == p.D) {
            z = 0;
            ++c;
            fresh = true;
          }
        }
      }
      if (!ok) {
        atomicExch(&g_tc_err, 1);
        // the copies in flight land before the CTA's shared memory goes away
        for (int j = max(0, na - p.stages_a); j < na; ++j) mbar_wait(afull0 + 8 * (j % p.stages_a), (uint32_t)(j / p.stages_a) & 1u);
        for (int j = max(0, nb - p.stages_b); j < nb; ++j) mbar_wait(bfull0 + 8 * (j % p.stages_b), (uint32_t)(j / p.stages_b) & 1u);
      }
    }
    __syncwarp();
  } else if (warp == 1) {
    // ---- MMAs, one warp in uniform control flow, issued by its lane 0 ----
    {
      const uint32_t leader = lane == 0 ? 1u : 0u;
      constexpr uint32_t kPitchA = 10 * kSpanA, kPitchB = 8 * kSpanB;
      const uint64_t a_desc = desc_mn(a_base, kSpanA, WA == 128 ? kABytes / 2 : kSpanA, kPitchA);
      const uint64_t b_desc = desc_mn(b_base, kSpanB, kPitchB, kPitchB);
      const uint32_t a_hi = (uint32_t)(a_desc >> 32), b_hi = (uint32_t)(b_desc >> 32);
      const uint32_t a_lo0 = (uint32_t)a_desc, b_lo0 = (uint32_t)b_desc;
      constexpr uint32_t idesc = (1u << 4) | (1u << 7) | (1u << 10) | (1u << 15) | (1u << 16) | ((uint32_t)(N >> 3) << 17) |
                                 ((uint32_t)(kM >> 4) << 24);
      int sa = 0, sb = 0, ts = 0;  // sb: B's stage of the tile's lowest plane
      uint32_t pa = 0u, pb = 0u, pt = 1u;
      bool ok = true;
      for (int u = blockIdx.x; u < units && ok; u += gridDim.x) {
        const WgUnit w(p, u);
        ok = warp_wait(tempty0 + 8 * ts, pt);
        int z = w.first % p.D;
        bool fresh = true;
        const uint32_t acc = tmem + (uint32_t)(ts * set);
        for (int k = 0; k < w.count && ok; ++k) {
          ok = warp_wait(afull0 + 8 * sa, pa);
          const bool end = k + 1 == w.count || z + 1 == p.D;  // B's planes go on with the next tile otherwise
#pragma unroll 1
          for (int e = 0; e < ZG && ok; ++e) {
            int s = sb + e;
            uint32_t ph = pb;
            if (s >= p.stages_b) {
              s -= p.stages_b;
              ph ^= 1u;
            }
            if (ZG == 1 || fresh || e == ZG - 1) ok = warp_wait(bfull0 + 8 * s, ph);
            if (!ok) break;
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            // 1x1x1: the unshifted voxels (column 1 of A's halo, row 1 of B's)
            const uint32_t a_lo = a_lo0 + (uint32_t)sa * (kABytes >> 4) + (FULL ? 0u : (kSpanA >> 4));
            const uint32_t b_lo = b_lo0 + (uint32_t)s * (kBBytes >> 4) + (FULL ? 0u : (kPitchB >> 4));
            for (int j = 0; j < p.groups; ++j) {
              const uint32_t dst = acc + (uint32_t)((e * p.groups + j) * N);
              const uint32_t aj = a_lo + (uint32_t)(WA == 64 ? 2 * j : j) * (kSpanA >> 4);
              if (k == 0)
                umma_first(leader, dst, a_hi, aj, b_hi, b_lo, idesc);
              else
                umma_bf16(leader, dst, a_hi, aj, b_hi, b_lo, idesc);
#pragma unroll
              for (int t = 1; t < 8; ++t)
                umma_bf16(leader, dst, a_hi, aj + (uint32_t)t * (2 * kPitchA >> 4), b_hi, b_lo + (uint32_t)t * (2 * kPitchB >> 4), idesc);
            }
          }
          if (!ok) break;
          umma_commit(leader, aempty0 + 8 * sa);
          if (++sa == p.stages_a) {
            sa = 0;
            pa ^= 1u;
          }
          const int free_b = ZG == 1 ? 1 : (end ? ZG : 1);
          for (int f = 0; f < free_b; ++f) {
            umma_commit(leader, bempty0 + 8 * sb);
            if (++sb == p.stages_b) {
              sb = 0;
              pb ^= 1u;
            }
          }
          fresh = end;
          if (++z == p.D) z = 0;
        }
        umma_commit(leader, tfull0 + 8 * ts);
        if (++ts == p.sets) {
          ts = 0;
          pt ^= 1u;
        }
      }
      if (!ok && lane == 0) atomicExch(&g_tc_err, 1);
    }
    __syncwarp();
  } else if (warp >= 4) {
    // ---- epilogue: add the set to dw.  Row: shift or channel group of A, and channel. ----
    const int row = (warp - 4) * 32 + lane;
    int ts = 0;
    uint32_t pt = 0u;
    for (int u = blockIdx.x; u < units; u += gridDim.x) {
      const WgUnit w(p, u);
      if (!warp_wait(tfull0 + 8 * ts, pt)) {
        if (lane == 0) atomicExch(&g_tc_err, 1);
        break;
      }
      asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
      const uint32_t mine = tmem + ((uint32_t)((warp - 4) * 32) << 16) + (uint32_t)(ts * set);
      const int ca = w.ba * WA + (WA == 128 ? row : row % RA);
      for (int q = 0; q < ZG * p.groups * (N / 16); ++q) {
        const int g = q / (N / 16), col = (q - g * (N / 16)) * 16;
        const int e = g / p.groups, j = g - e * p.groups;
        uint32_t r[16];
        tmem_ld16(mine + (uint32_t)(g * N + col), r);
        asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
        for (int i = 0; i < 16; ++i) asm volatile("" : "+r"(r[i]));
        // shifts 0, 1, 2 in x (of A), y and z (of B) and the tap they make
        const int sx = FULL ? (WA == 128 ? j : (WA == 64 ? 2 * j : 0) + row / RA) : (WA == 128 ? 1 : 1 + row / RA);
        const int sy = FULL ? col / WB : 1, sz = FULL ? (ZG == 3 ? e : w.zg) : 1;
        const int cb = w.bb * WB + (FULL ? col % WB : col);
        const bool use = ca < p.Ca && cb < p.Cb && (FULL ? sx < 3 : sx == 1);
        if (use) {
          const int tap = !FULL ? 0 : (p.a_is_dy ? (sz * 3 + sy) * 3 + 2 - sx : ((2 - sz) * 3 + 2 - sy) * 3 + sx);
          if (p.a_is_dy) {
            float* d = p.dw + ((int64_t)tap * p.Cout + ca) * p.Cin + cb;
#pragma unroll
            for (int i = 0; i < 16; i += 4)
              red4(d + i, __uint_as_float(r[i]), __uint_as_float(r[i + 1]), __uint_as_float(r[i + 2]),
                   __uint_as_float(r[i + 3]));
          } else {
            float* d = p.dw + ((int64_t)tap * p.Cout + cb) * p.Cin + ca;
#pragma unroll
            for (int i = 0; i < 16; ++i) red1(d + (int64_t)i * p.Cin, __uint_as_float(r[i]));
          }
        }
        __syncwarp();  // tcgen05.ld is warp-collective: every lane, converged
      }
      asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
      __syncwarp();
      if (lane == 0)
        asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(tempty0 + 8 * ts) : "memory");
      __syncwarp();
      if (++ts == p.sets) {
        ts = 0;
        pt ^= 1u;
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

// Tile of a weight gradient: which operand is A, the widths of the row groups, dz per
// unit, CTAs per SM, stages and sets.
struct WgPlan {
  int a_is_dy, wa, wb, zg, groups, sets, tmem, per_sm, stages_a, stages_b, smem;
};

constexpr int kWgSmemFixed = 1024 + 1024;  // reserved, static
constexpr int kWgSlack = 1024 + 1024;      // alignment of A's region; reads past A's last tile

// The plan with the fewest tensor cycles per K step (then the most loads in flight).
bool wg_plan(int cin, int cout, int taps, WgPlan& best) {
  double best_t = 0;
  bool found = false;
  for (int a_is_dy = 0; a_is_dy < 2; ++a_is_dy) {
    const int ca = a_is_dy ? cout : cin, cb = a_is_dy ? cin : cout;
    const int wa = ca <= 16 ? 16 : (ca <= 32 ? 32 : (ca <= 64 ? 64 : 128));
    const int groups = taps == 1 ? 1 : (wa <= 32 ? 1 : (wa == 64 ? 2 : 3));
    for (int wb = 16; wb <= 64; wb *= 2) {
      const int n = taps == 27 ? 3 * wb : wb;
      for (int zg = taps == 27 ? 3 : 1; zg >= 1; zg -= 2)
        for (int sets = 2; sets >= 1; --sets)
          for (int per_sm = 2; per_sm >= 1; --per_sm) {
            int tmem = 32;
            while (tmem < sets * zg * groups * n) tmem *= 2;
            if (tmem * per_sm > 512) continue;
            const int smem = std::min(kSmemSm / per_sm - kWgSmemFixed, kSmemDyn);
            const int room = smem - 1024 - kWgSlack;
            // as many tiles of A as fit beside theirs of B (ZG = 3: two planes more)
            int st = std::min(8, (room - (zg - 1) * wg_b_bytes(wb)) / (wg_a_bytes(wa) + wg_b_bytes(wb)));
            if (st < 2) continue;
            const int blocks = ((ca + wa - 1) / wa) * ((cb + wb - 1) / wb);
            // A K step of all dz and blocks: its MMAs or its TMA rows (one a cycle), and
            // some of the rows beside the MMAs.  One CTA an SM leaves the pipe idle between
            // units (less with two sets).  Factors from measured plans: 96^3 16 -> 16 (us)
            // 156 two CTAs, all dz, one set; 195 two CTAs, one dz; 197 one CTA, two sets;
            // 48^3 48 -> 48 89 two CTAs, 126 one with two sets of narrower blocks.
            const double mma = (taps == 27 ? 3.0 : 1.0) * groups * mma_cost(n);
            const double rows = ((wa == 128 ? 2 : 1) * 160.0 + 144.0) * (taps == 27 ? 3.0 / zg : 1.0) / 8.0;
            const double t = blocks * (std::max(mma, rows) + 0.5 * rows) *
                             (per_sm == 2 ? 1.0 : (sets == 2 ? 1.13 : 1.25)) * (st < 3 ? 1.05 : 1.0);
            if (!found || t < best_t) {
              found = true;
              best_t = t;
              best = WgPlan{a_is_dy, wa, wb, zg, groups, sets, tmem, per_sm, st, st + zg - 1, smem};
            }
          }
    }
  }
  return found;
}

template <int WA, int WB>
auto wg_kernel(int zg, int taps) {
  return taps == 1 ? k_wgrad_tc<WA, WB, 1, false> : (zg == 3 ? k_wgrad_tc<WA, WB, 3, true> : k_wgrad_tc<WA, WB, 1, true>);
}
template <int WA>
auto wg_kernel(int wb, int zg, int taps) {
  return wb == 16 ? wg_kernel<WA, 16>(zg, taps) : (wb == 32 ? wg_kernel<WA, 32>(zg, taps) : wg_kernel<WA, 64>(zg, taps));
}

// Modelled microseconds of a 3x3x3 gradient.  A CTA's units follow each other: a unit's
// MMAs (issued one every 0.0394 us, or the SM's pipe shared by its CTAs) and its epilogue
// (0.145 us a chunk of 16 columns), the two side by side where there are two sets.  The
// additions to dw bound it from below where runs are short, by their number (those of dy's
// rows, 16 bytes at a stride, cost twice those of x's) and by the runs that meet at an
// address; a volume a few voxels wide or high is mostly padding of the 8 x 16 tiles, so
// that its runs are many for what they add.  A 4-norm of the three over the launch's 2.77.
// A fit to 742 shapes, 10 % in the mean; so is wgrad_mma_time's.  Of the two kernels the
// faster one is chosen, or one within 5 %, for all but 25 of 754 other shapes (42 % at worst).
double wgrad_tc_time(const WgPlan& pl, const WgParams& p, int64_t units, int64_t ctas, int sms) {
  const double per_cta = (double)((units + ctas - 1) / ctas);
  const double resident = std::min((double)pl.per_sm, std::max(1.0, (double)units / sms));
  const int n = 3 * pl.wb, sums = pl.zg * pl.groups;
  const double mma = p.run * sums * 8.0 * std::max(0.0394, 0.00072 * mma_cost(n) * resident);
  const double epi = 0.145 * (sums * n / 16);
  const double chain = pl.sets == 2 && per_cta > 1 ? per_cta * std::max(mma, epi) + std::min(mma, epi)
                                                   : per_cta * (mma + epi);
  const double adds = p.runs * 27e-6 * p.Cin * p.Cout * (pl.a_is_dy ? 1.77 : 0.83), meet = 0.030 * p.runs;
  return 2.77 + std::sqrt(std::sqrt(chain * chain * chain * chain + adds * adds * adds * adds + meet * meet * meet * meet));
}

// `limit`: modelled time (us) above which the shape is not taken (3x3x3).
int wgrad_tc(const void* x, int cin, const void* dy, int cout, float* dw, int n, int d, int h, int wd, int taps,
             cudaStream_t st, double limit) {
  if (!x || !dy || !dw || cin <= 0 || cin % 16 || cout <= 0 || cout % 16 || n <= 0 || d <= 0 || h <= 0 || wd <= 0 ||
      (taps != 27 && taps != 1))
    return 1;
  if ((reinterpret_cast<uintptr_t>(x) | reinterpret_cast<uintptr_t>(dy) | reinterpret_cast<uintptr_t>(dw)) & 15u) return 1;
  auto enc = encode_fn();
  if (!enc) return 3;
  const int sms = hlbg::sm_count();
  WgPlan pl;
  if (!wg_plan(cin, cout, taps, pl)) return 1;
  WgParams p{};
  p.a_is_dy = pl.a_is_dy;
  p.Ca = pl.a_is_dy ? cout : cin;
  p.Cb = pl.a_is_dy ? cin : cout;
  p.D = d;
  p.H = h;
  p.W = wd;
  p.nbx = (wd + 7) / 8;
  p.nby = (h + 15) / 16;
  const int64_t tiles = (int64_t)n * p.nby * p.nbx * d;
  if (tiles > 0x3fffffff) return 1;
  p.tiles = (int)tiles;
  p.na = (p.Ca + pl.wa - 1) / pl.wa;
  p.nb = (p.Cb + pl.wb - 1) / pl.wb;
  p.nzg = taps == 27 ? 3 / pl.zg : 1;
  p.groups = pl.groups;
  p.stages_a = pl.stages_a;
  p.stages_b = pl.stages_b;
  p.sets = pl.sets;
  p.ncols = (uint32_t)pl.tmem;
  p.Cout = cout;
  p.Cin = cin;
  p.dw = dw;
  // Tiles of a unit: no more K steps than the mma.sync kernel sums on its tensor cores (8
  // per brick of 4 x 4 x 8 voxels; 1x1x1: 256), an eighth fewer where these are many;
  // shared out evenly over whole waves of CTAs.  The tensor cores' sums lose about 2^-26
  // of themselves a step (16 -> 16 at 96^3, error against 64 bits: 184 steps 2.4e-6, 136
  // steps 1.6e-6, mma.sync's 184 2.2e-6), so the run decides the accuracy.
  const int64_t blocks = (int64_t)p.na * p.nb * p.nzg, ctas = (int64_t)sms * pl.per_sm;
  const int64_t bricks = (int64_t)n * ((d + 3) / 4) * ((h + 3) / 4) * ((wd + 7) / 8);
  const int64_t shares = (int64_t)(cout / 16) * (cin / (cin % 32 == 0 ? 32 : 16));
  const int64_t theirs = taps == 27 ? (bricks * shares + 8 * sms - 1) / (8 * sms) : 32;
  const int64_t most = theirs >= 16 ? theirs - theirs / 8 : std::max<int64_t>(1, theirs);
  const int64_t waves = std::max<int64_t>(1, (tiles * blocks + most * ctas - 1) / (most * ctas));
  int64_t run = (tiles * blocks + waves * ctas - 1) / (waves * ctas);
  run = std::min(std::max<int64_t>(run, 1), most);
  p.run = (int)run;
  p.runs = (int)((tiles + run - 1) / run);
  const int64_t units = p.runs * blocks;
  if (units > 0x7fffffff) return 1;
  if (taps == 27 && wgrad_tc_time(pl, p, units, std::min(units, ctas), sms) > limit) return 1;
  auto map = [&](CUtensorMap& m, const void* ptr, int c, int w, int bx, int by) {
    const cuuint64_t dims[5] = {(cuuint64_t)c, (cuuint64_t)wd, (cuuint64_t)h, (cuuint64_t)d, (cuuint64_t)n};
    const cuuint64_t strides[4] = {(cuuint64_t)c * 2, (cuuint64_t)c * 2 * wd, (cuuint64_t)c * 2 * wd * h,
                                   (cuuint64_t)c * 2 * wd * h * d};
    const cuuint32_t box[5] = {(cuuint32_t)w, (cuuint32_t)bx, (cuuint32_t)by, 1, 1};
    const cuuint32_t es[5] = {1, 1, 1, 1, 1};
    return enc(&m, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 5, const_cast<void*>(ptr), dims, strides, box, es,
               CU_TENSOR_MAP_INTERLEAVE_NONE,
               w == 16 ? CU_TENSOR_MAP_SWIZZLE_32B : (w == 32 ? CU_TENSOR_MAP_SWIZZLE_64B : CU_TENSOR_MAP_SWIZZLE_128B),
               CU_TENSOR_MAP_L2_PROMOTION_L2_128B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
  };
  CUtensorMap ta, tb;
  if (!map(ta, pl.a_is_dy ? dy : x, p.Ca, std::min(pl.wa, 64), 10, 16) ||
      !map(tb, pl.a_is_dy ? x : dy, p.Cb, pl.wb, 8, 18))
    return 3;
  const auto kernel = pl.wa == 16   ? wg_kernel<16>(pl.wb, pl.zg, taps)
                      : pl.wa == 32 ? wg_kernel<32>(pl.wb, pl.zg, taps)
                      : pl.wa == 64 ? wg_kernel<64>(pl.wb, pl.zg, taps)
                                    : wg_kernel<128>(pl.wb, pl.zg, taps);
  // a per-device attribute of the kernel, always the same value (several threads may be here)
  if (cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kSmemDyn) != cudaSuccess) return 3;
  launch_overlapped(kernel, (unsigned)std::min<int64_t>(units, ctas), kWgThreads, pl.smem, st, ta, tb, p);
  return cudaGetLastError() == cudaSuccess ? 0 : 3;
}
