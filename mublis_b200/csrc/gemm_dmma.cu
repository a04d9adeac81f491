// gemm_dmma.cu -- plain FP64 GEMM on the FP64 tensor pipe: the device form
// of the reference's five-loop driver (frame/l3/l3_driver.c:126-239) plus
// its micro-kernel (include/mublis_instantiate.h:37-52) for double.
//
// B200 runs FP64 at the same peak on the tensor pipe (mma.sync .f64) as on
// the FMA pipe (37 TF/s).  What the tensor path saves is operand traffic: a
// warp's m16n8k4 MMA takes its 16x4 and 4x8 operands from registers the
// warp loaded once, where an FMA-pipe kernel streams every operand through
// shared memory per thread.  That traffic is what holds the FMA-pipe DGEMM
// well below peak.
//
// Persistent CTAs (one per SM) walk the 128 x 128 output tiles.  Warp 8
// produces: for every k-block of 16 it fills one stage (16 KB per operand) of a
// 4-stage shared-memory ring, completing on the stage's mbarrier.  Warps 0-7
// consume, each a 64 x 32 warp tile (4 x 4 m16n8k4 accumulators, 64 doubles a
// thread), then release the stage to the producer.  Every wait is bounded
// (tc_common.cuh); the producer waits for its own copies before it exits.
//
// An operand comes in one of three layouts, each read with 16-byte fragment
// loads that meet no bank conflict.  All share one k order: step ks of a
// k-block takes k = 8 (ks / 2) + 2 t + ks % 2 in lane t.
//   * packed (PACK_FRAG64, 1-D bulk copies): fragment order, every warp load
//     512 contiguous bytes;
//   * m / n contiguous, read in place: eight 16 (m) x 16 (k) TMA boxes with
//     128-byte swizzle.  MMA rows g and g + 8 are tile rows 2 g and 2 g + 1, so
//     one load brings both, and the XOR by k % 8 = 2 t + ks % 2 spreads the
//     lanes over all banks;
//   * k contiguous, read in place: one 128 x 16 TMA box with 128-byte swizzle.
//     One load brings the k of two steps; MMA row g is tile row bitrev(g), so
//     that the quarter-warp's two rows differ in the swizzle's top bit.
// Whole calls, before (8-byte fragment loads with 2- to 4-way conflicts, 168
// registers for all warps) -> now, in us: DGEMM 4096^3 NN 4105 -> 4090, NT 4027
// -> 3984 (34.5 TF/s, 93% of the pipe); 2048 x 1024 x 2048 TT 329 -> 315; DTRMM
// 2000^2 417 -> 385; DSYRK n = 1024, k = 8192 (split) 377 -> 328.
//
// Domain handling is the SIMT kernel's: ji skips tiles outside the written
// triangle and masks partial tiles, jp/pi clip each tile's k-range, an empty
// k-range writes beta * C, and beta == 0 never reads C.
#include <type_traits>

#include "kernels.cuh"
#include "tc_common.cuh"

namespace {

constexpr int BM = B200_DMMA_TILE, BN = B200_DMMA_TILE, BK = B200_DMMA_BK, STAGES = 4;
constexpr int CONSUMERS = 8;  // 2 (m) x 4 (n) warps of 64 x 32
// Two warpgroups of consumers and one that holds the producer warp.  Launched
// at 168 registers a thread (384 threads), the producer's warpgroup drops to 56
// and the consumers rise to 216: 128 for the sums, the rest for fragments and
// the epilogue, which spilled at 168.
constexpr int THREADS = (CONSUMERS + 4) * 32;
constexpr int PRODUCER_REGS = 56, CONSUMER_REGS = 216;
constexpr int TILE_BYTES = BM * BK * 8;  // 16 KB per operand per k-block
constexpr int STAGE_BYTES = 2 * TILE_BYTES;
constexpr int SMEM = STAGES * STAGE_BYTES + 128 + 1024;  // + alignment slack for swizzled tiles
constexpr int QUAD_DOUBLES = 8 * 32 * 2;  // one k-quad of a 128-row strip
constexpr int BOX_BYTES = 16 * 16 * 8;     // one 16 x 16 box of an m / n contiguous tile

__device__ __forceinline__ void dmma(double (&c)[4], double a0, double a1, double b0) {
  asm volatile(
      "mma.sync.aligned.m16n8k4.row.col.f64.f64.f64.f64 {%0,%1,%2,%3}, {%4,%5}, {%6}, "
      "{%0,%1,%2,%3};\n"
      : "+d"(c[0]), "+d"(c[1]), "+d"(c[2]), "+d"(c[3])
      : "d"(a0), "d"(a1), "d"(b0));
}

// Tile idx -> (tm, tn): from the host's tile list when the domain
// restricts the output or the k-ranges (only the tiles that write, heaviest
// first, so the strided assignment to persistent CTAs stays balanced), else
// rasterised in groups of 8 along M so that CTAs running together share B
// strips in L2.
__device__ __forceinline__ void tile_coords(const DmmaGemmArgs &p, int idx, int &tm, int &tn) {
  if (p.listed) {
    const int t = p.tiles[idx];
    tm = t >> 8;
    tn = t & 255;
    return;
  }
  if (p.tile_list) {
    const int2 t = p.tile_list[idx];
    tm = t.x;
    tn = t.y;
    return;
  }
  constexpr int G = 8;
  const int group = idx / (G * p.tiles_n);
  const int first_m = group * G;
  const int gsize = min(p.tiles_m - first_m, G);
  const int in_group = idx % (G * p.tiles_n);
  tm = first_m + in_group % gsize;
  tn = in_group / gsize;
}

// false for a tile wholly outside the written triangle (l3_driver.c:145-147,
// 165-171); else the tile's k-blocks [kt0, kt1) clipped to the product's
// support (:130,148-150,163,171).
__device__ __forceinline__ bool tile_krange(const DmmaGemmArgs &p, int tm, int tn, int &kt0,
                                            int &kt1) {
  const long m0 = (long)tm * BM, n0 = (long)tn * BN;
  if (p.ji == MUBLIS_L3_LOWER && n0 >= m0 + BM) return false;
  if (p.ji == MUBLIS_L3_UPPER && n0 + BN <= m0) return false;
  long kb = 0, ke = p.k;
  if (p.jp == MUBLIS_L3_LOWER) kb = max(kb, n0);       // j <= p
  if (p.jp == MUBLIS_L3_UPPER) ke = min(ke, n0 + BN);  // j >= p
  if (p.pi == MUBLIS_L3_LOWER) ke = min(ke, m0 + BM);  // p <= i
  if (p.pi == MUBLIS_L3_UPPER) kb = max(kb, m0);       // p >= i
  kt0 = (int)(kb / BK);
  kt1 = ke > kb ? (int)((ke + BK - 1) / BK) : kt0;
  return true;
}

// Chunk `chunk` of S of the k-blocks [kt0, kt1) (depends only on the
// tile's k range and S).
__device__ __forceinline__ void chunk_range(int chunk, int S, int &kt0, int &kt1) {
  const int per = (kt1 - kt0 + S - 1) / S;
  const int b = min(kt1, kt0 + chunk * per);
  kt1 = min(kt1, b + per);
  kt0 = b;
}

// Layouts of an operand's stage.
enum { PACKED = B200_DMMA_PACKED, MN_CONTIG = B200_DMMA_MN, K_CONTIG = B200_DMMA_K };

__device__ __forceinline__ int bitrev3(int x) { return (x & 1) << 2 | (x & 2) | (x >> 2 & 1); }

// Fragments of the 16 tile rows from 16 * blk of an operand for steps
// ks = 2 p and 2 p + 1: f[ks % 2][h] is MMA row (column) g of half h of the
// block.  `tile` is the operand's stage.
template <int LAYOUT>
__device__ __forceinline__ void load_fragments(const unsigned char *tile, int blk, int p, int g, int t,
                                               double (&f)[2][2]) {
  if constexpr (LAYOUT == K_CONTIG) {
    const int r = blk * 16 + bitrev3(g);
    const unsigned char *at = tile + r * 128 + (((4 * p + t) ^ (r & 7)) << 4);
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      const double2 v = *(const double2 *)(at + h * 8 * 128);
      f[0][h] = v.x;
      f[1][h] = v.y;
    }
  } else {
#pragma unroll
    for (int b = 0; b < 2; ++b) {
      const double2 v =
          LAYOUT == PACKED
              ? ((const double2 *)tile)[((2 * p + b) * 8 + blk) * 32 + 4 * g + t]
              : *(const double2 *)(tile + blk * BOX_BYTES + (8 * p + 2 * t + b) * 128 +
                                   ((g ^ (2 * t + b)) << 4));
      f[b][0] = v.x;
      f[b][1] = v.y;
    }
  }
}

// Tile row (column) of MMA row x + y, half h of 16-row block blk, is
// first_of(x) + offset_of(blk, h, y): x the lane's part (even where y may be
// 1), the rest known at compile time.
template <int LAYOUT>
__device__ __forceinline__ int first_of(int x) {
  return LAYOUT == K_CONTIG ? bitrev3(x) : 2 * x;
}
template <int LAYOUT>
__device__ __forceinline__ constexpr int offset_of(int blk, int h, int y) {
  return blk * 16 + (LAYOUT == K_CONTIG ? 4 * y + 8 * h : 2 * y + h);
}

// SPLIT: the split-K sums compiled in (without them the unsplit calls' main
// loop keeps its registers).
template <int LA, int LB, bool SPLIT>
__global__ void __launch_bounds__(THREADS, 1)
    dmma_gemm_kernel(const __grid_constant__ DmmaGemmArgs p) {
  extern __shared__ __align__(1024) unsigned char smem_raw[];
  // Swizzled TMA tiles need 1024-byte aligned destinations.
  unsigned char *smem = (unsigned char *)(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
  uint64_t *full = (uint64_t *)(smem + STAGES * STAGE_BYTES);
  uint64_t *empty = full + STAGES;
  volatile int *abort_flag = (volatile int *)(empty + STAGES);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  if (threadIdx.x == 0) {
    for (int s = 0; s < STAGES; ++s) {
      tc::mbar_init(&full[s], 1);
      tc::mbar_init(&empty[s], CONSUMERS);
    }
    *abort_flag = 0;
    tc::fence_barrier_init();
  }
  __syncthreads();
  const int num_tiles = p.ntiles;
  const int S = SPLIT ? p.splits : 1;
  const int num_units = num_tiles * S;

  if (warp >= CONSUMERS) {
    // ---------------- producer ----------------
    tc::setmaxnreg_dec<PRODUCER_REGS>();
    if (warp > CONSUMERS) return;
    // A stalled launch (armed by mublis_b200_test_stall_next) issues nothing:
    // the consumers' first bounded wait runs out, they raise the abort flag
    // and the error word, and the launch ends with status 4 on the host.
    if (lane != 0 || p.stall) return;
    int stage = 0, issued = 0;
    uint32_t phase = 0;
    bool ok = true;
    for (int u = blockIdx.x; u < num_units && ok; u += gridDim.x) {
      int tm, tn, kt0, kt1;
      tile_coords(p, u / S, tm, tn);
      if (!tile_krange(p, tm, tn, kt0, kt1)) continue;
      chunk_range(u % S, S, kt0, kt1);
      const int m0 = tm * BM, n0 = tn * BN;
      for (int kt = kt0; kt < kt1; ++kt) {
        if (!tc::mbar_wait(&empty[stage], phase ^ 1, abort_flag, p.err, p.wait_ns)) {
          ok = false;
          break;
        }
        tc::mbar_arrive_expect_tx(&full[stage], STAGE_BYTES);
        unsigned char *dst = smem + stage * STAGE_BYTES;
        // The k-block's pair and its k within the pair; TMA coordinates are
        // multiples of 16 doubles.
        auto load = [&](auto layout, unsigned char *to, const double *panel, const CUtensorMap *map,
                        long kpair, int t0) {
          if constexpr (decltype(layout)::value == PACKED) {
            tc::bulk_load_1d(to, panel + ((long)(t0 / BM) * p.kq + kt * 4) * QUAD_DOUBLES, TILE_BYTES,
                             &full[stage]);
          } else {
            const int q = kt * BK >= kpair, k = kt * BK - (q ? (int)kpair : 0);
            if constexpr (decltype(layout)::value == K_CONTIG) {
              tc::tma_load_2d(to, &map[q], &full[stage], k, t0);
            } else {
#pragma unroll
              for (int x = 0; x < 8; ++x)
                tc::tma_load_2d(to + x * BOX_BYTES, &map[q], &full[stage], t0 + 16 * x, k);
            }
          }
        };
        load(std::integral_constant<int, LA>(), dst, p.ap, p.ta, p.a_kpair, m0);
        load(std::integral_constant<int, LB>(), dst + TILE_BYTES, p.bp, p.tb, p.b_kpair, n0);
        ++issued;
        if (++stage == STAGES) { stage = 0; phase ^= 1; }
        // Behind the tile's first loads, its part of C.
        if (p.beta != 0 && u % S == S - 1 && kt == min(kt0 + STAGES, kt1) - 1)
          tc::prefetch_tile_l2(p.c, p.rs_c, p.cs_c, p.m, p.n, tm * BM, tn * BN, BM);
      }
    }
    const int pending = issued < STAGES ? issued : STAGES;
    for (int q = 0; q < pending; ++q) {
      if (--stage < 0) { stage = STAGES - 1; phase ^= 1; }
      if (!tc::mbar_wait_drain(&full[stage], phase)) break;
    }
    return;
  }

  // ---------------- consumers ----------------
  tc::setmaxnreg_inc<CONSUMER_REGS>();
  const int wm = warp & 1, wn = warp >> 1;
  const int g = lane >> 2, t = lane & 3;
  int stage = 0;
  uint32_t phase = 0;
  for (int u = blockIdx.x; u < num_units; u += gridDim.x) {
    int tm, tn, kt0, kt1;
    tile_coords(p, u / S, tm, tn);
    if (!tile_krange(p, tm, tn, kt0, kt1)) continue;
    chunk_range(u % S, S, kt0, kt1);
    double acc[4][4][4];
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
      for (int j = 0; j < 4; ++j)
#pragma unroll
        for (int e = 0; e < 4; ++e) acc[i][j][e] = 0.0;
    for (int kt = kt0; kt < kt1; ++kt) {
      const int wok = tc::mbar_wait(&full[stage], phase, abort_flag, p.err, p.wait_ns);
      if (!__all_sync(0xffffffffu, wok)) return;
      const unsigned char *At = smem + stage * STAGE_BYTES, *Bt = At + TILE_BYTES;
#pragma unroll
      for (int q = 0; q < BK / 8; ++q) {
        double b[2][2][2];  // [16-column block][step][half]
#pragma unroll
        for (int j = 0; j < 2; ++j) load_fragments<LB>(Bt, wn * 2 + j, q, g, t, b[j]);
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          double a[2][2];
          load_fragments<LA>(At, wm * 4 + i, q, g, t, a);
          if (q == BK / 8 - 1 && i == 3) {
            // The stage's last reads: the fence waits for them (an arrive alone
            // may pass reads still in flight) while the MMAs before them run;
            // behind the last MMAs it cost 1.2%.
            tc::fence_proxy_async();
            __syncwarp();
            if (lane == 0) tc::mbar_arrive(&empty[stage]);
          }
#pragma unroll
          for (int x = 0; x < 2; ++x)
#pragma unroll
            for (int j = 0; j < 4; ++j) dmma(acc[i][j], a[x][0], a[x][1], b[j >> 1][x][j & 1]);
        }
      }
      if (++stage == STAGES) { stage = 0; phase ^= 1; }
    }

    // Split-K: each warp stores its 64 x 32 sums of this chunk (element e of
    // lane l at e * 256 + 32 warp + l: 256 contiguous bytes per warp store);
    // the warp that finishes its sub-tile's last chunk (a per-(tile, warp)
    // counter -- no block-wide barrier, so a warp never waits on another)
    // adds the S chunks' sums in chunk order and runs the epilogue.
    if (SPLIT) {
      const int slot = threadIdx.x;  // consumer thread 0..255
      double *mine = p.partials + (size_t)u * 64 * 256;
#pragma unroll
      for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j)
#pragma unroll
          for (int e = 0; e < 4; ++e) mine[((i * 4 + j) * 4 + e) * 256 + slot] = acc[i][j][e];
      __threadfence();
      __syncwarp();
      int last = 0;
      if (lane == 0) last = atomicAdd(&p.arrivals[(u / S) * CONSUMERS + warp], 1) == S - 1;
      last = __shfl_sync(0xffffffffu, last, 0);
      if (!last) continue;
      __threadfence();
      // A 16 x 8 block's 4 sums at a time, each chunk's loads in flight
      // together (batches of 8 or 16 make the compiler spill in layouts that
      // do not otherwise: 1.3% of a split call at 16).
      const double *first = p.partials + (size_t)(u / S) * S * 64 * 256 + slot;
#pragma unroll
      for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j)
          for (int c = 0; c < S; ++c) {
            double v[4];
#pragma unroll
            for (int e = 0; e < 4; ++e)
              v[e] = __ldcg(first + ((size_t)c * 64 + (i * 4 + j) * 4 + e) * 256);
#pragma unroll
            for (int e = 0; e < 4; ++e) acc[i][j][e] = c ? acc[i][j][e] + v[e] : v[e];
          }
      if (lane == 0) p.arrivals[(u / S) * CONSUMERS + warp] = 0;
    }

    // Epilogue: accumulator e of block (i, j) is MMA row g, half e >> 1, of row
    // block i and MMA column 2 t + (e & 1) of column block j / 2, half j & 1.
    const double alpha = p.alpha, beta = p.beta;
    const bool inside = b200_whole_tile(p.m, p.n, tm, tn, BM, p.ji);
    // This lane's first element; every other is a fixed offset from it.
    // (Unsigned, and offsets compared with what is left of C: a tile's end may lie
    // past the largest int.)
    const unsigned i0 = tm * BM + wm * 64 + first_of<LA>(g), j0 = tn * BN + wn * 32 + first_of<LB>(2 * t);
    const int rows = p.m - i0, cols = p.n - j0, diag = j0 - i0;
    double *c0 = p.c + i0 * p.rs_c + j0 * p.cs_c;
    if (LA != K_CONTIG && inside && ((uintptr_t)p.c & 15) == 0 && p.rs_c == 1 && p.cs_c % 2 == 0) {
      // Rows 2 g and 2 g + 1 as 16 bytes; four loads go out before their stores.
#pragma unroll
      for (int j = 0; j < 4; ++j)
#pragma unroll
        for (int e = 0; e < 2; ++e) {
          double *col = c0 + offset_of<LB>(j >> 1, j & 1, e) * p.cs_c;
          double2 cv[4];
#pragma unroll
          for (int i = 0; i < 4; ++i)
            cv[i] = beta != 0.0 ? *(const double2 *)(col + 16 * i) : make_double2(0.0, 0.0);
#pragma unroll
          for (int i = 0; i < 4; ++i) {
            double2 v = make_double2(alpha * acc[i][j][e], alpha * acc[i][j][2 + e]);
            if (beta != 0.0) v.x = fma(beta, cv[i].x, v.x), v.y = fma(beta, cv[i].y, v.y);
            *(double2 *)(col + 16 * i) = v;
          }
        }
      continue;
    }
    // Otherwise element by element, a column's eight loads before their stores
    // (a load / store chain pays one memory round trip each: the compiler
    // cannot move a load of C above a store to C).
#pragma unroll
    for (int j = 0; j < 4; ++j)
#pragma unroll
      for (int e = 0; e < 2; ++e) {
        const int oj = offset_of<LB>(j >> 1, j & 1, e);
        if (oj >= cols) continue;
        double *col = c0 + oj * p.cs_c;
        double cv[8];
#pragma unroll
        for (int x = 0; x < 8; ++x) {
          const int o = offset_of<LA>(x >> 1, x & 1, 0);
          cv[x] = beta != 0.0 && o < rows && b200_rel(p.ji, diag + oj, o) ? col[o * p.rs_c] : 0.0;
        }
#pragma unroll
        for (int x = 0; x < 8; ++x) {
          const int o = offset_of<LA>(x >> 1, x & 1, 0);
          if (o >= rows || !b200_rel(p.ji, diag + oj, o)) continue;
          double v = alpha * acc[x >> 1][j][2 * (x & 1) + e];
          if (beta != 0.0) v = fma(beta, cv[x], v);
          col[o * p.rs_c] = v;
        }
      }
  }
}

template <int LA, int LB, bool SPLIT>
int launch_kernel(const DmmaGemmArgs &a, int grid, cudaStream_t s) {
  auto kern = dmma_gemm_kernel<LA, LB, SPLIT>;
  static B200Once once;
  B200_TRY(b200_once(once, "dmma kernel: set-up failed", [&]() -> int {
    B200_CUDA_TRY(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, SMEM));
    // An increase that the launch's registers cannot grant would wait forever.
    cudaFuncAttributes fa;
    B200_CUDA_TRY(cudaFuncGetAttributes(&fa, kern));
    if (fa.numRegs * THREADS < PRODUCER_REGS * 128 + CONSUMER_REGS * 256)
      return b200_set_error(B200_EINVAL, "dmma kernel: register split does not fit its launch");
    return B200_OK;
  }));
  B200ProfScope prof("dmma_dgemm", s);
  kern<<<grid, THREADS, SMEM, s>>>(a);
  B200_LAUNCH_CHECK();
  return B200_OK;
}

template <int LA, int LB>
int launch_layouts(const DmmaGemmArgs &a, int grid, cudaStream_t s) {
  return a.splits > 1 ? launch_kernel<LA, LB, true>(a, grid, s) : launch_kernel<LA, LB, false>(a, grid, s);
}

template <int LA>
int launch_a(const DmmaGemmArgs &a, int grid, cudaStream_t s) {
  return a.b_layout == PACKED      ? launch_layouts<LA, PACKED>(a, grid, s)
         : a.b_layout == MN_CONTIG ? launch_layouts<LA, MN_CONTIG>(a, grid, s)
                                   : launch_layouts<LA, K_CONTIG>(a, grid, s);
}

}  // namespace

int launch_dmma_gemm(const DmmaGemmArgs &a, cudaStream_t s) {
  const long tiles = (long)a.ntiles * a.splits;
  if (tiles <= 0) return B200_OK;
  if (tiles > 0x7fffffffL) return b200_set_error(B200_EINVAL, "dgemm: too many tiles");
  const int sms = b200_sm_count();
  const int grid = (int)(tiles < sms ? tiles : sms);
  return a.a_layout == PACKED      ? launch_a<PACKED>(a, grid, s)
         : a.a_layout == MN_CONTIG ? launch_a<MN_CONTIG>(a, grid, s)
                                   : launch_a<K_CONTIG>(a, grid, s);
}
