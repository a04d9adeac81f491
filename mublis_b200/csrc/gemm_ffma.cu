// gemm_ffma.cu -- plain FP32 GEMM on the FMA pipe for calls large enough for
// 128 x 128 tiles: the device form of the reference's five-loop driver
// (frame/l3/l3_driver.c:126-239) plus its micro-kernel
// (include/mublis_instantiate.h:37-52).
//
// Persistent CTAs, one per SM, walk the 128 x 128 output tiles.  Warp 8
// produces: per k-block of 16 one 2-D TMA tile (16 x 128, m / n innermost) of
// each operand into a 4-stage ring.  An operand whose unit stride runs along m
// (n) is read straight from the caller's matrix, out-of-range rows and k
// filling with zeros; any other (k-contiguous, structured, unaligned, or
// overlapping C) from an MN-major panel that pack.cu wrote.  Warps 0-7 consume
// (4 x 2 warps of 32 x 64): a thread holds 8 x 8 sums as column pairs updated
// with the packed FMA (__ffma2_rn: two correctly rounded fmaf), its fragments
// loaded one k ahead.
//
// What bounds it: the FMA pipe, 61-63 TF/s of the nominal 74.4.  Larger
// register tiles were measured and are slower (8192^3: 8 x 8 62.9, 16 x 8
// 58.8, 8 x 16 61.9 TF/s), as are pairs along k (53.4) or m (60.6) and two
// such CTAs per SM without the producer warp (62.6, and 53.6 at 4096^3).  Eight
// warps that never meet at a block barrier keep the pipe as busy as the
// sixteen of two cp.async CTAs did, so a call with about one tile per SM runs
// at full rate.  Whole calls, before (two cp.async CTAs of 256 threads per SM
// over packed panels) -> now, in us: SGEMM 4096^3 NT 2325 -> 2155 (63.8 TF/s),
// 2048^3 375 -> 333, 1500^3 NN 200 -> 151, SSYRK n = k = 2048 (136 tiles) 251 -> 175.
//
// Domain handling (ji skips and masks, jp / pi clip the k range, an empty k
// range writes beta * C, beta == 0 never reads C) and split-K are the FP64
// kernel's (gemm_dmma.cu).  Every wait is bounded (tc_common.cuh).
#include <algorithm>
#include <vector>

#include "kernels.cuh"
#include "tc_common.cuh"

namespace {

constexpr int BM = B200_FFMA_TILE, BN = B200_FFMA_TILE, BK = B200_FFMA_BK, STAGES = 4;
constexpr int WM = 4, WN = 2, CONSUMERS = WM * WN, THREADS = (CONSUMERS + 1) * 32;
constexpr int WTM = BM / WM, WTN = BN / WN, TM = WTM / 4, TN = WTN / 8;
constexpr int STAGE = (BM + BN) * BK;  // floats
constexpr int SUMS = TM * TN * CONSUMERS * 32;  // a tile's sums
constexpr int SMEM = (STAGES * STAGE + 2 * SUMS) * 4 + 2 * STAGES * 8 + 16;

__device__ __forceinline__ void tile_coords(const FfmaGemmArgs &p, int idx, int &tm, int &tn) {
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
  // Groups of 8 along M, so that CTAs running together share B tiles in L2.
  constexpr int G = 8;
  const int group = idx / (G * p.tiles_n);
  const int first_m = group * G;
  const int gsize = min(p.tiles_m - first_m, G);
  const int in_group = idx % (G * p.tiles_n);
  tm = first_m + in_group % gsize;
  tn = in_group / gsize;
}

// k-blocks [kt0, kt1) of chunk `chunk` of S of a tile, its k range clipped to
// the product's support (l3_driver.c:130,148-150,163,171).
__device__ __forceinline__ void unit_range(const FfmaGemmArgs &p, int tm, int tn, int chunk, int S,
                                           int &kt0, int &kt1) {
  const long m0 = (long)tm * BM, n0 = (long)tn * BN;
  long kb = 0, ke = p.k;
  if (p.jp == MUBLIS_L3_LOWER) kb = max(kb, n0);       // j <= p
  if (p.jp == MUBLIS_L3_UPPER) ke = min(ke, n0 + BN);  // j >= p
  if (p.pi == MUBLIS_L3_LOWER) ke = min(ke, m0 + BM);  // p <= i
  if (p.pi == MUBLIS_L3_UPPER) kb = max(kb, m0);       // p >= i
  const int t0 = (int)(kb / BK), t1 = ke > kb ? (int)((ke + BK - 1) / BK) : t0;
  const int per = (t1 - t0 + S - 1) / S;
  kt0 = min(t1, t0 + chunk * per);
  kt1 = min(t1, kt0 + per);
}

// How many k-blocks of a tile are added in a row.  (Formed anew at each use: held
// through the main loop it took 1% of every call.)
__device__ __forceinline__ int run_blocks(const FfmaGemmArgs &p, int tm, int tn) {
  if (p.runs == 1) return p.fold;
  int t0, t1;
  unit_range(p, tm, tn, 0, 1, t0, t1);
  return min(p.fold, (t1 - t0 + p.runs - 1) / p.runs);
}

__global__ void __launch_bounds__(THREADS, 1) ffma_gemm_kernel(const __grid_constant__ FfmaGemmArgs p) {
  extern __shared__ __align__(128) unsigned char smem_raw[];
  float *ring = (float *)smem_raw;
  float4 *folded = (float4 *)(ring + STAGES * STAGE);  // [TM * TN / 4][256 threads]
  uint64_t *full = (uint64_t *)(ring + STAGES * STAGE + 2 * SUMS);  // (behind the staged sums)
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
  const int S = p.splits, units = p.ntiles * S;
  // C's lines of 4 elements can move as 16 bytes: along m (1), along n (2).
  const bool base16 = ((uintptr_t)p.c & 15) == 0;
  const int vec = base16 && p.rs_c == 1 && p.cs_c % 4 == 0   ? 1
                  : base16 && p.cs_c == 1 && p.rs_c % 4 == 0 ? 2
                                                             : 0;

  if (warp == CONSUMERS) {
    // ---------------- producer ----------------
    if (lane != 0) return;
    int stage = 0, issued = 0;
    uint32_t phase = 0;
    bool ok = true;
    for (int u = blockIdx.x; u < units && ok; u += gridDim.x) {
      int tm, tn, kt0, kt1;
      tile_coords(p, u / S, tm, tn);
      unit_range(p, tm, tn, u % S, S, kt0, kt1);
      for (int kt = kt0; kt < kt1; ++kt) {
        if (!tc::mbar_wait(&empty[stage], phase ^ 1, abort_flag, p.err)) {
          ok = false;
          break;
        }
        tc::mbar_arrive_expect_tx(&full[stage], STAGE * 4);
        float *dst = ring + stage * STAGE;
        // The k-block's pair and its k within the pair (SYR2K read in place;
        // a packed operand holds both pairs as one).
        const int k = kt * BK, qa = k >= p.a_kpair, qb = k >= p.b_kpair;
        tc::tma_load_2d(dst, &p.ta[qa], &full[stage], tm * BM, qa ? k - p.a_kpair : k);
        tc::tma_load_2d(dst + BM * BK, &p.tb[qb], &full[stage], tn * BN, qb ? k - p.b_kpair : k);
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
  // Thread (ty, tx) of a warp holds rows 16 q + 4 ty + {0..3} and columns
  // 32 q + 4 tx + {0..3} (q = 0, 1) of its 32 x 64.
  const int wm = warp % WM, wn = warp / WM, ty = lane >> 3, tx = lane & 7;
  int stage = 0;
  uint32_t phase = 0;
  for (int u = blockIdx.x; u < units; u += gridDim.x) {
    int tm, tn, kt0, kt1;
    tile_coords(p, u / S, tm, tn);
    unit_range(p, tm, tn, u % S, S, kt0, kt1);
    float2 acc[TM][TN / 2];
#pragma unroll
    for (int i = 0; i < TM; ++i)
#pragma unroll
      for (int j = 0; j < TN / 2; ++j) acc[i][j] = make_float2(0.f, 0.f);
    for (int k0 = kt0, k1; k0 < kt1; k0 = k1) {
      k1 = k0 + min(kt1 - k0, run_blocks(p, tm, tn));
      for (int kt = k0; kt < k1; ++kt) {
        const int wok = tc::mbar_wait(&full[stage], phase, abort_flag, p.err);
        if (!__all_sync(0xffffffffu, wok)) return;
        const float *As = ring + stage * STAGE + wm * WTM + ty * 4;
        const float *Bs = ring + stage * STAGE + BM * BK + wn * WTN + tx * 4;
        float4 a[2][TM / 4], b[2][TN / 4];
        auto fragments = [&](int kk, int h) {
#pragma unroll
          for (int q = 0; q < TM / 4; ++q) a[h][q] = *(const float4 *)(As + kk * BM + q * 16);
#pragma unroll
          for (int q = 0; q < TN / 4; ++q) b[h][q] = *(const float4 *)(Bs + kk * BN + q * 32);
        };
        fragments(0, 0);
#pragma unroll
        for (int kk = 0; kk < BK; ++kk) {
          if (kk + 1 < BK) fragments(kk + 1, (kk + 1) & 1);
          const float *af = (const float *)a[kk & 1], *bf = (const float *)b[kk & 1];
#pragma unroll
          for (int i = 0; i < TM; ++i)
#pragma unroll
            for (int j = 0; j < TN / 2; ++j)
              acc[i][j] = __ffma2_rn(make_float2(af[i], af[i]), make_float2(bf[2 * j], bf[2 * j + 1]),
                                     acc[i][j]);
        }
        // The stage's shared-memory reads complete before the arrive that lets
        // the next copy overwrite it.  The fence is needed: without it the
        // arrive was seen to pass fragment loads still in flight (the products
        // that use them may be scheduled after it), and a warp multiplied the
        // next k-block's data once in some 10^6 k-blocks.  It costs nothing
        // measurable (62.7 TF/s at 4096^3 either way).
        tc::fence_proxy_async();
        __syncwarp();
        if (lane == 0) tc::mbar_arrive(&empty[stage]);
        if (++stage == STAGES) { stage = 0; phase ^= 1; }
      }
      // After each run of k-blocks the sums move to a total in shared memory (a
      // thread's own words).
      if (k1 < kt1) {
        const bool first = k0 == kt0;
#pragma unroll
        for (int i = 0; i < TM; ++i)
#pragma unroll
          for (int q = 0; q < TN / 4; ++q) {
            float4 *f = folded + (i * (TN / 4) + q) * CONSUMERS * 32 + threadIdx.x;
            float2 &x = acc[i][2 * q], &y = acc[i][2 * q + 1];
            float4 t = first ? make_float4(0.f, 0.f, 0.f, 0.f) : *f;
            *f = make_float4(t.x + x.x, t.y + x.y, t.z + y.x, t.w + y.y);
            x = y = make_float2(0.f, 0.f);
          }
      }
    }
    if (kt1 - kt0 > run_blocks(p, tm, tn)) {
#pragma unroll
      for (int i = 0; i < TM; ++i)
#pragma unroll
        for (int q = 0; q < TN / 4; ++q) {
          const float4 t = folded[(i * (TN / 4) + q) * CONSUMERS * 32 + threadIdx.x];
          float2 &x = acc[i][2 * q], &y = acc[i][2 * q + 1];
          x.x += t.x;
          x.y += t.y;
          y.x += t.z;
          y.y += t.w;
        }
    }

    // Split-K: each warp stores its sums of this chunk (element e of a thread
    // at e * 256 + thread); the warp that finishes its part's last chunk (a
    // counter per tile and warp: no warp waits on another) adds the S chunks'
    // sums in chunk order and runs the epilogue.
    if (S > 1) {
      const int slot = threadIdx.x;
      float *mine = p.partials + (size_t)u * SUMS;
#pragma unroll
      for (int i = 0; i < TM; ++i)
#pragma unroll
        for (int j = 0; j < TN / 2; ++j)
          *(float2 *)(mine + ((i * (TN / 2) + j) * CONSUMERS * 32 + slot) * 2) = acc[i][j];
      __threadfence();
      __syncwarp();
      int last = 0;
      if (lane == 0) last = atomicAdd(&p.arrivals[(u / S) * CONSUMERS + warp], 1) == S - 1;
      last = __shfl_sync(0xffffffffu, last, 0);
      if (!last) continue;
      __threadfence();
      const float *first = p.partials + (size_t)(u / S) * S * SUMS;
      // One chunk at a time, all its loads in flight together.
      for (int c = 0; c < S; ++c) {
        float2 w[TM][TN / 2];
#pragma unroll
        for (int i = 0; i < TM; ++i)
#pragma unroll
          for (int j = 0; j < TN / 2; ++j)
            w[i][j] = __ldcg((const float2 *)(first + (size_t)c * SUMS +
                                              ((i * (TN / 2) + j) * CONSUMERS * 32 + slot) * 2));
#pragma unroll
        for (int i = 0; i < TM; ++i)
#pragma unroll
          for (int j = 0; j < TN / 2; ++j) {
            acc[i][j].x = c ? acc[i][j].x + w[i][j].x : w[i][j].x;
            acc[i][j].y = c ? acc[i][j].y + w[i][j].y : w[i][j].y;
          }
      }
    }

    // Epilogue.  Tiles wholly inside C (and, under ji, inside the triangle)
    // move 16 bytes at a time along C's unit stride.
    const long m0 = (long)tm * BM + wm * WTM + ty * 4, n0 = (long)tn * BN + wn * WTN + tx * 4;
    const float alpha = p.alpha, beta = p.beta;
    const bool inside = b200_whole_tile(p.m, p.n, tm, tn, BM, p.ji);
    auto sum = [&](int i, int j) { return (j & 1) ? acc[i][j >> 1].y : acc[i][j >> 1].x; };
    if (vec && inside) {
      // Lines of four along m (rows 4 q + e of column j) or along n.
#pragma unroll
      for (int q = 0; q < 2; ++q) {
        float4 cv[8];
        float *line[8];
#pragma unroll
        for (int x = 0; x < 8; ++x) {
          line[x] = p.c + (vec == 1 ? (m0 + 16 * q) + (n0 + 32 * (x >> 2) + (x & 3)) * p.cs_c
                                    : (m0 + 16 * (x >> 2) + (x & 3)) * p.rs_c + (n0 + 32 * q));
          cv[x] = beta != 0.f ? *(const float4 *)line[x] : make_float4(0.f, 0.f, 0.f, 0.f);
        }
#pragma unroll
        for (int x = 0; x < 8; ++x) {
          float v[4];
          const float *c = (const float *)&cv[x];
#pragma unroll
          for (int e = 0; e < 4; ++e) {
            v[e] = alpha * (vec == 1 ? sum(4 * q + e, x) : sum(x, 4 * q + e));
            if (beta != 0.f) v[e] = fmaf(beta, c[e], v[e]);
          }
          *(float4 *)line[x] = make_float4(v[0], v[1], v[2], v[3]);
        }
      }
      continue;
    }
    // Otherwise (edges, diagonals, lines off 16 bytes) through the warp's own 32 x 64
    // floats of shared memory, so that its lanes run along C's smaller stride, 16
    // lines' loads before their stores.  Nothing else runs on the SM meanwhile: with
    // 4-byte accesses at the accumulators' places a tile's epilogue took about 9 us,
    // and 512 x 20000 x 512 with odd leading dimensions 311 us (260 so), 1000 x
    // 20000 x 200 310 (222), 967 x 2695 x 1123 207 (183).  alpha goes in here because
    // the products' own registers must not be tied to the float4 stores: the main loop
    // lost 1.5% to that.
    uint32_t id;  // (threadIdx.x, but not held through the main loop)
    asm volatile("mov.u32 %0, %%tid.x;" : "=r"(id));
    float *stage_c = ring + STAGES * STAGE + SUMS + (id >> 5) * (WTM * WTN);
    const int l = id & 31, row4 = l >> 3, col4 = l & 7;  // ty, tx
    const bool m_fast = labs(p.rs_c) <= labs(p.cs_c);
    if (m_fast) {  // [column][row], a column's groups of 4 rows XORed with column / 4
#pragma unroll
      for (int q = 0; q < 2; ++q)
#pragma unroll
        for (int x = 0; x < 8; ++x)
          *(float4 *)(stage_c + (32 * (x >> 2) + 4 * col4 + (x & 3)) * WTM + ((4 * q + row4) ^ col4) * 4) =
              make_float4(alpha * sum(4 * q, x), alpha * sum(4 * q + 1, x), alpha * sum(4 * q + 2, x),
                          alpha * sum(4 * q + 3, x));
    } else {  // [row][column]
#pragma unroll
      for (int i = 0; i < TM; ++i)
#pragma unroll
        for (int q = 0; q < 2; ++q)
          *(float4 *)(stage_c + (16 * (i >> 2) + 4 * row4 + (i & 3)) * WTN + 32 * q + 4 * col4) =
              make_float4(alpha * sum(i, 4 * q), alpha * sum(i, 4 * q + 1), alpha * sum(i, 4 * q + 2),
                          alpha * sum(i, 4 * q + 3));
    }
    __syncwarp();
#pragma unroll 1
    for (int h = 0; h < 4; ++h) {
      // Element y of a lane: row l, column 16 h + y, or row y + 16 (h & 1), column
      // 32 (h >> 1) + l.
      const long gi0 = (long)tm * BM + (id >> 5) % WM * WTM + (m_fast ? l : 16 * (h & 1));
      const long gj0 = (long)tn * BN + (id >> 5) / WM * WTN + (m_fast ? 16 * h : 32 * (h >> 1) + l);
      float *line = p.c + gi0 * p.rs_c + gj0 * p.cs_c;
      const long step = m_fast ? p.cs_c : p.rs_c;
      const long left = m_fast ? (gi0 < p.m ? p.n - gj0 : 0) : (gj0 < p.n ? p.m - gi0 : 0);
      // The lane's elements y that are written: those up to (from) the diagonal.
      int y0 = 0, y1 = (int)min(left, 16L);
      if (p.ji != MUBLIS_L3_ALL) {
        const long d = m_fast ? gi0 - gj0 : gj0 - gi0;
        const bool upto = (p.ji == MUBLIS_L3_LOWER) == m_fast;
        if (upto) y1 = (int)min((long)y1, d + 1);
        else y0 = (int)max(0L, min(d, 16L));
      }
      float cv[16];
#pragma unroll
      for (int y = 0; y < 16; ++y) cv[y] = beta != 0.f && y >= y0 && y < y1 ? line[y * step] : 0.f;
#pragma unroll
      for (int y = 0; y < 16; ++y) {
        float v = m_fast ? stage_c[(16 * h + y) * WTM + ((l >> 2) ^ ((4 * h + (y >> 2)) & 7)) * 4 + (l & 3)]
                         : stage_c[(y + 16 * (h & 1)) * WTN + 32 * (h >> 1) + l];
        if (beta != 0.f) v = fmaf(beta, cv[y], v);
        if (y >= y0 && y < y1) line[y * step] = v;
      }
    }
    __syncwarp();  // before the next tile's sums
  }
}

}  // namespace

int launch_ffma_gemm(FfmaGemmArgs &a, const FfmaPolicy *pol, cudaStream_t s) {
  static B200Once once;
  B200_TRY(b200_once(once, "sgemm: set-up failed", []() -> int {
    B200_CUDA_TRY(cudaFuncSetAttribute(ffma_gemm_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                       SMEM));
    return B200_OK;
  }));
  if (a.m <= 0 || a.n <= 0) return B200_OK;
  const int sms = b200_sm_count();
  a.tiles_m = (int)b200_ceil_div(a.m, BM);
  a.tiles_n = (int)b200_ceil_div(a.n, BN);
  if ((long)a.tiles_m * a.tiles_n > 0x7fffffffL / 16)
    return b200_set_error(B200_EINVAL, "gemm: too many tiles");
  a.ntiles = a.tiles_m * a.tiles_n;
  a.err = b200_device_error_word();
  const b200_tile_domain_t dom = {a.jp, a.ji, a.pi};
  // Restricted domains: the tiles that write, heaviest first; in the launch's
  // parameters when there are few, else uploaded.
  std::vector<int2> list;
  if (pol && (a.jp != MUBLIS_L3_ALL || a.ji != MUBLIS_L3_ALL || a.pi != MUBLIS_L3_ALL)) {
    b200_tile_list(a.m, a.n, a.k, BM, BN, BK, dom, &list, nullptr);
    if (list.empty()) return B200_OK;
    a.ntiles = (int)list.size();
    b200_snake(list, sms);
    a.listed = b200_list_tiles(list, a.tiles);
  }
  // Split-K from the whole call's shape (pol), so that column panels split
  // their tiles' k ranges as the whole call does.  A split unit's 64 KB of
  // sums cost about SPLIT_COST k-block times (1.3 us each).  With it the rule
  // took the fastest of S = 1, 2, 3, 4, 6, 8 or one within 3% of it on eleven
  // of twelve shapes timed, e.g. 2500 x 1000 x 4000: S = 1 634 us, 2 500, 4 451,
  // 6 447; 2048^3: 1 336, 2 364, 4 355.
  constexpr double SPLIT_COST = 4.0;
  a.splits = pol ? b200_split_for(pol->m_full, pol->n_full, a.k, BM, BN, BK, dom, sms, SPLIT_COST) : 1;
  // Sums are folded into a total where they would grow longer than the chunks into
  // which split-K cuts k for two CTAs per SM (the two that this kernel's full rate at
  // one tile per SM replaces; PAIR_COST: what a split unit cost them), and below
  // 1024 tiles every 1024 k as well.  Normwise error and us, in runs of 1024 and in
  // those chunks: 2000 x 2587 x 1300 (chunks of 336) 5.3e-7, 343; 3.3e-7, 346;
  // 4096 x 4096 x 8192 (4096) 1.6e-6, 4272; 1.1e-6, 4321.
  constexpr double PAIR_COST = 4.0;
  const long m_full = pol ? pol->m_full : a.m, n_full = pol ? pol->n_full : a.n;
  a.fold = b200_ceil_div(m_full, BM) * b200_ceil_div(n_full, BN) < 1024 ? 1024 / BK : 0x7fffffff;
  a.runs = pol ? b200_split_for(m_full, n_full, a.k, BM, BN, BK, dom, 2 * sms, PAIR_COST) : 1;
  const size_t list_bytes = list.empty() || a.listed ? 0 : sizeof(int2) * list.size();
  const size_t off_arr = b200_round_up((long)list_bytes, 256);
  const size_t arr_bytes = a.splits > 1 ? sizeof(int) * a.ntiles * CONSUMERS : 0;
  const size_t off_part = off_arr + b200_round_up((long)arr_bytes, 256);
  const size_t part_bytes = a.splits > 1 ? sizeof(float) * (size_t)a.ntiles * a.splits * SUMS : 0;
  char *ws = nullptr;
  int st = B200_OK;
  if (list_bytes || a.splits > 1) {
    B200_TRY(b200_alloc((void **)&ws, off_part + part_bytes));
    if ((list_bytes && cudaMemcpyAsync(ws, list.data(), list_bytes, cudaMemcpyHostToDevice, s) !=
                           cudaSuccess) ||
        (arr_bytes && cudaMemsetAsync(ws + off_arr, 0, arr_bytes, s) != cudaSuccess))
      st = b200_set_error(B200_ECUDA, "gemm: schedule upload failed");
    if (list_bytes) a.tile_list = (const int2 *)ws;
    a.arrivals = (int *)(ws + off_arr);
    a.partials = (float *)(ws + off_part);
  }
  if (st == B200_OK) {
    const long units = (long)a.ntiles * a.splits;
    B200ProfScope prof("ffma_sgemm", s);
    ffma_gemm_kernel<<<(unsigned)std::min<long>(units, sms), THREADS, SMEM, s>>>(a);
    if (cudaGetLastError() != cudaSuccess) st = b200_set_error(B200_ECUDA, "gemm: launch failed");
  }
  b200_free(ws);
  return st;
}

// Loads the kernel on the current device (the driver loads a kernel's code,
// and takes memory for it, at its first use).
int b200_ffma_preload() {
  cudaFuncAttributes fa;
  FfmaGemmArgs none;
  none.m = none.n = 0;
  B200_TRY(launch_ffma_gemm(none, nullptr, nullptr));  // no tiles: sets the kernel up only
  B200_CUDA_TRY(cudaFuncGetAttributes(&fa, ffma_gemm_kernel));
  return B200_OK;
}
