// gemm_direct.cu -- products too small to fill the GPU with 128 x 128 tiles,
// in one launch straight from the caller's operands.
//
// The packed path (l3.cu: two pack launches, then 128 x 128 tiles) costs a
// small call four allocations, three launches and a grid of a few CTAs.  Here
// a CTA of 128 threads computes a 64 x 64 or 32 x 32 tile of C, reads op(A)
// and op(B) itself -- op(), symmetric reflection, triangular zeros and the
// domain masks are resolved in the address of an asynchronous copy, as the
// reference's packm resolves them element by element (frame/l1m/packm.c:40-71)
// -- and a tile's k range may be cut over the 2, 4 or 8 CTAs of a cluster,
// which add their sums through distributed shared memory in rank order (the
// reference's pc loop, frame/l3/l3_driver.c:126-135, run side by side).
//
// What bounds it: latency (the call's launch and wait, 12.5 us on this host;
// one round trip for the operands, one for C) for the smallest calls,
// shared-memory and FMA issue for the larger ones: 64^3 SGEMM 40 -> 16 us a
// call, 301 x 177 x 211 DGEMM 79 -> 18, 512^3 SGEMM 86 -> 29.
//   * FP32: 8 x 4 (4 x 2) accumulators per thread as packed column pairs
//     (__ffma2_rn, each half a correctly rounded fmaf).
//   * FP64: m16n8k4 .f64 MMAs, a 32 x 32 (16 x 16) block per warp.  The
//     operand rows are padded to BM + 4 doubles, so the 16 lanes of a
//     fragment load's half-warp (4 k x 4 rows) fall on 16 different 8-byte
//     banks.
//   * Operands move in 16-byte copies where the unit stride runs along m (n)
//     and every row starts on 16 bytes, else element by element along
//     whichever stride is smaller; copies past the edge fill zeros.
//   * A group of many products (grouped.cu) runs the same tiles, one CTA each,
//     from a table of problems.
//   * The sums go through shared memory to C, so C is read and written along
//     its own unit stride.
#include <algorithm>
#include <cmath>

#include "kernels.cuh"

namespace {

template <typename T>
struct DirectOperand {
  const T *x[2];  // one per pair (SYR2K's two products are concatenated along k)
  long s_mn[2], s_k[2];  // strides along m (n) and along k
  int vec[2];            // 16-byte copies along m (n); of the transposed matrix
  int plain;             // general, unmasked: no element needs looking at
  int struc, uplo, diag, mask_rel;
};

template <typename T>
struct DirectArgs {
  DirectOperand<T> a, b;
  int npairs;
  T *c;
  long rs_c, cs_c;
  int m, n, k;  // k: of one pair
  int tiles_m;
  T alpha, beta;
  int jp, ji, pi;
  int splits;  // CTAs per cluster
};

__device__ __forceinline__ uint32_t smem_addr(const void *p) {
  return (uint32_t)__cvta_generic_to_shared(p);
}
// Asynchronous copy of BYTES, of which the first `valid` are read and the
// rest filled with zeros (valid = 0: nothing is read).
template <int BYTES>
__device__ __forceinline__ void cp_zfill(void *dst, const void *src, int valid) {
  if constexpr (BYTES == 16)
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(smem_addr(dst)), "l"(src),
                 "r"(valid)
                 : "memory");
  else
    asm volatile("cp.async.ca.shared.global [%0], [%1], %2, %3;" ::"r"(smem_addr(dst)), "l"(src),
                 "n"(BYTES), "r"(valid)
                 : "memory");
}
__device__ __forceinline__ void cp_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N>
__device__ __forceinline__ void cp_wait() {
  asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory");
}
__device__ __forceinline__ void cluster_barrier() {
  asm volatile("barrier.cluster.arrive.release.aligned;\nbarrier.cluster.wait.acquire.aligned;" ::
                   : "memory");
}
// Value at `p`'s offset in the shared memory of cluster rank `rank`.
__device__ __forceinline__ float ld_rank(const float *p, int rank) {
  uint32_t a;
  float v;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(a) : "r"(smem_addr(p)), "r"(rank));
  asm volatile("ld.shared::cluster.f32 %0, [%1];" : "=f"(v) : "r"(a) : "memory");
  return v;
}
__device__ __forceinline__ double ld_rank(const double *p, int rank) {
  uint32_t a;
  double v;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(a) : "r"(smem_addr(p)), "r"(rank));
  asm volatile("ld.shared::cluster.f64 %0, [%1];" : "=d"(v) : "r"(a) : "memory");
  return v;
}

__device__ __forceinline__ void dmma(double (&c)[4], double a0, double a1, double b0) {
  asm volatile(
      "mma.sync.aligned.m16n8k4.row.col.f64.f64.f64.f64 {%0,%1,%2,%3}, {%4,%5}, {%6}, "
      "{%0,%1,%2,%3};\n"
      : "+d"(c[0]), "+d"(c[1]), "+d"(c[2]), "+d"(c[3])
      : "d"(a0), "d"(a1), "d"(b0));
}

// Tile shapes.  TILE = 64: 128 threads.  TILE = 32: two groups of 128 threads,
// each taking half of every k-block, so that the small tile still has two
// warps per scheduler to hide one another's latency; their sums are added
// with the ranks' in the epilogue.
template <typename T, int TILE>
struct DirectCfg {
  static constexpr int GROUPS = TILE == 32 ? 2 : 1;
  static constexpr int NT = 128 * GROUPS;
  static constexpr int BK = 16 * GROUPS;
  static constexpr int STAGES = TILE == 64 && sizeof(T) == 8 ? 3 : 4;
  static constexpr int LD = TILE + 4;
  static constexpr int STAGE = 2 * BK * LD;  // elements
  static constexpr int CLD = TILE + 1;       // pitch of the staged sums
  static constexpr size_t SMEM = sizeof(T) * STAGES * STAGE;
  static_assert(GROUPS * CLD * TILE <= STAGES * STAGE, "the sums reuse the operand ring");
};

// One thread's share of a k-block of a general, unmasked operand: element
// (or 16-byte chunk) q is at src + q * q_src, goes to dst0 + q * q_dst and
// has k index kk0 + q * q_kk, so that the loop computes no addresses but
// increments.
template <typename T, int TILE>
struct PlainLoader {
  using C = DirectCfg<T, TILE>;
  static constexpr int VEC = 16 / sizeof(T);
  static constexpr int NV = C::BK * TILE / VEC / C::NT, NS = C::BK * TILE / C::NT;
  const T *src, *safe;
  long q_src, k_src;
  int dst0, q_dst, kk0, q_kk;
  int vec, valid;  // vec: bytes of each chunk; scalar: bit q set where element q is inside m (n)
  // swapped: the transposed matrix (a symmetric operand's unstored triangle).
  __device__ __forceinline__ void init(const DirectOperand<T> &o, int pair, int swapped, long mn0,
                                       int mn_len) {
    const int tid = threadIdx.x;
    const long s_mn = swapped ? o.s_k[pair] : o.s_mn[pair];
    const long s_k = swapped ? o.s_mn[pair] : o.s_k[pair];
    safe = o.x[pair];
    vec = o.vec[swapped];
    k_src = C::BK * s_k;
    int mn, q_mn;
    if (vec) {
      kk0 = tid / (TILE / VEC), mn = tid % (TILE / VEC) * VEC;
      q_kk = C::NT / (TILE / VEC), q_mn = 0;
    } else if (labs(s_mn) <= labs(s_k)) {
      kk0 = tid / TILE, mn = tid % TILE;
      q_kk = C::NT / TILE, q_mn = 0;
    } else {
      kk0 = tid % C::BK, mn = tid / C::BK;
      q_kk = 0, q_mn = C::NT / C::BK;
    }
    src = safe + (mn0 + mn) * s_mn + kk0 * s_k;
    q_src = q_mn * s_mn + q_kk * s_k;
    dst0 = kk0 * C::LD + mn;
    q_dst = q_kk * C::LD + q_mn;
    const long rest = mn_len - (mn0 + mn);
    if (vec) {
      valid = rest <= 0 ? 0 : (int)(rest < VEC ? rest : VEC) * (int)sizeof(T);
    } else {
      valid = 0;
#pragma unroll
      for (int q = 0; q < NS; ++q) valid |= (q * q_mn < rest ? 1 : 0) << q;
    }
  }
  // k-block kt of the pair; k_left: its rows that exist.
  __device__ __forceinline__ void load(T *dst, int kt, int k_left) const {
    const T *s = src + kt * k_src;
    T *d = dst + dst0;
    if (vec) {
#pragma unroll
      for (int q = 0; q < NV; ++q, s += q_src, d += q_dst) {
        const int bytes = kk0 + q * q_kk < k_left ? valid : 0;
        cp_zfill<16>(d, bytes ? s : safe, bytes);
      }
    } else {
#pragma unroll
      for (int q = 0; q < NS; ++q, s += q_src, d += q_dst) {
        const bool in = kk0 + q * q_kk < k_left && (valid >> q & 1);
        cp_zfill<sizeof(T)>(d, in ? s : safe, in ? (int)sizeof(T) : 0);
      }
    }
  }
};

// A k-block of a structured or masked operand, element by element: rows
// k0 .. k0 + BK - 1 into dst[kk][mn].  B_SIDE: the operand is op(B), element
// (r, c) = (k, mn); else op(A), (mn, k).
template <typename T, int TILE, bool B_SIDE>
__device__ __forceinline__ void load_general(const DirectOperand<T> &o, T *dst, long mn0, int mn_len,
                                             int k0, int k_len) {
  using C = DirectCfg<T, TILE>;
  const bool mn_fast = labs(o.s_mn[0]) <= labs(o.s_k[0]);
#pragma unroll 4
  for (int idx = threadIdx.x; idx < C::BK * TILE; idx += C::NT) {
    const int kk = mn_fast ? idx / TILE : idx % C::BK, mn = mn_fast ? idx % TILE : idx / C::BK;
    const long gm = mn0 + mn, gk = k0 + kk;
    T *d = dst + kk * C::LD + mn;
    // The logical element (r, c) of load_logical (kernels.cuh), resolved to
    // the address that holds it.
    const long r = B_SIDE ? gk : gm, c = B_SIDE ? gm : gk;
    long sr = B_SIDE ? o.s_k[0] : o.s_mn[0], sc = B_SIDE ? o.s_mn[0] : o.s_k[0];
    bool in = gk < k_len && gm < mn_len && b200_rel(o.mask_rel, c, r);
    const bool stored = o.uplo == MUBLIS_LOWER ? r >= c : (o.uplo == MUBLIS_UPPER ? r <= c : true);
    if (!stored) {
      if (o.struc == MUBLIS_STRUC_SYMMETRIC) {
        const long x = sr;
        sr = sc;
        sc = x;
      } else if (o.struc == MUBLIS_STRUC_TRIANGULAR) {
        in = false;
      }
    }
    if (in && o.struc == MUBLIS_STRUC_TRIANGULAR && r == c && o.diag != MUBLIS_PACKM_DIAG_NONUNIT) {
      *d = o.diag == MUBLIS_PACKM_DIAG_UNIT ? T(1) : T(1) / o.x[0][r * sr + c * sc];
      continue;
    }
    cp_zfill<sizeof(T)>(d, in ? o.x[0] + r * sr + c * sc : o.x[0], in ? (int)sizeof(T) : 0);
  }
}

// How a block of a structured or masked operand can be read: as stored (0),
// as its mirror image (1), or only element by element (2: it meets the
// diagonal, or lies outside the mask or triangle).
template <typename T, int TILE, bool B_SIDE>
__device__ __forceinline__ int block_class(const DirectOperand<T> &o, long mn0, long k0) {
  constexpr int BK = DirectCfg<T, TILE>::BK;
  // Extremes of r - c over the block.
  const long lo = B_SIDE ? k0 - (mn0 + TILE - 1) : mn0 - (k0 + BK - 1);
  const long hi = B_SIDE ? k0 + BK - 1 - mn0 : mn0 + TILE - 1 - k0;
  if ((o.mask_rel == MUBLIS_L3_LOWER && lo < 0) || (o.mask_rel == MUBLIS_L3_UPPER && hi > 0)) return 2;
  if (o.struc == MUBLIS_STRUC_GENERAL || (o.uplo != MUBLIS_LOWER && o.uplo != MUBLIS_UPPER))
    return o.struc == MUBLIS_STRUC_TRIANGULAR ? 2 : 0;
  if (o.uplo == MUBLIS_LOWER ? lo > 0 : hi < 0) return 0;
  return o.struc == MUBLIS_STRUC_SYMMETRIC && (o.uplo == MUBLIS_LOWER ? hi < 0 : lo > 0) ? 1 : 2;
}

// PLAIN: both operands general and unmasked.  (SYR2K's two pairs are plain;
// each pair takes whole k-blocks, the last one filled up with zeros.)
// FOLD: after every RUN k-blocks (128 products of a thread) the sums move to totals,
// in registers: at most three CTAs to an SM instead of four.
template <typename T, int TILE, bool PLAIN, bool FOLD>
__device__ __forceinline__ void direct_tile(const DirectArgs<T> &p, const int tile, const int rank,
                                            const int S) {
  using C = DirectCfg<T, TILE>;
  constexpr bool F64 = sizeof(T) == 8;
  constexpr int BM = TILE, BN = TILE, BK = C::BK, LD = C::LD, CLD = C::CLD, STAGES = C::STAGES;
  constexpr int NT = C::NT, GROUPS = C::GROUPS, GK = BK / GROUPS, RUN = B200_DIRECT_RUN / GK;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  T *ring = reinterpret_cast<T *>(smem_raw);

  const long m0 = (long)(tile % p.tiles_m) * BM, n0 = (long)(tile / p.tiles_m) * BN;
  // Outside the written triangle (l3_driver.c:145-147,165-171): the whole
  // cluster leaves.
  if (p.ji == MUBLIS_L3_LOWER && n0 >= m0 + BM) return;
  if (p.ji == MUBLIS_L3_UPPER && n0 + BN <= m0) return;
  long kb = 0, ke = p.k;  // (two pairs: no jp, pi)
  if (p.jp == MUBLIS_L3_LOWER) kb = max(kb, n0);       // j <= p
  if (p.jp == MUBLIS_L3_UPPER) ke = min(ke, n0 + BN);  // j >= p
  if (p.pi == MUBLIS_L3_LOWER) ke = min(ke, m0 + BM);  // p <= i
  if (p.pi == MUBLIS_L3_UPPER) kb = max(kb, m0);       // p >= i
  const int pair_blocks = (p.k + BK - 1) / BK;
  const int kt0 = (int)(kb / BK);
  const int kt1 = p.npairs == 2 ? 2 * pair_blocks : (ke > kb ? (int)((ke + BK - 1) / BK) : kt0);
  const int per = (kt1 - kt0 + S - 1) / S;
  const int begin = min(kt1, kt0 + rank * per), end = min(kt1, begin + per);

  const int tid = threadIdx.x & 127, group = threadIdx.x >> 7;
  const int warp = tid >> 5, lane = tid & 31;
  PlainLoader<T, TILE> la, lb;
  int va = 0, vb = 0;  // what the loaders are set up for: the pair, or a block class
  la.init(p.a, 0, 0, m0, p.m);
  lb.init(p.b, 0, 0, n0, p.n);
  auto load_stage = [&](int stage, int kt) {
    T *As = ring + stage * C::STAGE, *Bs = As + BK * LD;
    if constexpr (PLAIN) {
      if (p.npairs == 2 && va == 0 && kt >= pair_blocks) {
        va = 1;
        la.init(p.a, 1, 0, m0, p.m);
        lb.init(p.b, 1, 0, n0, p.n);
      }
      const int kl = kt - (va ? pair_blocks : 0);
      la.load(As, kl, p.k - kl * BK);
      lb.load(Bs, kl, p.k - kl * BK);
    } else {
      const int ca = block_class<T, TILE, false>(p.a, m0, kt * BK);
      if (ca == 2) {
        load_general<T, TILE, false>(p.a, As, m0, p.m, kt * BK, p.k);
      } else {
        if (ca != va) la.init(p.a, 0, va = ca, m0, p.m);
        la.load(As, kt, p.k - kt * BK);
      }
      const int cb = block_class<T, TILE, true>(p.b, n0, kt * BK);
      if (cb == 2) {
        load_general<T, TILE, true>(p.b, Bs, n0, p.n, kt * BK, p.k);
      } else {
        if (cb != vb) lb.init(p.b, 0, vb = cb, n0, p.n);
        lb.load(Bs, kt, p.k - kt * BK);
      }
    }
  };
#pragma unroll
  for (int s = 0; s < STAGES - 1; ++s) {
    if (begin + s < end) load_stage(s, begin + s);
    cp_commit();
  }
  // FP32: thread (ty, tx) of 8 x 16 holds rows 4 ty + 32 u + {0..3} and
  // columns TN tx + {0..TN-1}, as column pairs.  FP64: warp (wm, wn) of 2 x 2
  // holds MI x NI blocks of 16 x 8.
  constexpr int TM = TILE / 8, TN = TILE / 16;
  constexpr int MI = TILE / 32, NI = TILE / 16;
  float2 facc[F64 ? 1 : TM][F64 ? 1 : TN / 2];
  double dacc[F64 ? MI : 1][F64 ? NI : 1][4];
  const int ty = tid >> 4, tx = tid & 15;
  const int wm = warp & 1, wn = warp >> 1, g = lane >> 2, t = lane & 3;
  if constexpr (F64) {
#pragma unroll
    for (int i = 0; i < MI; ++i)
#pragma unroll
      for (int j = 0; j < NI; ++j)
#pragma unroll
        for (int e = 0; e < 4; ++e) dacc[i][j][e] = 0.0;
  } else {
#pragma unroll
    for (int i = 0; i < TM; ++i)
#pragma unroll
      for (int j = 0; j < TN / 2; ++j) facc[i][j] = make_float2(0.f, 0.f);
  }
  // The totals, and the step that moves the sums there.
  float2 ftot[FOLD && !F64 ? TM : 1][FOLD && !F64 ? TN / 2 : 1];
  double dtot[FOLD && F64 ? MI : 1][FOLD && F64 ? NI : 1][4];
  auto fold = [&](bool first) {
    if constexpr (FOLD && F64) {
#pragma unroll
      for (int i = 0; i < MI; ++i)
#pragma unroll
        for (int j = 0; j < NI; ++j)
#pragma unroll
          for (int e = 0; e < 4; ++e) {
            dtot[i][j][e] = first ? dacc[i][j][e] : dtot[i][j][e] + dacc[i][j][e];
            dacc[i][j][e] = 0.0;
          }
    } else if constexpr (FOLD) {
#pragma unroll
      for (int i = 0; i < TM; ++i)
#pragma unroll
        for (int j = 0; j < TN / 2; ++j) {
          ftot[i][j] = first ? facc[i][j] : __fadd2_rn(ftot[i][j], facc[i][j]);
          facc[i][j] = make_float2(0.f, 0.f);
        }
    }
  };
  fold(true);

  int stage = 0, next = STAGES - 1;
  for (int kt = begin; kt < end; fold(false)) {
    const int run_end = FOLD ? min(end, kt + RUN) : end;
    for (; kt < run_end; ++kt) {
      cp_wait<STAGES - 2>();
      __syncthreads();
      if (kt + STAGES - 1 < end) load_stage(next, kt + STAGES - 1);
      cp_commit();
      const T *As = ring + stage * C::STAGE + group * GK * LD, *Bs = As + BK * LD;
      if (++stage == STAGES) stage = 0;
      if (++next == STAGES) next = 0;
      if constexpr (F64) {
#pragma unroll
        for (int ks = 0; ks < GK / 4; ++ks) {
          const double *ar = As + (4 * ks + t) * LD + wm * (BM / 2) + g;
          const double *br = Bs + (4 * ks + t) * LD + wn * (BN / 2) + g;
          double a0[MI], a1[MI], b[NI];
#pragma unroll
          for (int i = 0; i < MI; ++i) a0[i] = ar[16 * i], a1[i] = ar[16 * i + 8];
#pragma unroll
          for (int j = 0; j < NI; ++j) b[j] = br[8 * j];
#pragma unroll
          for (int i = 0; i < MI; ++i)
#pragma unroll
            for (int j = 0; j < NI; ++j) dmma(dacc[i][j], a0[i], a1[i], b[j]);
        }
      } else {
        // Fragments one k ahead of the products that use them.
        float a[2][TM], b[2][TN];
        auto fragments = [&](int kk, int h) {
#pragma unroll
          for (int u = 0; u < TM / 4; ++u) {
            const float4 v = *reinterpret_cast<const float4 *>(As + kk * LD + 32 * u + 4 * ty);
            a[h][4 * u] = v.x, a[h][4 * u + 1] = v.y, a[h][4 * u + 2] = v.z, a[h][4 * u + 3] = v.w;
          }
          if constexpr (TN == 4) {
            const float4 v = *reinterpret_cast<const float4 *>(Bs + kk * LD + 4 * tx);
            b[h][0] = v.x, b[h][1] = v.y, b[h][2] = v.z, b[h][3] = v.w;
          } else {
            const float2 v = *reinterpret_cast<const float2 *>(Bs + kk * LD + 2 * tx);
            b[h][0] = v.x, b[h][1] = v.y;
          }
        };
        fragments(0, 0);
#pragma unroll
        for (int kk = 0; kk < GK; ++kk) {
          if (kk + 1 < GK) fragments(kk + 1, (kk + 1) & 1);
          const float *af = a[kk & 1], *bf = b[kk & 1];
#pragma unroll
          for (int i = 0; i < TM; ++i)
#pragma unroll
            for (int j = 0; j < TN / 2; ++j)
              facc[i][j] = __ffma2_rn(make_float2(af[i], af[i]), make_float2(bf[2 * j], bf[2 * j + 1]),
                                      facc[i][j]);
        }
      }
    }
  }
  cp_wait<0>();
  __syncthreads();  // every reader of the ring is done

  // The sums, column-major with an odd pitch, one copy per thread group.
  T *Cs = ring + group * CLD * TILE;
  if constexpr (F64) {
#pragma unroll
    for (int i = 0; i < MI; ++i)
#pragma unroll
      for (int j = 0; j < NI; ++j)
#pragma unroll
        for (int e = 0; e < 4; ++e)
          Cs[(wn * (BN / 2) + 8 * j + 2 * t + (e & 1)) * CLD + wm * (BM / 2) + 16 * i + g +
             8 * (e >> 1)] = FOLD ? dtot[FOLD ? i : 0][FOLD ? j : 0][e] : dacc[i][j][e];
  } else {
#pragma unroll
    for (int i = 0; i < TM; ++i)
#pragma unroll
      for (int j = 0; j < TN / 2; ++j) {
        const int r = 32 * (i / 4) + 4 * ty + i % 4;
        const float2 v = FOLD ? ftot[FOLD ? i : 0][FOLD ? j : 0] : facc[i][j];
        Cs[(TN * tx + 2 * j) * CLD + r] = v.x;
        Cs[(TN * tx + 2 * j + 1) * CLD + r] = v.y;
      }
  }
  if (S > 1) cluster_barrier();
  else __syncthreads();

  // Rank r writes slice r of the tile: lines of TILE elements along C's
  // smaller stride, a thread at one place of every (NT / TILE)-th line, adding
  // the sums of the ranks and groups in order.  A batch's loads of C go out
  // before its stores (one memory round trip per batch).
  const bool m_fast = labs(p.rs_c) <= labs(p.cs_c);
  const long fast0 = m_fast ? m0 : n0, slow0 = m_fast ? n0 : m0;
  const long fast_s = m_fast ? p.rs_c : p.cs_c, slow_s = m_fast ? p.cs_c : p.rs_c;
  const int fast = threadIdx.x % TILE;
  constexpr int STEP = NT / TILE, BATCH = 8;
  if (fast0 + fast < (m_fast ? p.m : p.n)) {
    const int slice = TILE / S;
    const int last = (int)min((long)(rank + 1) * slice, (m_fast ? p.n : p.m) - slow0);
    T *crow = p.c + (fast0 + fast) * fast_s + slow0 * slow_s;
    const T *sum = ring + fast * (m_fast ? 1 : CLD);
    const int sum_s = m_fast ? CLD : 1;
    auto written = [&](int line) {  // the ji relation, j against i
      return m_fast ? b200_rel(p.ji, slow0 + line, fast0 + fast)
                    : b200_rel(p.ji, fast0 + fast, slow0 + line);
    };
    for (int l0 = rank * slice + threadIdx.x / TILE; l0 < last; l0 += STEP * BATCH) {
      T cv[BATCH];
#pragma unroll
      for (int q = 0; q < BATCH; ++q) {
        const int line = l0 + q * STEP;
        cv[q] = T(0);
        if (p.beta != T(0) && line < last && written(line)) cv[q] = crow[line * slow_s];
      }
#pragma unroll
      for (int q = 0; q < BATCH; ++q) {
        const int line = l0 + q * STEP;
        if (line >= last || !written(line)) continue;
        const T *src = sum + line * sum_s;
        T v = T(0);
        if (S == 1) {
#pragma unroll
          for (int h = 0; h < GROUPS; ++h) v += src[h * CLD * TILE];
        } else {
#pragma unroll 1
          for (int r = 0; r < S; ++r)
#pragma unroll
            for (int h = 0; h < GROUPS; ++h) v += ld_rank(src + h * CLD * TILE, r);
        }
        v = p.alpha * v;
        if (p.beta != T(0)) v = fma(p.beta, cv[q], v);
        crow[line * slow_s] = v;
      }
    }
  }
  if (S > 1) cluster_barrier();  // no CTA leaves while another reads its sums
}

template <typename T, int TILE, bool PLAIN, bool FOLD>
__global__ void __launch_bounds__(DirectCfg<T, TILE>::NT, TILE == 32 && !PLAIN && FOLD ? 2 : (TILE == 32 && !PLAIN) || FOLD ? 3 : 4)
    direct_gemm_kernel(const __grid_constant__ DirectArgs<T> p) {
  direct_tile<T, TILE, PLAIN, FOLD>(p, blockIdx.x / p.splits, blockIdx.x % p.splits, p.splits);
}

// Many independent products: CTA b computes tile b of the group, of problem
// tile_prob[b] of the table.
template <typename T, int TILE>
__global__ void __launch_bounds__(DirectCfg<T, TILE>::NT, 4)
    direct_group_kernel(const b200_group_gemm_t *__restrict__ table, const int *__restrict__ tile_prob) {
  const b200_group_gemm_t &e = table[tile_prob[blockIdx.x]];
  DirectArgs<T> p;
  p.a.x[0] = (const T *)e.a;
  p.a.s_mn[0] = e.rs_a;
  p.a.s_k[0] = e.cs_a;
  p.a.vec[0] = e.vec & 1;
  p.b.x[0] = (const T *)e.b;
  p.b.s_mn[0] = e.cs_b;
  p.b.s_k[0] = e.rs_b;
  p.b.vec[0] = e.vec >> 1;
  p.npairs = 1;
  p.c = (T *)e.c;
  p.rs_c = e.rs_c;
  p.cs_c = e.cs_c;
  p.m = e.m;
  p.n = e.n;
  p.k = e.k;
  p.tiles_m = e.tiles_m;
  p.alpha = (T)e.alpha;
  p.beta = (T)e.beta;
  p.jp = p.ji = p.pi = MUBLIS_L3_ALL;
  direct_tile<T, TILE, true, false>(p, blockIdx.x - e.tile0, 0, 1);
}

template <typename T, int TILE, bool PLAIN, bool FOLD>
int launch_tile(DirectArgs<T> &p, cudaStream_t s) {
  using C = DirectCfg<T, TILE>;
  auto kern = direct_gemm_kernel<T, TILE, PLAIN, FOLD>;
  static B200Once once;
  B200_TRY(b200_once(once, "direct gemm: set-up failed", [&]() -> int {
    B200_CUDA_TRY(
        cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)C::SMEM));
    return B200_OK;
  }));
  p.tiles_m = (int)b200_ceil_div(p.m, TILE);
  const long ctas = (long)p.tiles_m * b200_ceil_div(p.n, TILE) * p.splits;
  if (ctas > 0x7fffffffL) return b200_set_error(B200_EINVAL, "direct gemm: too many tiles");
  cudaLaunchConfig_t cfg = {};
  cudaLaunchAttribute attr[1];
  cfg.gridDim = dim3((unsigned)ctas);
  cfg.blockDim = dim3(C::NT);
  cfg.dynamicSmemBytes = C::SMEM;
  cfg.stream = s;
  if (p.splits > 1) {
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = p.splits;
    attr[0].val.clusterDim.y = 1;
    attr[0].val.clusterDim.z = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
  }
  B200ProfScope prof(sizeof(T) == 4 ? "direct_sgemm" : "direct_dgemm", s);
  B200_CUDA_TRY(cudaLaunchKernelEx(&cfg, kern, (const DirectArgs<T> &)p));
  return B200_OK;
}

template <typename T, int TILE>
int launch_tile(DirectArgs<T> &p, bool plain, bool fold, cudaStream_t s) {
  if (fold) return plain ? launch_tile<T, TILE, true, true>(p, s) : launch_tile<T, TILE, false, true>(p, s);
  return plain ? launch_tile<T, TILE, true, false>(p, s) : launch_tile<T, TILE, false, false>(p, s);
}

template <typename T>
DirectOperand<T> operand(const void *const (&x)[2], const long (&s_mn)[2], const long (&s_k)[2],
                         int npairs, const mublis_l3_operand_t &o, int mask) {
  DirectOperand<T> d;
  constexpr int VEC = 16 / sizeof(T);
  d.struc = o.struc;
  d.uplo = o.uplo;
  d.diag = o.diag;
  d.mask_rel = mask;
  d.plain = o.struc == MUBLIS_STRUC_GENERAL && mask == MUBLIS_L3_ALL;
  d.vec[0] = d.vec[1] = 1;
  for (int t = 0; t < 2; ++t) {
    const int u = t < npairs ? t : 0;
    d.x[t] = (const T *)x[u];
    d.s_mn[t] = s_mn[u];
    d.s_k[t] = s_k[u];
    // 16-byte copies: unit stride along m (n), every k row on 16 bytes.
    const bool base = ((uintptr_t)x[u] & 15) == 0;
    if (!base || s_mn[u] != 1 || s_k[u] <= 0 || s_k[u] % VEC != 0) d.vec[0] = 0;
    if (!base || s_k[u] != 1 || s_mn[u] <= 0 || s_mn[u] % VEC != 0) d.vec[1] = 0;
  }
  return d;
}

template <typename T>
int run_direct(const b200_l3_desc_t *d, const b200_direct_choice_t &ch) {
  const mublis_l3_product_t &pr = d->product;
  DirectArgs<T> p;
  p.a = operand<T>(d->a, d->rs_a, d->cs_a, d->npairs, pr.a, pr.domain.pi);
  p.b = operand<T>(d->b, d->cs_b, d->rs_b, d->npairs, pr.b, pr.domain.jp);
  p.npairs = d->npairs;
  p.c = (T *)d->c;
  p.rs_c = d->rs_c;
  p.cs_c = d->cs_c;
  p.m = d->m;
  p.n = d->n;
  p.k = d->k;
  p.alpha = (T)d->alpha;
  p.beta = (T)d->beta;
  p.jp = pr.domain.jp;
  p.ji = pr.domain.ji;
  p.pi = pr.domain.pi;
  p.splits = ch.splits;
  cudaStream_t s = b200_cur_stream();
  const bool plain = p.a.plain && p.b.plain;
  if (!plain && d->npairs != 1) return b200_set_error(B200_EINVAL, "direct gemm: structured pairs");
  return ch.tile == 64 ? launch_tile<T, 64>(p, plain, ch.fold, s) : launch_tile<T, 32>(p, plain, ch.fold, s);
}

template <typename T, int TILE>
int launch_group_tile(const b200_group_gemm_t *table, const int *tile_prob, int tiles, cudaStream_t s) {
  using C = DirectCfg<T, TILE>;
  auto kern = direct_group_kernel<T, TILE>;
  static B200Once once;
  B200_TRY(b200_once(once, "grouped gemm: set-up failed", [&]() -> int {
    cudaFuncAttributes fa;
    B200_CUDA_TRY(
        cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)C::SMEM));
    B200_CUDA_TRY(cudaFuncGetAttributes(&fa, kern));  // loads it: a capture must not
    return B200_OK;
  }));
  if (tiles <= 0) return B200_OK;
  B200ProfScope prof(sizeof(T) == 4 ? "grouped_sgemm" : "grouped_dgemm", s);
  kern<<<tiles, C::NT, C::SMEM, s>>>(table, tile_prob);
  B200_LAUNCH_CHECK();
  return B200_OK;
}

}  // namespace

int b200_group_vec(const b200_group_gemm_t &e, int elt) {
  auto vec = [elt](const void *x, long s_mn, long s_k) {
    return s_mn == 1 && s_k > 0 && s_k * elt % 16 == 0 && ((uintptr_t)x & 15) == 0;
  };
  return (vec(e.a, e.rs_a, e.cs_a) ? 1 : 0) | (vec(e.b, e.cs_b, e.rs_b) ? 2 : 0);
}

int launch_direct_group(int dtype, int tile, const b200_group_gemm_t *table, const int *tile_prob,
                        int tiles, cudaStream_t s) {
  if (dtype == B200_F64)
    return tile == 64 ? launch_group_tile<double, 64>(table, tile_prob, tiles, s)
                      : launch_group_tile<double, 32>(table, tile_prob, tiles, s);
  return tile == 64 ? launch_group_tile<float, 64>(table, tile_prob, tiles, s)
                    : launch_group_tile<float, 32>(table, tile_prob, tiles, s);
}

// Which calls run here, and how: the least of the estimates below, in us, from
// the whole call's shape and structure (a column panel of a larger call carries
// the call's m and n, so every panel runs as the whole call would; strides and
// alignment differ between a panel and its call and are left out).
//
// Direct, with n CTAs on the fullest SM and kb k-blocks per CTA:
//   start + kb * max(alone, n * shared) + (n - 1) * next
// -- alone / shared: a k-block of a CTA that has the SM to itself / of one that
// shares it; next: filling and draining one more CTA; a triangle of C leaves half
// of the CTAs without work, but evens out only where an SM gets many.  Packed:
// start, the packs by the operands' size, and the rounds of 128 x 128 tiles, k cut
// into the best number of chunks.
//
// The constants are those that choose best among packed and both tiles at S = 1, 2,
// 4, 8, all nine timed on 566 calls (GEMM, SYMM, SYRK, SYR2K, TRMM; m, n, k 16 ..
// 4096, widths to 80000, k to 100000): the choice costs 0.8% (FP64 1.2%) more than
// the best of the nine on average.  Estimating the packed path by its rate alone
// sent these the slower way (us, then -> now): STRMM 256 x 40000 325 -> 153 and
// 512 x 10000 207 -> 112, SSYMM 256 x 20000 150 -> 104, SSYRK n = 2048, k = 512
// 83 -> 60, SGEMM 512 x 512 x 8192 158 -> 109 and 1024^3 84 -> 73 (packed); 64 x 64
// x 65536 FP32 351 -> 165 and FP64 622 -> 168, DGEMM 1719 x 1427 x 1060 341 -> 214
// (direct).
b200_direct_choice_t b200_direct_choice(const b200_l3_desc_t *d) {
  struct Direct {
    double start, alone, shared, next1, next;  // next1: S = 1
  };
  struct Packed {
    double start, packs, per_mb, structured_mb, block, tile, split;
  };
  // [FP64][general, symmetric, triangular or masked][tile 64]
  static const Direct cost[2][3][2] = {{{{13.5, 0.67, 0.44, 0.75, 0.97}, {18.3, 0.79, 0.45, 2.19, 2.00}},
                                        {{15.5, 0.97, 0.59, 1.46, 1.75}, {26.7, 1.01, 0.65, 2.00, 2.54}},
                                        {{30.8, 0.75, 0.28, 2.76, 2.42}, {47.9, 0.75, 0.40, 6.01, 3.13}}},
                                       {{{14.1, 0.86, 0.41, 1.01, 1.92}, {19.1, 0.98, 0.57, 2.02, 2.30}},
                                        {{15.3, 0.90, 0.61, 0.91, 1.92}, {26.8, 1.17, 0.86, 5.21, 2.89}},
                                        {{31.9, 0.75, 0.44, 2.27, 2.04}, {47.3, 1.29, 0.50, 8.91, 2.70}}}};
  static const Packed packed_cost[2] = {{27.5, 7.2, 0.38, 0.35, 1.03, 4.3, 4.0},
                                        {27.5, 12.7, 0.57, 0.25, 1.81, 4.0, 18.2}};
  const bool f64 = d->dtype == B200_F64;
  const long m = d->policy_m > 0 ? d->policy_m : d->m, n = d->policy_n > 0 ? d->policy_n : d->n;
  const long k = (long)d->k * d->npairs, sms = b200_sm_count();
  const mublis_l3_product_t &pr = d->product;
  const mublis_l3_domain_t &dom = pr.domain;
  const bool half_c = dom.ji != MUBLIS_L3_ALL, half_k = dom.jp != MUBLIS_L3_ALL || dom.pi != MUBLIS_L3_ALL;
  const bool triangular = half_k || pr.a.struc == MUBLIS_STRUC_TRIANGULAR || pr.b.struc == MUBLIS_STRUC_TRIANGULAR;
  const int kind = triangular ? 2
                   : pr.a.struc != MUBLIS_STRUC_GENERAL || pr.b.struc != MUBLIS_STRUC_GENERAL ? 1
                                                                                             : 0;
  const Packed &q = packed_cost[f64];
  const long tm = b200_ceil_div(m, 128), tn = b200_ceil_div(n, 128);
  const double tiles = half_c ? ((double)tm * tn + std::min(tm, tn)) / 2 : (double)tm * tn;
  const long blocks = b200_ceil_div(k, 16);
  double best = 1e30;
  for (int S = 1; S == 1 || (S <= 16 && blocks / S >= 8); ++S) {
    const double kb = (double)b200_ceil_div(blocks, S), unit = q.tile + (S > 1 ? q.split : 0.0);
    const double rounds = tiles * S / sms;
    best = std::min(best, half_k ? std::max(kb * q.block + unit, 1.05 * rounds * (0.5 * kb * q.block + unit))
                                 : std::ceil(rounds) * (kb * q.block + unit));
  }
  // Operands that are certain to be packed: a structured one, or a SYR2K's four whose
  // pairs do not meet on a k-block.
  const double mb = (f64 ? 8e-6 : 4e-6) * k;
  best += q.start + q.packs * (kind ? 1 : d->npairs == 2 && d->k % 16 ? 2 : 0) + q.per_mb * mb * (m + n) +
          (kind ? q.structured_mb * mb * k : 0.0);
  // Near ties in FP64 go to one launch without workspaces: in a solve's two column
  // chains it leaves the other chain's leaves more room (DTRSM 4096 x 4096 2528 us
  // without this, 2500 with).
  if (f64) best *= 1.05;

  b200_direct_choice_t ch = {0, 1, 0};
  long run = 0;  // products that a thread adds in a row
  for (int big = 0; big < 2; ++big) {
    const Direct &c = cost[f64][kind][big];
    const long tile = big ? 64 : 32, bk = big ? 16 : 32;
    const double ctas = (double)b200_ceil_div(m, tile) * b200_ceil_div(n, tile);
    for (int S = 1; S <= 8; S *= 2) {
      const long kb = b200_ceil_div(b200_ceil_div(k, bk), S);
      if (S > 1 && kb < 2) break;
      const double mean = ctas * S / sms, per_sm = std::ceil(half_c && mean > 3 ? 0.5 * mean + 1.5 : mean);
      const double t = c.start + kb * std::max(c.alone, per_sm * c.shared) + (per_sm - 1) * (S == 1 ? c.next1 : c.next);
      if (t < best) {
        best = t;
        ch = {big ? 64 : 32, S, 0};
        run = kb * 16;  // of each k-block, 16 to a thread
      }
    }
  }
  // Sums are to be no longer than under the packed path's split-K when that ran on
  // every SM's 1 (FP64) or 2 (FP32) CTAs, and in FP32 no longer than 1024: above
  // that they are folded.  Normwise error and us of FP32 696 x 389 x 1855, k cut in
  // 12 there, in 2 here: 2.4e-7 packed; 5.5e-7 and 65.6 in one sum, 2.1e-7 and 68.5
  // folded; 1236 x 788 x 1005 2.9e-7; 5.7e-7 and 85.8, 2.1e-7 and 83.2; FP64 254 x
  // 1050 x 1370 1.3e-15; 1.4e-15 and 56.3, 1.3e-15 and 54.8.  With four or more CTAs
  // to an SM folding takes 3-9% (360 x 1411 x 2847 114 -> 126; packed 170).
  if (ch.tile && run > B200_DIRECT_RUN) {
    const int cut = b200_split_for(m, n, k, 128, 128, 16, {dom.jp, dom.ji, dom.pi}, f64 ? sms : 2 * sms,
                                   f64 ? 8.0 : 4.0);
    const long chunk = b200_ceil_div(blocks, cut) * 16;
    ch.fold = run > (f64 ? chunk : std::min(chunk, 1024L));
  }
  return ch;
}

int launch_direct_gemm(const b200_l3_desc_t *d, const b200_direct_choice_t &ch) {
  return d->dtype == B200_F64 ? run_direct<double>(d, ch) : run_direct<float>(d, ch);
}
