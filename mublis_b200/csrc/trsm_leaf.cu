// trsm_leaf.cu -- the fused GEMMTRSM kernel: solves one leaf of a left
// triangular solve (up to 512 rows, every right-hand side) in one launch,
// the diagonal blocks by substitution in shared memory and the updates
// between them on the FP64 tensor pipe.
//
// Reference: the blocked solve of frame/l3/trsm.c:139-183 calls the
// gemmtrsm{l,u} micro-kernel (include/mublis_instantiate.h:95-114,
// targets/avx2/gemmtrsm_ukr.inc:95-215), which forms B11 - A1x * Bx1 and
// solves the MR x MR diagonal block A11 (packed with its diagonal already
// inverted, packm.c:143-144) in registers.  Here a CTA owns 8 or 16 columns (FP32:
// 32) of a leaf of 512 rows and keeps that whole block of B in registers.  A
// column group (8 columns of FP64, 32 of FP32) has 8 warps, and its
// 32 row blocks of 16 go to them in turn.  For each diagonal block d of 16 rows:
//   * the warp that owns block d + 1 first applies block d's update to it and
//     solves it, X = inv(D) R with the inverse of its 16 x 16 diagonal block, and
//     publishes it in shared memory on an mbarrier, so that the other warps find
//     it when their updates are done (look-ahead);
//   * every warp then applies X_d to its own blocks below: B_rb -= A_rb,d X_d, as
//     m16n8k4 .f64 MMAs on the tensor pipe, or FP32 FMAs on 4 x 4 register tiles.
// Nothing but these mbarriers and the ring's holds the warps together: there is no
// barrier of the CTA in the loop.  What bounds it is the chain from X_d to X_{d+1}
// (an update and a solve of one block, 1100-1400 clocks of 32 dependent steps;
// folding inv(D) into the update, so that the chain is one product, measured 2-5%
// slower and cost FP32 half a digit), then the FP64 pipe (a step's MMAs take half of
// it at 16 columns).  A CTA of 32 columns whose 8 warps each updated 16 x 32
// blocks, with a barrier per step, took 78 us a leaf in FP64 and 82 us in FP32
// (its FMAs took an A operand from shared memory for every two of them); now 28 us
// (8 columns) or 37 us (16, on 16 warps), and 52 us.  DTRSM 1000 x 1000 225 -> 123
// us, 4096 x 4096 2726 -> 2501; STRSM 1001 x 1500 231 -> 184.
//
// The leaf's A is packed once per solve (trsm_leaf_pack_kernel) into one contiguous
// segment per step -- the column of 16 x 16 blocks below the diagonal block (FP64 in
// MMA fragment order), then the inverse of the next diagonal block, formed by
// substitution against the reciprocal diagonal (the reference's inverted-diagonal
// packing, packm.c:143-144, carried to the whole 16 x 16 block) -- and one
// thread of a warpgroup of its own streams segments into a 3-deep shared-memory ring
// with 1-D bulk copies (TMA).  Every wait is bounded (tc_common.cuh); a
// CTA that gives up waits for its own copies and returns, and the call
// reports status 4.
//
// An upper-triangular leaf is the lower one with rows and columns reversed:
// the pack reads A from the bottom-right corner and the kernel addresses B
// from the leaf's last row with a negated row stride.
#include <type_traits>

#include "kernels.cuh"
#include "tc_common.cuh"

namespace {

constexpr int LB = 16;                     // rows of a diagonal block
constexpr int LEAF_BLOCKS = 32;            // diagonal blocks per leaf
constexpr int BLK = LB * LB;               // elements of a packed 16 x 16 block
constexpr int SEG_MAX = LEAF_BLOCKS * BLK; // largest segment: 31 panel blocks + 1 diagonal block
constexpr int RING = 3;
constexpr int XSLOTS = RING + 1;           // solved tiles kept: X_e is published once every warp is
                                           // done with step e - 1 - RING (its segment's slot)

// Offset (elements) of step d's segment in a leaf of nb blocks: the leaf
// starts with diagonal block 0, then segment d = (nb - 1 - d) panel blocks
// and diagonal block d + 1, for d = 0 .. nb - 2.
__host__ __device__ inline long seg_off(int d, int nb) {
  return (long)BLK * (1 + (long)d * nb - (long)d * (d - 1) / 2);
}

__device__ __forceinline__ void dmma(double (&c)[4], double a0, double a1, double b0) {
  asm volatile(
      "mma.sync.aligned.m16n8k4.row.col.f64.f64.f64.f64 {%0,%1,%2,%3}, {%4,%5}, {%6}, "
      "{%0,%1,%2,%3};\n"
      : "+d"(c[0]), "+d"(c[1]), "+d"(c[2]), "+d"(c[3])
      : "d"(a0), "d"(a1), "d"(b0));
}

__device__ __forceinline__ void lds128(double (&v)[2], uint32_t addr) {
  asm volatile("ld.shared.v2.f64 {%0, %1}, [%2];" : "=d"(v[0]), "=d"(v[1]) : "r"(addr));
}

struct LeafPackArgs {
  const void *a;
  long rs_a, cs_a;
  int m;          // order of the whole solve
  int leaf_rows;  // 512
  int lower, unit;
  void *out;
  long leaf_stride;  // elements per packed leaf
};

// Element (i, p) of a leaf in lower orientation (rows r0 .. r0 + rows); the
// identity outside it; the stored diagonal replaced by its reciprocal (or 1
// for a unit diagonal); the unstored triangle never read.
template <typename T>
__device__ T leaf_elem(const LeafPackArgs &a, long r0, int rows, int i, int p) {
  if (i >= rows || p >= rows) return i == p ? T(1) : T(0);
  if (p > i) return T(0);
  const long ri = a.lower ? r0 + i : r0 + rows - 1 - i;
  const long pj = a.lower ? r0 + p : r0 + rows - 1 - p;
  const T *x = (const T *)a.a;
  if (i == p) return a.unit ? T(1) : T(1) / x[ri * a.rs_a + pj * a.cs_a];
  return x[ri * a.rs_a + pj * a.cs_a];
}

// grid (LEAF_BLOCKS, leaves * LEAF_BLOCKS), 256 threads: blockIdx.y =
// leaf * LEAF_BLOCKS + s; s = 0 is diagonal block 0, s = d + 1 is step d's
// segment, whose block x is panel block d + 1 + x or, for the last x, the
// inverse of diagonal block d + 1.  FP64 blocks are stored in MMA
// A-fragment order; FP32 blocks column-major.
template <typename T>
__global__ void __launch_bounds__(256) trsm_leaf_pack_kernel(const LeafPackArgs a) {
  __shared__ T tile[LB][LB + 1];
  const int leaf = blockIdx.y / LEAF_BLOCKS, s = blockIdx.y % LEAF_BLOCKS, x = blockIdx.x;
  const long r0 = (long)leaf * a.leaf_rows;
  const int rows = (int)min((long)a.leaf_rows, a.m - r0);
  const int nb = (rows + LB - 1) / LB;
  int bi, bp;  // block coordinates in the leaf
  bool diag;
  long off;
  if (s == 0) {
    if (x > 0) return;
    bi = bp = 0;
    diag = true;
    off = 0;
  } else {
    const int d = s - 1;
    if (d > nb - 2 || x > nb - 1 - d) return;
    diag = x == nb - 1 - d;
    bi = diag ? d + 1 : d + 1 + x;
    bp = diag ? d + 1 : d;
    off = seg_off(d, nb) + (long)x * BLK;
  }
  const int tid = threadIdx.x;
  // Read with the stored matrix's unit stride running across the warp.
  const bool rows_fast = labs(a.rs_a) <= labs(a.cs_a);
  const int ri = rows_fast ? tid % LB : tid / LB, pi = rows_fast ? tid / LB : tid % LB;
  tile[ri][pi] = leaf_elem<T>(a, r0, rows, bi * LB + ri, bp * LB + pi);
  __syncthreads();
  if (diag) {
    // The block's inverse, column j by thread j: forward substitution
    // L x = e_j against the reciprocal diagonal (tile[i][i] = 1 / a_ii, as
    // the reference packs it, packm.c:143-144).
    T x[LB];
    if (tid < LB) {
#pragma unroll
      for (int i = 0; i < LB; ++i) {
        T r = i == tid ? T(1) : T(0);
#pragma unroll
        for (int q = 0; q < i; ++q) r = fma(-tile[i][q], x[q], r);
        x[i] = r * tile[i][i];
      }
    }
    __syncthreads();
    if (tid < LB) {
#pragma unroll
      for (int i = 0; i < LB; ++i) tile[i][tid] = x[i];
    }
    __syncthreads();
  }
  T *out = (T *)a.out + (long)leaf * a.leaf_stride + off;
  if (sizeof(T) == 8) {
    // MMA A-fragment order: (ks * 32 + lane) * 2 + h holds row g + 8h,
    // column 4 ks + t (lane = 4 g + t).
    const int ks = tid >> 6, lane = (tid >> 1) & 31, h = tid & 1;
    out[tid] = tile[(lane >> 2) + 8 * h][4 * ks + (lane & 3)];
  } else {
    out[tid] = tile[tid % LB][tid / LB];  // column-major
  }
}

template <typename T>
struct LeafArgs {
  const T *pack;  // this leaf's packed A
  int rows;       // rows of the leaf
  T *b;           // the leaf's first row (lower orientation)
  long rs_b, cs_b;
  int n;          // right-hand sides
  T alpha;        // B is scaled by it as it is read
  int *err;
  unsigned long long wait_ns;
};

// Shape of a CTA: NCG column groups (8 columns of FP64, 32 of FP32), the rows of
// each dealt out in blocks of 16 to its RG = W / NCG warps in turn.
template <typename T, int NCG, int W>
struct Leaf {
  static constexpr bool F64 = sizeof(T) == 8;
  // W warps solve; a warpgroup, of which one thread feeds the ring, gives them its
  // registers: 168 a thread at launch (65536 / 384), 4 * 32 * 56 + 8 * 32 * 216 =
  // 62464 of 64512, or 96 (65536 / 640), 4 * 32 * 32 + 16 * 32 * 112 = 61440.
  static constexpr int THREADS = 32 * (W + 4);
  static constexpr int FEED_REGS = W == 8 ? 56 : 32, SOLVE_REGS = W == 8 ? 216 : 112;
  static constexpr int RG = W / NCG;
  static constexpr int NBW = LEAF_BLOCKS / RG;  // row blocks of a warp
  static constexpr int CW = F64 ? 8 : 32;       // columns of a group
  static constexpr int NBC = NCG * CW;          // columns of a CTA
  // Rows of a solved tile in shared memory: 8 doubles make both the fragment's
  // 16-byte stores and its loads conflict-free; 36 floats keep 16-byte accesses
  // aligned and the transposed ones at two to a bank.
  static constexpr int XLD = F64 ? 8 : 36;
  static constexpr int TILE = LB * XLD;
  static constexpr int RHS = F64 ? 0 : LEAF_BLOCKS * TILE;  // FP32: B, apart from the sums
  static constexpr size_t SMEM = sizeof(T) * ((size_t)RING * SEG_MAX + BLK + XSLOTS * NCG * TILE + RHS) +
                                 sizeof(uint64_t) * (2 * RING + 1 + XSLOTS * NCG) + 16;
};

template <typename T, int NCG, int W>
__global__ void __launch_bounds__(32 * (W + 4), 1) trsm_leaf_kernel(const __grid_constant__ LeafArgs<T> p) {
  using L = Leaf<T, NCG, W>;
  constexpr bool F64 = L::F64;
  constexpr int RG = L::RG, NBW = L::NBW, XLD = L::XLD, AE = F64 ? 4 : 16;
  extern __shared__ __align__(128) unsigned char smem[];
  T *seg = (T *)smem;                  // [RING][SEG_MAX]
  T *diag0 = seg + RING * SEG_MAX;     // [BLK]
  T *xs = diag0 + BLK;                 // [XSLOTS][NCG][TILE]
  T *rhs = xs + XSLOTS * NCG * L::TILE;
  uint64_t *full = (uint64_t *)(rhs + L::RHS);  // [RING] segment landed
  uint64_t *empty = full + RING;                // [RING] every warp done with it
  uint64_t *dbar = empty + RING;                // diagonal block 0 landed
  uint64_t *ready = dbar + 1;                   // [XSLOTS][NCG] X_d published
  volatile int *abort_flag = (volatile int *)(ready + XSLOTS * NCG);
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int nb = (p.rows + LB - 1) / LB;

  if (tid == 0) {
    for (int i = 0; i < RING; ++i) {
      tc::mbar_init(&full[i], 1);
      tc::mbar_init(&empty[i], W);
    }
    tc::mbar_init(dbar, 1);
    for (int i = 0; i < XSLOTS * NCG; ++i) tc::mbar_init(&ready[i], 1);
    *abort_flag = 0;
    tc::fence_barrier_init();
  }
  __syncthreads();

  int issued = 0;  // segments issued (the producer's lane 0)
  if (warp >= W) {
    tc::setmaxnreg_dec<L::FEED_REGS>();
    if (warp == W && lane == 0) {
      tc::mbar_arrive_expect_tx(dbar, BLK * sizeof(T));
      tc::bulk_load_1d(diag0, p.pack, BLK * sizeof(T), dbar);
      for (int d = 0; d < nb - 1; ++d) {
        const int slot = d % RING;
        if (d >= RING &&
            !tc::mbar_wait(&empty[slot], (d / RING - 1) & 1, abort_flag, p.err, p.wait_ns))
          break;
        const uint32_t bytes = (uint32_t)((nb - d) * BLK * sizeof(T));
        tc::mbar_arrive_expect_tx(&full[slot], bytes);
        tc::bulk_load_1d(seg + slot * SEG_MAX, p.pack + seg_off(d, nb), bytes, &full[slot]);
        issued = d + 1;
      }
    }
  } else {
    tc::setmaxnreg_inc<L::SOLVE_REGS>();
    const int cg = warp % NCG, rg = warp / NCG;
    const long col0 = (long)blockIdx.x * L::NBC + cg * L::CW;
    const int g = F64 ? lane >> 2 : lane >> 3;  // FP64: rows g, g + 8; FP32: rows 4 g .. 4 g + 3
    const int t = F64 ? lane & 3 : lane & 7;    // FP64: columns 2 t, 2 t + 1; FP32: 4 t .. 4 t + 3
    const bool rows_fast = labs(p.rs_b) <= labs(p.cs_b);
    auto wait = [&](uint64_t *bar, int use) {
      const bool ok = tc::mbar_wait(bar, use & 1, abort_flag, p.err, p.wait_ns);
      return __all_sync(0xffffffffu, ok) != 0;
    };
    auto xtile = [&](int d) { return xs + ((d % XSLOTS) * NCG + cg) * L::TILE; };

    // acc[0] is always the warp's next block to solve.  FP64: B minus the updates
    // so far; FP32: minus the updates' sum, B itself waits in shared memory, so
    // that the updates' roundings are of their (smaller) sum.
    T acc[NBW][AE];
    // FP64: the lane's first element of B (row g of block 0, column 2 t).
    T *const b00 = p.b + g * p.rs_b + (col0 + 2 * t) * p.cs_b;
    const int ncol = (int)min(p.n - col0 - 2 * t, 2L);  // its columns that exist
    if constexpr (F64) {
      const T *src = b00 + rg * LB * p.rs_b;
#pragma unroll
      for (int q = 0; q < NBW; ++q) {
#pragma unroll
        for (int e = 0; e < 4; ++e) {
          const bool in = (rg + RG * q) * LB + g + 8 * (e >> 1) < p.rows && (e & 1) < ncol;
          acc[q][e] = in ? src[8 * (e >> 1) * p.rs_b + (e & 1) * p.cs_b] : T(0);
        }
        src += RG * LB * p.rs_b;
      }
      if (p.alpha != T(1)) {
#pragma unroll
        for (int q = 0; q < NBW; ++q)
#pragma unroll
          for (int e = 0; e < 4; ++e)
            acc[q][e] = (rg + RG * q) * LB + g + 8 * (e >> 1) < p.rows ? p.alpha * acc[q][e] : T(0);
      }
    } else {
#pragma unroll
      for (int q = 0; q < NBW; ++q) {
        T *tile = rhs + (rg + RG * q) * L::TILE;
#pragma unroll
        for (int e = 0; e < LB; ++e) {
          const int idx = e * 32 + lane;
          const int r = rows_fast ? idx % LB : idx / 32, c = rows_fast ? idx / LB : idx % 32;
          const int row = (rg + RG * q) * LB + r;
          const long col = col0 + c;
          tile[r * XLD + c] = row < p.rows && col < p.n ? p.b[row * p.rs_b + col * p.cs_b] : T(0);
        }
#pragma unroll
        for (int e = 0; e < AE; ++e) acc[q][e] = T(0);
      }
      __syncwarp();
    }

    // FP64: a tile x as B operand, the fragments of its four k steps, and
    // c += blk x for one 16 x 16 block of A.
    auto load_x = [&](double (&xf)[4], const T *x) {
#pragma unroll
      for (int ks = 0; ks < 4; ++ks) xf[ks] = x[(4 * ks + t) * XLD + g];
    };
    auto mma_block = [&](double (&c)[4], const T *blk, const double (&xf)[4]) {
#pragma unroll
      for (int ks = 0; ks < 4; ++ks) {
        const double2 a = ((const double2 *)blk)[ks * 32 + lane];
        dmma(c, a.x, a.y, xf[ks]);
      }
    };
    // FP32: c[i] += (MINUS: -=) the block at b[i] times the tile x, i < N.  One
    // block alone is unrolled for its latency, several only as far as their
    // independent chains need (the update's code stays in the instruction cache).
    auto fma_blocks = [&](auto nc, auto minus, auto &c, const T *const *b, const T *x) {
      constexpr int N = decltype(nc)::value, U = N == 1 ? LB : 4;
      constexpr bool MINUS = decltype(minus)::value;
#pragma unroll U
      for (int k = 0; k < LB; ++k) {
        const float4 v = *(const float4 *)&x[k * XLD + 4 * t];
        const float xv[4] = {MINUS ? -v.x : v.x, MINUS ? -v.y : v.y, MINUS ? -v.z : v.z,
                             MINUS ? -v.w : v.w};
#pragma unroll
        for (int i = 0; i < N; ++i) {
          const float4 a = *(const float4 *)&b[i][k * LB + 4 * g];
#pragma unroll
          for (int j = 0; j < 4; ++j) {
            c[i][j] = fmaf(a.x, xv[j], c[i][j]);
            c[i][4 + j] = fmaf(a.y, xv[j], c[i][4 + j]);
            c[i][8 + j] = fmaf(a.z, xv[j], c[i][8 + j]);
            c[i][12 + j] = fmaf(a.w, xv[j], c[i][12 + j]);
          }
        }
      }
    };
    using One = std::integral_constant<int, 1>;
    auto store_tile = [&](T *x, const T (&c)[AE]) {
      if constexpr (F64) {
        *(double2 *)&x[g * XLD + 2 * t] = make_double2(c[0], c[1]);
        *(double2 *)&x[(g + 8) * XLD + 2 * t] = make_double2(c[2], c[3]);
      } else {
#pragma unroll
        for (int i = 0; i < 4; ++i)
          *(float4 *)&x[(4 * g + i) * XLD + 4 * t] =
              make_float4(c[4 * i], c[4 * i + 1], c[4 * i + 2], c[4 * i + 3]);
      }
    };
    int next = rg;  // the row block in acc[0]
    // acc[0], fully updated: X = inv(D) R, published to the group's other warps
    // and written to B; the warp's blocks move up by one.
    auto solve = [&](const T *dinv) {
      T *x = xtile(next);
      if constexpr (!F64) {
        const T *tile = rhs + next * L::TILE;
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          const float4 b = *(const float4 *)&tile[(4 * g + i) * XLD + 4 * t];
          acc[0][4 * i] = fmaf(p.alpha, b.x, acc[0][4 * i]);
          acc[0][4 * i + 1] = fmaf(p.alpha, b.y, acc[0][4 * i + 1]);
          acc[0][4 * i + 2] = fmaf(p.alpha, b.z, acc[0][4 * i + 2]);
          acc[0][4 * i + 3] = fmaf(p.alpha, b.w, acc[0][4 * i + 3]);
        }
      }
      store_tile(x, acc[0]);
      __syncwarp();
      T c[1][AE];
#pragma unroll
      for (int e = 0; e < AE; ++e) c[0][e] = T(0);
      // The product multiplies the zeros above inv(D)'s diagonal as well: a
      // non-finite element of R spoils its whole column.  Then the rows before that
      // element are formed without it, and the others by inv(D)'s lower triangle
      // alone, as a substitution leaves them.  (FP64 votes on R's exponents before
      // the MMAs: 0-1.1% of a leaf, 1.4-6% on the product behind them.  FP32 looks
      // at a row of the product, in which a spoilt column shows: no cost.)
      if constexpr (F64) {
        const int top = max(max(__double2hiint(acc[0][0]) & 0x7fffffff, __double2hiint(acc[0][1]) & 0x7fffffff),
                            max(__double2hiint(acc[0][2]) & 0x7fffffff, __double2hiint(acc[0][3]) & 0x7fffffff));
        const bool spoilt = __any_sync(0xffffffffu, top >= 0x7ff00000);
        double r[4];
        load_x(r, x);
        if (!spoilt) {
          mma_block(c[0], dinv, r);
        } else {
#pragma unroll
          for (int i = 0; i < 4; ++i) r[i] = isfinite(r[i]) ? r[i] : 0.0;
          mma_block(c[0], dinv, r);
#pragma unroll
          for (int e = 0; e < 4; ++e) {
            const int row = g + 8 * (e >> 1);
            bool behind = false;
            double sum = 0.0;
#pragma unroll 1
            for (int q = 0; q <= row; ++q) {  // inv(D) is in MMA fragment order
              const double v = x[q * XLD + 2 * t + (e & 1)];
              sum = fma(dinv[((q >> 2) * 32 + 4 * g + (q & 3)) * 2 + (e >> 1)], v, sum);
              behind |= !isfinite(v);
            }
            if (behind) c[0][e] = sum;
          }
        }
        __syncwarp();
        store_tile(x, c[0]);
      } else {
        fma_blocks(One(), std::false_type(), c, &dinv, x);
        const bool spoilt = !isfinite(c[0][0]) || !isfinite(c[0][1]) || !isfinite(c[0][2]) ||
                            !isfinite(c[0][3]);
        const bool any = __any_sync(0xffffffffu, spoilt);
        __syncwarp();
        if (!any) {
          store_tile(x, c[0]);
        } else {
#pragma unroll 1
          for (int i = LB - 1; i >= 0; --i) {  // column `lane`, in place
            float sum = 0.f;
#pragma unroll 1
            for (int q = 0; q <= i; ++q) sum = fmaf(dinv[q * LB + i], x[q * XLD + lane], sum);
            x[i * XLD + lane] = sum;
          }
        }
      }
      __syncwarp();
      if (lane == 0) tc::mbar_arrive(&ready[(next % XSLOTS) * NCG + cg]);
      if constexpr (F64) {
        T *out = b00 + next * LB * p.rs_b;
#pragma unroll
        for (int e = 0; e < 4; ++e)
          if (next * LB + g + 8 * (e >> 1) < p.rows && (e & 1) < ncol)
            out[8 * (e >> 1) * p.rs_b + (e & 1) * p.cs_b] = c[0][e];
      } else if (rows_fast) {  // two columns of 16 rows to a store
        const int r = lane % LB, row = next * LB + r;
        const long col = col0 + lane / LB;
        T *out = p.b + row * p.rs_b + col * p.cs_b;
        const int left = row < p.rows ? (int)min(p.n - col, 32L) : 0;
#pragma unroll
        for (int e = 0; e < LB; ++e) {
          if (2 * e < left) *out = x[r * XLD + lane / LB + 2 * e];
          out += 2 * p.cs_b;
        }
      } else {  // a row to a store
        T *out = p.b + next * LB * p.rs_b + (col0 + lane) * p.cs_b;
        const int left = col0 + lane < p.n ? p.rows - next * LB : 0;
#pragma unroll
        for (int e = 0; e < LB; ++e) {
          if (e < left) *out = x[e * XLD + lane];
          out += p.rs_b;
        }
      }
#pragma unroll
      for (int q = 0; q + 1 < NBW; ++q)
#pragma unroll
        for (int e = 0; e < AE; ++e) acc[q][e] = acc[q + 1][e];
      next += RG;
    };

    bool ok = true;
    if (rg == 0) {
      ok = wait(dbar, 0);
      if (ok) solve(diag0);
    }
    for (int d = 0; ok && d + 1 < nb; ++d) {
      const int slot = d % RING;
      ok = wait(&full[slot], d / RING);
      if (!ok) break;
      if (next < nb) {
        ok = wait(&ready[(d % XSLOTS) * NCG + cg], d / XSLOTS);
        if (!ok) break;
        const T *sg = seg + slot * SEG_MAX;
        if constexpr (F64) {
          double xf[4];  // -X_d
          load_x(xf, xtile(d));
#pragma unroll
          for (int i = 0; i < 4; ++i) xf[i] = -xf[i];
          if (next == d + 1) {
            // The step's critical path comes first.
            mma_block(acc[0], sg, xf);
            solve(sg + (nb - 1 - d) * BLK);
          }
          // Two blocks at a time, for two chains of MMAs.  Where the second lies
          // past the leaf its accumulators are dead; it reads the first's block.
          constexpr int KS = W == 8 ? 4 : 2;  // k steps of fragments loaded ahead
          const uint32_t a0 = tc::smem_u32(sg) + lane * 16;
#pragma unroll
          for (int q = 0; q < NBW; q += 2) {
            const int rb = next + RG * q;
            if (rb < nb) {
              const uint32_t b0 = a0 + (rb - d - 1) * (BLK * 8);
              const uint32_t b1 = b0 + (rb + RG < nb ? RG * BLK * 8 : 0);
#pragma unroll
              for (int k0 = 0; k0 < 4; k0 += KS) {
                double f0[KS][2], f1[KS][2];
#pragma unroll
                for (int ks = 0; ks < KS; ++ks) {
                  lds128(f0[ks], b0 + (k0 + ks) * 512);
                  lds128(f1[ks], b1 + (k0 + ks) * 512);
                }
#pragma unroll
                for (int ks = 0; ks < KS; ++ks) {
                  dmma(acc[q], f0[ks][0], f0[ks][1], xf[k0 + ks]);
                  dmma(acc[q + 1], f1[ks][0], f1[ks][1], xf[k0 + ks]);
                }
              }
            }
          }
        } else {
          static_assert(F64 || NBW == 4, "four blocks a warp");
          const T *x = xtile(d);
          if (next == d + 1) {
            fma_blocks(One(), std::true_type(), acc, &sg, x);
            solve(sg + (nb - 1 - d) * BLK);
          }
          // Three or four blocks, or up to two; dead ones as above.
          const T *b[4];
          b[0] = sg + (next - d - 1) * BLK;
#pragma unroll
          for (int i = 1; i < 4; ++i) b[i] = next + RG * i < nb ? b[0] + RG * i * BLK : b[0];
          if (next + 2 * RG < nb)
            fma_blocks(std::integral_constant<int, 4>(), std::true_type(), acc, b, x);
          else if (next < nb)
            fma_blocks(std::integral_constant<int, 2>(), std::true_type(), acc, b, x);
        }
      }
      // Reads done before the copy that refills the slot.
      tc::fence_proxy_async();
      __syncwarp();
      if (lane == 0) tc::mbar_arrive(&empty[slot]);
    }
  }
  // Every wait above is bounded, so every thread comes here; if a warp gave up,
  // copies may still be in flight into this CTA's shared memory.
  __syncthreads();
  if (*abort_flag && warp == W && lane == 0) {
    tc::mbar_wait_drain(dbar, 0);
    for (int s = issued < RING ? 0 : issued - RING; s < issued; ++s)
      tc::mbar_wait_drain(&full[s % RING], (s / RING) & 1);
  }
}

}  // namespace

extern "C" long b200_trsm_leaf_rows(void) { return (long)LB * LEAF_BLOCKS; }

extern "C" long b200_trsm_leaf_stride(void) {
  return (long)BLK * LEAF_BLOCKS * (LEAF_BLOCKS + 1) / 2;
}

// Packs every leaf of op(A) (order m, normalised to lower / upper with
// strides) for trsm_leaf_kernel: leaves * b200_trsm_leaf_stride() elements.
extern "C" int b200_trsm_leaf_pack(int dtype, const void *a, long rs_a, long cs_a, int m,
                                   int lower, int unit, void *out) {
  if (m <= 0) return B200_OK;
  cudaStream_t s = b200_cur_stream();
  const long L = b200_trsm_leaf_rows();
  const long leaves = b200_ceil_div(m, L);
  if (leaves * LEAF_BLOCKS > 65535) return b200_set_error(B200_EINVAL, "trsm: order too large");
  LeafPackArgs pa{a, rs_a, cs_a, m, (int)L, lower, unit, out, b200_trsm_leaf_stride()};
  dim3 grid(LEAF_BLOCKS, (unsigned)(leaves * LEAF_BLOCKS));
  B200ProfScope prof(dtype == B200_F32 ? "trsm_leaf_pack_s" : "trsm_leaf_pack_d", s);
  if (dtype == B200_F32) trsm_leaf_pack_kernel<float><<<grid, 256, 0, s>>>(pa);
  else trsm_leaf_pack_kernel<double><<<grid, 256, 0, s>>>(pa);
  B200_LAUNCH_CHECK();
  return B200_OK;
}

// Solves one leaf (`rows` rows) of a packed solve for n right-hand sides, B
// scaled by alpha first:
// b points at the leaf's first row in lower orientation (for an upper leaf,
// its last row, with rs_b negated).
template <typename T, int NCG, int W>
int leaf_launch(const LeafArgs<T> &la, cudaStream_t s) {
  using L = Leaf<T, NCG, W>;
  static B200Once once;
  B200_TRY(b200_once(once, "trsm leaf kernel: set-up failed", []() -> int {
    // The register split adds up only for this allocation (an increase that cannot
    // be granted would wait for good).
    cudaFuncAttributes fa;
    B200_CUDA_TRY(cudaFuncGetAttributes(&fa, trsm_leaf_kernel<T, NCG, W>));
    if (fa.numRegs * L::THREADS < 128 * L::FEED_REGS + 32 * W * L::SOLVE_REGS)
      return b200_set_error(B200_ECUDA, "trsm leaf kernel: unexpected register allocation");
    B200_CUDA_TRY(cudaFuncSetAttribute(trsm_leaf_kernel<T, NCG, W>,
                                       cudaFuncAttributeMaxDynamicSharedMemorySize, (int)L::SMEM));
    return B200_OK;
  }));
  const long grid = b200_ceil_div(la.n, L::NBC);
  if (grid > 0x7fffffffL) return b200_set_error(B200_EINVAL, "trsm: too many right-hand sides");
  B200ProfScope prof(sizeof(T) == 4 ? "trsm_leaf_s" : "trsm_leaf_d", s);
  trsm_leaf_kernel<T, NCG, W><<<(unsigned)grid, L::THREADS, L::SMEM, s>>>(la);
  B200_LAUNCH_CHECK();
  return B200_OK;
}

template <typename T>
int leaf_solve(const void *pack, int rows, T *b, long rs_b, long cs_b, int n, double alpha) {
  if (rows <= 0 || n <= 0) return B200_OK;
  cudaStream_t s = b200_cur_stream();
  const LeafArgs<T> la{(const T *)pack, rows, b, rs_b, cs_b, n, (T)alpha, b200_device_error_word(),
                       B200_WAIT_NS};
  if constexpr (sizeof(T) == 4) {
    return leaf_launch<T, 1, 8>(la, s);  // 16 warps: 2-4% slower
  } else {
    // 16 columns to a CTA, or 8 where those still fit the SMs in one wave (twice
    // the SMs on the same columns).  DTRSM calls, us for 8 columns / 16 on 8 warps /
    // 16 on 16 warps: 500 x 300 57 / 72 / 67, 1000 x 1000 130 / 159 / 149, 1500 x
    // 1500 300 / 279 / 263, 700 x 8000 322 / 306 / 281, 4096 x 4096 2674 / 2573 /
    // 2501; 32 columns 82 us a leaf on 8 warps and 2734 a call on 16 (registers
    // spill).  Every column gets the same bits in each.
    if (n > 8L * b200_sm_count()) return leaf_launch<T, 2, 16>(la, s);
    return leaf_launch<T, 1, 8>(la, s);
  }
}

extern "C" int b200_trsm_leaf_solve(int dtype, const void *pack, int rows, void *b, long rs_b,
                                    long cs_b, int n, double alpha) {
  if (dtype == B200_F32) return leaf_solve<float>(pack, rows, (float *)b, rs_b, cs_b, n, alpha);
  return leaf_solve<double>(pack, rows, (double *)b, rs_b, cs_b, n, alpha);
}
