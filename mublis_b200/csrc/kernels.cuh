// kernels.cuh -- launchers shared between the CUDA translation units.
#pragma once

#include <cuda.h>
#include <cuda_bf16.h>
#include <cuda_fp16.h>

#include <vector>

#include "common.cuh"

// Logical operand view for packing.  Element (r, c) of the stored operand
// lives at x[r * rs + c * cs]; `struc/uplo/diag` give its logical view
// (frame/l1m/packm.c:40-71) and `mask_rel` a domain relation applied as
// rel(mask_rel, c, r) (pi on A's (i, p) or jp on B's (p, j)).
struct PackView {
  const void *x;
  long rs, cs;
  int struc, uplo, diag;
  int mask_rel;
};

// Logical element (r, c) of a view (frame/l1m/packm.c:40-71): zero outside
// the mask relation, the stored triangle reflected for a symmetric operand,
// zero outside it for a triangular one (unit / inverted diagonal applied).
// Elements outside the stored triangle are never read.
template <typename T>
__device__ __forceinline__ T load_logical(const PackView &v, long r, long c) {
  const T *x = (const T *)v.x;
  if (!b200_rel(v.mask_rel, c, r)) return T(0);
  long delta = r - c;
  bool stored = v.uplo == MUBLIS_LOWER ? delta >= 0 : (v.uplo == MUBLIS_UPPER ? delta <= 0 : true);
  if (v.struc == MUBLIS_STRUC_SYMMETRIC) {
    return stored ? x[r * v.rs + c * v.cs] : x[c * v.rs + r * v.cs];
  }
  if (v.struc == MUBLIS_STRUC_TRIANGULAR) {
    if (!stored) return T(0);
    if (delta == 0 && v.diag == MUBLIS_PACKM_DIAG_UNIT) return T(1);
    T val = x[r * v.rs + c * v.cs];
    if (delta == 0 && v.diag == MUBLIS_PACKM_DIAG_INVERT) val = T(1) / val;
    return val;
  }
  return x[r * v.rs + c * v.cs];
}

// Output orientation of a packed panel.  The panel covers mn in [0, mn_pad)
// and kk in [kk0, kk1); logical element (mn, kk - kk0) is taken from the
// view, as (r, c) = (mn, kk) for an A-side view or (kk, mn) for a B-side
// view; anything past mn_len / k_len is zero.
enum PackLayout {
  PACK_MN_MAJOR = 0,  // out[kk * ld + mn]       (SIMT kernels)
  PACK_K_MAJOR = 1,   // out[mn * ld + kk]       (tcgen05 kernels)
  PACK_FRAG64 = 2     // doubles in mma.m16n8k4 fragment order (FP64 MMA
                      // kernel), ld = Kpad: see b200_frag64_offset
};

// Offset of element (mn, kk) of a PACK_FRAG64 panel (Kpad = ld, a multiple
// of 16; Mpad a multiple of 128).  The panel is a sequence of 128-row
// strips; a strip is a sequence of MMA steps of 4 k (step s of a 16-k block
// holds k = 8 (s / 2) + 2 t + s % 2, t = 0..3); a step of a strip is 8 blocks
// of 16 rows, each 32 lanes x 2 doubles in the order an mma.m16n8k4 .f64
// fragment is held: lane = 4 (mn % 16 / 2) + t holds rows mn % 16 even and odd
// as one 16-byte pair.  An A operand strip is a 16-row block fragment (a0, a1)
// per lane; a B operand strip is two 8-column fragments (even columns, odd
// columns) per lane.  So one k-block of 16 of one strip is 16 KB contiguous,
// and every warp fragment load is 512 contiguous bytes.
__host__ __device__ inline long b200_frag64_offset(long mn, long kk, long kpad) {
  const long step = (kk >> 4) * 4 + ((kk >> 2) & 2) + (kk & 1);
  return (((((mn >> 7) * (kpad >> 2) + step) * 8 + ((mn & 127) >> 4)) * 32 +
           ((((mn >> 1) & 7) << 2) | ((kk >> 1) & 3))) << 1) |
         (mn & 1);
}

enum PackXform {
  PACK_COPY = 0,         // T -> T
  PACK_BF16_SPLIT = 1,   // f32 -> `terms` bf16 planes (hi, lo[, lo2])
  PACK_INT8_SLICES = 2,  // f64 -> `terms` int8 planes of 7-bit slices of
                         // x * 2^(7 - e), e from the row/column abs-max
  PACK_INT8_MODULI = 3,  // f64 -> `terms` int8 planes: the symmetric residues
                         // of X = rint(x * 2^(bits - e)) modulo each modulus
  PACK_FP16_SPLIT = 4    // f32 -> 2 fp16 planes of xs = x * 2^(15 - e) (e from
                         // the row/column abs-max, |xs| < 2^15): hi = rn(xs),
                         // lo = rn(xs - hi)
};

// fp16 split scaling: the row/column maximum lands just below 2^15, so that
// lo = rn(xs - hi) (about 2^-11 |xs|) stays a normal fp16 number for every
// element down to 2^-18 of its row's maximum (fp16 normals start at 2^-14;
// the tensor cores ran the product noticeably slower on subnormal halves).
constexpr int B200_FP16_SCALE_EXP = 15;

// Pairwise coprime moduli (<= 256, the first one 256) of the modular (CRT)
// Ozaki form and the constants of the pack pass's residues (b200_residue).
constexpr int B200_MAX_MODULI = 16;
struct B200Moduli {
  int n;
  int lo[B200_MAX_MODULI], hi[B200_MAX_MODULI];  // 256^0..3 and 256^4..7 mod m as signed bytes
  int base[B200_MAX_MODULI];                     // 2^23 as a float's bits, plus an offset
  float inv[B200_MAX_MODULI], neg_m[B200_MAX_MODULI];  // 1 / m, -m
};

struct PackOut {
  void *out;
  long ld;
  long plane_stride;  // elements between planes
  int layout, xform, terms;
  const int *exps;                   // scaled forms: e of each mn (b200_scale_exp)
  int bits;                          // PACK_INT8_MODULI: |X| <= 2^bits
  B200Moduli mod;                    // PACK_INT8_MODULI
};

// The symmetric residue of X + 2^56 - (2^56 mod m) ~ X modulo m in the low byte,
// for |X| <= 2^56 given as the two words of X + 2^56 (unsigned bytes b0 .. b7).
// v = sum of b_i (256^i mod m) + offset by two byte dot products; the offset (a
// multiple of m, less 2^56 mod m) keeps v in [0, 2^20), so that with `base` the
// sum is at once the bits of the float 2^23 + v.  Then r = v - m rint(v / m) in
// FP32: v < 2^20 and m >= 193 make the quotient's error below 4e-4, while v / m
// is at least 0.5 / m > 0.0019 away from a half for odd m, so the quotient is
// exact and r the unique residue in [-(m - 1) / 2, (m - 1) / 2].  (m = 256: the
// low byte itself.)  Eight instructions, most of them on the FP32 pipe; cutting X
// into 19-bit pieces in FP64 and reducing with integer multiplies took eleven.
__device__ __forceinline__ uint32_t b200_residue(uint32_t lo, uint32_t hi, const B200Moduli &mod,
                                                 int l) {
  if (l == 0) return lo;
  int v;
  asm("dp4a.u32.s32 %0, %1, %2, %3;" : "=r"(v) : "r"(lo), "r"(mod.lo[l]), "r"(mod.base[l]));
  asm("dp4a.u32.s32 %0, %1, %2, %3;" : "=r"(v) : "r"(hi), "r"(mod.hi[l]), "r"(v));
  const float f = __int_as_float(v) - 8388608.f;
  const float q = __fadd_rn(__fmaf_rn(f, mod.inv[l], 12582912.f), -12582912.f);
  const float r = __fmaf_rn(q, mod.neg_m[l], f);
  return (uint32_t)__float_as_int(__fadd_rn(r, 12582912.f));  // 1.5 2^23 + r
}

// Symmetric residue of t modulo m, in [-floor(m/2), m - 1 - floor(m/2)]
// (within [-128, 127] for m <= 256), for |t| <= 2^29.  u = t + bias lies in
// [0, 2^31); for u < 2^31 and m <= 2^8, floor(u / m) = umulhi(u, mg) >> 7
// with mg = ceil(2^39 / m) exactly (Granlund and Montgomery 1994: the error
// u (mg m - 2^39) / (m 2^39) stays below 1/m; for m = 256 mg is exact), so
// r = u - q m - floor(m/2) needs no correction.
__device__ __forceinline__ int b200_sym_mod(int t, int m, unsigned mg, int bias) {
  const unsigned u = (unsigned)(t + bias);
  const unsigned q = __umulhi(u, mg) >> 7;
  return (int)(u - q * (unsigned)m) - (m >> 1);
}

template <typename T>
int launch_absmax(const PackView &v, bool b_side, long mn_len, long k_len,
                  unsigned long long *absmax, cudaStream_t s);

// exps[i] = b200_scale_exp(absmax[i]) for i < count: the epilogues read one
// int per row / column instead of a 64-bit abs-max and its frexp.
int launch_scale_exps(const unsigned long long *absmax, int *exps, long count, cudaStream_t s);

// Exponent e with max|x| < 2^e (frexp), 0 for an all-zero row.
__device__ inline int b200_scale_exp(unsigned long long absmax_bits) {
  if (absmax_bits == 0) return 0;
  int e;
  frexp(__longlong_as_double((long long)absmax_bits), &e);
  return e;
}

// x * 2^e rounded once.
//  * float: the product is formed exactly in FP64 and rounded once to float;
//    valid for -1022 <= e <= 1023 (the fp16x3 epilogue's e = e_i + f_j - 30
//    stays within [-330, 230] for FP32 inputs).
//  * double: one multiply by the exact power of two where 2^e is a normal
//    number, else ldexp.
__device__ __forceinline__ float b200_pow2_scale(float x, int e) {
  return (float)((double)x * __longlong_as_double((long long)(e + 1023) << 52));
}
__device__ __forceinline__ double b200_pow2_scale(double x, int e) {
  return e >= -1022 && e <= 1023 ? x * __longlong_as_double((long long)(e + 1023) << 52)
                                 : ldexp(x, e);
}

// x * 2^sh for sh within [-252, 254], as two multiplications by exact powers
// of two: the first is the whole factor whenever 2^sh is a normal float (then
// it is one rounding of the exact product, as ldexpf gives); for larger |sh|
// the factor is cut in two.  (The fp16 splits' sh = 15 - e lies in [-113, 163]:
// e is frexp's exponent of an FP32 value, -148 .. 128.)
__device__ __forceinline__ void b200_pow2_factors(int sh, float &f1, float &f2) {
  const int s1 = sh > 127 ? 127 : (sh < -126 ? -126 : sh);
  f1 = __int_as_float((s1 + 127) << 23);
  f2 = __int_as_float((sh - s1 + 127) << 23);
}

// Scale exponents (exps, mn_pad of them) and packed planes of a whole operand in
// one pass over it, for k [0, kk1): false, with nothing launched, when the
// operand or the form is not one it takes (then absmax, scale_exps and pack).
template <typename T>
bool launch_scale_pack(const PackView &v, bool b_side, long mn_len, long k_len, long mn_pad, long kk1,
                       int *exps, const PackOut &o, cudaStream_t s);

template <typename T>
int launch_pack(const PackView &v, bool b_side, long mn_len, long k_len, long mn_pad,
                long kk0, long kk1, const PackOut &o, cudaStream_t s);

// Output tiles that a launch's parameters can list (restricted domains);
// longer lists are uploaded.
constexpr int B200_MAX_LISTED_TILES = 1024;

// Plain FP64 GEMM on the FMA pipe over packed MN-major panels.
template <typename T>
struct SimtGemmArgs {
  const T *ap;  // [Kpad][Mpad]
  const T *bp;  // [Kpad][Npad]
  long lda, ldb;
  T *c;
  long rs_c, cs_c;
  int m, n, k;
  T alpha, beta;
  int jp, ji, pi;
  // Scheduling, filled by the launcher when the caller passes a SimtPolicy:
  // persistent CTAs take units (tile, k-chunk) from a counter.  Left at
  // these defaults, every CTA computes the one tile of its block index.
  const int2 *tile_list = nullptr;  // (tm, tn) of the tiles to compute, or null: all tiles
  int ntiles = 0;                   // tiles scheduled (0: all tiles, one per CTA)
  int splits = 1;                   // k-chunks per tile (split-K)
  int *work = nullptr;              // unit counter (zeroed): persistent CTAs
  int *arrivals = nullptr;          // per tile: k-chunks finished (zeroed), splits > 1
  T *partials = nullptr;            // per unit: its k-chunk's sums, splits > 1
};

// What the launcher needs to schedule a call on persistent CTAs with
// split-K: the whole call's output size (a column panel of a larger call
// carries the call's m and n, so every panel splits its tiles' k ranges as
// the whole call would, and panels stay bit-identical to the one-call
// result).
struct SimtPolicy {
  long m_full, n_full;
};

// Plain FP32 GEMM on the FMA pipe (gemm_ffma.cu).  Each operand is one or two
// (SYR2K read in place) 2-D TMA sources with m (n) innermost.
constexpr int B200_FFMA_TILE = 128, B200_FFMA_BK = 16;
struct FfmaGemmArgs {
  CUtensorMap ta[2], tb[2];
  int a_kpair = 0x7fffffff, b_kpair = 0x7fffffff;  // k at which the second source begins
  float *c = nullptr;
  long rs_c = 1, cs_c = 1;
  int m = 0, n = 0, k = 0;
  float alpha = 0.f, beta = 0.f;
  int jp = MUBLIS_L3_ALL, ji = MUBLIS_L3_ALL, pi = MUBLIS_L3_ALL;
  // Filled by the launcher.
  int *err = nullptr;
  int tiles_m = 0, tiles_n = 0, ntiles = 0, splits = 1, listed = 0;
  int fold = 0x7fffffff;  // k-blocks added in a row, at most,
  int runs = 1;           // and at most this share of a tile's
  const int2 *tile_list = nullptr;
  int *arrivals = nullptr;    // per (tile, warp): k-chunks finished, splits > 1
  float *partials = nullptr;  // per unit: its k-chunk's sums, splits > 1
  uint16_t tiles[B200_MAX_LISTED_TILES];  // tm << 8 | tn
};
// The whole call's output size (a column panel carries the call's).
struct FfmaPolicy {
  long m_full, n_full;
};
// pol == nullptr: no split-K, no domain, nothing allocated.
int launch_ffma_gemm(FfmaGemmArgs &a, const FfmaPolicy *pol, cudaStream_t s);
int b200_ffma_preload();

// Plain FP64 GEMM on the FP64 tensor pipe over PACK_FRAG64 panels.
struct DmmaGemmArgs {
  const double *ap, *bp;  // PACK_FRAG64 panels, Mpad / Npad multiples of 128
  long kq;                // Kpad / 4
  double *c;
  long rs_c, cs_c;
  int m, n, k;
  int tiles_m, tiles_n;
  const int2 *tile_list;  // (tm, tn) of the tiles to compute, or null: all tiles
  int ntiles;             // tiles to compute
  int listed = 0;         // they are listed in `tiles`
  double alpha, beta;
  int jp, ji, pi;
  int *err;
  unsigned long long wait_ns;  // bound of every mbarrier wait
  int stall;                   // failure-detection test: the producer issues no loads
  // Split-K: each tile's k range in `splits` chunks (units tile * splits +
  // chunk, taken round-robin by the persistent CTAs); with splits > 1 every
  // chunk stores its sums in `partials` and the last of a tile's chunks to
  // finish (counted in `arrivals`, zeroed) adds them in chunk order.
  int splits = 1;
  int *arrivals = nullptr;
  double *partials = nullptr;
  // Each operand's layout (B200_DMMA_*): packed panels (ap / bp), or 2-D TMA
  // tiles straight from the caller's matrices, one tensor map per pair (a
  // SYR2K's second pair begins at k = a_kpair / b_kpair, a multiple of the
  // k-block).
  int a_layout = 0, b_layout = 0;
  long a_kpair = 0x7fffffff, b_kpair = 0x7fffffff;
  CUtensorMap ta[2], tb[2];
  uint16_t tiles[B200_MAX_LISTED_TILES];  // tm << 8 | tn
};
int launch_dmma_gemm(const DmmaGemmArgs &a, cudaStream_t s);
constexpr int B200_DMMA_TILE = 128, B200_DMMA_BK = 16;
enum { B200_DMMA_PACKED = 0, B200_DMMA_MN = 1 /* unit stride along m / n */, B200_DMMA_K = 2 /* along k */ };

template <typename T>
struct SimtConfig;

template <>
struct SimtConfig<double> {
  static constexpr int BM = 128, BN = 128, BK = 16;  // panel padding (tiles may be smaller)
};

// pol == nullptr: one tile per CTA, no scratch; otherwise persistent CTAs with
// split-K and stream-ordered scratch.
template <typename T>
int launch_simt_gemm(const SimtGemmArgs<T> &a, cudaStream_t s, const SimtPolicy *pol = nullptr);

// ---- output-tile scheduling shared by the persistent GEMM kernels (sched.cu)

// The product's domain relations (mublis_l3_relation_t values).
struct b200_tile_domain_t {
  int jp, ji, pi;
};

// The BM x BN tiles of an m x n output that write under ji (the reference's
// block_is_outside, l3_driver.c:145-147,165-171), heaviest first (stable),
// as (tm, tn); costs, when given, receives each tile's k-blocks of BK after
// clipping its k range to jp / pi (l3_driver.c:130,148-150,163,171).
void b200_tile_list(long m, long n, long k, int BM, int BN, int BK, b200_tile_domain_t dom,
                    std::vector<int2> *list, std::vector<int> *costs);

// Reverses every other round of `grid` entries of a heaviest-first list that
// `grid` persistent CTAs take round-robin, so that CTA 0 does not get the
// heaviest of every round.
void b200_snake(std::vector<int2> &list, int grid);
// Writes the list as tm << 8 | tn, if it fits `tiles`.
bool b200_list_tiles(const std::vector<int2> &list, uint16_t (&tiles)[B200_MAX_LISTED_TILES]);

// Split-K factor for a whole call (m_full x n_full x k) on `slots` resident
// persistent CTAs that take units (tile, k-chunk) heaviest tile first: the
// S in 1..16 (chunks of at least 8 k-blocks) whose simulated list schedule
// ends first, counting a fixed start-up cost per unit and split_cost
// (k-block times) more per split unit; S > 1 is taken only when it beats
// S = 1 by 10%.  Depends only on its arguments (cached per shape), so every
// column panel of a call splits its tiles as the whole call does.
int b200_split_for(long m_full, long n_full, long k, int BM, int BN, int BK,
                   b200_tile_domain_t dom, long slots, double split_cost);

// ---- small products in one launch (gemm_direct.cu)

// How a product runs there: tile 64 or 32 (0: not there), how many CTAs share a
// tile's k range, and whether sums are folded into totals every B200_DIRECT_RUN
// products.
constexpr int B200_DIRECT_RUN = 128;
struct b200_direct_choice_t {
  int tile, splits, fold;
};
b200_direct_choice_t b200_direct_choice(const b200_l3_desc_t *d);
// On the calling thread's stream; C must overlap no operand.
int launch_direct_gemm(const b200_l3_desc_t *d, const b200_direct_choice_t &ch);

// One problem of a group on the device: op(A) element (i, p) at a[i rs_a + p
// cs_a], op(B) (p, j) at b[p rs_b + j cs_b], C (i, j) at c[i rs_c + j cs_c].
struct b200_group_gemm_t {
  const void *a, *b;
  void *c;
  long rs_a, cs_a, rs_b, cs_b, rs_c, cs_c;
  double alpha, beta;
  int m, n, k;
  int tile0, tiles_m;  // the problem's first tile in the group, tiles along m
  int vec;             // b200_group_vec
};
// Operands that move in 16-byte copies: 1 op(A), 2 op(B).
int b200_group_vec(const b200_group_gemm_t &e, int elt);
// tile: 32 or 64; tile_prob: the problem of each of the `tiles` tiles (0: sets
// the kernel up only, as a stream capture of the launch needs).
int launch_direct_group(int dtype, int tile, const b200_group_gemm_t *table, const int *tile_prob,
                        int tiles, cudaStream_t s);

// b200_is_device_ptr for the many operands of one call (runtime.cu): a pointer
// inside an allocation that an earlier one of the call lay in needs no query.
// Lives for one call, on its thread: nothing is known of the next call's pointers.
class B200DevicePtrs {
 public:
  bool device(const void *p);

 private:
  static constexpr int RANGES = 8, PROBES = 32;
  struct Range {
    uintptr_t base, end;
  } range_[RANGES];
  int count_ = 0, last_ = 0, misses_ = 0, hits_ = 0;
};

// ---- small triangular solves (trsm_small.cu)

constexpr int B200_TRSM_SMALL = 256;      // largest order
constexpr int B200_TRSM_SMALL_COLS = 32;  // right-hand sides per CTA (slab)
// op(A) X = alpha B, X over B: op(A) element (i, p) at a[i rs_a + p cs_a], B
// (i, j) at b[i rs_b + j cs_b].
struct b200_small_trsm_t {
  const void *a;
  void *b;
  long rs_a, cs_a, rs_b, cs_b;
  double alpha;
  long n;
  int m, lower, unit;
  int slab0;  // the problem's first slab in the group
};
// Orders up to this one run on half the warps (a group's are best launched apart).
constexpr int B200_TRSM_SMALL_HALF = 128;
// A group's slabs first_slab ..: slab_prob names the problem of each (0 slabs:
// sets the kernel up only, as a stream capture of the launch needs).
int launch_small_trsm(int dtype, const b200_small_trsm_t *table, const int *slab_prob, int first_slab,
                      int slabs, int max_order, cudaStream_t s);
int launch_small_trsm_one(int dtype, const b200_small_trsm_t &e, cudaStream_t s);

template <typename T>
int launch_scale(int m, int n, T beta, T *c, long rs, long cs, int ji, cudaStream_t s);

// Load the kernels that the allocation-free SGEMM runs besides its GEMM.
int b200_pack_preload();
int b200_scale_preload();
