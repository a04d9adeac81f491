// l3.cu -- the device-side generic L3 driver: pack -> contraction ->
// masked epilogue, for every form.  This is what mublis_l3_{s,d}driver (and
// through it GEMM, SYMM, SYRK, SYR2K, TRMM and TRSM's updates) runs.
//
// Reference flow being replaced (frame/l3/l3_driver.c:49-249): a CPU loop
// nest that packs kc x nc panels of B (:133-142) and mc x kc panels of A
// (:152-161), calls the micro-kernel per MR x NR tile and patches edge and
// triangle tiles through a temporary (:192-234).  Here each operand is packed
// once for the whole call (one HBM pass, pack.cu) and the contraction kernel
// tiles the entire output on the device.
#include <cstdint>
#include <cstdlib>
#include <algorithm>
#include <cstring>
#include <vector>

#include "kernels.cuh"
#include "tc_common.cuh"
#include "tc_gemm.cuh"

// Whether an m x n view C and a rows x cols view X (elements of `elt` bytes)
// may share memory.  Exact for two blocks of one matrix (the same leading
// dimension and unit stride, as the blocks of a recursive solve have: their
// byte intervals interleave although no element is shared); otherwise by
// byte interval, and true for a negative stride.
extern "C" int b200_views_overlap(const void *c, long rs_c, long cs_c, long m, long n, const void *x,
                                  long rs_x, long cs_x, long rows, long cols, long elt) {
  if (rs_c < 0 || cs_c < 0 || rs_x < 0 || cs_x < 0) return 1;
  const intptr_t c0 = (intptr_t)c, x0 = (intptr_t)x;
  const intptr_t c1 = c0 + elt * ((m - 1) * rs_c + (n - 1) * cs_c + 1);
  const intptr_t x1 = x0 + elt * ((rows - 1) * rs_x + (cols - 1) * cs_x + 1);
  if (c1 <= x0 || x1 <= c0) return 0;
  // In one grid of lines of `ld` elements: C is cw x ch (along the unit
  // stride x lines), X is xw x xh.
  const bool c_row = rs_c == 1, x_row = rs_x == 1;
  const long ld = c_row ? cs_c : rs_c, cw = c_row ? m : n, ch = c_row ? n : m;
  const long xld = x_row ? cs_x : rs_x, xw = x_row ? rows : cols, xh = x_row ? cols : rows;
  if ((!c_row && cs_c != 1) || (!x_row && cs_x != 1) || ld != xld || cw > ld || xw > ld ||
      (x0 - c0) % elt != 0)
    return 1;
  const long off = (x0 - c0) / elt;
  long line = off / ld, at = off % ld;
  if (at < 0) at += ld, --line;  // X starts at (at, line) relative to C, 0 <= at < ld
  const bool lines = line < ch && line + xh > 0;
  if (lines && at < cw) return 1;
  // The part of X that runs past the line's end is on the next line.
  return at + xw > ld && line + 1 < ch && line + 1 + xh > 0;
}

namespace {

// "auto" picks, per call, the fastest form whose error is no worse than the
// plain kernel's: the tensor-core forms pay a split/residue pass and, for
// the integer forms, one int8 product per modulus, so below these sizes
// (crossovers measured on B200) plain wins.  FP32: BF16x6 (3-term split,
// error equal to plain FP32) when min(m, n) and k are >= 512 (at 256 x 8192
// x 256 plain is faster).  FP64: the modular Ozaki form with 16 moduli (error
// ~36x below plain FP64) when min(m, n) and k are >= 1024 and m n >= 2048^2,
// i.e. at least 64 of its 256 x 256 tiles (measured: 2048^3 0.65 vs 0.71 ms,
// 1024 x 8192 x 1024 0.58 vs 0.76, 2048 x 8192 x 2048 1.28 vs 2.26, 8192^3
// 8.8 vs 32.4; at 1024 x 1024 x 8192 the two tie).
int resolve_form(const b200_l3_desc_t *d) {
  int f = d->form == B200_FORM_AUTO ? b200_get_default_form(d->dtype) : d->form;
  if (f == B200_FORM_POLICY) {
    const long m = d->policy_m > 0 ? d->policy_m : d->m;
    const long n = d->policy_n > 0 ? d->policy_n : d->n;
    const long k = (long)d->k * d->npairs;
    const long mn = m < n ? m : n;
    // FP32: fp16x3 (normwise error ~0.6x plain) where it is at least as fast
    // as bf16x6 (error ~1.0x plain): from 4096 on (at 2048^3 its abs-max
    // pass and slower fp16 MMAs leave it ~10% behind).
    if (d->dtype == B200_F32) {
      if (mn >= 4096 && k >= 2048) return B200_FORM_FP16X3;
      return mn >= 512 && k >= 512 ? B200_FORM_BF16X6 : B200_FORM_PLAIN;
    }
    return mn >= 1024 && k >= 1024 && m * n >= 2048L * 2048 ? B200_FORM_OZAKI2 : B200_FORM_PLAIN;
  }
  if (d->dtype == B200_F32 && f == B200_FORM_OZAKI) f = B200_FORM_PLAIN;
  if (d->dtype == B200_F64 &&
      (f == B200_FORM_BF16X3 || f == B200_FORM_BF16X6 || f == B200_FORM_FP16X3))
    f = B200_FORM_PLAIN;
  return f;
}

// Pack every (A_t, B_t) pair of the descriptor, concatenated along k, into
// the given panel outputs.
template <typename T>
int pack_pairs(const b200_l3_desc_t *d, const PackOut &oa, long mpad, const PackOut &ob,
               long npad, long kpad, cudaStream_t s) {
  const mublis_l3_product_t &pr = d->product;
  for (int t = 0; t < d->npairs; ++t) {
    long kk0 = (long)t * d->k;
    long kk1 = t + 1 == d->npairs ? kpad : kk0 + d->k;
    PackView va{d->a[t], d->rs_a[t], d->cs_a[t], (int)pr.a.struc, (int)pr.a.uplo,
                (int)pr.a.diag, (int)pr.domain.pi};
    PackView vb{d->b[t], d->rs_b[t], d->cs_b[t], (int)pr.b.struc, (int)pr.b.uplo,
                (int)pr.b.diag, (int)pr.domain.jp};
    B200_TRY(launch_pack<T>(va, false, d->m, d->k, mpad, kk0, kk1, oa, s));
    B200_TRY(launch_pack<T>(vb, true, d->n, d->k, npad, kk0, kk1, ob, s));
  }
  return B200_OK;
}

// FP64 GEMM on the tensor pipe (gemm_dmma.cu) unless MUBLIS_B200_DGEMM=simt
// selects the FMA-pipe kernel.
bool use_dmma() {
  static const bool on = [] {
    const char *e = getenv("MUBLIS_B200_DGEMM");
    return !(e && !strcmp(e, "simt"));
  }();
  return on;
}

// MUBLIS_B200_DIRECT=0 keeps the pack pass for every call and operand;
// MUBLIS_B200_SMALL=0 sends small products (gemm_direct.cu) to the kernels of the
// large ones, which still read operands in place.
bool direct_on() {
  static const bool on = [] {
    const char *e = getenv("MUBLIS_B200_DIRECT");
    return !(e && !strcmp(e, "0"));
  }();
  return on;
}
bool small_on() {
  static const bool on = [] {
    const char *e = getenv("MUBLIS_B200_SMALL");
    return direct_on() && !(e && !strcmp(e, "0"));
  }();
  return on;
}

// A strided FP64 view (rows x cols, element (i, j) at x + i rs + j cs) as a
// TMA source: one stride must be 1 and the other a positive multiple of 2
// elements (16 bytes) at least the unit-stride extent, the base 16-byte
// aligned.  *first_contig: the unit stride runs along the rows index.
bool tma_view_ok(const void *x, long rs, long cs, long rows, long cols, bool *rows_contig) {
  if (((uintptr_t)x & 15) != 0 || rows <= 0 || cols <= 0) return false;
  if (rs == 1 && cs >= rows && cs % 2 == 0) {
    *rows_contig = true;
    return true;
  }
  if (cs == 1 && rs >= cols && rs % 2 == 0) {
    *rows_contig = false;
    return true;
  }
  return false;
}

// Whether C shares memory with an operand of the product.
bool overlaps_operand(const b200_l3_desc_t *d) {
  const long elt = d->dtype == B200_F64 ? 8 : 4;
  for (int t = 0; t < d->npairs; ++t)
    if (b200_views_overlap(d->c, d->rs_c, d->cs_c, d->m, d->n, d->a[t], d->rs_a[t], d->cs_a[t], d->m,
                      d->k, elt) ||
        b200_views_overlap(d->c, d->rs_c, d->cs_c, d->m, d->n, d->b[t], d->rs_b[t], d->cs_b[t], d->k,
                      d->n, elt))
      return true;
  return false;
}

// Whether a tensor map could be made; if not, the operand is packed, which is no
// error of the call's.
bool mapped(int status) {
  if (status != B200_OK) b200_set_error(B200_OK, "");
  return status == B200_OK;
}

// One operand of the FP64 tensor-pipe kernel: read in place (2-D TMA tiles)
// when no element needs changing on the way -- a general, unmasked operand,
// every pair with the same orientation, a SYR2K's pairs meeting on a k-block
// boundary -- and it shares no memory with C (an in-place product must read its
// operand before it is overwritten, which only a copy guarantees); else packed
// into *panel in fragment order, both pairs as one.  Every route adds the same
// products in the same order.
int dmma_operand(const b200_l3_desc_t *d, bool b_side, CUtensorMap (&map)[2], int *layout, long *kpair,
                 void **panel, cudaStream_t s) {
  const mublis_l3_product_t &pr = d->product;
  const mublis_l3_operand_t &o = b_side ? pr.b : pr.a;
  const int mask = b_side ? (int)pr.domain.jp : (int)pr.domain.pi;
  const void *const *x = b_side ? d->b : d->a;
  const long *rs = b_side ? d->rs_b : d->rs_a, *cs = b_side ? d->cs_b : d->cs_a;
  const long rows = b_side ? d->k : d->m, cols = b_side ? d->n : d->k, len = b_side ? d->n : d->m;
  const int T = B200_DMMA_TILE, BK = B200_DMMA_BK;
  bool direct = direct_on() && o.struc == MUBLIS_STRUC_GENERAL && mask == MUBLIS_L3_ALL &&
                (d->npairs == 1 || d->k % BK == 0);
  for (int t = 0; t < d->npairs && direct; ++t) {
    bool rows_contig;
    direct = tma_view_ok(x[t], rs[t], cs[t], rows, cols, &rows_contig) &&
             !b200_views_overlap(d->c, d->rs_c, d->cs_c, d->m, d->n, x[t], rs[t], cs[t], rows, cols, 8);
    if (!direct) break;
    const int lay = rows_contig == b_side ? B200_DMMA_K : B200_DMMA_MN;
    if (t == 0) *layout = lay;
    // k innermost: 16 k x 128 rows; m / n innermost: boxes of 16 x 16 k.
    direct = lay == *layout &&
             mapped(lay == B200_DMMA_K
                        ? b200_make_tmap_f64(&map[t], x[t], d->k, len, b_side ? cs[t] : rs[t], BK, T, 1)
                        : b200_make_tmap_f64(&map[t], x[t], len, d->k, b_side ? rs[t] : cs[t], 16, BK, 1));
  }
  if (direct) {
    if (d->npairs == 2) *kpair = d->k;
    return B200_OK;
  }
  *layout = B200_DMMA_PACKED;
  const long pad = b200_round_up(len, T), kpad = b200_round_up((long)d->k * d->npairs, BK);
  B200_TRY(b200_alloc(panel, sizeof(double) * pad * kpad));
  const PackOut out{*panel, kpad, 0, PACK_FRAG64, PACK_COPY, 1, nullptr};
  for (int t = 0; t < d->npairs; ++t) {
    const long kk0 = (long)t * d->k, kk1 = t + 1 == d->npairs ? kpad : kk0 + d->k;
    const PackView v{x[t], rs[t], cs[t], (int)o.struc, (int)o.uplo, (int)o.diag, mask};
    B200_TRY(launch_pack<double>(v, b_side, len, d->k, pad, kk0, kk1, out, s));
  }
  return B200_OK;
}

int run_dmma(const b200_l3_desc_t *d) {
  cudaStream_t s = b200_cur_stream();
  const long ktot = (long)d->k * d->npairs;
  const long mpad = b200_round_up(d->m, B200_DMMA_TILE);
  const long npad = b200_round_up(d->n, B200_DMMA_TILE);
  const long kpad = b200_round_up(ktot, B200_DMMA_BK);
  DmmaGemmArgs g;
  void *ap = nullptr, *bp = nullptr;
  int st = dmma_operand(d, false, g.ta, &g.a_layout, &g.a_kpair, &ap, s);
  if (st == B200_OK) st = dmma_operand(d, true, g.tb, &g.b_layout, &g.b_kpair, &bp, s);
  // Restricted domains: the tiles that write, heaviest first; in the launch's
  // parameters when there are few, else uploaded.
  const int tiles_m = (int)(mpad / B200_DMMA_TILE), tiles_n = (int)(npad / B200_DMMA_TILE);
  const mublis_l3_domain_t &dom = d->product.domain;
  void *list = nullptr;
  int ntiles = tiles_m * tiles_n;
  if (st == B200_OK &&
      (dom.ji != MUBLIS_L3_ALL || dom.jp != MUBLIS_L3_ALL || dom.pi != MUBLIS_L3_ALL)) {
    std::vector<int2> flat;
    b200_tile_list(d->m, d->n, ktot, B200_DMMA_TILE, B200_DMMA_TILE, B200_DMMA_BK,
                   {dom.jp, dom.ji, dom.pi}, &flat, nullptr);
    ntiles = (int)flat.size();
    b200_snake(flat, b200_sm_count());
    g.listed = b200_list_tiles(flat, g.tiles);
    if (!g.listed) {
      st = b200_alloc(&list, sizeof(int2) * ntiles);
      if (st == B200_OK &&
          cudaMemcpyAsync(list, flat.data(), sizeof(int2) * ntiles, cudaMemcpyHostToDevice, s) !=
              cudaSuccess)
        st = b200_set_error(B200_ECUDA, "dgemm: tile list upload failed");
    }
  }
  // Split-K from the whole call's shape (column panels carry the call's m
  // and n), so panels split their tiles' k ranges as the whole call does.
  const int S = b200_split_for(d->policy_m > 0 ? d->policy_m : d->m,
                               d->policy_n > 0 ? d->policy_n : d->n, ktot, B200_DMMA_TILE,
                               B200_DMMA_TILE, B200_DMMA_BK, {dom.jp, dom.ji, dom.pi},
                               b200_sm_count(), 8.0);  // 128 KB of partials per split unit
  const long sched_tiles = ntiles;
  void *split_ws = nullptr;
  if (st == B200_OK && S > 1 && ntiles > 0) {
    const size_t ints = b200_round_up(sizeof(int) * sched_tiles * 8, 256);
    st = b200_alloc(&split_ws, ints + sizeof(double) * (size_t)sched_tiles * S * 64 * 256);
    if (st == B200_OK && cudaMemsetAsync(split_ws, 0, ints, s) != cudaSuccess)
      st = b200_set_error(B200_ECUDA, "dgemm: split-K counters");
  }
  if (st == B200_OK && ntiles > 0) {
    g.ap = (const double *)ap;
    g.bp = (const double *)bp;
    g.kq = kpad / 4;
    g.c = (double *)d->c;
    g.rs_c = d->rs_c;
    g.cs_c = d->cs_c;
    g.m = d->m;
    g.n = d->n;
    g.k = (int)ktot;
    g.tiles_m = tiles_m;
    g.tiles_n = tiles_n;
    g.tile_list = (const int2 *)list;
    g.ntiles = ntiles;
    g.alpha = d->alpha;
    g.beta = d->beta;
    g.jp = d->product.domain.jp;
    g.ji = d->product.domain.ji;
    g.pi = d->product.domain.pi;
    g.err = b200_device_error_word();
    g.wait_ns = B200_WAIT_NS;
    g.stall = 0;
    if (const unsigned long long limit = b200_take_test_stall()) {
      g.wait_ns = limit;
      g.stall = 1;
    }
    g.splits = S;
    if (S > 1) {
      g.arrivals = (int *)split_ws;
      g.partials = (double *)((char *)split_ws +
                              b200_round_up(sizeof(int) * sched_tiles * 8, 256));
    }
    st = launch_dmma_gemm(g, s);
  }
  b200_free(split_ws);
  b200_free(list);
  b200_free(ap);
  b200_free(bp);
  return st;
}

// One operand of the FP32 kernel: read in place when it is general and
// unmasked, its unit stride runs along m (n), its lines start on 16 bytes and
// it shares no memory with C (SYR2K: and its first pair ends on a k-block);
// else packed into *panel (both pairs as one).
int ffma_operand(const b200_l3_desc_t *d, bool b_side, long len, CUtensorMap (&map)[2], int *kpair,
                 void **panel, cudaStream_t s) {
  const mublis_l3_product_t &pr = d->product;
  const mublis_l3_operand_t &o = b_side ? pr.b : pr.a;
  const int mask = b_side ? (int)pr.domain.jp : (int)pr.domain.pi;
  const void *const *x = b_side ? d->b : d->a;
  const long *rs = b_side ? d->rs_b : d->rs_a, *cs = b_side ? d->cs_b : d->cs_a;
  const int T = B200_FFMA_TILE, BK = B200_FFMA_BK;
  bool direct = direct_on() && o.struc == MUBLIS_STRUC_GENERAL && mask == MUBLIS_L3_ALL &&
                (d->npairs == 1 || d->k % BK == 0);
  for (int t = 0; t < d->npairs && direct; ++t) {
    const long s_mn = b_side ? cs[t] : rs[t], s_k = b_side ? rs[t] : cs[t];
    direct = s_mn == 1 && s_k >= len && s_k % 4 == 0 && ((uintptr_t)x[t] & 15) == 0 &&
             !b200_views_overlap(d->c, d->rs_c, d->cs_c, d->m, d->n, x[t], rs[t], cs[t],
                                 b_side ? d->k : d->m, b_side ? d->n : d->k, 4) &&
             mapped(b200_make_tmap_f32(&map[t], x[t], len, d->k, s_k, T, BK));
  }
  if (direct) {
    if (d->npairs == 2) *kpair = d->k;
    return B200_OK;
  }
  const long pad = b200_round_up(len, T), kpad = b200_round_up((long)d->k * d->npairs, BK);
  B200_TRY(b200_alloc(panel, sizeof(float) * pad * kpad));
  const PackOut out{*panel, pad, 0, PACK_MN_MAJOR, PACK_COPY, 1, nullptr};
  for (int t = 0; t < d->npairs; ++t) {
    const long kk0 = (long)t * d->k, kk1 = t + 1 == d->npairs ? kpad : kk0 + d->k;
    const PackView v{x[t], rs[t], cs[t], (int)o.struc, (int)o.uplo, (int)o.diag, mask};
    B200_TRY(launch_pack<float>(v, b_side, len, d->k, pad, kk0, kk1, out, s));
  }
  return b200_make_tmap_f32(&map[0], *panel, pad, kpad, pad, T, BK);
}

int run_sgemm(const b200_l3_desc_t *d) {
  cudaStream_t s = b200_cur_stream();
  FfmaGemmArgs g;
  void *ap = nullptr, *bp = nullptr;
  int st = ffma_operand(d, false, d->m, g.ta, &g.a_kpair, &ap, s);
  if (st == B200_OK) st = ffma_operand(d, true, d->n, g.tb, &g.b_kpair, &bp, s);
  if (st == B200_OK) {
    g.c = (float *)d->c;
    g.rs_c = d->rs_c;
    g.cs_c = d->cs_c;
    g.m = d->m;
    g.n = d->n;
    g.k = d->k * d->npairs;
    g.alpha = (float)d->alpha;
    g.beta = (float)d->beta;
    g.jp = d->product.domain.jp;
    g.ji = d->product.domain.ji;
    g.pi = d->product.domain.pi;
    const FfmaPolicy pol = {d->policy_m > 0 ? d->policy_m : d->m, d->policy_n > 0 ? d->policy_n : d->n};
    st = launch_ffma_gemm(g, &pol, s);
  }
  b200_free(ap);
  b200_free(bp);
  return st;
}

// FP64 on the FMA pipe (MUBLIS_B200_DGEMM=simt).
int run_simt_dgemm(const b200_l3_desc_t *d) {
  using C = SimtConfig<double>;
  cudaStream_t s = b200_cur_stream();
  const long ktot = (long)d->k * d->npairs;
  const long mpad = b200_round_up(d->m, C::BM), npad = b200_round_up(d->n, C::BN);
  const long kpad = b200_round_up(ktot, C::BK);
  void *ap = nullptr, *bp = nullptr;
  B200_TRY(b200_alloc(&ap, sizeof(double) * mpad * kpad));
  int st = b200_alloc(&bp, sizeof(double) * npad * kpad);
  if (st == B200_OK) {
    PackOut oa{ap, mpad, 0, PACK_MN_MAJOR, PACK_COPY, 1, nullptr};
    PackOut ob{bp, npad, 0, PACK_MN_MAJOR, PACK_COPY, 1, nullptr};
    st = pack_pairs<double>(d, oa, mpad, ob, npad, kpad, s);
  }
  if (st == B200_OK) {
    SimtGemmArgs<double> g;
    g.ap = (const double *)ap;
    g.bp = (const double *)bp;
    g.lda = mpad;
    g.ldb = npad;
    g.c = (double *)d->c;
    g.rs_c = d->rs_c;
    g.cs_c = d->cs_c;
    g.m = d->m;
    g.n = d->n;
    g.k = (int)ktot;
    g.alpha = d->alpha;
    g.beta = d->beta;
    g.jp = d->product.domain.jp;
    g.ji = d->product.domain.ji;
    g.pi = d->product.domain.pi;
    const SimtPolicy pol = {d->policy_m > 0 ? d->policy_m : d->m,
                            d->policy_n > 0 ? d->policy_n : d->n};
    st = launch_simt_gemm<double>(g, s, &pol);
  }
  b200_free(ap);
  b200_free(bp);
  return st;
}

// A small product in one launch (gemm_direct.cu), or 0 when the call is not
// one.  An in-place product (TRMM, a solve's diagonal products: C is the
// operand itself) reads a compact copy of that operand.
int try_direct(const b200_l3_desc_t *d, int *status) {
  // A stall armed by mublis_b200_test_stall_next waits for the FP64
  // tensor-pipe kernel of the packed path.
  if (!small_on() || (d->dtype == B200_F64 && (!use_dmma() || b200_test_stall_armed()))) return 0;
  const mublis_l3_product_t &pr = d->product;
  if (d->npairs == 2 &&
      (pr.a.struc != MUBLIS_STRUC_GENERAL || pr.b.struc != MUBLIS_STRUC_GENERAL ||
       pr.domain.jp != MUBLIS_L3_ALL || pr.domain.pi != MUBLIS_L3_ALL))
    return 0;
  const b200_direct_choice_t ch = b200_direct_choice(d);
  if (!ch.tile) return 0;
  if (!overlaps_operand(d)) {
    *status = launch_direct_gemm(d, ch);
    return 1;
  }
  const bool is_b = d->b[0] == d->c && d->rs_b[0] == d->rs_c && d->cs_b[0] == d->cs_c && d->k == d->m;
  const bool is_a = d->a[0] == d->c && d->rs_a[0] == d->rs_c && d->cs_a[0] == d->cs_c && d->k == d->n;
  const bool rows = d->rs_c == 1 && d->cs_c >= d->m, cols = d->cs_c == 1 && d->rs_c >= d->n;
  if (d->npairs != 1 || is_a == is_b || (!rows && !cols)) return 0;
  const size_t elt = d->dtype == B200_F64 ? 8 : 4;
  const long w = rows ? d->m : d->n, h = rows ? d->n : d->m;
  const long ld = b200_round_up(w, (long)(16 / elt));
  b200_l3_desc_t e = *d;
  (is_b ? e.rs_b : e.rs_a)[0] = rows ? 1 : ld;
  (is_b ? e.cs_b : e.cs_a)[0] = rows ? ld : 1;
  if (b200_views_overlap(e.c, e.rs_c, e.cs_c, e.m, e.n, is_b ? e.a[0] : e.b[0], is_b ? e.rs_a[0] : e.rs_b[0],
                    is_b ? e.cs_a[0] : e.cs_b[0], is_b ? e.m : e.k, is_b ? e.k : e.n, (long)elt))
    return 0;
  void *copy = nullptr;
  *status = b200_alloc(&copy, elt * ld * h);
  if (*status != B200_OK) return 1;
  (is_b ? e.b : e.a)[0] = copy;
  if (cudaMemcpy2DAsync(copy, ld * elt, d->c, (rows ? d->cs_c : d->rs_c) * elt, w * elt, h,
                        cudaMemcpyDeviceToDevice, b200_cur_stream()) != cudaSuccess)
    *status = b200_set_error(B200_ECUDA, "direct gemm: operand copy failed");
  else
    *status = launch_direct_gemm(&e, ch);
  b200_free(copy);
  return 1;
}

}  // namespace

extern "C" int b200_scale_strided(int dtype, int m, int n, double beta, void *c, long rs, long cs,
                                  mublis_l3_relation_t ji) {
  cudaStream_t s = b200_cur_stream();
  if (dtype == B200_F32) return launch_scale<float>(m, n, (float)beta, (float *)c, rs, cs, ji, s);
  return launch_scale<double>(m, n, beta, (double *)c, rs, cs, ji, s);
}

extern "C" int b200_l3_run(const b200_l3_desc_t *d) {
  if (d->m <= 0 || d->n <= 0) return B200_OK;
  if (d->npairs < 1 || d->npairs > 2) return b200_set_error(B200_EINVAL, "l3: npairs");
  // alpha == 0 (or no k): beta-scale the written part only, never touching
  // A or B (l3_driver.c:104,123).
  if (d->alpha == 0.0 || d->k <= 0)
    return b200_scale_strided(d->dtype, d->m, d->n, d->beta, d->c, d->rs_c, d->cs_c,
                              d->product.domain.ji);
  const int form = resolve_form(d);
  if (form == B200_FORM_BF16X3 || form == B200_FORM_BF16X6 || form == B200_FORM_FP16X3)
    return tc_run_bf16(d, form);
  if (form == B200_FORM_OZAKI || form == B200_FORM_OZAKI2) {
    b200_l3_desc_t e = *d;
    e.form = form;
    if (d->form == B200_FORM_POLICY || (d->form == B200_FORM_AUTO &&
                                        b200_get_default_form(d->dtype) == B200_FORM_POLICY))
      e.slices = form == B200_FORM_OZAKI ? 8 : 0;  // 0: the form's default count
    // "ozaki2@<target>": the modulus count measured for the target error
    // (cached per precision, k bucket and target).
    const double target = b200_get_default_target(d->dtype);
    if (form == B200_FORM_OZAKI2 && d->form == B200_FORM_AUTO && target > 0 && d->slices == 0 &&
        b200_get_default_form(d->dtype) == B200_FORM_OZAKI2 &&
        b200_get_default_slices(d->dtype) == 0)
      B200_TRY(b200_ozaki2_choice(&e, target, &e.slices, nullptr, 0));
    return tc_run_ozaki(&e);
  }
  int st;
  if (try_direct(d, &st)) return st;
  if (d->dtype == B200_F32) return run_sgemm(d);
  return use_dmma() ? run_dmma(d) : run_simt_dgemm(d);
}
