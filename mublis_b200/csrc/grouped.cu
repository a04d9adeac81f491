// grouped.cu -- many independent GEMMs / left TRSMs of uneven sizes in one
// launch per tile shape or order class, plus the plan object that autotunes the tile shape
// and captures the launches in a CUDA graph for replay.
//
// The reference has no batched interface: every call runs the full driver
// (frame/l3/l3_driver.c) on one host thread.  For many small calls the B200
// cost is launch latency and packing passes, not flops, so the grouped path
// (a) reads operands directly from caller memory with bounds checks (no
// pack pass), (b) maps every output tile of every problem into one global
// tile index space (prefix sums over per-problem tile counts), a CTA of the
// direct kernel (gemm_direct.cu) to a tile, and (c) solves each TRSM instance
// in slabs of 32 right-hand sides, a CTA of trsm_small.cu to a slab.
#include <algorithm>
#include <cstring>
#include <cstdio>
#include <cstdlib>
#include <mutex>
#include <string>
#include <type_traits>
#include <vector>

#include "kernels.cuh"
#include "../../include/mublis_b200.h"
#include "tc_gemm.cuh"

namespace {

using GemmEntry = b200_group_gemm_t;

using TrsmEntry = b200_small_trsm_t;
constexpr int TRSM_MAX_ORDER = B200_TRSM_SMALL;
constexpr int TRSM_SLAB = B200_TRSM_SMALL_COLS;

// ---- host side ------------------------------------------------------------------

// Tiles of the group kernel (gemm_direct.cu).
enum { TILE_32 = 0, TILE_64 = 1, TILE_VARIANTS = 2 };
const int kTile[TILE_VARIANTS] = {32, 64};

int sm_count() { return b200_sm_count(); }

template <typename T>
int launch_gemm_variant(int variant, const GemmEntry *dtable, int nprob, int tiles, cudaStream_t s) {
  return launch_direct_group(sizeof(T) == 8 ? B200_F64 : B200_F32, kTile[variant], dtable,
                             (const int *)(dtable + nprob), tiles, s);
}

// Size classes the autotuner chooses a tile shape for (by max(m, n)).
int size_class(long m, long n) {
  long x = std::max(m, n);
  return x <= 48 ? 0 : (x <= 160 ? 1 : 2);
}
constexpr int NCLASS = 3;

struct GemmGroup {
  std::vector<GemmEntry> entries;  // host copy, tile0/tiles_m filled for `variant`
  GemmEntry *dtable = nullptr;     // entries, then the tile -> problem map
  size_t bytes = 0;                // allocated at dtable
  int tiles = 0;
  int variant = TILE_64;
};

// Host image of a class's device table for tile variant v: the entries
// (tile0 / tiles_m filled) followed by one int per output tile, the index
// of the tile's problem, so that a CTA finds its tile's problem with one
// load (a binary search over tile0 was a chain of ~12 dependent loads per
// tile).
std::vector<char> table_image(std::vector<GemmEntry> &es, int v, int &tiles) {
  int t = 0;
  for (auto &e : es) {
    e.tile0 = t;
    e.tiles_m = (int)b200_ceil_div(e.m, kTile[v]);
    t += e.tiles_m * (int)b200_ceil_div(e.n, kTile[v]);
  }
  tiles = t;
  const size_t head = sizeof(GemmEntry) * es.size();
  std::vector<char> img(head + sizeof(int) * (size_t)t);
  if (!es.empty()) memcpy(img.data(), es.data(), head);
  int *map = reinterpret_cast<int *>(img.data() + head);
  for (size_t q = 0; q < es.size(); ++q) {
    const int end = q + 1 < es.size() ? es[q + 1].tile0 : t;
    for (int x = es[q].tile0; x < end; ++x) map[x] = (int)q;
  }
  return img;
}

// Builds the device table of one class for a tile variant.
int build_group(std::vector<GemmEntry> &src, int variant, GemmGroup &g, cudaStream_t s) {
  g.entries = src;
  g.variant = variant;
  const std::vector<char> img = table_image(g.entries, variant, g.tiles);
  if (g.entries.empty()) return B200_OK;
  if (img.size() > g.bytes) {  // stream-ordered: earlier launches keep the old table
    b200_free(g.dtable);
    g.dtable = nullptr;
    g.bytes = 0;
    B200_TRY(b200_alloc((void **)&g.dtable, img.size()));
    g.bytes = img.size();
  }
  B200_CUDA_TRY(cudaMemcpyAsync(g.dtable, img.data(), img.size(), cudaMemcpyHostToDevice, s));
  return B200_OK;
}

int to_entries(char dtype, const mublis_b200_gemm_problem_t *p, int count,
               std::vector<GemmEntry> (&cls)[NCLASS]) {
  B200DevicePtrs ptrs;
  for (int q = 0; q < count; ++q) {
    const mublis_b200_gemm_problem_t &x = p[q];
    if (x.m < 0 || x.n < 0 || x.k < 0) return b200_set_error(B200_EINVAL, "grouped gemm: negative size");
    if (x.m == 0 || x.n == 0) continue;
    if (x.ldc < std::max(1, x.m)) return b200_set_error(B200_EINVAL, "grouped gemm: ldc too small");
    const bool upd = x.alpha != 0.0 && x.k > 0;
    if (!ptrs.device(x.c) || (upd && (!ptrs.device(x.a) || !ptrs.device(x.b))))
      return b200_set_error(B200_EINVAL, "grouped gemm: operands must be device pointers");
    GemmEntry e;
    memset(&e, 0, sizeof e);
    e.m = x.m;
    e.n = x.n;
    e.k = upd ? x.k : 0;  // alpha == 0: beta * C only, A and B never read
    e.alpha = x.alpha;
    e.beta = x.beta;
    e.a = x.a;
    e.b = x.b;
    e.rs_a = x.trans_a == MUBLIS_TRANSPOSE ? x.lda : 1;
    e.cs_a = x.trans_a == MUBLIS_TRANSPOSE ? 1 : x.lda;
    e.rs_b = x.trans_b == MUBLIS_TRANSPOSE ? x.ldb : 1;
    e.cs_b = x.trans_b == MUBLIS_TRANSPOSE ? 1 : x.ldb;
    e.c = x.c;
    e.rs_c = 1;
    e.cs_c = x.ldc;
    e.vec = b200_group_vec(e, dtype == 'd' ? 8 : 4);
    cls[size_class(x.m, x.n)].push_back(e);
  }
  return B200_OK;
}

// Default tile per class, used until the autotuner has timed the classes.
const int kDefaultVariant[NCLASS] = {TILE_32, TILE_64, TILE_64};

template <typename T>
int run_groups(GemmGroup (&g)[NCLASS], cudaStream_t s) {
  for (int c = 0; c < NCLASS; ++c)
    if (g[c].tiles) B200_TRY(launch_gemm_variant<T>(g[c].variant, g[c].dtable, (int)g[c].entries.size(), g[c].tiles, s));
  return B200_OK;
}

// Autotuner: for each non-empty class time every tile variant on the
// class's actual problems (CUDA events, best of 2 after a warm-up) and keep
// the fastest.  Results are cached per (dtype, class, problem-count bucket)
// for the process.
std::mutex g_tune_mu;
int g_tuned[2][NCLASS][32];  // 0 = untuned, else variant + 1

// ---- tuned-table persistence ---------------------------------------------
//
// Text file: one key line, then one line per choice,
//   mublis_b200-tune <gpu name> sms=<n> cc=<major>.<minor> driver=<v> table=1
//   gemm <fp64 0/1> <size class> <count bucket> <tile variant>
// The key ties the file to a GPU model and driver (tile timings change with
// either); table=1 names this library's classes and variants.

constexpr int kTuneTable = 1;

std::string tune_key() {
  int dev = 0, drv = 0;
  cudaGetDevice(&dev);
  cudaDeviceProp prop;
  if (cudaGetDeviceProperties(&prop, dev) != cudaSuccess) return std::string();
  cudaDriverGetVersion(&drv);
  std::string name(prop.name);
  for (char &ch : name)
    if (ch == ' ' || ch == '\t') ch = '_';
  char buf[512];
  snprintf(buf, sizeof buf, "mublis_b200-tune %s sms=%d cc=%d.%d driver=%d table=%d",
           name.c_str(), prop.multiProcessorCount, prop.major, prop.minor, drv, kTuneTable);
  return buf;
}

int tune_save(const char *path) {
  if (!path || !*path) return b200_set_error(B200_EINVAL, "tune: empty path");
  const std::string key = tune_key();
  if (key.empty()) return b200_set_error(B200_ECUDA, "tune: no device to key the table to");
  std::string text = key + "\n";
  {
    std::lock_guard<std::mutex> lk(g_tune_mu);
    for (int dt = 0; dt < 2; ++dt)
      for (int c = 0; c < NCLASS; ++c)
        for (int b = 0; b < 32; ++b)
          if (g_tuned[dt][c][b]) {
            char line[64];
            snprintf(line, sizeof line, "gemm %d %d %d %d\n", dt, c, b, g_tuned[dt][c][b] - 1);
            text += line;
          }
  }
  b200_ozaki2_table_lines(&text);
  const std::string tmp = std::string(path) + ".tmp";
  FILE *f = fopen(tmp.c_str(), "w");
  if (!f) return b200_set_error(B200_EINVAL, "tune: cannot write the table file");
  const bool ok = fwrite(text.data(), 1, text.size(), f) == text.size();
  if (fclose(f) != 0 || !ok || rename(tmp.c_str(), path) != 0) {
    remove(tmp.c_str());
    return b200_set_error(B200_EINVAL, "tune: cannot write the table file");
  }
  return B200_OK;
}

int tune_load(const char *path, int *entries) {
  if (entries) *entries = 0;
  if (!path || !*path) return b200_set_error(B200_EINVAL, "tune: empty path");
  FILE *f = fopen(path, "r");
  if (!f) return B200_OK;  // no table yet
  const std::string key = tune_key();
  char line[512];
  int loaded = 0;
  if (!key.empty() && fgets(line, sizeof line, f)) {
    line[strcspn(line, "\r\n")] = 0;
    if (key == line) {
      while (fgets(line, sizeof line, f)) {
        if (!strncmp(line, "ozaki2 ", 7)) {
          if (b200_ozaki2_table_parse(line)) ++loaded;
          continue;
        }
        int dt, c, b, v;
        if (sscanf(line, "gemm %d %d %d %d", &dt, &c, &b, &v) != 4) continue;
        // (Variants 2 and 3 of older files named larger tiles.)
        if (dt < 0 || dt > 1 || c < 0 || c >= NCLASS || b < 0 || b >= 32 || v < 0 || v > 3) continue;
        v = std::min(v, TILE_VARIANTS - 1);
        std::lock_guard<std::mutex> lk(g_tune_mu);
        g_tuned[dt][c][b] = v + 1;
        ++loaded;
      }
    }
  }
  fclose(f);
  if (entries) *entries = loaded;
  return B200_OK;
}

const char *tune_env_path() {
  const char *p = getenv("MUBLIS_B200_TUNE_FILE");
  return p && *p ? p : nullptr;
}

void b200_tune_autosave() {
  if (const char *p = tune_env_path()) tune_save(p);  // best effort: tuning goes on regardless
}

template <typename T>
int autotune(std::vector<GemmEntry> (&cls)[NCLASS], GemmGroup (&g)[NCLASS], cudaStream_t s) {
  const int dt = sizeof(T) == 8;
  cudaEvent_t e0, e1;
  B200_CUDA_TRY(cudaEventCreate(&e0));
  B200_CUDA_TRY(cudaEventCreate(&e1));
  for (int c = 0; c < NCLASS; ++c) {
    if (cls[c].empty()) continue;
    int bucket = 31 - __builtin_clz((unsigned)cls[c].size());
    {
      std::lock_guard<std::mutex> lk(g_tune_mu);
      if (g_tuned[dt][c][bucket]) {
        B200_TRY(build_group(cls[c], g_tuned[dt][c][bucket] - 1, g[c], s));
        continue;
      }
    }
    float best = 1e30f;
    int best_v = kDefaultVariant[c];
    for (int v = 0; v < TILE_VARIANTS; ++v) {
      B200_TRY(build_group(cls[c], v, g[c], s));
      float ms_best = 1e30f;
      for (int rep = 0; rep < 3; ++rep) {
        B200_CUDA_TRY(cudaEventRecord(e0, s));
        B200_TRY(launch_gemm_variant<T>(v, g[c].dtable, (int)g[c].entries.size(), g[c].tiles, s));
        B200_CUDA_TRY(cudaEventRecord(e1, s));
        B200_CUDA_TRY(cudaEventSynchronize(e1));
        float ms = 0;
        cudaEventElapsedTime(&ms, e0, e1);
        if (rep > 0) ms_best = std::min(ms_best, ms);
      }
      if (ms_best < best) { best = ms_best; best_v = v; }
    }
    B200_TRY(build_group(cls[c], best_v, g[c], s));
    {
      std::lock_guard<std::mutex> lk(g_tune_mu);
      g_tuned[dt][c][bucket] = best_v + 1;
    }
    b200_tune_autosave();
  }
  cudaEventDestroy(e0);
  cudaEventDestroy(e1);
  return B200_OK;
}

// Note: the autotuner's trial launches write C (they are real executions of
// the grouped product); a plan therefore snapshots and restores every C
// before tuning.  See plan_gemm below.

struct TrsmGroup {
  std::vector<TrsmEntry> entries;
  TrsmEntry *dtable = nullptr;  // entries, then the slab -> problem map
  int slabs = 0;
  std::vector<int> fallback;  // problems too large for the one-CTA solve
};

// Host image of a TRSM group's device table: the entries followed by one
// int per 32-column slab, the index of the slab's problem.
std::vector<char> trsm_table_image(const TrsmGroup &g) {
  const size_t head = sizeof(TrsmEntry) * g.entries.size();
  std::vector<char> img(head + sizeof(int) * (size_t)g.slabs);
  if (!g.entries.empty()) memcpy(img.data(), g.entries.data(), head);
  int *map = reinterpret_cast<int *>(img.data() + head);
  for (size_t q = 0; q < g.entries.size(); ++q) {
    const int end = q + 1 < g.entries.size() ? g.entries[q + 1].slab0 : g.slabs;
    for (int x = g.entries[q].slab0; x < end; ++x) map[x] = (int)q;
  }
  return img;
}

// The group's entries by order (up to B200_TRSM_SMALL_HALF first: two launches),
// and their slabs.
void order_slabs(TrsmGroup &g) {
  std::stable_partition(g.entries.begin(), g.entries.end(),
                        [](const TrsmEntry &e) { return e.m <= B200_TRSM_SMALL_HALF; });
  g.slabs = 0;
  for (auto &e : g.entries) {
    e.slab0 = g.slabs;
    g.slabs += (int)b200_ceil_div(e.n, TRSM_SLAB);
  }
}

int to_trsm(const mublis_b200_trsm_problem_t *p, int count, TrsmGroup &g, cudaStream_t s) {
  B200DevicePtrs ptrs;
  for (int q = 0; q < count; ++q) {
    const mublis_b200_trsm_problem_t &x = p[q];
    if (x.m < 0 || x.n < 0) return b200_set_error(B200_EINVAL, "grouped trsm: negative size");
    if (x.m == 0 || x.n == 0) continue;
    if (x.uplo != MUBLIS_LOWER && x.uplo != MUBLIS_UPPER)
      return b200_set_error(B200_EINVAL, "grouped trsm: uplo must be lower or upper");
    if (!ptrs.device(x.b) || (x.alpha != 0.0 && !ptrs.device(x.a)))
      return b200_set_error(B200_EINVAL, "grouped trsm: operands must be device pointers");
    if (x.m > TRSM_MAX_ORDER || x.alpha == 0.0) {
      g.fallback.push_back(q);
      continue;
    }
    TrsmEntry e;
    memset(&e, 0, sizeof e);
    e.m = x.m;
    e.n = x.n;
    e.alpha = x.alpha;
    e.a = x.a;
    // trans folds into strides and flips the triangle (frame/l3/trsm.c:49-54)
    const bool tr = x.trans_a == MUBLIS_TRANSPOSE;
    e.rs_a = tr ? x.lda : 1;
    e.cs_a = tr ? 1 : x.lda;
    e.lower = (x.uplo == MUBLIS_LOWER) != tr;
    e.unit = x.diag == MUBLIS_UNIT_DIAG;
    e.b = x.b;
    e.rs_b = 1;
    e.cs_b = x.ldb;
    g.entries.push_back(e);
  }
  order_slabs(g);
  if (g.entries.empty()) return B200_OK;
  const std::vector<char> img = trsm_table_image(g);
  B200_TRY(b200_alloc((void **)&g.dtable, img.size()));
  B200_CUDA_TRY(cudaMemcpyAsync(g.dtable, img.data(), img.size(), cudaMemcpyHostToDevice, s));
  return B200_OK;
}

int launch_trsm_group(int dtype, const TrsmGroup &g, cudaStream_t s) {
  int order[2] = {0, 0}, slabs[2] = {0, 0};
  for (const auto &e : g.entries) {
    const int big = e.m > B200_TRSM_SMALL_HALF;
    order[big] = std::max(order[big], e.m);
    slabs[big] += (int)b200_ceil_div(e.n, TRSM_SLAB);
  }
  const int *slab_prob = (const int *)(g.dtable + g.entries.size());
  for (int big = 0; big < 2; ++big)
    if (slabs[big])
      B200_TRY(launch_small_trsm(dtype, g.dtable, slab_prob, big ? slabs[0] : 0, slabs[big], order[big], s));
  return B200_OK;
}

int trsm_fallback(char dtype, const mublis_b200_trsm_problem_t *p, const std::vector<int> &idx) {
  for (int q : idx) {
    const mublis_b200_trsm_problem_t &x = p[q];
    int st = dtype == 'd'
                 ? mublis_dtrsm(MUBLIS_LEFT, (mublis_uplo_t)x.uplo, (mublis_trans_t)x.trans_a,
                                (mublis_diag_t)x.diag, x.m, x.n, x.alpha, (const double *)x.a, 1,
                                x.lda, (double *)x.b, 1, x.ldb)
                 : mublis_strsm(MUBLIS_LEFT, (mublis_uplo_t)x.uplo, (mublis_trans_t)x.trans_a,
                                (mublis_diag_t)x.diag, x.m, x.n, (float)x.alpha, (const float *)x.a,
                                1, x.lda, (float *)x.b, 1, x.ldb);
    if (st) return st;
  }
  return B200_OK;
}

}  // namespace

// ---- plans ------------------------------------------------------------------------

struct mublis_b200_plan {
  char dtype = 's';
  int kind = 0;  // 0 gemm, 1 trsm
  GemmGroup gg[NCLASS];
  TrsmGroup tg;
  b200_tcg *tcg = nullptr;  // FP32 GEMMs in the fp16x3 form
  std::vector<mublis_b200_trsm_problem_t> trsm_problems;
  cudaGraph_t graph = nullptr;
  cudaGraphExec_t exec = nullptr;
};

namespace {

template <typename T>
int plan_gemm(mublis_b200_plan *pl, const mublis_b200_gemm_problem_t *p, int count) {
  cudaStream_t s = b200_cur_stream();
  std::vector<GemmEntry> cls[NCLASS];
  B200_TRY(to_entries(pl->dtype, p, count, cls));
  // Longest products first: a launch ends with its short ones.
  for (auto &c : cls)
    std::stable_sort(c.begin(), c.end(), [](const GemmEntry &x, const GemmEntry &y) { return x.k > y.k; });
  // The tuner's trials are real executions; keep every C and put it back.
  std::vector<void *> saved(count, nullptr);
  for (int q = 0; q < count; ++q) {
    if (p[q].m == 0 || p[q].n == 0) continue;
    size_t bytes = (size_t)p[q].ldc * (p[q].n - 1) * sizeof(T) + (size_t)p[q].m * sizeof(T);
    B200_TRY(b200_alloc(&saved[q], bytes));
    B200_CUDA_TRY(cudaMemcpyAsync(saved[q], p[q].c, bytes, cudaMemcpyDeviceToDevice, s));
  }
  int st = autotune<T>(cls, pl->gg, s);
  for (int q = 0; q < count; ++q) {
    if (!saved[q]) continue;
    size_t bytes = (size_t)p[q].ldc * (p[q].n - 1) * sizeof(T) + (size_t)p[q].m * sizeof(T);
    if (cudaMemcpyAsync(p[q].c, saved[q], bytes, cudaMemcpyDeviceToDevice, s) != cudaSuccess)
      st = b200_set_error(B200_ECUDA, "plan: restoring C failed");
    b200_free(saved[q]);
  }
  return st;
}

// FP32 groups run in the fp16x3 tensor-core form (tc_grouped.cu) when that
// is the FP32 form; every other form runs the plain grouped kernel.
bool tc_grouped(char dtype) {
  return dtype == 's' && b200_get_default_form(B200_F32) == B200_FORM_FP16X3;
}

// Sets up the kernels a plan launches: a capture fails when one of its launches
// is the process's first (loading code and taking host memory are not allowed
// then), and a plan whose tiles come from a table, or that has no trial runs,
// may be just that.
int setup(mublis_b200_plan *pl) {
  if (pl->tcg) return b200_tcg_setup();
  if (pl->kind == 1) {
    const int dt = pl->dtype == 'd' ? B200_F64 : B200_F32;
    B200_TRY(launch_small_trsm(dt, nullptr, nullptr, 0, 0, 1, nullptr));
    return launch_small_trsm(dt, nullptr, nullptr, 0, 0, B200_TRSM_SMALL, nullptr);
  }
  for (const auto &g : pl->gg)
    if (g.tiles)
      B200_TRY(pl->dtype == 'd' ? launch_gemm_variant<double>(g.variant, nullptr, 0, 0, nullptr)
                                : launch_gemm_variant<float>(g.variant, nullptr, 0, 0, nullptr));
  return B200_OK;
}

int capture(mublis_b200_plan *pl) {
  cudaStream_t s = b200_cur_stream();
  B200_TRY(setup(pl));
  B200_TRY(b200_stream_sync());
  B200_CUDA_TRY(cudaStreamBeginCapture(s, cudaStreamCaptureModeThreadLocal));
  int st;
  if (pl->tcg)
    st = b200_tcg_run(pl->tcg, s);
  else if (pl->kind == 0)
    st = pl->dtype == 'd' ? run_groups<double>(pl->gg, s) : run_groups<float>(pl->gg, s);
  else
    st = launch_trsm_group(pl->dtype == 'd' ? B200_F64 : B200_F32, pl->tg, s);
  cudaError_t e = cudaStreamEndCapture(s, &pl->graph);
  if (st != B200_OK) return st;
  B200_CUDA_TRY(e);
  B200_CUDA_TRY(cudaGraphInstantiate(&pl->exec, pl->graph, 0));
  return B200_OK;
}

}  // namespace

// ---- descriptor-based asynchronous entry points (the request server) --------

extern "C" int b200_l3_is_plain_gemm(const b200_l3_desc_t *d) {
  const mublis_l3_product_t &p = d->product;
  return d->npairs == 1 && p.domain.jp == MUBLIS_L3_ALL && p.domain.ji == MUBLIS_L3_ALL &&
         p.domain.pi == MUBLIS_L3_ALL && p.a.struc == MUBLIS_STRUC_GENERAL &&
         p.b.struc == MUBLIS_STRUC_GENERAL;
}

// Without a tuned choice: the class's default tile, or the small one when the
// group would leave more than half of the SMs without a tile.
int fill_variant(const std::vector<GemmEntry> &es, int v) {
  long tiles = 0;
  for (const auto &e : es) tiles += b200_ceil_div(e.m, kTile[v]) * b200_ceil_div(e.n, kTile[v]);
  return 2 * tiles < sm_count() ? TILE_32 : v;
}

extern "C" int b200_grouped_gemm_async(int dtype, const b200_l3_desc_t *const *descs, int count,
                                       void *stream) {
  cudaStream_t s = (cudaStream_t)stream;
  std::vector<GemmEntry> cls[NCLASS];
  for (int q = 0; q < count; ++q) {
    const b200_l3_desc_t &d = *descs[q];
    if (d.m <= 0 || d.n <= 0) continue;
    if (!b200_l3_is_plain_gemm(&d) || d.dtype != dtype)
      return b200_set_error(B200_EINVAL, "grouped: not a plain GEMM of this precision");
    GemmEntry e;
    memset(&e, 0, sizeof e);
    e.m = d.m;
    e.n = d.n;
    e.k = d.alpha != 0.0 ? d.k : 0;
    e.alpha = d.alpha;
    e.beta = d.beta;
    e.a = d.a[0];
    e.rs_a = d.rs_a[0];
    e.cs_a = d.cs_a[0];
    e.b = d.b[0];
    e.rs_b = d.rs_b[0];
    e.cs_b = d.cs_b[0];
    e.c = d.c;
    e.rs_c = d.rs_c;
    e.cs_c = d.cs_c;
    e.vec = b200_group_vec(e, dtype == B200_F64 ? 8 : 4);
    cls[size_class(d.m, d.n)].push_back(e);
  }
  GemmGroup g[NCLASS];
  int st = B200_OK;
  for (int c = 0; c < NCLASS && st == B200_OK; ++c) {
    if (cls[c].empty()) continue;
    int bucket = 31 - __builtin_clz((unsigned)cls[c].size());
    int v;
    bool tuned;
    {
      std::lock_guard<std::mutex> lk(g_tune_mu);
      tuned = g_tuned[dtype == B200_F64][c][bucket] != 0;
      v = tuned ? g_tuned[dtype == B200_F64][c][bucket] - 1 : kDefaultVariant[c];
    }
    if (!tuned) v = fill_variant(cls[c], v);
    g[c].entries = cls[c];
    g[c].variant = v;
    const std::vector<char> img = table_image(g[c].entries, v, g[c].tiles);
    if (cudaMallocAsync((void **)&g[c].dtable, img.size(), s) != cudaSuccess ||
        cudaMemcpyAsync(g[c].dtable, img.data(), img.size(), cudaMemcpyHostToDevice, s) !=
            cudaSuccess)
      st = b200_set_error(B200_ECUDA, "grouped: table upload failed");
  }
  if (st == B200_OK)
    st = dtype == B200_F64 ? run_groups<double>(g, s) : run_groups<float>(g, s);
  for (auto &x : g)
    if (x.dtable) cudaFreeAsync(x.dtable, s);
  return st;
}

extern "C" int b200_grouped_trsm_async(int dtype, const b200_trsm_desc_t *const *descs, int count,
                                       void *stream) {
  cudaStream_t s = (cudaStream_t)stream;
  TrsmGroup g;
  for (int q = 0; q < count; ++q) {
    const b200_trsm_desc_t &d = *descs[q];
    if (d.m <= 0 || d.n <= 0) continue;
    if (d.m > TRSM_MAX_ORDER || d.dtype != dtype || d.alpha == 0.0)
      return b200_set_error(B200_EINVAL, "grouped: TRSM not batchable");
    TrsmEntry e;
    memset(&e, 0, sizeof e);
    e.m = d.m;
    e.n = d.n;
    e.alpha = d.alpha;
    e.a = d.a;
    e.rs_a = d.rs_a;
    e.cs_a = d.cs_a;
    e.lower = d.uplo == MUBLIS_LOWER;
    e.unit = d.unit_diag != 0;
    e.b = d.b;
    e.rs_b = d.rs_b;
    e.cs_b = d.cs_b;
    g.entries.push_back(e);
  }
  order_slabs(g);
  if (g.entries.empty()) return B200_OK;
  const std::vector<char> img = trsm_table_image(g);
  if (cudaMallocAsync((void **)&g.dtable, img.size(), s) != cudaSuccess ||
      cudaMemcpyAsync(g.dtable, img.data(), img.size(), cudaMemcpyHostToDevice, s) != cudaSuccess)
    return b200_set_error(B200_ECUDA, "grouped: table upload failed");
  int st = launch_trsm_group(dtype, g, s);
  cudaFreeAsync(g.dtable, s);
  return st;
}

extern "C" {

int mublis_b200_gemm_grouped(char dtype, const mublis_b200_gemm_problem_t *problems, int count) {
  if (count < 0 || (count > 0 && !problems)) return b200_set_error(B200_EINVAL, "grouped gemm: bad arguments");
  if (dtype != 's' && dtype != 'd') return b200_set_error(B200_EINVAL, "grouped gemm: dtype is 's' or 'd'");
  if (count == 0) return B200_OK;
  B200_TRY(b200_init());
  cudaStream_t s = b200_cur_stream();
  if (tc_grouped(dtype)) {
    b200_tcg *g = nullptr;
    B200_TRY(b200_tcg_create(problems, count, &g));
    int st = b200_tcg_run(g, s);
    if (st == B200_OK) st = b200_stream_sync();
    b200_tcg_destroy(g);
    return st == B200_OK ? b200_stream_sync() : st;
  }
  std::vector<GemmEntry> cls[NCLASS];
  B200_TRY(to_entries(dtype, problems, count, cls));
  GemmGroup g[NCLASS];
  int st = B200_OK;
  for (int c = 0; c < NCLASS && st == B200_OK; ++c) {
    int bucket = cls[c].empty() ? 0 : 31 - __builtin_clz((unsigned)cls[c].size());
    int v;
    {
      std::lock_guard<std::mutex> lk(g_tune_mu);
      v = g_tuned[dtype == 'd'][c][bucket] ? g_tuned[dtype == 'd'][c][bucket] - 1 : kDefaultVariant[c];
    }
    st = build_group(cls[c], v, g[c], s);
  }
  if (st == B200_OK) st = dtype == 'd' ? run_groups<double>(g, s) : run_groups<float>(g, s);
  if (st == B200_OK) st = b200_stream_sync();
  for (auto &x : g) b200_free(x.dtable);
  return st == B200_OK ? b200_stream_sync() : st;
}

int mublis_b200_trsm_grouped(char dtype, const mublis_b200_trsm_problem_t *problems, int count) {
  if (count < 0 || (count > 0 && !problems)) return b200_set_error(B200_EINVAL, "grouped trsm: bad arguments");
  if (dtype != 's' && dtype != 'd') return b200_set_error(B200_EINVAL, "grouped trsm: dtype is 's' or 'd'");
  if (count == 0) return B200_OK;
  B200_TRY(b200_init());
  cudaStream_t s = b200_cur_stream();
  TrsmGroup g;
  int st = to_trsm(problems, count, g, s);
  if (st == B200_OK) st = launch_trsm_group(dtype == 'd' ? B200_F64 : B200_F32, g, s);
  if (st == B200_OK) st = b200_stream_sync();
  b200_free(g.dtable);
  if (st == B200_OK) st = b200_stream_sync();
  if (st == B200_OK) st = trsm_fallback(dtype, problems, g.fallback);
  return st;
}

int mublis_b200_plan_gemm_grouped(char dtype, const mublis_b200_gemm_problem_t *problems,
                                  int count, mublis_b200_plan_t **plan) {
  if (!plan || count < 0 || (count > 0 && !problems) || (dtype != 's' && dtype != 'd'))
    return b200_set_error(B200_EINVAL, "plan: bad arguments");
  *plan = nullptr;
  B200_TRY(b200_init());
  auto *pl = new mublis_b200_plan;
  pl->dtype = dtype;
  pl->kind = 0;
  int st = tc_grouped(dtype) ? b200_tcg_create(problems, count, &pl->tcg)
           : dtype == 'd'    ? plan_gemm<double>(pl, problems, count)
                             : plan_gemm<float>(pl, problems, count);
  if (st == B200_OK) st = capture(pl);
  if (st != B200_OK) {
    mublis_b200_plan_destroy(pl);
    return st;
  }
  *plan = pl;
  return b200_stream_sync();
}

int mublis_b200_plan_trsm_grouped(char dtype, const mublis_b200_trsm_problem_t *problems,
                                  int count, mublis_b200_plan_t **plan) {
  if (!plan || count < 0 || (count > 0 && !problems) || (dtype != 's' && dtype != 'd'))
    return b200_set_error(B200_EINVAL, "plan: bad arguments");
  *plan = nullptr;
  B200_TRY(b200_init());
  auto *pl = new mublis_b200_plan;
  pl->dtype = dtype;
  pl->kind = 1;
  int st = to_trsm(problems, count, pl->tg, b200_cur_stream());
  if (st == B200_OK && !pl->tg.fallback.empty())
    st = b200_set_error(B200_EINVAL, "plan: every TRSM must have order <= 256 and alpha != 0");
  if (st == B200_OK) st = capture(pl);
  if (st != B200_OK) {
    mublis_b200_plan_destroy(pl);
    return st;
  }
  *plan = pl;
  return b200_stream_sync();
}

int mublis_b200_plan_run(mublis_b200_plan_t *plan) {
  if (!plan || !plan->exec) return b200_set_error(B200_EINVAL, "plan: not instantiated");
  cudaStream_t s = b200_cur_stream();
  {
    B200ProfScope prof("plan_graph", s);
    B200_CUDA_TRY(cudaGraphLaunch(plan->exec, s));
  }
  return b200_stream_sync();
}

int mublis_b200_plan_destroy(mublis_b200_plan_t *plan) {
  if (!plan) return B200_OK;
  if (plan->exec) cudaGraphExecDestroy(plan->exec);
  if (plan->graph) cudaGraphDestroy(plan->graph);
  for (auto &g : plan->gg) b200_free(g.dtable);
  b200_free(plan->tg.dtable);
  b200_tcg_destroy(plan->tcg);
  b200_stream_sync();
  delete plan;
  return B200_OK;
}

}  // extern "C"

// ---- tuned-table API (include/mublis_b200.h) ---------------------------------

extern "C" void b200_tune_autoload(void) {
  if (const char *p = tune_env_path()) tune_load(p, nullptr);
}

extern "C" int mublis_b200_tune_save(const char *path) {
  B200_TRY(b200_init());
  return tune_save(path);
}

extern "C" int mublis_b200_tune_load(const char *path, int *entries) {
  if (entries) *entries = 0;
  B200_TRY(b200_init());
  return tune_load(path, entries);
}

void b200_tune_save_env() { b200_tune_autosave(); }

extern "C" int mublis_b200_tune_reset(void) {
  b200_ozaki2_table_reset();
  std::lock_guard<std::mutex> lk(g_tune_mu);
  memset(g_tuned, 0, sizeof g_tuned);
  return B200_OK;
}
