// trsm_small.cu -- left triangular solves of order up to 256 in one launch each,
// or one launch for many (grouped.cu): alpha, the solve and the updates between the
// blocks all in one kernel.
//
// Reference: the blocked solve of frame/l3/trsm.c:139-183 with gemmtrsm
// micro-kernels (include/mublis_instantiate.h:95-114) over a packed A whose
// diagonal is inverted (packm.c:143-144).  Here a CTA owns 32 right-hand-side
// columns of one problem and keeps them in registers, 16 rows to a warp: 8 warps
// up to order 128, 16 up to 256.  (Two blocks a warp duplicated the update and
// solve code; a kernel whose code runs once or a few times pays for its size in
// instruction fetches.)
//   * Start: the 16 x 16 diagonal blocks come in by asynchronous copies; their
//     diagonal becomes its reciprocal, as in the reference's packing.
//   * Step d: X_d (solved, in shared memory) updates the blocks below,
//     B_r -= A_rd X_d, and the warp of block d + 1 then solves it by substitution.
//     One block barrier per step.
//   * Column d of A's blocks arrives two steps ahead in a 3-deep ring of
//     asynchronous element copies, zeros past the matrix, nothing of the
//     unstored triangle or of a unit diagonal read.
// FP64 updates are m16n8k4 .f64 MMAs (16 x 20 blocks: a fragment load's half-warp
// falls on 16 different 8-byte banks); FP32 ones and both solves are FMAs with a
// lane per column and the blocks of A broadcast.
// An upper triangle is the lower one with rows and columns reversed.
//
// What bounds it: the latency of the order / 16 dependent steps; CTAs of other
// slabs and problems fill an SM meanwhile.  Measured (us, before -> now): groups
// of 1024 of order 32-256, FP64 1188 -> 165 and FP32 853 -> 139 (one warp
// substituted 32 rows at a time); a call of order 256 with 4000 right-hand sides,
// FP64 84 -> 60 (the leaf kernel after a scale and a pack); of order 128 with 1000,
// FP32 117 -> 46 (inverted blocks, a dozen launches).
#include <algorithm>
#include <type_traits>

#include "kernels.cuh"

namespace {

constexpr int LB = 16, NBC = 32, RING = 3;

template <typename T>
struct Layout {
  static constexpr bool F64 = sizeof(T) == 8;
  static constexpr int PITCH = F64 ? 20 : 16;  // of a 16 x 16 block
  static constexpr int BLK = LB * PITCH;
  static constexpr int XLD = F64 ? 36 : 33;    // of a solved 16 x 32 block
  // Element (r, c) of a block below the diagonal (FP64: row-major, FP32:
  // column-major) and of a diagonal block (column-major).
  __host__ __device__ static constexpr int panel(int r, int c) {
    return F64 ? r * PITCH + c : c * PITCH + r;
  }
  __host__ __device__ static constexpr int diag(int r, int c) { return c * PITCH + r; }
  // Elements of shared memory for problems of up to nb blocks.
  __host__ __device__ static constexpr int elements(int nb) {
    return nb * BLK + RING * (nb > 1 ? nb - 1 : 1) * BLK + 2 * LB * XLD;
  }
};

template <int BYTES>
__device__ __forceinline__ void cp_zfill(void *dst, const void *src, bool in) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], %2, %3;" ::"r"(
                   (uint32_t)__cvta_generic_to_shared(dst)),
               "l"(src), "n"(BYTES), "r"(in ? BYTES : 0)
               : "memory");
}
__device__ __forceinline__ void cp_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N>
__device__ __forceinline__ void cp_wait() {
  asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory");
}

__device__ __forceinline__ void dmma(double (&c)[4], double a0, double a1, double b0) {
  asm volatile(
      "mma.sync.aligned.m16n8k4.row.col.f64.f64.f64.f64 {%0,%1,%2,%3}, {%4,%5}, {%6}, "
      "{%0,%1,%2,%3};\n"
      : "+d"(c[0]), "+d"(c[1]), "+d"(c[2]), "+d"(c[3])
      : "d"(a0), "d"(a1), "d"(b0));
}

// A warp's 16 x 32 block of B.  FP64: c[j][e] is row g + 8 (e / 2), column 8 j +
// 2 t + e % 2.  FP32: c[r / 2] holds rows r and r + 1 of the lane's column.
template <typename T>
struct Block;
template <>
struct Block<double> {
  double c[4][4];
  template <typename F>
  __device__ __forceinline__ void each(F f) {  // f(row, column, element)
    const int g = (threadIdx.x & 31) >> 2, t = threadIdx.x & 3;
#pragma unroll
    for (int j = 0; j < 4; ++j)
#pragma unroll
      for (int e = 0; e < 4; ++e) f(g + 8 * (e >> 1), 8 * j + 2 * t + (e & 1), c[j][e]);
  }
};
template <>
struct Block<float> {
  float2 c[8];
  template <typename F>
  __device__ __forceinline__ void each(F f) {
    const int lane = threadIdx.x & 31;
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      f(2 * i, lane, c[i].x);
      f(2 * i + 1, lane, c[i].y);
    }
  }
};

// X as the operand of an update: FP64 B fragments, FP32 the lane's column.
template <typename T>
using XFrag = typename std::conditional<sizeof(T) == 8, double[4][4], float[LB]>::type;

template <typename T>
__device__ __forceinline__ void load_x(const T *x, XFrag<T> &f) {
  constexpr int LD = Layout<T>::XLD;
  const int lane = threadIdx.x & 31;
  if constexpr (sizeof(T) == 8) {
#pragma unroll
    for (int ks = 0; ks < 4; ++ks)
#pragma unroll
      for (int j = 0; j < 4; ++j) f[ks][j] = x[(4 * ks + (lane & 3)) * LD + 8 * j + (lane >> 2)];
  } else {
#pragma unroll
    for (int k = 0; k < LB; ++k) f[k] = x[k * LD + lane];
  }
}

// FP64: b -= A x, FP32: b += A x, for a 16 x 16 block A.
__device__ __forceinline__ void update(Block<double> &b, const double *a, const double (&x)[4][4]) {
  const int g = (threadIdx.x & 31) >> 2, t = threadIdx.x & 3;
#pragma unroll
  for (int ks = 0; ks < 4; ++ks) {
    const double a0 = -a[Layout<double>::panel(g, 4 * ks + t)];
    const double a1 = -a[Layout<double>::panel(g + 8, 4 * ks + t)];
#pragma unroll
    for (int j = 0; j < 4; ++j) dmma(b.c[j], a0, a1, x[ks][j]);
  }
}
__device__ __forceinline__ void update(Block<float> &b, const float *a, const float (&x)[LB]) {
#pragma unroll
  for (int k = 0; k < LB; ++k) {
    const float2 v = make_float2(x[k], x[k]);
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const float4 w = *(const float4 *)(a + Layout<float>::panel(4 * i, k));
      b.c[2 * i] = __ffma2_rn(make_float2(w.x, w.y), v, b.c[2 * i]);
      b.c[2 * i + 1] = __ffma2_rn(make_float2(w.z, w.w), v, b.c[2 * i + 1]);
    }
  }
}

// Solves a diagonal block D (lower triangle, reciprocal diagonal) for a warp's 32
// columns, a column to a lane, by substitution: x[i] = r[i] / D[i][i], then r[j] -=
// D[j][i] x[i] below.  D's columns are read as 16-byte broadcasts.  A product with
// the block's inverse instead (on the FP64 MMAs, or as many FMAs) took as long but
// was not backward stable -- diagonals of 0.05-1: residuals of 900 u |A||X| at order
// 16, 2 u so -- and its zeros spread a non-finite r to rows above it.
__device__ __forceinline__ void solve(Block<double> &b, const double *d, double *x) {
  constexpr int LD = Layout<double>::XLD;
  const int lane = threadIdx.x & 31;
  b.each([&](int r, int c, double v) { x[r * LD + c] = v; });
  __syncwarp();
  double r[LB];
#pragma unroll
  for (int i = 0; i < LB; ++i) r[i] = x[i * LD + lane];
#pragma unroll
  for (int i = 0; i < LB; ++i) {
    double col[LB];  // rows from i - i % 2 on
#pragma unroll
    for (int j = i / 2 * 2; j < LB; j += 2) {
      const double2 v = *(const double2 *)(d + Layout<double>::diag(j, i));
      col[j] = v.x, col[j + 1] = v.y;
    }
    r[i] *= col[i];
    x[i * LD + lane] = r[i];
#pragma unroll
    for (int j = i + 1; j < LB; ++j) r[j] = fma(-col[j], r[i], r[j]);
  }
}
// FP32: r = alpha rhs - sum, formed when its row is reached; the substitution's
// products go to the sum.
__device__ __forceinline__ void solve(Block<float> &sum, const Block<float> &rhs, float alpha,
                                      const float *d, float *x) {
  constexpr int LD = Layout<float>::XLD;
  const int lane = threadIdx.x & 31;
#pragma unroll
  for (int i = 0; i < LB; ++i) {
    float col[LB];  // rows from i - i % 4 on
#pragma unroll
    for (int j = i / 4 * 4; j < LB; j += 4) {
      const float4 v = *(const float4 *)(d + Layout<float>::diag(j, i));
      col[j] = v.x, col[j + 1] = v.y, col[j + 2] = v.z, col[j + 3] = v.w;
    }
    const float r = i % 2 ? fmaf(alpha, rhs.c[i / 2].y, -sum.c[i / 2].y)
                          : fmaf(alpha, rhs.c[i / 2].x, -sum.c[i / 2].x);
    const float xi = r * col[i];
    x[i * LD + lane] = xi;
    if (i % 2 == 0) sum.c[i / 2].y = fmaf(col[i + 1], xi, sum.c[i / 2].y);
#pragma unroll
    for (int j = i / 2 + 1; j < LB / 2; ++j)
      sum.c[j] = __ffma2_rn(make_float2(col[2 * j], col[2 * j + 1]), make_float2(xi, xi), sum.c[j]);
  }
}

// table may be null: then `one` is the only problem.
template <typename T, int WARPS>
__global__ void __launch_bounds__(WARPS * 32, 16 / WARPS)
    small_trsm_kernel(const b200_small_trsm_t *__restrict__ table, const int *__restrict__ slab_prob,
                      int first_slab, const __grid_constant__ b200_small_trsm_t one) {
  using L = Layout<T>;
  constexpr int THREADS = WARPS * 32;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const int slab = first_slab + blockIdx.x;
  const b200_small_trsm_t &e = table ? table[slab_prob[slab]] : one;
  const int m = e.m, nb = (m + LB - 1) / LB;
  T *dia = (T *)smem_raw;            // [nb] diagonal blocks, reciprocal diagonal
  T *ring = dia + nb * L::BLK;       // [RING][nb - 1] blocks
  const int seg = (nb > 1 ? nb - 1 : 1) * L::BLK;
  T *xs = ring + RING * seg;         // [2] solved blocks
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const T *A = (const T *)e.a;
  // Lower orientation: element (i, p) of op(A), or for an upper triangle
  // (m - 1 - i, m - 1 - p); likewise the rows of B.
  const long ars = e.lower ? e.rs_a : -e.rs_a, acs = e.lower ? e.cs_a : -e.cs_a;
  const T *a0 = e.lower ? A : A + (m - 1) * (e.rs_a + e.cs_a);
  const long brs = e.lower ? e.rs_b : -e.rs_b, bcs = e.cs_b;
  const long col0 = (long)(slab - e.slab0) * NBC;
  const int ncol = (int)min((long)NBC, e.n - col0);
  T *b0 = (T *)e.b + col0 * bcs + (e.lower ? 0 : (m - 1) * e.rs_b);
  const bool rows_fast = labs(ars) <= labs(acs);

  // Thread tid copies element (er, ec) of every (THREADS / 256)-th 16 x 16 block,
  // along A's unit stride.
  constexpr int STRIDE = THREADS / (LB * LB);
  const int ex = tid % (LB * LB), eb = tid / (LB * LB);
  const int er = rows_fast ? ex % LB : ex / LB, ec = rows_fast ? ex / LB : ex % LB;
  const T *ae = a0 + er * ars + ec * acs;
  // Blocks below the diagonal of block column d.
  auto load_segment = [&](int d) {
    T *dst = ring + (d % RING) * seg + eb * L::BLK + L::panel(er, ec);
    const T *src = ae + (long)(d + 1 + eb) * LB * ars + (long)d * LB * acs;
    for (int blk = d + 1 + eb; blk < nb; blk += STRIDE) {
      const bool in = blk * LB + er < m;  // (its column lies left of the last block: inside)
      cp_zfill<sizeof(T)>(dst, in ? src : A, in);
      src += STRIDE * LB * ars;
      dst += STRIDE * L::BLK;
    }
  };
  // The diagonal blocks: lower triangle, the identity past the matrix.
  for (int blk = eb; blk < nb; blk += STRIDE) {
    T *dst = dia + blk * L::BLK + L::diag(er, ec);
    if (blk * LB + er < m && (ec < er || (ec == er && !e.unit)))
      cp_zfill<sizeof(T)>(dst, ae + (long)blk * LB * (ars + acs), true);
    else
      *dst = ec == er ? T(1) : T(0);
  }
  cp_commit();
  for (int d = 0; d < 2; ++d) {
    if (d < nb - 1) load_segment(d);
    cp_commit();
  }

  // This warp's rows of B.  FP64 multiplies them by alpha and subtracts the updates
  // as they come; FP32 sums the updates by themselves and forms alpha B minus the
  // sum in one rounding, so that the others are of the (smaller) sum, not of B
  // (relative error of a solve 5.1e-8 with alpha B rounded by itself, 4.4e-8 so).
  const T alpha = (T)e.alpha;
  Block<T> acc, rhs;
  (L::F64 ? acc : rhs).each([&](int r, int c, T &v) {
    v = warp * LB + r < m && c < ncol ? b0[(warp * LB + r) * brs + c * bcs] : T(0);
    if constexpr (L::F64) v *= alpha;
  });
  if constexpr (!L::F64) acc.each([](int, int, T &v) { v = T(0); });

  cp_wait<2>();  // the diagonal blocks
  __syncthreads();
  if (warp < nb && lane < LB) {  // warp w: the reciprocal diagonal of block w
    T *d = dia + warp * L::BLK + L::diag(lane, lane);
    *d = T(1) / *d;
  }
  __syncthreads();

  // Solved block blk -> B, along B's unit stride.
  const bool b_rows_fast = labs(brs) <= labs(bcs);
  auto write_block = [&](int blk) {
    const T *x = xs + (blk & 1) * LB * L::XLD;
#pragma unroll
    for (int idx = tid; idx < LB * NBC; idx += THREADS) {
      const int r = b_rows_fast ? idx % LB : idx / NBC, c = b_rows_fast ? idx / LB : idx % NBC;
      if (blk * LB + r < m && c < ncol) b0[(blk * LB + r) * brs + c * bcs] = x[r * L::XLD + c];
    }
  };

  // Column 0 .. nb - 1: solve its block, then update the blocks below it.
  for (int d = 0; d < nb; ++d) {
    T *xd = xs + (d & 1) * LB * L::XLD;
    if (warp == d) {
      if constexpr (L::F64) solve(acc, dia + d * L::BLK, xd);
      else solve(acc, rhs, alpha, dia + d * L::BLK, xd);
    }
    cp_wait<1>();     // segment d
    __syncthreads();  // X_d and segment d are there; every warp is done with step d - 1
    if (d + 2 < nb - 1) load_segment(d + 2);
    cp_commit();
    if (warp > d && warp < nb) {
      XFrag<T> x;
      load_x<T>(xd, x);
      update(acc, ring + (d % RING) * seg + (warp - d - 1) * L::BLK, x);
    }
    write_block(d);
  }
}

template <typename T, int WARPS>
int launch(const b200_small_trsm_t *table, const int *slab_prob, const b200_small_trsm_t *one,
           int first_slab, int slabs, int max_order, cudaStream_t s) {
  using L = Layout<T>;
  auto kern = small_trsm_kernel<T, WARPS>;
  static B200Once once;
  B200_TRY(b200_once(once, "small trsm: set-up failed", [&]() -> int {
    cudaFuncAttributes fa;
    B200_CUDA_TRY(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                       (int)sizeof(T) * L::elements(WARPS)));
    B200_CUDA_TRY(cudaFuncGetAttributes(&fa, kern));  // loads it: a capture must not
    return B200_OK;
  }));
  if (slabs <= 0) return B200_OK;
  b200_small_trsm_t none = {};
  B200ProfScope prof(sizeof(T) == 4 ? "small_strsm" : "small_dtrsm", s);
  kern<<<slabs, WARPS * 32, sizeof(T) * L::elements((max_order + LB - 1) / LB), s>>>(
      table, slab_prob, first_slab, one ? *one : none);
  B200_LAUNCH_CHECK();
  return B200_OK;
}

template <typename T>
int launch_order(const b200_small_trsm_t *table, const int *slab_prob, const b200_small_trsm_t *one,
                 int first_slab, int slabs, int max_order, cudaStream_t s) {
  return max_order <= 128 ? launch<T, 8>(table, slab_prob, one, first_slab, slabs, max_order, s)
                          : launch<T, 16>(table, slab_prob, one, first_slab, slabs, max_order, s);
}

}  // namespace

int launch_small_trsm(int dtype, const b200_small_trsm_t *table, const int *slab_prob, int first_slab,
                      int slabs, int max_order, cudaStream_t s) {
  return dtype == B200_F64
             ? launch_order<double>(table, slab_prob, nullptr, first_slab, slabs, max_order, s)
             : launch_order<float>(table, slab_prob, nullptr, first_slab, slabs, max_order, s);
}

int launch_small_trsm_one(int dtype, const b200_small_trsm_t &e, cudaStream_t s) {
  const long slabs = b200_ceil_div(e.n, NBC);
  if (slabs > 0x7fffffffL) return b200_set_error(B200_EINVAL, "trsm: too many right-hand sides");
  return dtype == B200_F64 ? launch_order<double>(nullptr, nullptr, &e, 0, (int)slabs, e.m, s)
                           : launch_order<float>(nullptr, nullptr, &e, 0, (int)slabs, e.m, s);
}
