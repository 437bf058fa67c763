// pdot_aux.cu — the device passes around a solve: the feasibility rounding of
// a plan and the construction of a squared-Euclidean cost from coordinates.
//
// rounding (src/utils_gpu.jl:296-318): scale the rows by min(1, a / rowsum),
// then the columns by min(1, b / colsum) (a NaN ratio counts as 0), then add
// the rank-one correction err_r * err_c^T with err_r = a - rowsum normalised
// by its 1-norm (when that is not zero) and err_c = b - colsum. Sums are
// two-stage and in a fixed order; each product is rounded as the reference's
// `Diagonal(d) * X`, `X * Diagonal(d)` and `X .+= err_r * err_c'` round it.
#include <cstdint>

#include "pdot_common.cuh"
#include "pdot_pairs.cuh"

namespace pdot {
namespace {

constexpr int kAuxThreads = 256;
constexpr int kAuxWarps = kAuxThreads / 32;
constexpr int kColChunk = 64;  // columns per CTA of a warm-start plan's row sums

__device__ __forceinline__ double aux_warp_sum(double x) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) x += __shfl_xor_sync(0xffffffffu, x, o);
  return x;
}

__device__ __forceinline__ double row_sum(const double* part, int64_t m, int chunks, int64_t i) {
  double s = 0.0;
  int c = 0;
  for (; c + 8 <= chunks; c += 8) {  // eight loads in flight ahead of the ordered additions
    double v[8];
#pragma unroll
    for (int k = 0; k < 8; ++k) v[k] = part[(int64_t)(c + k) * m + i];
#pragma unroll
    for (int k = 0; k < 8; ++k) s += v[k];
  }
  for (; c < chunks; ++c) s += part[(int64_t)c * m + i];
  return s;
}

// min(1, dist / sum) with a NaN ratio replaced by 0 (src/utils_gpu.jl:302,305)
__device__ __forceinline__ double scale_of(double dist, double sum) {
  double t = __ddiv_rn(dist, sum);
  if (t != t) t = 0.0;
  return t < 1.0 ? t : 1.0;
}

// ---- rounding ----------------------------------------------------------------
// The scaled plans are never stored: each pass recomputes rs_i * X and
// cs_j * (rs_i * X) from X, rounding each product as the stored form would, so
// rounding streams the plan four times in and once out (40 B per entry: the row
// sums, the column sums of the row-scaled plan, both sums of the scaled plan,
// the write). With the scaled plans written back in place it was 80 B per entry
// and 11 launches: 10000 x 10000 took 1.81 ms on B200, now 0.75 with seven launches,
// where the five streams alone take 0.61 at the copy peak.
//
// CTA (p, c) of a summing pass covers panel p (kRoundRows rows) of column chunk c; a
// warp takes whole columns of the panel, lane rows in R-wide loads, so a column
// partial is one shuffle tree and row partials stay in registers until the chunk ends.
constexpr int kRoundRows = 256;
enum { kRoundRow = 1, kRoundCol = 2, kRoundRowScaled = 4, kRoundColScaled = 8 };

template <int R>
__device__ __forceinline__ void load_rows(const double* p, double (&v)[R]) {
  if constexpr (R == 2) {
    const double2 t = *reinterpret_cast<const double2*>(p);
    v[0] = t.x;
    v[1] = t.y;
  } else {
    v[0] = *p;
  }
}
template <int R>
__device__ __forceinline__ void store_rows(double* p, const double (&v)[R]) {
  if constexpr (R == 2)
    *reinterpret_cast<double2*>(p) = make_double2(v[0], v[1]);
  else
    *p = v[0];
}

template <int R, int MODE>
__global__ void __launch_bounds__(kAuxThreads, 3)
    k_round_sums(int64_t m, int64_t n, int64_t chunk, const double* __restrict__ X, const double* __restrict__ rscale,
                 const double* __restrict__ cscale, double* __restrict__ rowpart, double* __restrict__ colpart) {
  constexpr int RPL = kRoundRows / (32 * R);
  __shared__ double red[(MODE & kRoundRow) ? kAuxWarps : 1][(MODE & kRoundRow) ? kRoundRows : 1];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int64_t row0 = (int64_t)blockIdx.x * kRoundRows;
  const int64_t j0 = (int64_t)blockIdx.y * chunk, j1 = (j0 + chunk < n) ? j0 + chunk : n;
  double acc[RPL][R], rs[RPL][R];
  bool ok[RPL];
#pragma unroll
  for (int k = 0; k < RPL; ++k) {
    const int64_t i = row0 + k * 32 * R + lane * R;
    ok[k] = i < m;  // R divides m on the R-wide path
#pragma unroll
    for (int e = 0; e < R; ++e) {
      acc[k][e] = 0.0;
      rs[k][e] = ((MODE & kRoundRowScaled) && ok[k]) ? rscale[i + e] : 1.0;
    }
  }
  for (int64_t j = j0 + warp; j < j1; j += kAuxWarps) {
    const double cs = (MODE & kRoundColScaled) ? cscale[j] : 1.0;
    double x[RPL][R];
#pragma unroll
    for (int k = 0; k < RPL; ++k)
      if (ok[k]) load_rows<R>(X + j * m + row0 + k * 32 * R + lane * R, x[k]);
    double col = 0.0;
#pragma unroll
    for (int k = 0; k < RPL; ++k)
      if (ok[k]) {
#pragma unroll
        for (int e = 0; e < R; ++e) {
          double y = x[k][e];
          if (MODE & kRoundRowScaled) y = __dmul_rn(rs[k][e], y);
          if (MODE & kRoundColScaled) y = __dmul_rn(cs, y);
          if (MODE & kRoundRow) acc[k][e] += y;
          if (MODE & kRoundCol) col += y;
        }
      }
    if (MODE & kRoundCol) {
      col = aux_warp_sum(col);
      if (lane == 0) colpart[(int64_t)blockIdx.x * n + j] = col;
    }
  }
  if constexpr ((MODE & kRoundRow) != 0) {
#pragma unroll
    for (int k = 0; k < RPL; ++k)
#pragma unroll
      for (int e = 0; e < R; ++e) red[warp][k * 32 * R + lane * R + e] = acc[k][e];
    __syncthreads();
    const int64_t i = row0 + threadIdx.x;
    if (i < m) {
      double s = red[0][threadIdx.x];
#pragma unroll
      for (int w = 1; w < kAuxWarps; ++w) s += red[w][threadIdx.x];
      rowpart[(int64_t)blockIdx.y * m + i] = s;
    }
  }
}

// scale_i = min(1, dist_i / sum of the `parts` partials of i)
__global__ void k_round_scales(int64_t count, int parts, const double* __restrict__ part,
                               const double* __restrict__ dist, double* __restrict__ scale) {
  const int64_t i = (int64_t)blockIdx.x * kAuxThreads + threadIdx.x;
  if (i < count) scale[i] = scale_of(dist[i], row_sum(part, count, parts, i));
}

// err_r = a - rowsum and err_c = b - colsum of the scaled plan; block `bid` of the
// row blocks also leaves its share of ||err_r||_1 (a fixed-order tree).
__global__ void k_round_errors(int64_t m, int64_t n, int row_blocks, int chunks, int panels,
                               const double* __restrict__ rowpart, const double* __restrict__ colpart,
                               const double* __restrict__ a, const double* __restrict__ b, double* __restrict__ er,
                               double* __restrict__ ec, double* __restrict__ normpart) {
  if ((int)blockIdx.x >= row_blocks) {
    const int64_t j = (int64_t)(blockIdx.x - row_blocks) * kAuxThreads + threadIdx.x;
    if (j < n) ec[j] = __dsub_rn(b[j], row_sum(colpart, n, panels, j));
    return;
  }
  __shared__ double sh[kAuxThreads];
  const int64_t i = (int64_t)blockIdx.x * kAuxThreads + threadIdx.x;
  double e = 0.0;
  if (i < m) er[i] = e = __dsub_rn(a[i], row_sum(rowpart, m, chunks, i));
  sh[threadIdx.x] = fabs(e);
  __syncthreads();
  for (int w = kAuxThreads / 2; w > 0; w >>= 1) {
    if (threadIdx.x < w) sh[threadIdx.x] += sh[threadIdx.x + w];
    __syncthreads();
  }
  if (threadIdx.x == 0) normpart[blockIdx.x] = sh[0];
}

// X = cs_j * (rs_i * X) + (err_r / ||err_r||_1) * err_c^T. A thread keeps R rows and
// walks the columns of its chunk, four loads in flight.
template <int R>
__global__ void __launch_bounds__(kAuxThreads)
    k_round_write(int64_t m, int64_t n, int64_t chunk, double* __restrict__ X, const double* __restrict__ rscale,
                  const double* __restrict__ cscale, const double* __restrict__ er, const double* __restrict__ ec,
                  const double* __restrict__ normpart, int norm_blocks) {
  __shared__ double norm;
  if (threadIdx.x < 32) {
    double s = 0.0;
    for (int k = threadIdx.x; k < norm_blocks; k += 32) s += normpart[k];
    s = aux_warp_sum(s);
    if (threadIdx.x == 0) norm = s;
  }
  __syncthreads();
  const double nrm = norm;
  const int64_t i = ((int64_t)blockIdx.x * kAuxThreads + threadIdx.x) * R;
  if (i >= m) return;
  double rs[R], r[R];
#pragma unroll
  for (int e = 0; e < R; ++e) {
    rs[e] = rscale[i + e];
    r[e] = nrm != 0.0 ? __ddiv_rn(er[i + e], nrm) : er[i + e];
  }
  const int64_t j0 = (int64_t)blockIdx.y * chunk, j1 = (j0 + chunk < n) ? j0 + chunk : n;
  constexpr int U = 4;
  for (int64_t j = j0; j < j1; j += U) {
    double x[U][R];
#pragma unroll
    for (int k = 0; k < U; ++k)
      if (j + k < j1) load_rows<R>(X + (j + k) * m + i, x[k]);
#pragma unroll
    for (int k = 0; k < U; ++k)
      if (j + k < j1) {
        const double cs = cscale[j + k], c = ec[j + k];
#pragma unroll
        for (int e = 0; e < R; ++e)
          x[k][e] = __dadd_rn(__dmul_rn(cs, __dmul_rn(rs[e], x[k][e])), __dmul_rn(r[e], c));
        store_rows<R>(X + (j + k) * m + i, x[k]);
      }
  }
}

// ---- the squared-Euclidean cost ------------------------------------------------
// C_ij = ||x_i - y_j||^2 in FP64, divided by its maximum when `normalise`. The
// maximum is taken from the points, nothing stored, and the cost is then written
// once (8 B per entry); stored first, scanned and divided in place it took 32 B per
// entry: 0.93 ms at 10000 x 10000 in three dimensions on B200, now 0.20: 39 us for the
// maximum, 159 for the write, where a plain fill of the same bytes takes 116 to 120. The
// write is bound by latency, not by a unit: the FP64 pipe, issue and DRAM are each busy
// for half the time, and of the 13 cycles between two instructions of a warp 5 go to the
// loads of a column's coordinates and 4 to the chain of its 14 FP64 operations.
//
// DIM 1..4 are compiled in, 0 is any dimension (coordinates from global memory).
constexpr int kCostRows = 2;  // rows per thread of the write
template <int DIM>
__device__ __forceinline__ double sq_distance(const double* xi, const double* yj, int dim) {
  double s = 0.0;
  if constexpr (DIM > 0) {
#pragma unroll
    for (int d = 0; d < DIM; ++d) {
      const double t = __dsub_rn(xi[d], yj[d]);
      s = __dadd_rn(s, __dmul_rn(t, t));
    }
  } else {
    for (int d = 0; d < dim; ++d) {
      const double t = __dsub_rn(xi[d], yj[d]);
      s = __dadd_rn(s, __dmul_rn(t, t));
    }
  }
  return s;
}

// v / mx rounded to nearest for one divisor and many v >= 0 (quotient_of). The bounds on mx
// and v keep every term in the normal range; everything else, 0 and the entries next to
// mx and NaNs among it, takes the division itself.
struct DivideBy {
  double mx, y;
  unsigned low, span;  // high words of the v that take the corrections: low ... low + span
  __device__ __forceinline__ explicit DivideBy(double m) : mx(m) {
    const bool usable = m >= 0x1p-400 && m <= 0x1p+400;
    y = usable ? __drcp_rn(m) : 0.0;
    low = 0x20b00000u;  // 2^-500; the integer test costs an eighth of FP64 compares
    span = usable ? (unsigned)__double2hiint(m) - low : 0u;
  }
  __device__ __forceinline__ double operator()(double v) const {
    if ((unsigned)__double2hiint(v) - low < span) {
      return quotient_of(v, mx, y);
    }
    return __ddiv_rn(v, mx);
  }
};

// The largest entry (NaNs ignored), at least 0, by an atomicMax on its bits
// (non-negative doubles order as their bits do).
//
// DIM 1..4, large problems: a tile of columns is first passed over in FP32, with the
// coordinates taken relative to the first point. An FP32 distance is within
// E = 32 * 2^-24 * D A^2 of the FP64 one, A = |x|_max + |y|_max of those coordinates:
// narrowing moves a difference by 2^-24 A and its rounding by as much, a square then
// errs by 5 * 2^-24 A^2, and sum and test add less than that once more. Threads whose
// largest value cannot reach the CTA's largest lower bound, or the result so far, are
// done with the tile; the others take the FP64 distances of the columns, by fours, that
// can. Where E is not finite no pair is left out. 88 us in FP64 throughout at
// 10000 x 10000 in three dimensions, 39 this way; its FP32 operations alone take 17.
constexpr int kMaxTile = 128;  // columns of a tile
constexpr int kMaxRows = 2;    // rows per thread: a column's coordinates serve both
template <int D>
__global__ void __launch_bounds__(kAuxThreads)
    k_sqeuclid_max(int64_t m, int64_t n, int64_t share, const double* __restrict__ xs, const double* __restrict__ ys,
                   unsigned long long* __restrict__ out) {
  __shared__ double ty[kMaxTile * D];
  __shared__ __align__(16) float fy[D][kMaxTile];
  __shared__ double red[kAuxWarps];
  __shared__ float sbest;  // a lower bound of the result
  __shared__ int bound;    // bits of the tile's |y|_max
  double origin[D], x[kMaxRows][D];
  unsigned long long minus[kMaxRows][D];
  float reach[kMaxRows];
  bool ok[kMaxRows];
#pragma unroll
  for (int d = 0; d < D; ++d) origin[d] = fabs(xs[d]) < INFINITY ? xs[d] : 0.0;
#pragma unroll
  for (int q = 0; q < kMaxRows; ++q) {
    const int64_t i = ((int64_t)blockIdx.x * kMaxRows + q) * kAuxThreads + threadIdx.x;
    ok[q] = i < m;
    reach[q] = 0.0f;
#pragma unroll
    for (int d = 0; d < D; ++d) {
      x[q][d] = ok[q] ? xs[i * D + d] : origin[d];
      const float f = (float)(x[q][d] - origin[d]);
      reach[q] = fmaxf(reach[q], fabsf(f));
      minus[q][d] = pack2(-f, -f);
    }
  }
  if (threadIdx.x == 0)
    sbest = __double2float_rd(__longlong_as_double((long long)*reinterpret_cast<volatile unsigned long long*>(out)));
  double best = 0.0;
  const int64_t jb = (int64_t)blockIdx.y * share, je = (jb + share < n) ? jb + share : n;
  for (int64_t j0 = jb; j0 < je; j0 += kMaxTile) {
    const int cnt = (int)((je - j0) < kMaxTile ? (je - j0) : kMaxTile);
    __syncthreads();
    if (threadIdx.x == 0) bound = 0;
    __syncthreads();
    float my = 0.0f;
    // the FP32 entries past the last column repeat it
#pragma unroll
    for (int d = 0; d < D; ++d) {
      const int t = threadIdx.x, c = t < cnt ? t : cnt - 1;
      if (t >= kMaxTile) break;
      const double y = ys[(j0 + c) * D + d];
      const float f = (float)(y - origin[d]);
      ty[t * D + d] = y;
      fy[d][t] = f;
      my = fmaxf(my, fabsf(f));
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) my = fmaxf(my, __shfl_xor_sync(0xffffffffu, my, o));
    if ((threadIdx.x & 31) == 0) atomicMax(&bound, __float_as_int(my));
    __syncthreads();
    float top[kMaxRows], err[kMaxRows];
#pragma unroll
    for (int q = 0; q < kMaxRows; ++q) {
      const float A = reach[q] + __int_as_float(bound);
      err[q] = 32.0f * kUnit * (float)D * A * A + 1e-30f;
      top[q] = -1.0f;
    }
#pragma unroll 2
    for (int t = 0; t < cnt; t += 4) {
      ulonglong2 c[D];
#pragma unroll
      for (int d = 0; d < D; ++d) c[d] = *reinterpret_cast<const ulonglong2*>(&fy[d][t]);
#pragma unroll
      for (int q = 0; q < kMaxRows; ++q) top[q] = max_sqdist4<D>(minus[q], c, top[q]);
    }
    // the bits of non-negative floats order as the floats do
    float lower = 0.0f;
#pragma unroll
    for (int q = 0; q < kMaxRows; ++q)
      if (ok[q] && err[q] < INFINITY && top[q] < INFINITY) lower = fmaxf(lower, top[q] - err[q]);
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) lower = fmaxf(lower, __shfl_xor_sync(0xffffffffu, lower, o));
    if ((threadIdx.x & 31) == 0) atomicMax(reinterpret_cast<int*>(&sbest), __float_as_int(lower));
    __syncthreads();
    const float lim = sbest;
#pragma unroll
    for (int q = 0; q < kMaxRows; ++q) {
      // with a finite bound a tile of NaNs alone leaves top at -1 and has nothing to offer
      const bool finite = err[q] < INFINITY;
      if (!ok[q] || (finite && (top[q] < 0.0f || top[q] + err[q] < lim))) continue;
      for (int t = 0; t < cnt; t += 4) {
        ulonglong2 c[D];
#pragma unroll
        for (int d = 0; d < D; ++d) c[d] = *reinterpret_cast<const ulonglong2*>(&fy[d][t]);
        if (finite && max_sqdist4<D>(minus[q], c, -1.0f) + err[q] < lim) continue;
#pragma unroll
        for (int k = 0; k < 4; ++k)
          if (t + k < cnt) best = fmax(best, sq_distance<D>(x[q], ty + (t + k) * D, D));
      }
    }
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) best = fmax(best, __shfl_xor_sync(0xffffffffu, best, o));
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = best;
  __syncthreads();
  if (threadIdx.x == 0) {
#pragma unroll
    for (int w = 1; w < kAuxWarps; ++w) best = fmax(best, red[w]);
    atomicMax(out, (unsigned long long)__double_as_longlong(best));
  }
}

// The same in FP64 throughout: any dimension, and small problems, where the tiles' barriers
// and second passes cost more than the arithmetic (500 x 500 in one dimension, whole cost:
// 14.3 us against 17; 3000 x 2500 in two: 30.6 either way).
// rows per thread: a column's coordinates serve four distances where they are in registers
__host__ __device__ constexpr int small_rows(int dim) { return dim > 0 ? 4 : 1; }
constexpr int64_t kSmallPairs = int64_t(1) << 22;
template <int DIM>
__global__ void __launch_bounds__(kAuxThreads)
    k_sqeuclid_max_small(int64_t m, int64_t n, int dim, int64_t chunk, const double* __restrict__ xs,
                   const double* __restrict__ ys, unsigned long long* __restrict__ out) {
  constexpr int Q = small_rows(DIM);
  constexpr int D = DIM > 0 ? DIM : 1;
  const int64_t i0 = (int64_t)blockIdx.x * kAuxThreads * Q + threadIdx.x;
  double x[Q][D], mx[Q];
#pragma unroll
  for (int q = 0; q < Q; ++q) {
    mx[q] = 0.0;
    if constexpr (DIM > 0) {
      const int64_t i = i0 + q * kAuxThreads;
#pragma unroll
      for (int d = 0; d < D; ++d) x[q][d] = i < m ? xs[i * DIM + d] : 0.0;
    }
  }
  const int64_t j0 = (int64_t)blockIdx.y * chunk, j1 = (j0 + chunk < n) ? j0 + chunk : n;
#pragma unroll 2
  for (int64_t j = j0; j < j1; ++j) {
    if constexpr (DIM > 0) {
      double y[D];
#pragma unroll
      for (int d = 0; d < D; ++d) y[d] = __ldg(ys + j * DIM + d);
#pragma unroll
      for (int q = 0; q < Q; ++q) mx[q] = fmax(mx[q], sq_distance<DIM>(x[q], y, dim));
    } else {
#pragma unroll
      for (int q = 0; q < Q; ++q) {
        const int64_t i = i0 + q * kAuxThreads;
        if (i < m) mx[q] = fmax(mx[q], sq_distance<0>(xs + i * dim, ys + j * dim, dim));
      }
    }
  }
  double best = 0.0;
#pragma unroll
  for (int q = 0; q < Q; ++q)
    if (i0 + q * kAuxThreads < m) best = fmax(best, mx[q]);
  __shared__ double sh[kAuxWarps];
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) best = fmax(best, __shfl_xor_sync(0xffffffffu, best, o));
  if ((threadIdx.x & 31) == 0) sh[threadIdx.x >> 5] = best;
  __syncthreads();
  if (threadIdx.x == 0) {
#pragma unroll
    for (int w = 1; w < kAuxWarps; ++w) best = fmax(best, sh[w]);
    atomicMax(out, (unsigned long long)__double_as_longlong(best));
  }
}

// The cost's entries of a CTA's rows and column chunk, divided by *top when it is
// given and positive. Entry 0, where *top lies, is left to k_sqeuclid_first.
template <int DIM, int R>
__global__ void __launch_bounds__(kAuxThreads)
    k_sqeuclid_write(int64_t m, int64_t n, int64_t chunk, const double* __restrict__ xs, const double* __restrict__ ys,
                     const double* top, double* C) {
  const double mx = top ? *top : 0.0;
  const DivideBy by(mx);
  const int64_t i = ((int64_t)blockIdx.x * kAuxThreads + threadIdx.x) * R;
  if (i >= m) return;
  double x[R][DIM];
#pragma unroll
  for (int e = 0; e < R; ++e)
#pragma unroll
    for (int d = 0; d < DIM; ++d) x[e][d] = xs[(i + e) * DIM + d];
  const int64_t j0 = (int64_t)blockIdx.y * chunk, j1 = (j0 + chunk < n) ? j0 + chunk : n;
#pragma unroll 2
  for (int64_t j = j0; j < j1; ++j) {
    double v[R], y[DIM];
#pragma unroll
    for (int d = 0; d < DIM; ++d) y[d] = __ldg(ys + j * DIM + d);
#pragma unroll
    for (int e = 0; e < R; ++e) v[e] = sq_distance<DIM>(x[e], y, DIM);
    if (mx > 0.0) {
#pragma unroll
      for (int e = 0; e < R; ++e) v[e] = by(v[e]);
    }
    if (top && i == 0 && j == 0) {
      if constexpr (R == 2) C[1] = v[1];
    } else {
      store_rows<R>(C + j * m + i, v);
    }
  }
}

// The same an entry a thread, in the order of the matrix: for dimensions that are not
// compiled in, whose coordinates come from memory for every entry either way; for fewer
// than kEntryRows rows, which leave most lanes of the other form without one; and for few
// entries, which leave it too few CTAs. On B200, this and the other form: 10000 x 10000
// in six dimensions 548 and 742 us, 1000 x 3000 19 and 31; 8 x 10000 in the plane 4.1
// and 6.2, 64 x 10000 6.2 either way; 954 x 165 in four dimensions 4.4 and 6.3.
constexpr int kEntryRows = 64;
constexpr int64_t kFewEntries = 160000;
template <int DIM>
__global__ void __launch_bounds__(kAuxThreads)
    k_sqeuclid_entries(int64_t m, int64_t n, int dim, const double* __restrict__ xs, const double* __restrict__ ys,
                       const double* top, double* C) {
  const double mx = top ? *top : 0.0;
  const DivideBy by(mx);
  const int64_t N = m * n;
  for (int64_t e = (int64_t)blockIdx.x * kAuxThreads + threadIdx.x; e < N; e += (int64_t)gridDim.x * kAuxThreads) {
    const int64_t j = e / m, i = e - j * m;
    const int D = DIM > 0 ? DIM : dim;
    double v = sq_distance<DIM>(xs + i * D, ys + j * D, dim);
    if (mx > 0.0) v = by(v);
    if (!top || e != 0) C[e] = v;
  }
}

// Entry 0 in the place of the maximum that it held.
__global__ void k_sqeuclid_first(int dim, const double* __restrict__ xs, const double* __restrict__ ys,
                                 double* C) {
  const double mx = C[0], v = sq_distance<0>(xs, ys, dim);
  C[0] = mx > 0.0 ? __ddiv_rn(v, mx) : v;
}

// Row and column sums of a plan in storage type TX (the sums of a warm-start
// plan): row partials over column chunks, then their fixed-order total; one CTA
// per column for the column sums.
template <typename TX>
__global__ void k_plan_row_partials(int64_t m, int64_t n, const TX* __restrict__ X, double* __restrict__ part) {
  const int64_t i = (int64_t)blockIdx.x * kAuxThreads + threadIdx.x;
  const int64_t j0 = (int64_t)blockIdx.y * kColChunk;
  const int64_t j1 = (j0 + kColChunk < n) ? j0 + kColChunk : n;
  if (i >= m) return;
  double s = 0.0;
  for (int64_t j = j0; j < j1; ++j) s += (double)X[i + j * m];
  part[(int64_t)blockIdx.y * m + i] = s;
}

template <typename TX>
__global__ void k_plan_col_sums(int64_t m, const TX* __restrict__ X, double* __restrict__ out) {
  __shared__ double sh[kAuxThreads];
  const int64_t j = blockIdx.x;
  double s = 0.0;
  for (int64_t i = threadIdx.x; i < m; i += kAuxThreads) s += (double)X[i + j * m];
  sh[threadIdx.x] = s;
  __syncthreads();
  for (int w = kAuxThreads / 2; w > 0; w >>= 1) {
    if (threadIdx.x < w) sh[threadIdx.x] += sh[threadIdx.x + w];
    __syncthreads();
  }
  if (threadIdx.x == 0) out[j] = sh[0];
}

__global__ void k_plan_row_totals(int64_t m, int chunks, const double* __restrict__ part, double* __restrict__ r) {
  const int64_t i = (int64_t)blockIdx.x * kAuxThreads + threadIdx.x;
  if (i < m) r[i] = row_sum(part, m, chunks, i);
}

// Columns per CTA so that `strips` row strips times the chunks make about `target` CTAs,
// each with at least `least` columns.
int64_t column_chunk(int64_t n, int64_t strips, int64_t target, int64_t least) {
  const int64_t want = (target + strips - 1) / strips;
  const int64_t chunk = (n + want - 1) / want;
  const int64_t c = chunk < least ? least : chunk;
  return (n + c - 1) / c <= 65535 ? c : (n + 65534) / 65535;
}

struct RoundShape {
  int64_t panels, chunk, chunks, strips, wchunk;
  int rb, cb;
};
// About 16 CTAs per SM of the summing passes (3 resident): the ragged last
// panel's short CTAs then even out. A chunk has at least 4 columns per warp, so
// that the row partials stay below 1/32 of the plan.
RoundShape round_shape(int64_t m, int64_t n, int R) {
  RoundShape g;
  g.panels = (m + kRoundRows - 1) / kRoundRows;
  g.chunk = column_chunk(n, g.panels, 148 * 16, 32);
  g.chunks = (n + g.chunk - 1) / g.chunk;
  g.strips = (m + kAuxThreads * R - 1) / (kAuxThreads * R);
  g.wchunk = column_chunk(n, g.strips, 148 * 32, 8);
  g.rb = (int)((m + kAuxThreads - 1) / kAuxThreads);
  g.cb = (int)((n + kAuxThreads - 1) / kAuxThreads);
  return g;
}

template <int R>
cudaError_t rounding_passes(int64_t m, int64_t n, const double* a, const double* b, double* X, double* work,
                            cudaStream_t s) {
  const RoundShape g = round_shape(m, n, R);
  double* rowpart = work;
  double* colpart = rowpart + (size_t)g.chunks * m;
  double* rscale = colpart + (size_t)g.panels * n;
  double* cscale = rscale + m;
  double* er = cscale + n;
  double* ec = er + m;
  double* normpart = ec + n;
  const dim3 grid((unsigned)g.panels, (unsigned)g.chunks);
  const dim3 wgrid((unsigned)g.strips, (unsigned)((n + g.wchunk - 1) / g.wchunk));
  k_round_sums<R, kRoundRow><<<grid, kAuxThreads, 0, s>>>(m, n, g.chunk, X, nullptr, nullptr, rowpart, colpart);
  k_round_scales<<<g.rb, kAuxThreads, 0, s>>>(m, (int)g.chunks, rowpart, a, rscale);
  k_round_sums<R, kRoundCol | kRoundRowScaled>
      <<<grid, kAuxThreads, 0, s>>>(m, n, g.chunk, X, rscale, nullptr, rowpart, colpart);
  k_round_scales<<<g.cb, kAuxThreads, 0, s>>>(n, (int)g.panels, colpart, b, cscale);
  k_round_sums<R, kRoundRow | kRoundCol | kRoundRowScaled | kRoundColScaled>
      <<<grid, kAuxThreads, 0, s>>>(m, n, g.chunk, X, rscale, cscale, rowpart, colpart);
  k_round_errors<<<g.rb + g.cb, kAuxThreads, 0, s>>>(m, n, g.rb, (int)g.chunks, (int)g.panels, rowpart, colpart, a, b,
                                                     er, ec, normpart);
  k_round_write<R><<<wgrid, kAuxThreads, 0, s>>>(m, n, g.wchunk, X, rscale, cscale, er, ec, normpart, g.rb);
  return cudaGetLastError();
}

template <int DIM>
cudaError_t sqeuclid_passes(int64_t m, int64_t n, int dim, const double* xs, const double* ys, int normalise, double* C,
                            cudaStream_t s) {
  double* top = nullptr;
  if (normalise) {
    top = C;
    cudaError_t e = cudaMemsetAsync(top, 0, sizeof(double), s);
    if (e != cudaSuccess) return e;
    auto* bits = reinterpret_cast<unsigned long long*>(top);
    if (DIM == 0 || m * n <= kSmallPairs) {
      constexpr int Q = small_rows(DIM);
      const int64_t strips = (m + kAuxThreads * Q - 1) / (kAuxThreads * Q);
      const int64_t chunk = column_chunk(n, strips, 148 * 16, 4 * Q);
      k_sqeuclid_max_small<DIM>
          <<<dim3((unsigned)strips, (unsigned)((n + chunk - 1) / chunk)), kAuxThreads, 0, s>>>(m, n, dim, chunk, xs, ys, bits);
    } else if constexpr (DIM > 0) {
      const int64_t strips = (m + kAuxThreads * kMaxRows - 1) / (kAuxThreads * kMaxRows);
      // some 16 CTAs per SM, none with less than a tile
      const int64_t share = column_chunk(n, strips, 148 * 16, kMaxTile);
      k_sqeuclid_max<DIM><<<dim3((unsigned)strips, (unsigned)((n + share - 1) / share)), kAuxThreads, 0, s>>>(
          m, n, share, xs, ys, bits);
    }
  }
  if (DIM == 0 || m < kEntryRows || m * n <= kFewEntries) {
    const int64_t ctas = (m * n + kAuxThreads - 1) / kAuxThreads;
    k_sqeuclid_entries<DIM><<<(unsigned)(ctas < 148 * 16 ? ctas : 148 * 16), kAuxThreads, 0, s>>>(m, n, dim, xs, ys, top, C);
  } else if constexpr (DIM > 0) {
    const bool wide = m % kCostRows == 0 && (reinterpret_cast<uintptr_t>(C) & 15u) == 0;
    const int R = wide ? kCostRows : 1;
    const int64_t strips = (m + kAuxThreads * R - 1) / (kAuxThreads * R);
    const int64_t chunk = column_chunk(n, strips, 148 * 32, 8);
    const dim3 grid((unsigned)strips, (unsigned)((n + chunk - 1) / chunk));
    if (wide)
      k_sqeuclid_write<DIM, kCostRows><<<grid, kAuxThreads, 0, s>>>(m, n, chunk, xs, ys, top, C);
    else
      k_sqeuclid_write<DIM, 1><<<grid, kAuxThreads, 0, s>>>(m, n, chunk, xs, ys, top, C);
  }
  if (normalise) k_sqeuclid_first<<<1, 1, 0, s>>>(dim, xs, ys, C);
  return cudaGetLastError();
}

}  // namespace

size_t rounding_workspace_doubles(int64_t m, int64_t n) {
  const RoundShape g = round_shape(m, n, 1);  // the sums' shape does not depend on the load width
  return (size_t)g.chunks * m + (size_t)g.panels * n + 2 * (size_t)m + 2 * (size_t)n + g.rb;
}

cudaError_t launch_rounding(int64_t m, int64_t n, const double* a, const double* b, double* X, double* work,
                            cudaStream_t s) {
  // 16-byte loads where every column starts on a 16-byte boundary
  if (m % 2 == 0 && (reinterpret_cast<uintptr_t>(X) & 15u) == 0) return rounding_passes<2>(m, n, a, b, X, work, s);
  return rounding_passes<1>(m, n, a, b, X, work, s);
}

size_t plan_sums_workspace_doubles(int64_t m, int64_t n) {
  return (size_t)((n + kColChunk - 1) / kColChunk) * (size_t)m;
}

cudaError_t launch_plan_sums(int64_t m, int64_t n, const void* X, int plan_f32, double* r, double* c, double* work,
                             cudaStream_t s) {
  const int chunks = (int)((n + kColChunk - 1) / kColChunk);
  const dim3 rgrid((unsigned)((m + kAuxThreads - 1) / kAuxThreads), (unsigned)chunks);
  const int rb = (int)((m + kAuxThreads - 1) / kAuxThreads);
  if (plan_f32) {
    k_plan_row_partials<float><<<rgrid, kAuxThreads, 0, s>>>(m, n, static_cast<const float*>(X), work);
    k_plan_col_sums<float><<<(unsigned)n, kAuxThreads, 0, s>>>(m, static_cast<const float*>(X), c);
  } else {
    k_plan_row_partials<double><<<rgrid, kAuxThreads, 0, s>>>(m, n, static_cast<const double*>(X), work);
    k_plan_col_sums<double><<<(unsigned)n, kAuxThreads, 0, s>>>(m, static_cast<const double*>(X), c);
  }
  k_plan_row_totals<<<rb, kAuxThreads, 0, s>>>(m, chunks, work, r);
  return cudaGetLastError();
}

cudaError_t launch_sqeuclid_cost(int64_t m, int64_t n, int dim, const double* xs, const double* ys, int normalise,
                                 double* C, cudaStream_t s) {
  switch (dim) {
    case 1: return sqeuclid_passes<1>(m, n, dim, xs, ys, normalise, C, s);
    case 2: return sqeuclid_passes<2>(m, n, dim, xs, ys, normalise, C, s);
    case 3: return sqeuclid_passes<3>(m, n, dim, xs, ys, normalise, C, s);
    case 4: return sqeuclid_passes<4>(m, n, dim, xs, ys, normalise, C, s);
    default: return sqeuclid_passes<0>(m, n, dim, xs, ys, normalise, C, s);
  }
}

}  // namespace pdot
