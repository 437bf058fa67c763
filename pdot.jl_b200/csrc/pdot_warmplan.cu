// pdot_warmplan.cu — a warm-start plan recovered from warm-start duals (an
// addition; the reference always starts at zero, src/solver_gpu.jl:428-441).
//
// Given duals (u0, v0) and eps > 0, rounds of log-domain balancing
//   f_i = eps (log a_i - LSE_j((g_j - C_ij) / eps))        (rows sum to a)
//   g_j = eps (log b_j - LSE_i((f_i - C_ij) / eps))        (columns sum to b)
// start from (f, g) = (u0, v0); the plan is X_ij = exp((f_i + g_j - C_ij) / eps)
// and its row and column sums r, c. The solver keeps (u0, v0) as its duals.
// Every sum is in a fixed order (lane l of a warp takes entries l, l + 32, ... of
// a row or column, then a shuffle tree), so the result is deterministic. The
// balancing rounds take their exponentials in FP32 (the plan is only a starting
// point); the plan entries and their sums are FP64 (narrowed to the plan's storage
// type before they are summed).
//
// A warp takes up to Q neighbouring rows (columns) at once, with the cost kind and
// the point dimension compiled in: the other side's potential and coordinates are
// loaded once for Q entries and Q times four dependency chains overlap. What bounds a
// round is issue and the latency of those chains: 35 instructions an entry, four of
// them FP64 and two conversions; no round touches the plan. Measured on B200 per
// half-round (one row at a time with the kind and dimension read at run time, before;
// as here): 191 -> 71 us at 8000 x 6000 and 967 -> 369 us at 20000 x 15000 from
// planar points, 20 -> 12 us at 1024 x 1024, 272 -> 124 us for a stored FP64 cost of
// 6000 x 6000.
#include <cmath>
#include <cstdint>

#include "pdot_device.cuh"

namespace pdot {
namespace {

constexpr int kWpThreads = 256;
constexpr int kWpWarps = kWpThreads / 32;
// CTAs of two warps: a few thousand row groups then spread evenly over the SMs.
constexpr int kWpGroupThreads = 64;
constexpr int kWpGroupWarps = kWpGroupThreads / 32;
constexpr int kWpUnroll = 4;
// Rows of a warp's group: two, or four for a stored cost of 4 bytes or fewer an entry,
// whose 32-byte sectors they share (25 against 30 us at 3000 x 3000 in FP32; from
// points two beat four by 71 to 90 us at 8000 x 6000, where four leave 13 warps per SM).
constexpr int group_rows(int ck) { return ck == PDOT_COST_F32 || ck == PDOT_COST_BF16 ? 4 : 2; }
// Groups only where they still leave some 8 warps per SM; below, a warp takes one
// row, since then latency counts and not the work per entry.
constexpr bool grouped(long long total, int Q) { return total >= 148ll * 8 * Q; }

__device__ __forceinline__ int find_instance(const long long* prefix, int count, long long q) {
  int lo = 0, hi = count - 1;
  while (lo < hi) {
    const int mid = (lo + hi + 1) >> 1;
    if (__ldg(prefix + mid) <= q)
      lo = mid;
    else
      hi = mid - 1;
  }
  return lo;
}

// The solver's cost entries C_ij of instance I between the Q members of a group (rows
// if BY_ROWS, else columns) and one member of the other side: coordinate costs in FP32
// as the solver reads them, times the instance's cost scale, or the stored entry.
// Members past the group's end repeat its last one.
template <int CK, int Q, bool BY_ROWS>
struct GroupCost {
  static constexpr bool kPoints = is_point_cost(CK);
  static constexpr bool kL1 = is_l1_cost(CK);
  static constexpr int DIM = kPoints ? CK - (kL1 ? kCostL1Base : kCostSqBase) : 1;
  const void* C;
  const float* other;
  float scale;
  float own[Q][DIM];
  float oth[DIM];
  int64_t base[Q];
  int64_t stride;
  __device__ __forceinline__ GroupCost(const WarmPlanArgs& A, const PlanInstance& I, float scl, int64_t first, int count)
      : C(A.C), scale(scl) {
    if constexpr (kPoints) {
      const float* mine = BY_ROWS ? A.xs + I.row_off * DIM : A.ys + I.col_off * DIM;
      other = BY_ROWS ? A.ys + I.col_off * DIM : A.xs + I.row_off * DIM;
#pragma unroll
      for (int q = 0; q < Q; ++q)
#pragma unroll
        for (int d = 0; d < DIM; ++d) own[q][d] = __ldg(mine + (first + (q < count ? q : count - 1)) * DIM + d);
    } else {
      stride = BY_ROWS ? I.ld : 1;
#pragma unroll
      for (int q = 0; q < Q; ++q) {
        const int64_t k = first + (q < count ? q : count - 1);
        base[q] = I.x_off + (BY_ROWS ? k : k * I.ld);
      }
    }
  }
  // the other side's member `o` that get() pairs with the group's
  __device__ __forceinline__ void load(int64_t o) {
    if constexpr (kPoints) {
#pragma unroll
      for (int d = 0; d < DIM; ++d) oth[d] = __ldg(other + o * DIM + d);
    }
  }
  __device__ __forceinline__ double get(int q, int64_t o) const {
    if constexpr (CK == PDOT_COST_F64) {
      return __ldg(static_cast<const double*>(C) + base[q] + o * stride);
    } else if constexpr (CK == PDOT_COST_F32) {
      return (double)__ldg(static_cast<const float*>(C) + base[q] + o * stride);
    } else if constexpr (CK == PDOT_COST_BF16) {
      return (double)__bfloat162float(static_cast<const __nv_bfloat16*>(C)[base[q] + o * stride]);
    } else {
      float acc = 0.0f;
#pragma unroll
      for (int d = 0; d < DIM; ++d) {
        const float t = BY_ROWS ? own[q][d] - oth[d] : oth[d] - own[q][d];
        const float e = kL1 ? fabsf(t) : t * t;
        acc = d == 0 ? e : acc + e;
      }
      return (double)(acc * scale);
    }
  }
};

// log-sum-exp accumulator: value = mx + log(s)
struct Lse {
  double mx = -INFINITY;
  float s = 0.0f;
  // A new maximum rescales the sum by exp(mx - x) and adds 1, any other x adds
  // exp(x - mx): one exponential of -|x - mx| either way (0 from mx = -inf), so a
  // warp whose lanes disagree does not take it twice.
  __device__ __forceinline__ void add(double x) {
    const float e = expf((float)-fabs(x - mx));
    const bool up = x > mx;
    const float t = up ? s * e + 1.0f : s + e;
    s = x > -INFINITY ? t : s;  // -inf and NaN leave the sum alone
    mx = up ? x : mx;
  }
  __device__ __forceinline__ void merge_warp() {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      const double om = __shfl_xor_sync(0xffffffffu, mx, o);
      const float os = __shfl_xor_sync(0xffffffffu, s, o);
      const double M = om > mx ? om : mx;
      if (M == -INFINITY) continue;
      s = (mx == -INFINITY ? 0.0f : s * expf((float)(mx - M))) + (om == -INFINITY ? 0.0f : os * expf((float)(om - M)));
      mx = M;
    }
  }
};

// Calls f(instance, its index, first local row, rows) for the parts of a warp's group of
// Q global rows (columns) that lie in one active instance each.
template <int Q, typename F>
__device__ __forceinline__ void for_groups(const WarmPlanArgs& A, const long long* prefix, long long total, F&& f) {
  const long long groups = (total + Q - 1) / Q;
  for (long long w = (long long)blockIdx.x * kWpGroupWarps + (threadIdx.x >> 5); w < groups;
       w += (long long)gridDim.x * kWpGroupWarps) {
    long long q = w * Q;
    const long long qe = q + Q < total ? q + Q : total;
    while (q < qe) {
      const int k = find_instance(prefix, A.num, q);
      const long long b = __ldg(prefix + k), e = __ldg(prefix + k + 1);
      const long long to = e < qe ? e : qe;
      const PlanInstance I = A.inst[k];
      if (I.active) f(I, k, (int64_t)(q - b), (int)(to - q));
      q = to;
    }
  }
}

// One balancing half-round: rows (BY_ROWS) update f from g, columns g from f.
// `first` reads the other side from the warm duals.
template <int CK, int Q, bool BY_ROWS>
__global__ void __launch_bounds__(kWpGroupThreads) k_wp_balance(WarmPlanArgs A, int first) {
  const int lane = threadIdx.x & 31;
  for_groups<Q>(A, BY_ROWS ? A.row_prefix : A.col_prefix, BY_ROWS ? A.total_rows : A.total_cols,
                [&](const PlanInstance& I, int k, int64_t q0, int count) {
    const double inv = 1.0 / A.eps;
    GroupCost<CK, Q, BY_ROWS> cost(A, I, (float)A.st[k].cost_scale, q0, count);
    const double* other = BY_ROWS ? (first ? A.v0 : A.g) + I.col_off : (first ? A.u0 : A.f) + I.row_off;
    const int64_t len = BY_ROWS ? I.n : I.m;
    Lse acc[Q];
#pragma unroll kWpUnroll
    for (int64_t o = lane; o < len; o += 32) {
      const double h = other[o];
      cost.load(o);
#pragma unroll
      for (int q = 0; q < Q; ++q) acc[q].add((h - cost.get(q, o)) * inv);
    }
    const int64_t off = (BY_ROWS ? I.row_off : I.col_off) + q0;
    const double* mass = (BY_ROWS ? A.a : A.b) + off;
    double* out = (BY_ROWS ? A.f : A.g) + off;
#pragma unroll
    for (int q = 0; q < Q; ++q) {
      acc[q].merge_warp();
      if (lane == q && q < count) {
        const double lse = acc[q].mx + log((double)acc[q].s);
        out[q] = acc[q].mx == -INFINITY ? -INFINITY : A.eps * (log(mass[q]) - lse);
      }
    }
  });
}

// x / eps rounded to nearest, one divisor for many x of either sign (quotient_of); outside
// the range that keeps every term normal, the division itself.
struct OverEps {
  double eps, y;
  bool usable;
  __device__ __forceinline__ explicit OverEps(double e) : eps(e) {
    y = __drcp_rn(e);
    usable = e >= 0x1p-400 && e <= 0x1p+400;
  }
  __device__ __forceinline__ double operator()(double x) const {
    const double ax = fabs(x);
    if (usable && ax >= 0x1p-500 && ax <= 0x1p+500) {
      return quotient_of(x, eps, y);
    }
    return x / eps;
  }
};

// The plan by columns, stored in its type, with the column sums of what is stored.
template <typename TX, int CK, int Q>
__global__ void __launch_bounds__(kWpGroupThreads) k_wp_plan(WarmPlanArgs A) {
  const int lane = threadIdx.x & 31;
  TX* X = static_cast<TX*>(A.X);
  const OverEps over(A.eps);
  for_groups<Q>(A, A.col_prefix, A.total_cols, [&](const PlanInstance& I, int k, int64_t q0, int count) {
    GroupCost<CK, Q, false> cost(A, I, (float)A.st[k].cost_scale, q0, count);
    const double* f = A.f + I.row_off;
    double g[Q], s[Q];
#pragma unroll
    for (int q = 0; q < Q; ++q) {
      g[q] = A.g[I.col_off + q0 + (q < count ? q : count - 1)];
      s[q] = 0.0;
    }
    for (int64_t i = lane; i < I.m; i += 32) {
      const double fi = f[i];
      cost.load(i);
#pragma unroll
      for (int q = 0; q < Q; ++q)
        if (q < count) {
          const TX x = (TX)exp(over(fi + g[q] - cost.get(q, i)));
          X[I.x_off + i + (q0 + q) * I.ld] = x;
          s[q] += (double)x;
        }
    }
#pragma unroll
    for (int q = 0; q < Q; ++q) {
      s[q] = warp_sum(s[q]);
      if (lane == q && q < count) A.c[I.col_off + q0 + q] = s[q];
    }
  });
}

// The stored plan's row sums.
template <typename TX, int Q>
__global__ void __launch_bounds__(kWpGroupThreads) k_wp_row_sums(WarmPlanArgs A) {
  const int lane = threadIdx.x & 31;
  const TX* X = static_cast<const TX*>(A.X);
  for_groups<Q>(A, A.row_prefix, A.total_rows, [&](const PlanInstance& I, int, int64_t q0, int count) {
    double s[Q];
#pragma unroll
    for (int q = 0; q < Q; ++q) s[q] = 0.0;
    const TX* row = X + I.x_off + q0;
#pragma unroll 4
    for (int64_t j = lane; j < I.n; j += 32)
#pragma unroll
      for (int q = 0; q < Q; ++q)
        if (q < count) s[q] += (double)row[j * I.ld + q];
#pragma unroll
    for (int q = 0; q < Q; ++q) {
      s[q] = warp_sum(s[q]);
      if (lane == q && q < count) A.r[I.row_off + q0 + q] = s[q];
    }
  });
}

__global__ void k_wp_copy(const double* __restrict__ src, double* __restrict__ dst, long long count) {
  for (long long e = (long long)blockIdx.x * blockDim.x + threadIdx.x; e < count; e += (long long)gridDim.x * blockDim.x)
    dst[e] = src[e];
}

int wp_grid(long long warps) {
  long long g = (warps + kWpWarps - 1) / kWpWarps;
  return (int)(g < 1 ? 1 : (g > 148 * 16 ? 148 * 16 : g));
}

// CTAs of the group kernels: one per two groups, at most 32 per SM.
int group_grid(long long total, int Q) {
  const long long g = ((total + Q - 1) / Q + kWpGroupWarps - 1) / kWpGroupWarps;
  return (int)(g < 1 ? 1 : (g > 148 * 32 ? 148 * 32 : g));
}

template <int CK, int Q, bool BY_ROWS>
void balance(const WarmPlanArgs& A, int first, cudaStream_t s) {
  k_wp_balance<CK, Q, BY_ROWS>
      <<<group_grid(BY_ROWS ? A.total_rows : A.total_cols, Q), kWpGroupThreads, 0, s>>>(A, first);
}

template <typename TX, int CK>
void warm_plan(const WarmPlanArgs& A, int iterations, cudaStream_t s) {
  constexpr int Q = group_rows(CK);
  const bool rows = grouped(A.total_rows, Q), cols = grouped(A.total_cols, Q);
  for (int it = 0; it < iterations; ++it) {
    rows ? balance<CK, Q, true>(A, it == 0, s) : balance<CK, 1, true>(A, it == 0, s);
    cols ? balance<CK, Q, false>(A, 0, s) : balance<CK, 1, false>(A, 0, s);
  }
  if (cols)
    k_wp_plan<TX, CK, Q><<<group_grid(A.total_cols, Q), kWpGroupThreads, 0, s>>>(A);
  else
    k_wp_plan<TX, CK, 1><<<group_grid(A.total_cols, 1), kWpGroupThreads, 0, s>>>(A);
  k_wp_row_sums<TX, Q><<<group_grid(A.total_rows, Q), kWpGroupThreads, 0, s>>>(A);
}

}  // namespace

cudaError_t launch_warm_plan(const WarmPlanArgs& A, int iterations, cudaStream_t s) {
  // every array the kernels read or write must be in place
  const bool stored = A.kind == PDOT_COST_F64 || A.kind == PDOT_COST_F32 || A.kind == PDOT_COST_BF16;
  if (!A.inst || A.num < 1 || !A.row_prefix || !A.col_prefix || !A.st || !A.a || !A.b || !A.u0 || !A.v0 || !A.f ||
      !A.g || !A.X || !A.r || !A.c || !(A.eps > 0.0) || (stored ? !A.C : (!A.xs || !A.ys || A.dim < 1)))
    return cudaErrorInvalidValue;
  if (iterations <= 0) {
    // the plan from the warm duals themselves
    k_wp_copy<<<wp_grid(A.total_rows), kWpThreads, 0, s>>>(A.u0, A.f, A.total_rows);
    k_wp_copy<<<wp_grid(A.total_cols), kWpThreads, 0, s>>>(A.v0, A.g, A.total_cols);
  }
  // the FP64 plan goes with the FP64 cost, an FP32 plan with every other kind
  if (A.plan_f32 == (A.kind == PDOT_COST_F64)) return cudaErrorInvalidValue;
  switch (A.kind) {
    case PDOT_COST_F64: warm_plan<double, PDOT_COST_F64>(A, iterations, s); break;
    case PDOT_COST_F32: warm_plan<float, PDOT_COST_F32>(A, iterations, s); break;
    case PDOT_COST_BF16: warm_plan<float, PDOT_COST_BF16>(A, iterations, s); break;
    case kCostSqBase + 1: warm_plan<float, kCostSqBase + 1>(A, iterations, s); break;
    case kCostSqBase + 2: warm_plan<float, kCostSqBase + 2>(A, iterations, s); break;
    case kCostSqBase + 3: warm_plan<float, kCostSqBase + 3>(A, iterations, s); break;
    case kCostSqBase + 4: warm_plan<float, kCostSqBase + 4>(A, iterations, s); break;
    case kCostL1Base + 1: warm_plan<float, kCostL1Base + 1>(A, iterations, s); break;
    case kCostL1Base + 2: warm_plan<float, kCostL1Base + 2>(A, iterations, s); break;
    case kCostL1Base + 3: warm_plan<float, kCostL1Base + 3>(A, iterations, s); break;
    case kCostL1Base + 4: warm_plan<float, kCostL1Base + 4>(A, iterations, s); break;
    default: return cudaErrorInvalidValue;
  }
  return cudaGetLastError();
}

}  // namespace pdot
