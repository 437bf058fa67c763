// pdot_resident.cu — the iterations between two evaluations of a small problem as one
// launch that keeps the plan, its average and the cost in shared memory.
//
// A problem of a few megabytes is bound by latency: an iteration of primal pass and dual
// step took 17 us at 1000 x 1000 in FP64 and 12 us at 127 x 93 on B200 as two launches of
// a graph, where 40 MB from L2 take 4 us. Resident it takes 11 and 7.5 us, of which the
// barriers are 2.7 and 2.5, the dual step 2.2 and 1.8, the sums and the control 2.6 and
// 1.6; the primal pass, 3.2 and 1.7, is bound by FP64 issue and shared memory (2.2 k of
// its 6 k cycles at 1000 x 1000) and by the chain of one unit's sums.
//
// Here an iteration has two grid barriers and no launch:
//
//   primal   every CTA range of the primal pass from shared memory; row, column and
//            square partial sums to global memory
//   barrier
//   dual     every block of the dual step, its row sums, duals and averages in
//            registers; new duals and the blocks' sums to global memory. The last CTA
//            adds up the squares meanwhile
//   barrier
//   control  every CTA takes the step rule by itself from the same sums
//
// so nothing is elected, and no CTA waits for another's control. The two halves of a
// CTA (256 threads each) each run one CTA range of the primal pass and one block of the
// dual step, with the same lanes, warps, slots and orders of addition as those
// kernels: iterates, duals and state are the same bit for bit
// (tests/test_gpu_resident.py). What is read between two barriers was written before the
// first of them and is next written after the second.
//
// What counts is the length of the chain: a trip to L2 takes 360 cycles, a release 400
// and more, and lines that every CTA reads at once queue, so the sums are as few as
// they can be. Control by one CTA that publishes the result measured 25 % slower.
//
// What other CTAs wrote is read through L2 (__ldcg): the L1 of an SM may hold the last
// iteration's line.
//
// The CTAs take an SM each, and other work on the GPU may hold some. A cooperative launch
// would wait until all of them are free: a solve of 2.5 ms beside a kernel of one thread
// that runs for 1.6 s took 1.6 s, where the graph takes 3.7 ms. So the launch is an
// ordinary one, and its first barrier finds out whether its CTAs are all resident, as the
// discovery protocol of Sorensen et al. (OOPSLA 2016) does: after kGatherLimitNs without
// the last arrival the CTAs give up, nothing has been changed but partial sums, and the
// host runs the steps as launches of their own. Past the first barrier every CTA is on an
// SM and stays there; the other barriers are bounded by kWaitLimitNs, and a run-out there
// is an error.
#include <type_traits>

#include "pdot_device.cuh"

namespace pdot {
namespace {

constexpr int kHalf = 256;            // threads of a CTA range and of a dual block
constexpr int kResThreads = 2 * kHalf;
constexpr int kResSmem = 227 * 1024;  // shared memory of a CTA
constexpr int kResFixed = 37 * 1024;  // of it, static arrays (row-sum tiles, state)
// 148 CTAs are through their first primal pass 10 to 20 us after the launch; in 200 us a
// short kernel of another stream makes room too, and the SMs are not held longer for nothing.
constexpr unsigned long long kGatherLimitNs = 200000ull;
static_assert(kHalf == kThreads && kHalf == kVecThreads, "a half runs the other kernels' blocks");

__device__ __forceinline__ void half_sync(int half) { asm volatile("bar.sync %0, %1;" ::"r"(half + 1), "n"(kHalf) : "memory"); }

// Arrives and waits until `target` arrivals are counted (the counter is zero at the
// launch), but at most `limit_ns`. The CTA's writes are released by thread 0 after the
// CTA's own barrier, and what the others released is visible to the CTA after it. False
// when this wait or another CTA's ran out: a CTA gives up by setting the counter's top bit
// while arrivals are missing, and by nothing else, so either all CTAs pass a barrier or
// none does. (Each compare-and-swap that fails saw one more arrival.) A CTA that is to
// `give_up` (test hook) does so in place of arriving.
constexpr unsigned kGaveUp = 0x80000000u;  // above every target
__device__ __forceinline__ bool res_barrier(unsigned* count, unsigned target, unsigned long long limit_ns,
                                            bool give_up = false) {
  __shared__ int ok;
  __syncthreads();
  if (threadIdx.x == 0) {
    if (!give_up) asm volatile("red.release.gpu.global.add.u32 [%0], 1;" ::"l"(count) : "memory");
    int it = 0;
    unsigned long long t0 = 0;
    bool late = give_up;
    for (;;) {
      const unsigned seen = ld_acquire_gpu(count);
      if (seen >= target) {
        ok = (seen & kGaveUp) == 0;
        break;
      }
      if (late && atomicCAS(count, seen, seen | kGaveUp) == seen) {
        ok = 0;
        break;
      }
      if ((++it & 15) == 0) {
        const unsigned long long t = globaltimer_ns();
        if (t0 == 0) t0 = t;
        late |= t - t0 > limit_ns || it >= kSpinLimit;
      }
    }
  }
  __syncthreads();
  return ok != 0;
}

// sum_strided through L2
__device__ __forceinline__ double sum_strided_cg(const double* q, int64_t count, int64_t stride) {
  double s = 0.0;
  int64_t c = 0;
  for (; c + 8 <= count; c += 8) {
    double v[8];
#pragma unroll
    for (int k = 0; k < 8; ++k) v[k] = __ldcg(q + (c + k) * stride);
#pragma unroll
    for (int k = 0; k < 8; ++k) s += v[k];
  }
  for (; c < count; ++c) s += __ldcg(q + c * stride);
  return s;
}

// Bytes of a unit in shared memory: `rows` of the stored cost, the plan and the average.
__host__ __device__ __forceinline__ int unit_rows(int64_t m) {
  return m < kPanelRows ? (int)((m + 15) / 16 * 16) : kPanelRows;
}

// SPLIT: a unit's column and square sums by row load, added in load order at the end, as
// the staged primal pass has them; else one chain over the unit, as the direct pass.
template <typename TX, int CK, int R, bool SPLIT>
__global__ void __launch_bounds__(kResThreads, 1)
    k_resident(Buffers B, Geometry g, SolveConfig cfg, int steps, unsigned* bar) {
  constexpr int RPL = kPanelRows / (32 * R);
  constexpr bool kPts = is_point_cost(CK);
  using Reader = CostReader<CK, R, RPL>;
  using TC = typename Reader::value_t;
  extern __shared__ __align__(128) unsigned char smem[];
  __shared__ double red[2][kWarps][kPanelRows];
  __shared__ double us[2][kPanelRows];  // the range's source duals of a panel, loaded once for its warps
  __shared__ double sqw[2][kWarps], shv[2][kWarps][kStepSums];
  __shared__ double fin[2 * kStepSums + 1], sc[4];  // s, nw, aw, tw
  double* sqsum = reinterpret_cast<double*>(bar) + 1;  // total of the square sums
  __shared__ int sflags[2];                         // first average, zero gradient
  __shared__ StepPowers pw;
  __shared__ DevState loc;
  DevState* st = B.st;
  // One answer for the CTA: done and numerical_error stay as they are until every CTA is
  // here, but a CTA whose wait ran out may set kernel_error while this one starts, and
  // warps that left on it would be missed for good by the others' named barriers.
  if (__syncthreads_or(st->done | st->numerical_error | st->kernel_error)) return;
  const int buf = st->buf;
  const int half = threadIdx.x / kHalf, tid = threadIdx.x % kHalf, lane = tid & 31, warp = tid >> 5;
  const int64_t m = g.m, n = g.n, vcta = (int64_t)blockIdx.x * 2 + half;
  const unsigned ctas = gridDim.x;
  TX* X = static_cast<TX*>(B.X[buf]);
  TX* Xa = static_cast<TX*>(B.X[buf ^ 1]);
  double *u = B.u[buf], *v = B.v[buf];
  const bool active = vcta < g.grid;
  const int64_t q0 = active ? unit_begin(g, vcta) : 0, q1 = active ? unit_begin(g, vcta + 1) : 0;
  const int ur_rows = unit_rows(m);
  const int xb = ur_rows * (int)sizeof(TX), cb = kPts ? 0 : ur_rows * (int)sizeof(TC), ub = cb + 2 * xb;
  unsigned char* data = smem + (size_t)half * ((g.units + g.grid - 1) / g.grid) * ub;
  auto unit_ptr = [&](int64_t q) { return data + (q - q0) * ub; };

  // the range's units, a warp per unit: average, plan and cost
  auto each_unit = [&](auto&& f) {
    for (int64_t q = q0 + warp; q < q1; q += kWarps) {
      const int64_t p = q / n, j = q - p * n, row0 = p * kPanelRows;
      unsigned char* s = unit_ptr(q);
#pragma unroll
      for (int k = 0; k < RPL; ++k) {
        const int r = k * 32 * R + lane * R;
        if (row0 + r < m) f(s, r, j * m + row0 + r);
      }
    }
  };
  each_unit([&](unsigned char* s, int r, int64_t at) {
    TX x[R];
    if constexpr (!kPts) {
      TC c[R];
      vldg<TC, R>(static_cast<const TC*>(B.cost.C) + at, c);
      vst<TC, R>(reinterpret_cast<TC*>(s) + r, c);
    }
    vldcg<TX, R>(X + at, x);
    vst<TX, R>(reinterpret_cast<TX*>(s + cb) + r, x);
    vldcg<TX, R>(Xa + at, x);
    vst<TX, R>(reinterpret_cast<TX*>(s + cb + xb) + r, x);
  });

  // this thread's entry of the dual step: row or column `oi`, a warp's lane 0 or a thread
  const int64_t bid = vcta;
  const bool in_dual = bid < g.dual_row_blocks + g.col_blocks;
  const bool is_row = bid < g.dual_row_blocks;
  const bool by_warp = is_row && g.dual_row_blocks != g.row_blocks;
  const int64_t oi = by_warp ? bid * kWarps + warp : (is_row ? bid : bid - g.dual_row_blocks) * kHalf + tid;
  const bool valid = in_dual && oi < (is_row ? m : n);
  const bool own = valid && (!by_warp || lane == 0);
  double* osum[2] = {(is_row ? B.r : B.c)[buf], (is_row ? B.r : B.c)[buf ^ 1]};
  double* odual[2] = {is_row ? u : v, (is_row ? B.u : B.v)[buf ^ 1]};
  double o_dist = 0.0, o_sum = 0.0, o_dual = 0.0, o_sum_avg = 0.0, o_dual_avg = 0.0;
  if (own) {
    o_dist = (is_row ? B.a : B.b)[oi];
    o_sum = __ldcg(osum[0] + oi);
    o_dual = __ldcg(odual[0] + oi);
    o_sum_avg = __ldcg(osum[1] + oi);
    o_dual_avg = __ldcg(odual[1] + oi);
  }
  const double* part = nullptr;  // its partial sums, `parts` of them, `stride` apart
  int64_t parts = 0, stride = 0;
  if (valid && is_row) {
    const int64_t p = oi / kPanelRows, t = oi - p * kPanelRows;
    const int64_t lo = cta_of_unit(g, p * n), hi = cta_of_unit(g, (p + 1) * n - 1);
    part = B.rowpart + row_slot(lo, p) * kPanelRows + t;
    parts = hi - lo + 1;
    stride = kPanelRows;
  } else if (valid) {
    part = B.colpart + oi;
    parts = g.panels;
    stride = n;
  }

  // the step's weights of the state at hand: the three quotients by three lanes at once
  auto weights = [&] {
    const double tau = loc.step_size, omega = loc.primal_weight, S = loc.sum_weights;
    const bool first = !(S > 0.0);
    if (lane < 3) {
      const double q = __ddiv_rn(lane == 2 ? S : tau, lane == 0 ? omega : lane == 1 ? S : __dadd_rn(S, tau));
      sc[lane] = lane > 0 && first ? 1.0 : q;
    } else if (lane == 3) {
      sc[3] = __dmul_rn(tau, omega);
      sflags[0] = first;
      sflags[1] = loc.g_is_zero != 0;
    }
  };
  if (threadIdx.x < 32) {
    if (lane == 0) loc = *st;
    __syncwarp();
    weights();
  }
  Reader cost(B.cost, (float)st->cost_scale);
  const int64_t p_first = active ? q0 / n : 0;
  const bool one_panel = q1 <= (p_first + 1) * n;
  {
    bool ok[RPL];
#pragma unroll
    for (int k = 0; k < RPL; ++k) ok[k] = p_first * kPanelRows + k * 32 * R + lane * R < m;
    cost.panel(p_first * kPanelRows, lane, m, ok);
  }
  // the next pass's first duals and column, loaded while the control runs
  double un = 0.0, vn = 0.0;
  auto fetch = [&] {
    if (!active) return;
    const int64_t i = p_first * kPanelRows + tid;
    un = i < m ? __ldcg(u + i) : 0.0;
    const int64_t j = q0 - p_first * n + warp;
    if (j < n && p_first * n + j < q1) {
      vn = __ldcg(v + j);
      cost.prefetch(j);
    }
  };
  fetch();
  __syncthreads();

  unsigned round = 0;
  bool alive = true;
  for (int step = 0; step < steps; ++step) {
    const bool first = sflags[0] != 0, zero_g = sflags[1] != 0;
    const double s = sc[0], nw = sc[1], aw = sc[2];
    // PLAIN: every pass but a solve's first and those after an average reset
    auto primal = [&](auto plain) {
      constexpr bool PLAIN = decltype(plain)::value;
      const bool first = !PLAIN && sflags[0] != 0, zero_g = !PLAIN && sflags[1] != 0;
      double sq[SPLIT ? RPL : 1];
#pragma unroll
      for (int k = 0; k < (SPLIT ? RPL : 1); ++k) sq[k] = 0.0;
      for (int64_t p = p_first; p * n < q1; ++p) {
        const int64_t jb = (q0 > p * n ? q0 : p * n) - p * n;
        const int64_t je = (q1 < (p + 1) * n ? q1 : (p + 1) * n) - p * n;
        const int64_t row0 = p * kPanelRows;
        double acc[RPL][R];
        TX ur[RPL][R];
        bool ok[RPL];
        us[half][tid] = p == p_first ? un : (row0 + tid < m ? __ldcg(u + row0 + tid) : 0.0);
        half_sync(half);
#pragma unroll
        for (int k = 0; k < RPL; ++k) {
          ok[k] = row0 + k * 32 * R + lane * R < m;
#pragma unroll
          for (int e = 0; e < R; ++e) {
            acc[k][e] = 0.0;
            ur[k][e] = (ok[k] && !zero_g) ? (TX)us[half][k * 32 * R + lane * R + e] : (TX)0;
          }
        }
        if (!one_panel) cost.panel(row0, lane, m, ok);
        for (int64_t j = jb + warp; j < je; j += kWarps) {
          const bool ahead = p == p_first && j == jb + warp;
          const double vj = zero_g ? 0.0 : (ahead ? vn : __ldcg(v + j));
          if (ahead)
            cost.take();
          else
            cost.column(j);
          unsigned char* su = unit_ptr(p * n + j);
          double cs[SPLIT ? RPL : 1];
#pragma unroll
          for (int k = 0; k < (SPLIT ? RPL : 1); ++k) cs[k] = 0.0;
#pragma unroll
          for (int k = 0; k < RPL; ++k) {
            if (ok[k]) {
              const int r = k * 32 * R + lane * R;
              TX* px = reinterpret_cast<TX*>(su + cb) + r;
              TX* pa = reinterpret_cast<TX*>(su + cb + xb) + r;
              TC cv[R];
              TX xv[R], av[R];
              if constexpr (kPts)
                cost.get(0, k, cv);
              else
                vld<TC, R>(reinterpret_cast<const TC*>(su) + r, cv);
              vld<TX, R>(px, xv);
              if (!first) vld<TX, R>(pa, av);
              constexpr int q = SPLIT ? 1 : 0;
#pragma unroll
              for (int e = 0; e < R; ++e) {
                double d;
                primal_entry<TX>(widen(cv[e]), ur[k][e], vj, s, nw, aw, zero_g, first, xv[e], av[e], d);
                acc[k][e] += d;
                cs[q * k] += d;
                add_sq<TX>(sq[q * k], d);
              }
              vst<TX, R>(px, xv);
              vst<TX, R>(pa, av);
            }
          }
          double col = cs[0];
#pragma unroll
          for (int k = 1; k < (SPLIT ? RPL : 1); ++k) col += cs[k];
          col = warp_sum(col);
          if (lane == 0) B.colpart[p * n + j] = col;
        }
#pragma unroll
        for (int k = 0; k < RPL; ++k)
#pragma unroll
          for (int e = 0; e < R; ++e) red[half][warp][k * 32 * R + lane * R + e] = acc[k][e];
        half_sync(half);
        double s2 = red[half][0][tid];
#pragma unroll
        for (int w = 1; w < kWarps; ++w) s2 += red[half][w][tid];
        B.rowpart[row_slot(vcta, p) * kPanelRows + tid] = s2;
        half_sync(half);
      }
      double sqs = sq[0];
#pragma unroll
      for (int k = 1; k < (SPLIT ? RPL : 1); ++k) sqs += sq[k];
      sqs = warp_sum(sqs);
      if (lane == 0) sqw[half][warp] = sqs;
      half_sync(half);
      if (tid == 0) {
        double s2 = sqw[half][0];
#pragma unroll
        for (int w = 1; w < kWarps; ++w) s2 += sqw[half][w];
        B.sqpart[vcta] = s2;
      }
    };
    if (active) {
      if (first || zero_g)
        primal(std::false_type());
      else
        primal(std::true_type());
    }
    ++round;
    if (!(alive = res_barrier(bar, ctas * round, round == 1 ? kGatherLimitNs : kWaitLimitNs))) break;

    if (in_dual) {
      DualArgs A;
      A.first = first;
      A.tw = sc[3];
      A.nw = nw;
      A.aw = aw;
      double vals[kStepSums] = {0.0, 0.0};
      double sd = 0.0;
      if (by_warp) {
        for (int64_t c = lane; c < parts; c += 128) {  // four trips to L2 at once
          double q[4];
#pragma unroll
          for (int k = 0; k < 4; ++k) q[k] = c + 32 * k < parts ? __ldcg(part + (c + 32 * k) * stride) : 0.0;
#pragma unroll
          for (int k = 0; k < 4; ++k) sd += q[k];
        }
        sd = warp_sum(sd);
      } else if (own) {
        sd = sum_strided_cg(part, parts, stride);
      }
      if (own) {
        dual_entry(sd, o_dist, &o_sum, &o_dual, &o_sum_avg, &o_dual_avg, A, vals[0], vals[1]);
        odual[0][oi] = o_dual;
      }
      // a warp per row: its other lanes hold zeros, the sum is lane 0's
      if (!by_warp) vals[0] = warp_sum(vals[0]), vals[1] = warp_sum(vals[1]);
      if (lane == 0) shv[half][warp][0] = vals[0], shv[half][warp][1] = vals[1];
      half_sync(half);
      if (tid < kStepSums) {
        double x = shv[half][0][tid];
#pragma unroll
        for (int w = 1; w < kWarps; ++w) x = x + shv[half][w][tid];
        B.steppart[bid * kStepSums + tid] = x;
      }
    }
    if (blockIdx.x == ctas - 1 && threadIdx.x >= kResThreads - 32) {
      double xs[1];
      warp_reduce_partials<1>(B.sqpart, 0, g.grid, 0u, xs);
      if (lane == 0) *sqsum = xs[0];
    }
    const bool give_up = g.fail_waits && blockIdx.x == 0;
    if (!(alive = res_barrier(bar, ctas * ++round, kWaitLimitNs, give_up))) break;

    fetch();
    if (threadIdx.x < 32) {
      double rs[kStepSums];
      warp_reduce_partials<kStepSums>(B.steppart, 0, g.dual_row_blocks, 0u, rs);
      if (lane == 0) fin[0] = rs[0], fin[1] = rs[1];
    } else if (threadIdx.x < 64) {
      double cs[kStepSums];
      warp_reduce_partials<kStepSums>(B.steppart, g.dual_row_blocks, g.col_blocks, 0u, cs);
      if (lane == 0) fin[2] = cs[0], fin[3] = cs[1];
    } else if (threadIdx.x == 64) {
      fin[4] = __ldcg(sqsum);
    } else if (threadIdx.x == 96) {
      pw = step_powers(&loc, cfg);
    }
    __syncthreads();
    if (threadIdx.x < 32) {
      // step_control with the two norms taken by two lanes at once
      const double nrm = sqrt(lane == 0 ? fin[4] : fin[1] + fin[3]);
      const double interaction = fabs(fin[0] + fin[2]);
      const double movement = step_movement(loc.primal_weight, pw.half_over_omega, __shfl_sync(0xffffffffu, nrm, 0),
                                            __shfl_sync(0xffffffffu, nrm, 1));
      const double limit = step_limit(movement, interaction);
      if (lane == 0) step_attempts(&loc, cfg, interaction, movement, limit, pw);
      __syncwarp();
      weights();
    }
    __syncthreads();
    if (loc.numerical_error) break;  // the same in every CTA
  }
  if (!alive) {
    // before the first barrier only partial sums were written
    if (threadIdx.x == 0) atomicExch(&st->kernel_error, round == 1 ? kNotStarted : kWaitRanOut);
    return;
  }
  each_unit([&](unsigned char* s2, int r, int64_t at) {
    TX x[R];
    vld<TX, R>(reinterpret_cast<const TX*>(s2 + cb) + r, x);
    vst<TX, R>(X + at, x);
    vld<TX, R>(reinterpret_cast<const TX*>(s2 + cb + xb) + r, x);
    vst<TX, R>(Xa + at, x);
  });
  if (own) {
    osum[0][oi] = o_sum;
    osum[1][oi] = o_sum_avg;
    odual[1][oi] = o_dual_avg;
  }
  if (blockIdx.x == 0 && threadIdx.x == 0) {
    st->step_size = loc.step_size;
    st->kkt_passes = loc.kkt_passes;
    st->sum_weights = loc.sum_weights;
    st->avg_count = loc.avg_count;
    st->total_iters = loc.total_iters;
    st->iteration = loc.iteration;
    st->g_is_zero = loc.g_is_zero;
    st->numerical_error = loc.numerical_error;
    st->primal_passes = loc.primal_passes;
    st->fresh_passes = loc.fresh_passes;
  }
}

// Expands to the variant of geometry `g` (PDOT_VARIANT's cost sources and load widths;
// the staged order only where the primal pass is staged).
#define PDOT_RES_KIND(g, TX, CK, VEC, LAUNCH)                                  \
  do {                                                                         \
    if ((g).tma) { auto kfn = k_resident<TX, CK, VEC, true>; LAUNCH; }         \
    else if ((g).vec > 1) { auto kfn = k_resident<TX, CK, VEC, false>; LAUNCH; } \
    else { auto kfn = k_resident<TX, CK, 1, false>; LAUNCH; }                  \
  } while (0)
#define PDOT_RES_VARIANT(g, LAUNCH)                                                                    \
  do {                                                                                                 \
    if (!(g).plan_f32) PDOT_RES_KIND(g, double, PDOT_COST_F64, 2, LAUNCH);                             \
    else switch ((g).cost_kind) {                                                                      \
      case PDOT_COST_F32: PDOT_RES_KIND(g, float, PDOT_COST_F32, 4, LAUNCH); break;                    \
      case PDOT_COST_BF16: PDOT_RES_KIND(g, float, PDOT_COST_BF16, 4, LAUNCH); break;                  \
      case kCostSqBase + 1: PDOT_RES_KIND(g, float, kCostSqBase + 1, 4, LAUNCH); break;                \
      case kCostSqBase + 2: PDOT_RES_KIND(g, float, kCostSqBase + 2, 4, LAUNCH); break;                \
      case kCostSqBase + 3: PDOT_RES_KIND(g, float, kCostSqBase + 3, 4, LAUNCH); break;                \
      case kCostSqBase + 4: PDOT_RES_KIND(g, float, kCostSqBase + 4, 4, LAUNCH); break;                \
      case kCostL1Base + 1: PDOT_RES_KIND(g, float, kCostL1Base + 1, 4, LAUNCH); break;                \
      case kCostL1Base + 2: PDOT_RES_KIND(g, float, kCostL1Base + 2, 4, LAUNCH); break;                \
      case kCostL1Base + 3: PDOT_RES_KIND(g, float, kCostL1Base + 3, 4, LAUNCH); break;                \
      default: PDOT_RES_KIND(g, float, kCostL1Base + 4, 4, LAUNCH); break;                             \
    }                                                                                                  \
  } while (0)

int cost_bytes(const Geometry& g) {
  return !g.plan_f32 ? 8 : g.cost_kind == PDOT_COST_F32 ? 4 : g.cost_kind == PDOT_COST_BF16 ? 2 : 0;
}

size_t resident_smem(const Geometry& g) {
  const size_t unit = (size_t)unit_rows(g.m) * (cost_bytes(g) + 2 * (g.plan_f32 ? 4 : 8));
  return 2 * (size_t)((g.units + g.grid - 1) / g.grid) * unit;
}

}  // namespace

// The CTAs of the resident steps, 0 where they cannot run: the two CTA ranges of a CTA
// must fit its shared memory (some 1.1 M entries in FP64, 3.6 M with an FP32 plan and
// coordinate costs), every block of the dual step a half of its own, and all CTAs an
// otherwise idle device at once. Over that range they are as fast as the graph or faster,
// us per iteration against the graph's: FP64 6.6 and 8.9 at 16 x 16, 9.5 and 15.1 at 256 x
// 256, 10.7 and 14.9 at 1000 x 1000, 12.2 and 15.0 at 100 x 8000, 10.4 and 14.1 at 8000 x
// 100, 14.9 and 15.3 at 2400 x 440; an FP32 plan with an FP32 cost 7.8 and 10.2 at 127 x
// 93, 11.4 and 17.3 at 1200 x 1200, with a BF16 cost 12.6 and 19.6 at 1300 x 1300, with
// planar coordinates 10.2 and 14.9 at 1000 x 1000, 14.6 and 18.5 at 1500 x 1500, 21.2 and
// 21.3 at 1800 x 1800, 24.9 and 24.7 at 300 x 10000; single-row loads 10.6 and 14.3 at
// 1023 x 1021 in FP64, 14.5 and 18.8 at 1501 x 1499 from planar coordinates.
int resident_ctas(const Geometry& g, int device) {
  const int ctas = (g.grid + 1) / 2;
  if (g.dual_row_blocks + g.col_blocks > 2 * ctas) return 0;
  const size_t smem = resident_smem(g);
  if (smem > (size_t)(kResSmem - kResFixed)) return 0;
  int sms = 0, occ = 0;
  if (cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, device) != cudaSuccess) sms = 0;
  PDOT_RES_VARIANT(g, {
    if (cudaFuncSetAttribute(kfn, cudaFuncAttributeMaxDynamicSharedMemorySize, kResSmem - kResFixed) != cudaSuccess ||
        cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ, kfn, kResThreads, smem) != cudaSuccess)
      occ = 0;
  });
  cudaGetLastError();
  return (int64_t)occ * sms >= ctas ? ctas : 0;
}

size_t resident_scratch_bytes() { return 64; }

cudaError_t launch_resident(const Buffers& B, const Geometry& g, const SolveConfig& cfg, cudaStream_t s, int ctas,
                            int steps, void* scratch) {
  // two arrivals of every CTA a step stay below the counter's top bit
  if (steps < 1 || steps > kMaxResidentSteps || (int64_t)ctas * 2 * steps >= (int64_t)kGaveUp) return cudaErrorInvalidValue;
  unsigned* bar = static_cast<unsigned*>(scratch);
  cudaError_t e = cudaMemsetAsync(bar, 0, sizeof(unsigned), s);
  if (e != cudaSuccess) return e;
  Buffers b = B;
  Geometry gg = g;
  SolveConfig c = cfg;
  void* args[] = {&b, &gg, &c, &steps, &bar};
  PDOT_RES_VARIANT(g, (e = cudaLaunchKernel((const void*)kfn, dim3((unsigned)ctas), dim3(kResThreads), args,
                                            resident_smem(g), s)));
  return e;
}

}  // namespace pdot
