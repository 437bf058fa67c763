// pdot_multiscale.cu — device passes of the coarse-to-fine warm start for
// point clouds (pdot/multiscale.py): the largest squared distance between two
// point sets, which normalises the squared-Euclidean cost, and the
// semi-discrete c-transform that extends duals known on coarse cells to every
// point, u_i = min_J (scale * ||x_i - c_J||^2 - V_J).
//
// Both visit every pair, but only pairs that can decide the result are computed in
// FP64. A pass over a tile of the second set in FP32 finds what the tile holds for a
// point, to a known error; where that cannot beat the best value so far by more than
// the error, the tile is done, and else the FP64 values of the pairs within the error
// are taken. The results are those of FP64 throughout, bit for bit (a maximum and a
// minimum do not depend on the pairs that are left out). FP64 arithmetic was what
// bounded them: B200 does two FP32 operations for one in FP64, and none of the FP32
// ones needs the conversions. The FP32 pass is bound by issue, so it does two pairs in
// an instruction and one comparison for two distances; the c-transform keeps the
// minima of groups of eight centres, and which groups hold the smallest ones, in place
// of every centre's. 20000 x 15000 points in the plane: the maximum 80 us a pair at a
// time, 60 this way (the FP32 operations alone take 33); 20000 points against 6000
// centres: 96 and 53 (17).
//
// The second set is split over CTAs too, so that 20000 points, 79 CTAs of 256, fill
// the 148 SMs: the maximum by atomicMax, the minimum by a cluster's shared memory. Tiles
// of 128 points for the maximum, which took 74 us with 512, and of 256 centres, which
// took 58 with 128.
#include <cooperative_groups.h>

#include <cfloat>
#include <cmath>

#include "pdot_common.cuh"
#include "pdot_pairs.cuh"

namespace pdot {
namespace {

constexpr int kFarTile = 128;   // points of the second set per shared-memory tile of the maximum
constexpr int kTile = 256;      // and of the c-transform
constexpr int kMaxThreads = 256;  // threads of a CTA of the maximum
constexpr int kMinThreads = 128;  // and of the c-transform
constexpr int kGroup = 8;       // centres whose minimum the c-transform takes as one
constexpr int kPointsPer = 2;   // points of the first set per thread: a tile entry read once serves both
constexpr int kSplit = 8;       // CTAs of a cluster, each with a share of the centres

// Threads keep max_j ||x_i - y_j||^2 of their points (FP64 from FP32 coordinates) over a
// share of the y_j; a CTA reduces its threads and one atomicMax on the bit pattern
// combines the CTAs (non-negative doubles order like their bit patterns).
//
// The FP32 distance of FP32 points has a relative error below (D + 3) 2^-24, and below
// 1e-36 from underflow, so a tile's FP32 maximum t holds an FP64 distance of at least
// t (1 - 2e-6) - 1e-30 and none above t (1 + 2e-6) + 1e-30. Threads whose upper bound
// stays below the CTA's largest lower bound (or below the result so far) are done with
// the tile; the others take its FP64 distances. Which threads those are can differ
// from run to run, the maximum cannot.
template <int D>
__global__ void __launch_bounds__(kMaxThreads) k_max_sqdist(int64_t m, int64_t n, int64_t share, const float* __restrict__ xs,
                                                      const float* __restrict__ ys,
                                                      unsigned long long* __restrict__ out_bits) {
  __shared__ __align__(16) float ty[D][kFarTile];
  __shared__ double red[kMaxThreads / 32];
  __shared__ float sbest;  // a lower bound of the result
  float xi[kPointsPer][D];
  unsigned long long minus[kPointsPer][D];
  bool ok[kPointsPer];
#pragma unroll
  for (int q = 0; q < kPointsPer; ++q) {
    const int64_t i = ((int64_t)blockIdx.x * kPointsPer + q) * kMaxThreads + threadIdx.x;
    ok[q] = i < m;
#pragma unroll
    for (int d = 0; d < D; ++d) {
      xi[q][d] = ok[q] ? xs[i * D + d] : 0.0f;
      minus[q][d] = pack2(-xi[q][d], -xi[q][d]);
    }
  }
  double best = 0.0;
  if (threadIdx.x == 0)
    sbest = __double2float_rd(__longlong_as_double((long long)*reinterpret_cast<volatile unsigned long long*>(out_bits)));
  const int64_t jb = (int64_t)blockIdx.y * share, je = (jb + share < n) ? jb + share : n;
  for (int64_t j0 = jb; j0 < je; j0 += kFarTile) {
    const int cnt = (int)((je - j0) < kFarTile ? (je - j0) : kFarTile);
    __syncthreads();
    // the entries past the last point repeat it
    for (int t = threadIdx.x; t < kFarTile * D; t += kMaxThreads) {
      const int j = t / D < cnt ? t / D : cnt - 1;
      ty[t % D][t / D] = ys[(j0 + j) * D + t % D];
    }
    __syncthreads();
    float top[kPointsPer];
#pragma unroll
    for (int q = 0; q < kPointsPer; ++q) top[q] = -1.0f;
#pragma unroll 2
    for (int t = 0; t < cnt; t += 4) {
      ulonglong2 c[D];
#pragma unroll
      for (int d = 0; d < D; ++d) c[d] = *reinterpret_cast<const ulonglong2*>(&ty[d][t]);
#pragma unroll
      for (int q = 0; q < kPointsPer; ++q) top[q] = max_sqdist4<D>(minus[q], c, top[q]);
    }
    // the bits of non-negative floats order as the floats do
    float lower = 0.0f;
#pragma unroll
    for (int q = 0; q < kPointsPer; ++q)
      if (ok[q] && top[q] < INFINITY) lower = fmaxf(lower, top[q] * 0.999998f - 1e-30f);
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) lower = fmaxf(lower, __shfl_xor_sync(0xffffffffu, lower, o));
    if ((threadIdx.x & 31) == 0) atomicMax(reinterpret_cast<int*>(&sbest), __float_as_int(lower));
    __syncthreads();
    const float lim = sbest;
#pragma unroll
    for (int q = 0; q < kPointsPer; ++q) {
      // a tile of NaNs leaves top at -1 and has nothing to offer
      if (!ok[q] || top[q] < 0.0f || top[q] * 1.000002f + 1e-30f < lim) continue;
      for (int t = 0; t < cnt; t += 4) {
        ulonglong2 c[D];
#pragma unroll
        for (int d = 0; d < D; ++d) c[d] = *reinterpret_cast<const ulonglong2*>(&ty[d][t]);
        if (max_sqdist4<D>(minus[q], c, -1.0f) * 1.000002f + 1e-30f < lim) continue;
#pragma unroll
        for (int k = 0; k < 4; ++k) {
          double s = 0.0;
#pragma unroll
          for (int d = 0; d < D; ++d) {
            const double e = (double)xi[q][d] - (double)ty[d][t + k];
            s += e * e;
          }
          best = s > best ? s : best;
        }
      }
    }
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    const double y = __shfl_xor_sync(0xffffffffu, best, o);
    best = y > best ? y : best;
  }
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = best;
  __syncthreads();
  if (threadIdx.x == 0) {
    double b = red[0];
    for (int w = 1; w < kMaxThreads / 32; ++w) b = red[w] > b ? red[w] : b;
    atomicMax(out_bits, (unsigned long long)__double_as_longlong(b));
  }
}

// out_i = min_J (scale * ||p_i - c_J||^2 - dual_J), p in FP32, centres and duals in
// FP64, arithmetic in FP64. The CTAs of a cluster take the centres of a point block in
// equal shares; the cluster's first CTA reads the others' minima from their shared
// memory.
//
// What FP32 makes of a pair (centre, dual and scale rounded to it): with u = 2^-24 and A =
// |p|_max + |c|_max over the tile, a coordinate difference errs by at most 2 u A, the
// squared distance s by 4 u A sqrt(D s) + 4 D u^2 A^2 + 4 u s, the value scale s - v by
// |scale| times that, another 2 u |scale| s and u (|v| + |value|). Where the scale is
// positive a pair whose value is at most x has scale s <= x + V, V = |dual|_max, so that
// error(x) below, twice the sum and more, holds for every pair that counts; it is some
// twenty times less than with the largest distance for s, which let through many more
// pairs on the line (20000 points and 6000 centres with the duals 0.3 c^2 + 0.1 c: 141 us
// then, 131 now, 121 in FP64 throughout; with duals of 1e-3 51, 41 and 121). A pair whose FP32 value exceeds
// M + error(M), M = min(best so far, tile's FP32 minimum + its error), cannot be the
// minimum: only the groups whose minima are within that are taken up again, at most two,
// or the whole tile where a third one is.
//
// The screen's coordinates are taken relative to the first centre, so that A is the
// extent of the points and not their distance from the origin: for points of a unit
// square at (1000, 1000) the error would let most pairs through (3000 centres, 5000
// points: 109 us, 19 this way, 82 in FP64 throughout). No pair is left out where a bound
// is not finite, where a distance may exceed FP32 (the screen's infinity is then a finite
// value times a small scale), or where the scale is below the normal FP32 numbers and
// errs by more than a rounding.
template <int D>
__global__ void __cluster_dims__(1, kSplit, 1) __launch_bounds__(kMinThreads)
    k_c_transform(int64_t np, int64_t nc, const float* __restrict__ pts, const double* __restrict__ centres,
                  const double* __restrict__ duals, double scale, double* __restrict__ out) {
  __shared__ double tc[kTile * D];
  __shared__ double tv[kTile];
  __shared__ __align__(16) float fc[D][kTile];
  __shared__ __align__(16) float fv[kTile];  // minus the duals
  __shared__ int bound_c, bound_v;  // bits of the tile's |c|_max and |dual|_max
  __shared__ double part[kMinThreads * kPointsPer];
  float p[kPointsPer][D], reach[kPointsPer];
  unsigned long long minus[kPointsPer][D];
  double best[kPointsPer], origin[D];
  bool ok[kPointsPer];
#pragma unroll
  for (int d = 0; d < D; ++d) origin[d] = fabs(centres[d]) < INFINITY ? centres[d] : 0.0;
#pragma unroll
  for (int q = 0; q < kPointsPer; ++q) {
    const int64_t i = ((int64_t)blockIdx.x * kPointsPer + q) * kMinThreads + threadIdx.x;
    ok[q] = i < np;
    best[q] = INFINITY;
    reach[q] = 0.0f;
#pragma unroll
    for (int d = 0; d < D; ++d) {
      p[q][d] = ok[q] ? pts[i * D + d] : 0.0f;
      const float f = ok[q] ? (float)((double)p[q][d] - origin[d]) : 0.0f;
      reach[q] = fmaxf(reach[q], fabsf(f));
      minus[q][d] = pack2(-f, -f);
    }
  }
  const float sc = (float)scale;
  const unsigned long long sc2 = pack2(sc, sc);
  const bool screened = scale == 0.0 || (fabsf(sc) >= FLT_MIN && fabsf(sc) < INFINITY);
  const int64_t share = (nc + kSplit - 1) / kSplit;
  const int64_t jb = (int64_t)blockIdx.y * share, je = (jb + share < nc) ? jb + share : nc;
  for (int64_t j0 = jb; j0 < je; j0 += kTile) {
    const int cnt = (int)((je - j0) < kTile ? (je - j0) : kTile);
    __syncthreads();
    if (threadIdx.x == 0) bound_c = bound_v = 0;
    __syncthreads();
    float mc = 0.0f, mv = 0.0f;
    bool odd = false;  // a value that FP32 cannot hold or that is not a number
    for (int t = threadIdx.x; t < cnt * D; t += kMinThreads) {
      const double c = centres[j0 * D + t];
      double o = origin[0];
#pragma unroll
      for (int d = 1; d < D; ++d) o = t % D == d ? origin[d] : o;
      const float f = (float)(c - o);
      tc[t] = c;
      fc[t % D][t / D] = f;
      mc = fmaxf(mc, fabsf(f));
      odd |= !(fabsf(f) < INFINITY);
    }
    for (int t = threadIdx.x; t < cnt; t += kMinThreads) {
      const double v = duals[j0 + t];
      const float f = (float)v;
      tv[t] = v;
      fv[t] = -f;
      mv = fmaxf(mv, fabsf(f));
      odd |= !(fabsf(f) < INFINITY);
    }
    // a last group is filled up with centres that are never the smallest
    if (const int t = cnt + (int)threadIdx.x; t < ((cnt + kGroup - 1) / kGroup) * kGroup) {
      fv[t] = INFINITY;
#pragma unroll
      for (int d = 0; d < D; ++d) fc[d][t] = 0.0f;
    }
    if (odd) mc = INFINITY;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      mc = fmaxf(mc, __shfl_xor_sync(0xffffffffu, mc, o));
      mv = fmaxf(mv, __shfl_xor_sync(0xffffffffu, mv, o));
    }
    if ((threadIdx.x & 31) == 0) {
      atomicMax(&bound_c, __float_as_int(mc));
      atomicMax(&bound_v, __float_as_int(mv));
    }
    __syncthreads();
    // the three smallest minima of a group and where the first two are
    float low[kPointsPer], next[kPointsPer], third[kPointsPer];
    int at[kPointsPer], at2[kPointsPer];
#pragma unroll
    for (int q = 0; q < kPointsPer; ++q) {
      low[q] = next[q] = third[q] = INFINITY;
      at[q] = at2[q] = 0;
    }
    for (int t = 0; t < cnt; t += kGroup) {
      float least[kPointsPer];
#pragma unroll
      for (int h = 0; h < kGroup; h += 4) {
        ulonglong2 c[D];
#pragma unroll
        for (int d = 0; d < D; ++d) c[d] = *reinterpret_cast<const ulonglong2*>(&fc[d][t + h]);
        const ulonglong2 w = *reinterpret_cast<const ulonglong2*>(&fv[t + h]);
#pragma unroll
        for (int q = 0; q < kPointsPer; ++q) {
          unsigned long long s[2];
          sqdist4<D>(minus[q], c, s);
          float v0, v1, v2, v3;
          unpack2(fma2(sc2, s[0], w.x), v0, v1);
          unpack2(fma2(sc2, s[1], w.y), v2, v3);
          least[q] = h == 0 ? fminf(min3(v0, v1, v2), v3) : min3(min3(least[q], v0, v1), v2, v3);
        }
      }
#pragma unroll
      for (int q = 0; q < kPointsPer; ++q) {
        const bool first = least[q] < low[q];
        third[q] = fminf(third[q], fmaxf(least[q], next[q]));
        at2[q] = first ? at[q] : least[q] < next[q] ? t : at2[q];
        next[q] = fminf(next[q], fmaxf(least[q], low[q]));
        at[q] = first ? t : at[q];
        low[q] = fminf(low[q], least[q]);
      }
    }
#pragma unroll
    for (int q = 0; q < kPointsPer; ++q) {
      const float A = reach[q] + __int_as_float(bound_c), V = __int_as_float(bound_v);
      const float far = 2.0f * (float)D * A * A;  // no squared distance is larger
      const float least = fabsf(sc) * (64.0f * kUnit * kUnit * far + 1e-38f) + 1e-30f;
      // the error of a pair whose value is at most x
      auto error = [&](float x) {
        const float t = sc < 0.0f ? fabsf(sc) * far : fminf(fmaxf(x + V, 0.0f), sc * far);
        return kUnit * (8.0f * A * sqrtf((float)D * fabsf(sc) * t) + 16.0f * t + 4.0f * (V + fabsf(x))) + least;
      };
      const float have = __double2float_ru(best[q]);
      float lim = low[q] + error(low[q]);
      lim = lim < have ? lim : have;
      lim += error(lim);
      const bool all = !screened || !(far < INFINITY) || !(fabsf(lim) < INFINITY);
      auto take = [&](int t) {
        double s = 0.0;
#pragma unroll
        for (int d = 0; d < D; ++d) {
          const double e = (double)p[q][d] - tc[t * D + d];
          s += e * e;
        }
        const double val = scale * s - tv[t];
        best[q] = val < best[q] ? val : best[q];
      };
      if (ok[q] && (all || !(low[q] > lim))) {
        auto scan = [&](int t0, int t1) {
          for (int t = t0; t < t1; ++t) {
            if (!all) {
              float s = 0.0f;
#pragma unroll
              for (int d = 0; d < D; ++d) {
                const float e = fc[d][t] + unpack_low(minus[q][d]);
                s = d == 0 ? e * e : __fmaf_rn(e, e, s);
              }
              if (__fmaf_rn(sc, s, fv[t]) > lim) continue;
            }
            take(t);
          }
        };
        auto group = [&](int t) { scan(t, t + kGroup < cnt ? t + kGroup : cnt); };
        // the pairs within the error are in the groups whose minima are
        if (all || !(third[q] > lim)) {
          scan(0, cnt);
        } else {
          group(at[q]);
          if (!(next[q] > lim)) group(at2[q]);
        }
      }
    }
  }
#pragma unroll
  for (int q = 0; q < kPointsPer; ++q) part[q * kMinThreads + threadIdx.x] = best[q];
  cooperative_groups::cluster_group cluster = cooperative_groups::this_cluster();
  cluster.sync();
  if (cluster.block_rank() == 0) {
#pragma unroll
    for (int q = 0; q < kPointsPer; ++q) {
      double b = best[q];
      for (int r = 1; r < kSplit; ++r) {
        const double o = *cluster.map_shared_rank(part + q * kMinThreads + threadIdx.x, r);
        b = o < b ? o : b;
      }
      const int64_t i = ((int64_t)blockIdx.x * kPointsPer + q) * kMinThreads + threadIdx.x;
      if (ok[q]) out[i] = b;
    }
  }
  cluster.sync();  // no CTA leaves while its shared memory is read
}

// Both in FP64 throughout, a point of the first set a thread, for a second set of few
// points: there is little to split over CTAs and a screen has no best value to measure a
// tile against, so that its passes and barriers only come on top. On B200, this and the
// screened form, 5000 points: the c-transform in the plane 4.1 and 6.2 us for 32 centres,
// 6.2 and 8.2 for 128, 10.3 and 8.2 for 256, on the line, where a distance is two
// operations less, 6.3 and 8.4 for 189, 8.2 and 8.3 for 256; the maximum in the plane 5.2 and 5.7 us for one
// point, 8.2 and 8.3 for 128, 10.3 and 8.5 for 256, on the line 6.2 and 8.2 for 128, 8.2
// and 8.2 for 256.
__host__ __device__ constexpr int few_points(int dim) { return dim == 1 ? 256 : 160; }
constexpr int kFewThreads = 256;
template <int D>
__global__ void __launch_bounds__(kFewThreads) k_max_sqdist_few(int64_t m, int64_t n, const float* __restrict__ xs,
                                                                const float* __restrict__ ys,
                                                                unsigned long long* __restrict__ out_bits) {
  __shared__ float ty[few_points(D) * D];
  __shared__ double red[kFewThreads / 32];
  const int64_t i = (int64_t)blockIdx.x * kFewThreads + threadIdx.x;
  double x[D];
#pragma unroll
  for (int d = 0; d < D; ++d) x[d] = i < m ? (double)xs[i * D + d] : 0.0;
  double best = 0.0;
  for (int t = threadIdx.x; t < n * D; t += kFewThreads) ty[t] = ys[t];
  __syncthreads();
  if (i < m)
    for (int t = 0; t < n; ++t) {
      double s = 0.0;
#pragma unroll
      for (int d = 0; d < D; ++d) {
        const double e = x[d] - (double)ty[t * D + d];
        s += e * e;
      }
      best = s > best ? s : best;
    }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    const double y = __shfl_xor_sync(0xffffffffu, best, o);
    best = y > best ? y : best;
  }
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = best;
  __syncthreads();
  if (threadIdx.x == 0) {
    double b = red[0];
    for (int w = 1; w < kFewThreads / 32; ++w) b = red[w] > b ? red[w] : b;
    atomicMax(out_bits, (unsigned long long)__double_as_longlong(b));
  }
}

template <int D>
__global__ void __launch_bounds__(kFewThreads)
    k_c_transform_few(int64_t np, int64_t nc, const float* __restrict__ pts, const double* __restrict__ centres,
                      const double* __restrict__ duals, double scale, double* __restrict__ out) {
  __shared__ double tc[few_points(D) * D];
  __shared__ double tv[few_points(D)];
  const int64_t i = (int64_t)blockIdx.x * kFewThreads + threadIdx.x;
  double p[D];
#pragma unroll
  for (int d = 0; d < D; ++d) p[d] = i < np ? (double)pts[i * D + d] : 0.0;
  double best = INFINITY;
  for (int t = threadIdx.x; t < nc * D; t += kFewThreads) tc[t] = centres[t];
  for (int t = threadIdx.x; t < nc; t += kFewThreads) tv[t] = duals[t];
  __syncthreads();
  if (i < np)
    for (int t = 0; t < nc; ++t) {
      double s = 0.0;
#pragma unroll
      for (int d = 0; d < D; ++d) {
        const double e = p[d] - tc[t * D + d];
        s += e * e;
      }
      const double val = scale * s - tv[t];
      best = val < best ? val : best;
    }
  if (i < np) out[i] = best;
}

template <int D>
void max_sqdist(int64_t m, int64_t n, const float* xs, const float* ys, unsigned long long* bits, cudaStream_t s) {
  if (n <= few_points(D)) {
    k_max_sqdist_few<D><<<(unsigned)((m + kFewThreads - 1) / kFewThreads), kFewThreads, 0, s>>>(m, n, xs, ys, bits);
    return;
  }
  const int64_t blocks = (m + kMaxThreads * kPointsPer - 1) / (kMaxThreads * kPointsPer);
  // the second set in shares of whole tiles, some 16 CTAs per SM
  const int64_t tiles = (n + kFarTile - 1) / kFarTile;
  int64_t shares = (148 * 16 + blocks - 1) / blocks;
  shares = shares < tiles ? shares : tiles;
  const int64_t share = (tiles + shares - 1) / shares * kFarTile;
  const dim3 grid((unsigned)blocks, (unsigned)((n + share - 1) / share));
  k_max_sqdist<D><<<grid, kMaxThreads, 0, s>>>(m, n, share, xs, ys, bits);
}

template <int D>
void c_transform(int64_t np, int64_t nc, const float* pts, const double* centres, const double* duals, double scale,
                 double* out, cudaStream_t s) {
  if (nc <= few_points(D)) {
    k_c_transform_few<D><<<(unsigned)((np + kFewThreads - 1) / kFewThreads), kFewThreads, 0, s>>>(
        np, nc, pts, centres, duals, scale, out);
    return;
  }
  const dim3 grid((unsigned)((np + kMinThreads * kPointsPer - 1) / (kMinThreads * kPointsPer)), kSplit);
  k_c_transform<D><<<grid, kMinThreads, 0, s>>>(np, nc, pts, centres, duals, scale, out);
}

int report(int code, const char* msg) {
  set_last_error(msg);
  return code;
}

}  // namespace
}  // namespace pdot

extern "C" int pdot_points_max_sqdist(int64_t m, int64_t n, int32_t dim, const float* source_points,
                                      const float* target_points, double* out, void* stream) {
  using namespace pdot;
  set_last_error("");
  if (m < 1 || n < 1) return report(PDOT_ERR_INVALID_ARGUMENT, "empty point set");
  if (dim < 1 || dim > 3) return report(PDOT_ERR_INVALID_ARGUMENT, "point dimension must be 1..3");
  if (!source_points || !target_points || !out) return report(PDOT_ERR_INVALID_ARGUMENT, "null pointer argument");
  const cudaStream_t s = static_cast<cudaStream_t>(stream);
  cudaError_t e = cudaMemsetAsync(out, 0, sizeof(double), s);
  if (e != cudaSuccess) return report(PDOT_ERR_CUDA, cudaGetErrorString(e));
  auto* bits = reinterpret_cast<unsigned long long*>(out);
  if (dim == 1)
    max_sqdist<1>(m, n, source_points, target_points, bits, s);
  else if (dim == 2)
    max_sqdist<2>(m, n, source_points, target_points, bits, s);
  else
    max_sqdist<3>(m, n, source_points, target_points, bits, s);
  e = cudaGetLastError();
  if (e != cudaSuccess) return report(PDOT_ERR_CUDA, cudaGetErrorString(e));
  return PDOT_OK;
}

extern "C" int pdot_points_c_transform(int64_t num_points, int64_t num_centres, int32_t dim, const float* points,
                                       const double* centres, const double* duals, double scale, double* out,
                                       void* stream) {
  using namespace pdot;
  set_last_error("");
  if (num_points < 1 || num_centres < 1) return report(PDOT_ERR_INVALID_ARGUMENT, "empty point set");
  if (dim < 1 || dim > 3) return report(PDOT_ERR_INVALID_ARGUMENT, "point dimension must be 1..3");
  if (!points || !centres || !duals || !out) return report(PDOT_ERR_INVALID_ARGUMENT, "null pointer argument");
  if (!std::isfinite(scale)) return report(PDOT_ERR_INVALID_ARGUMENT, "scale must be finite");
  const cudaStream_t s = static_cast<cudaStream_t>(stream);
  if (dim == 1)
    c_transform<1>(num_points, num_centres, points, centres, duals, scale, out, s);
  else if (dim == 2)
    c_transform<2>(num_points, num_centres, points, centres, duals, scale, out, s);
  else
    c_transform<3>(num_points, num_centres, points, centres, duals, scale, out, s);
  const cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) return report(PDOT_ERR_CUDA, cudaGetErrorString(e));
  return PDOT_OK;
}
