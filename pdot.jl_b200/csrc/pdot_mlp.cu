// pdot_mlp.cu — the network of the learned warm start: an MLP
// input -> hidden -> hidden -> output with GELU, BF16 weights (FP32 master
// copies and AdamW state), BF16 activations and FP32 accumulation.
//
// Every matrix product runs on the 5th-generation tensor cores through one
// hand-written kernel, k_gemm: D[M x N] = A[M x K] . B[N x K]^T with A and B
// BF16 and K-major (K contiguous). TMA moves 128 x 64 tiles of A and B into
// shared memory with the 128-byte swizzle, one thread issues tcgen05.mma
// (M = 128, N = 128, K = 16 per instruction) into a TMEM accumulator, each
// stage of the 4-deep ring is released by tcgen05.commit on its mbarrier, and
// the eight warps read the accumulator back with tcgen05.ld for a fused
// epilogue (bias, GELU or the GELU derivative) that also writes the transposed
// BF16 copy the backward products read. With every operand K-major:
//
//   forward   Z1 = X  W1^T + b1, H1 = gelu(Z1)     A = X  [B x I],  B = W1 [H x I]
//             Z2 = H1 W2^T + b2, H2 = gelu(Z2)     A = H1,          B = W2
//             Y  = H2 W3^T + b3                    A = H2,          B = W3 [O x H]
//   backward  dW3 = dY^T H2                        A = dY^T [O x B], B = H2^T [H x B]
//             dZ2 = (dY W3) * gelu'(Z2)            A = dY [B x O],   B = W3^T [H x O]
//             dW2 = dZ2^T H1,  dZ1 = (dZ2 W2) * gelu'(Z1),  dW1 = dZ1^T X
//
// The loss is the mean squared error over the output entries of the real rows
// of the batch. All reductions (loss, bias gradients) are in a fixed order.
//
// A training step of 256 rows (2048 -> 1024 -> 1024 -> 2048) takes 127 us on B200, 305
// before the transposed copies went through shared memory, the bias gradients, AdamW
// and the loss took one parallel launch each and the kernels were launched dependent on
// one another: features 5, split products 4 x 15, the output layer's 11, weight
// gradients 7 each, loss 6, bias gradients 5, AdamW 32 us. The products are bound by
// latency (their bytes take 1 to 3 us from L2), AdamW by its bytes.
#include <cooperative_groups.h>
#include <cuda.h>
#include <cuda_bf16.h>
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <cstdarg>
#include <cstdint>
#include <cstdio>
#include <cstring>
#include <functional>
#include <memory>
#include <mutex>
#include <new>
#include <string>
#include <vector>

#include "pdot_device.cuh"

namespace pdot {
namespace {

// Build knob: PDOT_MLP_SPLIT_K 0 runs every product as one tile per CTA.
#ifndef PDOT_MLP_SPLIT_K
#define PDOT_MLP_SPLIT_K 1
#endif
constexpr int kGemmThreads = 256;  // two warps per 32 accumulator rows: the epilogues are latency-bound
constexpr int kBM = 128;  // rows of A per tile (= TMEM lanes)
constexpr int kBN = 128;  // rows of B per tile (= accumulator columns)
constexpr int kBK = 64;   // K per stage: one 128-byte swizzle row of BF16
constexpr int kUmmaK = 16;
constexpr int kStages = 4;
constexpr int kTileABytes = kBM * kBK * 2;
constexpr int kTileBBytes = kBN * kBK * 2;
constexpr int kStageBytes = kTileABytes + kTileBBytes;
constexpr int kGemmSmem = kStages * kStageBytes + 1024 + 256;

enum { EPI_F32 = 0, EPI_BIAS_GELU = 1, EPI_BIAS = 2, EPI_GELU_BWD = 3 };

// Error codes a kernel leaves in the error word.
enum { kErrWaitFull = 1, kErrWaitEmpty = 2, kErrWaitDone = 3 };

struct Epi {
  float* f32;                  // row-major M x N (ld_f32)
  __nv_bfloat16* bf16;         // row-major M x N (ld_bf16)
  __nv_bfloat16* bf16_t;       // transposed: entry (r, c) at [c * ld_t + r]
  const float* bias;           // N
  const float* z;              // saved pre-activation, row-major (ld_z)
  int64_t ld_f32, ld_bf16, ld_t, ld_z;
};

__device__ __forceinline__ uint32_t smem_addr(const void* p) {
  return static_cast<uint32_t>(__cvta_generic_to_shared(p));
}

// UMMA shared-memory descriptor of a K-major operand tile written by TMA with
// the 128-byte swizzle: rows of 128 bytes, 8-row groups 1024 bytes apart
// (stride byte offset), descriptor version 1, layout SWIZZLE_128B (2).
__device__ __forceinline__ uint64_t sw128_kmajor_desc(uint32_t saddr) {
  uint64_t d = 0;
  d |= (uint64_t)((saddr & 0x3FFFFu) >> 4);
  d |= (uint64_t)1 << 16;            // leading byte offset (unused by swizzled K-major)
  d |= (uint64_t)(1024 >> 4) << 32;  // stride byte offset
  d |= (uint64_t)1 << 46;            // version
  d |= (uint64_t)2 << 61;            // SWIZZLE_128B
  return d;
}

// Instruction descriptor: kind::f16 with BF16 A and B, FP32 accumulator,
// both K-major, N = kBN, M = kBM.
constexpr uint32_t kIdesc = (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(kBN >> 3) << 17) |
                            ((uint32_t)(kBM >> 4) << 24);

__device__ __forceinline__ void tc_fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tc_fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }

__device__ __forceinline__ void tma_load_2d(uint32_t dst, const CUtensorMap* map, uint32_t bar, int x, int y) {
  asm volatile(
      "cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4}], [%2];" ::"r"(
          dst),
      "l"(reinterpret_cast<uint64_t>(map)), "r"(bar), "r"(x), "r"(y)
      : "memory");
}

// D (+)= A B^T for one K = 16 step; no output lane disabled.
__device__ __forceinline__ void umma_bf16(uint32_t tmem_d, uint64_t da, uint64_t db, uint32_t accumulate) {
  const uint32_t z = 0u;
  asm volatile(
      "{\n .reg .pred p;\n setp.ne.b32 p, %4, 0;\n"
      " tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, {%5, %6, %7, %8}, p;\n}" ::"r"(tmem_d),
      "l"(da), "l"(db), "r"(kIdesc), "r"(accumulate), "r"(z), "r"(z), "r"(z), "r"(z)
      : "memory");
}

__device__ __forceinline__ void umma_commit(uint32_t bar) {
  asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(bar) : "memory");
}

__device__ __forceinline__ void tmem_ld16(uint32_t taddr, float (&v)[16]) {
  uint32_t r[16];
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, "
      "[%16];"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]),
        "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
      : "r"(taddr));
  asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
  for (int k = 0; k < 16; ++k) v[k] = __uint_as_float(r[k]);
}

// GELU with the error function, and its derivative.
__device__ __forceinline__ float gelu(float z) { return 0.5f * z * (1.0f + erff(z * 0.70710678118654752f)); }
__device__ __forceinline__ float gelu_grad(float z) {
  return 0.5f * (1.0f + erff(z * 0.70710678118654752f)) + z * 0.39894228040143268f * expf(-0.5f * z * z);
}

__device__ __forceinline__ void store_f32x8(float* p, const float* v) {
  asm volatile("st.global.v8.f32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8};" ::"l"(p), "f"(v[0]), "f"(v[1]), "f"(v[2]),
               "f"(v[3]), "f"(v[4]), "f"(v[5]), "f"(v[6]), "f"(v[7])
               : "memory");
}

// The fused epilogue of W (a multiple of 4) accumulator columns [col, col + W)
// of one row.
template <int EPI, int W>
__device__ __forceinline__ void epilogue_cols(const Epi& ep, int64_t row, int64_t col, float (&v)[W]) {
  if (EPI == EPI_BIAS_GELU || EPI == EPI_BIAS) {
#pragma unroll
    for (int k = 0; k < W; ++k) v[k] += __ldg(ep.bias + col + k);
  }
  if (EPI == EPI_GELU_BWD) {
    const float* zr = ep.z + row * ep.ld_z + col;
#pragma unroll
    for (int k = 0; k < W; k += 4) {
      const float4 z4 = *reinterpret_cast<const float4*>(zr + k);
      v[k] *= gelu_grad(z4.x);
      v[k + 1] *= gelu_grad(z4.y);
      v[k + 2] *= gelu_grad(z4.z);
      v[k + 3] *= gelu_grad(z4.w);
    }
  }
  float* fo = ep.f32 + row * ep.ld_f32 + col;
  if constexpr (W % 8 == 0) {
#pragma unroll
    for (int k = 0; k < W; k += 8) store_f32x8(fo + k, v + k);  // whole sectors
  } else {
#pragma unroll
    for (int k = 0; k < W; k += 4) *reinterpret_cast<float4*>(fo + k) = make_float4(v[k], v[k + 1], v[k + 2], v[k + 3]);
  }
  if (EPI == EPI_BIAS_GELU || EPI == EPI_GELU_BWD) {
    __align__(16) __nv_bfloat16 h[W];
#pragma unroll
    for (int k = 0; k < W; ++k) h[k] = __float2bfloat16_rn(EPI == EPI_BIAS_GELU ? gelu(v[k]) : v[k]);
    if (ep.bf16) {
      __nv_bfloat16* bo = ep.bf16 + row * ep.ld_bf16 + col;
      if constexpr (W % 8 == 0) {
#pragma unroll
        for (int k = 0; k < W; k += 8) *reinterpret_cast<uint4*>(bo + k) = *reinterpret_cast<const uint4*>(h + k);
      } else {
#pragma unroll
        for (int k = 0; k < W; k += 4) *reinterpret_cast<uint2*>(bo + k) = *reinterpret_cast<const uint2*>(h + k);
      }
    }
#pragma unroll
    for (int k = 0; k < W; ++k) ep.bf16_t[(col + k) * ep.ld_t + row] = h[k];
  }
}

// One 128 x 128 tile of D = A B^T per CTA; K a multiple of kBK. With split > 1 the K
// blocks are cut into `split` slices, slice z the blocks [z * KB / split, (z + 1) * KB /
// split), and a cluster of gridDim.z CTAs shares the tile, each with split / gridDim.z
// neighbouring slices in accumulators of their own: products with few output tiles (the
// batch is 256 rows) thus spread over the SMs instead of 16 of them. The CTAs leave
// their partial tiles in shared memory; each then adds its share of the rows over the
// cluster, slice by slice in order, and runs their epilogue. (With the partial tiles in
// global memory and a second kernel for the ordered sum, 256 x 1024 x 2048 took 8.9 +
// 6.3 us.)
constexpr int kMaxSplit = 16;
constexpr int kTileF4 = kBN / 4;  // float4 columns of a tile
static_assert(2 * kBM * kBN * 4 <= kStages * kStageBytes, "two partial tiles fit the ring");
// Float4 slot of (row, column group) of a partial tile: lanes of a warp hold the same
// group of 32 rows when they write and neighbouring rows when they read; the exclusive
// or spreads both over the banks.
__device__ __forceinline__ int tile_slot(int row, int c4) { return row * kTileF4 + (c4 ^ (row & (kTileF4 - 1))); }

template <int EPI>
__global__ void __launch_bounds__(kGemmThreads, 1)
    k_gemm(const __grid_constant__ CUtensorMap ta, const __grid_constant__ CUtensorMap tb, int K, int split, Epi ep,
           int* err) {
  extern __shared__ uint8_t smem_raw[];
  const uint32_t raw = smem_addr(smem_raw);
  const uint32_t tiles = (raw + 1023u) & ~1023u;  // the swizzle atoms need 1024-byte alignment
  const uint32_t bars = tiles + kStages * kStageBytes;
  auto full = [&](int s) { return bars + 8u * s; };
  auto empty = [&](int s) { return bars + 8u * (kStages + s); };
  const uint32_t done = bars + 8u * (2 * kStages);
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(smem_raw + (bars - raw) + 8 * (2 * kStages + 1));
  __shared__ int s_err;

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int m0 = blockIdx.y * kBM, n0 = blockIdx.x * kBN;
  const int kb_all = K / kBK;
  const int per = split / (int)gridDim.z;  // slices of this CTA, 1 or 2
  auto slice_begin = [&](int z) { return (int)((long long)z * kb_all / split); };
  const int z0 = (int)blockIdx.z * per;
  const int kb0 = slice_begin(z0), kblocks = slice_begin(z0 + per) - kb0;
  const int cut = slice_begin(z0 + 1) - kb0;  // first K block of the second slice
  const uint32_t tmem_cols = (uint32_t)(per * kBN);
  if (threadIdx.x == 0) {
    asm volatile("prefetch.tensormap [%0];" ::"l"(reinterpret_cast<uint64_t>(&ta)) : "memory");
    asm volatile("prefetch.tensormap [%0];" ::"l"(reinterpret_cast<uint64_t>(&tb)) : "memory");
    s_err = 0;
    for (int s = 0; s < kStages; ++s) {
      mbar_init(full(s), 1);
      mbar_init(empty(s), 1);
    }
    mbar_init(done, 1);
    fence_mbar_init();
  }
  if (warp == 2) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_addr(tmem_slot)),
                 "r"(tmem_cols)
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = *tmem_slot;
  pdl_enter();  // barriers and accumulators are set up while the kernel before this one ends

  if (warp == 0 && lane == 0) {
    // producer: TMA loads of the A and B tiles of each K block
    int issued = 0;
    for (int kb = 0; kb < kblocks; ++kb) {
      const int s = kb % kStages;
      if (kb >= kStages && !mbar_wait_bounded(empty(s), ((kb / kStages) & 1) ^ 1)) {
        atomicCAS(&s_err, 0, kErrWaitEmpty);
        break;
      }
      mbar_expect_tx(full(s), kStageBytes);
      tma_load_2d(tiles + s * kStageBytes, &ta, full(s), (kb0 + kb) * kBK, m0);
      tma_load_2d(tiles + s * kStageBytes + kTileABytes, &tb, full(s), (kb0 + kb) * kBK, n0);
      issued = kb + 1;
    }
    // every copy issued has landed before the CTA may leave (already true on
    // the normal path, where the MMAs consumed them)
    for (int kb = (issued > kStages ? issued - kStages : 0); kb < issued; ++kb)
      if (!mbar_wait_bounded(full(kb % kStages), (kb / kStages) & 1)) atomicCAS(&s_err, 0, kErrWaitFull);
  } else if (warp == 1 && lane == 0) {
    // MMA issuer
    for (int kb = 0; kb < kblocks; ++kb) {
      const int s = kb % kStages;
      if (!mbar_wait_bounded(full(s), (kb / kStages) & 1)) {
        atomicCAS(&s_err, 0, kErrWaitFull);
        break;
      }
      tc_fence_after();
      const uint64_t da = sw128_kmajor_desc(tiles + s * kStageBytes);
      const uint64_t db = sw128_kmajor_desc(tiles + s * kStageBytes + kTileABytes);
#pragma unroll
      for (int kk = 0; kk < kBK / kUmmaK; ++kk)  // +32 bytes along the swizzled row per K step
        umma_bf16(tmem + (kb >= cut ? (uint32_t)kBN : 0u), da + (uint64_t)(2 * kk), db + (uint64_t)(2 * kk),
                  (kb != 0 && kb != cut) || kk != 0 ? 1u : 0u);
      umma_commit(empty(s));
    }
    umma_commit(done);
  }
  __syncwarp();
  if (!mbar_wait_bounded(done, 0)) atomicCAS(&s_err, 0, kErrWaitDone);
  __syncwarp();
  tc_fence_after();

  // thread (warp w, lane l) owns half a row of the accumulator: row 32 (w mod 4) + l,
  // columns from (w / 4) kBN / 2
  const int trow = (warp & 3) * 32 + lane, tcol = (warp >> 2) * (kBN / 2);
  const uint32_t lane_base = tmem + ((uint32_t)((warp & 3) * 32) << 16);
  if (split == 1) {
#pragma unroll 2
    for (int c0 = tcol; c0 < tcol + kBN / 2; c0 += 16) {
      float v[16];
      tmem_ld16(lane_base + (uint32_t)c0, v);
      epilogue_cols<EPI, 16>(ep, m0 + trow, n0 + c0, v);
    }
  } else {
    // the ring is free: every copy has landed and every product has read it
    float4* tile = reinterpret_cast<float4*>(smem_raw + (tiles - raw));
    for (int t = 0; t < per; ++t) {
#pragma unroll 2
      for (int c0 = tcol; c0 < tcol + kBN / 2; c0 += 16) {
        float v[16];
        tmem_ld16(lane_base + (uint32_t)(t * kBN + c0), v);
#pragma unroll
        for (int k = 0; k < 4; ++k)
          tile[t * kBM * kTileF4 + tile_slot(trow, c0 / 4 + k)] =
              make_float4(v[4 * k], v[4 * k + 1], v[4 * k + 2], v[4 * k + 3]);
      }
    }
    cooperative_groups::cluster_group cluster = cooperative_groups::this_cluster();
    cluster.sync();
    // lanes on neighbouring rows (the transposed BF16 copy's stores coalesce), two
    // column groups per warp (the row-major ones fill their sectors)
    const int rows = kBM / (int)gridDim.z;  // 16 and more
    const int two = per - 1;                // log2 of the slices per CTA
#pragma unroll 2
    for (int item = threadIdx.x; item < rows * kTileF4; item += kGemmThreads) {
      const int c4 = (item >> 4) & (kTileF4 - 1);
      const int r = (int)blockIdx.z * rows + (item / (16 * kTileF4)) * 16 + (item & 15);
      const int slot = tile_slot(r, c4);
      float4 q[kMaxSplit];
#pragma unroll
      for (int z = 0; z < kMaxSplit; ++z)
        if (z < split) q[z] = cluster.map_shared_rank(tile, z >> two)[(z & two) * kBM * kTileF4 + slot];
      float v[4] = {q[0].x, q[0].y, q[0].z, q[0].w};
#pragma unroll
      for (int z = 1; z < kMaxSplit; ++z)
        if (z < split) v[0] += q[z].x, v[1] += q[z].y, v[2] += q[z].z, v[3] += q[z].w;
      epilogue_cols<EPI, 4>(ep, m0 + r, n0 + 4 * c4, v);
    }
    cluster.sync();  // no CTA leaves while its tile is read
  }
  tc_fence_before();
  __syncthreads();
  if (warp == 2) {
    tc_fence_after();
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(tmem_cols) : "memory");
  }
  if (threadIdx.x == 0 && s_err != 0) atomicCAS(err, 0, s_err);
}

constexpr int kEw = 256;  // threads of the elementwise kernels

// Tiles of kTr x kTr entries of a row-major matrix whose BF16 form is also stored
// transposed: the tile goes through shared memory, so that both copies are written in
// whole sectors. (Written entry by entry, the transposed copy took a 32-byte sector
// for 2 bytes and most of these kernels' time.) Rows and columns are multiples of kTr.
constexpr int kTr = 64;
struct TransposeTile {
  __nv_bfloat16 h[kTr][kTr + 2];
};
// the 4 x 4 entries of a thread: rows (t >> 4) + 16 k, columns 4 (t & 15) ...
__device__ __forceinline__ void tile_put(TransposeTile& T, int r, int c, const __nv_bfloat16 (&b)[4]) {
#pragma unroll
  for (int e = 0; e < 4; ++e) T.h[r][c + e] = b[e];
}
// dst[(c0 + c) * ld + r0 + r] for the whole tile; 16 rows of a column per thread
__device__ __forceinline__ void tile_write_transposed(const TransposeTile& T, __nv_bfloat16* dst, int64_t ld,
                                                      int64_t r0, int64_t c0) {
  const int c = threadIdx.x >> 2, r = (threadIdx.x & 3) * 16;
  __align__(16) __nv_bfloat16 o[16];
#pragma unroll
  for (int e = 0; e < 16; ++e) o[e] = T.h[r + e][c];
  uint4* p = reinterpret_cast<uint4*>(dst + (c0 + c) * ld + r0 + r);
  p[0] = reinterpret_cast<const uint4*>(o)[0];
  p[1] = reinterpret_cast<const uint4*>(o)[1];
}
__device__ __forceinline__ void store_bf16x4(__nv_bfloat16* p, const __nv_bfloat16 (&b)[4]) {
  uint2 w;
  memcpy(&w, b, 8);
  *reinterpret_cast<uint2*>(p) = w;
}

// x[r, k] = bf16((log(max(h, 1e-30)) + shift) * scale) for real rows, 0 for the
// padding rows up to bp; also the transposed copy xt (leading dimension ld_t). A CTA
// takes kTr rows of kFeatCols columns, four FP64 logarithms a thread: their latency,
// not the bytes, is what counts, so the tiles are narrow and many.
constexpr int kFeatCols = 16;
__global__ void __launch_bounds__(kEw) k_features(const double* __restrict__ hist, int64_t batch, int64_t dim,
                                                  double shift, double scale, __nv_bfloat16* __restrict__ x,
                                                  __nv_bfloat16* __restrict__ xt, int64_t ld_t) {
  __shared__ __nv_bfloat16 T[kTr][kFeatCols + 2];
  pdl_enter();
  const int64_t r0 = (int64_t)blockIdx.y * kTr, c0 = (int64_t)blockIdx.x * kFeatCols;
  const int r = threadIdx.x >> 2, c = 4 * (threadIdx.x & 3);
  __align__(8) __nv_bfloat16 b[4];
#pragma unroll
  for (int e = 0; e < 4; ++e) {
    double f = 0.0;
    if (r0 + r < batch) {
      const double h = hist[(r0 + r) * dim + c0 + c + e];
      f = (log(h > 1e-30 ? h : 1e-30) + shift) * scale;
    }
    b[e] = __double2bfloat16(f);
    T[r][c + e] = b[e];
  }
  store_bf16x4(x + (r0 + r) * dim + c0 + c, b);
  __syncthreads();
  const int tc = threadIdx.x >> 4, tr = 4 * (threadIdx.x & 15);
#pragma unroll
  for (int e = 0; e < 4; ++e) b[e] = T[tr + e][tc];
  store_bf16x4(xt + (c0 + tc) * ld_t + r0 + tr, b);
}

// dY = 2 (Y - T) / (batch * O) on real rows (0 on padding), its BF16 copy and
// transpose, and per-CTA partial sums of (Y - T)^2.
__global__ void __launch_bounds__(kEw) k_loss(const float* __restrict__ y, const float* __restrict__ t, int64_t batch,
                                              int64_t dim, float* __restrict__ dy, __nv_bfloat16* __restrict__ dyb,
                                              __nv_bfloat16* __restrict__ dyt, int64_t ld_t,
                                              double* __restrict__ part) {
  __shared__ TransposeTile T;
  __shared__ double sh[kEw / 32];
  pdl_enter();
  const int64_t r0 = (int64_t)blockIdx.y * kTr, c0 = (int64_t)blockIdx.x * kTr;
  const int c = 4 * (threadIdx.x & 15);
  const float g = 2.0f / (float)(batch * dim);
  double acc = 0.0;
#pragma unroll
  for (int k = 0; k < 4; ++k) {
    const int r = (threadIdx.x >> 4) + 16 * k;
    const int64_t at = (r0 + r) * dim + c0 + c;
    float d[4] = {0.0f, 0.0f, 0.0f, 0.0f};
    if (r0 + r < batch) {
      const float4 yv = *reinterpret_cast<const float4*>(y + at);
      float tv[4];
#pragma unroll
      for (int e = 0; e < 4; ++e) tv[e] = t[at + e];  // the caller's array: any alignment
      const float diff[4] = {yv.x - tv[0], yv.y - tv[1], yv.z - tv[2], yv.w - tv[3]};
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        acc += (double)diff[e] * (double)diff[e];
        d[e] = g * diff[e];
      }
    }
    *reinterpret_cast<float4*>(dy + at) = make_float4(d[0], d[1], d[2], d[3]);
    __align__(8) __nv_bfloat16 b[4];
#pragma unroll
    for (int e = 0; e < 4; ++e) b[e] = __float2bfloat16_rn(d[e]);
    store_bf16x4(dyb + at, b);
    tile_put(T, r, c, b);
  }
  acc = warp_sum(acc);
  if ((threadIdx.x & 31) == 0) sh[threadIdx.x >> 5] = acc;
  __syncthreads();
  tile_write_transposed(T, dyt, ld_t, r0, c0);
  if (threadIdx.x == 0) {
    double s = sh[0];
#pragma unroll
    for (int w = 1; w < kEw / 32; ++w) s += sh[w];
    part[blockIdx.y * gridDim.x + blockIdx.x] = s;
  }
}

// One CTA: thread t adds partials t, t + kEw, ..., then a tree (50 us by one thread).
__global__ void __launch_bounds__(kEw) k_loss_total(const double* __restrict__ part, int parts, int64_t count,
                                                    double* __restrict__ loss) {
  __shared__ double sh[kEw / 32];
  pdl_enter();
  double s = 0.0;
  for (int k = threadIdx.x; k < parts; k += kEw) s += part[k];
  s = warp_sum(s);
  if ((threadIdx.x & 31) == 0) sh[threadIdx.x >> 5] = s;
  __syncthreads();
  if (threadIdx.x == 0) {
#pragma unroll
    for (int w = 1; w < kEw / 32; ++w) s += sh[w];
    *loss = s / (double)count;
  }
}

// The bias gradients of all layers: out[c] = sum over the first `rows` rows of in[r, c].
// A CTA takes 32 columns of one layer with 16 row groups side by side, added in order
// (one thread per column, a launch per layer: 25 us each at 256 rows).
constexpr int kColGroups = 16;
struct ColSums {
  const float* in[3];
  float* out[3];
  int blocks[3];  // CTAs of each layer: columns / 32
  int64_t cols[3];
};
__global__ void __launch_bounds__(32 * kColGroups) k_colsum(ColSums S, int64_t rows) {
  __shared__ double sh[kColGroups][32];
  pdl_enter();
  int l = 0, b = blockIdx.x;
  while (b >= S.blocks[l]) b -= S.blocks[l++];
  const int lane = threadIdx.x & 31, grp = threadIdx.x >> 5;
  const int64_t cols = S.cols[l], c = (int64_t)b * 32 + lane;
  const float* in = S.in[l] + c;
  double s = 0.0;
#pragma unroll 8
  for (int64_t r = grp; r < rows; r += kColGroups) s += (double)in[r * cols];
  sh[grp][lane] = s;
  __syncthreads();
  if (grp == 0) {
#pragma unroll
    for (int g = 1; g < kColGroups; ++g) s += sh[g][lane];
    S.out[l][c] = (float)s;
  }
}

// AdamW on every tensor in one launch: CTAs of kTr x kTr tiles of the three weight
// matrices, then CTAs of kEw entries of the three biases (no decay, no BF16 copies).
// m = b1 m + (1 - b1) g, v = b2 v + (1 - b2) g^2,
// p -= lr (m / (1 - b1^t) / (sqrt(v / (1 - b2^t)) + eps) + wd p);
// then the BF16 copy and its transpose. Bound by the 32 B per parameter it streams: 32 us for
// 5.2 M parameters on B200, 82 us with a launch per tensor and the transposes entry by entry.
struct AdamTensors {
  float* p[3];         // weights
  const float* g[3];
  float* m[3];
  float* v[3];
  __nv_bfloat16* pb[3];
  __nv_bfloat16* pt[3];
  int64_t rows[3], cols[3];
  int tiles[3];
  float* bp[3];        // biases, rows[l] entries
  const float* bg[3];
  float* bm[3];
  float* bv[3];
  int bias_blocks[3];
};
struct AdamStep {
  float lr, b1, b2, eps, wd, c1, c2;
};
__device__ __forceinline__ float adamw_entry(const AdamStep& A, float wd, float p, float gr, float& m, float& v) {
  const float mm = A.b1 * m + (1.0f - A.b1) * gr;
  const float vv = A.b2 * v + (1.0f - A.b2) * gr * gr;
  m = mm;
  v = vv;
  const float upd = (mm / A.c1) / (sqrtf(vv / A.c2) + A.eps) + wd * p;
  return p - A.lr * upd;
}
__global__ void __launch_bounds__(kEw) k_adamw(AdamTensors T, AdamStep A) {
  __shared__ TransposeTile tile;
  pdl_enter();
  int l = 0, b = blockIdx.x;
  while (l < 3 && b >= T.tiles[l]) b -= T.tiles[l++];
  if (l == 3) {  // a bias
    l = 0;
    while (b >= T.bias_blocks[l]) b -= T.bias_blocks[l++];
    const int64_t e = (int64_t)b * kEw + threadIdx.x;
    if (e < T.rows[l]) {
      float m = T.bm[l][e], v = T.bv[l][e];
      T.bp[l][e] = adamw_entry(A, 0.0f, T.bp[l][e], T.bg[l][e], m, v);
      T.bm[l][e] = m;
      T.bv[l][e] = v;
    }
    return;
  }
  const int64_t rows = T.rows[l], cols = T.cols[l], across = cols / kTr;
  const int64_t r0 = b / across * kTr, c0 = b % across * kTr;
  const int c = 4 * (threadIdx.x & 15);
  float4 p[4], g[4], m[4], v[4];
#pragma unroll
  for (int k = 0; k < 4; ++k) {
    const int64_t at = (r0 + (threadIdx.x >> 4) + 16 * k) * cols + c0 + c;
    p[k] = *reinterpret_cast<const float4*>(T.p[l] + at);
    g[k] = *reinterpret_cast<const float4*>(T.g[l] + at);
    m[k] = *reinterpret_cast<const float4*>(T.m[l] + at);
    v[k] = *reinterpret_cast<const float4*>(T.v[l] + at);
  }
#pragma unroll
  for (int k = 0; k < 4; ++k) {
    const int r = (threadIdx.x >> 4) + 16 * k;
    const int64_t at = (r0 + r) * cols + c0 + c;
    p[k].x = adamw_entry(A, A.wd, p[k].x, g[k].x, m[k].x, v[k].x);
    p[k].y = adamw_entry(A, A.wd, p[k].y, g[k].y, m[k].y, v[k].y);
    p[k].z = adamw_entry(A, A.wd, p[k].z, g[k].z, m[k].z, v[k].z);
    p[k].w = adamw_entry(A, A.wd, p[k].w, g[k].w, m[k].w, v[k].w);
    *reinterpret_cast<float4*>(T.p[l] + at) = p[k];
    *reinterpret_cast<float4*>(T.m[l] + at) = m[k];
    *reinterpret_cast<float4*>(T.v[l] + at) = v[k];
    const __nv_bfloat16 h[4] = {__float2bfloat16_rn(p[k].x), __float2bfloat16_rn(p[k].y), __float2bfloat16_rn(p[k].z),
                                __float2bfloat16_rn(p[k].w)};
    store_bf16x4(T.pb[l] + at, h);
    tile_put(tile, r, c, h);
  }
  __syncthreads();
  tile_write_transposed(tile, T.pt[l], rows, r0, c0);
}

// BF16 copies (and transposes) of the weight matrices from the FP32 masters.
__global__ void __launch_bounds__(kEw) k_to_bf16(const float* __restrict__ p, int64_t rows, int64_t cols,
                                                 __nv_bfloat16* __restrict__ pb, __nv_bfloat16* __restrict__ pt) {
  __shared__ TransposeTile T;
  pdl_enter();
  const int64_t r0 = (int64_t)blockIdx.y * kTr, c0 = (int64_t)blockIdx.x * kTr;
  const int c = 4 * (threadIdx.x & 15);
#pragma unroll
  for (int k = 0; k < 4; ++k) {
    const int r = (threadIdx.x >> 4) + 16 * k;
    const int64_t at = (r0 + r) * cols + c0 + c;
    const float4 w = *reinterpret_cast<const float4*>(p + at);
    const __nv_bfloat16 h[4] = {__float2bfloat16_rn(w.x), __float2bfloat16_rn(w.y), __float2bfloat16_rn(w.z),
                                __float2bfloat16_rn(w.w)};
    store_bf16x4(pb + at, h);
    tile_put(T, r, c, h);
  }
  __syncthreads();
  tile_write_transposed(T, pt, rows, r0, c0);
}

dim3 tile_grid(int64_t rows, int64_t cols) { return dim3((unsigned)(cols / kTr), (unsigned)(rows / kTr)); }

}  // namespace
}  // namespace pdot

// ---------------------------------------------------------------------------
// Host side
namespace {

struct MlpFailure {
  int code;
  std::string msg;
};

[[noreturn]] void mfail(int code, const char* fmt, ...) {
  char buf[1024];
  va_list ap;
  va_start(ap, fmt);
  vsnprintf(buf, sizeof(buf), fmt, ap);
  va_end(ap);
  throw MlpFailure{code, buf};
}

void mck(cudaError_t e, const char* what, int line) {
  if (e != cudaSuccess) {
    cudaGetLastError();
    mfail(e == cudaErrorMemoryAllocation ? PDOT_ERR_OUT_OF_MEMORY : PDOT_ERR_CUDA, "%s failed: %s (pdot_mlp.cu:%d)",
          what, cudaGetErrorString(e), line);
  }
}
#define MCK(x) mck((x), #x, __LINE__)

typedef CUresult (*EncodeTiledFn)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*,
                                  const cuuint64_t*, const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave,
                                  CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

EncodeTiledFn encode_fn() {
  static std::mutex mu;
  static EncodeTiledFn fn = nullptr;
  std::lock_guard<std::mutex> lock(mu);
  if (!fn) {
    void* p = nullptr;
    cudaDriverEntryPointQueryResult q = cudaDriverEntryPointSymbolNotFound;
    if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &p, cudaEnableDefault, &q) != cudaSuccess ||
        q != cudaDriverEntryPointSuccess || !p) {
      cudaGetLastError();
      mfail(PDOT_ERR_CUDA, "cuTensorMapEncodeTiled is not available from the driver");
    }
    fn = reinterpret_cast<EncodeTiledFn>(p);
  }
  return fn;
}

// Tensor map of a row-major BF16 matrix [rows x cols] read in 128 x 64 boxes
// with the 128-byte swizzle (cols a multiple of 64, rows of 128).
CUtensorMap make_map(const __nv_bfloat16* base, int64_t rows, int64_t cols) {
  CUtensorMap map;
  memset(&map, 0, sizeof(map));
  const cuuint64_t dims[2] = {(cuuint64_t)cols, (cuuint64_t)rows};
  const cuuint64_t strides[1] = {(cuuint64_t)cols * 2};
  const cuuint32_t box[2] = {(cuuint32_t)pdot::kBK, (cuuint32_t)pdot::kBM};
  const cuuint32_t estr[2] = {1, 1};
  const CUresult r = encode_fn()(&map, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, const_cast<__nv_bfloat16*>(base), dims,
                                 strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B,
                                 CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  if (r != CUDA_SUCCESS) mfail(PDOT_ERR_CUDA, "cuTensorMapEncodeTiled failed (%d) for a %lld x %lld matrix", (int)r,
                               (long long)rows, (long long)cols);
  return map;
}

using bf16 = __nv_bfloat16;

}  // namespace

struct pdot_mlp {
  int device = 0;
  int64_t I = 0, H = 0, O = 0, Bp = 0;  // dimensions; Bp = batch capacity (multiple of 128)
  int64_t P = 0;                        // parameters
  int64_t step = 0;                     // AdamW steps taken
  cudaStream_t stream = nullptr;
  std::vector<void*> allocs;
  // FP32 masters, gradients, AdamW moments (layout W1, b1, W2, b2, W3, b3)
  float *theta = nullptr, *grad = nullptr, *m1 = nullptr, *m2 = nullptr;
  float *W[3] = {}, *b[3] = {}, *gW[3] = {}, *gb[3] = {};
  bf16 *Wb[3] = {}, *Wt[3] = {};
  // activations
  bf16 *x = nullptr, *xt = nullptr, *h1 = nullptr, *h1t = nullptr, *h2 = nullptr, *h2t = nullptr;
  float *z1 = nullptr, *z2 = nullptr, *y = nullptr;
  float *dy = nullptr, *dz2 = nullptr, *dz1 = nullptr;
  bf16 *dyb = nullptr, *dyt = nullptr, *dz2b = nullptr, *dz2t = nullptr, *dz1t = nullptr;
  double *loss_part = nullptr, *loss = nullptr;
  int* err = nullptr;
  int sms = 148;
  int loss_parts = 0;
  int64_t batch = 0;  // rows of the current input
  // tensor maps of every GEMM operand
  CUtensorMap mx, mW[3], mh1, mh2, mdyt, mh2t, mdyb, mWt[3], mdz2t, mh1t, mdz2b, mdz1t, mxt;

  template <typename T>
  T* alloc(size_t count) {
    void* p = nullptr;
    MCK(cudaMalloc(&p, std::max<size_t>(count, 1) * sizeof(T)));
    allocs.push_back(p);
    MCK(cudaMemsetAsync(p, 0, std::max<size_t>(count, 1) * sizeof(T), stream));
    return static_cast<T*>(p);
  }

  ~pdot_mlp() {
    if (stream) cudaStreamSynchronize(stream);
    for (void* p : allocs) cudaFree(p);
    if (stream) cudaStreamDestroy(stream);
  }

  // the network's kernels are launched with programmatic dependent launch (pdot::pdl_launch)
  template <typename... P, typename... A>
  void launch(void (*kfn)(P...), dim3 grid, A... args) {
    MCK(pdot::pdl_launch(kfn, grid, dim3(pdot::kEw), 0, stream, P(args)...));
  }

  void sync_bf16() {
    const int64_t rows[3] = {H, H, O}, cols[3] = {I, H, H};
    for (int l = 0; l < 3; ++l)
      launch(pdot::k_to_bf16, pdot::tile_grid(rows[l], cols[l]), W[l], rows[l], cols[l], Wb[l], Wt[l]);
  }

  void check_err() {
    int e = 0;
    MCK(cudaMemcpyAsync(&e, err, sizeof(int), cudaMemcpyDeviceToHost, stream));
    MCK(cudaStreamSynchronize(stream));
    if (e != 0) {
      MCK(cudaMemsetAsync(err, 0, sizeof(int), stream));
      mfail(PDOT_ERR_CUDA, "a tensor-core GEMM gave up waiting on its pipeline (code %d)", e);
    }
  }

  template <int EPI>
  void gemm(const CUtensorMap& a, const CUtensorMap& bm, int64_t M, int64_t N, int64_t K, const pdot::Epi& ep) {
    if (M % pdot::kBM || N % pdot::kBN || K % pdot::kBK || K <= 0)
      mfail(PDOT_ERR_INVALID_ARGUMENT, "GEMM shape %lld x %lld x %lld is not tiled by 128 x 128 x 64", (long long)M,
            (long long)N, (long long)K);
    MCK(cudaFuncSetAttribute(pdot::k_gemm<EPI>, cudaFuncAttributeMaxDynamicSharedMemorySize, pdot::kGemmSmem));
    // split K where the tiles cover at most an eighth of the SMs (the batch's
    // 256-row products with a 1024-wide output), while the slices fill at
    // most every SM and each keeps at least two K blocks. 256 x 2048 x 1024 (32
    // tiles) split in four measured 16.6 us against 14.4 us whole, so it and the
    // weight gradients (64 and more tiles) are not split.
    const int64_t tiles = (N / pdot::kBN) * (M / pdot::kBM), kb = K / pdot::kBK;
    int S = 1;
    if (PDOT_MLP_SPLIT_K && tiles * 8 <= sms)
      while (tiles * S * 2 <= sms && kb / (S * 2) >= 2 && S * 2 <= pdot::kMaxSplit) S *= 2;
    // eight slices to four CTAs, two each: 16 clusters of eight wait for room on the
    // GPCs (20 us a product against 14)
    const int ctas = S >= 8 ? S / 2 : S;
    cudaLaunchConfig_t c = {};
    c.gridDim = dim3((unsigned)(N / pdot::kBN), (unsigned)(M / pdot::kBM), (unsigned)ctas);
    c.blockDim = dim3(pdot::kGemmThreads);
    c.dynamicSmemBytes = pdot::kGemmSmem;
    c.stream = stream;
    cudaLaunchAttribute at[2];
    at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at[0].val.programmaticStreamSerializationAllowed = PDOT_PDL;
    at[1].id = cudaLaunchAttributeClusterDimension;
    at[1].val.clusterDim.x = at[1].val.clusterDim.y = 1;
    at[1].val.clusterDim.z = c.gridDim.z;
    c.attrs = at;
    c.numAttrs = 2;
    MCK(cudaLaunchKernelEx(&c, pdot::k_gemm<EPI>, a, bm, (int)K, S, ep, err));
  }

  int64_t padded(int64_t rows) const { return (rows + pdot::kBM - 1) / pdot::kBM * pdot::kBM; }

  void forward() {
    const int64_t bp = padded(batch);
    pdot::Epi e{};
    e.f32 = z1; e.ld_f32 = H; e.bf16 = h1; e.ld_bf16 = H; e.bf16_t = h1t; e.ld_t = Bp; e.bias = b[0];
    gemm<pdot::EPI_BIAS_GELU>(mx, mW[0], bp, H, I, e);
    e = pdot::Epi{};
    e.f32 = z2; e.ld_f32 = H; e.bf16 = h2; e.ld_bf16 = H; e.bf16_t = h2t; e.ld_t = Bp; e.bias = b[1];
    gemm<pdot::EPI_BIAS_GELU>(mh1, mW[1], bp, H, H, e);
    e = pdot::Epi{};
    e.f32 = y; e.ld_f32 = O; e.bias = b[2];
    gemm<pdot::EPI_BIAS>(mh2, mW[2], bp, O, H, e);
  }

  // want_loss: the caller reads `loss` afterwards
  void backward(const float* target, bool want_loss) {
    const int64_t bp = padded(batch);
    const dim3 lg = pdot::tile_grid(bp, O);
    launch(pdot::k_loss, lg, y, target, batch, O, dy, dyb, dyt, Bp, loss_part);
    if (want_loss) launch(pdot::k_loss_total, dim3(1), loss_part, (int)(lg.x * lg.y), batch * O, loss);
    // the transposed operands were written with leading dimension Bp; the
    // products over the batch read the first bp columns of them
    pdot::Epi e{};
    e.f32 = gW[2]; e.ld_f32 = H;
    gemm<pdot::EPI_F32>(mdyt, mh2t, O, H, bp, e);
    e = pdot::Epi{};
    e.f32 = dz2; e.ld_f32 = H; e.bf16 = dz2b; e.ld_bf16 = H; e.bf16_t = dz2t; e.ld_t = Bp; e.z = z2; e.ld_z = H;
    gemm<pdot::EPI_GELU_BWD>(mdyb, mWt[2], bp, H, O, e);
    e = pdot::Epi{};
    e.f32 = gW[1]; e.ld_f32 = H;
    gemm<pdot::EPI_F32>(mdz2t, mh1t, H, H, bp, e);
    e = pdot::Epi{};
    e.f32 = dz1; e.ld_f32 = H; e.bf16 = nullptr; e.bf16_t = dz1t; e.ld_t = Bp; e.z = z1; e.ld_z = H;
    gemm<pdot::EPI_GELU_BWD>(mdz2b, mWt[1], bp, H, H, e);
    e = pdot::Epi{};
    e.f32 = gW[0]; e.ld_f32 = I;
    gemm<pdot::EPI_F32>(mdz1t, mxt, H, I, bp, e);
    pdot::ColSums cs{{dy, dz2, dz1}, {gb[2], gb[1], gb[0]}, {(int)(O / 32), (int)(H / 32), (int)(H / 32)}, {O, H, H}};
    MCK(pdot::pdl_launch(pdot::k_colsum, dim3((unsigned)((O + 2 * H) / 32)), dim3(32 * pdot::kColGroups), 0, stream, cs,
                         bp));
  }

  void adamw(float lr, float b1_, float b2_, float eps, float wd) {
    ++step;
    const float c1 = 1.0f - powf(b1_, (float)step), c2 = 1.0f - powf(b2_, (float)step);
    const int64_t rows[3] = {H, H, O}, cols[3] = {I, H, H};
    pdot::AdamTensors t{};
    unsigned blocks = 0;
    for (int l = 0; l < 3; ++l) {
      const int64_t off_w = W[l] - theta, off_b = b[l] - theta;
      t.p[l] = W[l], t.g[l] = grad + off_w, t.m[l] = m1 + off_w, t.v[l] = m2 + off_w;
      t.pb[l] = Wb[l], t.pt[l] = Wt[l], t.rows[l] = rows[l], t.cols[l] = cols[l];
      t.tiles[l] = (int)(rows[l] / pdot::kTr * (cols[l] / pdot::kTr));
      t.bp[l] = b[l], t.bg[l] = grad + off_b, t.bm[l] = m1 + off_b, t.bv[l] = m2 + off_b;
      t.bias_blocks[l] = (int)((rows[l] + pdot::kEw - 1) / pdot::kEw);
      blocks += (unsigned)(t.tiles[l] + t.bias_blocks[l]);
    }
    launch(pdot::k_adamw, dim3(blocks), t, pdot::AdamStep{lr, b1_, b2_, eps, wd, c1, c2});
  }
};

namespace {

int mguarded(const std::function<void()>& f) {
  try {
    f();
    return PDOT_OK;
  } catch (const MlpFailure& e) {
    pdot::set_last_error(e.msg.c_str());
    return e.code;
  } catch (const std::bad_alloc&) {
    pdot::set_last_error("host allocation failed");
    return PDOT_ERR_OUT_OF_MEMORY;
  } catch (...) {
    pdot::set_last_error("unknown failure");
    return PDOT_ERR_CUDA;
  }
}

// splitmix64, for the initial weights
uint64_t splitmix(uint64_t& s) {
  uint64_t z = (s += 0x9E3779B97F4A7C15ull);
  z = (z ^ (z >> 30)) * 0xBF58476D1CE4E5B9ull;
  z = (z ^ (z >> 27)) * 0x94D049BB133111EBull;
  return z ^ (z >> 31);
}
}  // namespace

extern "C" int pdot_mlp_create(int32_t device, int64_t input_dim, int64_t hidden_dim, int64_t output_dim,
                               int64_t max_batch, uint64_t seed, pdot_mlp** out) {
  return mguarded([&] {
    if (!out) mfail(PDOT_ERR_INVALID_ARGUMENT, "null output handle");
    *out = nullptr;
    if (input_dim <= 0 || hidden_dim <= 0 || output_dim <= 0 || input_dim % 128 || hidden_dim % 128 ||
        output_dim % 128)
      mfail(PDOT_ERR_INVALID_ARGUMENT, "the layer widths must be positive multiples of 128");
    if (max_batch <= 0 || max_batch > (1 << 20)) mfail(PDOT_ERR_INVALID_ARGUMENT, "max_batch must be 1..2^20");
    int count = 0;
    MCK(cudaGetDeviceCount(&count));
    if (device < 0 || device >= count) mfail(PDOT_ERR_NO_DEVICE, "no CUDA device %d", device);
    cudaDeviceProp prop;
    MCK(cudaGetDeviceProperties(&prop, device));
    if (prop.major != 10) mfail(PDOT_ERR_NO_DEVICE, "the tensor-core kernels need an sm_100 device");
    MCK(cudaSetDevice(device));
    std::unique_ptr<pdot_mlp> m(new pdot_mlp);
    m->device = device;
    m->I = input_dim;
    m->H = hidden_dim;
    m->O = output_dim;
    m->Bp = (max_batch + 127) / 128 * 128;
    MCK(cudaDeviceGetAttribute(&m->sms, cudaDevAttrMultiProcessorCount, device));
    MCK(cudaStreamCreateWithFlags(&m->stream, cudaStreamNonBlocking));
    const int64_t I = m->I, H = m->H, O = m->O, Bp = m->Bp;
    const int64_t sizes[6] = {H * I, H, H * H, H, O * H, O};
    int64_t P = 0;
    for (int64_t s : sizes) P += s;
    m->P = P;
    m->theta = m->alloc<float>(P);
    m->grad = m->alloc<float>(P);
    m->m1 = m->alloc<float>(P);
    m->m2 = m->alloc<float>(P);
    int64_t off = 0;
    for (int l = 0; l < 3; ++l) {
      m->W[l] = m->theta + off;
      m->gW[l] = m->grad + off;
      off += sizes[2 * l];
      m->b[l] = m->theta + off;
      m->gb[l] = m->grad + off;
      off += sizes[2 * l + 1];
    }
    const int64_t rows[3] = {H, H, O}, cols[3] = {I, H, H};
    for (int l = 0; l < 3; ++l) {
      m->Wb[l] = m->alloc<bf16>(rows[l] * cols[l]);
      m->Wt[l] = m->alloc<bf16>(rows[l] * cols[l]);
    }
    m->x = m->alloc<bf16>(Bp * I);
    m->xt = m->alloc<bf16>(I * Bp);
    m->z1 = m->alloc<float>(Bp * H);
    m->h1 = m->alloc<bf16>(Bp * H);
    m->h1t = m->alloc<bf16>(H * Bp);
    m->z2 = m->alloc<float>(Bp * H);
    m->h2 = m->alloc<bf16>(Bp * H);
    m->h2t = m->alloc<bf16>(H * Bp);
    m->y = m->alloc<float>(Bp * O);
    m->dy = m->alloc<float>(Bp * O);
    m->dyb = m->alloc<bf16>(Bp * O);
    m->dyt = m->alloc<bf16>(O * Bp);
    m->dz2 = m->alloc<float>(Bp * H);
    m->dz2b = m->alloc<bf16>(Bp * H);
    m->dz2t = m->alloc<bf16>(H * Bp);
    m->dz1 = m->alloc<float>(Bp * H);
    m->dz1t = m->alloc<bf16>(H * Bp);
    m->loss_parts = (int)(Bp / pdot::kTr * (O / pdot::kTr));
    m->loss_part = m->alloc<double>(m->loss_parts);
    m->loss = m->alloc<double>(1);
    m->err = m->alloc<int>(1);
    // initial weights and biases uniform in +-1/sqrt(fan_in)
    std::vector<float> h(P);
    uint64_t s = seed;
    const int64_t fan[6] = {I, I, H, H, H, H};
    off = 0;
    for (int k = 0; k < 6; ++k) {
      const double bound = 1.0 / std::sqrt((double)fan[k]);
      for (int64_t e = 0; e < sizes[k]; ++e) {
        const double u = (double)(splitmix(s) >> 11) * (1.0 / 9007199254740992.0);
        h[off + e] = (float)((2.0 * u - 1.0) * bound);
      }
      off += sizes[k];
    }
    MCK(cudaMemcpyAsync(m->theta, h.data(), P * sizeof(float), cudaMemcpyHostToDevice, m->stream));
    m->sync_bf16();
    // tensor maps: activations have Bp rows (products over the batch read the
    // transposed copies, Bp columns), weights their own shapes
    m->mx = make_map(m->x, Bp, I);
    m->mxt = make_map(m->xt, I, Bp);
    m->mh1 = make_map(m->h1, Bp, H);
    m->mh1t = make_map(m->h1t, H, Bp);
    m->mh2 = make_map(m->h2, Bp, H);
    m->mh2t = make_map(m->h2t, H, Bp);
    m->mdyb = make_map(m->dyb, Bp, O);
    m->mdyt = make_map(m->dyt, O, Bp);
    m->mdz2b = make_map(m->dz2b, Bp, H);
    m->mdz2t = make_map(m->dz2t, H, Bp);
    m->mdz1t = make_map(m->dz1t, H, Bp);
    for (int l = 0; l < 3; ++l) {
      m->mW[l] = make_map(m->Wb[l], rows[l], cols[l]);
      m->mWt[l] = make_map(m->Wt[l], cols[l], rows[l]);
    }
    MCK(cudaStreamSynchronize(m->stream));
    *out = m.release();
  });
}

extern "C" int pdot_mlp_destroy(pdot_mlp* m) {
  delete m;
  return PDOT_OK;
}

extern "C" int64_t pdot_mlp_num_parameters(const pdot_mlp* m) { return m ? m->P : 0; }

extern "C" void* pdot_mlp_stream(pdot_mlp* m) { return m ? (void*)m->stream : nullptr; }

extern "C" int pdot_mlp_get_parameters(pdot_mlp* m, float* host, int64_t count) {
  return mguarded([&] {
    if (!m || !host || count != m->P) mfail(PDOT_ERR_INVALID_ARGUMENT, "bad arguments");
    MCK(cudaSetDevice(m->device));
    MCK(cudaMemcpyAsync(host, m->theta, count * sizeof(float), cudaMemcpyDeviceToHost, m->stream));
    MCK(cudaStreamSynchronize(m->stream));
  });
}

extern "C" int pdot_mlp_set_parameters(pdot_mlp* m, const float* host, int64_t count) {
  return mguarded([&] {
    if (!m || !host || count != m->P) mfail(PDOT_ERR_INVALID_ARGUMENT, "bad arguments");
    MCK(cudaSetDevice(m->device));
    MCK(cudaMemcpyAsync(m->theta, host, count * sizeof(float), cudaMemcpyHostToDevice, m->stream));
    MCK(cudaMemsetAsync(m->m1, 0, count * sizeof(float), m->stream));
    MCK(cudaMemsetAsync(m->m2, 0, count * sizeof(float), m->stream));
    m->step = 0;
    m->sync_bf16();
    MCK(cudaStreamSynchronize(m->stream));
  });
}

extern "C" int pdot_mlp_get_gradients(pdot_mlp* m, float* host, int64_t count) {
  return mguarded([&] {
    if (!m || !host || count != m->P) mfail(PDOT_ERR_INVALID_ARGUMENT, "bad arguments");
    MCK(cudaSetDevice(m->device));
    MCK(cudaMemcpyAsync(host, m->grad, count * sizeof(float), cudaMemcpyDeviceToHost, m->stream));
    MCK(cudaStreamSynchronize(m->stream));
  });
}

extern "C" int pdot_mlp_set_input(pdot_mlp* m, int64_t batch, const double* histograms, double shift, double scale) {
  return mguarded([&] {
    if (!m || !histograms) mfail(PDOT_ERR_INVALID_ARGUMENT, "bad arguments");
    if (batch < 1 || batch > m->Bp) mfail(PDOT_ERR_INVALID_ARGUMENT, "batch must be 1..%lld", (long long)m->Bp);
    MCK(cudaSetDevice(m->device));
    m->batch = batch;
    const int64_t bp = m->padded(batch);
    // rows past bp stay as they are: no product reads them
    m->launch(pdot::k_features, dim3((unsigned)(m->I / pdot::kFeatCols), (unsigned)(bp / pdot::kTr)), histograms, batch, m->I, shift, scale, m->x, m->xt, m->Bp);
  });
}

extern "C" int pdot_mlp_forward(pdot_mlp* m, float* out) {
  return mguarded([&] {
    if (!m || m->batch < 1) mfail(PDOT_ERR_INVALID_ARGUMENT, "no input set");
    MCK(cudaSetDevice(m->device));
    m->forward();
    if (out)
      MCK(cudaMemcpyAsync(out, m->y, m->batch * m->O * sizeof(float), cudaMemcpyDeviceToDevice, m->stream));
    m->check_err();
  });
}

extern "C" int pdot_mlp_backward(pdot_mlp* m, const float* target, double* loss) {
  return mguarded([&] {
    if (!m || !target || m->batch < 1) mfail(PDOT_ERR_INVALID_ARGUMENT, "bad arguments");
    MCK(cudaSetDevice(m->device));
    m->backward(target, loss != nullptr);
    if (loss) MCK(cudaMemcpyAsync(loss, m->loss, sizeof(double), cudaMemcpyDeviceToHost, m->stream));
    m->check_err();
  });
}

extern "C" int pdot_mlp_adamw(pdot_mlp* m, float lr, float beta1, float beta2, float eps, float weight_decay) {
  return mguarded([&] {
    if (!m) mfail(PDOT_ERR_INVALID_ARGUMENT, "null network");
    MCK(cudaSetDevice(m->device));
    m->adamw(lr, beta1, beta2, eps, weight_decay);
  });
}

extern "C" int pdot_mlp_train_step(pdot_mlp* m, const float* target, float lr, float weight_decay, double* loss) {
  return mguarded([&] {
    if (!m || !target || m->batch < 1) mfail(PDOT_ERR_INVALID_ARGUMENT, "bad arguments");
    MCK(cudaSetDevice(m->device));
    m->forward();
    m->backward(target, loss != nullptr);
    m->adamw(lr, 0.9f, 0.999f, 1e-8f, weight_decay);
    if (loss) {
      MCK(cudaMemcpyAsync(loss, m->loss, sizeof(double), cudaMemcpyDeviceToHost, m->stream));
      m->check_err();
    }
  });
}
