// C = A . W^T with fp32 operands to fp32 precision: the product of models that are run in true 32-bit.  Groups, two ways:
//   tile_group != null   the rows of A come in 128-row tiles, tile i using the weights of group
//                        tile_group[i]; tiles from *live_tiles on are skipped
//   groups > 1           blockIdx.z = group: strides between the groups' operands
// A single product may add a bias and apply xIELU to its first columns.  Two kernels:
//   gemm_f32_tc_kernel   tensor cores, every operand split into three bf16 pieces
//   gemm_f32_kernel      what it does not take: operands that 16-byte loads cannot read, a K below 64 or, for many columns, 128
#include <cfloat>

#include "common.cuh"
#include "tc_ops.cuh"
#include "xielu.cuh"

namespace eb {
namespace {

constexpr int kT = 64, kStep = 16, kF32Threads = 256;

struct F32Params {
  const float *A, *W;
  float *C;
  long long lda, ldw, ldc, a_gs, w_gs, c_gs;
  int M, N, K;
  const int *tile_group, *live_tiles;
  const float *bias, *act_params;   // both or either may be null; xIELU on the columns below act_cols
  int act_cols;
};

// ---- tensor cores -------------------------------------------------------------------------------------------------
// A CTA computes 128 rows of A x 64 rows of W.  An fp32 number is the sum of three bf16 numbers (rounded, and twice the exact
// remainder rounded); of the nine products of pieces the three smallest, below 2^-25 of the whole and of either sign, are left out.
// Per chunk of 64 columns six products of 128 x 64 x 64 go to the tensor core, the smallest first, into an accumulator that starts at zero;
// four warps add the finished chunk to sums in registers.  The tensor core truncates when it accumulates (a K of 2048 summed there is off
// by 2e-6 and too small on average, one of 4096 by 4e-6); over one chunk that is 7e-8, and the whole is closer to 64-bit results than a
// chain of fp32 multiply-adds: K = 64 7.7e-8 against 1.4e-7, K = 2048 1.3e-7 against 8.1e-7, K = 5632 1.9e-7 against 1.3e-6 (2-norm, normal operands).
// Bound by the trip to L2 for a chunk's operands, of which one chunk is requested ahead (48 registers a thread), and by splitting them.
// Warps 0-3 add up and store, 4-11 load, split and write the swizzled operand tiles, 12 issues the products.
// Some outputs are computed again from the operands, by the whole CTA, in 64 bits (all 128 x 64 of a tile with a K of 2048: 0.8 ms, at
// the rate of 64-bit multiply-adds):
//   not finite   an infinity or a number that bf16 rounds to infinity has no such split, and where a product overflows, products of
//                pieces overflow each by itself, to either side
//   small        below 2^-100 a number's lower pieces, or what they are multiplied to, can lie below the normal range (2^-126; bf16 ends at
//                2^-133): an absolute error of up to 2^-126 per term and unit of the other operand.  That counts where one side's row is that
//                small throughout, or the sum is not 2^24 times what the errors can add up to.
// A NaN among the operands stays one in the pieces and in the sum, which is then right as it is.
constexpr int kF32Cols = 64, kF32Chunk = 64, kSplitWarps = 8, kF32TcThreads = 32 * (4 + kSplitWarps + 1), kF32Stages = 3;
constexpr uint32_t kPlaneA = kRows * 128, kPlaneW = kF32Cols * 128, kF32StageBytes = 3 * (kPlaneA + kPlaneW);
constexpr size_t kF32TcSmem = 1024 + 1024 + (size_t)kF32Stages * kF32StageBytes;

// Pieces of two numbers, packed.
__device__ __forceinline__ uint32_t round2(float x0, float x1) {
  uint32_t v;
  asm("cvt.rn.bf16x2.f32 %0, %1, %2;" : "=r"(v) : "f"(x1), "f"(x0));
  return v;
}
__device__ __forceinline__ void split2(float x0, float x1, uint32_t &hi, uint32_t &mid, uint32_t &lo) {
  hi = round2(x0, x1);
  x0 -= __uint_as_float(hi << 16); x1 -= __uint_as_float(hi & 0xffff0000u);
  mid = round2(x0, x1);
  lo = round2(x0 - __uint_as_float(mid << 16), x1 - __uint_as_float(mid & 0xffff0000u));
}

// The largest magnitude; a NaN stays.
__device__ __forceinline__ float largest(float x, float y, float z) {
  float r;
  asm("max.NaN.abs.f32 %0, %1, %2, %3;" : "=f"(r) : "f"(x), "f"(y), "f"(z));
  return r;
}

__device__ __forceinline__ void store_f32(const F32Params &p, float *C, int m, int n, float v, float up, float down) {
  v += p.bias ? p.bias[n] : 0.f;
  if (p.act_params && n < p.act_cols) v = xielu_exact(v, up, down);
  C[(long long)m * p.ldc + n] = v;
}

// The outputs of a tile that `redo` marks (a word of column bits per row), by all warps: one has 4 rows x 4 columns at a time, its lanes
// share K.  A marked output costs its block's 8 rows of operands on their way from L2.
__device__ __noinline__ void redo_marked(const F32Params &p, const float *A, const float *W, float *C, int m0, int n0, const unsigned long long *redo, float up,
                                         float down) {
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  for (int block = warp; block < kRows / 4 * (kF32Cols / 4); block += kF32TcThreads / 32) {
    const int row = block / (kF32Cols / 4) * 4, col = block % (kF32Cols / 4) * 4;
    uint32_t marked = 0;                                 // bit 4 r + c
#pragma unroll
    for (int r = 0; r < 4; ++r) marked |= ((uint32_t)(redo[row + r] >> col) & 15u) << (4 * r);
    if (!marked) continue;
    const float *a[4], *w[4];
    double sum[4][4];
#pragma unroll
    for (int i = 0; i < 4; ++i) {                        // (rows and columns that are not there: the last ones, never marked)
      a[i] = A + (long long)min(m0 + row + i, p.M - 1) * p.lda;
      w[i] = W + (long long)min(n0 + col + i, p.N - 1) * p.ldw;
#pragma unroll
      for (int c = 0; c < 4; ++c) sum[i][c] = 0.;
    }
    for (int k = lane * 4; k < p.K; k += 128) {
      float4 x[4], y[4];
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        x[i] = __ldg(reinterpret_cast<const float4 *>(a[i] + k));
        y[i] = __ldg(reinterpret_cast<const float4 *>(w[i] + k));
      }
#pragma unroll
      for (int r = 0; r < 4; ++r)
#pragma unroll
        for (int c = 0; c < 4; ++c)
          sum[r][c] = fma((double)x[r].w, (double)y[c].w, fma((double)x[r].z, (double)y[c].z, fma((double)x[r].y, (double)y[c].y, fma((double)x[r].x, (double)y[c].x, sum[r][c]))));
    }
#pragma unroll
    for (int i = 0; i < 16; ++i) {
      double v = sum[i >> 2][i & 3];
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
      if (lane == i && (marked >> i & 1u)) store_f32(p, C, m0 + row + (i >> 2), n0 + col + (i & 3), (float)v, up, down);
    }
  }
}

__global__ void __launch_bounds__(kF32TcThreads, 1) gemm_f32_tc_kernel(const F32Params p) {
  extern __shared__ uint8_t smem_raw[];
  const uint32_t raw_addr = s32(smem_raw);
  uint8_t *smem = smem_raw + (((raw_addr + 1023u) & ~1023u) - raw_addr);
  uint64_t *bars = reinterpret_cast<uint64_t *>(smem);
  const uint32_t full = s32(bars), empty = full + 8 * kF32Stages, tfull = empty + 8 * kF32Stages, tempty = tfull + 16;
  uint32_t *tmem_slot = reinterpret_cast<uint32_t *>(bars + 2 * kF32Stages + 4);
  volatile int *abort_flag = reinterpret_cast<volatile int *>(tmem_slot + 1);
  float *top = reinterpret_cast<float *>(smem + 256);  // per row of A, then of W: its largest magnitude, or NaN
  const uint32_t tiles = s32(smem) + 1024;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int m0 = blockIdx.y * kRows, n0 = blockIdx.x * kF32Cols, chunks = (p.K + kF32Chunk - 1) / kF32Chunk;

  if (threadIdx.x == 0) {
    for (int s = 0; s < kF32Stages; ++s) { bar_init(full + 8 * s, kSplitWarps); bar_init(empty + 8 * s, 1); }
    for (int a = 0; a < 2; ++a) { bar_init(tfull + 8 * a, 1); bar_init(tempty + 8 * a, 4); }
    *abort_flag = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == 12) {
    __syncwarp();
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(s32(tmem_slot)), "r"(2u * kF32Cols) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = *tmem_slot;
  griddep_wait();
  griddep_launch();
  long long group = blockIdx.z;
  bool live = true;
  if (p.tile_group) {
    live = (int)blockIdx.y < *p.live_tiles;
    group = live ? p.tile_group[blockIdx.y] : 0;
  }
  const float *A = p.A + (p.tile_group ? 0 : group * p.a_gs), *W = p.W + group * p.w_gs;
  float *C = p.C + (p.tile_group ? 0 : group * p.c_gs);
  float acc[kF32Cols];
  bool odd = false;

  if (!live) {
  } else if (warp < 4) {
    // ---------------- sums of the chunks: a thread has a row ----------------
#pragma unroll
    for (int j = 0; j < kF32Cols; ++j) acc[j] = 0.f;
    for (int c = 0; c < chunks; ++c) {
      const int b = c & 1;
      if (!__all_sync(0xffffffffu, bar_wait(tfull + 8 * b, (c >> 1) & 1, abort_flag, 1))) break;
      tc_fence_after();
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        float v[32];
        tc_ld32(tmem + ((uint32_t)(warp * 32) << 16) + b * kF32Cols + h * 32, v);
#pragma unroll
        for (int j = 0; j < 32; ++j) acc[h * 32 + j] += v[j];
      }
      tc_fence_before();
      __syncwarp();
      if (lane == 0) bar_arrive(tempty + 8 * b);
    }
  } else if (warp < 12) {
    // ---------------- loads and splits: eight threads per row, 8 columns each ----------------
    constexpr int kPasses = (kRows + kF32Cols) / 32;
    const int t = threadIdx.x - 128, unit = t & 7, row_in = t >> 3;
    float4 x[kPasses][2];
    float most[kPasses] = {};
    auto load = [&](int q, int c) {
      const int row = q * 32 + row_in, k = c * kF32Chunk + unit * 8;
      const bool of_a = q < kRows / 32;
      const int r = of_a ? m0 + row : n0 + row - kRows;
      const bool ok = r < (of_a ? p.M : p.N);
      const float *src = (of_a ? A + (long long)r * p.lda : W + (long long)r * p.ldw) + k;
#pragma unroll
      for (int h = 0; h < 2; ++h)
        x[q][h] = ok && k + 4 * h < p.K ? __ldg(reinterpret_cast<const float4 *>(src) + h) : make_float4(0.f, 0.f, 0.f, 0.f);
    };
#pragma unroll
    for (int q = 0; q < kPasses; ++q) load(q, 0);
    int stage = 0;
    uint32_t phase = 0;
    for (int c = 0; c < chunks; ++c) {
      if (!__all_sync(0xffffffffu, bar_wait(empty + 8 * stage, phase ^ 1u, abort_flag, 2))) break;
      uint8_t *at = smem + 1024 + (size_t)stage * kF32StageBytes;
#pragma unroll
      for (int q = 0; q < kPasses; ++q) {
        const bool of_a = q < kRows / 32;
        const int row = (of_a ? q : q - kRows / 32) * 32 + row_in;
        uint8_t *dst = at + (of_a ? 0 : 3 * kPlaneA) + row * 128 + ((unit ^ (row & 7)) << 4);
        const uint32_t plane = of_a ? kPlaneA : kPlaneW;
        uint4 hi, mid, lo;
        split2(x[q][0].x, x[q][0].y, hi.x, mid.x, lo.x);
        split2(x[q][0].z, x[q][0].w, hi.y, mid.y, lo.y);
        split2(x[q][1].x, x[q][1].y, hi.z, mid.z, lo.z);
        split2(x[q][1].z, x[q][1].w, hi.w, mid.w, lo.w);
        most[q] = largest(largest(x[q][0].x, x[q][0].y, x[q][0].z), largest(x[q][0].w, x[q][1].x, x[q][1].y), largest(x[q][1].z, x[q][1].w, most[q]));
        *reinterpret_cast<uint4 *>(dst) = hi;
        *reinterpret_cast<uint4 *>(dst + plane) = mid;
        *reinterpret_cast<uint4 *>(dst + 2 * plane) = lo;
        if (c + 1 < chunks) load(q, c + 1);
      }
      asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
      __syncwarp();
      if (lane == 0) bar_arrive(full + 8 * stage);
      if (++stage == kF32Stages) { stage = 0; phase ^= 1u; }
    }
    // the hand-backs of the last stages, which nothing orders before the sums' signal, do not find the CTA gone
    for (int s = 0; s < kF32Stages; ++s) {
      if (!__all_sync(0xffffffffu, bar_wait(empty + 8 * stage, phase ^ 1u, abort_flag, 5))) break;
      if (++stage == kF32Stages) { stage = 0; phase ^= 1u; }
    }
#pragma unroll
    for (int q = 0; q < kPasses; ++q) {
#pragma unroll
      for (int o = 1; o < 8; o <<= 1) most[q] = largest(most[q], __shfl_xor_sync(0xffffffffu, most[q], o), 0.f);
      if (unit == 0) top[q * 32 + row_in] = most[q];
    }
  } else {
    // ---------------- products ----------------
    constexpr uint32_t idesc = tc_idesc(kF32Cols, 1);
    int stage = 0;
    uint32_t phase = 0;
    for (int c = 0; c < chunks; ++c) {
      const int b = c & 1;
      if (!__all_sync(0xffffffffu, bar_wait(tempty + 8 * b, ((c >> 1) & 1) ^ 1u, abort_flag, 3))) break;
      if (!__all_sync(0xffffffffu, bar_wait(full + 8 * stage, phase, abort_flag, 4))) break;
      tc_fence_after();
      const uint32_t at = tiles + stage * kF32StageBytes, wt = at + 3 * kPlaneA, d = tmem + b * kF32Cols;
      // (piece of A, piece of W), smallest products first
      constexpr int pa[6] = {2, 0, 1, 1, 0, 0}, pw[6] = {0, 2, 1, 0, 1, 0};
#pragma unroll
      for (int i = 0; i < 6; ++i) {
        const uint64_t da = tc_desc(at + pa[i] * kPlaneA), dw = tc_desc(wt + pw[i] * kPlaneW);
#pragma unroll
        for (int k = 0; k < kF32Chunk / 16; ++k) tc_mma_warp(d, da + 2 * k, dw + 2 * k, idesc, i > 0 || k > 0 ? 1u : 0u);
      }
      tc_commit_warp(empty + 8 * stage);
      tc_commit_warp(tfull + 8 * b);
      if (++stage == kF32Stages) { stage = 0; phase ^= 1u; }
    }
  }

  tc_fence_before();
  __syncthreads();
  if (warp == 12) {
    __syncwarp();
    tc_fence_after();
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(2u * kF32Cols) : "memory");
  }
  if (!live || *abort_flag) return;                    // (uniform)
  float up = 0.f, down = 0.f;
  if (p.act_params) { up = p.act_params[0]; down = p.act_params[1]; }
  unsigned long long *redo = reinterpret_cast<unsigned long long *>(smem + 1024);      // per row: the columns to compute again (the stages are free)
  if (warp < 4) {
    const int row = warp * 32 + lane, m = m0 + row;
    unsigned long long again = 0;
    // (Magnitudes are in the order of their bits; a NaN above all.  A row of zeros has exact sums.)
    const uint32_t w0 = __float_as_uint(top[kRows + lane]), w1 = __float_as_uint(top[kRows + 32 + lane]);
    const float tw_least = __uint_as_float(__reduce_min_sync(0xffffffffu, min(w0 ? w0 : 0x7f7fffffu, w1 ? w1 : 0x7f7fffffu)));
    const float tw_most = __uint_as_float(__reduce_max_sync(0xffffffffu, max(w0, w1)));
    if (m < p.M) {
      // Mostly the whole row is fine by its least and largest sum.  Zeros are, unless every product fell below the range.
      const float ta = top[row], least = (float)p.K * 0x1p-102f;
      float v_least = FLT_MAX, v_most = 0.f;
#pragma unroll
      for (int j = 0; j < kF32Cols; ++j) {
        v_least = fminf(v_least, acc[j] == 0.f ? FLT_MAX : fabsf(acc[j]));
        v_most = largest(v_most, acc[j], 0.f);
      }
      if (!(v_most <= FLT_MAX && (ta == 0.f || (fminf(fminf(ta, tw_least), ta * tw_least) >= 0x1p-100f && v_least >= fmaxf(0x1p-100f, least * fmaxf(ta, tw_most)))))) {
#pragma unroll
        for (int j = 0; j < kF32Cols; ++j) {
          const float tw = top[kRows + j], v = fabsf(acc[j]), small = fminf(ta, tw);
          const bool lost = small > 0.f && (small < 0x1p-100f || (v < fmaxf(0x1p-100f, least * fmaxf(ta, tw)) && (v > 0.f || ta * tw < 0x1p-100f)));
          if (n0 + j < p.N && !isnan(ta) && !isnan(tw) && (!(v <= FLT_MAX) || lost)) again |= 1ull << j;
        }
      }
      const bool wide = !p.bias && !p.act_params && ((uintptr_t)C & 15) == 0 && p.ldc % 4 == 0;
#pragma unroll
      for (int j = 0; j < kF32Cols; j += 4) {
        if (n0 + j >= p.N) break;
        if (wide && n0 + j + 4 <= p.N) {
          *reinterpret_cast<float4 *>(C + (long long)m * p.ldc + n0 + j) = make_float4(acc[j], acc[j + 1], acc[j + 2], acc[j + 3]);
        } else {
#pragma unroll
          for (int e = 0; e < 4; ++e)
            if (n0 + j + e < p.N) store_f32(p, C, m, n0 + j + e, acc[j + e], up, down);
        }
      }
    }
    redo[row] = again;
    odd = again != 0;
  }
  if (!__syncthreads_or(odd)) return;
  redo_marked(p, A, W, C, m0, n0, redo, up, down);
}

// ---- any operands: a tiled CUDA-core kernel, 64 x 64 outputs per CTA ----------------------------------------------------------------
__global__ void __launch_bounds__(kF32Threads) gemm_f32_kernel(const F32Params p) {
  __shared__ float sa[kStep][kT + 4], sw[kStep][kT + 4];
  griddep_wait();
  griddep_launch();
  const int m0 = blockIdx.y * kT, n0 = blockIdx.x * kT;
  long long group = blockIdx.z;
  if (p.tile_group) {
    const int tile = m0 / 128;
    if (tile >= *p.live_tiles) return;
    group = p.tile_group[tile];
  }
  const float *A = p.A + (p.tile_group ? 0 : group * p.a_gs), *W = p.W + group * p.w_gs;
  float *C = p.C + (p.tile_group ? 0 : group * p.c_gs);
  const int tx = threadIdx.x & 15, ty = threadIdx.x >> 4;
  float acc[4][4] = {};
  for (int k0 = 0; k0 < p.K; k0 += kStep) {
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const int e = threadIdx.x + i * kF32Threads, r = e / kStep, k = e % kStep;
      sa[k][r] = (m0 + r < p.M && k0 + k < p.K) ? A[(long long)(m0 + r) * p.lda + k0 + k] : 0.f;
      sw[k][r] = (n0 + r < p.N && k0 + k < p.K) ? W[(long long)(n0 + r) * p.ldw + k0 + k] : 0.f;
    }
    __syncthreads();
#pragma unroll
    for (int k = 0; k < kStep; ++k) {
      float a[4], w[4];
#pragma unroll
      for (int i = 0; i < 4; ++i) { a[i] = sa[k][ty * 4 + i]; w[i] = sw[k][tx * 4 + i]; }
#pragma unroll
      for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) acc[i][j] = fmaf(a[i], w[j], acc[i][j]);
    }
    __syncthreads();
  }
  float up = 0.f, down = 0.f;
  if (p.act_params) { up = p.act_params[0]; down = p.act_params[1]; }
#pragma unroll
  for (int i = 0; i < 4; ++i)
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const int m = m0 + ty * 4 + i, n = n0 + tx * 4 + j;
      if (m >= p.M || n >= p.N) continue;
      store_f32(p, C, m, n, acc[i][j], up, down);
    }
}

}  // namespace

// Status words of this file's kernels, for eb_device_status.
int f32_status(int *out4, bool clear) { return tc_status(out4, clear); }

}  // namespace eb

using namespace eb;

extern "C" int eb_gemm_f32(const float *A, long long lda, long long a_group_stride, const float *W, long long ldw, long long w_group_stride,
                           float *C, long long ldc, long long c_group_stride, int M, int N, int K, int groups, const int32_t *tile_group,
                           const int32_t *live_tiles, const float *bias, int act_cols, const float *act_params, void *stream) {
  if (M == 0 || N == 0 || groups == 0) return EB_OK;
  EB_REQUIRE(A && W && C, "gemm_f32: null pointer");
  EB_REQUIRE(M > 0 && N > 0 && K > 0 && groups > 0 && groups <= 65535, "gemm_f32: bad sizes");
  EB_REQUIRE(lda >= K && ldw >= K && ldc >= N, "gemm_f32: leading dimensions smaller than the rows they hold");
  EB_REQUIRE((tile_group == nullptr) == (live_tiles == nullptr) && (!tile_group || groups == 1),
             "gemm_f32: tile_group goes with live_tiles and without strided groups");
  EB_REQUIRE((!bias && !act_params) || (groups == 1 && !tile_group), "gemm_f32: bias and activation belong to a single product");
  EB_REQUIRE((M + kT - 1) / kT <= 65535, "gemm_f32: too many rows");
  F32Params p{};
  p.A = A; p.W = W; p.C = C; p.lda = lda; p.ldw = ldw; p.ldc = ldc; p.a_gs = a_group_stride; p.w_gs = w_group_stride; p.c_gs = c_group_stride;
  p.M = M; p.N = N; p.K = K; p.tile_group = tile_group; p.live_tiles = live_tiles;
  p.bias = bias; p.act_cols = act_cols; p.act_params = act_params;
  cudaStream_t st = as_stream(stream);
  // 16-byte loads need rows that begin and end on 16 bytes, and below a chunk the multiply-adds are the closer ones (K = 4: 4.0e-8 against
  // 4.6e-8).  However many rows there are: a row's result is the same in every batch.  333 x 11264 x 2048: 881 us by multiply-adds, 202 so; one
  // row x 2048 x 2048 149 and 39.  With a short K a tile is little but the way in and out, which tiles of one SM go one after the other, while several
  // of the multiply-add kernel's share it: beyond a wave of columns the line lies at two chunks (one row x 32768: K = 64 17 us against 24, K = 96 24
  // against 28, K = 128 30 against 28).
  const bool many = (long long)((N + kF32Cols - 1) / kF32Cols) * groups > sm_count();
  const bool packs = K >= (many ? 2 : 1) * kF32Chunk && K % 4 == 0 && lda % 4 == 0 && ldw % 4 == 0 && a_group_stride % 4 == 0 && w_group_stride % 4 == 0 && aligned16(A) && aligned16(W);
  if (packs) {
    static bool configured[64] = {};
    int dev = 0;
    cudaGetDevice(&dev);
    if (dev >= 0 && dev < 64 && !configured[dev]) {
      if (cudaFuncSetAttribute(gemm_f32_tc_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kF32TcSmem) != cudaSuccess) {
        cudaGetLastError();
        return fail(EB_ECUDA, "gemm_f32: cannot reserve shared memory");
      }
      configured[dev] = true;
    }
    launch_pdl(gemm_f32_tc_kernel, dim3((N + kF32Cols - 1) / kF32Cols, (M + kRows - 1) / kRows, groups), dim3(kF32TcThreads), kF32TcSmem, st, p);
    return check_launch("gemm_f32");
  }
  launch_pdl(gemm_f32_kernel, dim3((N + kT - 1) / kT, (M + kT - 1) / kT, groups), dim3(kF32Threads), 0, st, p);
  return check_launch("gemm_f32");
}
