// C = act(A · Wᵀ + bias) + residual for a generation step's few rows, where the latency of a launch and
// not the weight stream sets the time (included by gemm.cu).
//
// A CTA of eight warps owns 16 weight rows at a time; the warps split K.  A lane quartet loads 16 bytes of weight
// rows g and g + 8 and of activation row g at the same 8 columns and feeds them to two mma.sync (which
// columns an MMA calls k = 0..15 does not matter as long as both operands agree, so nothing is rearranged).  mma.sync
// and not tcgen05: there is no tensor memory to allocate, no descriptor to fetch and no stage to hand over, and the
// products are far below either's rate.  The weights of the first eight k-steps of every warp are requested
// before the preceding kernel of the stream is waited for, so behind that wait a launch consists of one L2
// trip for the activations (one cp.async per 16 bytes, all at once), the MMAs, one sum over the warps in shared memory
// and the store.  The sums of a slice's first 256 columns wait in shared memory for the others: mma.sync truncates as it accumulates, and with 512
// columns in one accumulator a K of 4096 was off by 6.4e-7 where the tcgen05 form is by 3.5e-7 (fp16 operands, 2-norm; now 3.4e-7; a K of 768 1.6e-7
// against 9.5e-7).  At most 128 registers, so that the next launch's CTAs fit beside these and fetch their weights meanwhile.
// Launches one behind the other, each with other weights (tcgen05 form before): 768 x 768 with one row 5.2 -> 2.4 us, 2304 x 768
// with eight rows and the LayerNorm 5.4 -> 3.3, 768 x 3072 7.7 -> 4.4, 2048 x 2048 with 16 rows 7.3 -> 5.1.
constexpr int kStepWarps = 8, kStepThreads = kStepWarps * 32;
constexpr int kStepUnroll = 4;                      // k-steps (32 columns of a warp's slice) per weight request
constexpr int kStepRun = 256;                       // columns that a warp adds up in one accumulator
constexpr int kStepPart = 33;                       // floats per accumulator element and warp (32 lanes and one against bank conflicts)

struct StepGeometry {
  int slice;                                        // columns of K per warp, a multiple of 32
  int pitch;                                        // bytes per activation row of a slice in shared memory: 64 more than a multiple of 128
  size_t smem;
};

// Where this form is the faster one.  In a row of such products it wins up to 64 M weights with 8 rows (16384 x 4096: 24.6 us against
// 26.9), but in a model the tcgen05 form asks for more of its weights while the attention before it still runs.  33 steps of two layers of 12 h^2
// weights, 8 rows: h = 1536 5.4 -> 5.2 ms, h = 3072 with all of them in this form 7.5 -> 8.6, with the square ones alone 7.7 -> 8.0; a head of 50257 x 768
// with 8 rows, 18.5 us against 21.3, is better off in this form (31 steps of 12 layers 11.9 ms against 12.6).  A longer K
// leaves a CTA too little in flight (2048 x 5632: 17.4 us against 11.7), and with a short one a tile is little but its rendezvous and sums, of which a CTA
// should not have many one after the other (8192 x 256 3.3 us against 3.8, 16384 x 256 5.4 against 4.8, 50264 x 512 13.9 against 13.3).
// With more rows the reads of the activations from shared memory, once per 16 weight rows, set the
// pace: 4096 x 2048 elements are the line for 16 rows (2048 x 2048: 5.1 against 7.3; 3072 x 3072: 10.9 against 8.1), 2048 x 2048
// for 32 (7.3 against 10.2), and a CTA has to be done with one tile.  Of 16 rows two CTAs run well side by side up to a K of 2048 (4096 x 1024 5.4 us
// against 6.5, 3072 x 2048 6.9 against 9.1, 3072 x 2304 8.0 against 7.9, 2720 x 2816 11.4 against 9.3; from K = 2817 on one fills the shared memory), of 32 rows
// one (2304 x 768 6.4 against 6.8, 3072 x 1024 10.8 against 7.6).
// A row is summed in another order here than in the tcgen05 form, so its rounding depends on which of the two its batch takes, as it does between
// steps and prompts; within a form it does not depend on the batch.
inline bool step_form_pays(int M, int N, int K, size_t smem) {
  const long long weights = (long long)N * K, most = M <= 8 && K <= 1024 ? 64ll << 20 : M <= 8 && K <= 2048 ? 16ll << 20 : M <= 16 ? 8ll << 20 : 4ll << 20;
  const int tiles = (N + 15) / 16, per_sm = M <= 8 ? (K <= 512 ? 4 : 1 << 20) : M <= 16 && K <= 2048 ? 2 : 1;
  return M <= 32 && K <= 4096 && weights <= most && tiles <= (long long)per_sm * sm_count() && smem <= 200 * 1024;
}

inline StepGeometry step_geometry(int M, int K) {
  StepGeometry s;
  const int rows = M <= 8 ? 8 : M <= 16 ? 16 : 32;
  s.slice = ((K + kStepWarps - 1) / kStepWarps + 31) / 32 * 32;
  s.pitch = s.slice * 2 + (s.slice * 2 % 128 == 0 ? 64 : 0);
  s.smem = (size_t)kStepWarps * rows * s.pitch + (size_t)2 * kStepWarps * (rows / 2) * kStepPart * sizeof(float) +
           (size_t)kStepWarps * rows * 2 * sizeof(float);
  return s;
}

// 16 bytes to shared memory, zeros if !ok
__device__ __forceinline__ void step_cp16(uint32_t dst, const void *src, bool ok) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst), "l"(src), "r"(ok ? 16 : 0) : "memory");
}

// NT: batch rows in eights (1, 2 or 4)
template <typename T, int NT>
__global__ void __launch_bounds__(kStepThreads, 2)
gemm_step_kernel(const GemmParams p, const void *weights, long long ldw, int slice, int pitch) {
  constexpr int kRows = NT * 8, U = NT == 4 ? kStepUnroll / 2 : kStepUnroll;
  constexpr int kOuts = 16 * kRows, kPer = (kOuts + kStepThreads - 1) / kStepThreads;      // outputs of a tile, per thread
  constexpr int kThreadsUsed = kOuts < kStepThreads ? kOuts : kStepThreads;
  extern __shared__ __align__(128) uint8_t step_smem[];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
  uint8_t *xs = step_smem + (size_t)warp * kRows * pitch;                                  // this warp's slice of the activations
  float *part = reinterpret_cast<float *>(step_smem + (size_t)kStepWarps * kRows * pitch); // [2][warps][NT * 4][kStepPart]
  float *stats = part + 2 * kStepWarps * NT * 4 * kStepPart;                               // [warps][rows][2]
  griddep_launch();
  const T *W = reinterpret_cast<const T *>(weights);
  const int kb = warp * slice, ke = min(p.K, kb + slice);
  const int tiles = (p.N + 15) / 16, chunks = (slice + 32 * U - 1) / (32 * U);

  // ---- the weight stream: chunk after chunk, tile after tile, two chunks ahead of the products ----
  int ld_tile = blockIdx.x, ld_chunk = 0;
  auto load = [&](uint4 (&w)[U][2]) {
    const int ra = min(ld_tile * 16 + g, p.N - 1), rb = min(ld_tile * 16 + g + 8, p.N - 1);      // rows beyond N: multiplied, not stored
    const int k0 = kb + ld_chunk * 32 * U + t * 8;
    const T *wa = W + (long long)ra * ldw + k0, *wb = W + (long long)rb * ldw + k0;
    const bool live = ld_tile < tiles;
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const bool ok = live && k0 + u * 32 < ke;
      w[u][0] = ok ? ld_stream(wa + u * 32) : make_uint4(0, 0, 0, 0);
      w[u][1] = ok ? ld_stream(wb + u * 32) : make_uint4(0, 0, 0, 0);
    }
    if (++ld_chunk == chunks) { ld_chunk = 0; ld_tile += gridDim.x; }
  };
  uint4 w0[U][2], w1[U][2];
  if (!p.static_w) griddep_wait();
  load(w0);
  load(w1);
  if (p.static_w) griddep_wait();

  // ---- the activations of the warp's slice; columns beyond K as zeros ----
  const T *X = reinterpret_cast<const T *>(p.ln_x);
  {
    const int per_row = slice / 8, total = p.M * per_row;
    const uint32_t dst = smem_u32(xs);
    for (int i = lane; i < total; i += 32) {
      const int r = i / per_row, c = i - r * per_row;
      const bool ok = kb + c * 8 < p.K;
      step_cp16(dst + r * pitch + c * 16, X + (long long)r * p.ln_ldx + (ok ? kb + c * 8 : 0), ok);
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
  }
  const bool fold = p.ln_colsum != nullptr;
  // LayerNorm folded in: shifted sums of the rows, taken from the operands as they pass by
  float sum[NT][2], sq[NT][2], pivot[NT];
#pragma unroll
  for (int j = 0; j < NT; ++j) {
    sum[j][0] = sum[j][1] = sq[j][0] = sq[j][1] = 0.f;
    pivot[j] = fold && j * 8 + g < p.M ? to_f32<T>(__ldcg(X + (long long)(j * 8 + g) * p.ln_ldx)) : 0.f;
  }
  // what this thread's outputs need: row of C, and per tile bias, column sum and residual, requested before the products
  const T *bias = reinterpret_cast<const T *>(p.bias), *res = reinterpret_cast<const T *>(p.residual);
  const int n_local = p.gated ? threadIdx.x & 7 : threadIdx.x & 15;
  const int m_first = p.gated ? threadIdx.x >> 3 : threadIdx.x >> 4, m_step = kStepThreads / (p.gated ? 8 : 16);
  const int c_row = p.c_row_offset_dev ? __ldg(p.c_row_offset_dev) : 0;
  const bool row_ok = row_in_limit(p, c_row);
  float mean[kPer], rstd[kPer];
#pragma unroll
  for (int i = 0; i < kPer; ++i) { mean[i] = 0.f; rstd[i] = 1.f; }
  float act0 = 0.f, act1 = 0.f;
  if (p.act_params) { act0 = __ldg(p.act_params); act1 = __ldg(p.act_params + 1); }
  asm volatile("cp.async.wait_group 0;" ::: "memory");
  __syncwarp();

  int tile = blockIdx.x, chunk = 0, buf = 0;
  bool first = true;
  float acc[NT][4];
  float b_n = 0.f, colsum = 0.f;
  T r_mn[kPer];
  // The lane's accumulators to its places in this tile's half of `part`, on top of what they hold or not.  (The half's last readers have passed the
  // preceding tile's rendezvous, and so has this warp.)
  auto leave_sums = [&](bool add) {
    float *mine = part + (size_t)(buf * kStepWarps + warp) * (NT * 4) * kStepPart + lane;
#pragma unroll
    for (int j = 0; j < NT; ++j)
#pragma unroll
      for (int e = 0; e < 4; ++e) mine[(j * 4 + e) * kStepPart] = add ? mine[(j * 4 + e) * kStepPart] + acc[j][e] : acc[j][e];
  };
  auto clear_sums = [&]() {
#pragma unroll
    for (int j = 0; j < NT; ++j) acc[j][0] = acc[j][1] = acc[j][2] = acc[j][3] = 0.f;
  };
  auto begin_tile = [&]() {
    clear_sums();
    const int n = tile * 16 + n_local;
    const bool n_ok = n < p.N && !p.gated;
    b_n = !n_ok ? 0.f : fold ? __ldg(p.ln_bias + n) : bias ? to_f32<T>(bias[n]) : 0.f;
    colsum = n_ok && fold ? __ldg(p.ln_colsum + n) : 0.f;
#pragma unroll
    for (int i = 0; i < kPer; ++i) {
      const int m = m_first + i * m_step;
      r_mn[i] = n_ok && res && m < p.M ? __ldcg(res + (long long)m * p.ldr + n) : from_f32<T>(0.f);
    }
  };
  auto finish_tile = [&]() {
    leave_sums(slice > kStepRun);
    if (fold && first) {
#pragma unroll
      for (int j = 0; j < NT; ++j) {
        float s = sum[j][0] + sum[j][1], q = sq[j][0] + sq[j][1];
        s += __shfl_xor_sync(0xffffffffu, s, 1); q += __shfl_xor_sync(0xffffffffu, q, 1);
        s += __shfl_xor_sync(0xffffffffu, s, 2); q += __shfl_xor_sync(0xffffffffu, q, 2);
        if (t == 0) { stats[(warp * kRows + j * 8 + g) * 2] = s; stats[(warp * kRows + j * 8 + g) * 2 + 1] = q; }
      }
    }
    // One rendezvous per tile: the sums of tile i are read from one half while tile i + 1 fills the other, and nobody
    // writes a half again before everybody has passed the next tile's rendezvous.
    __syncthreads();
    if (fold && first) {
#pragma unroll
      for (int i = 0; i < kPer; ++i) {
        const int m = m_first + i * m_step;
        if (m < p.M) {
          float s = 0.f, q = 0.f;
#pragma unroll
          for (int w = 0; w < kStepWarps; ++w) { s += stats[(w * kRows + m) * 2]; q += stats[(w * kRows + m) * 2 + 1]; }
          const float inv_k = 1.f / (float)p.K, ms = s * inv_k;
          mean[i] = to_f32<T>(__ldcg(X + (long long)m * p.ln_ldx)) + ms;
          rstd[i] = rsqrtf(fmaxf(q * inv_k - ms * ms, 0.f) + p.ln_eps);
        }
      }
    }
    first = false;
    const float *sums = part + (size_t)buf * kStepWarps * (NT * 4) * kStepPart;
    buf ^= 1;
    // accumulator element of weight row (n_local, + 8: hi) and batch row m: lane (n_local & 7) * 4 + (m % 8) / 2
    auto total = [&](int row, int m) {
      const float *at = sums + ((m >> 3) * 4 + (row >> 3) * 2 + (m & 1)) * kStepPart + (row & 7) * 4 + ((m & 7) >> 1);
      float v = 0.f;
#pragma unroll
      for (int w = 0; w < kStepWarps; ++w) v += at[w * (NT * 4) * kStepPart];
      return v;
    };
    if (p.gated) {
#pragma unroll
      for (int i = 0; i < kPer; ++i) {
        const int m = m_first + i * m_step, c = tile * 8 + n_local;
        if (m < p.M && row_ok)                                          // (N is a multiple of 16)
          reinterpret_cast<T *>(p.C)[c_row_offset(p, m) + c] = from_f32<T>(unit_value(p.gated, total(n_local, m), total(n_local + 8, m), p.gate_limit, p.gate_alpha));
      }
      return;
    }
    const int n = tile * 16 + n_local;
    if (threadIdx.x < kThreadsUsed && n < p.N && row_ok) {
      const int act = n < p.act_cols ? p.act : EB_ACT_NONE;
#pragma unroll
      for (int i = 0; i < kPer; ++i) {
        const int m = m_first + i * m_step;
        if (m >= p.M) continue;
        float y = rstd[i] * (total(n_local, m) - mean[i] * colsum) + b_n;
        y = act == EB_ACT_XIELU ? xielu_fast(y, act0, act1) : apply_act(y, act);
        y += to_f32<T>(r_mn[i]);
        if (n >= p.tail_col) p.tail[(long long)m * p.ld_tail + (n - p.tail_col)] = y;
        else if (p.out_f32) reinterpret_cast<float *>(p.C)[c_row_offset(p, m) + n] = y;
        else reinterpret_cast<T *>(p.C)[c_row_offset(p, m) + n] = from_f32<T>(y);
      }
    }
  };
  auto step = [&](uint4 (&w)[U][2]) {
    const uint8_t *xk = xs + (size_t)g * pitch + (chunk * 32 * U + t * 8) * 2;
#pragma unroll
    for (int u = 0; u < U; ++u) {
      if (chunk * 32 * U + u * 32 < slice) {                            // (uniform: the slice is a multiple of 32)
#pragma unroll
        for (int j = 0; j < NT; ++j) {
          const uint4 x = *reinterpret_cast<const uint4 *>(xk + (size_t)j * 8 * pitch + u * 64);
          mma_16816<T>(acc[j], w[u][0].x, w[u][1].x, w[u][0].y, w[u][1].y, x.x, x.y);
          mma_16816<T>(acc[j], w[u][0].z, w[u][1].z, w[u][0].w, w[u][1].w, x.z, x.w);
          if (fold && first && kb + chunk * 32 * U + u * 32 + t * 8 < p.K) {
            Vec16<T> v;
            v.raw = x;
            float f[8];
            v.unpack(f);
#pragma unroll
            for (int e = 0; e < 8; e += 2) {
              add2(f[e], f[e + 1], f[e], f[e + 1], -pivot[j], -pivot[j]);
              add2(sum[j][0], sum[j][1], sum[j][0], sum[j][1], f[e], f[e + 1]);
              fma2(sq[j][0], sq[j][1], f[e], f[e + 1], f[e], f[e + 1], sq[j][0], sq[j][1]);
            }
          }
        }
      }
    }
    load(w);
    if (++chunk == chunks) {
      finish_tile();
      chunk = 0;
      tile += gridDim.x;
      if (tile < tiles) begin_tile();
    } else if (chunk == kStepRun / (32 * U)) {            // (once: a slice has at most 512 columns)
      leave_sums(false);
      clear_sums();
    }
    return tile < tiles;
  };
  begin_tile();
  while (step(w0) && step(w1)) {}
}

template <typename T, int NT>
int launch_step_gemm(const GemmParams &p, const void *W, long long ldw, const StepGeometry &s, cudaStream_t st) {
  auto kern = gemm_step_kernel<T, NT>;
  static bool configured[64] = {};
  int dev = 0;
  cudaGetDevice(&dev);
  if (dev >= 0 && dev < 64 && !configured[dev]) {
    if (cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, 227 * 1024) != cudaSuccess) {
      cudaGetLastError();
      return fail(EB_ECUDA, "gemm: cannot reserve shared memory");
    }
    configured[dev] = true;
  }
  const int tiles = (p.N + 15) / 16, most = 2 * sm_count();
  launch_pdl(kern, dim3(tiles < most ? tiles : most), dim3(kStepThreads), s.smem, st, p, W, ldw, s.slice, s.pitch);
  return check_launch("gemm");
}
