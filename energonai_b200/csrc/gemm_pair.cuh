// C = act(A · Wᵀ + bias) + residual for prompt-sized products, a tile of 256 rows x BN columns per pair of SMs
// (included by gemm.cu).
//
// With one SM per tile the operands' way through shared memory sets the pace: a 128 x 256 x 64 block is written (48 KB) and
// read (48 KB) in the 512 cycles its MMAs take.  Here the two CTAs of a cluster share one tcgen05.mma of 256 x BN: each
// holds 128 rows of A, half of the BN rows of W and half of the accumulator (its 128 rows, all BN columns), so a
// k-block moves 32 KB instead of 48.  Two k-blocks per stage: with one, the hand-over of a stage (0.25-0.3 us) set the pace of the
// narrow tiles.
//
// Who signals whom (rank 0 of the pair leads):
//   full    leader's: the copies of both CTAs complete on it; its one arrival announces the bytes of both
//   empty   each CTA's own: the leader's commit arrives on both once the MMAs have read the stage
//   tfull   each CTA's own: accumulator complete, likewise
//   tempty  leader's: one arrival per epilogue warp of either CTA
// Waits are bounded as in the one-SM kernel; a CTA leaves only when its peer has passed the same rendezvous, so no signal
// goes to a CTA that is gone.
constexpr int kPairBlocks = 2;                       // k-blocks per stage
constexpr uint32_t kPairStagingBytes = 2048 + 64;    // per epilogue warp: 32 rows x 32 columns of C, 32 columns of the bias

__device__ __forceinline__ uint32_t leader_addr(uint32_t addr) {
  uint32_t r;
  asm volatile("mapa.shared::cluster.u32 %0, %1, 0;" : "=r"(r) : "r"(addr));
  return r;
}
__device__ __forceinline__ void pair_load_2d(uint32_t dst, const CUtensorMap *map, uint32_t leader_bar, int x, int y) {
  asm volatile(
      "cp.async.bulk.tensor.2d.shared::cluster.global.tile.mbarrier::complete_tx::bytes.cta_group::2 [%0], [%1, {%2, %3}], [%4];"
      ::"r"(dst), "l"(map), "r"(x), "r"(y), "r"(leader_bar)
      : "memory");
}
__device__ __forceinline__ void pair_commit(uint32_t bar) {
  asm volatile(
      "{\n\t.reg .pred q;\n\telect.sync _|q, 0xffffffff;\n\t"
      "@q tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], %1;\n\t}" ::"r"(bar), "h"((uint16_t)3)
      : "memory");
}
// The four MMAs of a k-block (16 columns = 32 bytes = 2 in the descriptors' address field apart), issued by one elected lane of a
// converged warp.
__device__ __forceinline__ void pair_mma_block(uint32_t d_tmem, uint64_t a, uint64_t b, uint32_t idesc, uint32_t accumulate) {
  asm volatile(
      "{\n\t.reg .pred p, q;\n\t"
      "elect.sync _|q, 0xffffffff;\n\t"
      "setp.ne.b32 p, %10, 0;\n\t"
      "@q tcgen05.mma.cta_group::2.kind::f16 [%0], %1, %5, %9, p;\n\t"
      "@q tcgen05.mma.cta_group::2.kind::f16 [%0], %2, %6, %9, 1;\n\t"
      "@q tcgen05.mma.cta_group::2.kind::f16 [%0], %3, %7, %9, 1;\n\t"
      "@q tcgen05.mma.cta_group::2.kind::f16 [%0], %4, %8, %9, 1;\n\t}"
      ::"r"(d_tmem), "l"(a), "l"(a + 2), "l"(a + 4), "l"(a + 6), "l"(b), "l"(b + 2), "l"(b + 4), "l"(b + 6), "r"(idesc), "r"(accumulate)
      : "memory");
}
__device__ __forceinline__ void cluster_rendezvous() {
  asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}

// Output tile number `pos` of the raster: groups of kGroup / 2 row tiles, so that the pairs running at the same time share
// panels of both operands in L2.
__device__ __forceinline__ void pair_tile(int pos, int row_tiles, int col_tiles, int &row_tile, int &col_tile) {
  constexpr int kRows = kGroup / 2;
  const int per_group = kRows * col_tiles, group = pos / per_group, in_group = pos - group * per_group;
  const int first = group * kRows, size = min(kRows, row_tiles - first);
  col_tile = in_group / size;
  row_tile = first + in_group - col_tile * size;
}

// 32 accumulator columns of 32 rows, requested; `tmem_ld32_wait` makes them valid.
__device__ __forceinline__ void tmem_ld32_request(uint32_t taddr, uint32_t (&r)[32]) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x32.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16,%17,%18,%19,%20,%21,%22,%23,%24,%25,%26,"
      "%27,%28,%29,%30,%31}, [%32];"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]), "=r"(r[9]), "=r"(r[10]),
        "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15]), "=r"(r[16]), "=r"(r[17]), "=r"(r[18]), "=r"(r[19]), "=r"(r[20]),
        "=r"(r[21]), "=r"(r[22]), "=r"(r[23]), "=r"(r[24]), "=r"(r[25]), "=r"(r[26]), "=r"(r[27]), "=r"(r[28]), "=r"(r[29]), "=r"(r[30]),
        "=r"(r[31])
      : "r"(taddr));
}
__device__ __forceinline__ void tmem_ld32_wait(uint32_t (&r)[32]) {
  asm volatile("tcgen05.wait::ld.sync.aligned;"
               : "+r"(r[0]), "+r"(r[1]), "+r"(r[2]), "+r"(r[3]), "+r"(r[4]), "+r"(r[5]), "+r"(r[6]), "+r"(r[7]), "+r"(r[8]), "+r"(r[9]),
                 "+r"(r[10]), "+r"(r[11]), "+r"(r[12]), "+r"(r[13]), "+r"(r[14]), "+r"(r[15]), "+r"(r[16]), "+r"(r[17]), "+r"(r[18]),
                 "+r"(r[19]), "+r"(r[20]), "+r"(r[21]), "+r"(r[22]), "+r"(r[23]), "+r"(r[24]), "+r"(r[25]), "+r"(r[26]), "+r"(r[27]),
                 "+r"(r[28]), "+r"(r[29]), "+r"(r[30]), "+r"(r[31])::"memory");
}

// A warp's 32 rows from m0 on x COLS columns from n0 on, out of tensor memory.  There a thread holds one row, and 32 rows
// stored (or a residual read) 16 bytes at a time are 32 transactions per instruction.  32 columns at a time go through shared memory in the
// output type instead (`stage`: 64 bytes per row, its 16-byte units permuted by the row against bank conflicts): the residual comes in and
// the result leaves as 64 contiguous bytes per row.  `acquire` waits for the accumulator (false: it never came), `release` is called when it
// has been read.
template <typename T, int COLS, typename Acquire, typename Release>
__device__ __forceinline__ bool store_staged(const GemmParams &p, uint32_t t_base, int m0, int n0, uint4 *stage, Acquire acquire, Release release) {
  constexpr int kChunks = COLS / 32;
  const int lane = threadIdx.x & 31, unit = lane & 3, row_in = lane >> 2;
  const T *bias = reinterpret_cast<const T *>(p.bias), *res = reinterpret_cast<const T *>(p.residual);
  const bool row_ok = row_in_limit(p, p.c_row_offset_dev ? __ldg(p.c_row_offset_dev) : 0);
  const int rows = row_ok ? min(32, p.M - m0) : 0;       // (may be negative: nothing is stored)
  uint4 *bias_stage = stage + 128;
  auto slot = [&](int row, int u) { return stage + row * 4 + (u ^ ((row >> 1) & 3)); };
  // The bias of a chunk (lanes 0 to 3, a unit each) and this lane's part of its residual, requested a chunk ahead: loaded where they are
  // used, the units' trips to L2 came one after the other.
  uint4 rq[4], bq = make_uint4(0u, 0u, 0u, 0u);
  auto fetch = [&](int n_chunk) {
    if (bias && lane < 4 && n_chunk + lane * 8 < p.N) bq = *reinterpret_cast<const uint4 *>(bias + n_chunk + lane * 8);
    if (res) {
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const int row = row_in + 8 * i, n = n_chunk + unit * 8;
        rq[i] = row < rows && n < p.N ? *reinterpret_cast<const uint4 *>(res + (long long)(m0 + row) * p.ldr + n) : make_uint4(0u, 0u, 0u, 0u);
      }
    }
  };
  fetch(n0);
  if (!acquire()) return false;
#pragma unroll 1
  for (int c = 0; c < kChunks; ++c) {
    const int n_chunk = n0 + c * 32;
    uint32_t r[32];
    tmem_ld32_request(t_base + c * 32, r);
    __syncwarp();                                        // the previous chunk (the previous tile's last) has left
    if (lane < 4) bias_stage[lane] = bq;
    if (res) {
#pragma unroll
      for (int i = 0; i < 4; ++i) *slot(row_in + 8 * i, unit) = rq[i];
    }
    __syncwarp();
    if (c + 1 < kChunks) fetch(n_chunk + 32);
    tmem_ld32_wait(r);
    if (c == kChunks - 1) release();
    if (n_chunk >= p.N || rows <= 0) continue;           // warp-uniform
    if (p.gated) {                                       // 16 columns: 8 gates and their 8 ups (N is a multiple of 16)
#pragma unroll
      for (int q = 0; q < 2; ++q) {
        float y[8];
#pragma unroll
        for (int j = 0; j < 8; ++j) {
          const float g = __uint_as_float(r[q * 16 + j]), up = __uint_as_float(r[q * 16 + 8 + j]);
          y[j] = p.gated == EB_UNIT_GEGLU ? gelu_tanh_value(g) * up : gated_value(g, up, p.gate_limit, p.gate_alpha);
        }
        Vec16<T> o;
        o.pack(y);
        *slot(lane, q) = o.raw;
      }
      __syncwarp();
#pragma unroll
      for (int i = 0; i < 2; ++i) {
        const int row = (lane >> 1) + 16 * i, q = lane & 1;
        const uint4 o = *slot(row, q);
        if (row < rows && n_chunk + q * 16 < p.N)
          *reinterpret_cast<uint4 *>(reinterpret_cast<T *>(p.C) + (long long)(m0 + row) * p.ldc + n_chunk / 2 + q * 8) = o;
      }
      continue;
    }
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      const int n = n_chunk + u * 8;                     // (N is a multiple of 8)
      if (n >= p.N) break;
      const int act = n < p.act_cols ? p.act : EB_ACT_NONE;
      float v[8];
      Vec16<T> b;
      b.raw = bias_stage[u];
      b.unpack(v);
#pragma unroll
      for (int j = 0; j < 8; ++j) v[j] += __uint_as_float(r[u * 8 + j]);
      if (act == EB_ACT_RELU) {
#pragma unroll
        for (int j = 0; j < 8; ++j) v[j] = fmaxf(v[j], 0.f);
      } else if (act == EB_ACT_XIELU) {
        const float act0 = __ldg(p.act_params), act1 = __ldg(p.act_params + 1);
#pragma unroll
        for (int j = 0; j < 8; ++j) v[j] = xielu_fast(v[j], act0, act1);
      } else if (act == EB_ACT_GELU_ERF) {
#pragma unroll
        for (int j = 0; j < 8; ++j) v[j] = gelu_erf_fast(v[j]);
      } else if (act != EB_ACT_NONE) {
#pragma unroll
        for (int j = 0; j < 8; ++j) v[j] = apply_act(v[j], act);
      }
      if (res) {
        Vec16<T> q;
        float rf[8];
        q.raw = *slot(lane, u);
        q.unpack(rf);
#pragma unroll
        for (int j = 0; j < 8; ++j) v[j] += rf[j];
      }
      if (n >= p.tail_col || p.out_f32) {                // fp32 results leave straight from the registers
        if (lane < rows) {
          float4 *o = reinterpret_cast<float4 *>(n >= p.tail_col ? p.tail + (long long)(m0 + lane) * p.ld_tail + (n - p.tail_col)
                                                                : reinterpret_cast<float *>(p.C) + c_row_offset(p, m0 + lane) + n);
          o[0] = make_float4(v[0], v[1], v[2], v[3]);
          o[1] = make_float4(v[4], v[5], v[6], v[7]);
        }
      } else {
        Vec16<T> o;
        o.pack(v);
        *slot(lane, u) = o.raw;
      }
    }
    if (p.out_f32) continue;
    __syncwarp();
    const int n = n_chunk + unit * 8;
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const int row = row_in + 8 * i;
      const uint4 o = *slot(row, unit);
      if (row < rows && n < p.N && n < p.tail_col) *reinterpret_cast<uint4 *>(reinterpret_cast<T *>(p.C) + c_row_offset(p, m0 + row) + n) = o;
    }
  }
  return true;
}

// EW: epilogue warps, 8 or 16 (see the launch)
template <typename T, int BN, int EW>
__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(64 + 32 * EW, 1)
gemm_pair_kernel(const __grid_constant__ CUtensorMap tm_a, const __grid_constant__ CUtensorMap tm_w, const GemmParams p) {
  constexpr uint32_t kABytes = kLanes * 128u, kWBytes = BN / 2 * 128u, kBlock = kABytes + kWBytes, kStage = kPairBlocks * kBlock;
  constexpr uint32_t kTmemCols = 2 * BN;
  constexpr uint32_t kIdesc = (make_idesc(BN, std::is_same<T, __nv_bfloat16>::value ? 1 : 0) & ~(31u << 24)) | (256u >> 4) << 24;
  constexpr int kCols = BN / (EW / 4);                 // columns per epilogue warp
  extern __shared__ uint8_t smem_raw[];
  const uint32_t raw_addr = smem_u32(smem_raw);
  uint8_t *smem = smem_raw + (((raw_addr + 1023u) & ~1023u) - raw_addr);
  uint64_t *bars = reinterpret_cast<uint64_t *>(smem);
  const uint32_t full_bar = smem_u32(bars), empty_bar = full_bar + 8 * kMaxStages;
  const uint32_t tfull_bar = empty_bar + 8 * kMaxStages, tempty_bar = tfull_bar + 16;
  uint32_t *tmem_slot = reinterpret_cast<uint32_t *>(bars + 2 * kMaxStages + 4);
  volatile int *abort_flag = reinterpret_cast<volatile int *>(tmem_slot + 1), *came = abort_flag + 1;
  const uint32_t tiles_addr = smem_u32(smem) + kBarrierBytes;
  const int stages = p.stages, warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int rank = blockIdx.x & 1, pair = blockIdx.x >> 1, pairs = gridDim.x >> 1;
  const int row_tiles = (p.M + 255) / 256, col_tiles = (p.N + BN - 1) / BN, tiles = row_tiles * col_tiles;

  if (threadIdx.x == 0) {
    asm volatile("prefetch.tensormap [%0];" ::"l"(&tm_a) : "memory");
    asm volatile("prefetch.tensormap [%0];" ::"l"(&tm_w) : "memory");
    for (int s = 0; s < stages; ++s) {
      mbar_init(full_bar + 8 * s, 1);
      mbar_init(empty_bar + 8 * s, 1);
    }
    for (int a = 0; a < 2; ++a) {
      mbar_init(tfull_bar + 8 * a, 1);
      mbar_init(tempty_bar + 8 * a, 2 * EW);
    }
    *abort_flag = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == 1) {
    __syncwarp();
    asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmem_slot)), "r"(kTmemCols) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
  }
  tcgen05_fence_before();
  __syncthreads();
  cluster_rendezvous();                                // the peer's barriers are ready as well
  tcgen05_fence_after();
  const uint32_t tmem_base = *tmem_slot;
  griddep_launch();

  if (warp == 0) {
    // ---------------- copies: this CTA's rows of A and its half of the tile's rows of W ----------------
    if (lane == 0) {
      const uint32_t leader_full = leader_addr(full_bar);
      const int nsk = (p.kblocks + kPairBlocks - 1) / kPairBlocks;
      // A stage holds [block][rows of A][rows of W]; the last one of a tile may have fewer blocks.
      auto expect = [&](int stage, int sk) {
        if (rank == 0) mbar_expect_tx(full_bar + 8 * stage, 2 * kBlock * (uint32_t)min(kPairBlocks, p.kblocks - sk * kPairBlocks));
      };
      auto fetch = [&](const CUtensorMap *map, int stage, uint32_t off, int sk, int row) {
#pragma unroll
        for (int j = 0; j < kPairBlocks; ++j)
          if (sk * kPairBlocks + j < p.kblocks)
            pair_load_2d(tiles_addr + stage * kStage + j * kBlock + off, map, leader_full + 8 * stage, (sk * kPairBlocks + j) * kBlockK, row);
      };
      int pre = 0;
      if (!p.static_w) griddep_wait();
      for (int pos = pair; pos < tiles && pre < stages; pos += pairs) {       // weights of the first stages, ahead of the preceding kernel
        int rt, ct;
        pair_tile(pos, row_tiles, col_tiles, rt, ct);
        for (int sk = 0; sk < nsk && pre < stages; ++sk, ++pre) {
          expect(pre, sk);
          fetch(&tm_w, pre, kABytes, sk, ct * BN + rank * (BN / 2));
        }
      }
      if (p.static_w) griddep_wait();
      int stage = 0, iter = 0;
      uint32_t phase = 0;
      bool ok = true;
      for (int pos = pair; ok && pos < tiles; pos += pairs) {
        int rt, ct;
        pair_tile(pos, row_tiles, col_tiles, rt, ct);
        for (int sk = 0; sk < nsk; ++sk, ++iter) {
          if (iter >= pre) {
            if (!mbar_wait(empty_bar + 8 * stage, phase ^ 1u, abort_flag, 11)) { ok = false; break; }
            expect(stage, sk);
            fetch(&tm_w, stage, kABytes, sk, ct * BN + rank * (BN / 2));
          }
          fetch(&tm_a, stage, 0, sk, rt * 256 + rank * kLanes);
          if (++stage == stages) { stage = 0; phase ^= 1u; }
        }
      }
      // The hand-backs of the last stages, which no copy waits for: nothing orders them before the accumulator's signal, and the leader
      // must not send them to a CTA that has left.  (A stage that was never filled counts as handed back.)
      for (int s = 0; ok && s < stages; ++s) {
        ok = mbar_wait(empty_bar + 8 * stage, phase ^ 1u, abort_flag, 15);
        if (++stage == stages) { stage = 0; phase ^= 1u; }
      }
    }
    __syncwarp();
  } else if (warp == 1) {
    // ---------------- MMAs: the leader's warp, for both ----------------
    griddep_wait();
    if (rank == 0) {
      auto wait = [&](uint32_t bar, uint32_t parity, int where) { return __all_sync(0xffffffffu, mbar_wait(bar, parity, abort_flag, where)) != 0; };
      int stage = 0, acc = 0;
      uint32_t phase = 0, acc_phase = 0;
      bool ok = true;
      for (int pos = pair; ok && pos < tiles; pos += pairs) {
        if (!wait(tempty_bar + 8 * acc, acc_phase ^ 1u, 12)) break;
        tcgen05_fence_after();
        for (int kb = 0; kb < p.kblocks; kb += kPairBlocks) {
          if (!wait(full_bar + 8 * stage, phase, 13)) { ok = false; break; }
          tcgen05_fence_after();
          const uint32_t at = tiles_addr + stage * kStage;
#pragma unroll
          for (int j = 0; j < kPairBlocks; ++j)
            if (kb + j < p.kblocks)
              pair_mma_block(tmem_base + acc * BN, make_smem_desc(at + j * kBlock), make_smem_desc(at + j * kBlock + kABytes), kIdesc, kb + j > 0 ? 1u : 0u);
          pair_commit(empty_bar + 8 * stage);
          if (++stage == stages) { stage = 0; phase ^= 1u; }
        }
        if (!ok) break;
        pair_commit(tfull_bar + 8 * acc);
        if (++acc == 2) { acc = 0; acc_phase ^= 1u; }
      }
    }
  } else {
    // ---------------- epilogue: a warp has 32 of the CTA's 128 rows and kCols of the columns ----------------
    griddep_wait();
    const int quarter = warp & 3, part = (warp - 2) >> 2;
    const uint32_t leader_tempty = leader_addr(tempty_bar);
    uint4 *stage = reinterpret_cast<uint4 *>(smem + kBarrierBytes + stages * kStage + (warp - 2) * kPairStagingBytes);
    int acc = 0;
    uint32_t acc_phase = 0;
    for (int pos = pair; pos < tiles; pos += pairs) {
      int rt, ct;
      pair_tile(pos, row_tiles, col_tiles, rt, ct);
      const uint32_t t_base = tmem_base + ((uint32_t)(quarter * 32) << 16) + acc * BN + part * kCols;
      auto acquire = [&]() {
        // One warp looks; the others sleep at a hardware barrier, which it always reaches (with all of them looking the main loop ran 4-8 %
        // slower).  Its answer has a place per accumulator, so that nobody reads the next one's.
        if (warp == 2) {
          const bool ok = __all_sync(0xffffffffu, mbar_wait(tfull_bar + 8 * acc, acc_phase, abort_flag, 14)) != 0;
          if (lane == 0) came[acc] = ok;
        }
        asm volatile("bar.sync 1, %0;" ::"n"(32 * EW) : "memory");
        tcgen05_fence_after();
        return came[acc] != 0;
      };
      auto release = [&]() {
        tcgen05_fence_before();
        __syncwarp();
        if (lane == 0) asm volatile("mbarrier.arrive.release.cluster.shared::cluster.b64 _, [%0];" ::"r"(leader_tempty + 8 * acc) : "memory");
      };
      if (!store_staged<T, kCols>(p, t_base, rt * 256 + rank * kLanes + quarter * 32, ct * BN + part * kCols, stage, acquire, release)) break;
      if (++acc == 2) { acc = 0; acc_phase ^= 1u; }
    }
  }

  tcgen05_fence_before();
  __syncthreads();
  if (*abort_flag) {                                   // bounded grace period for copies in flight to this CTA's shared memory
    const unsigned long long t0 = globaltimer();
    while (globaltimer() - t0 < 2000000ull) __nanosleep(1000);
    __syncthreads();
  }
  cluster_rendezvous();
  if (warp == 1) {
    __syncwarp();
    tcgen05_fence_after();
    asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"(kTmemCols) : "memory");
  }
}
