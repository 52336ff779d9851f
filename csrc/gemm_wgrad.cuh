// CTA-pair kernel for weight gradients of little depth.  Included by gemm_sm100.cu, whose helpers it uses.
//
//   C_g[M, N] (+)= alpha * A[rows of g, M]^T B[rows of g, N],  C in bf16
//
// What bounds it: the result.  A micro-batch of 576 tokens gives each of 8 experts three 64-row k blocks of depth, 0.8 us of MMAs
// a 256 x 256 tile, and 128 KB to write, as much again to read where gradients are added to: 1.5 or 2.9 us at the rate of the
// memory.  The general pair kernel moves C through registers (fetch, add, flush, one chunk after the other in each warp), which
// leaves its latency exposed once a tile.  Here each epilogue warp owns a small ring of 32 x 64 pieces of C in shared memory: pieces are
// brought in by TMA three ahead, added to in place, and written back by TMA, so that a warp waits for neither direction.  The
// ring takes shared memory from the operands' stages (3 with addition, 5 without), which the little depth does not need.
//
// 8 experts of 14336 x 4096, microseconds, pair kernel / this one (floor: C at the measured copy rate, 143 written, 287 added to):
// 576 tokens 353 / 182 and 533 / 355, 77 tokens 309 / 185 and 530 / 350, 2000 tokens 414 / 348 and 636 / 490.

template <bool ACC> struct WgShape {
  static constexpr int STAGES = ACC ? 3 : 5;
  static constexpr int SLOTS = ACC ? 4 : 2;              // pieces of C per warp
  static constexpr int RING = STAGES * PAIR_STAGE_BYTES, PIECES = EPI_WARPS * SLOTS * EPI_STAGE_BYTES;
};
constexpr int WG_GROUPS = 64;
struct WgTable { int krow0[WG_GROUPS], kb[WG_GROUPS]; };
constexpr int WG_SMEM = WgShape<true>::RING + WgShape<true>::PIECES + 1024 + 512 + (int)sizeof(WgTable);
static_assert(WgShape<true>::RING + WgShape<true>::PIECES == WgShape<false>::RING + WgShape<false>::PIECES, "both forms use the same amount");
static_assert(WG_SMEM <= 227 * 1024, "weight gradient kernel: shared memory of a CTA");

struct WgParams {
  CUtensorMap tmA, tmB, tmC;      // boxes: A, B 64 columns x 64 rows of depth; C 64 columns x 32 rows
  int M, N, K, G;
  const int* offsets; const int* group_rows;
  float alpha; const float* alpha_dev;
  int* status;
};

__host__ __device__ __forceinline__ bool wg_tile(int M, int N, int G, int t, int& g, int& m0, int& n0) {
  const int mb = (M + 255) / 256, nb = (N + 255) / 256;
  g = t / (mb * nb);
  if (g >= G) return false;
  int m, n;
  panel_order(t - g * mb * nb, mb, nb, PANEL_ROWS / 256, m, n);
  m0 = m * 256; n0 = n * 256;
  return true;
}

// A warp's pieces of C in the order in which it meets them: 32 rows from r0, 64 columns from c0 of group g, inside the matrix and of
// groups that have depth.
struct WgPieces {
  int tile, ch, g, r0, c0;
  __device__ __forceinline__ bool next(const WgParams& p, const WgTable* tb, int pairs, int row, int col) {
    while (true) {
      if (++ch == 2) { ch = 0; tile += pairs; }
      int m0, n0;
      if (!wg_tile(p.M, p.N, p.G, tile, g, m0, n0)) return false;
      r0 = m0 + row; c0 = n0 + col + ch * 64;
      if (r0 < p.M && c0 < p.N && tb->kb[g] > 0) return true;
    }
  }
};

template <bool ACC>
__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(GEMM_THREADS, 1) gemm_sm100_wgrad_kernel(const __grid_constant__ WgParams p) {
  constexpr int STAGES = WgShape<ACC>::STAGES, SLOTS = WgShape<ACC>::SLOTS;
  constexpr uint32_t TMEM_COLS = 512;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  uint8_t* pieces = smem + WgShape<ACC>::RING;
  uint64_t* full_bar = reinterpret_cast<uint64_t*>(pieces + WgShape<ACC>::PIECES);
  uint64_t* empty_bar = full_bar + STAGES;
  uint64_t* tfull_bar = empty_bar + STAGES;
  uint64_t* tempty_bar = tfull_bar + 2;
  uint64_t* piece_bar = tempty_bar + 2;                  // [warp][slot]
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(piece_bar + EPI_WARPS * 4);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);
  WgTable* tb = reinterpret_cast<WgTable*>(pieces + WgShape<ACC>::PIECES + 512);

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int rank = (int)cluster_ctarank();
  const int pair_id = (int)cluster_id_x(), num_pairs = (int)num_clusters_x();

  if (threadIdx.x == 0) {
    for (int s = 0; s < STAGES; ++s) { mbar_init(&full_bar[s], 1); mbar_init(&empty_bar[s], 1); }
    for (int b = 0; b < 2; ++b) { mbar_init(&tfull_bar[b], 1); mbar_init(&tempty_bar[b], 2 * EPI_WARPS); }
    for (int i = 0; i < EPI_WARPS * 4; ++i) mbar_init(&piece_bar[i], 1);
    *abort_flag = 0;
    fence_barrier_init();
  }
  if (warp == 1) { tmem_alloc_pair(tmem_slot, TMEM_COLS); tmem_relinquish_pair(); }
  if (warp == 2) {
    wait_for_predecessor();
    for (int g = lane; g < p.G; g += 32) {
      const int begin = p.offsets != nullptr ? p.offsets[g] : 0;
      int rows = p.offsets != nullptr ? p.offsets[g + 1] - begin : p.K;
      if (p.group_rows != nullptr && p.group_rows[g] < rows) rows = p.group_rows[g];      // (the rest of the group is zero)
      tb->krow0[g] = begin;
      tb->kb[g] = (rows + BK - 1) / BK;
    }
  }
  tc_fence_before();
  cluster_sync_all();
  tc_fence_after();
  const uint32_t tmem_base = *tmem_slot;
  after_predecessor();
  auto fail = [&](int code) {
    *abort_flag = 1;
    if (p.status != nullptr) atomicCAS(p.status, 0, code);
  };

  if (warp == 0) {
    // ------------------------------------------------------------------ TMA producer (one per CTA)
    if (elect_one()) { prefetch_tensormap(&p.tmA); prefetch_tensormap(&p.tmB); prefetch_tensormap(&p.tmC); }
    int s = 0, g, m0, n0;
    uint32_t ph = 0;
    bool ok = true;
    for (int tile = pair_id; ok && wg_tile(p.M, p.N, p.G, tile, g, m0, n0); tile += num_pairs) {
      const int kb_n = tb->kb[g], krow0 = tb->krow0[g], m = m0 + rank * BM, n = n0 + rank * 128;
      for (int kb = 0; kb < kb_n; ++kb) {
        if (!wait_parity_warp(&empty_bar[s], ph ^ 1, abort_flag)) { fail(ST_TIMEOUT_EMPTY); ok = false; break; }
        uint8_t* sA = smem + s * PAIR_STAGE_BYTES;
        uint8_t* sB = sA + A_BYTES;
        const uint32_t bar = mapa_shared(smem_u32(&full_bar[s]), 0);      // (only the leader arrives, see the pair kernel)
        const int krow = krow0 + kb * BK;
        if (elect_one()) {
          if (rank == 0) mbar_expect_tx(&full_bar[s], 2 * PAIR_STAGE_BYTES);
          tma_load_2d_pair(sA, &p.tmA, bar, m, krow);
          tma_load_2d_pair(sA + 8192, &p.tmA, bar, m + 64, krow);
          tma_load_2d_pair(sB, &p.tmB, bar, n, krow);
          tma_load_2d_pair(sB + 8192, &p.tmB, bar, n + 64, krow);
        }
        if (++s == STAGES) { s = 0; ph ^= 1; }
      }
    }
    if (!ok) {  // give this CTA's copies already in flight a bounded time to land before it leaves
      const uint64_t t0 = global_timer_ns();
      while (global_timer_ns() - t0 < 2000000ull) {}
    }
  } else if (warp == 1 && rank == 0) {
    // ------------------------------------------------------------------ MMA issuer (leader only)
    const uint32_t idesc = make_idesc_bf16(2 * BM, 256, 1, 1);
    int s = 0, g, m0, n0;
    uint32_t ph = 0, acc_it = 0;
    bool ok = true;
    for (int tile = pair_id; ok && wg_tile(p.M, p.N, p.G, tile, g, m0, n0); tile += num_pairs) {
      const int kb_n = tb->kb[g];
      if (kb_n == 0) continue;
      const int buf = acc_it & 1;
      if (!wait_parity_warp(&tempty_bar[buf], ((acc_it >> 1) & 1) ^ 1, abort_flag)) { fail(ST_TIMEOUT_TMEM_EMPTY); break; }
      tc_fence_after();
      const uint32_t d_tmem = tmem_base + buf * 256;
      for (int kb = 0; kb < kb_n; ++kb) {
        if (!wait_parity_warp(&full_bar[s], ph, abort_flag)) { fail(ST_TIMEOUT_FULL); ok = false; break; }
        tc_fence_after();
        const uint32_t sA = smem_u32(smem + s * PAIR_STAGE_BYTES);
        const uint64_t da = operand_desc(sA, 1), db = operand_desc(sA + A_BYTES, 1);
        const uint32_t step = operand_kstep(1);
        if (elect_one()) {
#pragma unroll
          for (int k = 0; k < BK / 16; ++k) umma_bf16_pair(d_tmem, da + k * step, db + k * step, idesc, (kb > 0 || k > 0) ? 1u : 0u);
          umma_commit_pair(&empty_bar[s], 3);
        }
        if (++s == STAGES) { s = 0; ph ^= 1; }
      }
      if (!ok) break;
      if (elect_one()) umma_commit_pair(&tfull_bar[buf], 3);
      ++acc_it;
    }
  } else if (warp >= 2) {
    // ------------------------------------------------------------------ epilogue (both CTAs, own 128 rows)
    const int q = warp & 3, half = (warp - 2) >> 2, row = rank * BM + q * 32, col = half * 128;
    uint8_t* my = pieces + (warp - 2) * SLOTS * EPI_STAGE_BYTES;
    uint64_t* bars = piece_bar + (warp - 2) * 4;
    const float alpha = p.alpha_dev != nullptr ? p.alpha * *p.alpha_dev : p.alpha;
    uint32_t acc_it = 0, c = 0;                 // tiles with depth, pieces so far
    WgPieces ahead = {pair_id, -1, 0, 0, 0};    // the piece that is brought in next
    auto bring = [&](uint32_t slot) {
      if (ahead.next(p, tb, num_pairs, row, col) && lane == 0) {
        mbar_expect_tx(&bars[slot], EPI_STAGE_BYTES);
        tma_load_3d(my + slot * EPI_STAGE_BYTES, &p.tmC, &bars[slot], ahead.c0, ahead.r0, ahead.g);
      }
    };
    if (ACC) { for (uint32_t i = 0; i < SLOTS - 1; ++i) bring(i); }
    int g, m0, n0;
    bool ok = true;
    for (int tile = pair_id; ok && wg_tile(p.M, p.N, p.G, tile, g, m0, n0); tile += num_pairs) {
      const bool depth = tb->kb[g] > 0;
      if (ACC && !depth) continue;                                  // nothing is added
      const int buf = acc_it & 1;
      if (depth) {
        if (!wait_parity_warp(&tfull_bar[buf], (acc_it >> 1) & 1, abort_flag)) { fail(ST_TIMEOUT_TMEM_FULL); break; }
        tc_fence_after();
      }
      const int r0 = m0 + row;
#pragma unroll 1
      for (int ch = 0; ch < 2; ++ch) {
        const int c0 = n0 + col + ch * 64;
        if (r0 >= p.M || c0 >= p.N) continue;
        const uint32_t slot = c % SLOTS;
        uint8_t* piece = my + slot * EPI_STAGE_BYTES;
        if (ACC) {
          if (!wait_parity_warp(&bars[slot], (c / SLOTS) & 1, abort_flag)) { fail(ST_TIMEOUT_FULL); ok = false; break; }
        } else {
          if (lane == 0) bulk_wait_read<1>();                       // the store of two pieces ago has left the slot
          __syncwarp();
        }
#pragma unroll
        for (int part = 0; part < 2; ++part) {
          float v[32];
          if (depth) {
            uint32_t acc[32];
            tmem_ld_32x32(tmem_base + buf * 256 + ((uint32_t)(q * 32) << 16) + col + ch * 64 + part * 32, acc);
            tmem_ld_wait();
#pragma unroll
            for (int i = 0; i < 32; ++i) v[i] = __uint_as_float(acc[i]) * alpha;
          } else {
#pragma unroll
            for (int i = 0; i < 32; ++i) v[i] = 0.f;
          }
          epi_stage_row<ACC>(piece, v, part, lane);
        }
        fence_proxy_async();
        __syncwarp();
        if (lane == 0) { tma_store_3d(&p.tmC, piece, c0, r0, g); bulk_commit(); }
        ++c;
        if (ACC) {
          if (lane == 0) bulk_wait_read<1>();                       // the store before this one has left its slot
          __syncwarp();
          bring((c + SLOTS - 2) % SLOTS);
        }
      }
      if (!ok) break;
      if (depth) {
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive_cluster(mapa_shared(smem_u32(&tempty_bar[buf]), 0));
        ++acc_it;
      }
    }
    if (lane == 0) bulk_wait_all();
    if (*abort_flag) {       // pieces that were on their way
      const uint64_t t0 = global_timer_ns();
      while (global_timer_ns() - t0 < 2000000ull) {}
    }
  }

  // Neither CTA may leave while its partner can still read its shared memory or arrive on its barriers.
  __syncwarp();
  tc_fence_before();
  cluster_sync_all();
  if (warp == 1) { tc_fence_after(); tmem_dealloc_pair(tmem_base, TMEM_COLS); }
}
