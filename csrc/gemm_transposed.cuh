// Transposed CTA-pair kernel of the GEMM family: the weight matrix is the 256-row operand of the MMA, the token rows are its N.
// Included by gemm_sm100.cu, whose helpers it uses.
//
//   D[features, rows] = W[features, k] * X[rows, k]^T,   C[row, feature] = D^T through SwiGLU, its backward, or nothing
//
// Why: the token rows of an expert come in any number (a micro-batch leaves 30 to 300 for each of 8), the weights always in
// thousands.  With tokens as M a group of 144 rows is two 128-row tiles, one of them holding 16 rows, and the weights pass
// through the SMs once for each; as N it is one 160-wide tile.  Shared memory bounds a k block of n rows at 256 + n clocks of a
// pair (2 x (32 KB of weights + n x 128 bytes) through 2 SMs' 128 bytes per clock); measured are 430 at 128 rows and 640 at 256
// (tp_clocks), against 700 that the weights' 32 KB take from HBM, so that up to 256 rows a group the products run at the
// rate of the weights.
//
// Rows of a group are cut into tiles of equal numbers of 32-row units, at most 8 (256 rows), or 16 where tp_joint_pays says so: such a
// tile is two products with one copy of the weights in shared memory, in both accumulators.  Only rows that exist are
// multiplied where the caller passes their number (group_rows); the padding up to the next 128-row boundary, zero by contract,
// gives zeros, which are written without being computed.  Every tile is multiplied by one pair, its depth in ascending order as in the
// pair kernel: results are the same bits in every run, and those of that kernel.
//
// Epilogue: TMEM is read in 16 x 256-bit pieces, whose register layout is the one that stmatrix transposes, so that rows of C
// leave through a 4 KB stage per warp in 16-byte pieces without shuffles.  In the gate / up form the 128 rows of a CTA's
// operand alternate between 16 gate and 16 up features: both values of one output then land in the same thread.

constexpr int TP_GROUPS = 64;      // row groups that fit the table in shared memory
constexpr int TP_UNIT = 32;        // rows: N of a pair's MMA is a multiple of 32
constexpr int TP_A_BYTES = BM * BK * 2;
// The ring: stages of 16 KB of weights and as many rows as the widest tile has.  Six of 256 rows, ten of 32: what bounds the
// products of few rows is the bytes of weights in flight.
constexpr int TP_RING_BYTES = 6 * (TP_A_BYTES + 128 * BK * 2);
constexpr int TP_MAX_STAGES = 10;
// (groups in the order of the rows of their tiles, most first: see tp_work; units, groups, row_tiles: totals that the host check of the
// enumeration keeps)
struct TPTable { int group[TP_GROUPS], start[TP_GROUPS], rows[TP_GROUPS], end[TP_GROUPS], tile0[TP_GROUPS + 1], widest, units, groups, row_tiles, cap; };
constexpr int TP_SMEM = TP_RING_BYTES + 1024 + 256 + EPI_WARPS * EPI_STAGE_BYTES + (int)sizeof(TPTable);
static_assert(TP_SMEM <= 227 * 1024, "transposed pair kernel: shared memory of a CTA");

enum : int { TP_PLAIN = 0, TP_DUAL = 1, TP_SWIGLU_BWD = 2 };

struct TPParams {
  CUtensorMap tmW, tmW2, tmW_l, tmW2_l;   // weights (tmW2: the up matrix of the gate / up form), main and short depth segment
  CUtensorMap tmX[4], tmX_l[4];           // token rows in boxes of 16, 32, 64 and 128 rows
  int M, N, K, K_l, G, mode, w_mn, w_mn_l;
  const int* offsets; const int* group_rows;
  void* C; void* C2; void* C3;
  const void* swiglu_g; const void* swiglu_u;
  long long ldc;
  float alpha; const float* alpha_dev;
  int* status;
};
// rows [row0, row0 + n) x features [f0, f0 + 256 or 128), rows below `end` are stored; zero0: first row to be cleared (= end: none)
struct TPTile { int g, f0, row0, n, end, zero0; };
// A pair's work: a tile and its k blocks.  No tile is shared along the depth, so these are all of them: split < 0, one contributor.
struct TPWork { TPTile t; int kb0, kb1, split, contributors; };

__host__ __device__ __forceinline__ int tp_tiles_of_rows(int rows, int cap) { return ((rows + TP_UNIT - 1) / TP_UNIT + cap - 1) / cap; }
// rows of its widest tile
__host__ __device__ __forceinline__ int tp_tile_rows(int rows, int cap) {
  const int units = (rows + TP_UNIT - 1) / TP_UNIT, nt = tp_tiles_of_rows(rows, cap);
  return nt > 0 ? (units + nt - 1) / nt * TP_UNIT : 0;
}
// rows of the first accumulator of a tile of n rows
__host__ __device__ __forceinline__ int tp_first(int n) { return n > 256 ? (n / TP_UNIT + 1) / 2 * TP_UNIT : n; }

// Clocks of a k block for a tile of n rows with little else on the chip (measured: n = 128 430, 160 525, 192 556, 256 640), and for one
// with two accumulators, which copies the weights to shared memory once: what the measurements below ask for.
__host__ __device__ __forceinline__ float tp_clocks(int n) { return n <= 256 ? 220.f + 1.64f * (float)n : 150.f + 2.1f * (float)n; }
// Clocks of a pair for all tiles: `row_tiles` of them for each of f_tiles, `step` a k block of one (`longest`: of the longest),
// `rows` rows each.
__host__ __device__ __forceinline__ float tp_clocks_of_all(int row_tiles, int f_tiles, int pairs, int kbt, float step, float longest, float rows, float epilogue) {
  const int total = row_tiles * f_tiles, rounds = (total + pairs - 1) / pairs;
  return (float)rounds * ((float)kbt * (total <= pairs ? longest : step) + epilogue * rows);
}
// Whether tiles of up to 512 rows are taken (sums over the groups: tiles, k block clocks; longest, of both forms).  Such a tile reads
// its weights once for twice the rows, but takes both accumulators, so that nothing hides its epilogue (8 clocks a row), and there are
// fewer of them to go round.  us in turn, up to 256 / up to 512 rows, 8 experts of 4096 x 14336: down 800 tokens 247 / 194, 1250 345 / 271,
// 1750 425 / 462, 2000 386 / 427, 4000 794 / 736, 9200 1494 / 1457; dx (two matrices) 474 / 366, 658 / 511, 763 / 821, 816 / 902,
// 1568 / 1449, 3652 / 3557; 2 experts of 1000 tokens, half of whose tiles are too few, 175 / 261; dense of depth 14336 2300 x 4096
// 208 / 349.  Where the two are close the model may miss: 4 experts of 3001 tokens, 14336 x 4096, 552 / 572 and dense 576 x 32000 of
// depth 4096 151 / 140 run with the slower.  Not for more than one result a product: gate and up of 2000 tokens 892 / 937, with
// their inputs kept of 9200 3320 / 3856, SwiGLU backward 1896 / 2704.
struct TPForm { int row_tiles; float step, longest; };
__host__ __device__ __forceinline__ bool tp_joint_pays(const TPForm& one, const TPForm& two, int units, int f_tiles, int pairs, int kbt, bool = false) {
  if (two.row_tiles == one.row_tiles || two.row_tiles == 0) return false;
  const float rows = 32.f * (float)units;
  const float a = tp_clocks_of_all(one.row_tiles, f_tiles, pairs, kbt, one.step / (float)one.row_tiles, one.longest, rows / (float)one.row_tiles, 0.f);
  const float b = tp_clocks_of_all(two.row_tiles, f_tiles, pairs, kbt, two.step / (float)two.row_tiles, two.longest, rows / (float)two.row_tiles, 8.f);
  return b < 0.98f * a;
}
__host__ __device__ __forceinline__ void tp_add_group(TPForm& f, int rows, int cap) {
  const int nt = tp_tiles_of_rows(rows, cap);
  if (nt == 0) return;
  const float most = tp_clocks(tp_tile_rows(rows, cap));
  f.row_tiles += nt;
  f.step += (float)nt * most;
  f.longest = fmaxf(f.longest, most);
}

__device__ __forceinline__ int tp_rows_of(const TPParams& p, int g, int& start, int& end) {
  start = p.mode == 1 ? p.offsets[g] : 0;
  end = p.mode == 1 ? p.offsets[g + 1] : p.M;
  const int rows = end - start;
  return p.group_rows != nullptr && p.group_rows[g] < rows ? p.group_rows[g] : rows;
}
// One thread per group fills the table, after the groups' places in it are counted; a warp scan gives the first tile of each.
template <bool JOINT>
__device__ __forceinline__ void tp_fill_table(const TPParams& p, TPTable* tb, int f_tiles, int kbt, int pairs, int lane) {
  int cap = 8, start, end;
  if (JOINT) {
    TPForm one{0, 0.f, 0.f}, two{0, 0.f, 0.f};
    int units = 0;
    for (int g = lane; g < p.G; g += 32) {
      const int rows = tp_rows_of(p, g, start, end);
      units += (rows + TP_UNIT - 1) / TP_UNIT;
      tp_add_group(one, rows, 8);
      tp_add_group(two, rows, 16);
    }
    auto over_lanes = [&](TPForm& f) {
      f.row_tiles = __reduce_add_sync(0xffffffffu, f.row_tiles);
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) { f.step += __shfl_xor_sync(0xffffffffu, f.step, o); f.longest = fmaxf(f.longest, __shfl_xor_sync(0xffffffffu, f.longest, o)); }
    };
    over_lanes(one); over_lanes(two);
    units = __reduce_add_sync(0xffffffffu, units);
    if (tp_joint_pays(one, two, units, f_tiles, pairs, kbt)) cap = 16;
  }
  for (int g = lane; g < p.G; g += 32) tb->tile0[g] = tp_tile_rows(tp_rows_of(p, g, start, end), cap);
  __syncwarp();
  for (int g = lane; g < p.G; g += 32) {
    const int rows = tp_rows_of(p, g, start, end), mine = tb->tile0[g];
    int place = 0;
    for (int o = 0; o < p.G; ++o) place += tb->tile0[o] > mine || (tb->tile0[o] == mine && o < g) ? 1 : 0;
    tb->group[place] = g; tb->start[place] = start; tb->rows[place] = rows; tb->end[place] = end;
  }
  __syncwarp();
  int carry = 0, widest = 0;
  for (int g0 = 0; g0 < p.G; g0 += 32) {
    const int g = g0 + lane;
    int tiles = 0;
    if (g < p.G) {
      const int rows = tb->rows[g];
      tiles = tp_tiles_of_rows(rows, cap) * f_tiles;
      widest = max(widest, tp_tile_rows(rows, cap));
    }
    int incl = tiles;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) { const int v = __shfl_up_sync(0xffffffffu, incl, o); if (lane >= o) incl += v; }
    if (g < p.G) tb->tile0[g] = carry + incl - tiles;
    carry += __shfl_sync(0xffffffffu, incl, 31);
  }
  widest = __reduce_max_sync(0xffffffffu, widest);
  if (lane == 0) { tb->tile0[p.G] = carry; tb->widest = widest; tb->cap = cap; }
}

__host__ __device__ __forceinline__ void tp_tile(const TPTable* tb, int G, int f_tiles, int f_width, int t, TPTile& o) {
  int g = 0;
  while (g + 1 < G && t >= tb->tile0[g + 1]) ++g;
  const int units = (tb->rows[g] + TP_UNIT - 1) / TP_UNIT, nt = tp_tiles_of_rows(tb->rows[g], tb->cap);
  int n, f;
  panel_order(t - tb->tile0[g], nt, f_tiles, 8, n, f);      // rows fastest: the tiles that share weights run together
  const int base = units / nt, extra = units % nt;
  o.g = tb->group[g];
  o.f0 = f * f_width;
  o.row0 = tb->start[g] + (n * base + (n < extra ? n : extra)) * TP_UNIT;
  o.n = (base + (n < extra ? 1 : 0)) * TP_UNIT;
  o.end = tb->end[g];
  o.zero0 = n == nt - 1 && o.row0 + o.n < o.end ? o.row0 + o.n : o.end;
}

// it = 0, 1, ...: the tile of pair `pair` of `pairs`.  The tiles come by their rows, most first, and every second round goes through
// the pairs backwards, so that all have about the same to do (us, groups in their own order, each round forwards /
// so: SwiGLU backward of 600 tokens 226 / 214, down 1000 tokens 271 / 261, dx 527 / 513).
// (The unnamed flags here and in tp_joint_pays asked for a last round shared along the depth; its sums came in any order.)
__host__ __device__ __forceinline__ bool tp_work(const TPTable* tb, int G, int f_tiles, int f_width, int kbt, bool, int pair, int pairs, int it, TPWork& w) {
  const int i = it * pairs + (it & 1 ? pairs - 1 - pair : pair);
  if (i >= tb->tile0[G]) return false;
  tp_tile(tb, G, f_tiles, f_width, i, w.t);
  w.kb0 = 0; w.kb1 = kbt; w.split = -1; w.contributors = 1;
  return true;
}

__device__ __forceinline__ uint32_t pack_bf16(float lo, float hi) {
  const __nv_bfloat162 v = __floats2bfloat162_rn(lo, hi);
  return *reinterpret_cast<const uint32_t*>(&v);
}
// A warp's stage: rows of 64 bytes (32 features) or, in the gate / up form, of 32 bytes (16 features); the 16-byte pieces are
// swizzled by the row so that eight consecutive rows' pieces fall into different banks.
__device__ __forceinline__ uint32_t tp_slot64(int row, int piece) { return row * 64 + ((piece ^ ((row >> 1) & 3)) << 4); }
__device__ __forceinline__ uint32_t tp_slot32(int row, int piece) { return row * 32 + ((piece ^ ((row >> 2) & 1)) << 4); }

// Rows [first, end) of a warp's features are cleared.
template <int KIND>
__device__ __forceinline__ void tp_clear(const TPParams& p, int first, int end, int col, int half, int lane) {
  constexpr int PIECES = KIND == TP_DUAL ? 2 : 4, STEP = 32 / PIECES;
  const int c = col + (lane % PIECES) * 8;
  if (c >= p.N) return;
  const uint4 z = make_uint4(0u, 0u, 0u, 0u);
  for (int row = first + half * STEP + lane / PIECES; row < end; row += 2 * STEP) {
    const long long at = (long long)row * p.ldc + c;
    *reinterpret_cast<uint4*>(reinterpret_cast<__nv_bfloat16*>(p.C) + at) = z;
    if (KIND != TP_PLAIN && p.C2 != nullptr) *reinterpret_cast<uint4*>(reinterpret_cast<__nv_bfloat16*>(p.C2) + at) = z;
    if (KIND == TP_DUAL && p.C3 != nullptr) *reinterpret_cast<uint4*>(reinterpret_cast<__nv_bfloat16*>(p.C3) + at) = z;
  }
}
// The stage's 32 rows to the rows of `out` from `row0` on.
template <int KIND>
__device__ __forceinline__ void tp_store(const TPParams& p, void* out, const uint8_t* stage, int row0, int end, int col, int lane) {
  constexpr int PIECES = KIND == TP_DUAL ? 2 : 4, STEP = 32 / PIECES;
  const int piece = lane % PIECES, c = col + piece * 8;
#pragma unroll
  for (int i = 0; i < PIECES; ++i) {
    const int r = i * STEP + lane / PIECES;
    const uint4 v = *reinterpret_cast<const uint4*>(stage + (KIND == TP_DUAL ? tp_slot32(r, piece) : tp_slot64(r, piece)));
    if (row0 + r < end && c < p.N) *reinterpret_cast<uint4*>(reinterpret_cast<__nv_bfloat16*>(out) + (long long)(row0 + r) * p.ldc + c) = v;
  }
}
// 32 rows of `src` into registers, as tp_store lays them out
__device__ __forceinline__ void tp_fetch(uint4 (&v)[4], const TPParams& p, const void* src, int row0, int end, int col, int lane) {
  const int c = col + (lane & 3) * 8;
  const uint4* at[4];
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const int row = row0 + i * 8 + (lane >> 2);
    at[i] = reinterpret_cast<const uint4*>(reinterpret_cast<const __nv_bfloat16*>(src) + (row < end && c < p.N ? (long long)row * p.ldc + c : 0));
  }
#pragma unroll
  for (int i = 0; i < 4; ++i) v[i] = __ldcg(at[i]);
}

// One warp's part of a tile: its 32 TMEM lanes (from `acc`), every second chunk of 32 rows from `half` on.  `ready` is called before the
// first read of the accumulator.
template <int KIND, class Ready>
__device__ __forceinline__ bool tp_epilogue(const TPParams& p, uint8_t* stage, const TPTile& t, int col, int half, int lane, float alpha, uint32_t acc, Ready ready) {
  const int chunks = t.n / TP_UNIT;
  const uint32_t st = smem_u32(stage);
  uint4 pg[4], pu[4];
  if constexpr (KIND == TP_SWIGLU_BWD) {
    if (half < chunks) { tp_fetch(pg, p, p.swiglu_g, t.row0 + half * 32, t.end, col, lane); tp_fetch(pu, p, p.swiglu_u, t.row0 + half * 32, t.end, col, lane); }
  }
  if (!ready()) return false;
#pragma unroll 1
  for (int c = half; c < chunks; c += 2) {
    const int row0 = t.row0 + c * 32;
    uint32_t lo[16], hi[16];                      // lanes 0-15 and 16-31 of the warp's quarter
    tmem_ld_16x256b_x4(acc + c * 32, lo);
    tmem_ld_16x256b_x4(acc + c * 32 + (16u << 16), hi);
    tmem_ld_wait();
    if constexpr (KIND == TP_PLAIN) {
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        auto v = [&](const uint32_t (&a)[16], int i) { return __uint_as_float(a[4 * j + i]) * alpha; };
        stmatrix_x4_trans(st + tp_slot64(8 * j + (lane & 7), lane >> 3), pack_bf16(v(lo, 0), v(lo, 1)), pack_bf16(v(lo, 2), v(lo, 3)),
                          pack_bf16(v(hi, 0), v(hi, 1)), pack_bf16(v(hi, 2), v(hi, 3)));
      }
      __syncwarp();
      tp_store<KIND>(p, p.C, stage, row0, t.end, col, lane);
    } else if constexpr (KIND == TP_DUAL) {
      auto put = [&](int mat, auto value) {
#pragma unroll
        for (int j = 0; j < 2; ++j) {
          const int r = 16 * j + (lane >> 4) * 8 + (lane & 7);
          stmatrix_x4_trans(st + mat * 1024 + tp_slot32(r, (lane >> 3) & 1), pack_bf16(value(8 * j), value(8 * j + 1)), pack_bf16(value(8 * j + 2), value(8 * j + 3)),
                            pack_bf16(value(8 * j + 4), value(8 * j + 5)), pack_bf16(value(8 * j + 6), value(8 * j + 7)));
        }
      };
      const bool keep = p.C2 != nullptr;
      if (keep) {
        put(1, [&](int i) { return __uint_as_float(lo[i]); });
        put(2, [&](int i) { return __uint_as_float(hi[i]); });
      }
      put(0, [&](int i) { const float g = __uint_as_float(lo[i]); return g / (1.0f + __expf(-g)) * __uint_as_float(hi[i]); });
      __syncwarp();
      tp_store<KIND>(p, p.C, stage, row0, t.end, col, lane);
      if (keep) {
        tp_store<KIND>(p, p.C2, stage + 1024, row0, t.end, col, lane);
        tp_store<KIND>(p, p.C3, stage + 2048, row0, t.end, col, lane);
      }
    } else {
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const int r = i * 8 + (lane >> 2);
        *reinterpret_cast<uint4*>(stage + tp_slot64(r, lane & 3)) = pg[i];
        *reinterpret_cast<uint4*>(stage + 2048 + tp_slot64(r, lane & 3)) = pu[i];
      }
      __syncwarp();
      if (c + 2 < chunks) { tp_fetch(pg, p, p.swiglu_g, row0 + 64, t.end, col, lane); tp_fetch(pu, p, p.swiglu_u, row0 + 64, t.end, col, lane); }
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        // (each piece of the stage is read here by the lanes of one instruction before the same instruction group writes it)
        const uint32_t at = st + tp_slot64(8 * j + (lane & 7), lane >> 3);
        uint32_t g[4], u[4];
        ldmatrix_x4_trans(at, g[0], g[1], g[2], g[3]);
        ldmatrix_x4_trans(at + 2048, u[0], u[1], u[2], u[3]);
        uint32_t dg[4], du[4];
#pragma unroll
        for (int m = 0; m < 4; ++m) {
          const float2 gf = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&g[m])), uf = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&u[m]));
          const float d0 = __uint_as_float(m < 2 ? lo[4 * j + 2 * m] : hi[4 * j + 2 * (m - 2)]) * alpha;
          const float d1 = __uint_as_float(m < 2 ? lo[4 * j + 2 * m + 1] : hi[4 * j + 2 * (m - 2) + 1]) * alpha;
          const float s0 = 1.f / (1.f + __expf(-gf.x)), s1 = 1.f / (1.f + __expf(-gf.y));
          du[m] = pack_bf16(d0 * (gf.x * s0), d1 * (gf.y * s1));
          dg[m] = pack_bf16(d0 * uf.x * s0 * (1.f + gf.x * (1.f - s0)), d1 * uf.y * s1 * (1.f + gf.y * (1.f - s1)));
        }
        __syncwarp();
        stmatrix_x4_trans(at, dg[0], dg[1], dg[2], dg[3]);
        stmatrix_x4_trans(at + 2048, du[0], du[1], du[2], du[3]);
      }
      __syncwarp();
      tp_store<KIND>(p, p.C, stage, row0, t.end, col, lane);
      tp_store<KIND>(p, p.C2, stage + 2048, row0, t.end, col, lane);
    }
    __syncwarp();       // the stage is free again
  }
  return true;
}

template <int KIND>
__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(GEMM_THREADS, 1) gemm_sm100_tpair_kernel(const __grid_constant__ TPParams p) {
  constexpr int F_WIDTH = KIND == TP_DUAL ? 128 : 256;      // output features of a tile
  constexpr bool JOINT = KIND == TP_PLAIN;                  // tiles of two accumulators at all (tp_joint_pays)
  constexpr uint32_t TMEM_COLS = 512;

  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  uint64_t* full_bar = reinterpret_cast<uint64_t*>(smem + TP_RING_BYTES);
  uint64_t* empty_bar = full_bar + TP_MAX_STAGES;
  uint64_t* tfull_bar = empty_bar + TP_MAX_STAGES;
  uint64_t* tempty_bar = tfull_bar + 2;
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(tempty_bar + 2);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);
  uint8_t* epi_stage = smem + TP_RING_BYTES + 256;
  TPTable* tb = reinterpret_cast<TPTable*>(epi_stage + EPI_WARPS * EPI_STAGE_BYTES);

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int rank = (int)cluster_ctarank();          // 0 = leader
  const int pair_id = (int)cluster_id_x(), num_pairs = (int)num_clusters_x();
  const int f_tiles = (p.N + F_WIDTH - 1) / F_WIDTH;
  const int num_kb = (p.K + BK - 1) / BK, kbt = num_kb + (p.K_l + BK - 1) / BK;

  if (threadIdx.x == 0) {
    for (int s = 0; s < TP_MAX_STAGES; ++s) { mbar_init(&full_bar[s], 1); mbar_init(&empty_bar[s], 1); }
    for (int b = 0; b < 2; ++b) { mbar_init(&tfull_bar[b], 1); mbar_init(&tempty_bar[b], 2 * EPI_WARPS); }
    *abort_flag = 0;
    fence_barrier_init();
  }
  if (warp == 1) { tmem_alloc_pair(tmem_slot, TMEM_COLS); tmem_relinquish_pair(); }
  if (warp == 2) { wait_for_predecessor(); tp_fill_table<JOINT>(p, tb, f_tiles, kbt, num_pairs, lane); }
  tc_fence_before();
  cluster_sync_all();
  tc_fence_after();
  const uint32_t tmem_base = *tmem_slot;
  after_predecessor();
  const int stage_bytes = TP_A_BYTES + tb->widest * (BK * 2 / 2);
  const int stages = min(TP_RING_BYTES / stage_bytes, TP_MAX_STAGES);

  auto fail = [&](int code) {
    *abort_flag = 1;
    if (p.status != nullptr) atomicCAS(p.status, 0, code);
  };
  TPWork w;
  auto next = [&](int it) { return tp_work(tb, p.G, f_tiles, F_WIDTH, kbt, false, pair_id, num_pairs, it, w); };

  if (warp == 0) {
    // ------------------------------------------------------------------ TMA producer (one per CTA)
    if (elect_one()) { prefetch_tensormap(&p.tmW); prefetch_tensormap(&p.tmX[3]); }
    int s = 0;
    uint32_t ph = 0;
    bool ok = true;
    for (int wi = 0; ok && next(wi); ++wi) {
      const TPTile& t = w.t;
      const int f0 = t.f0 + rank * (F_WIDTH / 2);
      const uint32_t bytes = 2 * (TP_A_BYTES + t.n / 2 * (BK * 2));
      // (a loop for each of one and two accumulators, here and in the issuer: with the choice inside, tiles of 256 rows took 25 % longer)
      auto load = [&](auto two) {
        const int n0 = decltype(two)::value ? tp_first(t.n) : t.n;
        for (int kb = 0; kb < kbt; ++kb) {
          if (!wait_parity_warp(&empty_bar[s], ph ^ 1, abort_flag)) { fail(ST_TIMEOUT_EMPTY); ok = false; break; }
          uint8_t* sW = smem + s * stage_bytes;
          uint8_t* sX = sW + TP_A_BYTES;
          // (only the leader arrives, see the pair kernel)
          const uint32_t bar = mapa_shared(smem_u32(&full_bar[s]), 0);
          const bool second = kb >= num_kb;
          const int kk = (second ? kb - num_kb : kb) * BK;
          const CUtensorMap* mW = second ? &p.tmW_l : &p.tmW;
          const CUtensorMap* mW2 = second ? &p.tmW2_l : &p.tmW2;
          const int w_mn = second ? p.w_mn_l : p.w_mn;
          if (elect_one()) {
            if (rank == 0) mbar_expect_tx(&full_bar[s], bytes);
            if (KIND == TP_DUAL) {
#pragma unroll
              for (int j = 0; j < 4; ++j) {
                tma_load_3d_pair(sW + j * 4096, mW, bar, kk, f0 + 16 * j, t.g);
                tma_load_3d_pair(sW + j * 4096 + 2048, mW2, bar, kk, f0 + 16 * j, t.g);
              }
            } else if (w_mn == 0) {
              tma_load_3d_pair(sW, mW, bar, kk, f0, t.g);
            } else {
              tma_load_3d_pair(sW, mW, bar, f0, kk, t.g);
              tma_load_3d_pair(sW + 8192, mW, bar, f0 + 64, kk, t.g);
            }
            const CUtensorMap* mX = second ? p.tmX_l : p.tmX;
            auto rows = [&](uint8_t* to, int n, int first) {      // this CTA's half of n rows
              int done = 0;
#pragma unroll
              for (int b = 3; b >= 0; --b)
                if ((n / 2) & (16 << b)) { tma_load_2d_pair(to + done * (BK * 2), mX + b, bar, kk, first + rank * (n / 2) + done); done += 16 << b; }
            };
            rows(sX, n0, t.row0);
            if (decltype(two)::value) rows(sX + n0 / 2 * (BK * 2), t.n - n0, t.row0 + n0);
          }
          if (++s == stages) { s = 0; ph ^= 1; }
        }
      };
      if (!JOINT || t.n <= 256) load(std::false_type());
      else load(std::integral_constant<bool, JOINT>());
    }
    if (!ok) {  // give this CTA's copies already in flight a bounded time to land before it leaves
      const uint64_t t0 = global_timer_ns();
      while (global_timer_ns() - t0 < 2000000ull) {}
    }
  } else if (warp == 1 && rank == 0) {
    // ------------------------------------------------------------------ MMA issuer (leader only)
    int s = 0;
    uint32_t ph = 0, acc_it = 0;
    bool ok = true;
    for (int wi = 0; ok && next(wi); ++wi) {
      auto multiply = [&](auto two) {
        const int n0 = decltype(two)::value ? tp_first(w.t.n) : w.t.n, n1 = w.t.n - n0, buf = acc_it & 1;
        if (!wait_parity_warp(&tempty_bar[buf], ((acc_it >> 1) & 1) ^ 1, abort_flag)) { fail(ST_TIMEOUT_TMEM_EMPTY); ok = false; return; }
        if (decltype(two)::value && !wait_parity_warp(&tempty_bar[buf ^ 1], (((acc_it + 1) >> 1) & 1) ^ 1, abort_flag)) { fail(ST_TIMEOUT_TMEM_EMPTY); ok = false; return; }
        tc_fence_after();
        const uint32_t d_tmem = tmem_base + buf * 256, d_tmem1 = tmem_base + (buf ^ 1) * 256;
        for (int kb = 0; kb < kbt; ++kb) {
          if (!wait_parity_warp(&full_bar[s], ph, abort_flag)) { fail(ST_TIMEOUT_FULL); ok = false; return; }
          tc_fence_after();
          const int w_mn = kb >= num_kb ? p.w_mn_l : p.w_mn;
          const uint32_t idesc = make_idesc_bf16(2 * BM, n0, w_mn, 0);
          const uint32_t sW = smem_u32(smem + s * stage_bytes);
          const uint64_t dw = operand_desc(sW, w_mn), dx = operand_desc(sW + TP_A_BYTES, 0);
          const uint32_t kw = operand_kstep(w_mn), kx = operand_kstep(0);
          if (elect_one()) {
#pragma unroll
            for (int k = 0; k < BK / 16; ++k)
              umma_bf16_pair(d_tmem, dw + k * kw, dx + k * kx, idesc, (kb > 0 || k > 0) ? 1u : 0u);
            if (decltype(two)::value) {
              const uint32_t idesc1 = make_idesc_bf16(2 * BM, n1, w_mn, 0);
              const uint64_t dx1 = operand_desc(sW + TP_A_BYTES + n0 / 2 * (BK * 2), 0);
#pragma unroll
              for (int k = 0; k < BK / 16; ++k)
                umma_bf16_pair(d_tmem1, dw + k * kw, dx1 + k * kx, idesc1, (kb > 0 || k > 0) ? 1u : 0u);
            }
            umma_commit_pair(&empty_bar[s], 3);   // frees the stage in both CTAs
          }
          if (++s == stages) { s = 0; ph ^= 1; }
        }
        if (elect_one()) {                          // accumulators complete, in both CTAs
          umma_commit_pair(&tfull_bar[buf], 3);
          if (decltype(two)::value) umma_commit_pair(&tfull_bar[buf ^ 1], 3);
        }
        acc_it += decltype(two)::value ? 2 : 1;
      };
      if (!JOINT || w.t.n <= 256) multiply(std::false_type());
      else multiply(std::integral_constant<bool, JOINT>());
    }
  } else if (warp >= 2) {
    // ------------------------------------------------------------------ epilogue (both CTAs, own 128 operand rows)
    const int q = warp & 3, half = (warp - 2) >> 2;
    uint8_t* stage = epi_stage + (warp - 2) * EPI_STAGE_BYTES;
    const float alpha = p.alpha_dev != nullptr ? p.alpha * *p.alpha_dev : p.alpha;
    uint32_t acc_it = 0;
    bool ok = true;
    for (int wi = 0, sub = 0; ok && (sub > 0 || next(wi)); sub > 0 ? 0 : ++wi) {
      // (a tile of more than 256 rows: its two accumulators one after the other)
      TPTile t = w.t;
      const int mine = sub;
      if (JOINT) {
        const int n0 = tp_first(t.n);
        sub = mine == 0 && t.n > n0 ? 1 : 0;
        t.row0 += mine * n0;
        t.n = mine == 0 ? n0 : t.n - n0;
      }
      const int col = t.f0 + rank * (F_WIDTH / 2) + q * (F_WIDTH / 8);        // this warp's first output feature
      const int buf = acc_it & 1;
      const uint32_t aph = (acc_it >> 1) & 1;
      const uint32_t tacc = tmem_base + buf * 256 + ((uint32_t)(q * 32) << 16);
      if (mine == 0) tp_clear<KIND>(p, t.zero0, t.end, col, half, lane);     // under the wait for the accumulator
      auto ready = [&]() {
        if (!wait_parity_warp(&tfull_bar[buf], aph, abort_flag)) { fail(ST_TIMEOUT_TMEM_FULL); return false; }
        tc_fence_after();
        return true;
      };
      ok = tp_epilogue<KIND>(p, stage, t, col, half, lane, alpha, tacc, ready);
      if (!ok) break;
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive_cluster(mapa_shared(smem_u32(&tempty_bar[buf]), 0));
      ++acc_it;
    }
  }

  // Neither CTA may leave while its partner can still read its shared memory or arrive on its barriers.
  __syncwarp();
  tc_fence_before();
  cluster_sync_all();
  if (warp == 1) { tc_fence_after(); tmem_dealloc_pair(tmem_base, TMEM_COLS); }
}
