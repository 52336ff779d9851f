// Persistent warp-specialised bf16 GEMM family for sm_100a.
//
//   TMA (cp.async.bulk.tensor, 128-byte swizzle) -> shared memory ring -> tcgen05.mma (one issuing
//   thread, fp32 accumulators in TMEM, two accumulator buffers) -> tcgen05.ld epilogue.
//
// One kernel covers every matrix product of the training step:
//   mode 0  dense          C[M,N]        = A[M,K] * B[K,N]
//   mode 1  grouped rows   C[rows of g]  = A[rows of g] * B_g      (expert forward / dgrad; row groups
//                                                                   start on 128-row boundaries)
//   mode 2  grouped depth  C_g[M,N]      = sum over rows of g  A[row,:]^T B[row,:]   (weight gradients)
// Operands may be K-major or MN-major (the tensor core transposes from shared memory), so the same
// kernel serves x*W^T, dy*W and dy^T*x without materialising a transpose.
// Options: a second, short depth segment (LoRA: += (s*X*A) * B with its own tensor maps), a dual-B
// mode that computes gate and up projections in one 256-wide MMA and applies SwiGLU in the
// epilogue, alpha scaling and accumulation into C (gradient accumulation), fp32 or bf16 C.
//
// Role layout of a 320-thread CTA: warp 0 = TMA producer, warp 1 = MMA issuer (owns TMEM), warps 2-9 = epilogue
// (a warp reads the 32-lane quarter warp % 4 of TMEM; two warps share a quarter, half of the columns each).
#include <cuda.h>
#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <stdint.h>
#include <math.h>
#include <stdio.h>
#include <stdlib.h>

#include <map>
#include <unordered_map>
#include <string.h>
#include <mutex>
#include <type_traits>
#include <tuple>

#include "api.h"
#include "comm.h"
#include "common/host.h"
#include "common/ptx.cuh"

namespace mdt {

constexpr int BM = 128;
constexpr int BK = 64;
constexpr int A_BYTES = BM * BK * 2;
constexpr int GEMM_THREADS = 320;
constexpr int SPLIT_COUNTERS = 12;   // of a shared tile: 8 parts (row quarter x column half), 4 row quarters

struct GemmParams {
  CUtensorMap tmA, tmB, tmB2;        // main depth segment (tmB2: second B matrix of the dual mode)
  CUtensorMap tmA_l, tmB_l, tmB2_l;  // optional LoRA depth segment
  int M, N, K, K_l, G, mode;
  int a_mn, b_mn, a_mn_l, b_mn_l, dual;
  const int* offsets;
  void* C; void* C2; void* C3; const void* R;
  const void* swiglu_g; const void* swiglu_u;
  long long ldc, c_group_stride;
  int c_fp32, accumulate;
  float alpha;
  const float* alpha_dev;
  int store_gate_up;
  int* status;
  const unsigned* tile_ready; const int* tile_expected;
  const int* row_dest_rank; const int* row_dest_row; const long long* peer_out; const long long* peer_arrive; int num_peers;
  unsigned long long peer_wait_ns;   // limit of the waits for operands that other GPUs or streams deliver
  // B (and B2) may be part of a buffer that an all-gather is still filling: see MdtGemmDesc::b_ready
  MdtOperandReady rdy_b, rdy_b2, rdy_bl;
  long long b_rows, ldb, b_group_stride, bl_rows, ldb_l, bl_group_stride;
  // split of the last, partly filled wave of tiles along the depth (128-row kernel; see get_work)
  float* sk_ws; unsigned* sk_ctr;
};

// Bounded wait until the chunks of the gathered buffer that hold bytes [off, off + len) of an operand have landed.
__device__ __forceinline__ bool wait_operand_ready(const MdtOperandReady& r, long long off, long long len, unsigned long long limit_ns) {
  if (r.ready == nullptr || len <= 0) return true;
  const long long o0 = r.offset_bytes + off, o1 = o0 + len - 1;
  const int c0 = (int)(o0 / r.shard_bytes) * r.chunks_per_rank + (int)((o0 % r.shard_bytes) / r.chunk_bytes);
  const int c1 = (int)(o1 / r.shard_bytes) * r.chunks_per_rank + (int)((o1 % r.shard_bytes) / r.chunk_bytes);
  for (int c = c0; c <= c1; ++c)
    if (!wait_ge(r.ready + c, r.epoch, limit_ns)) return false;
  return true;
}
// The part of B that the tile (group g, columns from n0, `rows` output columns) reads: whole rows of a K-major B,
// the whole matrix of the group for an MN-major one.
__device__ __forceinline__ bool wait_b_tile(const GemmParams& p, int g, int n0, int rows) {
  if (p.rdy_bl.ready != nullptr && p.K_l > 0 &&
      !wait_operand_ready(p.rdy_bl, (long long)g * p.bl_group_stride * 2, p.bl_rows * p.ldb_l * 2, p.peer_wait_ns)) return false;   // whole matrix
  if (p.rdy_b.ready == nullptr && p.rdy_b2.ready == nullptr) return true;
  long long off, len;
  if (p.b_mn == 0) {
    const long long r = (long long)rows < p.b_rows - n0 ? rows : p.b_rows - n0;
    off = ((long long)g * p.b_group_stride + (long long)n0 * p.ldb) * 2;
    len = r * p.ldb * 2;
  } else {
    off = (long long)g * p.b_group_stride * 2;
    len = p.b_rows * p.ldb * 2;
  }
  return wait_operand_ready(p.rdy_b, off, len, p.peer_wait_ns) && wait_operand_ready(p.rdy_b2, off, len, p.peer_wait_ns);
}
// A GEMM that takes part in an exchange does nothing when the status word is already set (an earlier wait of the
// exchange ran out: its metadata describe no rows and nothing may be stored into a peer on the strength of them).
__device__ __forceinline__ bool gemm_dead(const GemmParams& p) {
  return p.status != nullptr && (p.tile_ready != nullptr || p.row_dest_rank != nullptr) && *reinterpret_cast<const volatile int*>(p.status) != 0;
}

// Set-up is done: from here on the kernel touches what others touch.  One that waits for peers or for a gather on another stream
// keeps its successors out until it ends, so that their CTAs never take the place of those it waits for.
__device__ __forceinline__ void gemm_begin(const GemmParams& p) {
  wait_for_predecessor();
  if (p.tile_ready == nullptr && p.row_dest_rank == nullptr && p.rdy_b.ready == nullptr && p.rdy_b2.ready == nullptr && p.rdy_bl.ready == nullptr) admit_successor();
}

// Order of the output tiles.  A persistent grid works on a window of consecutive tiles at a time; what that window
// reads should stay in L2.  Tiles therefore go through panels of at most 2048 rows (16 blocks of 128 or 8 of 256),
// m fastest inside a panel, then n: 148 CTAs then share about 2048 rows of A and 9 column blocks of B.  With m fastest
// over all rows, a window of the expert products (18 400 rows x K 14336) streamed the whole 530 MB of A once per column
// block, 1.0-1.2 PFLOP/s instead of the 1.4 that the same kernel reaches when the window fits.  Row groups are
// enumerated one after the other for the same reason: a window then holds one expert's weights.
constexpr int PANEL_ROWS = 2048;
__host__ __device__ __forceinline__ void panel_order(int r, int m_blocks, int n_blocks, int panel, int& m, int& n) {
  const int first = r / (panel * n_blocks) * panel;
  const int width = m_blocks - first < panel ? m_blocks - first : panel;
  const int q = r - first * n_blocks;
  m = first + q % width;
  n = q / width;
}

struct Tile {
  int g, m0, n0, krow0, num_kb, num_kb_l, second_ok;
};
typedef Tile PairTile;

// Maps a linear tile index to its coordinates, for tiles of ROWS rows (128, or 256 for the CTA pair); returns false past
// the last tile.  In the grouped-rows mode a 256-row tile never straddles two groups: a group with an odd number of
// 128-row blocks ends with a tile whose second half is idle (second_ok = 0).  (Also callable on the host, where a unit
// test enumerates the tiles of random problems and checks that they cover every block exactly once.)
template <int BN_OUT, int ROWS>
__host__ __device__ __forceinline__ bool locate_tile(const GemmParams& p, int t, Tile& o) {
  const int n_blocks = (p.N + BN_OUT - 1) / BN_OUT;
  int m, n;
  o.num_kb_l = (p.K_l + BK - 1) / BK;
  o.second_ok = 1;
  o.krow0 = 0;
  o.num_kb = (p.K + BK - 1) / BK;
  if (p.mode == 1) {
    for (int g = 0; g < p.G; ++g) {
      const int begin = p.offsets[g], end = p.offsets[g + 1];
      const int m_blocks = (end - begin + ROWS - 1) / ROWS;
      if (t < m_blocks * n_blocks) {
        panel_order(t, m_blocks, n_blocks, PANEL_ROWS / ROWS, m, n);
        o.g = g;
        o.m0 = begin + m * ROWS;
        o.n0 = n * BN_OUT;
        if (ROWS > BM) o.second_ok = (o.m0 + BM < end) ? 1 : 0;
        return true;
      }
      t -= m_blocks * n_blocks;
    }
    return false;
  }
  const int m_blocks = (p.M + ROWS - 1) / ROWS;
  const int per_group = m_blocks * n_blocks;
  o.g = 0;
  if (p.mode == 2) {
    if (t >= per_group * p.G) return false;
    o.g = t / per_group;
    t -= o.g * per_group;
    if (p.offsets != nullptr) {
      o.krow0 = p.offsets[o.g];
      o.num_kb = (p.offsets[o.g + 1] - o.krow0 + BK - 1) / BK;
    }
  } else if (t >= per_group) {
    return false;
  }
  panel_order(t, m_blocks, n_blocks, PANEL_ROWS / ROWS, m, n);
  o.m0 = m * ROWS;
  o.n0 = n * BN_OUT;
  return true;
}
template <int BN_OUT>
__host__ __device__ __forceinline__ bool get_tile(const GemmParams& p, int t, Tile& o) { return locate_tile<BN_OUT, BM>(p, t, o); }
template <int BN_OUT>
__host__ __device__ __forceinline__ bool get_pair_tile(const GemmParams& p, int t, PairTile& o) { return locate_tile<BN_OUT, 2 * BM>(p, t, o); }

// One unit of work of a CTA: a whole output tile, or a piece [kb0, kb1) of the depth of a tile that several CTAs share.
struct Work {
  Tile t;
  int kb0, kb1;        // k blocks of the tile this CTA computes (main segment first, then the LoRA segment)
  int split;           // -1: whole tile.  Otherwise the index of the shared tile (its slot in the fp32 workspace)
  int contributors;    // CTAs that share the tile
};

// Tiles are dealt to the CTAs round robin; when the last round would leave most SMs idle (fewer than 7/8 of them
// get a tile), the tiles of that round are not handed out whole: their k blocks, taken together, are cut into one
// contiguous piece per CTA (a piece spans at most two tiles).  Every CTA adds its piece's partial sums into an fp32
// workspace tile and counts itself in, per 32-row quarter and column half of the tile, i.e. per epilogue warp; the warp that
// arrives last at such a part reads the sums back and runs the normal epilogue for it.  Nobody waits for anybody.  With 160
// tiles of depth 224 on 148 SMs that is 1 round + 18 k blocks per CTA instead of 2 rounds (0.136 instead of 0.192 ms).
// Products of less than one round are left alone.
// it = 0, 1, ... enumerates the CTA's work in order; returns false when there is no more.
template <int BN_OUT>
__host__ __device__ __forceinline__ bool get_work(const GemmParams& p, int cta, int num_ctas, int it, Work& w) {
  const int n_blocks = (p.N + BN_OUT - 1) / BN_OUT;
  int total_tiles;
  if (p.mode == 2) {
    total_tiles = ((p.M + BM - 1) / BM) * n_blocks * p.G;
  } else {
    const int rows = (p.mode == 1) ? p.offsets[p.G] : p.M;
    total_tiles = ((rows + BM - 1) / BM) * n_blocks;
  }
  const int kbt = (p.K + BK - 1) / BK + (p.K_l + BK - 1) / BK;        // k blocks per tile (modes 0 and 1)
  int whole = total_tiles;
  if (p.sk_ws != nullptr && p.mode != 2 && !p.dual && kbt >= 8) {
    const int rem = total_tiles % num_ctas;
    // (pieces shorter than 8 k blocks are not worth their partial-sum traffic, and a product of less than one full round
    // stays as it is: 80 tiles of depth 64 cut into 148 pieces lose more to the partial sums than they gain)
    if (rem != 0 && total_tiles > num_ctas && rem * 8 < num_ctas * 7 && (long long)rem * kbt >= 8ll * num_ctas) whole = total_tiles - rem;
  }
  const int n_whole = whole > cta ? (whole - cta + num_ctas - 1) / num_ctas : 0;
  w.split = -1; w.contributors = 1;
  if (it < n_whole) {
    if (!get_tile<BN_OUT>(p, cta + it * num_ctas, w.t)) return false;
    w.kb0 = 0;
    w.kb1 = w.t.num_kb + (w.t.num_kb > 0 || p.mode != 2 ? w.t.num_kb_l : 0);
    return true;
  }
  const int rem = total_tiles - whole;
  if (rem == 0) return false;
  const long long units = (long long)rem * kbt;
  const long long per = (units + num_ctas - 1) / num_ctas;
  const long long u0 = (long long)cta * per, u1 = (u0 + per < units) ? u0 + per : units;
  if (u0 >= u1) return false;
  const int t_first = (int)(u0 / kbt), t_last = (int)((u1 - 1) / kbt);
  const int tt = t_first + (it - n_whole);
  if (tt > t_last) return false;
  if (!get_tile<BN_OUT>(p, whole + tt, w.t)) return false;
  const long long lo = (long long)tt * kbt, hi = lo + kbt;
  w.kb0 = (int)((u0 > lo ? u0 : lo) - lo);
  w.kb1 = (int)((u1 < hi ? u1 : hi) - lo);
  w.contributors = (int)((hi - 1) / per) - (int)(lo / per) + 1;
  w.split = w.contributors > 1 ? tt : -1;
  return true;
}

__device__ __forceinline__ void store8(void* C, long long idx, const float (&v0)[8], int c_fp32, int accumulate, const void* R = nullptr) {
  float v[8];
#pragma unroll
  for (int i = 0; i < 8; ++i) v[i] = v0[i];
  if (R != nullptr) {   // residual connection: a bf16 matrix laid out like C
    const uint4 rv = *reinterpret_cast<const uint4*>(reinterpret_cast<const __nv_bfloat16*>(R) + idx);
    const __nv_bfloat162* r2 = reinterpret_cast<const __nv_bfloat162*>(&rv);
#pragma unroll
    for (int i = 0; i < 4; ++i) { float2 f = __bfloat1622float2(r2[i]); v[2 * i] += f.x; v[2 * i + 1] += f.y; }
  }
  if (c_fp32) {
    float4* dst = reinterpret_cast<float4*>(reinterpret_cast<float*>(C) + idx);
    float4 a = make_float4(v[0], v[1], v[2], v[3]), b = make_float4(v[4], v[5], v[6], v[7]);
    if (accumulate) {
      float4 oa = dst[0], ob = dst[1];
      a.x += oa.x; a.y += oa.y; a.z += oa.z; a.w += oa.w;
      b.x += ob.x; b.y += ob.y; b.z += ob.z; b.w += ob.w;
    }
    dst[0] = a; dst[1] = b;
  } else {
    uint4* dst = reinterpret_cast<uint4*>(reinterpret_cast<__nv_bfloat16*>(C) + idx);
    float w[8];
#pragma unroll
    for (int i = 0; i < 8; ++i) w[i] = v[i];
    if (accumulate) {
      uint4 old = *dst;
      const __nv_bfloat162* o2 = reinterpret_cast<const __nv_bfloat162*>(&old);
#pragma unroll
      for (int i = 0; i < 4; ++i) { float2 f = __bfloat1622float2(o2[i]); w[2 * i] += f.x; w[2 * i + 1] += f.y; }
    }
    uint4 out;
    __nv_bfloat162* q = reinterpret_cast<__nv_bfloat162*>(&out);
#pragma unroll
    for (int i = 0; i < 4; ++i) q[i] = __floats2bfloat162_rn(w[2 * i], w[2 * i + 1]);
    *dst = out;
  }
}

// ---- epilogue: eight warps, warp -> (32-row quarter of the tile = its TMEM lanes, half of the tile's columns) ----------
// bf16 results leave through a 4 KB stage per warp, 32 rows x 64 columns: a lane holds one row of the accumulator, so
// storing from registers would write 16 bytes to each of 32 rows per instruction.  From the stage a warp writes whole
// 128-byte lines, four rows per instruction.  What is added to the result (C itself when accumulating, or the residual)
// comes in the same way, the first chunk fetched before the warp waits for the accumulator and the next one while the
// first is processed, so that the latency passes under other work.  Weight gradients of one micro-batch
// (3 k blocks per 128 x 256 tile of an 8 x 14336 x 4096 matrix, read and written) are bound by exactly this traffic:
// 1400 us with per-row accesses by four warps.
// 16-byte slots are XOR-swizzled by the row, so that row-wise and line-wise accesses are both free of bank conflicts.
constexpr int EPI_WARPS = 8;
constexpr int EPI_STAGE_BYTES = 32 * 128;
__device__ __forceinline__ uint4* epi_slot(uint8_t* stage, int row, int slot) {
  return reinterpret_cast<uint4*>(stage + row * 128 + ((slot ^ (row & 7)) << 4));
}
// the 64-column chunk at `col` of the matrix whose rows start at `mine` (one per lane), line-wise: 8 x 16 bytes per lane
// (`safe`: an address that may be read instead of one that is out of range, so that the loads need no branches)
__device__ __forceinline__ void epi_fetch(uint4 (&v)[8], unsigned long long mine, unsigned row_ok, int lane, int col, int N, const void* safe) {
  const int c = col + (lane & 7) * 8;
  const uint4* src[8];
#pragma unroll
  for (int i = 0; i < 8; ++i) {
    const int row = i * 4 + (lane >> 3);
    const unsigned long long ptr = __shfl_sync(0xffffffffu, mine, row);
    src[i] = ((row_ok >> row) & 1u) && c < N ? reinterpret_cast<const uint4*>(reinterpret_cast<const __nv_bfloat16*>(ptr) + c)
                                             : reinterpret_cast<const uint4*>(safe);
  }
#pragma unroll
  for (int i = 0; i < 8; ++i)
    asm volatile("ld.global.cg.v4.u32 {%0, %1, %2, %3}, [%4];" : "=r"(v[i].x), "=r"(v[i].y), "=r"(v[i].z), "=r"(v[i].w) : "l"(src[i]));
}
__device__ __forceinline__ void epi_stage_in(uint8_t* stage, const uint4 (&v)[8], int lane) {
#pragma unroll
  for (int i = 0; i < 8; ++i) *epi_slot(stage, i * 4 + (lane >> 3), lane & 7) = v[i];
  __syncwarp();
}
// this lane's row, columns [32 * part, 32 * part + 32) of the chunk; ADD: plus what the stage holds there
template <bool ADD>
__device__ __forceinline__ void epi_stage_row(uint8_t* stage, const float (&v)[32], int part, int lane) {
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    uint4* slot = epi_slot(stage, lane, part * 4 + j);
    float f[8];
#pragma unroll
    for (int i = 0; i < 8; ++i) f[i] = v[j * 8 + i];
    if (ADD) {
      const uint4 old = *slot;
      const __nv_bfloat162* o2 = reinterpret_cast<const __nv_bfloat162*>(&old);
#pragma unroll
      for (int i = 0; i < 4; ++i) { const float2 t = __bfloat1622float2(o2[i]); f[2 * i] += t.x; f[2 * i + 1] += t.y; }
    }
    uint4 out;
    __nv_bfloat162* q = reinterpret_cast<__nv_bfloat162*>(&out);
#pragma unroll
    for (int i = 0; i < 4; ++i) q[i] = __floats2bfloat162_rn(f[2 * i], f[2 * i + 1]);
    *slot = out;
  }
}
__device__ __forceinline__ void epi_flush(uint8_t* stage, unsigned long long mine, unsigned row_ok, int lane, int col, int N) {
  __syncwarp();
  const int c = col + (lane & 7) * 8;
#pragma unroll
  for (int i = 0; i < 8; ++i) {
    const int row = i * 4 + (lane >> 3);
    const unsigned long long ptr = __shfl_sync(0xffffffffu, mine, row);
    const uint4 val = *epi_slot(stage, row, lane & 7);
    if (((row_ok >> row) & 1u) && c < N) *reinterpret_cast<uint4*>(reinterpret_cast<__nv_bfloat16*>(ptr) + c) = val;
  }
  __syncwarp();
}
// The row of C (or of a peer's buffer) that a lane of an epilogue warp owns.
struct EpiRow { void* C; long long base; bool ok; int dest; };
__device__ __forceinline__ EpiRow epi_row(const GemmParams& p, int g, int row, bool row_ok) {
  EpiRow r;
  r.base = (p.mode == 2 ? (long long)g * p.c_group_stride : 0) + (long long)row * p.ldc;
  r.C = p.C;
  r.dest = -1;
  r.ok = row_ok;
  if (p.row_dest_rank != nullptr) {          // result rows go straight into peers' buffers
    r.dest = row_ok ? p.row_dest_rank[row] : -1;
    const int drow = row_ok ? p.row_dest_row[row] : -1;
    if (r.dest >= p.num_peers || drow < 0) r.dest = -1;
    r.ok = r.dest >= 0;
    if (r.ok) { r.C = reinterpret_cast<void*>(p.peer_out[r.dest]); r.base = (long long)drow * p.ldc; }
  }
  return r;
}
__device__ __forceinline__ float gemm_alpha(const GemmParams& p) { return p.alpha_dev != nullptr ? p.alpha * *p.alpha_dev : p.alpha; }
// publish a warp's delivered rows: one count per (row, column tile) and destination
__device__ __forceinline__ void epi_publish(const GemmParams& p, int dest, int lane) {
  __threadfence_system();
  __syncwarp();
  for (int d = 0; d < p.num_peers; ++d) {
    const unsigned m = __ballot_sync(0xffffffffu, dest == d);
    if (lane == 0 && m != 0) red_add_release_sys(reinterpret_cast<unsigned*>(p.peer_arrive[d]), __popc(m));
  }
}
// a tile without any depth (an empty group of a weight gradient): zeros unless accumulating
template <int COLS>
__device__ __forceinline__ void epi_zero(const GemmParams& p, const EpiRow& r, bool row_ok, int col0) {
  if (p.accumulate || !row_ok) return;
  const float z[8] = {0, 0, 0, 0, 0, 0, 0, 0};
  for (int c = 0; c < COLS; c += 8)
    if (col0 + c < p.N) store8(p.C, r.base + col0 + c, z, p.c_fp32, 0);
}

// One warp's part of a tile: COLS = BN / 2 accumulator columns from TMEM column `taddr` on (dual: COLS / 2 outputs, the
// up accumulators being 2 * COLS / 2 = BN / 2 columns further).  `wait` is called once, before the first TMEM load.
// SWIGLU: the form for p.swiglu_g, in kernels of its own: beside the other forms its registers make them spill (weight
// gradients of one micro-batch, accumulated, lost 15 %).
template <int BN, bool SWIGLU, class Wait>
__device__ __forceinline__ bool epi_tile(const GemmParams& p, uint8_t* stage, uint32_t tacc, int half, int lane, int n0, const EpiRow& r, Wait wait) {
  const bool fast = !p.c_fp32 && !(p.accumulate && p.R != nullptr);
  const unsigned row_ok = __ballot_sync(0xffffffffu, r.ok);
  const unsigned long long mine = reinterpret_cast<unsigned long long>(reinterpret_cast<__nv_bfloat16*>(r.C) + r.base);
  if (!SWIGLU && p.dual) {
    constexpr int OUT = BN / 4;                   // output columns of this warp
    if (!wait()) return false;
    const int n_mats = p.store_gate_up ? 3 : 1;
#pragma unroll 1
    for (int c = 0; c < OUT; c += 64) {
      const int col = n0 + half * OUT + c;
      if (col >= p.N) break;
#pragma unroll 1
      for (int mat = 0; mat < n_mats; ++mat) {    // h, gate, up
#pragma unroll 1
        for (int part = 0; part < (OUT < 64 ? 1 : 2); ++part) {
          const uint32_t ta = tacc + half * OUT + c + part * 32;
          uint32_t r0[32], r1[32];                // gate and up; or only the one that is stored
          float v[32];
          tmem_ld_32x32(mat == 2 ? ta + BN / 2 : ta, r0);
          if (mat == 0) {
            tmem_ld_32x32(ta + BN / 2, r1);
            tmem_ld_wait();
#pragma unroll
            for (int i = 0; i < 32; ++i) {
              const float g = __uint_as_float(r0[i]);
              v[i] = g / (1.0f + __expf(-g)) * __uint_as_float(r1[i]);
            }
          } else {
            tmem_ld_wait();
#pragma unroll
            for (int i = 0; i < 32; ++i) v[i] = __uint_as_float(r0[i]);
          }
          epi_stage_row<false>(stage, v, part, lane);
        }
        const void* out = mat == 0 ? p.C : (mat == 1 ? p.C2 : p.C3);
        epi_flush(stage, reinterpret_cast<unsigned long long>(reinterpret_cast<const __nv_bfloat16*>(out) + r.base), row_ok, lane, col, min(p.N, n0 + (half + 1) * OUT));
      }
    }
    return true;
  }
  constexpr int CHUNKS = BN / 128;                // 64-column chunks of this warp
  const int col0 = n0 + half * (BN / 2);
  const float alpha = gemm_alpha(p);
  if constexpr (SWIGLU) {
    // dh in the accumulator -> dg, du.  As a kernel of its own this read dh, g and u and wrote both for 12 000 tokens x
    // 14336 in 685 us (41 us for 576 tokens), dh rounded to bf16 on the way; here it passes under the next tile's MMAs.
    if (!wait()) return false;
    const unsigned long long grow = reinterpret_cast<unsigned long long>(reinterpret_cast<const __nv_bfloat16*>(p.swiglu_g) + r.base);
    const unsigned long long urow = reinterpret_cast<unsigned long long>(reinterpret_cast<const __nv_bfloat16*>(p.swiglu_u) + r.base);
    const unsigned long long durow = reinterpret_cast<unsigned long long>(reinterpret_cast<__nv_bfloat16*>(p.C2) + r.base);
#pragma unroll 1
    for (int ch = 0; ch < CHUNKS; ++ch) {
      const int col = col0 + ch * 64;
      if (col >= p.N) break;
      uint4 gk[8], du[8];
      {
        uint4 pu[8];
        epi_fetch(gk, grow, row_ok, lane, col, p.N, p.swiglu_g);
        epi_fetch(pu, urow, row_ok, lane, col, p.N, p.swiglu_u);
        epi_stage_in(stage, gk, lane);
#pragma unroll
        for (int j = 0; j < 8; ++j) gk[j] = *epi_slot(stage, lane, j);     // this lane's row of g
        __syncwarp();
        epi_stage_in(stage, pu, lane);                                     // u: row by row from the stage
      }
#pragma unroll
      for (int part = 0; part < 2; ++part) {
        uint32_t acc[32];
        tmem_ld_32x32(tacc + half * (BN / 2) + ch * 64 + part * 32, acc);
        tmem_ld_wait();
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          uint4* slot = epi_slot(stage, lane, part * 4 + j);
          const uint4 uv = *slot;
          const __nv_bfloat162* g2 = reinterpret_cast<const __nv_bfloat162*>(&gk[part * 4 + j]);
          const __nv_bfloat162* u2 = reinterpret_cast<const __nv_bfloat162*>(&uv);
          uint4 dgv;
          __nv_bfloat162* dg2 = reinterpret_cast<__nv_bfloat162*>(&dgv);
          __nv_bfloat162* du2 = reinterpret_cast<__nv_bfloat162*>(&du[part * 4 + j]);
#pragma unroll
          for (int i = 0; i < 4; ++i) {
            const float2 gf = __bfloat1622float2(g2[i]), uf = __bfloat1622float2(u2[i]);
            const float d0 = __uint_as_float(acc[j * 8 + 2 * i]) * alpha, d1 = __uint_as_float(acc[j * 8 + 2 * i + 1]) * alpha;
            const float s0 = 1.f / (1.f + __expf(-gf.x)), s1 = 1.f / (1.f + __expf(-gf.y));
            du2[i] = __floats2bfloat162_rn(d0 * (gf.x * s0), d1 * (gf.y * s1));
            dg2[i] = __floats2bfloat162_rn(d0 * uf.x * s0 * (1.f + gf.x * (1.f - s0)), d1 * uf.y * s1 * (1.f + gf.y * (1.f - s1)));
          }
          *slot = dgv;
        }
      }
      epi_flush(stage, mine, row_ok, lane, col, p.N);
#pragma unroll
      for (int j = 0; j < 8; ++j) *epi_slot(stage, lane, j) = du[j];
      epi_flush(stage, durow, row_ok, lane, col, p.N);
    }
  } else {
    const bool add = fast && (p.accumulate || p.R != nullptr);
    const unsigned long long src = p.accumulate ? mine : reinterpret_cast<unsigned long long>(reinterpret_cast<const __nv_bfloat16*>(p.R) + r.base);
    uint4 pre[8];                                   // (two chunks' worth of registers would spill, and serialise the loads)
    if (add) epi_fetch(pre, src, row_ok, lane, col0, p.N, p.accumulate ? p.C : p.R);
    if (!wait()) return false;
#pragma unroll 1
    for (int ch = 0; ch < CHUNKS; ++ch) {
      const int col = col0 + ch * 64;
      if (col >= p.N) break;
      if (add) {
        epi_stage_in(stage, pre, lane);
        if (ch + 1 < CHUNKS) epi_fetch(pre, src, row_ok, lane, col + 64, p.N, p.accumulate ? p.C : p.R);
      }
#pragma unroll 1
      for (int part = 0; part < 2; ++part) {
        uint32_t acc[32];
        float v[32];
        tmem_ld_32x32(tacc + half * (BN / 2) + ch * 64 + part * 32, acc);
        tmem_ld_wait();
#pragma unroll
        for (int i = 0; i < 32; ++i) v[i] = __uint_as_float(acc[i]) * alpha;
        if (add) {
          epi_stage_row<true>(stage, v, part, lane);
        } else if (fast) {
          epi_stage_row<false>(stage, v, part, lane);
        } else if (r.ok) {
#pragma unroll
          for (int w = 0; w < 4; ++w) {
            const int cc = col + part * 32 + w * 8;
            if (cc < p.N) {
              float o[8];
#pragma unroll
              for (int i = 0; i < 8; ++i) o[i] = v[w * 8 + i];
              store8(r.C, r.base + cc, o, p.c_fp32, p.accumulate, p.R);
            }
          }
        }
        __syncwarp();   // the next TMEM load is warp-aligned
      }
      if (fast) epi_flush(stage, mine, row_ok, lane, col, p.N);
    }
  }
  return true;
}

// Descriptor of a 64-deep operand tile in shared memory, and its step per 16 k (in descriptor units of 16 bytes; the
// address field never carries out of its 14 bits, shared memory being smaller than 256 KB).
__device__ __forceinline__ uint64_t operand_desc(uint32_t addr, int mn_major) {
  return mn_major ? make_smem_desc(addr, 8192, 1024) : make_smem_desc(addr, 16, 1024);
}
__device__ __forceinline__ uint32_t operand_kstep(int mn_major) { return mn_major ? 2048 >> 4 : 32 >> 4; }

template <int BN, int STAGES, bool SWIGLU>
__global__ void __launch_bounds__(GEMM_THREADS, 1) gemm_sm100_kernel(const __grid_constant__ GemmParams p) {
  constexpr int B_BYTES = BN * BK * 2;
  constexpr int STAGE_BYTES = A_BYTES + B_BYTES;
  constexpr uint32_t TMEM_COLS = 2 * BN;  // 256 or 512: a power of two >= 32

  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  uint64_t* full_bar = reinterpret_cast<uint64_t*>(smem + STAGES * STAGE_BYTES);
  uint64_t* empty_bar = full_bar + STAGES;
  uint64_t* tfull_bar = empty_bar + STAGES;
  uint64_t* tempty_bar = tfull_bar + 2;
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(tempty_bar + 2);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);
  // [accumulator buffer][row quarter]: column halves whose rows have been delivered to peers.  A buffer's two halves
  // count the same tile: a warp reaches the buffer's next tile only after both have released the accumulator.
  unsigned* rows_done = reinterpret_cast<unsigned*>(tmem_slot + 2);
  uint8_t* epi_stage = smem + STAGES * STAGE_BYTES + 256;

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int BN_OUT = p.dual ? BN / 2 : BN;

  if (threadIdx.x == 0) {
    for (int s = 0; s < STAGES; ++s) { mbar_init(&full_bar[s], 1); mbar_init(&empty_bar[s], 1); }
    for (int b = 0; b < 2; ++b) { mbar_init(&tfull_bar[b], 1); mbar_init(&tempty_bar[b], EPI_WARPS); }
    for (int i = 0; i < 8; ++i) rows_done[i] = 0;
    *abort_flag = 0;
    fence_barrier_init();
  }
  if (warp == 1) { tmem_alloc(tmem_slot, TMEM_COLS); tmem_relinquish(); }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = *tmem_slot;
  gemm_begin(p);

  auto fail = [&](int code) {
    *abort_flag = 1;
    if (p.status != nullptr) atomicCAS(p.status, 0, code);
  };

  const bool dead = __any_sync(0xffffffffu, gemm_dead(p));
  if (dead) {
    // nothing to do; fall through to the common exit
  } else if (warp == 0) {
    // ------------------------------------------------------------------ TMA producer
    if (elect_one()) { prefetch_tensormap(&p.tmA); prefetch_tensormap(&p.tmB); }
    uint32_t it = 0;
    Work w;
    bool ok = true;
    for (int wi = 0; ok && (p.dual ? get_work<BN / 2>(p, blockIdx.x, gridDim.x, wi, w) : get_work<BN>(p, blockIdx.x, gridDim.x, wi, w)); ++wi) {
      const Tile& t = w.t;
      const int total_kb = w.kb1 - w.kb0;
      if (p.tile_ready != nullptr) {
        // rows of this tile are stored by peer GPUs: wait for them, then order the TMA reads after the acquire
        const int ti = t.m0 / BM;
        if (!__all_sync(0xffffffffu, wait_ge(p.tile_ready + ti, (unsigned)p.tile_expected[ti], p.peer_wait_ns))) { fail(ST_TIMEOUT_PEER); ok = false; break; }
        fence_proxy_async_all();
      }
      if (p.mode != 2 && total_kb > 0 && (p.rdy_b.ready != nullptr || p.rdy_b2.ready != nullptr || p.rdy_bl.ready != nullptr)) {
        // the weight operand is part of a buffer that an all-gather on another stream is still filling
        if (!__all_sync(0xffffffffu, wait_b_tile(p, t.g, t.n0, BN_OUT))) { fail(ST_TIMEOUT_PEER); ok = false; break; }
        fence_proxy_async_all();
      }
      for (int kb = w.kb0; kb < w.kb1; ++kb, ++it) {
        const int s = it % STAGES;
        const uint32_t ph = (it / STAGES) & 1;
        if (!wait_parity_warp(&empty_bar[s], ph ^ 1, abort_flag)) { fail(ST_TIMEOUT_EMPTY); ok = false; break; }
        uint8_t* sA = smem + s * STAGE_BYTES;
        uint8_t* sB = sA + A_BYTES;
        const bool lora = kb >= t.num_kb;
        const int kk = (lora ? kb - t.num_kb : kb) * BK;
        const CUtensorMap* mA = lora ? &p.tmA_l : &p.tmA;
        const CUtensorMap* mB = lora ? &p.tmB_l : &p.tmB;
        const CUtensorMap* mB2 = lora ? &p.tmB2_l : &p.tmB2;
        const int a_mn = lora ? p.a_mn_l : p.a_mn, b_mn = lora ? p.b_mn_l : p.b_mn;
        const int krow = (lora ? 0 : t.krow0) + kk;
        const int zB = (p.mode == 2) ? 0 : t.g;
        if (elect_one()) {
          mbar_expect_tx(&full_bar[s], STAGE_BYTES);
          if (a_mn == 0) {
            tma_load_2d(sA, mA, &full_bar[s], kk, t.m0);
          } else {
            tma_load_2d(sA, mA, &full_bar[s], t.m0, krow);
            tma_load_2d(sA + 8192, mA, &full_bar[s], t.m0 + 64, krow);
          }
          if (b_mn == 0) {
            if (p.dual) {
              tma_load_3d(sB, mB, &full_bar[s], kk, t.n0, zB);
              tma_load_3d(sB + B_BYTES / 2, mB2, &full_bar[s], kk, t.n0, zB);
            } else {
              tma_load_3d(sB, mB, &full_bar[s], kk, t.n0, zB);
            }
          } else {
            if (p.dual) {
#pragma unroll
              for (int c = 0; c < BN / 128; ++c) {
                tma_load_3d(sB + c * 8192, mB, &full_bar[s], t.n0 + 64 * c, krow, zB);
                tma_load_3d(sB + B_BYTES / 2 + c * 8192, mB2, &full_bar[s], t.n0 + 64 * c, krow, zB);
              }
            } else {
#pragma unroll
              for (int c = 0; c < BN / 64; ++c) tma_load_3d(sB + c * 8192, mB, &full_bar[s], t.n0 + 64 * c, krow, zB);
            }
          }
        }
      }
    }
    if (!ok) {  // give copies already in flight a bounded time to land before the CTA exits
      for (int s = 0; s < STAGES; ++s) {
        uint64_t t0 = global_timer_ns();
        while (!mbar_try_wait(&full_bar[s], 0) && !mbar_try_wait(&full_bar[s], 1) && global_timer_ns() - t0 < 1000000ull) {}
      }
    }
  } else if (warp == 1) {
    // ------------------------------------------------------------------ MMA issuer
    uint32_t it = 0, acc_it = 0;
    Work w;
    bool ok = true;
    for (int wi = 0; ok && (p.dual ? get_work<BN / 2>(p, blockIdx.x, gridDim.x, wi, w) : get_work<BN>(p, blockIdx.x, gridDim.x, wi, w)); ++wi) {
      const Tile& t = w.t;
      const int total_kb = w.kb1 - w.kb0;
      if (total_kb == 0) continue;
      const int buf = acc_it & 1;
      const uint32_t aph = (acc_it >> 1) & 1;
      if (!wait_parity_warp(&tempty_bar[buf], aph ^ 1, abort_flag)) { fail(ST_TIMEOUT_TMEM_EMPTY); break; }
      tc_fence_after();
      const uint32_t d_tmem = tmem_base + buf * BN;
      for (int kb = w.kb0; kb < w.kb1; ++kb, ++it) {
        const int s = it % STAGES;
        const uint32_t ph = (it / STAGES) & 1;
        if (!wait_parity_warp(&full_bar[s], ph, abort_flag)) { fail(ST_TIMEOUT_FULL); ok = false; break; }
        tc_fence_after();
        const bool lora = kb >= t.num_kb;
        const int a_mn = lora ? p.a_mn_l : p.a_mn, b_mn = lora ? p.b_mn_l : p.b_mn;
        const uint32_t idesc = make_idesc_bf16(BM, BN, a_mn, b_mn);
        const uint32_t sA = smem_u32(smem + s * STAGE_BYTES);
        const uint64_t da = operand_desc(sA, a_mn), db = operand_desc(sA + A_BYTES, b_mn);
        const uint32_t ka = operand_kstep(a_mn), kbs = operand_kstep(b_mn);
        if (elect_one()) {
#pragma unroll
          for (int k = 0; k < BK / 16; ++k)
            umma_bf16(d_tmem, da + k * ka, db + k * kbs, idesc, (kb > w.kb0 || k > 0) ? 1u : 0u);
          umma_commit(&empty_bar[s]);   // frees the stage when these MMAs have read it
        }
      }
      if (!ok) break;
      if (elect_one()) umma_commit(&tfull_bar[buf]);   // accumulator complete
      ++acc_it;
    }
  } else if (warp >= 2) {
    // ------------------------------------------------------------------ epilogue
    const int q = warp & 3, half = (warp - 2) >> 2;
    uint8_t* stage = epi_stage + (warp - 2) * EPI_STAGE_BYTES;
    uint32_t acc_it = 0;
    Work w;
    for (int wi = 0; (p.dual ? get_work<BN / 2>(p, blockIdx.x, gridDim.x, wi, w) : get_work<BN>(p, blockIdx.x, gridDim.x, wi, w)); ++wi) {
      const Tile& t = w.t;
      const int row = t.m0 + q * 32 + lane;
      const bool row_ok = row < ((p.mode == 1) ? p.offsets[p.G] : p.M);
      const EpiRow r = epi_row(p, t.g, row, row_ok);
      if (w.kb1 == w.kb0) {
        if (p.dual) epi_zero<BN / 4>(p, r, row_ok, t.n0 + half * (BN / 4));
        else epi_zero<BN / 2>(p, r, row_ok, t.n0 + half * (BN / 2));
        continue;
      }
      const int buf = acc_it & 1;
      const uint32_t aph = (acc_it >> 1) & 1;
      auto wait = [&]() {
        // (one answer for the warp: the TMEM loads and shuffles that follow are warp-wide)
        if (!wait_parity_warp(&tfull_bar[buf], aph, abort_flag)) { fail(ST_TIMEOUT_TMEM_FULL); return false; }
        tc_fence_after();
        return true;
      };
      const uint32_t tacc = tmem_base + buf * BN + ((uint32_t)(q * 32) << 16);
      bool publish = p.row_dest_rank != nullptr;
      if (w.split >= 0) {
        // A piece of a shared tile: add the partial sums into the tile's fp32 workspace (four columns of a row at a time,
        // rows adjacent, so that a warp's reduction covers 512 contiguous bytes), release the accumulator, count this
        // warp in, and if it is the last of the contributors to its part, read the sums back and finish that part.
        // Each (32-row quarter, column half) has its own counter, so no warp ever has to meet another one of its CTA.
        if (!wait()) break;
        float4* ws = reinterpret_cast<float4*>(p.sk_ws) + (long long)w.split * (BM * BN / 4) + half * (BN / 8) * BM + (q * 32 + lane);
#pragma unroll 1
        for (int c = 0; c < BN / 2; c += 32) {
          uint32_t acc[32];
          tmem_ld_32x32(tacc + half * (BN / 2) + c, acc);
          tmem_ld_wait();
#pragma unroll
          for (int i = 0; i < 32; i += 4)
            red_add_v4_f32(reinterpret_cast<float*>(ws + (c + i) / 4 * BM), __uint_as_float(acc[i]), __uint_as_float(acc[i + 1]),
                           __uint_as_float(acc[i + 2]), __uint_as_float(acc[i + 3]));
          __syncwarp();
        }
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(&tempty_bar[buf]);
        ++acc_it;
        __threadfence();
        __syncwarp();
        unsigned* ctr = p.sk_ctr + w.split * SPLIT_COUNTERS;
        unsigned before = 0;
        if (lane == 0) before = atomicAdd(ctr + q * 2 + half, 1u);
        before = __shfl_sync(0xffffffffu, before, 0);
        if (before != (unsigned)w.contributors - 1u) continue;
        __threadfence();
        const float alpha = gemm_alpha(p);
#pragma unroll 1
        for (int c = 0; c < BN / 2; c += 8) {
          float o[8];
#pragma unroll
          for (int i = 0; i < 8; i += 4) {
            float4* src = ws + (c + i) / 4 * BM;
            const float4 v = __ldcg(src);
            __stcg(src, make_float4(0.f, 0.f, 0.f, 0.f));   // leave the workspace clean
            o[i] = v.x * alpha; o[i + 1] = v.y * alpha; o[i + 2] = v.z * alpha; o[i + 3] = v.w * alpha;
          }
          const int col = t.n0 + half * (BN / 2) + c;
          if (r.ok && col < p.N) store8(r.C, r.base + col, o, p.c_fp32, p.accumulate, p.R);
        }
        __syncwarp();
        if (lane == 0) ctr[q * 2 + half] = 0;
        if (publish) {          // by the half that finishes second
          __threadfence_system();
          __syncwarp();
          if (lane == 0) { before = atomicAdd(ctr + 8 + q, 1u); if (before == 1u) ctr[8 + q] = 0; }
          before = __shfl_sync(0xffffffffu, before, 0);
          if (before == 1u) epi_publish(p, r.dest, lane);
        }
        continue;
      }
      if (!epi_tile<BN, SWIGLU>(p, stage, tacc, half, lane, t.n0, r, wait)) break;
      if (publish) {            // by the half that finishes second (before the accumulator is released, see rows_done)
        __threadfence_system();
        __syncwarp();
        unsigned before = 0;
        if (lane == 0) before = atomicAdd(&rows_done[buf * 4 + q], 1u);
        before = __shfl_sync(0xffffffffu, before, 0);
        if (before & 1u) epi_publish(p, r.dest, lane);
      }
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(&tempty_bar[buf]);
      ++acc_it;
    }
  }

  __syncwarp();
  tc_fence_before();
  __syncthreads();
  if (warp == 1) { tc_fence_after(); tmem_dealloc(tmem_base, TMEM_COLS); }
}

// ---------------------------------------------------------------------------------------------
// CTA-pair variant (cta_group::2).  Two CTAs of a cluster share one 256 x 256 MMA tile: each CTA loads its own
// 128 rows of A and half of B's 256 columns (in the dual mode: the leader the gate matrix, its peer the up
// matrix), the leader's MMA thread reads both CTAs' shared memory, and each CTA's TMEM receives the accumulators
// of its own 128 rows.  Per CTA and 64-deep k block that is 32 KB of operands instead of 48 KB.  What bounds the
// single-CTA kernel is the ~64 bytes per clock that an SM takes in (0.38 us for 48 KB; with the MMAs left out it runs
// no faster), and a 256 x 256 tile in one CTA is bound by shared memory (64 KB written, 96 KB read by the MMAs per k
// block).  The pair needs 64 KB of either for 512 clocks of MMA.  8192^3: 1634 TFLOP/s (128-row kernel 1390, torch's
// library call 1670); 9200 x 4096 x 4096: 183 us, 1684 TFLOP/s (before: 212 us).  Its roles run as whole warps: with a
// single lane in the loops (922 us at 8192^3) the issue of the MMAs was the limit.
//   full_bar[s]   (leader's is used): the leader's producer arrives and announces both CTAs' TMA bytes
//   empty_bar[s]  (one per CTA)     : arrives by the leader's commit, delivered to both CTAs
//   tfull_bar[b]  (one per CTA)     : same, when a tile's accumulators are complete
//   tempty_bar[b] (leader's is used): 16 arrivals, the 8 epilogue warps of each CTA
// Every load lands in the shared memory of the CTA that issued it.
// ---------------------------------------------------------------------------------------------
constexpr int PAIR_BN = 256;
constexpr int PAIR_STAGES = 6;
constexpr int PAIR_B_BYTES = 128 * BK * 2;
constexpr int PAIR_STAGE_BYTES = A_BYTES + PAIR_B_BYTES;
constexpr int PAIR_SMEM = PAIR_STAGES * PAIR_STAGE_BYTES + 1024 + 256 + EPI_WARPS * EPI_STAGE_BYTES;
static_assert(PAIR_SMEM <= 227 * 1024, "pair kernel: stages + barriers + epilogue stages exceed the shared memory of a CTA");

template <bool SWIGLU>
__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(GEMM_THREADS, 1) gemm_sm100_pair_kernel(const __grid_constant__ GemmParams p) {
  constexpr int STAGES = PAIR_STAGES;
  constexpr int BN = PAIR_BN;
  constexpr uint32_t TMEM_COLS = 2 * BN;

  extern __shared__ uint8_t smem_raw[];
  // the dynamic shared memory starts at the same offset in both CTAs, so the aligned tile addresses match too
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  uint64_t* full_bar = reinterpret_cast<uint64_t*>(smem + STAGES * PAIR_STAGE_BYTES);
  uint64_t* empty_bar = full_bar + STAGES;
  uint64_t* tfull_bar = empty_bar + STAGES;
  uint64_t* tempty_bar = tfull_bar + 2;
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(tempty_bar + 2);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);
  unsigned* rows_done = reinterpret_cast<unsigned*>(tmem_slot + 2);   // as in the 128-row kernel
  uint8_t* epi_stage = smem + STAGES * PAIR_STAGE_BYTES + 256;

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const uint32_t cta_rank = cluster_ctarank();          // 0 = leader
  const int pair_id = (int)cluster_id_x(), num_pairs = (int)num_clusters_x();
  const int BN_OUT = p.dual ? BN / 2 : BN;

  if (threadIdx.x == 0) {
    for (int s = 0; s < STAGES; ++s) { mbar_init(&full_bar[s], 1); mbar_init(&empty_bar[s], 1); }
    for (int b = 0; b < 2; ++b) { mbar_init(&tfull_bar[b], 1); mbar_init(&tempty_bar[b], 2 * EPI_WARPS); }
    for (int i = 0; i < 8; ++i) rows_done[i] = 0;
    *abort_flag = 0;
    fence_barrier_init();
  }
  if (warp == 1) { tmem_alloc_pair(tmem_slot, TMEM_COLS); tmem_relinquish_pair(); }
  tc_fence_before();
  cluster_sync_all();
  tc_fence_after();
  const uint32_t tmem_base = *tmem_slot;
  gemm_begin(p);

  auto fail = [&](int code) {
    *abort_flag = 1;
    if (p.status != nullptr) atomicCAS(p.status, 0, code);
  };

  const bool dead = __any_sync(0xffffffffu, gemm_dead(p));   // the same in both CTAs of the pair: the word never returns to zero while kernels run
  if (dead) {
    // nothing to do; fall through to the common exit
  } else if (warp == 0) {
    // ------------------------------------------------------------------ TMA producer (one per CTA)
    if (elect_one()) { prefetch_tensormap(&p.tmA); prefetch_tensormap(&p.tmB); }
    uint32_t it = 0;
    PairTile t;
    bool ok = true;
    for (int tile = pair_id; ok && (p.dual ? get_pair_tile<BN / 2>(p, tile, t) : get_pair_tile<BN>(p, tile, t)); tile += num_pairs) {
      const int total_kb = t.num_kb + (t.num_kb > 0 || p.mode != 2 ? t.num_kb_l : 0);
      const int my_m0 = t.m0 + (int)cta_rank * BM;
      const bool half_ok = cta_rank == 0 || t.second_ok;
      if (p.tile_ready != nullptr && half_ok && total_kb > 0) {
        const int ti = my_m0 / BM;
        if (!__all_sync(0xffffffffu, wait_ge(p.tile_ready + ti, (unsigned)p.tile_expected[ti], p.peer_wait_ns))) { fail(ST_TIMEOUT_PEER); ok = false; break; }
        fence_proxy_async_all();
      }
      if (p.mode != 2 && total_kb > 0 && (p.rdy_b.ready != nullptr || p.rdy_b2.ready != nullptr || p.rdy_bl.ready != nullptr)) {
        if (!__all_sync(0xffffffffu, wait_b_tile(p, t.g, t.n0, BN_OUT))) { fail(ST_TIMEOUT_PEER); ok = false; break; }
        fence_proxy_async_all();
      }
      for (int kb = 0; kb < total_kb; ++kb, ++it) {
        const int s = it % STAGES;
        const uint32_t ph = (it / STAGES) & 1;
        if (!wait_parity_warp(&empty_bar[s], ph ^ 1, abort_flag)) { fail(ST_TIMEOUT_EMPTY); ok = false; break; }
        uint8_t* sA = smem + s * PAIR_STAGE_BYTES;
        uint8_t* sB = sA + A_BYTES;
        // Only the leader arrives, announcing both CTAs' bytes: a cluster-scope arrive from the peer would put a
        // memory barrier into every stage of its producer loop.  The peer's bytes may be counted before the
        // leader's announcement (the transaction count goes negative for a moment; the phase cannot complete
        // before the leader's arrival).
        const uint32_t bar = mapa_shared(smem_u32(&full_bar[s]), 0);
        const bool lora = kb >= t.num_kb;
        const int kk = (lora ? kb - t.num_kb : kb) * BK;
        const CUtensorMap* mA = lora ? &p.tmA_l : &p.tmA;
        const CUtensorMap* mB = lora ? &p.tmB_l : &p.tmB;
        const int a_mn = lora ? p.a_mn_l : p.a_mn, b_mn = lora ? p.b_mn_l : p.b_mn;
        const int krow = (lora ? 0 : t.krow0) + kk;
        const int zB = (p.mode == 2) ? 0 : t.g;
        // this CTA's half of B: columns n0 + 128*rank, or in the dual mode the gate (leader) / up (peer) matrix
        if (p.dual && cta_rank == 1) mB = lora ? &p.tmB2_l : &p.tmB2;
        const int my_n0 = p.dual ? t.n0 : t.n0 + (int)cta_rank * 128;
        if (elect_one()) {
          if (cta_rank == 0) mbar_expect_tx(&full_bar[s], 2 * PAIR_STAGE_BYTES);
          if (a_mn == 0) {
            tma_load_2d_pair(sA, mA, bar, kk, my_m0);
          } else {
            tma_load_2d_pair(sA, mA, bar, my_m0, krow);
            tma_load_2d_pair(sA + 8192, mA, bar, my_m0 + 64, krow);
          }
          if (b_mn == 0) {
            tma_load_3d_pair(sB, mB, bar, kk, my_n0, zB);
          } else {
            tma_load_3d_pair(sB, mB, bar, my_n0, krow, zB);
            tma_load_3d_pair(sB + 8192, mB, bar, my_n0 + 64, krow, zB);
          }
        }
      }
    }
    if (!ok) {  // give this CTA's copies already in flight a bounded time to land before it leaves
      const uint64_t t0 = global_timer_ns();
      while (global_timer_ns() - t0 < 2000000ull) {}
    }
  } else if (warp == 1 && cta_rank == 0) {
    // ------------------------------------------------------------------ MMA issuer (leader only)
    uint32_t it = 0, acc_it = 0;
    PairTile t;
    bool ok = true;
    for (int tile = pair_id; ok && (p.dual ? get_pair_tile<BN / 2>(p, tile, t) : get_pair_tile<BN>(p, tile, t)); tile += num_pairs) {
      const int total_kb = t.num_kb + (t.num_kb > 0 || p.mode != 2 ? t.num_kb_l : 0);
      if (total_kb == 0) continue;
      const int buf = acc_it & 1;
      const uint32_t aph = (acc_it >> 1) & 1;
      if (!wait_parity_warp(&tempty_bar[buf], aph ^ 1, abort_flag)) { fail(ST_TIMEOUT_TMEM_EMPTY); break; }
      tc_fence_after();
      const uint32_t d_tmem = tmem_base + buf * BN;
      for (int kb = 0; kb < total_kb; ++kb, ++it) {
        const int s = it % STAGES;
        const uint32_t ph = (it / STAGES) & 1;
        if (!wait_parity_warp(&full_bar[s], ph, abort_flag)) { fail(ST_TIMEOUT_FULL); ok = false; break; }
        tc_fence_after();
        const bool lora = kb >= t.num_kb;
        const int a_mn = lora ? p.a_mn_l : p.a_mn, b_mn = lora ? p.b_mn_l : p.b_mn;
        const uint32_t idesc = make_idesc_bf16(2 * BM, BN, a_mn, b_mn);
        const uint32_t sA = smem_u32(smem + s * PAIR_STAGE_BYTES);
        const uint64_t da = operand_desc(sA, a_mn), db = operand_desc(sA + A_BYTES, b_mn);
        const uint32_t ka = operand_kstep(a_mn), kbs = operand_kstep(b_mn);
        if (elect_one()) {
#pragma unroll
          for (int k = 0; k < BK / 16; ++k)
            umma_bf16_pair(d_tmem, da + k * ka, db + k * kbs, idesc, (kb > 0 || k > 0) ? 1u : 0u);
          umma_commit_pair(&empty_bar[s], 3);   // frees the stage in both CTAs
        }
      }
      if (!ok) break;
      if (elect_one()) umma_commit_pair(&tfull_bar[buf], 3);   // accumulators complete, in both CTAs
      ++acc_it;
    }
  } else if (warp >= 2) {
    // ------------------------------------------------------------------ epilogue (both CTAs, own 128 rows)
    const int q = warp & 3, half = (warp - 2) >> 2;
    uint8_t* stage = epi_stage + (warp - 2) * EPI_STAGE_BYTES;
    uint32_t acc_it = 0;
    PairTile t;
    for (int tile = pair_id; (p.dual ? get_pair_tile<BN / 2>(p, tile, t) : get_pair_tile<BN>(p, tile, t)); tile += num_pairs) {
      const int total_kb = t.num_kb + (t.num_kb > 0 || p.mode != 2 ? t.num_kb_l : 0);
      const int row = t.m0 + (int)cta_rank * BM + q * 32 + lane;
      const bool row_ok = (cta_rank == 0 || t.second_ok) && row < ((p.mode == 1) ? p.offsets[p.G] : p.M);
      const EpiRow r = epi_row(p, t.g, row, row_ok);
      if (total_kb == 0) {
        if (p.dual) epi_zero<BN / 4>(p, r, row_ok, t.n0 + half * (BN / 4));
        else epi_zero<BN / 2>(p, r, row_ok, t.n0 + half * (BN / 2));
        continue;
      }
      const int buf = acc_it & 1;
      const uint32_t aph = (acc_it >> 1) & 1;
      auto wait = [&]() {
        // (one answer for the warp: the TMEM loads and shuffles that follow are warp-wide)
        if (!wait_parity_warp(&tfull_bar[buf], aph, abort_flag)) { fail(ST_TIMEOUT_TMEM_FULL); return false; }
        tc_fence_after();
        return true;
      };
      if (!epi_tile<BN, SWIGLU>(p, stage, tmem_base + buf * BN + ((uint32_t)(q * 32) << 16), half, lane, t.n0, r, wait)) break;
      if (p.row_dest_rank != nullptr) {            // by the half that finishes second (see the 128-row kernel)
        __threadfence_system();
        __syncwarp();
        unsigned before = 0;
        if (lane == 0) before = atomicAdd(&rows_done[buf * 4 + q], 1u);
        before = __shfl_sync(0xffffffffu, before, 0);
        if (before & 1u) epi_publish(p, r.dest, lane);
      }
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

// ---------------------------------------------------------------------------------------------
// Products with few output tiles: a cluster of S CTAs shares one 128 x BN tile along the depth.
//
// 16 tiles of a 4096-deep projection of one prompt leave 132 SMs idle while each tile's 64 k blocks wait for memory one
// ring at a time (43 us); the adapters' down projections are one column of tiles, 224 deep for the experts.  Here
// CTA c of a cluster takes the c-th part of the k blocks; the S partial tiles then go to shared memory (the ring is
// free by then) and every CTA adds up its share of the tile from all S of them, in the order of the ranks, so that the
// result does not depend on timing.  BN = 64 serves the adapter ranks (64 columns are one swizzle atom).  Same roles as the 128-row kernel, one tile per cluster, no peers' rows (those products keep the other kernels).
// ---------------------------------------------------------------------------------------------
constexpr int MAX_CLUSTER = 8;
template <int BN> struct SplitShape {
  static constexpr int STAGE = A_BYTES + BN * BK * 2;
  static constexpr int STAGES = BN == 256 ? 4 : (BN == 128 ? 6 : 8);   // 192 KB
  static constexpr int SMEM = STAGES * STAGE + 1024 + 256;
  static_assert(STAGES * STAGE >= BM * BN * 4, "the ring must hold the fp32 tile");
  static_assert(SMEM <= 227 * 1024, "shared memory of a CTA");
};

template <int BN>
__device__ __forceinline__ void cluster_product(const GemmParams& p, int index) {
  constexpr int STAGES = SplitShape<BN>::STAGES, STAGE_BYTES = SplitShape<BN>::STAGE;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  uint64_t* full_bar = reinterpret_cast<uint64_t*>(smem + STAGES * STAGE_BYTES);
  uint64_t* empty_bar = full_bar + STAGES;
  uint64_t* done_bar = empty_bar + STAGES;
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(done_bar + 1);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int rank = (int)cluster_ctarank(), S = (int)cluster_nctarank();
  Tile t;
  if (p.offsets != nullptr) wait_for_predecessor();
  if (!locate_tile<BN, BM>(p, index, t)) return;                    // the same for the whole cluster
  if (threadIdx.x == 0) {
    for (int s = 0; s < STAGES; ++s) { mbar_init(&full_bar[s], 1); mbar_init(&empty_bar[s], 1); }
    mbar_init(done_bar, 1);
    *abort_flag = 0;
    fence_barrier_init();
  }
  if (warp == 1) { tmem_alloc(tmem_slot, BN); tmem_relinquish(); }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = *tmem_slot;
  gemm_begin(p);
  auto fail = [&](int code) {
    *abort_flag = 1;
    if (p.status != nullptr) atomicCAS(p.status, 0, code);
  };
  const int total = t.num_kb + (t.num_kb > 0 || p.mode != 2 ? t.num_kb_l : 0);
  const int kb0 = total * rank / S, kb1 = total * (rank + 1) / S;

  if (warp == 0) {
    // ------------------------------------------------------------------ TMA producer
    if (elect_one()) { prefetch_tensormap(&p.tmA); prefetch_tensormap(&p.tmB); }
    bool ok = true;
    if (p.mode != 2 && kb1 > kb0 && (p.rdy_b.ready != nullptr || p.rdy_bl.ready != nullptr)) {
      ok = __all_sync(0xffffffffu, wait_b_tile(p, t.g, t.n0, BN));
      if (!ok) fail(ST_TIMEOUT_PEER);
      fence_proxy_async_all();
    }
    for (int kb = kb0, it = 0; ok && kb < kb1; ++kb, ++it) {
      const int s = it % STAGES;
      ok = wait_parity_warp(&empty_bar[s], ((it / STAGES) & 1) ^ 1, abort_flag);
      if (!ok) { fail(ST_TIMEOUT_EMPTY); break; }
      uint8_t* sA = smem + s * STAGE_BYTES;
      uint8_t* sB = sA + A_BYTES;
      const bool lora = kb >= t.num_kb;
      const int kk = (lora ? kb - t.num_kb : kb) * BK;
      const CUtensorMap* mA = lora ? &p.tmA_l : &p.tmA;
      const CUtensorMap* mB = lora ? &p.tmB_l : &p.tmB;
      const int a_mn = lora ? p.a_mn_l : p.a_mn, b_mn = lora ? p.b_mn_l : p.b_mn;
      const int krow = (lora ? 0 : t.krow0) + kk;
      const int zB = (p.mode == 2) ? 0 : t.g;
      if (elect_one()) {
        mbar_expect_tx(&full_bar[s], STAGE_BYTES);
        if (a_mn == 0) {
          tma_load_2d(sA, mA, &full_bar[s], kk, t.m0);
        } else {
          tma_load_2d(sA, mA, &full_bar[s], t.m0, krow);
          tma_load_2d(sA + 8192, mA, &full_bar[s], t.m0 + 64, krow);
        }
        if (b_mn == 0) {
          tma_load_3d(sB, mB, &full_bar[s], kk, t.n0, zB);
        } else {
#pragma unroll
          for (int c = 0; c < BN / 64; ++c) tma_load_3d(sB + c * 8192, mB, &full_bar[s], t.n0 + 64 * c, krow, zB);
        }
      }
    }
    if (!ok) {   // give copies in flight a bounded time to land before the CTA leaves
      const uint64_t t0 = global_timer_ns();
      while (global_timer_ns() - t0 < 2000000ull) {}
    }
  } else if (warp == 1) {
    // ------------------------------------------------------------------ MMA issuer
    bool ok = true;
    for (int kb = kb0, it = 0; kb < kb1; ++kb, ++it) {
      const int s = it % STAGES;
      ok = wait_parity_warp(&full_bar[s], (it / STAGES) & 1, abort_flag);
      if (!ok) { fail(ST_TIMEOUT_FULL); break; }
      tc_fence_after();
      const bool lora = kb >= t.num_kb;
      const int a_mn = lora ? p.a_mn_l : p.a_mn, b_mn = lora ? p.b_mn_l : p.b_mn;
      const uint32_t idesc = make_idesc_bf16(BM, BN, a_mn, b_mn);
      const uint32_t sA = smem_u32(smem + s * STAGE_BYTES);
      const uint64_t da = operand_desc(sA, a_mn), db = operand_desc(sA + A_BYTES, b_mn);
      const uint32_t ka = operand_kstep(a_mn), kbs = operand_kstep(b_mn);
      if (elect_one()) {
#pragma unroll
        for (int k = 0; k < BK / 16; ++k) umma_bf16(tmem, da + k * ka, db + k * kbs, idesc, (kb > kb0 || k > 0) ? 1u : 0u);
        umma_commit(&empty_bar[s]);
      }
    }
    if (ok && kb1 > kb0 && elect_one()) umma_commit(done_bar);
  } else {
    // ------------------------------------------------------------------ partial tile: TMEM -> shared memory [column / 4][row][4]
    const int q = warp & 3, half = (warp - 2) >> 2;
    float4* part = reinterpret_cast<float4*>(smem) + q * 32 + lane;
    if (kb1 > kb0) {
      const bool ok = wait_parity_warp(done_bar, 0, abort_flag);
      if (!ok) fail(ST_TIMEOUT_TMEM_FULL);
      tc_fence_after();
#pragma unroll 1
      for (int c = half * (BN / 2); ok && c < (half + 1) * (BN / 2); c += 16) {
        uint32_t acc[16];
        tmem_ld_32x16(tmem + c + ((uint32_t)(q * 32) << 16), acc);
        tmem_ld_wait();
#pragma unroll
        for (int i = 0; i < 16; i += 4)
          part[(c + i) / 4 * BM] = make_float4(__uint_as_float(acc[i]), __uint_as_float(acc[i + 1]), __uint_as_float(acc[i + 2]), __uint_as_float(acc[i + 3]));
      }
    } else {
      for (int c = half * (BN / 2); c < (half + 1) * (BN / 2); c += 4) part[c / 4 * BM] = make_float4(0.f, 0.f, 0.f, 0.f);
    }
  }
  __syncwarp();
  tc_fence_before();
  cluster_sync_all();                                             // all partial tiles are in place
  if (warp == 1) { tc_fence_after(); tmem_dealloc(tmem, BN); }
  // this CTA's share: units of one row x 8 columns, rows fastest
  constexpr int UNITS = BM * (BN / 8);
  const float alpha = gemm_alpha(p);
  const int row_limit = (p.mode == 1) ? p.offsets[p.G] : p.M;
  const bool empty = total == 0 && p.accumulate;
  const uint32_t part0 = smem_u32(smem);
  for (int u = UNITS * rank / S + (int)threadIdx.x; u < UNITS * (rank + 1) / S && !empty; u += GEMM_THREADS) {
    const int r = u % BM, g8 = u / BM;
    const int row = t.m0 + r, col = t.n0 + g8 * 8;
    if (row >= row_limit || col >= p.N) continue;
    float o[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
    const uint32_t at = part0 + ((2 * g8) * BM + r) * 16;
    for (int c = 0; c < S; ++c) {
      const uint32_t a = mapa_shared(at, c);
      const float4 x = ld_cluster_v4(a), y = ld_cluster_v4(a + BM * 16);
      o[0] += x.x; o[1] += x.y; o[2] += x.z; o[3] += x.w; o[4] += y.x; o[5] += y.y; o[6] += y.z; o[7] += y.w;
    }
#pragma unroll
    for (int i = 0; i < 8; ++i) o[i] *= alpha;
    store8(p.C, (p.mode == 2 ? (long long)t.g * p.c_group_stride : 0) + (long long)row * p.ldc + col, o, p.c_fp32, p.accumulate, p.R);
  }
  cluster_sync_all();                                             // nobody leaves while its partial tile is read
}
template <int BN>
__global__ void __launch_bounds__(GEMM_THREADS, 1) gemm_sm100_cluster_kernel(const __grid_constant__ GemmParams p) {
  cluster_product<BN>(p, (int)cluster_id_x());
}
// Several small products in one launch: the adapter products of a block, each a few tiles of some microseconds, of which the
// launch, the set-up of the CTAs and the exchange are most.
constexpr int MAX_PRODUCTS = 8;
struct ProductList { int count, tile0[MAX_PRODUCTS + 1]; GemmParams p[MAX_PRODUCTS]; };
template <int BN>
__global__ void __launch_bounds__(GEMM_THREADS, 1) gemm_sm100_list_kernel(const __grid_constant__ ProductList list) {
  const int c = (int)cluster_id_x();
  int i = 0;
  while (i + 1 < list.count && c >= list.tile0[i + 1]) ++i;
  cluster_product<BN>(list.p[i], c - list.tile0[i]);
}

#include "gemm_transposed.cuh"
#include "gemm_wgrad.cuh"

// ---------------------------------------------------------------------------------------------
// host side
// ---------------------------------------------------------------------------------------------
typedef CUresult (*EncodeTiledFn)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*,
                                  const cuuint64_t*, const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave,
                                  CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

static EncodeTiledFn encode_fn() {
  static EncodeTiledFn fn = nullptr;
  static std::once_flag once;
  std::call_once(once, [] {
    void* ptr = nullptr;
    cudaDriverEntryPointQueryResult qres;
    if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &ptr, cudaEnableDefault, &qres) == cudaSuccess &&
        qres == cudaDriverEntryPointSuccess)
      fn = reinterpret_cast<EncodeTiledFn>(ptr);
  });
  return fn;
}

// bf16 tensor [d2][d1][d0] (d0 contiguous), strides in elements; box = {b0, b1, 1}
// Encoded maps are cached per host thread: a training step re-uses the same (pointer, shape, box) combinations
// (weights, pooled gather buffers, allocator-recycled activations) thousands of times.
struct MapKey {
  uint64_t v[8];
  bool operator==(const MapKey& o) const { return memcmp(v, o.v, sizeof(v)) == 0; }
};
struct MapKeyHash {
  size_t operator()(const MapKey& k) const {
    uint64_t h = 1469598103934665603ull;
    for (int i = 0; i < 8; ++i) { h ^= k.v[i]; h *= 1099511628211ull; }
    return (size_t)h;
  }
};
static int make_map_uncached(CUtensorMap* m, const void* ptr, uint64_t d0, uint64_t d1, uint64_t d2, uint64_t s1, uint64_t s2,
                             uint32_t b0, uint32_t b1, int rank);
static int make_map(CUtensorMap* m, const void* ptr, uint64_t d0, uint64_t d1, uint64_t d2, uint64_t s1, uint64_t s2,
                    uint32_t b0, uint32_t b1, int rank) {
  static thread_local std::unordered_map<MapKey, CUtensorMap, MapKeyHash> cache;
  MapKey k{{(uint64_t)reinterpret_cast<uintptr_t>(ptr), d0, d1, d2, s1, s2, ((uint64_t)b0 << 32) | b1, (uint64_t)rank}};
  auto it = cache.find(k);
  if (it != cache.end()) { *m = it->second; return 0; }
  int rc = make_map_uncached(m, ptr, d0, d1, d2, s1, s2, b0, b1, rank);
  if (rc == 0) {
    if (cache.size() > 65536) cache.clear();
    cache.emplace(k, *m);
  }
  return rc;
}
static int make_map_uncached(CUtensorMap* m, const void* ptr, uint64_t d0, uint64_t d1, uint64_t d2, uint64_t s1, uint64_t s2,
                             uint32_t b0, uint32_t b1, int rank) {
  EncodeTiledFn fn = encode_fn();
  if (fn == nullptr) return -1;
  cuuint64_t dims[3] = {d0, d1, d2};
  cuuint64_t strides[2] = {s1 * 2, s2 * 2};
  cuuint32_t box[3] = {b0, b1, 1};
  cuuint32_t estr[3] = {1, 1, 1};
  if ((reinterpret_cast<uintptr_t>(ptr) & 15) || (strides[0] & 15) || (rank == 3 && (strides[1] & 15))) return -2;
  CUresult r = fn(m, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, rank, const_cast<void*>(ptr), dims, strides, box, estr,
                  CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                  CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  return r == CUDA_SUCCESS ? 0 : -3;
}

static int g_num_sms = 0;
static long long g_launches = 0;

// Workspace of the split last wave: one fp32 tile per SM plus SPLIT_COUNTERS counters per tile, zero between launches (the
// warp that finishes a shared tile clears what it read).  One workspace per stream, since launches on different streams may
// overlap on the GPU; created on the stream's first product that can use it and cleared by that stream itself: a clear on
// the default stream is not ordered against a non-blocking stream, and one that comes late takes back partial sums and
// counts, so that a part never sees its last contributor and stays unwritten.  MDT_GEMM_SPLIT=0 switches the split off.
struct SplitWorkspace { float* ws; unsigned* ctr; };
static std::mutex g_split_mutex;
static std::map<std::pair<int, cudaStream_t>, SplitWorkspace> g_split_ws;
static int g_split_enabled = -1;
static bool split_enabled() {
  if (g_split_enabled < 0) {
    const char* e = getenv("MDT_GEMM_SPLIT");
    g_split_enabled = (e != nullptr && e[0] == '0') ? 0 : 1;
  }
  return g_split_enabled == 1;
}
static bool split_workspace(cudaStream_t stream, SplitWorkspace* out) {
  int dev = 0;
  cudaGetDevice(&dev);
  std::lock_guard<std::mutex> lock(g_split_mutex);
  auto key = std::make_pair(dev, stream);
  auto it = g_split_ws.find(key);
  if (it == g_split_ws.end()) {
    if (g_split_ws.size() >= 64) return false;          // more streams than expected: those products run unsplit
    // (a capture can neither allocate nor clear for the launches that run outside it: unsplit)
    cudaStreamCaptureStatus capturing = cudaStreamCaptureStatusNone;
    if (cudaStreamIsCapturing(stream, &capturing) != cudaSuccess || capturing != cudaStreamCaptureStatusNone) { cudaGetLastError(); return false; }
    SplitWorkspace w{nullptr, nullptr};
    const size_t ws_bytes = (size_t)g_num_sms * BM * 256 * sizeof(float), ctr_bytes = (size_t)g_num_sms * SPLIT_COUNTERS * sizeof(unsigned);
    if (cudaMalloc(&w.ws, ws_bytes) != cudaSuccess) { cudaGetLastError(); return false; }
    if (cudaMalloc(&w.ctr, ctr_bytes) != cudaSuccess) { cudaGetLastError(); cudaFree(w.ws); return false; }
    if (cudaMemsetAsync(w.ws, 0, ws_bytes, stream) != cudaSuccess || cudaMemsetAsync(w.ctr, 0, ctr_bytes, stream) != cudaSuccess) {
      cudaGetLastError();
      cudaFree(w.ws);
      cudaFree(w.ctr);
      return false;
    }
    it = g_split_ws.emplace(key, w).first;
  }
  *out = it->second;
  return true;
}

template <int BN, int STAGES, bool SWIGLU>
static cudaError_t launch(const GemmParams& p, int grid, cudaStream_t stream) {
  constexpr int smem = STAGES * (A_BYTES + BN * BK * 2) + 1024 + 256 + EPI_WARPS * EPI_STAGE_BYTES;
  static_assert(smem <= 227 * 1024, "stages + barriers + epilogue stages exceed the shared memory of a CTA");
  static bool configured = false;
  if (!configured) {
    cudaError_t e = cudaFuncSetAttribute(gemm_sm100_kernel<BN, STAGES, SWIGLU>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
    if (e != cudaSuccess) return e;
    configured = true;
  }
  launch_after(gemm_sm100_kernel<BN, STAGES, SWIGLU>, grid, GEMM_THREADS, smem, stream, p);
  ++g_launches;
  return cudaGetLastError();
}

// Number of CTA pairs that can be resident at once (pairs never span GPCs, so this can be below SMs / 2); the
// persistent grid is sized to it because tiles are assigned to pairs statically.
static int g_max_pairs = 0;
static int g_pair_cap = 0;   // optional upper bound set through mdt_gemm_set_pair_cap (0 = none)

template <class Kernel>
static int resident_pairs(Kernel kernel, int smem) {
  cudaLaunchConfig_t cfg;
  memset(&cfg, 0, sizeof(cfg));
  cfg.gridDim = dim3((unsigned)(g_num_sms & ~1)); cfg.blockDim = dim3(GEMM_THREADS); cfg.dynamicSmemBytes = smem;
  cudaLaunchAttribute attr;
  attr.id = cudaLaunchAttributeClusterDimension;
  attr.val.clusterDim.x = 2; attr.val.clusterDim.y = 1; attr.val.clusterDim.z = 1;
  cfg.attrs = &attr; cfg.numAttrs = 1;
  int n = 0;
  if (cudaOccupancyMaxActiveClusters(&n, kernel, &cfg) != cudaSuccess || n < 1) { cudaGetLastError(); n = g_num_sms / 2; }
  return n < g_num_sms / 2 ? n : g_num_sms / 2;
}

template <bool SWIGLU>
static cudaError_t launch_pair(const GemmParams& p, int pairs_wanted, cudaStream_t stream) {
  constexpr int smem = PAIR_SMEM;
  static bool configured = false;
  if (!configured) {
    cudaError_t e = cudaFuncSetAttribute(gemm_sm100_pair_kernel<SWIGLU>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
    if (e != cudaSuccess) return e;
    g_max_pairs = resident_pairs(gemm_sm100_pair_kernel<SWIGLU>, smem);
    configured = true;
  }
  const int limit = (g_pair_cap > 0 && g_pair_cap < g_max_pairs) ? g_pair_cap : g_max_pairs;
  const int grid = 2 * (pairs_wanted < limit ? pairs_wanted : limit);
  launch_after(gemm_sm100_pair_kernel<SWIGLU>, grid, GEMM_THREADS, smem, stream, p);
  ++g_launches;
  return cudaGetLastError();
}

// The transposed pair kernel: what it can run at all.
static bool transposed_ok(const MdtGemmDesc* d) {
  const int G = d->G < 1 ? 1 : d->G;
  return (d->mode == 0 || d->mode == 1) && G <= TP_GROUPS && d->a_mn == 0 && (d->K_l == 0 || d->a_mn_l == 0) && !d->c_fp32 && !d->accumulate &&
         d->R == nullptr && d->tile_ready == nullptr && d->row_dest_rank == nullptr && d->b_ready.ready == nullptr && d->b2_ready.ready == nullptr &&
         d->bl_ready.ready == nullptr && d->N > 128 && (!d->dual || (d->b_mn == 0 && (d->K_l == 0 || d->b_mn_l == 0)));
}

// The weight gradient kernel: what it can run at all.
static bool wgrad_ok(const MdtGemmDesc* d) {
  const int G = d->G < 1 ? 1 : d->G;
  return d->mode == 2 && G <= WG_GROUPS && d->a_mn == 1 && d->b_mn == 1 && !d->c_fp32 && d->K_l == 0 && !d->dual && (reinterpret_cast<uintptr_t>(d->C) & 15) == 0 &&
         d->N > 128 && d->M > 128 && (G == 1 || (d->c_group_stride % 8 == 0 && d->c_group_stride >= 0));
}

// Which weight gradients it takes under the default policy: those of up to 12 k blocks, where the result bounds them, and deeper ones
// that are written and that the cluster kernel leaves alone (adding to C costs the ring stages that a deep product needs).
// Microseconds, pair / this kernel, 8 x 14336 x 4096: 576 tokens (3 k blocks) written 353 / 182, added to 533 / 355; 2000 tokens (8)
// 414 / 348, 636 / 490; 4000 tokens (16) 687 / 627, 810 / 835; 12000 tokens 1787 / 1742, 2233 / 2688.  Dense 32000 x 4096 of 576 rows
// 165 / 147, 235 / 183, of 1000 rows 182 / 168, 195 / 214.
static bool wgrad_preferred(const MdtGemmDesc* d, long long thread_rows_hint, int cluster) {
  const int G = d->G < 1 ? 1 : d->G;
  double depth = (double)d->K;
  if (d->offsets != nullptr) {
    double n = (double)d->capacity_rows - 127.0 * G;
    if (thread_rows_hint > 0 && (double)thread_rows_hint < n) n = (double)thread_rows_hint;
    depth = n / G;
  }
  return depth <= 12.0 * BK || (!d->accumulate && cluster == 0);
}

template <bool ACC>
static cudaError_t launch_wgrad(const WgParams& p, cudaStream_t stream) {
  static int max_pairs = 0;
  if (max_pairs == 0) {
    cudaError_t e = cudaFuncSetAttribute(gemm_sm100_wgrad_kernel<ACC>, cudaFuncAttributeMaxDynamicSharedMemorySize, WG_SMEM);
    if (e != cudaSuccess) return e;
    max_pairs = resident_pairs(gemm_sm100_wgrad_kernel<ACC>, WG_SMEM);
  }
  const long long tiles = (long long)p.G * ((p.M + 255) / 256) * ((p.N + 255) / 256);
  const int limit = (g_pair_cap > 0 && g_pair_cap < max_pairs) ? g_pair_cap : max_pairs;
  launch_after(gemm_sm100_wgrad_kernel<ACC>, 2 * (int)(tiles < limit ? tiles : limit), GEMM_THREADS, WG_SMEM, stream, p);
  ++g_launches;
  return cudaGetLastError();
}

// Which row-grouped products it takes under the default policy (those that the cluster kernel would take stay there).
// Measured in turn, microseconds, 128-row or pair kernel / transposed with tiles of up to 256 rows (tp_joint_pays has the larger ones),
// 8 experts of 4096 x 14336:
//   tokens                     77           576          1000         2000         9200
//   gate and up (K-major)      333 / 301    395 / 342    540 / 466    800 / 735    3130 / 3110
//   dy W2^T, SwiGLU (K-major)  208 / 175    253 / 218    330 / 300    530 / 490    1900 / 1860
//   down (MN-major)            146 / 150    176 / 165    275 / 255    430 / 360    1940 / 1900
//   dx, two matrices (MN)      275 / 289    360 / 322    545 / 505    920 / 785    3800 / 3950
// MN-major weights of up to about 96 rows a group stay: 128 x 256 tiles ask for 512 adjacent bytes at a time, one CTA per tile,
// and at one row block a group nothing is gained by exact rows.
// Dense products of more than 128 rows (those that the cluster kernel leaves): where 256-row tiles of tokens would hold an eighth more
// rows than there are in 32-row units, if the tiles give five pairs of eight something to do and, past two rounds, the last round
// wastes no more than a fifth.  us, pair or 128-row kernel / transposed, rows x features x depth: 200 x 32000 x 4096 60 / 60, 300 123 / 71,
// 576 141 / 130, 800 168 / 161, 1300 259 / 249; 576 x 4096 x 4096 34 / 32, x 32000 170 / 155, 1300 284 / 249; 1300 x 4096 x 4096 53 / 50.
// Left: 512 x 4096 x 4096 28 / 34 and 1024 35 / 36 (whole tiles), 300 27 / 30 (32 tiles), 640 x 14336 x 4096 70 / 73 (2.3 rounds).
static bool transposed_preferred_dense(const MdtGemmDesc* d) {
  if (d->dual || d->swiglu_g != nullptr || d->M <= BM) return false;
  const long long pairs = g_num_sms / 2, exact = (d->M + 31) / 32 * 32ll, whole = (d->M + 255) / 256 * 256ll;
  const long long tiles = (whole / 256) * ((d->N + 255) / 256), rounds = (tiles + pairs - 1) / pairs;
  return 8 * whole >= 9 * exact && 8 * tiles >= 5 * pairs && (tiles <= 2 * pairs || 4 * rounds * pairs <= 5 * tiles);
}
static bool transposed_preferred(const MdtGemmDesc* d, long long thread_rows_hint) {
  if (d->mode != 1) return d->mode == 0 && transposed_preferred_dense(d);
  const int G = d->G < 1 ? 1 : d->G;
  long long rows = d->capacity_rows - 127ll * G;
  if (thread_rows_hint > 0 && thread_rows_hint < rows) rows = thread_rows_hint;
  return d->b_mn == 0 || rows > 96ll * G;
}

template <int KIND>
static cudaError_t launch_transposed(const TPParams& p, long long tiles, cudaStream_t stream) {
  static bool configured = false;
  static int max_pairs = 0;
  if (!configured) {
    cudaError_t e = cudaFuncSetAttribute(gemm_sm100_tpair_kernel<KIND>, cudaFuncAttributeMaxDynamicSharedMemorySize, TP_SMEM);
    if (e != cudaSuccess) return e;
    max_pairs = resident_pairs(gemm_sm100_tpair_kernel<KIND>, TP_SMEM);
    configured = true;
  }
  const int limit = (g_pair_cap > 0 && g_pair_cap < max_pairs) ? g_pair_cap : max_pairs;
  const int grid = 2 * (int)(tiles < limit ? tiles : limit);
  launch_after(gemm_sm100_tpair_kernel<KIND>, grid, GEMM_THREADS, TP_SMEM, stream, p);
  ++g_launches;
  return cudaGetLastError();
}

// Expected number of rows of the row-grouped products issued by this thread (0 = unknown); see mdt_gemm_rows_hint.
static thread_local long long t_rows_hint = 0;

// Which kernel takes the 256-wide tiles: 0 = the 128-row kernel always, 1 = the CTA-pair kernel where the shape
// fills 256-row tiles, 2 and 4 = the CTA-pair kernel always (4: an older name of it), 3 = the CTA-pair kernel only where
// 256-row tiles would win by a wide margin, 5 = whichever is faster by the measured models (default; the cluster and the
// transposed pair kernel only here), 6 = the transposed pair kernel wherever it can run.  Initial value from
// MDT_GEMM_PAIR; mdt_gemm_set_pair_policy() changes it.
constexpr int MAX_POLICY = 6;
constexpr int DEFAULT_POLICY = 5;
static int g_pair_policy = -1;
static int pair_policy() {
  if (g_pair_policy < 0) {
    const char* e = getenv("MDT_GEMM_PAIR");
    g_pair_policy = (e != nullptr && e[0] >= '0' && e[0] <= '0' + MAX_POLICY) ? e[0] - '0' : DEFAULT_POLICY;
  }
  return g_pair_policy;
}

// The default rule: rounds x time per round of either kernel, microseconds, as measured on B200.
//   128-row kernel: 0.48 per 64-deep k block and CTA (bound by the 48 KB it brings in) + 1 per tile
//   pair kernel:    0.34 per k block and pair (32 KB per CTA; near the tensor core's 0.27) + 2 per tile
//   a tile takes at least its epilogue: 3.4 / 3.1, and 2.3 more where C is read as well
//   weights arrive at no more than 5.6 TB/s, so below that the two are taken for the same and the smaller tiles stay (not
//   always right: dy W2^T of 576 tokens, 8 experts, 226 us against the pair's 208, with the SwiGLU epilogue 254 / 241)
// E.g. gate/up of 8 experts, 4096 -> 14336: 400 tokens 342 against 387, 800 tokens 467 / 439, 2000 tokens 929 / 846, 9200
// tokens 3058 / 2853; dense 9200 x 4096 x 4096 249 / 183; dense 1152 x 4096 x 4096 (144 or 80 tiles) 40 / 52.
static bool pair_is_faster(const MdtGemmDesc* d, long long thread_rows_hint, int num_sms, int bn_out) {
  const int G = d->G < 1 ? 1 : d->G;
  const double pairs = num_sms / 2;
  double rows = d->mode == 1 ? (double)d->capacity_rows : (double)d->M;
  double depth = (double)d->K;
  if (d->mode == 1) {
    // row groups padded to 128: the capacity leaves 127 rows of padding for each; a hint says what to expect instead
    rows = rows - 127.0 * G > G ? rows - 127.0 * G : G;
    if (thread_rows_hint > 0 && (double)thread_rows_hint < rows) rows = (double)thread_rows_hint;
  }
  if (d->mode == 2 && d->offsets != nullptr) {
    double n = (double)d->capacity_rows;
    if (thread_rows_hint > 0 && (double)thread_rows_hint < n) n = (double)thread_rows_hint;
    depth = n / G;
  }
  const double nb = (double)((d->N + bn_out - 1) / bn_out) * (d->mode == 2 ? G : 1);
  double m1 = ceil(rows / BM), m2 = ceil(rows / (2 * BM));
  if (d->mode == 1) {   // the last block of a group is half full on average
    m1 = fmax(rows / BM + 0.5 * G, (double)G);
    m2 = fmax(rows / (2 * BM) + 0.5 * G, (double)G);
  }
  const double kb = ceil(depth / BK) + ceil((double)d->K_l / BK);
  const double more = d->accumulate ? 2.3 : 0.0;
  const double e1 = m1 * nb / num_sms, e2 = m2 * nb / pairs;
  // rounds: whole ones where the row count is known
  double r1 = d->mode == 1 ? fmax(1.0, e1 + 0.3) : ceil(e1), r2 = d->mode == 1 ? fmax(1.0, e2 + 0.3) : ceil(e2);
  double extra1 = 0.0;
  if (split_enabled() && d->mode != 2 && !d->dual && d->swiglu_g == nullptr && e1 > 1.0 && e1 - floor(e1) < 0.875 && kb >= 8.0) {   // shared last round
    r1 = e1 + (d->mode == 1 ? 0.38 : 0.08);
    extra1 = 15.0;
  }
  const double weights = d->mode == 2 ? 0.0 : (double)d->K * d->N * G * (d->dual ? 4.0 : 2.0) / 5.6e6;
  const double t1 = fmax(r1 * fmax(kb * 0.48 + 1.0, 3.4 + more) + extra1, weights);
  const double t2 = fmax(r2 * fmax(kb * 0.34 + 2.0, 3.1 + more), weights);
  return t2 < 0.97 * t1;
}

// Which kernel runs a product: 0 = 128-row tiles, otherwise the CTA pair (1: policies 1 and 2, 2: policies 3 to 5).
// Pure arithmetic on the descriptor (no CUDA call), so that it can be examined without a GPU.
static int choose_tiling(const MdtGemmDesc* d, int policy, long long thread_rows_hint, int num_sms) {
  const int G = d->G < 1 ? 1 : d->G;
  const int BN = (d->dual || d->N > 128) ? 256 : 128;
  const int bn_out = d->dual ? BN / 2 : BN;
  if (BN != 256) return 0;
  // The CTA-pair kernel needs 256-row pair tiles that are mostly full: dense and depth-grouped products with
  // M >= 256, and row-grouped products whose groups average at least four 128-row blocks.
  const long long rows_hint = (d->mode == 1) ? d->capacity_rows : d->M;
  const bool fills = rows_hint >= 2 * BM && (d->mode != 1 || rows_hint >= (long long)G * 4 * BM);
  if (policy == 2 || (policy == 1 && fills)) return 1;
  if (policy == 4) return 2;
  if (policy == 5) return pair_is_faster(d, thread_rows_hint, num_sms, bn_out) ? 2 : 0;
  if (policy != 3) return 0;
  // Policy 3, for comparisons: a cautious rule that charges 256-row tiles more than the pair kernel takes (0.70 us per k
  // block and an epilogue of 5 us, 14 with SwiGLU, that nothing hides: the costs of a single CTA with 256 rows) and wants
  // 10 % in return; without a row count it takes them for products of >= 2048 rows and >= 3 waves of 128-row tiles only.
  long long r = rows_hint;
  const bool hinted = d->mode == 1 && thread_rows_hint > 0;
  if (hinted && thread_rows_hint < r) r = thread_rows_hint;
  long long grouped_depth = d->capacity_rows;          // mode 2 over row groups: the depth is the group's rows
  if (thread_rows_hint > 0 && thread_rows_hint < grouped_depth) grouped_depth = thread_rows_hint;
  const double blocks = (double)r / BM + (d->mode == 1 ? 0.5 * G : 0.0);
  const double nb = (double)((d->N + bn_out - 1) / bn_out) * (d->mode == 2 ? G : 1);
  const double depth = (d->mode == 2 && d->offsets != nullptr) ? (double)grouped_depth / G : (double)d->K;
  const double kb = ceil(depth / BK) + ceil((double)d->K_l / BK);
  bool wide;
  if (d->mode != 1 || hinted) {
    const double sms = num_sms;
    const double slow_epilogue = (!d->c_fp32 && !d->accumulate) ? 0.0 : 6.0;
    // rounds of 128-row tiles: whole rounds, except that a last round that fills less than 7/8 of the SMs is shared
    // by all of them along the depth (get_work), which costs about its share plus the partial-sum traffic
    double rounds = ceil(ceil(blocks) * nb / sms);
    if (split_enabled() && d->mode != 2 && !d->dual) {
      const double exact = ceil(blocks) * nb / sms, frac = exact - floor(exact);
      if (exact > 1.0 && frac > 0.0 && frac < 0.875 && kb >= 8.0) rounds = exact + 0.08;
    }
    const double t1 = rounds * (fmax(kb * 0.47, 2.0) + 1.0);
    const double t2 = ceil(ceil(blocks / 2 + (d->mode == 1 ? 0.25 * G : 0.0)) * nb / sms) * (kb * 0.70 + 5.0 + (d->dual ? 9.0 : 0.0) + slow_epilogue);
    wide = r >= 2 * BM && kb >= 32.0 && t2 < 0.9 * t1;
  } else {
    wide = r >= 16 * BM && ceil(blocks) * nb >= 3.0 * num_sms && kb >= 32.0;
  }
  return wide ? 2 : 0;
}

// Clusters of S CTAs of the cluster kernel that are resident at once (all its widths take the SM's shared memory).
static int max_clusters(int S) {
  static int cached[MAX_CLUSTER + 1];
  static std::mutex mu;
  std::lock_guard<std::mutex> lock(mu);
  if (cached[S] == 0) {
    cudaLaunchConfig_t cfg;
    memset(&cfg, 0, sizeof(cfg));
    cfg.gridDim = dim3((unsigned)(g_num_sms / S * S)); cfg.blockDim = dim3(GEMM_THREADS); cfg.dynamicSmemBytes = SplitShape<256>::SMEM;
    cudaLaunchAttribute attr;
    attr.id = cudaLaunchAttributeClusterDimension;
    attr.val.clusterDim.x = S; attr.val.clusterDim.y = 1; attr.val.clusterDim.z = 1;
    cfg.attrs = &attr; cfg.numAttrs = 1;
    int n = 0;
    if (cudaFuncSetAttribute(gemm_sm100_cluster_kernel<256>, cudaFuncAttributeMaxDynamicSharedMemorySize, SplitShape<256>::SMEM) != cudaSuccess ||
        cudaOccupancyMaxActiveClusters(&n, gemm_sm100_cluster_kernel<256>, &cfg) != cudaSuccess || n < 1) { cudaGetLastError(); n = g_num_sms / 2 / S; }
    cached[S] = n;
  }
  return cached[S];
}

// Whether a product with few tiles is cut along the depth, and how: cluster size (0 = not) and tile width.  Times in
// microseconds, measured on B200: 0.48 / 0.28 / 0.22 per k block of a 256 / 128 / 64-wide tile, 5 for the exchange of the
// partial tiles; against one CTA per tile (0.28 + 1, 128-wide outputs) or the faster of the two 256-wide kernels in one
// round.  All clusters have to be resident at once (max_clusters: a cluster needs its SMs in one GPC, so 16 clusters of 8
// are more than a B200 holds: 16 tiles 64 deep took 25 us that way, in two rounds, 4 tiles 13).  That counts each product as
// alone on the GPU; the q, k and v projections of a block run at the same time (bindings.cpp) and share it.
// `resident`: clusters of S CTAs that the GPU holds at once.
template <class Resident>
static int choose_cluster(const MdtGemmDesc* d, long long thread_rows_hint, Resident resident, int* bn) {
  if (d->dual || d->swiglu_g != nullptr || d->tile_ready != nullptr || d->row_dest_rank != nullptr || (d->accumulate && d->R != nullptr)) return 0;
  const int G = d->G < 1 ? 1 : d->G;
  *bn = d->N <= 64 ? 64 : (d->N <= 128 ? 128 : 256);
  double rows = (double)d->M, depth = (double)d->K, n = (double)d->capacity_rows - 127.0 * G;
  if (n < G) n = G;
  if (thread_rows_hint > 0 && (double)thread_rows_hint < n) n = (double)thread_rows_hint;
  double blocks = ceil(rows / BM);
  if (d->mode == 1) blocks = fmax(n / BM + 0.5 * G, (double)G);
  if (d->mode == 2 && d->offsets != nullptr) depth = n / G;
  const double tiles = blocks * ((d->N + *bn - 1) / *bn) * (d->mode == 2 ? G : 1);
  const double kb = ceil(depth / BK) + ceil((double)d->K_l / BK);
  const double per = *bn == 256 ? 0.48 : (*bn == 128 ? 0.28 : 0.22);
  const double whole = d->N <= 128 ? kb * 0.28 + 1.0 : fmin(kb * 0.48 + 1.0, kb * 0.34 + 2.0);
  for (int S = MAX_CLUSTER; S >= 2; S /= 2)
    if (kb >= 4.0 * S && tiles <= resident(S)) return ceil(kb / S) * per + 5.0 < whole ? S : 0;
  return 0;
}

template <int BN>
static cudaError_t launch_cluster(const GemmParams& p, int tiles, int S, cudaStream_t stream) {
  static bool configured = false;
  if (!configured) {
    cudaError_t e = cudaFuncSetAttribute(gemm_sm100_cluster_kernel<BN>, cudaFuncAttributeMaxDynamicSharedMemorySize, SplitShape<BN>::SMEM);
    if (e != cudaSuccess) return e;
    configured = true;
  }
  cudaLaunchConfig_t cfg;
  memset(&cfg, 0, sizeof(cfg));
  cfg.gridDim = dim3((unsigned)(tiles * S)); cfg.blockDim = dim3(GEMM_THREADS); cfg.dynamicSmemBytes = SplitShape<BN>::SMEM; cfg.stream = stream;
  cudaLaunchAttribute attr[2];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = S; attr[0].val.clusterDim.y = 1; attr[0].val.clusterDim.z = 1;
  attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;         // (see launch_after)
  attr[1].val.programmaticStreamSerializationAllowed = early_setup_pays(cfg.gridDim.x);
  cfg.attrs = attr; cfg.numAttrs = 2;
  cudaError_t e = cudaLaunchKernelEx(&cfg, gemm_sm100_cluster_kernel<BN>, p);
  ++g_launches;
  return e != cudaSuccess ? e : cudaGetLastError();
}

}  // namespace mdt

extern "C" long long mdt_gemm_launch_count() { return mdt::g_launches; }
extern "C" void mdt_gemm_rows_hint(long long rows) { mdt::t_rows_hint = rows; }
extern "C" int mdt_gemm_max_pairs() { return mdt::g_max_pairs; }
extern "C" int mdt_gemm_choose_tiling(const MdtGemmDesc* d, int policy, long long rows_hint, int num_sms) {
  return mdt::choose_tiling(d, policy, rows_hint, num_sms);
}
extern "C" int mdt_gemm_choose_cluster(const MdtGemmDesc* d, long long rows_hint, int num_sms, int* width) {
  *width = 0;
  return mdt::choose_cluster(d, rows_hint, [num_sms](int S) { return num_sms / S; }, width);
}
extern "C" void mdt_gemm_set_pair_cap(int pairs) { mdt::g_pair_cap = pairs; }
extern "C" int mdt_gemm_set_split(int on) {
  const int old = mdt::split_enabled() ? 1 : 0;
  if (on == 0 || on == 1) mdt::g_split_enabled = on;
  return old;
}
extern "C" int mdt_gemm_set_pair_policy(int policy) {
  const int old = mdt::pair_policy();
  if (policy >= 0 && policy <= mdt::MAX_POLICY) mdt::g_pair_policy = policy;
  return old;
}

namespace mdt {
// The descriptor for the transposed pair kernel (transposed_ok has answered for it).
static int gemm_transposed(const MdtGemmDesc* d, cudaStream_t stream) {
  TPParams p;
  memset(&p, 0, sizeof(p));
  p.M = d->M; p.N = d->N; p.K = d->K; p.K_l = d->K_l; p.G = d->G < 1 ? 1 : d->G; p.mode = d->mode;
  p.w_mn = d->b_mn; p.w_mn_l = d->b_mn_l;
  p.offsets = d->offsets; p.group_rows = d->group_rows;
  p.C = d->C; p.C2 = d->C2; p.C3 = d->C3; p.swiglu_g = d->swiglu_g; p.swiglu_u = d->swiglu_u;
  p.ldc = d->ldc; p.alpha = d->alpha; p.alpha_dev = d->alpha_dev; p.status = d->status;
  const uint32_t w_rows = d->dual ? 16 : (d->b_mn ? 64 : BM), wl_rows = d->dual ? 16 : (d->b_mn_l ? 64 : BM);
  int rc = make_map(&p.tmW, d->B, d->b_cols, d->b_rows, p.G, d->ldb, d->b_group_stride, 64, w_rows, 3);
  if (d->dual) rc |= make_map(&p.tmW2, d->B2, d->b_cols, d->b_rows, p.G, d->ldb, d->b_group_stride, 64, w_rows, 3);
  for (int i = 0; i < 4; ++i) rc |= make_map(&p.tmX[i], d->A, d->a_cols, d->a_rows, 1, d->lda, 0, 64, 16u << i, 2);
  if (d->K_l > 0) {
    rc |= make_map(&p.tmW_l, d->B_l, d->bl_cols, d->bl_rows, p.G, d->ldb_l, d->bl_group_stride, 64, wl_rows, 3);
    if (d->dual) rc |= make_map(&p.tmW2_l, d->B2_l, d->bl_cols, d->bl_rows, p.G, d->ldb_l, d->bl_group_stride, 64, wl_rows, 3);
    for (int i = 0; i < 4; ++i) rc |= make_map(&p.tmX_l[i], d->A_l, d->al_cols, d->al_rows, 1, d->lda_l, 0, 64, 16u << i, 2);
  }
  if (rc != 0) return rc;
  const int width = d->dual ? 128 : 256;
  const long long rows = d->mode == 1 ? d->capacity_rows : d->M;
  const long long tiles = ((rows + 255) / 256 + (d->mode == 1 ? p.G : 0)) * ((p.N + width - 1) / width);       // an upper bound
  const cudaError_t e = d->dual ? launch_transposed<TP_DUAL>(p, tiles, stream)
                      : (d->swiglu_g != nullptr ? launch_transposed<TP_SWIGLU_BWD>(p, tiles, stream) : launch_transposed<TP_PLAIN>(p, tiles, stream));
  return e == cudaSuccess ? 0 : -100 - (int)e;
}
}  // namespace mdt

namespace mdt {
static int gemm_wgrad(const MdtGemmDesc* d, cudaStream_t stream) {
  WgParams p;
  memset(&p, 0, sizeof(p));
  p.M = d->M; p.N = d->N; p.K = d->K; p.G = d->G < 1 ? 1 : d->G;
  p.offsets = d->offsets; p.group_rows = d->group_rows;
  p.alpha = d->alpha; p.alpha_dev = d->alpha_dev; p.status = d->status;
  int rc = make_map(&p.tmA, d->A, d->a_cols, d->a_rows, 1, d->lda, 0, 64, 64, 2);
  rc |= make_map(&p.tmB, d->B, d->b_cols, d->b_rows, 1, d->ldb, 0, 64, 64, 2);
  // (a stride that one matrix does not use still has to be a valid one)
  rc |= make_map(&p.tmC, d->C, d->N, d->M, p.G, d->ldc, p.G > 1 ? d->c_group_stride : d->ldc * (long long)d->M, 64, 32, 3);
  if (rc != 0) return rc;
  const cudaError_t e = d->accumulate ? launch_wgrad<true>(p, stream) : launch_wgrad<false>(p, stream);
  return e == cudaSuccess ? 0 : -100 - (int)e;
}
}  // namespace mdt

namespace mdt {
// The parameter block without its tensor maps; negative: a combination that no kernel takes.
static int fill_params(const MdtGemmDesc* d, GemmParams& p) {
  memset(&p, 0, sizeof(p));
  p.M = d->M; p.N = d->N; p.K = d->K; p.K_l = d->K_l; p.G = d->G < 1 ? 1 : d->G; p.mode = d->mode;
  p.a_mn = d->a_mn; p.b_mn = d->b_mn; p.a_mn_l = d->a_mn_l; p.b_mn_l = d->b_mn_l; p.dual = d->dual;
  p.offsets = d->offsets; p.C = d->C; p.C2 = d->C2; p.C3 = d->C3; p.ldc = d->ldc; p.c_group_stride = d->c_group_stride;
  p.c_fp32 = d->c_fp32; p.accumulate = d->accumulate; p.alpha = d->alpha; p.alpha_dev = d->alpha_dev; p.store_gate_up = d->C2 != nullptr;
  p.status = d->status;
  p.tile_ready = d->tile_ready; p.tile_expected = d->tile_expected;
  p.row_dest_rank = d->row_dest_rank; p.row_dest_row = d->row_dest_row; p.peer_out = d->peer_out; p.peer_arrive = d->peer_arrive;
  p.num_peers = d->num_peers;
  p.peer_wait_ns = mdt_peer_wait_limit_ns();
  p.rdy_b = d->b_ready; p.rdy_b2 = d->b2_ready; p.rdy_bl = d->bl_ready;
  if (p.mode == 2) { p.rdy_b.ready = nullptr; p.rdy_b2.ready = nullptr; p.rdy_bl.ready = nullptr; }
  p.b_rows = d->b_rows; p.ldb = d->ldb; p.b_group_stride = d->b_group_stride;
  p.bl_rows = d->bl_rows; p.ldb_l = d->ldb_l; p.bl_group_stride = d->bl_group_stride;
  p.R = d->R;
  p.swiglu_g = d->swiglu_g; p.swiglu_u = d->swiglu_u;
  if (p.swiglu_g != nullptr && (p.dual || p.mode == 2 || p.c_fp32 || p.accumulate || p.R != nullptr || p.row_dest_rank != nullptr || p.swiglu_u == nullptr || p.C2 == nullptr))
    return -14;
  if (p.R != nullptr && (p.dual || p.mode == 2 || p.row_dest_rank != nullptr || (reinterpret_cast<uintptr_t>(p.R) & 15))) return -13;
  if (p.row_dest_rank != nullptr && (p.dual || p.c_fp32 || p.accumulate || p.mode == 2)) return -12;
  if (p.N % 8 != 0 || p.ldc % 8 != 0) return -10;
  if (p.dual && (p.b_mn != 0 || p.c_fp32 || p.accumulate)) return -11;
  return 0;
}
// Tensor maps; b_rows: rows of a box of a K-major B.
static int fill_maps(const MdtGemmDesc* d, GemmParams& p, int b_rows) {
  int rc = 0;
  // A: [a_rows, a_cols] row-major, a_cols contiguous.  K-major: rows = M, cols = K.  MN-major: rows = depth, cols = M.
  rc |= make_map(&p.tmA, d->A, d->a_cols, d->a_rows, 1, d->lda, 0, 64, d->a_mn ? 64 : BM, 2);
  // B: [G, b_rows, b_cols].  K-major: rows = N, cols = K.  MN-major: rows = depth, cols = N.
  const uint32_t box = d->b_mn ? 64 : b_rows;
  rc |= make_map(&p.tmB, d->B, d->b_cols, d->b_rows, p.mode == 2 ? 1 : p.G, d->ldb, d->b_group_stride, 64, box, 3);
  if (p.dual) rc |= make_map(&p.tmB2, d->B2, d->b_cols, d->b_rows, p.G, d->ldb, d->b_group_stride, 64, box, 3);
  if (p.K_l > 0) {
    rc |= make_map(&p.tmA_l, d->A_l, d->al_cols, d->al_rows, 1, d->lda_l, 0, 64, d->a_mn_l ? 64 : BM, 2);
    const uint32_t box_l = d->b_mn_l ? 64 : b_rows;
    rc |= make_map(&p.tmB_l, d->B_l, d->bl_cols, d->bl_rows, p.G, d->ldb_l, d->bl_group_stride, 64, box_l, 3);
    if (p.dual) rc |= make_map(&p.tmB2_l, d->B2_l, d->bl_cols, d->bl_rows, p.G, d->ldb_l, d->bl_group_stride, 64, box_l, 3);
  }
  return rc;
}
static void prepare_host() {
  // Tensor-map encoding is a driver call: make sure this host thread has the device's primary context
  // bound (a thread that has issued no runtime work yet, e.g. a fresh autograd worker, has none).
  static thread_local bool context_bound = false;
  if (!context_bound) { cudaFree(nullptr); context_bound = true; }
  if (g_num_sms == 0) {
    int dev = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&g_num_sms, cudaDevAttrMultiProcessorCount, dev);
  }
}

// Whether a product may be one of a list: what the cluster kernel computes, with one 64-wide column of tiles in one of its directions.
static bool listable(const MdtGemmDesc* d) {
  return !d->dual && d->swiglu_g == nullptr && d->tile_ready == nullptr && d->row_dest_rank == nullptr && !(d->accumulate && d->R != nullptr) &&
         d->mode != 1 && d->G <= 1 && d->offsets == nullptr && d->N % 8 == 0 && (d->mode == 2 ? (d->M <= BM || d->N <= 64) : d->N <= 64);
}
static int list_tiles(const MdtGemmDesc* d, int n, int bn) {
  int tiles = 0;
  for (int i = 0; i < n; ++i) tiles += ((d[i].M + BM - 1) / BM) * ((d[i].N + bn - 1) / bn);
  return tiles;
}
template <int BN>
static int launch_list(const MdtGemmDesc* d, int n, cudaStream_t stream) {
  ProductList list;
  memset(&list, 0, sizeof(list));
  list.count = n;
  int kb = 0;
  for (int i = 0; i < n; ++i) {
    const int refused = fill_params(d + i, list.p[i]);
    if (refused != 0) return refused;
    const int rc = fill_maps(d + i, list.p[i], BN);
    if (rc != 0) return rc;
    list.tile0[i + 1] = list.tile0[i] + list_tiles(d + i, 1, BN);
    const int k = (d[i].K + BK - 1) / BK + (d[i].K_l + BK - 1) / BK;
    if (k > kb) kb = k;
  }
  const int tiles = list.tile0[n];
  if (tiles == 0) return 0;
  // the depth over as many CTAs as are there at once, four k blocks for each of the deepest product
  int S = MAX_CLUSTER;
  while (S > 1 && (kb < 4 * S || tiles > max_clusters(S))) S /= 2;
  static bool configured = false;
  if (!configured) {
    const cudaError_t e = cudaFuncSetAttribute(gemm_sm100_list_kernel<BN>, cudaFuncAttributeMaxDynamicSharedMemorySize, SplitShape<BN>::SMEM);
    if (e != cudaSuccess) return -100 - (int)e;
    configured = true;
  }
  cudaLaunchConfig_t cfg;
  memset(&cfg, 0, sizeof(cfg));
  cfg.gridDim = dim3((unsigned)(tiles * S)); cfg.blockDim = dim3(GEMM_THREADS); cfg.dynamicSmemBytes = SplitShape<BN>::SMEM; cfg.stream = stream;
  cudaLaunchAttribute attr[2];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = S; attr[0].val.clusterDim.y = 1; attr[0].val.clusterDim.z = 1;
  attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;         // (see launch_after)
  attr[1].val.programmaticStreamSerializationAllowed = early_setup_pays(cfg.gridDim.x);
  cfg.attrs = attr; cfg.numAttrs = 2;
  cudaError_t e = cudaLaunchKernelEx(&cfg, gemm_sm100_list_kernel<BN>, list);
  ++g_launches;
  if (e == cudaSuccess) e = cudaGetLastError();
  return e == cudaSuccess ? 0 : -100 - (int)e;
}
// Tiles as narrow as leaves one round of them: a k block costs 0.22 us of a 64-wide tile and 0.48 of a 256-wide one, a round 5 besides.
// The eight adapter gradients of an attention block (rank 16, 4096 columns, 576 rows) are 352 tiles of 64 columns or 144 of 256:
// 30 and 15 us, one by one 8 of 11 to 15 and the gaps between them.
static int launch_products(const MdtGemmDesc* d, int n, cudaStream_t stream) {
  if (list_tiles(d, n, 64) <= g_num_sms) return launch_list<64>(d, n, stream);
  return list_tiles(d, n, 128) <= g_num_sms ? launch_list<128>(d, n, stream) : launch_list<256>(d, n, stream);
}
}  // namespace mdt

extern "C" int mdt_gemm_list(const MdtGemmDesc* d, int n, cudaStream_t stream) {
  using namespace mdt;
  prepare_host();
  bool together = pair_policy() >= DEFAULT_POLICY && n > 1;
  for (int i = 0; i < n; ++i) together = together && listable(d + i);
  for (int i = 0; i < n; ) {
    const int m = together ? (n - i < MAX_PRODUCTS ? n - i : MAX_PRODUCTS) : 1;
    const int rc = m > 1 ? launch_products(d + i, m, stream) : mdt_gemm(d + i, stream);
    if (rc != 0) return rc;
    i += m;
  }
  return 0;
}

extern "C" int mdt_gemm(const MdtGemmDesc* d, cudaStream_t stream) {
  using namespace mdt;
  prepare_host();
  GemmParams p;
  const int refused = fill_params(d, p);
  if (refused != 0) return refused;
  const int BN = (p.dual || p.N > 128) ? 256 : 128;
  const int bn_out = p.dual ? BN / 2 : BN;
  int cluster_bn = 0;
  const int cluster = pair_policy() == DEFAULT_POLICY ? choose_cluster(d, t_rows_hint, max_clusters, &cluster_bn) : 0;
  if (cluster == 0 && pair_policy() >= DEFAULT_POLICY && transposed_ok(d) && (pair_policy() == MAX_POLICY || transposed_preferred(d, t_rows_hint)))
    return gemm_transposed(d, stream);
  if (pair_policy() >= DEFAULT_POLICY && wgrad_ok(d) && (pair_policy() == MAX_POLICY || wgrad_preferred(d, t_rows_hint, cluster))) return gemm_wgrad(d, stream);
  const bool pair = cluster == 0 && choose_tiling(d, pair_policy(), t_rows_hint, g_num_sms) != 0;
  // (each CTA of a pair loads its half of B in boxes of 128 rows)
  const int rc = fill_maps(d, p, cluster ? cluster_bn : (pair ? 128 : bn_out));
  if (rc != 0) return rc;
  // upper bound on the number of tiles (the exact count may depend on device-side offsets)
  long long rows = (p.mode == 1) ? d->capacity_rows : p.M;
  long long tiles = ((rows + BM - 1) / BM) * ((p.N + bn_out - 1) / bn_out) * (p.mode == 2 ? p.G : 1);
  int grid = (int)(tiles < g_num_sms ? (tiles < 1 ? 1 : tiles) : g_num_sms);
  if (cluster) {
    const int nt = (int)(((rows + BM - 1) / BM) * ((p.N + cluster_bn - 1) / cluster_bn) * (p.mode == 2 ? p.G : 1));
    const cudaError_t e4 = cluster_bn == 256 ? launch_cluster<256>(p, nt, cluster, stream)
                         : (cluster_bn == 128 ? launch_cluster<128>(p, nt, cluster, stream) : launch_cluster<64>(p, nt, cluster, stream));
    return e4 == cudaSuccess ? 0 : -100 - (int)e4;
  }
  if (pair) {
    long long pairs = ((rows + 2 * BM - 1) / (2 * BM) + (p.mode == 1 ? p.G : 0)) * ((p.N + bn_out - 1) / bn_out) * (p.mode == 2 ? p.G : 1);
    const int np = (int)(pairs < 1 ? 1 : (pairs > g_num_sms ? g_num_sms : pairs));
    cudaError_t e2 = p.swiglu_g != nullptr ? launch_pair<true>(p, np, stream) : launch_pair<false>(p, np, stream);
    return e2 == cudaSuccess ? 0 : -100 - (int)e2;
  }
  if (split_enabled() && p.mode != 2 && !p.dual && p.swiglu_g == nullptr) {
    // the last, partly filled round of tiles may be cut along the depth and shared by all SMs (get_work)
    const long long kbt = (p.K + BK - 1) / BK + (p.K_l + BK - 1) / BK;
    SplitWorkspace w;
    if (kbt >= 8 && tiles > g_num_sms && split_workspace(stream, &w)) {
      p.sk_ws = w.ws; p.sk_ctr = w.ctr;
      grid = g_num_sms;
    }
  }
  cudaError_t e;
  if (p.swiglu_g != nullptr) e = (BN == 256) ? launch<256, 4, true>(p, grid, stream) : launch<128, 6, true>(p, grid, stream);
  else e = (BN == 256) ? launch<256, 4, false>(p, grid, stream) : launch<128, 6, false>(p, grid, stream);
  return e == cudaSuccess ? 0 : -100 - (int)e;
}
