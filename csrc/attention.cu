// Causal grouped-query attention over packed variable-length sequences, head_dim 128, on tcgen05.
//
// Forward (attn_fwd_pipelined_kernel): one CTA per (sequence, 128-row query block, query head).  One warp loads key / value
// blocks of 64 rows by TMA and issues the MMAs, four warps do the softmax with one thread per query row; the probabilities
// stay in TMEM, where they are the A operand of P V.  attn_fwd_kernel is the serial form, one 128-row block at a time with P
// through shared memory, for comparisons and for scales that are not positive.
//
// Backward: attn_bwd_prepare_kernel (row statistics, schedule, zeros for rows outside the sequences) and attn_bwd_kernel, whose
// CTAs are of two kinds: dK, dV of a key block and a set of query heads, and dQ of a query block and head.
//
// A [128 x 128] bf16 tile in shared memory is always held as two [128 rows x 128 bytes] swizzled atoms; the same bytes serve
// as a K-major or an MN-major operand, only the descriptor changes, so the transposed products need no data movement.
#include <cuda.h>
#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <math.h>
#include <stdint.h>

#include <stdlib.h>
#include <string.h>

#include <mutex>

#include "api.h"
#include "common/host.h"
#include "common/ptx.cuh"

namespace mdt {

typedef __nv_bfloat16 bf16;
static long long g_att_launches = 0;
constexpr int AB = 128;            // rows per query / key block
constexpr int HD = 128;            // head dimension
constexpr int TILE_BYTES = AB * HD * 2;   // 32 KB
constexpr int ATOM_BYTES = AB * 128;      // 16 KB: [128 rows x 64 bf16]

struct AttnParams {
  CUtensorMap tmQ, tmK, tmV;
  CUtensorMap tmK64, tmV64;                  // key / value maps with 64-row boxes (pipelined forward)
  const int* cu_seqlens;
  int num_seqs, heads_q, heads_kv, tokens;
  float scale_log2e;
  bf16* o; float* lse;
  int* status;
};

// descriptors over the canonical tile form (two swizzled atoms of [128 rows x 128 B])
__device__ __forceinline__ uint64_t desc_kmajor(uint32_t tile, int kstep) {   // depth = the 128 columns
  return make_smem_desc(tile + (kstep >> 2) * ATOM_BYTES + (kstep & 3) * 32, 16, 1024);
}
__device__ __forceinline__ uint64_t desc_mnmajor(uint32_t tile, int kstep) {  // depth = the 128 rows
  return make_smem_desc(tile + kstep * 2048, ATOM_BYTES, 1024);
}
// byte offset of 8 consecutive bf16 (columns c..c+7, c % 8 == 0) of row r inside a canonical tile
__device__ __forceinline__ uint32_t tile_offset(int r, int c) {
  return (c >> 6) * ATOM_BYTES + r * 128 + ((((c & 63) >> 3) ^ (r & 7)) << 4);
}
__device__ __forceinline__ void load_tile(uint8_t* dst, const CUtensorMap* map, uint64_t* bar, int col0, int row0) {
  tma_load_2d(dst, map, bar, col0, row0);
  tma_load_2d(dst + ATOM_BYTES, map, bar, col0 + 64, row0);
}
__device__ __forceinline__ uint32_t pack2(float a, float b) {
  __nv_bfloat162 h = __floats2bfloat162_rn(a, b);
  return *reinterpret_cast<uint32_t*>(&h);
}
// 128-row blocks of a sequence; none if it is empty or reaches outside the tensors' rows
__device__ __forceinline__ int blocks_of(int seq_start, int seq_end, int tokens) {
  return seq_start >= 0 && seq_end > seq_start && seq_end <= tokens ? (seq_end - seq_start + AB - 1) / AB : 0;
}
// Locate block `flat` of the 128-row blocks over all sequences: its sequence (-1: there is no such block, and blk is its number
// past the last one) and its place there.  Called by whole warps: 32 sequences at a time, a scan over their block counts
// (one sequence after the other, each step waiting for its bounds, a CTA of 1024 sequences took 70 us to find its block).
// Grids have at least one block more than the sequences do; the CTA that comes past the last one reports (`status`, optional)
// sequences that were left out because they reach outside the tensors.  1024 sequences of 8 tokens, 32 heads: forward 10.0 ->
// 1.23 ms, backward 11.2 -> 3.2 ms.
__device__ __forceinline__ int find_block(const int* cu, int num_seqs, int tokens, int flat, int& seq_start, int& seq_end, int& blk, int* status) {
  const int lane = threadIdx.x & 31;
  bool outside = false;
  for (int s0 = 0; s0 < num_seqs; s0 += 32) {
    const bool live = s0 + lane < num_seqs;
    const int a = live ? cu[s0 + lane] : 0, b = live ? cu[s0 + lane + 1] : 0;
    const int nb = blocks_of(a, b, tokens);
    outside = outside || (nb == 0 && b > a);
    int upto = nb;                               // blocks of the window's sequences up to this lane's
#pragma unroll
    for (int off = 1; off < 32; off <<= 1) {
      const int v = __shfl_up_sync(0xffffffffu, upto, off);
      if (lane >= off) upto += v;
    }
    const unsigned past = __ballot_sync(0xffffffffu, flat < upto);
    if (past != 0) {
      const int l = __ffs(past) - 1;
      seq_start = __shfl_sync(0xffffffffu, a, l);
      seq_end = __shfl_sync(0xffffffffu, b, l);
      blk = flat - __shfl_sync(0xffffffffu, upto - nb, l);
      return s0 + l;
    }
    flat -= __shfl_sync(0xffffffffu, upto, 31);
  }
  if (__any_sync(0xffffffffu, outside) && threadIdx.x == 0 && status != nullptr) atomicCAS(status, 0, ST_CAPACITY);
  blk = flat;
  return -1;
}

// ------------------------------------------------------------------------------------------- forward
__global__ void __launch_bounds__(128, 1) attn_fwd_kernel(const __grid_constant__ AttnParams p) {
  wait_for_predecessor();
  int seq_start, seq_end, qb;
  if (find_block(p.cu_seqlens, p.num_seqs, p.tokens, blockIdx.x, seq_start, seq_end, qb, p.status) < 0) return;
  const int h = blockIdx.y, kvh = h / (p.heads_q / p.heads_kv);
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  uint8_t* sQ = smem;
  uint8_t* sK = smem + TILE_BYTES;          // two stages
  uint8_t* sV = smem + 3 * TILE_BYTES;      // two stages
  uint8_t* sP = smem + 5 * TILE_BYTES;
  uint64_t* bars = reinterpret_cast<uint64_t*>(smem + 6 * TILE_BYTES);
  uint64_t* barQ = bars; uint64_t* barKV = bars + 1; uint64_t* barS = bars + 3; uint64_t* barO = bars + 4;
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + 5);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);
  const int tid = threadIdx.x, warp = tid >> 5;
  if (tid == 0) {
    mbar_init(barQ, 1); mbar_init(&barKV[0], 1); mbar_init(&barKV[1], 1); mbar_init(barS, 1); mbar_init(barO, 1);
    *abort_flag = 0;
    fence_barrier_init();
  }
  if (warp == 1) { tmem_alloc(tmem_slot, 256); tmem_relinquish(); }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = *tmem_slot;
  admit_successor();              // (not before TMEM is allocated: a product's CTA could take the columns and wait for this kernel)
  const uint32_t t_row = tmem + ((uint32_t)(warp * 32) << 16);   // this warp's lane quarter
  const int q0 = seq_start + qb * AB;
  const int n_kv = qb + 1;
  const uint32_t idesc = make_idesc_bf16(128, 128, 0, 0);
  const uint32_t idesc_pv = make_idesc_bf16(128, 128, 0, 1);
  if (tid == 0) {
    mbar_expect_tx(barQ, TILE_BYTES);
    load_tile(sQ, &p.tmQ, barQ, h * HD, q0);
    mbar_expect_tx(&barKV[0], 2 * TILE_BYTES);
    load_tile(sK, &p.tmK, &barKV[0], kvh * HD, seq_start);
    load_tile(sV, &p.tmV, &barKV[0], kvh * HD, seq_start);
  }
  float o[HD];
#pragma unroll
  for (int i = 0; i < HD; ++i) o[i] = 0.f;
  float m = -INFINITY, l = 0.f;
  const int r = tid;                         // query row inside the block == TMEM lane
  bool ok = true;
  for (int j = 0; j < n_kv && ok; ++j) {
    const int st = j & 1;
    if (tid == 0) {
      if (j + 1 < n_kv) {
        mbar_expect_tx(&barKV[st ^ 1], 2 * TILE_BYTES);
        load_tile(sK + (st ^ 1) * TILE_BYTES, &p.tmK, &barKV[st ^ 1], kvh * HD, seq_start + (j + 1) * AB);
        load_tile(sV + (st ^ 1) * TILE_BYTES, &p.tmV, &barKV[st ^ 1], kvh * HD, seq_start + (j + 1) * AB);
      }
      bool w = (j > 0) || wait_parity(barQ, 0, abort_flag);
      w = w && wait_parity(&barKV[st], (j >> 1) & 1, abort_flag);
      if (w) {
        tc_fence_after();
        const uint32_t a = smem_u32(sQ), b = smem_u32(sK + st * TILE_BYTES);
#pragma unroll
        for (int k = 0; k < 8; ++k) umma_bf16(tmem, desc_kmajor(a, k), desc_kmajor(b, k), idesc, k > 0);
        umma_commit(barS);
      } else {
        *abort_flag = 1;
        if (p.status) atomicCAS(p.status, 0, ST_TIMEOUT_FULL);
      }
    }
    __syncwarp();
    if (!wait_parity_warp(barS, j & 1, abort_flag)) { ok = false; break; }
    tc_fence_after();
    // ---- online softmax on this thread's row (two passes over TMEM: row maximum, then exponentials)
    float mx = m;
    const bool diag = (j == qb);
#pragma unroll
    for (int c = 0; c < 4; ++c) {
      uint32_t raw[32];
      tmem_ld_32x32(t_row + c * 32, raw);
      tmem_ld_wait();
#pragma unroll
      for (int i = 0; i < 32; ++i) {
        if (!(diag && (c * 32 + i) > r)) mx = fmaxf(mx, __uint_as_float(raw[i]) * p.scale_log2e);
      }
    }
    const float alpha = exp2f(m - mx);
    float rs = 0.f;
#pragma unroll
    for (int c = 0; c < 4; ++c) {
      uint32_t raw[32];
      tmem_ld_32x32(t_row + c * 32, raw);
      tmem_ld_wait();
#pragma unroll
      for (int i = 0; i < 32; i += 8) {
        float e[8];
#pragma unroll
        for (int t = 0; t < 8; ++t) {
          const bool masked = diag && (c * 32 + i + t) > r;
          e[t] = masked ? 0.f : exp2f(__uint_as_float(raw[i + t]) * p.scale_log2e - mx);
          rs += e[t];
        }
        uint4 u = make_uint4(pack2(e[0], e[1]), pack2(e[2], e[3]), pack2(e[4], e[5]), pack2(e[6], e[7]));
        *reinterpret_cast<uint4*>(sP + tile_offset(r, c * 32 + i)) = u;
      }
    }
    l = l * alpha + rs;
    m = mx;
    fence_proxy_async();
    tc_fence_before();
    __syncthreads();
    if (tid == 0) {
      tc_fence_after();
      const uint32_t a = smem_u32(sP), b = smem_u32(sV + st * TILE_BYTES);
#pragma unroll
      for (int k = 0; k < 8; ++k) umma_bf16(tmem + 128, desc_kmajor(a, k), desc_mnmajor(b, k), idesc_pv, k > 0);
      umma_commit(barO);
    }
#pragma unroll
    for (int i = 0; i < HD; ++i) o[i] *= alpha;
    __syncwarp();
    if (!wait_parity_warp(barO, j & 1, abort_flag)) { ok = false; break; }
    tc_fence_after();
#pragma unroll
    for (int c = 0; c < 4; ++c) {
      uint32_t raw[32];
      tmem_ld_32x32(t_row + 128 + c * 32, raw);
      tmem_ld_wait();
#pragma unroll
      for (int i = 0; i < 32; ++i) o[c * 32 + i] += __uint_as_float(raw[i]);
    }
    tc_fence_before();
    __syncthreads();
  }
  if (!ok && tid == 0 && p.status) atomicCAS(p.status, 0, ST_TIMEOUT_TMEM_FULL);
  const int row = q0 + r;
  if (ok && row < seq_end) {
    const float inv = 1.f / l;
    bf16* dst = p.o + ((long long)row * p.heads_q + h) * HD;
#pragma unroll
    for (int i = 0; i < HD; i += 8) {
      uint4 u = make_uint4(pack2(o[i] * inv, o[i + 1] * inv), pack2(o[i + 2] * inv, o[i + 3] * inv),
                           pack2(o[i + 4] * inv, o[i + 5] * inv), pack2(o[i + 6] * inv, o[i + 7] * inv));
      *reinterpret_cast<uint4*>(dst + i) = u;
    }
    p.lse[(long long)row * p.heads_q + h] = (m + log2f(l)) * 0.6931471805599453f;
  }
  tc_fence_before();
  __syncthreads();
  if (warp == 1) { tc_fence_after(); tmem_dealloc(tmem, 256); }
}

// ------------------------------------------------------------------------------------------- forward, pipelined
// Warp-specialised forward: warps 0-3 do the softmax (one query row per thread), warp 4 loads (TMA) and issues the
// MMAs.  Keys / values come in blocks of 64 rows; S = Q K^T lives in two 64-column TMEM buffers, so the tensor core
// computes S of block j+1 while the softmax warps work on block j.  The probabilities go back into the first half of
// their S buffer as bf16 and are the A operand of P V from there: through shared memory they cost 16 KB written and 16
// read per block, where the products already take 64 KB per 512 clocks of MMA.  O is accumulated in TMEM by the P V
// products themselves.  The running row maximum used for the exponentials is only raised when the true maximum has grown
// by more than 2^8 (the sum and O are rescaled then, rarely after the first blocks; the final division by the row
// sum makes the result independent of the reference point); only then does the softmax wait for a P V product.  96 KB of
// shared memory and 256 TMEM columns per CTA: two CTAs share an SM, so that one's softmax also overlaps the other's
// products.  The query blocks with the most keys come first in the grid.
//   TMEM columns: [0,64) S / P buffer 0, [64,128) S / P buffer 1, [128,256) O
//   barriers: Q, K[2], V[2] (loaded), S[2] (S ready), P[2] (probabilities stored: S read too), O[2] (P V done: O updated,
//             V tile and P buffer free)
constexpr int FB = 64;                        // key rows per block
constexpr int KV_TILE = FB * HD * 2;          // 16 KB: two atoms of [64 rows x 128 B]
constexpr int KV_ATOM = FB * 128;             // 8 KB
constexpr int FWD2_THREADS = 160;
constexpr int FWD2_SMEM = TILE_BYTES + 4 * KV_TILE + 1024 + 128;
static_assert(2 * (FWD2_SMEM + 1024) <= 228 * 1024, "two CTAs of the pipelined forward must fit one SM");
constexpr float RESCALE_THRESHOLD = 8.0f;     // log2 units

__device__ __forceinline__ void load_kv_tile(uint8_t* dst, const CUtensorMap* map, uint64_t* bar, int col0, int row0) {
  tma_load_2d(dst, map, bar, col0, row0);               // box {64 columns, 64 rows}
  tma_load_2d(dst + KV_ATOM, map, bar, col0 + 64, row0);
}

__global__ void __launch_bounds__(FWD2_THREADS, 2) attn_fwd_pipelined_kernel(const __grid_constant__ AttnParams p) {
  wait_for_predecessor();
  int seq_start, seq_end, qb;
  if (find_block(p.cu_seqlens, p.num_seqs, p.tokens, blockIdx.x / p.heads_q, seq_start, seq_end, qb, p.status) < 0) return;
  qb = (seq_end - seq_start + AB - 1) / AB - 1 - qb;          // last (longest) block of a sequence first
  const int h = blockIdx.x % p.heads_q, kvh = h / (p.heads_q / p.heads_kv);
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  uint8_t* sQ = smem;
  uint8_t* sK = smem + TILE_BYTES;            // two stages
  uint8_t* sV = sK + 2 * KV_TILE;             // two stages
  uint64_t* bars = reinterpret_cast<uint64_t*>(sV + 2 * KV_TILE);
  uint64_t *barQ = bars, *barK = bars + 1, *barV = bars + 3, *barS = bars + 5, *barP = bars + 7, *barO = bars + 9;
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + 11);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  if (tid == 0) {
    mbar_init(barQ, 1);
    for (int i = 0; i < 2; ++i) { mbar_init(&barK[i], 1); mbar_init(&barV[i], 1); mbar_init(&barS[i], 1); mbar_init(&barP[i], 4); mbar_init(&barO[i], 1); }
    *abort_flag = 0;
    fence_barrier_init();
  }
  if (warp == 4) { tmem_alloc(tmem_slot, 256); tmem_relinquish(); }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = *tmem_slot;
  admit_successor();              // (not before TMEM is allocated: a product's CTA could take the columns and wait for this kernel)
  const int q0 = seq_start + qb * AB;
  // key blocks up to the diagonal, and not past the end of the sequence
  const int len = seq_end - seq_start;
  int n_kv = 2 * qb + 2;
  const int n_seq = (len + FB - 1) / FB;
  if (n_kv > n_seq) n_kv = n_seq;
  auto fail = [&](int code) {
    *abort_flag = 1;
    if (p.status != nullptr) atomicCAS(p.status, 0, code);
  };

  if (warp == 4) {
    // ------------------------------------------------------------------ loads and MMA issue
    const uint32_t idesc_s = make_idesc_bf16(128, FB, 0, 0);       // Q (K-major) x K^T (K-major)
    const uint32_t idesc_pv = make_idesc_bf16(128, HD, 0, 1);      // P (TMEM) x V (MN-major)
    const uint32_t aQ = smem_u32(sQ), aK = smem_u32(sK), aV = smem_u32(sV);
    auto load_k = [&](int j) { mbar_expect_tx(&barK[j & 1], KV_TILE); load_kv_tile(sK + (j & 1) * KV_TILE, &p.tmK64, &barK[j & 1], kvh * HD, seq_start + j * FB); };
    auto load_v = [&](int j) { mbar_expect_tx(&barV[j & 1], KV_TILE); load_kv_tile(sV + (j & 1) * KV_TILE, &p.tmV64, &barV[j & 1], kvh * HD, seq_start + j * FB); };
    if (elect_one()) {
      mbar_expect_tx(barQ, TILE_BYTES);
      load_tile(sQ, &p.tmQ, barQ, h * HD, q0);
      load_k(0);
      load_v(0);
      if (n_kv > 1) { load_k(1); load_v(1); }
    }
    bool ok = wait_parity_warp(barQ, 0, abort_flag) && wait_parity_warp(&barK[0], 0, abort_flag);
    if (!ok) fail(ST_TIMEOUT_FULL);
    auto issue_s = [&](int j) {     // S_j = Q K_j^T into buffer j & 1 (P_{j-2} V was issued before: products execute in order)
      tc_fence_after();
      if (elect_one()) {
        const uint32_t k0 = aK + (j & 1) * KV_TILE;
#pragma unroll
        for (int k = 0; k < 8; ++k)
          umma_bf16(tmem + (j & 1) * FB, desc_kmajor(aQ, k), make_smem_desc(k0 + (k >> 2) * KV_ATOM + (k & 3) * 32, 16, 1024), idesc_s, k > 0);
        umma_commit(&barS[j & 1]);
      }
    };
    if (ok) issue_s(0);
    for (int j = 0; j < n_kv && ok; ++j) {
      if (j + 1 < n_kv) {
        ok = wait_parity_warp(&barK[(j + 1) & 1], ((j + 1) >> 1) & 1, abort_flag);
        if (!ok) { fail(ST_TIMEOUT_FULL); break; }
        issue_s(j + 1);
      }
      if (j + 2 < n_kv) {           // K tile j free: S_j done
        ok = wait_parity_warp(&barS[j & 1], (j >> 1) & 1, abort_flag);
        if (!ok) { fail(ST_TIMEOUT_TMEM_FULL); break; }
        if (elect_one()) load_k(j + 2);
      }
      ok = wait_parity_warp(&barP[j & 1], (j >> 1) & 1, abort_flag);
      if (!ok) { fail(ST_TIMEOUT_EMPTY); break; }
      ok = wait_parity_warp(&barV[j & 1], (j >> 1) & 1, abort_flag);
      if (!ok) { fail(ST_TIMEOUT_FULL); break; }
      tc_fence_after();
      if (elect_one()) {
        const uint32_t v0 = aV + (j & 1) * KV_TILE;
#pragma unroll
        for (int k = 0; k < FB / 16; ++k)
          umma_bf16_ta(tmem + 128, tmem + (j & 1) * FB + k * 8, make_smem_desc(v0 + k * 2048, KV_ATOM, 1024), idesc_pv, (j > 0 || k > 0) ? 1u : 0u);
        umma_commit(&barO[j & 1]);
      }
      if (j >= 1 && j + 1 < n_kv) { // V tile j-1 free: its product done (this one is under way)
        ok = wait_parity_warp(&barO[(j - 1) & 1], ((j - 1) >> 1) & 1, abort_flag);
        if (!ok) { fail(ST_TIMEOUT_TMEM_FULL); break; }
        if (elect_one()) load_v(j + 1);
      }
    }
    if (!ok) {   // give copies in flight a bounded time to land before the CTA leaves
      const uint64_t t0 = global_timer_ns();
      while (global_timer_ns() - t0 < 20000ull) {}
    }
  } else {
    // ------------------------------------------------------------------ softmax warps: thread = query row
    const int r = tid;
    const uint32_t t_row = tmem + ((uint32_t)(warp * 32) << 16);
    float m_ref = -INFINITY, l = 0.f;         // reference point (log2 units) and row sum
    bool ok = true;
    for (int j = 0; j < n_kv; ++j) {
      if (!wait_parity_warp(&barS[j & 1], (j >> 1) & 1, abort_flag)) { ok = false; break; }
      // the product two blocks back is long done (S_j came after it); waiting for it keeps barO's phases in step
      if (j >= 2 && !wait_parity_warp(&barO[j & 1], ((j - 2) >> 1) & 1, abort_flag)) { ok = false; break; }
      tc_fence_after();
      uint32_t s0[32], s1[32];
      tmem_ld_32x32(t_row + (j & 1) * FB, s0);
      tmem_ld_32x32(t_row + (j & 1) * FB + 32, s1);
      tmem_ld_wait();
      // causal mask: key column 64j + c is visible to query row 128qb + r iff it is not to the right of it
      const int visible = qb * AB + r - j * FB;         // columns c <= visible are kept
      if (qb * AB - j * FB < FB - 1) {                  // some row of the block sees less than all columns
#pragma unroll
        for (int c = 0; c < 32; ++c) {
          if (c > visible) s0[c] = __float_as_uint(-INFINITY);
          if (c + 32 > visible) s1[c] = __float_as_uint(-INFINITY);
        }
      }
      float mx0 = -INFINITY, mx1 = -INFINITY, mx2 = -INFINITY, mx3 = -INFINITY;
#pragma unroll
      for (int c = 0; c < 32; c += 2) {
        mx0 = fmaxf(mx0, __uint_as_float(s0[c])); mx1 = fmaxf(mx1, __uint_as_float(s0[c + 1]));
        mx2 = fmaxf(mx2, __uint_as_float(s1[c])); mx3 = fmaxf(mx3, __uint_as_float(s1[c + 1]));
      }
      const float mx = fmaxf(fmaxf(mx0, mx1), fmaxf(mx2, mx3)) * p.scale_log2e;
      // raise the reference point only when the maximum has outgrown it by more than the threshold
      const bool raise = mx > m_ref + RESCALE_THRESHOLD;    // (also true for the first visible block: m_ref = -inf)
      if (__any_sync(0xffffffffu, raise)) {
        float alpha = 1.f;
        if (raise) { alpha = (m_ref == -INFINITY) ? 0.f : fast_exp2(m_ref - mx); m_ref = mx; l *= alpha; }
        if (j > 0) {
          if (!wait_parity_warp(&barO[(j - 1) & 1], ((j - 1) >> 1) & 1, abort_flag)) { ok = false; break; }   // O of the blocks so far is complete
          tc_fence_after();
#pragma unroll 1
          for (int c = 0; c < 8; ++c) {
            uint32_t o[16];
            tmem_ld_32x16(t_row + 128 + c * 16, o);
            tmem_ld_wait();
#pragma unroll
            for (int i = 0; i < 16; ++i) o[i] = __float_as_uint(__uint_as_float(o[i]) * alpha);
            tmem_st_32x16(t_row + 128 + c * 16, o);
          }
        }
      }
      // (a row with nothing visible yet has m_ref = -inf: subtract 0 instead, exp2(-inf) = 0)
      const float ref = m_ref == -INFINITY ? 0.f : m_ref;
      float rs0 = 0.f, rs1 = 0.f, rs2 = 0.f, rs3 = 0.f;
      uint32_t pk[32];
#pragma unroll
      for (int c = 0; c < 32; c += 4) {
        const float a = fast_exp2(fmaf(__uint_as_float(s0[c]), p.scale_log2e, -ref)), b = fast_exp2(fmaf(__uint_as_float(s0[c + 1]), p.scale_log2e, -ref));
        const float e = fast_exp2(fmaf(__uint_as_float(s0[c + 2]), p.scale_log2e, -ref)), f = fast_exp2(fmaf(__uint_as_float(s0[c + 3]), p.scale_log2e, -ref));
        rs0 += a; rs1 += b; rs2 += e; rs3 += f;
        pk[c / 2] = pack2(a, b); pk[c / 2 + 1] = pack2(e, f);
      }
#pragma unroll
      for (int c = 0; c < 32; c += 4) {
        const float a = fast_exp2(fmaf(__uint_as_float(s1[c]), p.scale_log2e, -ref)), b = fast_exp2(fmaf(__uint_as_float(s1[c + 1]), p.scale_log2e, -ref));
        const float e = fast_exp2(fmaf(__uint_as_float(s1[c + 2]), p.scale_log2e, -ref)), f = fast_exp2(fmaf(__uint_as_float(s1[c + 3]), p.scale_log2e, -ref));
        rs0 += a; rs1 += b; rs2 += e; rs3 += f;
        pk[16 + c / 2] = pack2(a, b); pk[16 + c / 2 + 1] = pack2(e, f);
      }
      tmem_st_32x32(t_row + (j & 1) * FB, pk);
      tmem_st_wait();
      l += (rs0 + rs1) + (rs2 + rs3);
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(&barP[j & 1]);
    }
    for (int j = n_kv > 1 ? n_kv - 2 : 0; ok && j < n_kv; ++j) ok = wait_parity_warp(&barO[j & 1], (j >> 1) & 1, abort_flag);
    if (!ok && lane == 0) fail(ST_TIMEOUT_TMEM_FULL);
    if (ok) {
      tc_fence_after();
      const int row = q0 + r;
      const bool valid = row < seq_end;
      const float inv = l > 0.f ? 1.f / l : 0.f;
      bf16* dst = p.o + ((long long)row * p.heads_q + h) * HD;
#pragma unroll 1
      for (int c = 0; c < 4; ++c) {
        uint32_t o[32];
        tmem_ld_32x32(t_row + 128 + c * 32, o);
        tmem_ld_wait();
        if (valid) {
#pragma unroll
          for (int i = 0; i < 32; i += 8) {
            uint4 u = make_uint4(pack2(__uint_as_float(o[i]) * inv, __uint_as_float(o[i + 1]) * inv),
                                 pack2(__uint_as_float(o[i + 2]) * inv, __uint_as_float(o[i + 3]) * inv),
                                 pack2(__uint_as_float(o[i + 4]) * inv, __uint_as_float(o[i + 5]) * inv),
                                 pack2(__uint_as_float(o[i + 6]) * inv, __uint_as_float(o[i + 7]) * inv));
            *reinterpret_cast<uint4*>(dst + c * 32 + i) = u;
          }
        }
        __syncwarp();
      }
      if (valid) p.lse[(long long)row * p.heads_q + h] = (m_ref + log2f(l)) * 0.6931471805599453f;
    }
  }
  __syncwarp();
  tc_fence_before();
  __syncthreads();
  if (warp == 4) { tc_fence_after(); tmem_dealloc(tmem, 256); }
}

// ------------------------------------------------------------------------------------------- backward
// Two launches.  `attn_bwd_prepare_kernel` computes, per (128-row block, query head), delta = rowsum(o * do) and the row statistics in
// log2 units, ranks the blocks by the work they mean as key blocks, and clears the gradients of rows outside the sequences.
// `attn_bwd_kernel` holds two kinds of CTAs, most work first within each kind:
//   dK, dV: one per (key block, HPC query heads of one kv head); its loop runs over the query blocks at or below the diagonal
//   dQ:     one per (query block, head); its loop runs over the key blocks up to the diagonal
// Each forms S and dP for itself, 7 products a 128 x 128 block instead of the 5 of a kernel that also adds dQ up from its key
// blocks.  Those additions were what bounded it: 64 KB of fp32 reductions into L2 a block (25 % of its loop), dQ's place in TMEM that held
// up the next block's dP, and a buffer of 128 floats a token and head to be cleared and converted.  Without them nothing leaves TMEM
// but the results: P^T and dS^T (dK, dV) and dS (dQ) are operands of their products from there.
// Whole calls, 32 / 8 heads, us, with dQ by reductions -> so: 77 tokens 33.8 -> 21.5, 613 62.5 -> 48.1, 2048 207.9 -> 187.4, 8192
// 1716 -> 1578, 16384 6741 -> 6720 (8192: dK, dV of all blocks about 0.56 of it, dQ 0.44).  What bounds it is the chain of a CTA, scores ->
// exponentials -> product, with one CTA an SM (its operands fill shared memory and its accumulators TMEM) and half a block to overlap with.
// dS = P (scale dP - scale delta) has its factor before it is rounded (it is no power of two: on the sums it would put every rounding
// elsewhere), in the statistics and a fused multiply-add; a multiplication of its own took 3 % at 8192 tokens.
// Slower at 8192 (of 1543 then): 16 softmax warps (2379, they spill), two blocks in flight through halves of TMEM (1581), one wait for scores and
// statistics together (1912), a share of the exponentials on the fp32 units (1604 with a quarter, 1688 with half).
//
// dK, dV keep keys as rows (TMEM lanes): S^T = K Q^T, P^T = exp2(S^T - lse) over S^T, dV += P^T dO, dS^T over dP^T = V dO^T, dK += dS^T Q.
// 4 products of 512 clocks a block, 1024 clocks of exponentials; while the softmax warps form dS_i the tensor core works on dV_i and
// S_{i+1}, while they form P_{i+1} on dK_i and dP_{i+1}.   TMEM columns: [0,128) S^T / P^T, [128,256) dP^T / dS^T, dV, dK
// dQ keeps queries as rows: S = Q K^T in two buffers, dP = dO V^T, dS over dP, dQ += dS K; 3 products.   TMEM: S, S, dP / dS, dQ
// (P^T and dS^T are stored by two warps for half of the columns each: the first 32 columns of each half's 64.)
// Warps 0-7 softmax (warp -> 32 rows, 64 columns), 8 TMA, 9 MMA issue.
// Where the query heads of a kv head are spread over several CTAs these form a cluster, which adds their dK, dV in the order of the
// ranks through distributed shared memory; all results are the same in every run.
constexpr int BWD_THREADS = 320;
constexpr int BWD_STATS = 2 * AB;                              // lse2 | scale * delta of a block, floats
constexpr int BWD_SMEM = 7 * TILE_BYTES + 2 * BWD_STATS * 4 + 256 + 768;   // (768: what alignment to 1024 may take)
constexpr int MAX_SETS = 8;                                    // CTAs that share a kv head's query heads: a cluster
static_assert(BWD_SMEM <= 227 * 1024, "attention backward: shared memory of a CTA");

struct AttnBwdParams {
  CUtensorMap tmQ, tmK, tmV, tmdO;
  const int4* sched;            // by rank: {seq_start, seq_end, block, flat block}; seq_start < 0: none
  const float* stats;           // [flat block][head][lse2 x 128 | scale * delta x 128]
  bf16* dq; bf16* dk; bf16* dv;
  int heads_q, heads_kv, hpc;   // hpc: query heads per dK, dV CTA
  int tokens, blocks;           // rows of the tensors; entries of the schedule
  float scale_log2e, scale;
  int* status;
};

__global__ void __launch_bounds__(256, 2) attn_bwd_prepare_kernel(const bf16* __restrict__ o, const bf16* __restrict__ dout, const float* __restrict__ lse,
                                                               const int* __restrict__ cu, int num_seqs, int tokens, int heads, int heads_kv, float scale, int4* __restrict__ sched,
                                                               float* __restrict__ stats, bf16* __restrict__ dq, bf16* __restrict__ dk, bf16* __restrict__ dv, int* status) {
  after_predecessor();
  int seq_start, seq_end, blk;
  const int flat = blockIdx.x, h = blockIdx.y;
  const int seq = find_block(cu, num_seqs, tokens, flat, seq_start, seq_end, blk, status);
  if (seq < 0) {
    if (h == 0 && threadIdx.x == 0) sched[flat] = make_int4(-1, 0, 0, 0);
    // rows before the first and after the last sequence: zeros, from the CTAs that have no block
    const int first = num_seqs > 0 ? min(max(cu[0], 0), tokens) : 0, end = num_seqs > 0 ? min(max(cu[num_seqs], first), tokens) : 0;
    const int idle = (int)gridDim.x - (flat - blk), sub = threadIdx.x & 15;            // CTAs like this one, per head
    const uint4 zero = make_uint4(0, 0, 0, 0);
    for (int u = blk * 16 + (threadIdx.x >> 4); u < first + tokens - end; u += idle * 16) {
      const long long row = u < first ? u : end + (u - first);
      reinterpret_cast<uint4*>(dq + (row * heads + h) * HD)[sub] = zero;
      if (h < heads_kv) {
        reinterpret_cast<uint4*>(dk + (row * heads_kv + h) * HD)[sub] = zero;
        reinterpret_cast<uint4*>(dv + (row * heads_kv + h) * HD)[sub] = zero;
      }
    }
    return;
  }
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  if (h == 0 && warp == 0) {
    // rank by the number of query blocks that a key block meets, most first
    const int n = blocks_of(seq_start, seq_end, tokens) - blk;
    int rank = 0;
    for (int s = lane; s < num_seqs; s += 32) {
      const int nb = blocks_of(cu[s], cu[s + 1], tokens);
      rank += (nb > n ? nb - n : 0) + (s < seq && nb >= n ? 1 : 0);
    }
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) rank += __shfl_xor_sync(0xffffffffu, rank, off);
    // (sequences that overlap may have more blocks than the schedule has entries)
    if (lane == 0 && rank < (int)gridDim.x) sched[rank] = make_int4(seq_start, seq_end, blk, flat);
  }
  const long long tile = (long long)flat * heads + h;
  // 16 lanes x 16 bytes hold a row, 16 rows per pass; all loads of the block are in flight at once
  const int sub = lane & 15, r0 = warp * 2 + (lane >> 4);
  const int row0 = seq_start + blk * AB, rows = min(AB, seq_end - row0);
  uint4 a[8], b[8];
#pragma unroll
  for (int k = 0; k < 8; ++k) {
    const int r = k * 16 + r0;
    const long long at = ((long long)(row0 + (r < rows ? r : 0)) * heads + h) * HD;     // (past the end: one row again and again)
    a[k] = reinterpret_cast<const uint4*>(o + at)[sub];
    b[k] = reinterpret_cast<const uint4*>(dout + at)[sub];
  }
  float* st = stats + tile * BWD_STATS;
#pragma unroll
  for (int k = 0; k < 8; ++k) {
    const int r = k * 16 + r0;
    const long long row = row0 + r;
    const bool valid = r < rows;
    const __nv_bfloat162* pa = reinterpret_cast<const __nv_bfloat162*>(&a[k]);
    const __nv_bfloat162* pb = reinterpret_cast<const __nv_bfloat162*>(&b[k]);
    float s = 0.f;
#pragma unroll
    for (int i = 0; i < 4; ++i) { const float2 x = __bfloat1622float2(pa[i]), y = __bfloat1622float2(pb[i]); s += x.x * y.x + x.y * y.y; }
#pragma unroll
    for (int off = 8; off > 0; off >>= 1) s += __shfl_xor_sync(0xffffffffu, s, off);
    if (sub == 0) { st[r] = valid ? lse[row * heads + h] * 1.4426950408889634f : 0.f; st[AB + r] = valid ? s * scale : 0.f; }
  }
}

__device__ __forceinline__ uint4 pack8(const uint32_t* a) {
  return make_uint4(pack2(__uint_as_float(a[0]), __uint_as_float(a[1])), pack2(__uint_as_float(a[2]), __uint_as_float(a[3])),
                    pack2(__uint_as_float(a[4]), __uint_as_float(a[5])), pack2(__uint_as_float(a[6]), __uint_as_float(a[7])));
}

__global__ void __launch_bounds__(BWD_THREADS, 1) attn_bwd_kernel(const __grid_constant__ AttnBwdParams p) {
  wait_for_predecessor();
  const int sets = p.heads_q / p.hpc, per = sets / p.heads_kv;     // head sets; of one kv head: a cluster of the dK, dV CTAs
  const int kv_ctas = p.blocks * sets;
  const bool is_dq = (int)blockIdx.x >= kv_ctas;
  const int unit = is_dq ? (int)blockIdx.x - kv_ctas : (int)blockIdx.x, width = is_dq ? p.heads_q : sets;   // the sets / heads of a block are neighbours
  const int4 work = p.sched[unit / width];
  const int seq_start = work.x, seq_end = work.y, kb = work.z;
  if (seq_start < 0) return;
  const int nb = blocks_of(seq_start, seq_end, p.tokens);
  // an entry of sequences that overlap, or one that nobody wrote for them: what it leads to has to exist
  if (kb < 0 || kb >= nb || work.w - kb < 0 || work.w + nb - kb > p.blocks) {
    if (threadIdx.x == 0 && p.status != nullptr) atomicCAS(p.status, 0, ST_CAPACITY);
    return;
  }
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  if (smem + BWD_SMEM - 768 > smem_raw + BWD_SMEM) {       // uniform; never seen: dynamic shared memory starts 1024-aligned
    if (threadIdx.x == 0 && p.status != nullptr) atomicCAS(p.status, 0, ST_CAPACITY);
    return;
  }
  float* sStats = reinterpret_cast<float*>(smem + 7 * TILE_BYTES);
  uint64_t* bars = reinterpret_cast<uint64_t*>(smem + 7 * TILE_BYTES + 2 * BWD_STATS * 4);
  // fixed operands | streamed ones, three stages of X and two of Y: loaded, free | row statistics loaded | S, P (by columns), dP, dS | all products done
  uint64_t *barFix = bars, *barX = bars + 1, *barXfree = bars + 4, *barY = bars + 7, *barYfree = bars + 9, *barT = bars + 11, *barS = bars + 13, *barP = bars + 15,
           *bardP = bars + 17, *bardS = bars + 18, *barDone = bars + 19;
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + 20);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  if (tid == 0) {
    mbar_init(barFix, 1); mbar_init(bardP, 1); mbar_init(bardS, 8); mbar_init(barDone, 1);
    for (int i = 0; i < 3; ++i) { mbar_init(&barX[i], 1); mbar_init(&barXfree[i], 1); }
    for (int i = 0; i < 2; ++i) { mbar_init(&barY[i], 1); mbar_init(&barYfree[i], 1); mbar_init(&barT[i], 1); mbar_init(&barS[i], 1); mbar_init(&barP[i], 8); }
    *abort_flag = 0;
    fence_barrier_init();
  }
  if (warp == 9) { tmem_alloc(tmem_slot, 512); tmem_relinquish(); }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = *tmem_slot;
  admit_successor();              // (not before TMEM is allocated: a product's CTA could take the columns and wait for this kernel)
  auto fail = [&](int code) {
    *abort_flag = 1;
    if (p.status != nullptr) atomicCAS(p.status, 0, code);
  };
  const int half = warp >> 2, r = (warp & 3) * 32 + lane;         // softmax warps: 64 columns, row
  const uint32_t t_lane = (uint32_t)((warp & 3) * 32) << 16;
  const uint32_t id_kk = make_idesc_bf16(128, 128, 0, 0), id_km = make_idesc_bf16(128, 128, 0, 1);
  // fixed: K, V or Q, dO; streamed: X = Q or K, Y = dO or V
  uint8_t *sF0 = smem, *sF1 = smem + TILE_BYTES, *sX = smem + 2 * TILE_BYTES, *sY = smem + 5 * TILE_BYTES;
  const uint32_t aF0 = smem_u32(sF0), aF1 = smem_u32(sF1), aX = smem_u32(sX), aY = smem_u32(sY);

  if (!is_dq) {
    // ================================================================== dK, dV of a key block
    const int set = unit % width, h0 = set * p.hpc, kvh = h0 / (p.heads_q / p.heads_kv);
    const int k0 = seq_start + kb * AB, nq = nb - kb, n_it = nq * p.hpc;
    const uint32_t tS = tmem, tdP = tmem + 128, tdV = tmem + 256, tdK = tmem + 384;
    if (warp == 8) {
      // ---------------------------------------------------------------- loads
      bool ok = true;
      if (elect_one()) {
        mbar_expect_tx(barFix, 2 * TILE_BYTES);
        load_tile(sF0, &p.tmK, barFix, kvh * HD, k0);
        load_tile(sF1, &p.tmV, barFix, kvh * HD, k0);
      }
      // (the statistics of a block go into one of two places, free once dK of two blocks ago is done: they come one block behind X)
      auto load_stats = [&](int it, int h, int i) {
        mbar_expect_tx(&barT[it & 1], BWD_STATS * 4);
        bulk_load(sStats + (it & 1) * BWD_STATS, p.stats + ((long long)(work.w + i) * p.heads_q + h) * BWD_STATS, BWD_STATS * 4, &barT[it & 1]);
      };
      int head = 0, i = 0, h_last = h0, i_last = 0;
      for (int it = 0; it < n_it; ++it) {
        const int h = h0 + head, q0 = seq_start + (kb + i) * AB;
        ok = wait_parity_warp(&barXfree[it % 3], (it / 3 & 1) ^ 1, abort_flag);
        if (!ok) { fail(ST_TIMEOUT_EMPTY); break; }
        if (elect_one()) {
          mbar_expect_tx(&barX[it % 3], TILE_BYTES);
          load_tile(sX + it % 3 * TILE_BYTES, &p.tmQ, &barX[it % 3], h * HD, q0);
          if (it > 0) load_stats(it - 1, h_last, i_last);
          if (it == n_it - 1 && it < 2) load_stats(it, h, i);
        }
        h_last = h; i_last = i;
        ok = wait_parity_warp(&barYfree[it & 1], ((it >> 1) & 1) ^ 1, abort_flag);
        if (!ok) { fail(ST_TIMEOUT_EMPTY); break; }
        if (elect_one()) {
          mbar_expect_tx(&barY[it & 1], TILE_BYTES);
          load_tile(sY + (it & 1) * TILE_BYTES, &p.tmdO, &barY[it & 1], h * HD, q0);
        }
        if (++i == nq) { i = 0; ++head; }
      }
      if (ok && n_it > 2) {
        ok = wait_parity_warp(&barXfree[n_it % 3], (n_it / 3 & 1) ^ 1, abort_flag);
        if (!ok) fail(ST_TIMEOUT_EMPTY);
        else if (elect_one()) load_stats(n_it - 1, h_last, i_last);
      }
      if (!ok) {   // give copies in flight a bounded time to land before the CTA leaves
        const uint64_t t0 = global_timer_ns();
        while (global_timer_ns() - t0 < 20000ull) {}
      }
    } else if (warp == 9) {
      // ---------------------------------------------------------------- MMA issue (products execute in the order of issue)
      auto issue_s = [&](int it) {      // S^T = K Q^T
        tc_fence_after();
        if (elect_one()) {
#pragma unroll
          for (int s = 0; s < 8; ++s) umma_bf16(tS, desc_kmajor(aF0, s), desc_kmajor(aX + it % 3 * TILE_BYTES, s), id_kk, s > 0);
          umma_commit(barS);
        }
      };
      auto issue_dp = [&](int it) {     // dP^T = V dO^T
        tc_fence_after();
        if (elect_one()) {
#pragma unroll
          for (int s = 0; s < 8; ++s) umma_bf16(tdP, desc_kmajor(aF1, s), desc_kmajor(aY + (it & 1) * TILE_BYTES, s), id_kk, s > 0);
          umma_commit(bardP);
        }
      };
      bool ok = wait_parity_warp(barFix, 0, abort_flag) && wait_parity_warp(&barX[0], 0, abort_flag);
      if (ok) { issue_s(0); ok = wait_parity_warp(&barY[0], 0, abort_flag); }
      if (ok) issue_dp(0);
      for (int it = 0; it < n_it && ok; ++it) {
        const int st = it & 1;
        for (int c = 0; c < 2 && ok; ++c) {     // dV += P^T dO: the first 32 columns of both halves while the others are formed
          ok = wait_parity_warp(&barP[c], it & 1, abort_flag);
          if (!ok) break;
          tc_fence_after();
          if (elect_one()) {
#pragma unroll
            for (int x = 0; x < 4; ++x) {
              const int s = (x >> 1) * 4 + c * 2 + (x & 1);
              umma_bf16_ta(tdV, tS + (s >> 2) * 64 + (s & 3) * 8, desc_mnmajor(aY + st * TILE_BYTES, s), id_km, it > 0 || c > 0 || x > 0);
            }
            if (c == 1) umma_commit(&barYfree[st]);
          }
        }
        if (!ok) break;
        if (it + 1 < n_it) {            // over P^T
          ok = wait_parity_warp(&barX[(it + 1) % 3], (it + 1) / 3 & 1, abort_flag);
          if (!ok) break;
          issue_s(it + 1);
        }
        ok = wait_parity_warp(bardS, it & 1, abort_flag);
        if (!ok) break;
        tc_fence_after();
        if (elect_one()) {              // dK += dS^T Q
#pragma unroll
          for (int s = 0; s < 8; ++s) umma_bf16_ta(tdK, tdP + (s >> 2) * 64 + (s & 3) * 8, desc_mnmajor(aX + it % 3 * TILE_BYTES, s), id_km, it > 0 || s > 0);
          umma_commit(&barXfree[it % 3]);
        }
        if (it + 1 < n_it) {            // over dS^T
          ok = wait_parity_warp(&barY[st ^ 1], ((it + 1) >> 1) & 1, abort_flag);
          if (!ok) break;
          issue_dp(it + 1);
        }
      }
      if (ok) { if (elect_one()) umma_commit(barDone); }
      else fail(ST_TIMEOUT_FULL);
    } else {
      // ---------------------------------------------------------------- softmax (lane = key row, 64 query columns)
      const uint32_t t_row = tmem + half * 64 + t_lane;
      const bool k_valid = k0 + r < seq_end;
      bool ok = true;
      int i = 0;
      for (int it = 0; it < n_it; ++it) {
        const int st = it & 1;
        const int q0 = seq_start + (kb + i) * AB;
        const float* lse2 = sStats + st * BWD_STATS + half * 64;
        const float* delta = lse2 + AB;
        // block on the diagonal or last query block: elements are masked one by one (rows past the sequence are not stored)
        const bool masked = i == 0 || q0 + AB > seq_end;
        auto hidden = [&](int c) {       // query column half * 64 + c
          const int q = half * 64 + c;
          return (i == 0 && q < r) || q0 + q >= seq_end;
        };
        // (statistics come into registers before the waits: between the tensor core's reads of its operands a load from shared
        // memory takes long, and 64 of them one by one made the loop a third longer)
        if (!wait_parity_warp(&barT[st], (it >> 1) & 1, abort_flag)) { ok = false; break; }
        float pr[64];
#pragma unroll
        for (int x = 0; x < 64; x += 4) {
          const float4 l = *reinterpret_cast<const float4*>(lse2 + x);
          pr[x] = l.x; pr[x + 1] = l.y; pr[x + 2] = l.z; pr[x + 3] = l.w;
        }
        if (!wait_parity_warp(barS, it & 1, abort_flag)) { ok = false; break; }
        tc_fence_after();
        {
          uint32_t s[2][32];
          tmem_ld_32x32(t_row, s[0]);
          tmem_ld_32x32(t_row + 32, s[1]);
          tmem_ld_wait();
#pragma unroll
          for (int c = 0; c < 2; ++c) {
            uint32_t pk[16];
#pragma unroll
            for (int x = 0; x < 32; ++x) {
              float& v = pr[c * 32 + x];
              v = fast_exp2(fmaf(__uint_as_float(s[c][x]), p.scale_log2e, -v));
            }
            if (masked) {
#pragma unroll
              for (int x = 0; x < 32; ++x) if (hidden(c * 32 + x)) pr[c * 32 + x] = 0.f;
            }
#pragma unroll
            for (int x = 0; x < 16; ++x) pk[x] = pack2(pr[c * 32 + 2 * x], pr[c * 32 + 2 * x + 1]);
            tmem_st_32x16(t_row + c * 16, pk);      // over this warp's own part of S^T
            tmem_st_wait();
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(&barP[c]);
          }
        }
        float dl[32];
#pragma unroll
        for (int x = 0; x < 32; x += 4) {
          const float4 v = *reinterpret_cast<const float4*>(delta + x);
          dl[x] = v.x; dl[x + 1] = v.y; dl[x + 2] = v.z; dl[x + 3] = v.w;
        }
        if (!wait_parity_warp(bardP, it & 1, abort_flag)) { ok = false; break; }
        tc_fence_after();
        uint32_t pk[32];                 // dS^T with the factor `scale`, then rounded once
#pragma unroll
        for (int c = 0; c < 64; c += 32) {
          uint32_t d[32];
          tmem_ld_32x32(t_row + 128 + c, d);
          tmem_ld_wait();
#pragma unroll
          for (int x = 0; x < 32; ++x) d[x] = __float_as_uint(pr[c + x] * fmaf(__uint_as_float(d[x]), p.scale, -dl[x]));
          if (masked) {                  // (a branch of its own: tests between the products cost 900 clocks a block)
#pragma unroll
            for (int x = 0; x < 32; ++x) if (hidden(c + x)) d[x] = 0u;
          }
#pragma unroll
          for (int x = 0; x < 16; ++x) pk[c / 2 + x] = pack2(__uint_as_float(d[2 * x]), __uint_as_float(d[2 * x + 1]));
          if (c == 0) {
#pragma unroll
            for (int x = 0; x < 32; x += 4) {
              const float4 v = *reinterpret_cast<const float4*>(delta + 32 + x);
              dl[x] = v.x; dl[x + 1] = v.y; dl[x + 2] = v.z; dl[x + 3] = v.w;
            }
          }
        }
        tmem_st_32x32(t_row + 128, pk);  // over this warp's own part of dP^T
        tmem_st_wait();
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(bardS);
        if (++i == nq) i = 0;
      }
      ok = ok && wait_parity_warp(barDone, 0, abort_flag);
      if (!ok) { if (lane == 0) fail(ST_TIMEOUT_TMEM_FULL); }
      else {
        // warps 0-3 write dV, warps 4-7 dK
        tc_fence_after();
        const uint32_t acc = tmem + 256 + half * 128 + t_lane;
        bf16* out = (half == 0 ? p.dv : p.dk) + ((long long)(k0 + r) * p.heads_kv + kvh) * HD;
        float4* part = reinterpret_cast<float4*>(smem + half * 2 * TILE_BYTES) + r;      // [column / 4][row], over the operands
#pragma unroll 1
        for (int c = 0; c < HD; c += 32) {
          uint32_t a[32];
          tmem_ld_32x32(acc + c, a);
          tmem_ld_wait();
          if (per > 1) {
#pragma unroll
            for (int x = 0; x < 32; x += 4)
              part[(c + x) / 4 * AB] = make_float4(__uint_as_float(a[x]), __uint_as_float(a[x + 1]), __uint_as_float(a[x + 2]), __uint_as_float(a[x + 3]));
          } else if (k_valid) {
#pragma unroll
            for (int x = 0; x < 32; x += 8) *reinterpret_cast<uint4*>(out + c + x) = pack8(a + x);
          }
          __syncwarp();
        }
      }
    }
    if (per > 1) {
      // add up the cluster's partial tiles, an equal share of dV | dK by each CTA
      cluster_sync_all();
      const int rank = (int)cluster_ctarank();
      constexpr int UNITS = 2 * AB * (HD / 8);                    // eight columns of a row; rows fastest
      const uint32_t base = smem_u32(smem);
      for (int u = UNITS * rank / per + tid; u < UNITS * (rank + 1) / per; u += BWD_THREADS) {
        const int row = u % AB, g8 = u / AB % (HD / 8), mat = u / (AB * (HD / 8));
        if (k0 + row >= seq_end) continue;
        float s[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
        const uint32_t at = base + mat * 2 * TILE_BYTES + (2 * g8 * AB + row) * 16;
        for (int c = 0; c < per; ++c) {
          const uint32_t a = mapa_shared(at, c);
          const float4 x = ld_cluster_v4(a), y = ld_cluster_v4(a + AB * 16);
          s[0] += x.x; s[1] += x.y; s[2] += x.z; s[3] += x.w; s[4] += y.x; s[5] += y.y; s[6] += y.z; s[7] += y.w;
        }
        *reinterpret_cast<uint4*>((mat == 0 ? p.dv : p.dk) + ((long long)(k0 + row) * p.heads_kv + kvh) * HD + g8 * 8) =
            make_uint4(pack2(s[0], s[1]), pack2(s[2], s[3]), pack2(s[4], s[5]), pack2(s[6], s[7]));
      }
      cluster_sync_all();                                         // nobody leaves while its tiles are read
    }
  } else {
    // ================================================================== dQ of a query block: as many key blocks as its mirror image has query blocks
    const int h = unit % width, kvh = h / (p.heads_q / p.heads_kv);
    const int qb = nb - 1 - kb, q0 = seq_start + qb * AB, n = qb + 1;
    const uint32_t tdP = tmem + 256, tdQ = tmem + 384;
    if (warp == 8) {
      // ---------------------------------------------------------------- loads
      bool ok = true;
      if (elect_one()) {
        mbar_expect_tx(barFix, 2 * TILE_BYTES);
        load_tile(sF0, &p.tmQ, barFix, h * HD, q0);
        load_tile(sF1, &p.tmdO, barFix, h * HD, q0);
      }
      for (int j = 0; j < n; ++j) {
        const int st = j & 1, sx = j % 3;
        ok = wait_parity_warp(&barXfree[sx], (j / 3 & 1) ^ 1, abort_flag);
        if (!ok) { fail(ST_TIMEOUT_EMPTY); break; }
        if (elect_one()) { mbar_expect_tx(&barX[sx], TILE_BYTES); load_tile(sX + sx * TILE_BYTES, &p.tmK, &barX[sx], kvh * HD, seq_start + j * AB); }
        ok = wait_parity_warp(&barYfree[st], ((j >> 1) & 1) ^ 1, abort_flag);
        if (!ok) { fail(ST_TIMEOUT_EMPTY); break; }
        if (elect_one()) { mbar_expect_tx(&barY[st], TILE_BYTES); load_tile(sY + st * TILE_BYTES, &p.tmV, &barY[st], kvh * HD, seq_start + j * AB); }
      }
      if (!ok) {   // give copies in flight a bounded time to land before the CTA leaves
        const uint64_t t0 = global_timer_ns();
        while (global_timer_ns() - t0 < 20000ull) {}
      }
    } else if (warp == 9) {
      // ---------------------------------------------------------------- MMA issue
      auto issue_s = [&](int j) {       // S = Q K^T (the buffer's scores of two blocks ago were read before dS of that block came)
        tc_fence_after();
        if (elect_one()) {
#pragma unroll
          for (int s = 0; s < 8; ++s) umma_bf16(tmem + (j & 1) * 128, desc_kmajor(aF0, s), desc_kmajor(aX + j % 3 * TILE_BYTES, s), id_kk, s > 0);
          umma_commit(&barS[j & 1]);
        }
      };
      auto issue_dp = [&](int j) {      // dP = dO V^T
        tc_fence_after();
        if (elect_one()) {
#pragma unroll
          for (int s = 0; s < 8; ++s) umma_bf16(tdP, desc_kmajor(aF1, s), desc_kmajor(aY + (j & 1) * TILE_BYTES, s), id_kk, s > 0);
          umma_commit(bardP);
          umma_commit(&barYfree[j & 1]);
        }
      };
      bool ok = wait_parity_warp(barFix, 0, abort_flag) && wait_parity_warp(&barX[0], 0, abort_flag);
      if (ok) { issue_s(0); ok = wait_parity_warp(&barY[0], 0, abort_flag); }
      if (ok) issue_dp(0);
      for (int j = 0; j < n && ok; ++j) {
        if (j + 1 < n) {
          ok = wait_parity_warp(&barX[(j + 1) % 3], (j + 1) / 3 & 1, abort_flag);
          if (!ok) break;
          issue_s(j + 1);
        }
        ok = wait_parity_warp(bardS, j & 1, abort_flag);
        if (!ok) break;
        tc_fence_after();
        if (elect_one()) {              // dQ += dS K
#pragma unroll
          for (int s = 0; s < 8; ++s) umma_bf16_ta(tdQ, tdP + (s >> 2) * 64 + (s & 3) * 8, desc_mnmajor(aX + j % 3 * TILE_BYTES, s), id_km, j > 0 || s > 0);
          umma_commit(&barXfree[j % 3]);
        }
        if (j + 1 < n) {                // over dS
          ok = wait_parity_warp(&barY[(j + 1) & 1], ((j + 1) >> 1) & 1, abort_flag);
          if (!ok) break;
          issue_dp(j + 1);
        }
      }
      if (ok) { if (elect_one()) umma_commit(barDone); }
      else fail(ST_TIMEOUT_FULL);
    } else {
      // ---------------------------------------------------------------- softmax (lane = query row, 64 key columns)
      const float* st = p.stats + ((long long)(work.w - kb + qb) * p.heads_q + h) * BWD_STATS;
      const float lse2 = st[r], delta = st[AB + r];
      bool ok = true;
      for (int j = 0; j < n; ++j) {
        const uint32_t t_s = tmem + (j & 1) * 128 + half * 64 + t_lane, t_dp = tdP + half * 64 + t_lane;
        if (!wait_parity_warp(&barS[j & 1], (j >> 1) & 1, abort_flag)) { ok = false; break; }
        tc_fence_after();
        float pr[64];
        {
          uint32_t s[2][32];
          tmem_ld_32x32(t_s, s[0]);
          tmem_ld_32x32(t_s + 32, s[1]);
          tmem_ld_wait();
#pragma unroll
          for (int x = 0; x < 64; ++x) pr[x] = fast_exp2(fmaf(__uint_as_float(s[x >> 5][x & 31]), p.scale_log2e, -lse2));
        }
        if (!wait_parity_warp(bardP, j & 1, abort_flag)) { ok = false; break; }
        tc_fence_after();
        uint32_t pk[32];
#pragma unroll
        for (int c = 0; c < 64; c += 32) {
          uint32_t d[32];
          tmem_ld_32x32(t_dp + c, d);
          tmem_ld_wait();
#pragma unroll
          for (int x = 0; x < 32; ++x) d[x] = __float_as_uint(pr[c + x] * fmaf(__uint_as_float(d[x]), p.scale, -delta));
          if (j == qb) {                 // diagonal: keys to the right of the query
#pragma unroll
            for (int x = 0; x < 32; ++x) if (half * 64 + c + x > r) d[x] = 0u;
          }
#pragma unroll
          for (int x = 0; x < 16; ++x) pk[c / 2 + x] = pack2(__uint_as_float(d[2 * x]), __uint_as_float(d[2 * x + 1]));
        }
        tmem_st_32x32(t_dp, pk);         // over this warp's own part of dP
        tmem_st_wait();
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(bardS);
      }
      ok = ok && wait_parity_warp(barDone, 0, abort_flag);
      if (!ok) { if (lane == 0) fail(ST_TIMEOUT_TMEM_FULL); }
      else {
        tc_fence_after();
        const bool valid = q0 + r < seq_end;
        bf16* out = p.dq + ((long long)(q0 + r) * p.heads_q + h) * HD + half * 64;
#pragma unroll 1
        for (int c = 0; c < 64; c += 32) {
          uint32_t a[32];
          tmem_ld_32x32(tdQ + half * 64 + t_lane + c, a);
          tmem_ld_wait();
          if (valid) {
#pragma unroll
            for (int x = 0; x < 32; x += 8) *reinterpret_cast<uint4*>(out + c + x) = pack8(a + x);
          }
          __syncwarp();
        }
      }
    }
  }
  __syncwarp();
  tc_fence_before();
  __syncthreads();
  if (warp == 9) { tc_fence_after(); tmem_dealloc(tmem, 512); }
}

typedef CUresult (*EncodeTiledFnA)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*, const cuuint64_t*,
                                   const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave, CUtensorMapSwizzle,
                                   CUtensorMapL2promotion, CUtensorMapFloatOOBfill);
static EncodeTiledFnA att_encode_fn() {
  static EncodeTiledFnA fn = nullptr;
  static std::once_flag once;
  std::call_once(once, [] {
    void* ptr = nullptr;
    cudaDriverEntryPointQueryResult q;
    if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &ptr, cudaEnableDefault, &q) == cudaSuccess && q == cudaDriverEntryPointSuccess)
      fn = reinterpret_cast<EncodeTiledFnA>(ptr);
  });
  return fn;
}
// [tokens, heads*128] bf16, box 64 columns x `box_rows` rows
static int att_map(CUtensorMap* m, const void* ptr, long long tokens, int heads, int box_rows = AB) {
  EncodeTiledFnA fn = att_encode_fn();
  if (fn == nullptr) return -1;
  if (reinterpret_cast<uintptr_t>(ptr) & 15) return -2;
  cuuint64_t dims[2] = {(cuuint64_t)heads * HD, (cuuint64_t)tokens};
  cuuint64_t strides[1] = {(cuuint64_t)heads * HD * 2};
  cuuint32_t box[2] = {64, (cuuint32_t)box_rows};
  cuuint32_t es[2] = {1, 1};
  return fn(m, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, const_cast<void*>(ptr), dims, strides, box, es, CU_TENSOR_MAP_INTERLEAVE_NONE,
            CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS ? 0 : -3;
}
constexpr int ATT_SMEM = 6 * TILE_BYTES + 1024 + 128;

}  // namespace mdt

using namespace mdt;

extern "C" long long mdt_attention_launch_count() { return g_att_launches; }

extern "C" int mdt_attention_fwd(const void* q, const void* k, const void* v, void* o, float* lse, const int* cu_seqlens,
                                 int num_seqs, int total_tokens, int max_seqlen, int heads_q, int heads_kv, int head_dim,
                                 float scale, int* status, cudaStream_t s) {
  if (head_dim != HD || heads_q % heads_kv != 0) return -1;
  if (total_tokens == 0) return 0;
  static thread_local bool bound = false;
  if (!bound) { cudaFree(nullptr); bound = true; }
  AttnParams p;
  memset(&p, 0, sizeof(p));
  // MDT_ATTN_FWD=serial selects the one-block-at-a-time kernel (for comparisons); default: the pipelined kernel
  static const bool forced = []() { const char* e = getenv("MDT_ATTN_FWD"); return e != nullptr && e[0] == 's'; }();
  // The pipelined kernel masks and compares scores before they are scaled, which takes a positive scale; any other one goes
  // through the serial kernel, which scales first.
  const bool serial = forced || !(scale > 0.f);
  int rc = att_map(&p.tmQ, q, total_tokens, heads_q);
  if (serial) rc |= att_map(&p.tmK, k, total_tokens, heads_kv) | att_map(&p.tmV, v, total_tokens, heads_kv);
  else rc |= att_map(&p.tmK64, k, total_tokens, heads_kv, FB) | att_map(&p.tmV64, v, total_tokens, heads_kv, FB);
  if (rc) return rc;
  p.cu_seqlens = cu_seqlens; p.num_seqs = num_seqs; p.heads_q = heads_q; p.heads_kv = heads_kv; p.tokens = total_tokens;
  p.status = status;
  p.scale_log2e = scale * 1.4426950408889634f;
  p.o = (bf16*)o; p.lse = lse;
  static bool configured = false;
  if (!configured) {
    if (cudaFuncSetAttribute(attn_fwd_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, ATT_SMEM) != cudaSuccess) return -4;
    if (cudaFuncSetAttribute(attn_fwd_pipelined_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, FWD2_SMEM) != cudaSuccess) return -4;
    configured = true;
  }
  dim3 grid((total_tokens + AB - 1) / AB + num_seqs, heads_q);
  if (serial) launch_after(attn_fwd_kernel, grid, 128, ATT_SMEM, s, p);
  else launch_after(attn_fwd_pipelined_kernel, grid.x * grid.y, FWD2_THREADS, FWD2_SMEM, s, p);
  ++g_att_launches;
  cudaError_t e = cudaGetLastError();
  return e == cudaSuccess ? 0 : -100 - (int)e;
}

namespace {
// How the backward pass is cut: 128-row blocks (upper bound: the sequences are ragged) and query heads per dK, dV CTA.
struct BwdPlan { long long blocks; int hpc, sets; long long off_stats, floats; };
BwdPlan bwd_plan(int num_seqs, int total_tokens, int max_seqlen, int heads_q, int heads_kv) {
  BwdPlan b;
  b.blocks = ((long long)total_tokens + AB - 1) / AB + num_seqs;
  // A CTA that takes all query heads of a kv head adds their dK, dV in TMEM; but its loop is that much longer.  The longest loop may be
  // a third of an SM's share of all work (sequences taken as equally long, one block at least; a round of dK, dV is 1.3 of dQ's),
  // else fewer heads per CTA, in clusters of at most 8 CTAs: 613 tokens, 32 / 8 heads run with one head, four sequences of 1024-8192
  // with all four.
  const int group = heads_q / heads_kv;
  const double seqs = num_seqs > 0 ? num_seqs : 1, n = fmax((double)total_tokens / (AB * seqs), 1.0);
  const double share = 2.3 * seqs * n * (n + 1.0) / 2.0 * heads_q / sm_count_of_current_device();
  const int longest = ((max_seqlen < total_tokens ? max_seqlen : total_tokens) + AB - 1) / AB;
  b.hpc = group;
  for (int h = group - 1; h >= 1 && 1.3 * b.hpc * longest > 0.33 * share; --h)
    if (group % h == 0 && group / h <= MAX_SETS) b.hpc = h;
  b.sets = heads_q / b.hpc;
  b.off_stats = (b.blocks * 4 + 31) / 32 * 32;                                   // after the schedule
  b.floats = b.off_stats + b.blocks * heads_q * BWD_STATS;
  return b;
}
}  // namespace

extern "C" long long mdt_attention_bwd_scratch(int num_seqs, int total_tokens, int max_seqlen, int heads_q, int heads_kv) {
  return bwd_plan(num_seqs, total_tokens, max_seqlen, heads_q, heads_kv).floats;
}

extern "C" int mdt_attention_bwd(const void* q, const void* k, const void* v, const void* o, const void* dout, const float* lse,
                                 void* dq, void* dk, void* dv, float* scratch, const int* cu_seqlens, int num_seqs, int total_tokens,
                                 int max_seqlen, int heads_q, int heads_kv, int head_dim, float scale, int* status, cudaStream_t s) {
  // scratch: mdt_attention_bwd_scratch() floats, 128-byte aligned: schedule | row statistics
  if (head_dim != HD || heads_q % heads_kv != 0) return -1;
  if (total_tokens == 0) return 0;
  if (reinterpret_cast<uintptr_t>(scratch) & 127) return -2;
  static thread_local bool bound = false;
  if (!bound) { cudaFree(nullptr); bound = true; }
  const BwdPlan b = bwd_plan(num_seqs, total_tokens, max_seqlen, heads_q, heads_kv);
  AttnBwdParams p;
  memset(&p, 0, sizeof(p));
  int rc = att_map(&p.tmQ, q, total_tokens, heads_q) | att_map(&p.tmK, k, total_tokens, heads_kv) |
           att_map(&p.tmV, v, total_tokens, heads_kv) | att_map(&p.tmdO, dout, total_tokens, heads_q);
  if (rc) return rc;
  p.sched = reinterpret_cast<const int4*>(scratch); p.stats = scratch + b.off_stats;
  p.dq = (bf16*)dq; p.dk = (bf16*)dk; p.dv = (bf16*)dv;
  p.heads_q = heads_q; p.heads_kv = heads_kv; p.hpc = b.hpc; p.tokens = total_tokens; p.blocks = (int)b.blocks;
  p.status = status;
  p.scale = scale; p.scale_log2e = scale * 1.4426950408889634f;
  static bool configured = false;
  if (!configured) {
    if (cudaFuncSetAttribute(attn_bwd_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, BWD_SMEM) != cudaSuccess) return -4;
    configured = true;
  }
  launch_after(attn_bwd_prepare_kernel, dim3((unsigned)b.blocks, heads_q), 256, 0, s, (const bf16*)o, (const bf16*)dout, lse, cu_seqlens, num_seqs,
               total_tokens, heads_q, heads_kv, scale, reinterpret_cast<int4*>(scratch), scratch + b.off_stats, p.dq, p.dk, p.dv, status);
  ++g_att_launches;
  cudaLaunchConfig_t cfg;
  memset(&cfg, 0, sizeof(cfg));
  cfg.gridDim = dim3((unsigned)(b.blocks * (b.sets + heads_q))); cfg.blockDim = dim3(BWD_THREADS); cfg.dynamicSmemBytes = BWD_SMEM; cfg.stream = s;
  cudaLaunchAttribute attr[2];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = early_setup_pays(cfg.gridDim.x);
  attr[1].id = cudaLaunchAttributeClusterDimension;                                // the sets of a kv head add up their dK, dV
  attr[1].val.clusterDim.x = b.sets / heads_kv; attr[1].val.clusterDim.y = 1; attr[1].val.clusterDim.z = 1;
  cfg.attrs = attr; cfg.numAttrs = b.sets > heads_kv ? 2 : 1;
  cudaLaunchKernelEx(&cfg, attn_bwd_kernel, p);
  ++g_att_launches;
  cudaError_t e = cudaGetLastError();
  return e == cudaSuccess ? 0 : -100 - (int)e;
}
