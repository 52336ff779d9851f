// Memory-bound kernels: RMSNorm, RoPE, SwiGLU, embedding, softmax cross-entropy, AdamW, reductions.
// All of them move 16 bytes per thread per access and keep intermediate math in fp32.
#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <stdint.h>

#include "api.h"
#include "common/host.h"
#include "common/ptx.cuh"

namespace mdt {

static long long g_ew_launches = 0;
typedef __nv_bfloat16 bf16;
typedef __nv_bfloat162 bf162;

__device__ __forceinline__ void unpack8(const uint4& u, float (&f)[8]) {
  const bf162* h = reinterpret_cast<const bf162*>(&u);
#pragma unroll
  for (int i = 0; i < 4; ++i) { float2 t = __bfloat1622float2(h[i]); f[2 * i] = t.x; f[2 * i + 1] = t.y; }
}
__device__ __forceinline__ uint4 pack8(const float (&f)[8]) {
  uint4 u;
  bf162* h = reinterpret_cast<bf162*>(&u);
#pragma unroll
  for (int i = 0; i < 4; ++i) h[i] = __floats2bfloat162_rn(f[2 * i], f[2 * i + 1]);
  return u;
}
__device__ __forceinline__ float warp_sum(float v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}
__device__ __forceinline__ float warp_max(float v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v = fmaxf(v, __shfl_xor_sync(0xffffffffu, v, o));
  return v;
}
// block-wide sum; `red` is shared memory for 32 floats; every thread receives the result
__device__ __forceinline__ float block_sum(float v, float* red) {
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5, nw = (blockDim.x + 31) >> 5;
  v = warp_sum(v);
  __syncthreads();
  if (lane == 0) red[w] = v;
  __syncthreads();
  float t = (lane < nw) ? red[lane] : 0.f;
  return warp_sum(t);
}
__device__ __forceinline__ float block_max(float v, float* red) {
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5, nw = (blockDim.x + 31) >> 5;
  v = warp_max(v);
  __syncthreads();
  if (lane == 0) red[w] = v;
  __syncthreads();
  float t = (lane < nw) ? red[lane] : -INFINITY;
  return warp_max(t);
}

// ------------------------------------------------------------------------------------ RMSNorm
__global__ void rmsnorm_fwd_kernel(const bf16* __restrict__ x, const bf16* __restrict__ w, bf16* __restrict__ y,
                                   float* __restrict__ rstd, int rows, int cols, float eps) {
  after_predecessor();
  __shared__ float red[32];
  const int row = blockIdx.x;
  const uint4* xr = reinterpret_cast<const uint4*>(x + (long long)row * cols);
  const uint4* wr = reinterpret_cast<const uint4*>(w);
  uint4* yr = reinterpret_cast<uint4*>(y + (long long)row * cols);
  const int nv = cols / 8;
  float ss = 0.f;
  for (int i = threadIdx.x; i < nv; i += blockDim.x) {
    float f[8]; unpack8(xr[i], f);
#pragma unroll
    for (int j = 0; j < 8; ++j) ss += f[j] * f[j];
  }
  ss = block_sum(ss, red);
  const float r = rsqrtf(ss / cols + eps);
  if (threadIdx.x == 0 && rstd != nullptr) rstd[row] = r;
  for (int i = threadIdx.x; i < nv; i += blockDim.x) {
    float f[8], g[8]; unpack8(xr[i], f); unpack8(wr[i], g);
#pragma unroll
    for (int j = 0; j < 8; ++j) f[j] = f[j] * r * g[j];
    yr[i] = pack8(f);
  }
}

// dx = rstd * (dy*w - x * rstd^2 * mean(dy*w*x)) (+ dres, the gradient that reaches x past the norm through the
// residual connection);  dw partial sums per CTA (CTA loops over rows), unless dw_partial is NULL (frozen norm).
// Bound by one pass over x, dy, dres and dx.  A thread holds its NV vectors of the row and of the next one in registers,
// so a row costs one barrier-separated sum and its loads are in flight while the row before it is reduced; several CTAs
// share an SM.  8000 x 4096 with dres: 165 us with the row read twice by one CTA per SM, without a look ahead.
template <int NV>
__global__ void __launch_bounds__(256) rmsnorm_bwd_kernel(const bf16* __restrict__ x, const bf16* __restrict__ w, const bf16* __restrict__ dy,
                                                          const float* __restrict__ rstd, const bf16* __restrict__ dres, bf16* __restrict__ dx,
                                                          float* __restrict__ dw_partial, int rows, int cols) {
  after_predecessor();
  __shared__ float red[32];
  const int nv = cols / 8;
  const uint4* xr = reinterpret_cast<const uint4*>(x);
  const uint4* dr = reinterpret_cast<const uint4*>(dy);
  const uint4* rr = reinterpret_cast<const uint4*>(dres);
  uint4* ox = reinterpret_cast<uint4*>(dx);
  const uint4 zero = make_uint4(0, 0, 0, 0);
  float acc[NV][8];
  uint4 wv[NV], xn[NV], dn[NV], rn[NV];
  float rs = 0.f;
  auto load = [&](int row) {
#pragma unroll
    for (int k = 0; k < NV; ++k) {
      const int i = threadIdx.x + k * 256;
      const bool in = i < nv;
      const long long at = (long long)row * nv + i;
      xn[k] = in ? xr[at] : zero; dn[k] = in ? dr[at] : zero; rn[k] = in && rr != nullptr ? rr[at] : zero;
    }
    rs = rstd[row];
  };
#pragma unroll
  for (int k = 0; k < NV; ++k) {
    const int i = threadIdx.x + k * 256;
    wv[k] = i < nv ? reinterpret_cast<const uint4*>(w)[i] : zero;
#pragma unroll
    for (int j = 0; j < 8; ++j) acc[k][j] = 0.f;
  }
  constexpr bool AHEAD = NV <= 4;      // (more columns: no registers for the next row)
  if (AHEAD && (int)blockIdx.x < rows) load(blockIdx.x);
  for (int row = blockIdx.x; row < rows; row += gridDim.x) {
    if (!AHEAD) load(row);
    uint4 xv[NV], dv[NV], rv[NV];
    const float r = rs;
#pragma unroll
    for (int k = 0; k < NV; ++k) { xv[k] = xn[k]; dv[k] = dn[k]; rv[k] = rn[k]; }
    if (AHEAD && row + (int)gridDim.x < rows) load(row + gridDim.x);
    float dot = 0.f;
#pragma unroll
    for (int k = 0; k < NV; ++k) {
      float xf[8], df[8], wf[8]; unpack8(xv[k], xf); unpack8(dv[k], df); unpack8(wv[k], wf);
#pragma unroll
      for (int j = 0; j < 8; ++j) dot += df[j] * wf[j] * xf[j];
    }
    dot = block_sum(dot, red);
    const float c = dot * r * r / cols;
#pragma unroll
    for (int k = 0; k < NV; ++k) {
      const int i = threadIdx.x + k * 256;
      float xf[8], df[8], wf[8], rf[8], o[8]; unpack8(xv[k], xf); unpack8(dv[k], df); unpack8(wv[k], wf); unpack8(rv[k], rf);
#pragma unroll
      for (int j = 0; j < 8; ++j) {
        o[j] = r * (df[j] * wf[j] - xf[j] * c) + rf[j];
        acc[k][j] += df[j] * xf[j] * r;
      }
      if (i < nv) ox[(long long)row * nv + i] = pack8(o);
    }
  }
  if (dw_partial == nullptr) return;
#pragma unroll
  for (int k = 0; k < NV; ++k) {
    const int i = threadIdx.x + k * 256;
    if (i < nv) {
      float4* dst = reinterpret_cast<float4*>(dw_partial + (long long)blockIdx.x * cols + i * 8);
      dst[0] = make_float4(acc[k][0], acc[k][1], acc[k][2], acc[k][3]);
      dst[1] = make_float4(acc[k][4], acc[k][5], acc[k][6], acc[k][7]);
    }
  }
}

// dw[c] = sum over the partial rows (+ cast): finishes the weight gradient of rmsnorm_bwd_kernel in one launch.  The
// partial rows are spread over the 8 warps of a CTA (32 columns each), eight loads in flight per lane.
__global__ void __launch_bounds__(256) rmsnorm_dw_finalize_kernel(const float* __restrict__ partial, int n_partial, int cols, bf16* __restrict__ dw_bf16,
                                                                  float* __restrict__ dw_f32) {
  after_predecessor();
  __shared__ float part[8][33];
  const int lane = threadIdx.x & 31, wp = threadIdx.x >> 5;
  const int c = blockIdx.x * 32 + lane;
  float s = 0.f;
  if (c < cols) {
#pragma unroll 8
    for (int r = wp; r < n_partial; r += 8) s += partial[(long long)r * cols + c];
  }
  part[wp][lane] = s;
  __syncthreads();
  if (wp != 0 || c >= cols) return;
#pragma unroll
  for (int k = 1; k < 8; ++k) s += part[k][lane];
  if (dw_bf16 != nullptr) dw_bf16[c] = __float2bfloat16(s);
  if (dw_f32 != nullptr) dw_f32[c] = s;
}

// ------------------------------------------------------------------------------------ RoPE
// x: [tokens, heads, d]; pairs (i, i + d/2) rotated by pos * theta^(-2i/d); inverse negates the angle
// One CTA per token: its d/2 angles are evaluated once, into shared memory, and used for all heads; a thread then
// rotates eight pairs with 16-byte accesses (head sizes that are a multiple of 16; else pair by pair).
// 8000 tokens x 32 heads of 128: 85 us with one sincosf and 2-byte accesses per pair.
__global__ void __launch_bounds__(256) rope_kernel(const bf16* __restrict__ x, bf16* __restrict__ y, const int* __restrict__ pos, int tokens,
                                                   int heads, int d, float log2_theta, int inverse, int vec) {
  after_predecessor();
  extern __shared__ float angles[];            // cos [half] | sin [half]
  const int t = blockIdx.x;
  const int half = d / 2;
  const float p = (float)pos[t];
  for (int i = threadIdx.x; i < half; i += blockDim.x) {
    const float inv_freq = exp2f(-log2_theta * (2.0f * i / d));
    float s, c;
    sincosf(p * inv_freq, &s, &c);
    angles[i] = c;
    angles[half + i] = inverse ? -s : s;
  }
  __syncthreads();
  const long long row = (long long)t * heads * d;
  if (vec) {
    const int per = half / 8;
    for (int idx = threadIdx.x; idx < heads * per; idx += blockDim.x) {
      const int h = idx / per, i = (idx - h * per) * 8;
      const long long base = row + (long long)h * d + i;
      float a[8], b[8], u[8], v[8];
      unpack8(*reinterpret_cast<const uint4*>(x + base), a);
      unpack8(*reinterpret_cast<const uint4*>(x + base + half), b);
#pragma unroll
      for (int j = 0; j < 8; ++j) {
        const float c = angles[i + j], s = angles[half + i + j];
        u[j] = a[j] * c - b[j] * s;
        v[j] = b[j] * c + a[j] * s;
      }
      *reinterpret_cast<uint4*>(y + base) = pack8(u);
      *reinterpret_cast<uint4*>(y + base + half) = pack8(v);
    }
    return;
  }
  for (int idx = threadIdx.x; idx < heads * half; idx += blockDim.x) {
    const int h = idx / half, i = idx - h * half;
    const float s = angles[half + i], c = angles[i];
    const long long base = row + (long long)h * d;
    const float a = __bfloat162float(x[base + i]), b = __bfloat162float(x[base + i + half]);
    y[base + i] = __float2bfloat16(a * c - b * s);
    y[base + i + half] = __float2bfloat16(b * c + a * s);
  }
}

// ------------------------------------------------------------------------------------ SwiGLU
__global__ void swiglu_fwd_kernel(const uint4* __restrict__ g, const uint4* __restrict__ u, uint4* __restrict__ h, long long nv) {
  after_predecessor();
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < nv; i += (long long)gridDim.x * blockDim.x) {
    float a[8], b[8]; unpack8(g[i], a); unpack8(u[i], b);
#pragma unroll
    for (int j = 0; j < 8; ++j) a[j] = a[j] / (1.f + __expf(-a[j])) * b[j];
    h[i] = pack8(a);
  }
}
// Copy of a capacity-sized row buffer that touches only the rows in use (count read from device memory).
__global__ void copy_rows_used_kernel(const uint4* __restrict__ src, uint4* __restrict__ dst, long long nv,
                                      const int* __restrict__ rows_used, long long vecs_per_row) {
  after_predecessor();
  const long long lim = (long long)rows_used[0] * vecs_per_row;
  nv = lim < nv ? lim : nv;
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < nv; i += (long long)gridDim.x * blockDim.x) dst[i] = src[i];
}

// ------------------------------------------------------------------------------------ embedding
__global__ void embedding_kernel(const bf16* __restrict__ table, const long long* __restrict__ ids, bf16* __restrict__ out, int cols) {
  after_predecessor();
  const long long id = ids[blockIdx.x];
  const uint4* src = reinterpret_cast<const uint4*>(table + id * cols);
  uint4* dst = reinterpret_cast<uint4*>(out + (long long)blockIdx.x * cols);
  for (int i = threadIdx.x; i < cols / 8; i += blockDim.x) dst[i] = src[i];
}
// Gradient of the table: rows that tokens name are written with, or (add) increased by, the sum of their tokens' rows of dout, in fp32
// and rounded once (the others are left alone).  Text is not uniform: most ids have one or two tokens, a filler token may have nearly all.  The
// first EMB_LIST tokens of an id form a list (head[id], then next[token]) that the CTA of the token at its head adds up.  Later ones are
// added to a row of fp32 sums that the id gets then, 16 tokens by a CTA, equal ids among them first; the CTA at the head adds that.
// 32000 x 4096, us, of which clearing the table takes about 75: 576 tokens uniform 87, 90 % of one id 110; 8192 tokens 116 and 136.  Lists
// of all tokens took 83, 617, 108 and 7630 (one CTA walks them), a table in fp32, added to with atomics and converted, 204 to 286.
constexpr int EMB_LIST = 32, EMB_LATE = 16, EMB_LATE_MARK = -2;
__global__ void __launch_bounds__(256) embedding_list_kernel(const long long* __restrict__ ids, int* __restrict__ next, int* __restrict__ head, int* __restrict__ count,
                                                             int* __restrict__ sum_row, int* __restrict__ sum_rows, float4* __restrict__ sums, long long nv, int tokens) {
  after_predecessor();
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < nv; i += (long long)gridDim.x * blockDim.x) sums[i] = make_float4(0.f, 0.f, 0.f, 0.f);
  const int t = blockIdx.x * blockDim.x + threadIdx.x, lane = threadIdx.x & 31;
  const long long id = t < tokens ? ids[t] : -1;
  // (one addition for all lanes of an id; head, count, sum_row and sum_rows start at -1)
  const unsigned same = __match_any_sync(0xffffffffu, id);
  const int first = __ffs(same) - 1;
  int rank = 0;
  if (id >= 0 && lane == first) rank = atomicAdd(count + id, __popc(same)) + 1;
  rank = __shfl_sync(0xffffffffu, rank, first) + __popc(same & ((1u << lane) - 1));
  if (id < 0) return;
  next[t] = rank < EMB_LIST ? atomicExch(head + id, t) : EMB_LATE_MARK;
  if (rank == EMB_LIST) sum_row[id] = atomicAdd(sum_rows, 1) + 1;
}
__global__ void __launch_bounds__(256) embedding_late_kernel(const bf16* __restrict__ dout, const long long* __restrict__ ids, const int* __restrict__ next,
                                                             const int* __restrict__ sum_row, float* __restrict__ sums, int tokens, int cols) {
  after_predecessor();
  __shared__ int rows[EMB_LATE];
  const int t0 = blockIdx.x * EMB_LATE;
  int row = -1;
  if (threadIdx.x < EMB_LATE) {
    const int t = t0 + threadIdx.x;
    if (t < tokens && next[t] == EMB_LATE_MARK) row = sum_row[ids[t]];
    rows[threadIdx.x] = row;
  }
  if (!__syncthreads_or(row >= 0)) return;
  const int col = (blockIdx.y * 256 + threadIdx.x) * 8;
  if (col >= cols) return;
  uint4 v[EMB_LATE];
#pragma unroll
  for (int i = 0; i < EMB_LATE; ++i)
    if (rows[i] >= 0) v[i] = *reinterpret_cast<const uint4*>(dout + (long long)(t0 + i) * cols + col);
#pragma unroll
  for (int i = 0; i < EMB_LATE; ++i) {
    const int r = rows[i];
    bool done = r < 0;
#pragma unroll
    for (int j = 0; j < i; ++j) done = done || rows[j] == r;
    if (done) continue;
    float f[8] = {0, 0, 0, 0, 0, 0, 0, 0};
#pragma unroll
    for (int j = i; j < EMB_LATE; ++j)
      if (rows[j] == r) {
        float g[8];
        unpack8(v[j], g);
#pragma unroll
        for (int k = 0; k < 8; ++k) f[k] += g[k];
      }
    float* to = sums + (long long)r * cols + col;
    red_add_v4_f32(to, f[0], f[1], f[2], f[3]);
    red_add_v4_f32(to + 4, f[4], f[5], f[6], f[7]);
  }
}
template <bool F32>
__global__ void __launch_bounds__(256) embedding_bwd_kernel(const bf16* __restrict__ dout, const long long* __restrict__ ids, const int* __restrict__ next,
                                                            const int* __restrict__ head, const int* __restrict__ sum_row, const float* __restrict__ sums,
                                                            void* __restrict__ dtable, int cols, int add) {
  after_predecessor();
  const long long id = ids[blockIdx.x];
  if (head[id] != (int)blockIdx.x) return;
  __shared__ int list[EMB_LIST], length;
  if (threadIdx.x == 0) {
    int n = 0;
    for (int t = blockIdx.x; t >= 0 && n < EMB_LIST; t = next[t]) list[n++] = t;
    length = n;
  }
  __syncthreads();
  const int n = length, row = sum_row[id];
  for (int i = threadIdx.x; i < cols / 8; i += blockDim.x) {
    float f[8] = {0, 0, 0, 0, 0, 0, 0, 0};
    auto plus = [&](const float* src) {
      const float4 x = reinterpret_cast<const float4*>(src)[0], y = reinterpret_cast<const float4*>(src)[1];
      f[0] += x.x; f[1] += x.y; f[2] += x.z; f[3] += x.w; f[4] += y.x; f[5] += y.y; f[6] += y.z; f[7] += y.w;
    };
    const long long at = id * cols + i * 8;
    if (add) {
      if (F32) plus(reinterpret_cast<const float*>(dtable) + at);
      else unpack8(*reinterpret_cast<const uint4*>(reinterpret_cast<const bf16*>(dtable) + at), f);
    }
    if (row >= 0) plus(sums + (long long)row * cols + i * 8);
#pragma unroll 4
    for (int k = 0; k < n; ++k) {
      float g[8];
      unpack8(reinterpret_cast<const uint4*>(dout + (long long)list[k] * cols)[i], g);
#pragma unroll
      for (int j = 0; j < 8; ++j) f[j] += g[j];
    }
    if (F32) {
      float4* o = reinterpret_cast<float4*>(reinterpret_cast<float*>(dtable) + at);
      o[0] = make_float4(f[0], f[1], f[2], f[3]); o[1] = make_float4(f[4], f[5], f[6], f[7]);
    } else {
      *reinterpret_cast<uint4*>(reinterpret_cast<bf16*>(dtable) + at) = pack8(f);
    }
  }
}

// ------------------------------------------------------------------------------------ expert adapters
// The gate and up adapters of a layer as their products want them: A13 [E, H, 2r] = [s1 A1 | s3 A3], and K-major B1p = [B1^T | 0],
// B3p = [0 | B3^T], both [E, F, 2r].  One pass over 14 MB (8 experts, rank 16, 4096 -> 14336) instead of the six that scaling,
// concatenating and transposing them with library operations takes: 10 us against 48 and five launches more.
// CTA: 64 columns of one expert's B (transposed through shared memory), or a stretch of A's rows.
// (The products want ranks that are multiples of 4.)
constexpr int ADAPTER_COLS = 64, ADAPTER_RANKS = 64;
__global__ void __launch_bounds__(256) adapter_pack_kernel(const bf16* __restrict__ A1, const bf16* __restrict__ A3, float s1, float s3, const bf16* __restrict__ B1,
                                                           const bf16* __restrict__ B3, bf16* __restrict__ A13, bf16* __restrict__ B1p, bf16* __restrict__ B3p,
                                                           int E, int H, int F, int r) {
  after_predecessor();
  __shared__ bf16 tile[2][ADAPTER_RANKS][ADAPTER_COLS + 2];
  const int strips = (F + ADAPTER_COLS - 1) / ADAPTER_COLS;
  if ((int)blockIdx.x < E * strips) {
    const int e = blockIdx.x / strips, f0 = (blockIdx.x - e * strips) * ADAPTER_COLS, n = min(ADAPTER_COLS, F - f0);
    for (int k0 = 0; k0 < r; k0 += ADAPTER_RANKS) {
      const int ranks = min(ADAPTER_RANKS, r - k0);
      for (int i = threadIdx.x; i < ranks * ADAPTER_COLS; i += blockDim.x) {
        const int k = i / ADAPTER_COLS, f = i % ADAPTER_COLS;
        if (f < n) {
          const long long at = ((long long)e * r + k0 + k) * F + f0 + f;
          tile[0][k][f] = B1[at];
          tile[1][k][f] = B3[at];
        }
      }
      __syncthreads();
      for (int i = threadIdx.x; i < n * (ranks / 4); i += blockDim.x) {
        const int f = i / (ranks / 4), k = i % (ranks / 4) * 4;
        const long long row = ((long long)e * F + f0 + f) * 2 * r + k0 + k;
        uint2 v[2];
#pragma unroll
        for (int m = 0; m < 2; ++m) {
          bf16* q = reinterpret_cast<bf16*>(&v[m]);
#pragma unroll
          for (int j = 0; j < 4; ++j) q[j] = tile[m][k + j][f];
        }
        *reinterpret_cast<uint2*>(B1p + row) = v[0];
        *reinterpret_cast<uint2*>(B1p + row + r) = make_uint2(0u, 0u);
        *reinterpret_cast<uint2*>(B3p + row) = make_uint2(0u, 0u);
        *reinterpret_cast<uint2*>(B3p + row + r) = v[1];
      }
      __syncthreads();
    }
    return;
  }
  const long long rows = (long long)E * H;
  const int ctas = gridDim.x - E * strips, b = blockIdx.x - E * strips;
  for (long long i = (long long)b * blockDim.x + threadIdx.x; i < rows * (r / 4); i += (long long)ctas * blockDim.x) {
    const long long row = i / (r / 4);
    const int k = (int)(i - row * (r / 4)) * 4;
    const uint2 v[2] = {*reinterpret_cast<const uint2*>(A1 + row * r + k), *reinterpret_cast<const uint2*>(A3 + row * r + k)};
#pragma unroll
    for (int m = 0; m < 2; ++m) {
      const float s = m == 0 ? s1 : s3;
      const float2 lo = __bfloat1622float2(reinterpret_cast<const bf162*>(&v[m])[0]), hi = __bfloat1622float2(reinterpret_cast<const bf162*>(&v[m])[1]);
      uint2 o;
      reinterpret_cast<bf162*>(&o)[0] = __floats2bfloat162_rn(lo.x * s, lo.y * s);
      reinterpret_cast<bf162*>(&o)[1] = __floats2bfloat162_rn(hi.x * s, hi.y * s);
      *reinterpret_cast<uint2*>(A13 + row * 2 * r + m * r + k) = o;
    }
  }
}

// ------------------------------------------------------------------------------------ cross entropy
// One CTA per row.  The row (vocab bf16 values) is staged in shared memory, so global memory is read
// once and written once.  Output: logits <- (softmax - onehot) * grad_scale / max(count,1), or 0 for
// ignored rows; loss_sum += lse - logit[label].  `count` must already hold the number of counted rows.
__global__ void cross_entropy_kernel(bf16* __restrict__ logits, const long long* __restrict__ labels, float* __restrict__ loss_sum,
                                     const float* __restrict__ count, int vocab, long long ld, int ignore_index, float grad_scale) {
  after_predecessor();
  extern __shared__ uint4 row_smem[];
  __shared__ float red[32];
  const int row = blockIdx.x;
  uint4* gr = reinterpret_cast<uint4*>(logits + (long long)row * ld);
  const int nv = vocab / 8;
  const long long label = labels[row];
  if (label == ignore_index) {
    for (int i = threadIdx.x; i < nv; i += blockDim.x) gr[i] = make_uint4(0, 0, 0, 0);
    return;
  }
  float mx = -INFINITY;
  for (int i = threadIdx.x; i < nv; i += blockDim.x) {
    uint4 u = gr[i]; row_smem[i] = u;
    float f[8]; unpack8(u, f);
#pragma unroll
    for (int j = 0; j < 8; ++j) mx = fmaxf(mx, f[j]);
  }
  mx = block_max(mx, red);
  float se = 0.f;
  for (int i = threadIdx.x; i < nv; i += blockDim.x) {
    float f[8]; unpack8(row_smem[i], f);
#pragma unroll
    for (int j = 0; j < 8; ++j) se += __expf(f[j] - mx);
  }
  se = block_sum(se, red);
  const float lse = mx + logf(se);
  const float scale = grad_scale / fmaxf(*count, 1.f);
  const float inv = 1.f / se;
  for (int i = threadIdx.x; i < nv; i += blockDim.x) {
    float f[8]; unpack8(row_smem[i], f);
#pragma unroll
    for (int j = 0; j < 8; ++j) {
      float pz = __expf(f[j] - mx) * inv;
      if ((long long)i * 8 + j == label) {
        pz -= 1.f;
        atomicAdd(loss_sum, lse - f[j]);
      }
      f[j] = pz * scale;
    }
    gr[i] = pack8(f);
  }
}
__global__ void count_labels_kernel(const long long* __restrict__ labels, int rows, int ignore_index, float* __restrict__ count) {
  after_predecessor();
  __shared__ float red[32];
  float c = 0.f;
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < rows; i += gridDim.x * blockDim.x) c += labels[i] != ignore_index ? 1.f : 0.f;
  c = block_sum(c, red);
  if (threadIdx.x == 0 && c != 0.f) atomicAdd(count, c);
}

// ------------------------------------------------------------------------------------ AdamW
template <typename T> __device__ __forceinline__ float ldf(const T* p, long long i);
template <> __device__ __forceinline__ float ldf<float>(const float* p, long long i) { return p[i]; }
template <> __device__ __forceinline__ float ldf<bf16>(const bf16* p, long long i) { return __bfloat162float(p[i]); }
template <typename T> __device__ __forceinline__ void stf(T* p, long long i, float v);
template <> __device__ __forceinline__ void stf<float>(float* p, long long i, float v) { p[i] = v; }
template <> __device__ __forceinline__ void stf<bf16>(bf16* p, long long i, float v) { p[i] = __float2bfloat16(v); }

// bias corrections enter as reciprocals (ibc1 = 1 / (1 - beta1^t), ibc2 likewise) so that the update costs one
// square root and one division per element; both use the fast single-precision forms, whose error (a few ulp of
// fp32) is far below the bf16 resolution of the parameters and moments they are rounded to
__device__ __forceinline__ void adam_update(float& p, float g, float& m, float& v, float lr, float b1, float b2, float eps,
                                            float wd, float ibc1, float ibc2, float gscale) {
  const float gg = g * gscale;
  m = b1 * m + (1.f - b1) * gg;
  v = b2 * v + (1.f - b2) * gg * gg;
  const float denom = __fsqrt_rn(v * ibc2) + eps;
  p = p * (1.f - lr * wd) - __fdividef(lr * (m * ibc1), denom);
}
__device__ __forceinline__ bool aligned16(const void* a, const void* b, const void* c, const void* d) {
  return ((reinterpret_cast<uintptr_t>(a) | reinterpret_cast<uintptr_t>(b) | reinterpret_cast<uintptr_t>(c) |
           reinterpret_cast<uintptr_t>(d)) & 15) == 0;
}

// One launch for all tensors (blockIdx.y = tensor).  All-bf16, 16-byte aligned tensors go eight elements per
// thread and iteration through 128-bit loads (four loads in flight per thread, 32 warps per SM); everything else,
// and the tail, element by element.
__global__ void __launch_bounds__(256, 4) adamw_kernel(const MdtAdamTensor* __restrict__ tensors, float lr, float b1, float b2,
                                                       float eps, float wd, float ibc1, float ibc2, float gscale,
                                                       const float* __restrict__ gscale_dev) {
  after_predecessor();
  const MdtAdamTensor t = tensors[blockIdx.y];
  if (gscale_dev != nullptr) gscale *= *gscale_dev;
  const long long tid = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  const long long nthreads = (long long)gridDim.x * blockDim.x;
  long long done = 0;
  if (!t.p_fp32 && !t.g_fp32 && !t.s_fp32 && aligned16(t.p, t.g, t.m, t.v)) {
    const long long nv = t.n / 8;
    uint4* __restrict__ pp = reinterpret_cast<uint4*>(t.p);
    const uint4* __restrict__ gp = reinterpret_cast<const uint4*>(t.g);
    uint4* __restrict__ mp = reinterpret_cast<uint4*>(t.m);
    uint4* __restrict__ vp = reinterpret_cast<uint4*>(t.v);
    for (long long i = tid; i < nv; i += nthreads) {
      uint4 P = pp[i], G = __ldcs(gp + i), M = mp[i], V = vp[i];
      bf162* ph = reinterpret_cast<bf162*>(&P); const bf162* gh = reinterpret_cast<const bf162*>(&G);
      bf162* mh = reinterpret_cast<bf162*>(&M); bf162* vh = reinterpret_cast<bf162*>(&V);
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        float2 p = __bfloat1622float2(ph[j]), g = __bfloat1622float2(gh[j]), m = __bfloat1622float2(mh[j]), v = __bfloat1622float2(vh[j]);
        adam_update(p.x, g.x, m.x, v.x, lr, b1, b2, eps, wd, ibc1, ibc2, gscale);
        adam_update(p.y, g.y, m.y, v.y, lr, b1, b2, eps, wd, ibc1, ibc2, gscale);
        ph[j] = __floats2bfloat162_rn(p.x, p.y); mh[j] = __floats2bfloat162_rn(m.x, m.y); vh[j] = __floats2bfloat162_rn(v.x, v.y);
      }
      pp[i] = P; mp[i] = M; vp[i] = V;
    }
    done = nv * 8;
  }
  for (long long i = done + tid; i < t.n; i += nthreads) {
    float p = t.p_fp32 ? ldf((const float*)t.p, i) : ldf((const bf16*)t.p, i);
    const float g = t.g_fp32 ? ldf((const float*)t.g, i) : ldf((const bf16*)t.g, i);
    float m = t.s_fp32 ? ldf((const float*)t.m, i) : ldf((const bf16*)t.m, i);
    float v = t.s_fp32 ? ldf((const float*)t.v, i) : ldf((const bf16*)t.v, i);
    adam_update(p, g, m, v, lr, b1, b2, eps, wd, ibc1, ibc2, gscale);
    if (t.p_fp32) stf((float*)t.p, i, p); else stf((bf16*)t.p, i, p);
    if (t.s_fp32) { stf((float*)t.m, i, m); stf((float*)t.v, i, v); }
    else { stf((bf16*)t.m, i, m); stf((bf16*)t.v, i, v); }
  }
}

__global__ void __launch_bounds__(256) sumsq_kernel(const void* __restrict__ x, long long n, int fp32, float* __restrict__ out) {
  after_predecessor();
  __shared__ float red[32];
  const long long tid = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  const long long nthreads = (long long)gridDim.x * blockDim.x;
  float s = 0.f;
  long long done = 0;
  if ((reinterpret_cast<uintptr_t>(x) & 15) == 0) {
    const uint4* __restrict__ xv = reinterpret_cast<const uint4*>(x);
    const int per = fp32 ? 4 : 8;
    const long long nv = n / per;
    for (long long i = tid; i < nv; i += nthreads) {
      const uint4 u = xv[i];
      if (fp32) {
        const float4 f = *reinterpret_cast<const float4*>(&u);
        s += f.x * f.x + f.y * f.y + f.z * f.z + f.w * f.w;
      } else {
        const bf162* h = reinterpret_cast<const bf162*>(&u);
#pragma unroll
        for (int j = 0; j < 4; ++j) { const float2 f = __bfloat1622float2(h[j]); s += f.x * f.x + f.y * f.y; }
      }
    }
    done = nv * per;
  }
  for (long long i = done + tid; i < n; i += nthreads) {
    const float v = fp32 ? ((const float*)x)[i] : __bfloat162float(((const bf16*)x)[i]);
    s += v * v;
  }
  s = block_sum(s, red);
  if (threadIdx.x == 0) atomicAdd(out, s);
}

// y = a*y + b*x
__global__ void __launch_bounds__(256) axpby_kernel(void* __restrict__ y, const void* __restrict__ x, long long n, float a, float b,
                                                    int y_fp32, int x_fp32) {
  after_predecessor();
  const long long tid = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  const long long nthreads = (long long)gridDim.x * blockDim.x;
  long long done = 0;
  if (!y_fp32 && !x_fp32 && ((reinterpret_cast<uintptr_t>(y) | reinterpret_cast<uintptr_t>(x)) & 15) == 0) {
    const long long nv = n / 8;
    uint4* __restrict__ yv = reinterpret_cast<uint4*>(y);
    const uint4* __restrict__ xv = reinterpret_cast<const uint4*>(x);
    for (long long i = tid; i < nv; i += nthreads) {
      const uint4 X = xv[i];
      uint4 Y = a == 0.f ? make_uint4(0, 0, 0, 0) : yv[i];
      bf162* yh = reinterpret_cast<bf162*>(&Y); const bf162* xh = reinterpret_cast<const bf162*>(&X);
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const float2 yf = __bfloat1622float2(yh[j]), xf = __bfloat1622float2(xh[j]);
        yh[j] = __floats2bfloat162_rn(a * yf.x + b * xf.x, a * yf.y + b * xf.y);
      }
      yv[i] = Y;
    }
    done = nv * 8;
  }
  for (long long i = done + tid; i < n; i += nthreads) {
    const float xv = x_fp32 ? ((const float*)x)[i] : __bfloat162float(((const bf16*)x)[i]);
    const float yv = a == 0.f ? 0.f : a * (y_fp32 ? ((float*)y)[i] : __bfloat162float(((bf16*)y)[i]));
    const float r = yv + b * xv;
    if (y_fp32) ((float*)y)[i] = r; else ((bf16*)y)[i] = __float2bfloat16(r);
  }
}

// cap: upper bound on the grid in CTAs; <= 0 means -cap CTAs per SM of the current device (default 16 per SM)
// dst_i (fp32) += src_i (bf16 or fp32) for up to MDT_MULTI_ADD_MAX tensors in one launch (pointers passed by value)
__global__ void multi_add_kernel(const MdtMultiAdd a) {
  after_predecessor();
  const int t = blockIdx.y;
  if (t >= a.count) return;
  float* __restrict__ dst = a.dst[t];
  const long long n = a.n[t];
  if (a.src_fp32[t]) {
    const float* __restrict__ src = reinterpret_cast<const float*>(a.src[t]);
    for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x) dst[i] += src[i];
  } else {
    const bf16* __restrict__ src = reinterpret_cast<const bf16*>(a.src[t]);
    for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x)
      dst[i] += __bfloat162float(src[i]);
  }
}

static inline int grid_for(long long work_items, int block, int cap = -16) {
  if (cap <= 0) cap = sm_count_of_current_device() * -cap;
  long long g = (work_items + block - 1) / block;
  return (int)(g < 1 ? 1 : (g > cap ? cap : g));
}
#define MDT_CHECK_LAUNCH() do { ++g_ew_launches; cudaError_t e_ = cudaGetLastError(); if (e_ != cudaSuccess) return -100 - (int)e_; } while (0)

}  // namespace mdt

using namespace mdt;

extern "C" long long mdt_elementwise_launch_count() { return g_ew_launches; }

extern "C" int mdt_rmsnorm_fwd(const void* x, const void* w, void* y, float* rstd, int rows, int cols, float eps, cudaStream_t s) {
  if (cols % 8 != 0) return -1;
  if (rows == 0) return 0;
  launch_after(rmsnorm_fwd_kernel, rows, 256, 0, s, (const bf16*)x, (const bf16*)w, (bf16*)y, rstd, rows, cols, eps);
  MDT_CHECK_LAUNCH();
  return 0;
}
extern "C" int mdt_rmsnorm_bwd(const void* x, const void* w, const void* dy, const float* rstd, const void* dres, void* dx,
                               float* dw_partial, int rows, int cols, int n_partial, cudaStream_t s) {
  if (cols % 8 != 0 || cols > 8 * 8 * 256) return -1;
  const int nv = (cols / 8 + 255) / 256;
#define RMS_BWD(NV) launch_after(rmsnorm_bwd_kernel<NV>, n_partial, 256, 0, s, (const bf16*)x, (const bf16*)w, (const bf16*)dy, rstd, (const bf16*)dres, (bf16*)dx, dw_partial, rows, cols)
  if (nv <= 1) RMS_BWD(1); else if (nv <= 2) RMS_BWD(2); else if (nv <= 4) RMS_BWD(4); else RMS_BWD(8);
#undef RMS_BWD
  MDT_CHECK_LAUNCH();
  return 0;
}
extern "C" int mdt_rmsnorm_dw_finalize(const float* dw_partial, int n_partial, int cols, void* dw_bf16, float* dw_f32, cudaStream_t s) {
  launch_after(rmsnorm_dw_finalize_kernel, (cols + 31) / 32, 256, 0, s, dw_partial, n_partial, cols, (bf16*)dw_bf16, dw_f32);
  MDT_CHECK_LAUNCH();
  return 0;
}
extern "C" int mdt_rope(const void* x, void* y, const int* positions, int tokens, int heads, int head_dim, float theta,
                        int inverse, cudaStream_t s) {
  if (tokens == 0) return 0;
  const int vec = head_dim % 16 == 0 && ((reinterpret_cast<uintptr_t>(x) | reinterpret_cast<uintptr_t>(y)) & 15) == 0;
  const int work = vec ? heads * (head_dim / 16) : heads * (head_dim / 2);          // threads that have something to do
  const int threads = work <= 64 ? 64 : (work <= 128 ? 128 : 256);
  launch_after(rope_kernel, tokens, threads, (head_dim / 2) * 2 * sizeof(float), s, (const bf16*)x, (bf16*)y, positions, tokens, heads, head_dim, log2f(theta), inverse, vec);
  MDT_CHECK_LAUNCH();
  return 0;
}
extern "C" int mdt_swiglu_fwd(const void* g, const void* u, void* h, long long n, cudaStream_t s) {
  if (n % 8 != 0) return -1;
  if (n == 0) return 0;
  launch_after(swiglu_fwd_kernel, grid_for(n / 8, 256), 256, 0, s, (const uint4*)g, (const uint4*)u, (uint4*)h, n / 8);
  MDT_CHECK_LAUNCH();
  return 0;
}
extern "C" int mdt_copy_rows_used(const void* src, void* dst, long long n, const int* rows_used, long long cols, cudaStream_t s) {
  if (n % 8 != 0 || cols % 8 != 0 || rows_used == nullptr) return -1;
  if (n == 0) return 0;
  launch_after(copy_rows_used_kernel, grid_for(n / 8, 256), 256, 0, s, (const uint4*)src, (uint4*)dst, n / 8, rows_used, cols / 8);
  MDT_CHECK_LAUNCH();
  return 0;
}
extern "C" int mdt_embedding(const void* table, const long long* ids, void* out, int tokens, int cols, cudaStream_t s) {
  if (cols % 8 != 0) return -1;
  if (tokens == 0) return 0;
  launch_after(embedding_kernel, tokens, 128, 0, s, (const bf16*)table, ids, (bf16*)out, cols);
  MDT_CHECK_LAUNCH();
  return 0;
}
extern "C" void mdt_embedding_bwd_scratch(int tokens, int rows, int cols, long long* ints, long long* floats) {
  *ints = (long long)tokens + 3ll * rows + 1;
  *floats = (long long)(tokens / (EMB_LIST + 1)) * cols;       // ids with more tokens than a list takes
}
extern "C" int mdt_embedding_bwd(const void* dout, const long long* ids, void* dtable, int table_fp32, int add, int* scratch, float* sums, int tokens, int rows, int cols,
                                 cudaStream_t s) {
  if (cols % 8 != 0) return -1;
  if (tokens == 0) return 0;
  int *next = scratch, *head = next + tokens, *count = head + rows, *sum_row = count + rows, *sum_rows = sum_row + rows;
  if (cudaMemsetAsync(head, 0xff, (3 * (size_t)rows + 1) * sizeof(int), s) != cudaSuccess) return -2;
  const int late = tokens / (EMB_LIST + 1);
  launch_after(embedding_list_kernel, (tokens + 255) / 256, 256, 0, s, ids, next, head, count, sum_row, sum_rows, (float4*)sums, (long long)late * cols / 4, tokens);
  MDT_CHECK_LAUNCH();
  if (late > 0) {
    launch_after(embedding_late_kernel, dim3((tokens + EMB_LATE - 1) / EMB_LATE, (cols + 2047) / 2048), 256, 0, s, (const bf16*)dout, ids, next, sum_row, sums, tokens, cols);
    MDT_CHECK_LAUNCH();
  }
  if (table_fp32) launch_after(embedding_bwd_kernel<true>, tokens, 256, 0, s, (const bf16*)dout, ids, next, head, sum_row, sums, dtable, cols, add);
  else launch_after(embedding_bwd_kernel<false>, tokens, 256, 0, s, (const bf16*)dout, ids, next, head, sum_row, sums, dtable, cols, add);
  MDT_CHECK_LAUNCH();
  return 0;
}
extern "C" int mdt_adapter_pack(const void* A1, const void* A3, float s1, float s3, const void* B1, const void* B3, void* A13, void* B1p, void* B3p, int E, int H, int F,
                                int r, cudaStream_t s) {
  if (r < 4 || r % 4 != 0) return -1;
  const int strips = (F + ADAPTER_COLS - 1) / ADAPTER_COLS;
  const long long stretch = ((long long)E * H * r / 4 + 255) / 256;
  launch_after(adapter_pack_kernel, E * strips + (int)(stretch < 1024 ? stretch : 1024), 256, 0, s, (const bf16*)A1, (const bf16*)A3, s1, s3, (const bf16*)B1, (const bf16*)B3, (bf16*)A13,
                                                                                        (bf16*)B1p, (bf16*)B3p, E, H, F, r);
  MDT_CHECK_LAUNCH();
  return 0;
}
extern "C" int mdt_cross_entropy(void* logits, const long long* labels, float* loss_sum, float* count, int rows, int vocab,
                                 long long ld, int ignore_index, float grad_scale, cudaStream_t s) {
  if (vocab % 8 != 0 || ld % 8 != 0) return -1;
  if (rows == 0) return 0;
  const int smem = vocab * 2;
  static int configured = 0;
  if (smem > 48 * 1024 && configured < smem) {
    if (cudaFuncSetAttribute(cross_entropy_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, smem) != cudaSuccess) return -2;
    configured = smem;
  }
  launch_after(count_labels_kernel, grid_for(rows, 256, 64), 256, 0, s, labels, rows, ignore_index, count);
  MDT_CHECK_LAUNCH();
  launch_after(cross_entropy_kernel, rows, 512, smem, s, (bf16*)logits, labels, loss_sum, count, vocab, ld, ignore_index, grad_scale);
  MDT_CHECK_LAUNCH();
  return 0;
}
extern "C" int mdt_adamw(const MdtAdamTensor* tensors_device, int num_tensors, long long max_n, float lr, float beta1, float beta2,
                         float eps, float weight_decay, float bc1, float bc2, float grad_scale, const float* grad_scale_dev, cudaStream_t s) {
  if (num_tensors == 0) return 0;
  dim3 grid(grid_for((max_n + 7) / 8, 256, -16), num_tensors);
  launch_after(adamw_kernel, grid, 256, 0, s, tensors_device, lr, beta1, beta2, eps, weight_decay, 1.0f / bc1, 1.0f / bc2, grad_scale, grad_scale_dev);
  MDT_CHECK_LAUNCH();
  return 0;
}
extern "C" int mdt_multi_add(const MdtMultiAdd* a, cudaStream_t s) {
  if (a->count < 1) return 0;
  if (a->count > MDT_MULTI_ADD_MAX) return -1;
  long long max_n = 0;
  for (int i = 0; i < a->count; ++i) max_n = a->n[i] > max_n ? a->n[i] : max_n;
  if (max_n == 0) return 0;
  dim3 grid(grid_for(max_n, 256, -4), a->count);
  launch_after(multi_add_kernel, grid, 256, 0, s, *a);
  MDT_CHECK_LAUNCH();
  return 0;
}
extern "C" int mdt_sumsq(const void* x, long long n, int fp32, float* out_accum, cudaStream_t s) {
  if (n == 0) return 0;
  launch_after(sumsq_kernel, grid_for(n, 256 * 8, -4), 256, 0, s, x, n, fp32, out_accum);
  MDT_CHECK_LAUNCH();
  return 0;
}
extern "C" int mdt_axpby(void* y, const void* x, long long n, float a, float b, int y_fp32, int x_fp32, cudaStream_t s) {
  if (n == 0) return 0;
  launch_after(axpby_kernel, grid_for(n, 256 * 4), 256, 0, s, y, x, n, a, b, y_fp32, x_fp32);
  MDT_CHECK_LAUNCH();
  return 0;
}
