// Gated DeltaNet layers: a/b gate projection, fused causal conv(4) + SiLU + q/k L2 norm with the conv
// state carry, and the 128x128 fp32 recurrent-state update with the gated RMSNorm, over ragged
// sequences. Replaces kernels::gdn_ab, gdn_conv and gdn_recurrence of the reference
// (src/kernels/kernels.h:184-228, src/kernels/gdn.cu). State layouts (reference docs/FORMAT.md 3.2):
// recurrent fp32 [slot][gdn_layer][v_head][128 dv][128 dk]; conv bf16 [slot][gdn_layer][3][conv_dim],
// tap 0 oldest.
#include <algorithm>
#include <type_traits>

#include "common.cuh"
#include "host_util.h"
#include "tcgen05.cuh"

namespace q38 {
extern int g_chunk_scan_tensor_cores;  // 1: the chunk scan runs its products on the tensor cores
namespace {

constexpr int kDk = 128, kDv = 128;

// ---------------------------------------------------------------------------------------------------
// gdn_ab: ab[m][j] = rs[m] * sum_k xbf[m][k] * w[j][k]  (fp32; rows j < nv are b, the rest a).
// One CTA per (16 TM tokens, 8 TN weight rows); the sixteen warps take the 32-wide k blocks in turn and their partial sums
// meet in shared memory, added in warp order. Products on mma.sync m16n8k16 (bf16 products are exact in fp32). The order of
// the contraction index is free, so a lane takes 16 contiguous bytes of its token row and of its weight row per k block and
// they are two k16 steps of both operands as they stand: no shared memory, no ldmatrix.
// Bound by the round trips to L2: every load of a warp's k blocks is independent of the others. One tile per warp up to 256
// tokens (as many CTAs as possible), two by two above, where the re-reads of x and w through L2 count.
// 96 rows, hidden 5120: 1531 tokens 144 us on the CUDA cores, 27 us now; 64 tokens 13 and 8 us.
// ---------------------------------------------------------------------------------------------------
constexpr int kAbWarps = 16;
// 16 bytes of global memory, zero where `live` is false; volatile, so that a batch of them is issued as written
__device__ __forceinline__ uint4 load16_if(const uint4* p, bool live) {
  uint4 v;
  asm volatile(
      "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %5, 0;\n\tmov.u32 %0, 0;\n\tmov.u32 %1, 0;\n\tmov.u32 %2, 0;\n\tmov.u32 %3, 0;\n\t"
      "@p ld.global.v4.u32 {%0,%1,%2,%3}, [%4];\n\t}"
      : "=&r"(v.x), "=&r"(v.y), "=&r"(v.z), "=&r"(v.w)
      : "l"(p), "r"(int(live))
      : "memory");
  return v;
}
template <int TM, int TN>
__global__ void __launch_bounds__(kAbWarps * 32) gdn_ab_kernel(const __nv_bfloat16* __restrict__ xbf, int m, int hidden,
                                                               const __nv_bfloat16* __restrict__ w, int rows,
                                                               const float* __restrict__ partials_in, float eps,
                                                               float* __restrict__ ab_out) {
  // The weights are written by no kernel: their lines are on the way to L2 while the previous kernel still runs.
  for (int i = threadIdx.x; i < 8 * TN * (hidden / 64); i += kAbWarps * 32) {
    const int j = blockIdx.x * (8 * TN) + i / (hidden / 64);
    if (blockIdx.y == 0 && j < rows)
      asm volatile("prefetch.global.L2 [%0];" ::"l"(w + (size_t)j * hidden + 64 * (i % (hidden / 64))));
  }
  pdl_wait();               // everything written by earlier kernels of the stream is visible from here on
  pdl_launch_dependents();  // the next kernel may be scheduled now; it holds its own dependent work back the same way
  __shared__ float red[kAbWarps][TM * 16][TN * 8 + 1];
  __shared__ float rs_sm[TM * 16];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, g = lane >> 2, t = lane & 3;
  const int j0 = blockIdx.x * (8 * TN), m0 = blockIdx.y * (16 * TM);
  const uint4* xr[TM][2];
  const uint4* wr[TN];
#pragma unroll
  for (int i = 0; i < TM; ++i)
#pragma unroll
    for (int h = 0; h < 2; ++h)
      xr[i][h] = reinterpret_cast<const uint4*>(xbf + (size_t)min(m0 + 16 * i + 8 * h + g, m - 1) * hidden) + t;
#pragma unroll
  for (int j = 0; j < TN; ++j) wr[j] = reinterpret_cast<const uint4*>(w + (size_t)min(j0 + 8 * j + g, rows - 1) * hidden) + t;
  float acc[TM][TN][4];
#pragma unroll
  for (int i = 0; i < TM; ++i)
#pragma unroll
    for (int j = 0; j < TN; ++j)
#pragma unroll
      for (int c = 0; c < 4; ++c) acc[i][j][c] = 0.0f;
  constexpr int kBatch = TM * TN == 1 ? 5 : 3;  // k blocks requested together (hidden 5120: two round trips per warp)
  const int nkb = hidden / 32;
  for (int k0 = warp; k0 < nkb; k0 += kAbWarps * kBatch) {
    uint4 x[kBatch][TM][2], wv[kBatch][TN];
#pragma unroll
    for (int u = 0; u < kBatch; ++u) {
      const int kb = k0 + kAbWarps * u;
      const bool live = kb < nkb;
#pragma unroll
      for (int i = 0; i < TM; ++i)
#pragma unroll
        for (int h = 0; h < 2; ++h) x[u][i][h] = load16_if(xr[i][h] + 4 * kb, live);
#pragma unroll
      for (int j = 0; j < TN; ++j) wv[u][j] = load16_if(wr[j] + 4 * kb, live);
    }
#pragma unroll
    for (int u = 0; u < kBatch; ++u)
#pragma unroll
      for (int i = 0; i < TM; ++i) {
        const uint32_t a0[4] = {x[u][i][0].x, x[u][i][1].x, x[u][i][0].y, x[u][i][1].y};
        const uint32_t a1[4] = {x[u][i][0].z, x[u][i][1].z, x[u][i][0].w, x[u][i][1].w};
#pragma unroll
        for (int j = 0; j < TN; ++j) {
          mma_bf16_16816(acc[i][j], a0, wv[u][j].x, wv[u][j].y);
          mma_bf16_16816(acc[i][j], a1, wv[u][j].z, wv[u][j].w);
        }
      }
  }
#pragma unroll
  for (int i = 0; i < TM; ++i)
#pragma unroll
    for (int j = 0; j < TN; ++j)
#pragma unroll
      for (int c = 0; c < 4; ++c) red[warp][16 * i + g + 8 * (c >> 1)][8 * j + 2 * t + (c & 1)] = acc[i][j][c];
  row_scales_to_smem(partials_in ? partials_in + (size_t)m0 * (hidden / 128) : nullptr, min(16 * TM, m - m0), 16 * TM, hidden, eps,
                     rs_sm, tid, kAbWarps * 32);
  __syncthreads();
  for (int i = tid; i < TM * 16 * TN * 8; i += kAbWarps * 32) {
    const int r = i / (TN * 8), j = i % (TN * 8);
    if (m0 + r < m && j0 + j < rows) {
      float total = 0.0f;
#pragma unroll
      for (int wi = 0; wi < kAbWarps; ++wi) total += red[wi][r][j];
      ab_out[(size_t)(m0 + r) * rows + j0 + j] = total * rs_sm[r];
    }
  }
}

// ---------------------------------------------------------------------------------------------------
// gdn_conv: depthwise causal conv (width 4) + SiLU over the [q | k | v] channels; q/k heads are
// L2-normalised (x * rsqrt(sum x^2 + 1e-6)), q additionally scaled by 1/sqrt(128).
// Any alignment: one CTA per (128-channel head block, 1 or 8 consecutive tokens). The three previous inputs of a channel
// come from the same chunk's earlier rows of `proj`, or from the conv state for the first tokens of a
// sequence's chunk. A second small kernel then rolls the conv state forward by the chunk.
// ---------------------------------------------------------------------------------------------------
__global__ void __launch_bounds__(128) gdn_conv_kernel(const __nv_bfloat16* __restrict__ proj, int ld_proj,
                                                       const float* __restrict__ conv_w, float* __restrict__ qkv,
                                                       int conv_dim, int key_dim, int layer, int num_layers,
                                                       __nv_bfloat16* __restrict__ conv_state,
                                                       const int* __restrict__ seq_start,
                                                       const int* __restrict__ seq_slot,
                                                       const int* __restrict__ tok_seq, int roll_state, int num_tokens,
                                                       int tokens_per_cta, int one_token_each) {
  pdl_wait();               // everything written by earlier kernels of the stream is visible from here on
  pdl_launch_dependents();  // the next kernel may be scheduled now; it holds its own dependent work back the same way
  __shared__ float red[4];
  const int c = blockIdx.x * 128 + threadIdx.x;
  const float4 w = *reinterpret_cast<const float4*>(conv_w + (size_t)c * 4);
  const int m_end = min(num_tokens, (int(blockIdx.y) + 1) * tokens_per_cta);
  for (int m = blockIdx.y * tokens_per_cta; m < m_end; ++m) {
    // one_token_each (a decode batch: every sequence has exactly one token, so token m is sequence m's and the first of
    // its run): two dependent loads fewer on the way to the taps
    const int b = one_token_each ? m : tok_seq[m];
    const int i = one_token_each ? 0 : m - seq_start[b];  // index of the token inside its sequence's chunk
    __nv_bfloat16* st = conv_state + ((size_t)seq_slot[b] * num_layers + layer) * 3 * conv_dim;
    float x[4];
    __nv_bfloat16 xb[4];
#pragma unroll
    for (int j = 0; j < 4; ++j) {  // x[j] = input 3 - j steps back
      const int back = 3 - j;
      xb[j] = back <= i ? proj[(size_t)(m - back) * ld_proj + c] : st[(size_t)(3 + i - back) * conv_dim + c];
      x[j] = __bfloat162float(xb[j]);
    }
    if (roll_state) {  // one token per sequence: this thread is the only reader of its channel's taps, so it also rolls them
      st[c] = xb[1];
      st[(size_t)conv_dim + c] = xb[2];
      st[(size_t)2 * conv_dim + c] = xb[3];
    }
    float acc = 0.0f;
    acc += w.x * x[0];
    acc += w.y * x[1];
    acc += w.z * x[2];
    acc += w.w * x[3];
    float y = silu_f(acc);
    if (c < 2 * key_dim) {  // block-uniform: the 128 channels of a CTA are one q or k head
      const float ss = warp_sum(y * y);
      __syncthreads();  // the previous token's readers of red[] are done
      if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = ss;
      __syncthreads();
      const float total = red[0] + red[1] + red[2] + red[3];
      y *= 1.0f / sqrtf(total + 1e-6f);
      if (c < key_dim) y *= 0.08838834764831845f;  // 1 / sqrt(128)
    }
    qkv[(size_t)m * conv_dim + c] = y;
  }
}

// The same by vectors, where proj, qkv and the conv state allow 8- and 16-byte accesses: a warp takes the 128 channels of a
// head, four per lane (the norm is a warp sum, no barrier), of TOK consecutive tokens. TOK = 4, prefill-sized steps: the
// seven input rows of the window and the tokens' sequence data are requested before anything is computed; taps that a
// sequence's first three tokens take from the conv state are fetched on demand; the state is not rolled here. TOK = 1: a
// token's four taps come from the rows before it or from the state, which is rolled where every sequence has one token.
// Bound by latency (two round trips and TOK norms per warp): 1000 tokens of 10,240 channels (61 MB in and out) 35 us with one
// channel per thread, 22 us now; 512 tokens 20 and 13 us; 256 tokens of 4096 channels 7.0 and 6.4 us (8.2 with eight tokens per
// warp, which were slower at every size; two: 23.5 us at 1000 tokens).
constexpr int kConvBlock = 4;
constexpr int kConvWarps = 8;
__device__ __forceinline__ float4 bf16x4_to_float4(uint2 v) {
  return make_float4(__uint_as_float(v.x << 16), __uint_as_float(v.x & 0xffff0000u), __uint_as_float(v.y << 16),
                     __uint_as_float(v.y & 0xffff0000u));
}
template <int TOK>
__global__ void __launch_bounds__(kConvWarps * 32) gdn_conv_vec_kernel(
    const __nv_bfloat16* __restrict__ proj, int ld_proj, const float* __restrict__ conv_w, float* __restrict__ qkv, int conv_dim,
    int key_dim, int layer, int num_layers, __nv_bfloat16* __restrict__ conv_state, const int* __restrict__ seq_start,
    const int* __restrict__ seq_slot, const int* __restrict__ tok_seq, int num_tokens, int roll_state, int one_token_each) {
  pdl_wait();               // everything written by earlier kernels of the stream is visible from here on
  pdl_launch_dependents();  // the next kernel may be scheduled now; it holds its own dependent work back the same way
  const int lane = threadIdx.x & 31, c = blockIdx.x * 128 + 4 * lane;
  const int m0 = (blockIdx.y * kConvWarps + (threadIdx.x >> 5)) * TOK;
  if (m0 >= num_tokens) return;
  const int nt = min(TOK, num_tokens - m0);
  float4 w[4];  // taps of channel c + i
#pragma unroll
  for (int i = 0; i < 4; ++i) w[i] = *reinterpret_cast<const float4*>(conv_w + (size_t)(c + i) * 4);
  auto load4 = [](const __nv_bfloat16* p) { return *reinterpret_cast<const uint2*>(p); };
  auto finish = [&](const float4 (&x)[4], int m) {  // x[j]: input 3 - j steps back
    float y[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      auto at = [&](int j) { return i == 0 ? x[j].x : i == 1 ? x[j].y : i == 2 ? x[j].z : x[j].w; };
      float acc = 0.0f;
      acc += w[i].x * at(0);
      acc += w[i].y * at(1);
      acc += w[i].z * at(2);
      acc += w[i].w * at(3);
      y[i] = silu_f(acc);
    }
    if (c < 2 * key_dim) {  // warp-uniform: the 128 channels of a warp are one q or k head
      const float total = warp_sum((y[0] * y[0] + y[1] * y[1]) + (y[2] * y[2] + y[3] * y[3]));
      float r = 1.0f / sqrtf(total + 1e-6f);
      const float scale = c < key_dim ? 0.08838834764831845f : 1.0f;  // 1 / sqrt(128)
#pragma unroll
      for (int i = 0; i < 4; ++i) y[i] = y[i] * r * scale;
    }
    *reinterpret_cast<float4*>(qkv + (size_t)m * conv_dim + c) = make_float4(y[0], y[1], y[2], y[3]);
  };
  if constexpr (TOK == 1) {
    const int b = one_token_each ? m0 : tok_seq[m0];
    const int i = one_token_each ? 0 : m0 - seq_start[b];  // index of the token inside its sequence's chunk
    __nv_bfloat16* st = conv_state + ((size_t)seq_slot[b] * num_layers + layer) * 3 * conv_dim + c;
    uint2 raw[4];
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const int back = 3 - j;
      raw[j] = load4(back <= i ? proj + (size_t)(m0 - back) * ld_proj + c : st + (size_t)(3 + i - back) * conv_dim);
    }
    if (roll_state) {  // one token per sequence: this lane is the only reader of its channels' taps
#pragma unroll
      for (int j = 0; j < 3; ++j) *reinterpret_cast<uint2*>(st + (size_t)j * conv_dim) = raw[j + 1];
    }
    const float4 x[4] = {bf16x4_to_float4(raw[0]), bf16x4_to_float4(raw[1]), bf16x4_to_float4(raw[2]), bf16x4_to_float4(raw[3])};
    finish(x, m0);
  } else {
    uint2 win[TOK + 3];  // inputs of rows m0 - 3 + k
#pragma unroll
    for (int k = 0; k < TOK + 3; ++k) {
      const int row = m0 - 3 + k;
      win[k] = row >= 0 && row < num_tokens ? load4(proj + (size_t)row * ld_proj + c) : make_uint2(0u, 0u);
    }
    int seq[TOK], idx[TOK];
#pragma unroll
    for (int t = 0; t < TOK; ++t) seq[t] = t < nt ? tok_seq[m0 + t] : 0;
#pragma unroll
    for (int t = 0; t < TOK; ++t) idx[t] = t < nt ? m0 + t - seq_start[seq[t]] : 3;  // index inside its sequence's chunk
#pragma unroll
    for (int t = 0; t < TOK; ++t) {
      if (t >= nt) break;
      uint2 raw[4] = {win[t], win[t + 1], win[t + 2], win[t + 3]};
      if (idx[t] < 3) {  // the sequence's chunk starts here: older inputs come from its conv state
        const __nv_bfloat16* st = conv_state + ((size_t)seq_slot[seq[t]] * num_layers + layer) * 3 * conv_dim + c;
#pragma unroll
        for (int j = 0; j < 3; ++j)
          if (3 - j > idx[t]) raw[j] = load4(st + (size_t)(idx[t] + j) * conv_dim);
      }
      const float4 x[4] = {bf16x4_to_float4(raw[0]), bf16x4_to_float4(raw[1]), bf16x4_to_float4(raw[2]), bf16x4_to_float4(raw[3])};
      finish(x, m0 + t);
    }
  }
}

// The same at any alignment for prefill-sized steps: one CTA per (128-channel head block, 8 consecutive tokens), state not rolled here.
// A thread requests its channel's eleven inputs of the window (rows m0 - 3 .. m0 + 7 of `proj`) and the tokens' sequence
// data before it computes anything, so the CTA pays one round trip to memory instead of one per token; the taps a
// sequence's first three tokens take from the conv state are fetched on demand. The arithmetic per token is that of
// gdn_conv_kernel, in the same order.
constexpr int kConvWindow = 8;
__global__ void __launch_bounds__(128) gdn_conv_block_kernel(const __nv_bfloat16* __restrict__ proj, int ld_proj,
                                                             const float* __restrict__ conv_w, float* __restrict__ qkv,
                                                             int conv_dim, int key_dim, int layer, int num_layers,
                                                             const __nv_bfloat16* __restrict__ conv_state,
                                                             const int* __restrict__ seq_start,
                                                             const int* __restrict__ seq_slot,
                                                             const int* __restrict__ tok_seq, int num_tokens) {
  pdl_wait();               // everything written by earlier kernels of the stream is visible from here on
  pdl_launch_dependents();  // the next kernel may be scheduled now; it holds its own dependent work back the same way
  __shared__ float red[kConvWindow][4];
  const int c = blockIdx.x * 128 + threadIdx.x;
  const int m0 = blockIdx.y * kConvWindow;
  const int nt = min(kConvWindow, num_tokens - m0);
  const float4 w = *reinterpret_cast<const float4*>(conv_w + (size_t)c * 4);
  float win[kConvWindow + 3];  // inputs of rows m0 - 3 + k
#pragma unroll
  for (int k = 0; k < kConvWindow + 3; ++k) {
    const int row = m0 - 3 + k;
    win[k] = row >= 0 && row < num_tokens ? __bfloat162float(proj[(size_t)row * ld_proj + c]) : 0.0f;
  }
  int seq[kConvWindow], idx[kConvWindow];
#pragma unroll
  for (int t = 0; t < kConvWindow; ++t) seq[t] = t < nt ? tok_seq[m0 + t] : 0;
#pragma unroll
  for (int t = 0; t < kConvWindow; ++t) idx[t] = t < nt ? m0 + t - seq_start[seq[t]] : 3;  // index inside its sequence's chunk
  float y[kConvWindow];
#pragma unroll
  for (int t = 0; t < kConvWindow; ++t) {
    float x[4];
#pragma unroll
    for (int j = 0; j < 4; ++j) x[j] = win[t + j];  // input 3 - j steps back
    if (t < nt && idx[t] < 3) {  // the sequence's chunk starts here: older inputs come from its conv state
      const __nv_bfloat16* st = conv_state + ((size_t)seq_slot[seq[t]] * num_layers + layer) * 3 * conv_dim;
#pragma unroll
      for (int j = 0; j < 3; ++j) {
        const int back = 3 - j;
        if (back > idx[t]) x[j] = __bfloat162float(st[(size_t)(3 + idx[t] - back) * conv_dim + c]);
      }
    }
    float acc = 0.0f;
    acc += w.x * x[0];
    acc += w.y * x[1];
    acc += w.z * x[2];
    acc += w.w * x[3];
    y[t] = silu_f(acc);
  }
  if (c < 2 * key_dim) {  // block-uniform: the 128 channels of a CTA are one q or k head
#pragma unroll
    for (int t = 0; t < kConvWindow; ++t) {
      const float ss = warp_sum(y[t] * y[t]);
      if ((threadIdx.x & 31) == 0) red[t][threadIdx.x >> 5] = ss;
    }
    __syncthreads();
#pragma unroll
    for (int t = 0; t < kConvWindow; ++t) {
      const float total = red[t][0] + red[t][1] + red[t][2] + red[t][3];
      y[t] *= 1.0f / sqrtf(total + 1e-6f);
      if (c < key_dim) y[t] *= 0.08838834764831845f;  // 1 / sqrt(128)
    }
  }
#pragma unroll
  for (int t = 0; t < kConvWindow; ++t)
    if (t < nt) qkv[(size_t)(m0 + t) * conv_dim + c] = y[t];
}

__global__ void __launch_bounds__(128) gdn_conv_state_kernel(const __nv_bfloat16* __restrict__ proj, int ld_proj,
                                                             int conv_dim, int layer, int num_layers,
                                                             __nv_bfloat16* __restrict__ conv_state,
                                                             const int* __restrict__ seq_start,
                                                             const int* __restrict__ seq_slot) {
  pdl_wait();               // everything written by earlier kernels of the stream is visible from here on
  pdl_launch_dependents();  // the next kernel may be scheduled now; it holds its own dependent work back the same way
  const int c = blockIdx.x * 128 + threadIdx.x, b = blockIdx.y;
  const int s = seq_start[b], n = seq_start[b + 1] - s;
  if (n <= 0) return;
  __nv_bfloat16* st = conv_state + ((size_t)seq_slot[b] * num_layers + layer) * 3 * conv_dim;
  __nv_bfloat16 old[3], nw[3];
#pragma unroll
  for (int t = 0; t < 3; ++t) old[t] = st[(size_t)t * conv_dim + c];
#pragma unroll
  for (int t = 0; t < 3; ++t) {  // history = [old0 old1 old2 x0 .. x(n-1)], keep its last three
    const int idx = n + t;
    nw[t] = idx < 3 ? old[idx] : proj[(size_t)(s + idx - 3) * ld_proj + c];
  }
#pragma unroll
  for (int t = 0; t < 3; ++t) st[(size_t)t * conv_dim + c] = nw[t];
}

// ---------------------------------------------------------------------------------------------------
// gdn_recurrence: one CTA per (v head, sequence). The 128x128 fp32 state lives in registers for the
// whole chunk: 16 warps x 8 rows, a lane owns 4 consecutive columns of each row, so a row is one
// coalesced 512-byte access. Per token (reference src/kernels/gdn.cu:275-334, oracle
// src/ref/ops.cpp:210-240):
//   beta = sigmoid(b); decay = exp(A * softplus(a + dt_bias));
//   S *= decay; kv = S k; delta = beta (v - kv); S += delta k^T; o = S q;
//   out = bf16(o * rsqrt(mean(o^2) + eps) * norm_w * silu(z)).
// ---------------------------------------------------------------------------------------------------
constexpr int kRecWarps = 16;
constexpr int kRowsPerWarp = kDv / kRecWarps;

__global__ void __launch_bounds__(kRecWarps * 32, 1) gdn_recurrence_kernel(
    const float* __restrict__ qkv, int conv_dim, const float* __restrict__ ab, const float* __restrict__ A,
    const float* __restrict__ dt_bias, const __nv_bfloat16* __restrict__ z, int ld_z,
    const float* __restrict__ norm_w, float eps, __nv_bfloat16* __restrict__ out, int layer, int num_layers, int nk,
    int nv, float* __restrict__ recurrent, const int* __restrict__ seq_start, const int* __restrict__ seq_slot) {
  pdl_wait();               // everything written by earlier kernels of the stream is visible from here on
  pdl_launch_dependents();  // the next kernel may be scheduled now; it holds its own dependent work back the same way
  const int vh = blockIdx.x, b = blockIdx.y;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int s0 = seq_start[b], s1 = seq_start[b + 1];
  if (s1 <= s0) return;
  const int kh = vh / (nv / nk);
  float* S = recurrent + (((size_t)seq_slot[b] * num_layers + layer) * nv + vh) * kDv * kDk;
  const int row0 = warp * kRowsPerWarp;
  float4 st[kRowsPerWarp];
#pragma unroll
  for (int r = 0; r < kRowsPerWarp; ++r) st[r] = *reinterpret_cast<const float4*>(S + (size_t)(row0 + r) * kDk + 4 * lane);

  __shared__ float o_sm[kDv];
  __shared__ float red[kRecWarps];
  const float a_h = A[vh], dt_h = dt_bias[vh];
  const size_t q_off = (size_t)kh * kDk, k_off = (size_t)nk * kDk + (size_t)kh * kDk, v_off = (size_t)2 * nk * kDk + (size_t)vh * kDv;

  for (int m = s0; m < s1; ++m) {
    const float* row = qkv + (size_t)m * conv_dim;
    const float4 q4 = *reinterpret_cast<const float4*>(row + q_off + 4 * lane);
    const float4 k4 = *reinterpret_cast<const float4*>(row + k_off + 4 * lane);
    const float bb = ab[(size_t)m * 2 * nv + vh], aa = ab[(size_t)m * 2 * nv + nv + vh];
    const float beta = 1.0f / (1.0f + expf(-bb));
    const float xsp = aa + dt_h;
    const float sp = xsp > 20.0f ? xsp : log1pf(expf(xsp));
    const float decay = expf(a_h * sp);
    float ov[kRowsPerWarp];
#pragma unroll
    for (int r = 0; r < kRowsPerWarp; ++r) {
      float4 sv = st[r];
      sv.x *= decay;
      sv.y *= decay;
      sv.z *= decay;
      sv.w *= decay;
      const float kv = warp_sum(sv.x * k4.x + sv.y * k4.y + sv.z * k4.z + sv.w * k4.w);
      const float delta = beta * (row[v_off + row0 + r] - kv);
      sv.x += delta * k4.x;
      sv.y += delta * k4.y;
      sv.z += delta * k4.z;
      sv.w += delta * k4.w;
      st[r] = sv;
      ov[r] = warp_sum(sv.x * q4.x + sv.y * q4.y + sv.z * q4.z + sv.w * q4.w);
    }
    // gated RMSNorm over the 128 outputs of the head
    float ss = 0.0f;
#pragma unroll
    for (int r = 0; r < kRowsPerWarp; ++r) ss += ov[r] * ov[r];
    if (lane == 0) red[warp] = ss;
    if (lane < kRowsPerWarp) {
      float mine = ov[0];
#pragma unroll
      for (int r = 1; r < kRowsPerWarp; ++r)
        if (lane == r) mine = ov[r];
      o_sm[row0 + lane] = mine;
    }
    __syncthreads();
    if (threadIdx.x < kDv) {
      float total = 0.0f;
#pragma unroll
      for (int w = 0; w < kRecWarps; ++w) total += red[w];
      const float r = 1.0f / sqrtf(total / float(kDv) + eps);
      const int d = threadIdx.x;
      const float zz = __bfloat162float(z[(size_t)m * ld_z + (size_t)vh * kDv + d]);
      out[(size_t)m * nv * kDv + (size_t)vh * kDv + d] = __float2bfloat16_rn(o_sm[d] * r * norm_w[d] * silu_f(zz));
    }
    __syncthreads();
  }
#pragma unroll
  for (int r = 0; r < kRowsPerWarp; ++r) *reinterpret_cast<float4*>(S + (size_t)(row0 + r) * kDk + 4 * lane) = st[r];
}


// ---------------------------------------------------------------------------------------------------
// gdn_recurrence for decode batches (every sequence advances by at most one token): the step is a pure
// stream over the recurrent state (64 KB read + 64 KB written per (sequence, head), a few hundred FMAs per
// thread), so it is organised around the memory pipeline instead of one CTA per (sequence, head):
//   * one persistent CTA per SM walks the (sequence, head) items cta, cta + grid, ...;
//   * a producer warp brings each item's state and its token's q / k / v / z rows into a three-slot
//     shared-memory ring with 1-D bulk (TMA) copies, so up to three states per SM are in flight while
//     a fourth is being computed;
//   * 16 compute warps take the state into registers (a slot is handed back as soon as it has been read),
//     run exactly the arithmetic of gdn_recurrence_kernel for one token, and write the new state straight
//     from registers with 16-byte stores.
// ---------------------------------------------------------------------------------------------------
constexpr int kDecSlots = 3;
constexpr int kDecStateBytes = kDv * kDk * 4;
constexpr int kDecQOff = kDecStateBytes, kDecKOff = kDecQOff + 512, kDecVOff = kDecKOff + 512, kDecZOff = kDecVOff + 512;
constexpr int kDecSlotBytes = kDecStateBytes + 2048;
constexpr int kDecTxBytes = kDecStateBytes + 3 * 512 + 256;
constexpr int kDecSmemBytes = 128 + kDecSlots * kDecSlotBytes + 2 * (kDv + 2 * kRecWarps) * 4 + 2 * kDecSlots * 8 + 16;
constexpr int kDecThreads = (kRecWarps + 1) * 32;

__global__ void __launch_bounds__(kDecThreads, 1) gdn_recurrence_decode_kernel(
    const float* __restrict__ qkv, int conv_dim, const float* __restrict__ ab, const float* __restrict__ A,
    const float* __restrict__ dt_bias, const __nv_bfloat16* __restrict__ z, int ld_z,
    const float* __restrict__ norm_w, float eps, __nv_bfloat16* __restrict__ out, int layer, int num_layers, int nk,
    int nv, float* __restrict__ recurrent, const int* __restrict__ seq_start, const int* __restrict__ seq_slot,
    int num_seqs) {
  extern __shared__ uint8_t dec_smem_raw[];
  uint8_t* smem = dec_smem_raw + ((128 - (smem_u32(dec_smem_raw) & 127)) & 127);
  uint8_t* slots = smem;
  // outputs, partial sums of squares and the warps' wait results of an item: two sets used in turn, so that one barrier
  // per item is enough (a warp may start the next item while the others still read this one's set)
  float* o_sm_all = reinterpret_cast<float*>(smem + kDecSlots * kDecSlotBytes);
  float* red_all = o_sm_all + 2 * kDv;
  int* okf_all = reinterpret_cast<int*>(red_all + 2 * kRecWarps);
  uint64_t* full = reinterpret_cast<uint64_t*>(okf_all + 2 * kRecWarps);
  uint64_t* empty = full + kDecSlots;
  volatile int* abort_flag = reinterpret_cast<volatile int*>(empty + kDecSlots);  // [0] compute warps, [1] producer

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int items = num_seqs * nv;
  if (threadIdx.x == 0) {
    for (int s = 0; s < kDecSlots; ++s) {
      mbar_init(&full[s], 1);
      mbar_init(&empty[s], kRecWarps);
    }
    abort_flag[0] = 0;
    abort_flag[1] = 0;
    mbar_fence_init();
  }
  __syncthreads();

  if (warp == kRecWarps) {
    // ------------------------------ producer ------------------------------
    const uint64_t pol = policy_evict_first();
    uint32_t it = 0;
    bool waited = false;
    for (int item = blockIdx.x; item < items; item += gridDim.x) {
      const int b = item / nv, vh = item - b * nv;
      const int m = seq_start[b];
      if (seq_start[b + 1] <= m) continue;
      const int slot = it % kDecSlots;
      int ok = 1;
      if (lane == 0) {
        ok = (!abort_flag[0] && mbar_wait(&empty[slot], ((it / kDecSlots) & 1) ^ 1, 0x401)) ? 1 : 0;
        if (ok) mbar_expect_tx(&full[slot], kDecTxBytes);
        else abort_flag[1] = 1;
      }
      ok = __shfl_sync(0xffffffffu, ok, 0);
      if (!ok) break;
      uint8_t* dst = slots + (size_t)slot * kDecSlotBytes;
      const float* S = recurrent + (((size_t)seq_slot[b] * num_layers + layer) * nv + vh) * kDv * kDk;
      const float* row = qkv + (size_t)m * conv_dim;
      const int kh = vh / (nv / nk);
      if (lane < 4)
        bulk_g2s(dst + lane * (kDecStateBytes / 4), reinterpret_cast<const uint8_t*>(S) + lane * (kDecStateBytes / 4),
                 kDecStateBytes / 4, &full[slot], pol);
      if (!waited) {  // the state and the batch metadata are older than the previous kernel; the token rows may not be
        pdl_wait();
        waited = true;
      }
      if (lane == 4)
        bulk_g2s(dst + kDecQOff, row + (size_t)kh * kDk, 512, &full[slot], pol);
      else if (lane == 5)
        bulk_g2s(dst + kDecKOff, row + (size_t)nk * kDk + (size_t)kh * kDk, 512, &full[slot], pol);
      else if (lane == 6)
        bulk_g2s(dst + kDecVOff, row + (size_t)2 * nk * kDk + (size_t)vh * kDv, 512, &full[slot], pol);
      else if (lane == 7)
        bulk_g2s(dst + kDecZOff, z + (size_t)m * ld_z + (size_t)vh * kDv, 256, &full[slot], pol);
      __syncwarp();
      ++it;
    }
    return;
  }

  // ------------------------------ compute warps ------------------------------
  pdl_wait();
  pdl_launch_dependents();
  const int row0 = warp * kRowsPerWarp;
  const int tid = threadIdx.x;
  uint32_t it = 0;
  for (int item = blockIdx.x; item < items; item += gridDim.x) {
    const int b = item / nv, vh = item - b * nv;
    const int m = seq_start[b];
    if (seq_start[b + 1] <= m) continue;
    const int slot = it % kDecSlots;
    // scalars of this (token, head): requested before the wait so that their latency hides behind it
    const float bb = ab[(size_t)m * 2 * nv + vh], aa = ab[(size_t)m * 2 * nv + nv + vh];
    const float a_h = A[vh], dt_h = dt_bias[vh];
    const float nw = tid < kDv ? norm_w[tid] : 0.0f;
    float* S = recurrent + (((size_t)seq_slot[b] * num_layers + layer) * nv + vh) * kDv * kDk;
    // a wait that runs out marks the launch as failed; the warps leave the loop together below
    const bool ok = mbar_wait(&full[slot], (it / kDecSlots) & 1, 0x402);
    if (!ok) abort_flag[0] = 1;
    float* o_sm = o_sm_all + (it & 1u) * kDv;
    float* red = red_all + (it & 1u) * kRecWarps;
    int* okf = okf_all + (it & 1u) * kRecWarps;
    const uint8_t* src = slots + (size_t)slot * kDecSlotBytes;
    float4 st[kRowsPerWarp];
    float vv[kRowsPerWarp];
#pragma unroll
    for (int r = 0; r < kRowsPerWarp; ++r) {
      st[r] = *reinterpret_cast<const float4*>(src + (size_t)(row0 + r) * kDk * 4 + 16 * lane);
      vv[r] = *reinterpret_cast<const float*>(src + kDecVOff + 4 * (row0 + r));
    }
    const float4 q4 = *reinterpret_cast<const float4*>(src + kDecQOff + 16 * lane);
    const float4 k4 = *reinterpret_cast<const float4*>(src + kDecKOff + 16 * lane);
    const float zz = tid < kDv ? __bfloat162float(*reinterpret_cast<const __nv_bfloat16*>(src + kDecZOff + 2 * tid)) : 0.0f;
    __syncwarp();
    if (lane == 0) mbar_arrive(&empty[slot]);  // everything of the slot is in registers now

    const float beta = 1.0f / (1.0f + expf(-bb));
    const float xsp = aa + dt_h;
    const float sp = xsp > 20.0f ? xsp : log1pf(expf(xsp));
    const float decay = expf(a_h * sp);
    float ov[kRowsPerWarp];
#pragma unroll
    for (int r = 0; r < kRowsPerWarp; ++r) {
      float4 sv = st[r];
      sv.x *= decay;
      sv.y *= decay;
      sv.z *= decay;
      sv.w *= decay;
      const float kv = warp_sum(sv.x * k4.x + sv.y * k4.y + sv.z * k4.z + sv.w * k4.w);
      const float delta = beta * (vv[r] - kv);
      sv.x += delta * k4.x;
      sv.y += delta * k4.y;
      sv.z += delta * k4.z;
      sv.w += delta * k4.w;
      st[r] = sv;
      ov[r] = warp_sum(sv.x * q4.x + sv.y * q4.y + sv.z * q4.z + sv.w * q4.w);
    }
    if (ok) {
#pragma unroll
      for (int r = 0; r < kRowsPerWarp; ++r)
        *reinterpret_cast<float4*>(S + (size_t)(row0 + r) * kDk + 4 * lane) = st[r];
    }
    // gated RMSNorm over the 128 outputs of the head
    float ss = 0.0f;
#pragma unroll
    for (int r = 0; r < kRowsPerWarp; ++r) ss += ov[r] * ov[r];
    if (lane == 0) {
      red[warp] = ss;
      okf[warp] = ok ? 1 : 0;
    }
    if (lane < kRowsPerWarp) {
      float mine = ov[0];
#pragma unroll
      for (int r = 1; r < kRowsPerWarp; ++r)
        if (lane == r) mine = ov[r];
      o_sm[row0 + lane] = mine;
    }
    named_bar_sync(1, kRecWarps * 32);
    // a wait of any warp ran out: all of them leave after this item (the item's set was written before the barrier, so
    // every warp reads the same value)
    int stop = 0;
#pragma unroll
    for (int w = 0; w < kRecWarps; ++w) stop |= okf[w] ^ 1;
    if (tid < kDv && ok) {
      float total = 0.0f;
#pragma unroll
      for (int w = 0; w < kRecWarps; ++w) total += red[w];
      const float r = 1.0f / sqrtf(total / float(kDv) + eps);
      out[(size_t)m * nv * kDv + (size_t)vh * kDv + tid] = __float2bfloat16_rn(o_sm[tid] * r * nw * silu_f(zz));
    }
    if (stop) break;
    ++it;
  }
}


// ---------------------------------------------------------------------------------------------------
// gdn_recurrence for prefill chunks: the chunked (WY) form of the gated delta rule. The token recurrence
//     S_t = a_t S_{t-1} + beta_t (v_t - a_t S_{t-1} k_t) k_t^T,   o_t = S_t q_t        (S is [dv][dk])
// is sequential in t; over a chunk of C = 64 tokens with lg_i = sum_{t<=i} log a_t it is equivalent to
//     A[i][j] = beta_i e^{lg_i - lg_j} (k_i . k_j)  (j < i)          P[i][j] = e^{lg_i - lg_j} (q_i . k_j)  (j <= i)
//     (I + A) U0 = diag(beta) V         (I + A) W = diag(beta e^{lg}) K                       (prep, no state)
//     U = U0 - W S_0^T      O = diag(e^{lg}) Q S_0^T + P U      S_C = e^{lg_C} S_0 + U^T diag(e^{lg_C - lg}) K
// so everything that does not touch the state is computed for all chunks in parallel (gdn_chunk_prep_kernel,
// one CTA per (chunk, up to three v heads of a k head, sequence)), and the sequential part is four small matrix products per chunk with
// the state resident in shared memory (gdn_chunk_scan_kernel, one CTA per (v head, sequence)). All arithmetic is fp32 (the
// scan's products on the tensor cores in three bf16 terms a factor); the log decays are added token by token, so their sums never
// rise and every exponent is <= 0: nothing overflows however strong the decay is.
// Tokens beyond a sequence's ragged tail are treated as beta = 0, log a = 0, q = k = v = 0 (no effect).
// Scratch per (chunk slot, v head): U0 [64][128], W [64][128], P [64][64], lg [64] floats; the chunk slots of
// sequence b start at (seq_start[b] - seq_start[0]) / 64 + b (never fewer than the chunks before it, so slots do not collide).
// ---------------------------------------------------------------------------------------------------
constexpr int kCh = 64;
constexpr int kLd = 132;   // padded row stride (floats) of 128-wide shared tiles: 16-byte reads of 8 rows hit 32 banks
constexpr int kLdP = 68;   // the same for 64-wide tiles
constexpr int kChunkFloats = 2 * kCh * 128 + kCh * kCh + kCh;
constexpr int kChunkThreads = 512;

__device__ __forceinline__ void token_gates(const float* __restrict__ ab, int m, int nv, int vh, float a_h, float dt_h,
                                            float& beta, float& log_decay) {
  const float bb = ab[(size_t)m * 2 * nv + vh], aa = ab[(size_t)m * 2 * nv + nv + vh];
  beta = 1.0f / (1.0f + expf(-bb));
  const float xsp = aa + dt_h;
  const float sp = xsp > 20.0f ? xsp : log1pf(expf(xsp));
  log_decay = a_h * sp;
}

// Rows [0, nc) of a [.][128] fp32 row block -> shared [64][kLd], rows >= nc zero, as asynchronous 16-byte copies: no register staging, so all of a tile's requests are in
// flight at once and the copy overlaps whatever the threads do until they wait for its group.
__device__ __forceinline__ void cp_async16(void* dst, const void* src, bool valid) {
  const int bytes = valid ? 16 : 0;  // 0: the destination is zero-filled, nothing is read
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(smem_u32(dst)), "l"(src), "r"(bytes) : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N>
__device__ __forceinline__ void cp_async_wait() {
  asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory");
}
__device__ __forceinline__ void rows_async_128(float* dst, const float* __restrict__ src, size_t ld, int nc, int tid,
                                               int threads = kChunkThreads) {
  for (int i = tid; i < kCh * 32; i += threads) {
    const int r = i >> 5, c4 = i & 31;
    cp_async16(dst + r * kLd + 4 * c4, src + (size_t)(r < nc ? r : 0) * ld + 4 * c4, r < nc);
  }
}

// HEADS value heads of one key head per CTA: K K^T and Q K^T are the same for all of them, only the gates differ; V comes in by
// cp.async under the products. One head per CTA (two CTAs per SM) where the grid is too small to fill the SMs otherwise.
// Bound by the substitution, 42,000 of 67,000 cycles of a CTA of three heads: 64 x 63 / 2 FMAs per column behind broadcasts of A's
// rows and a fetch of straight-line code. 1531 tokens, 16 / 48 heads, whole mixer: 653 us in one run, 581 in four with a column per
// thread, 635 and 555 with two; one head per CTA keeps one column (300 tokens: 206 us, 207 with two, which spill at its registers).
// Two heads per CTA gain little by it: 16 / 32 heads, 1024 tokens 326 and 325 us, three runs of 1531 tokens in all 413 and 408; 8 / 16 heads
// 220 and 221, 227 and 225.
constexpr bool prep_stages_v(int heads) { return heads > 1; }
constexpr int prep_smem_bytes(int heads) {
  return (2 * kCh * kLd + heads * (kCh * kLdP + 3 * kCh) + (prep_stages_v(heads) ? heads * kCh * kDv : 0)) * 4;
}
static_assert(prep_smem_bytes(3) <= 227 * 1024, "shared memory");

template <int HEADS, int THREADS>
__global__ void __launch_bounds__(THREADS, HEADS == 1 && THREADS == 256 ? 2 : 1) gdn_chunk_prep_kernel(
    const float* __restrict__ qkv, int conv_dim, const float* __restrict__ ab, const float* __restrict__ A,
    const float* __restrict__ dt_bias, int nk, int nv, const int* __restrict__ seq_start, float* __restrict__ scratch) {
  pdl_wait();               // everything written by earlier kernels of the stream is visible from here on
  pdl_launch_dependents();  // the next kernel may be scheduled now; it holds its own dependent work back the same way
  constexpr int kThreads = THREADS;  // 128 * HEADS (one head: 256) for the substitution, more take part in the products only
  constexpr bool kStageV = prep_stages_v(HEADS);
  extern __shared__ float prep_sm[];
  float* Ks = prep_sm;
  float* Qs = Ks + kCh * kLd;
  float* As = Qs + kCh * kLd;                 // [HEADS][64][kLdP]
  float* beta_s = As + HEADS * kCh * kLdP;    // [HEADS][64]
  float* lg_s = beta_s + HEADS * kCh;
  float* bg_s = lg_s + HEADS * kCh;           // beta e^lg
  float* Vs = bg_s + HEADS * kCh;             // [HEADS][64][128]
  const int ratio = nv / nk, parts = (ratio + HEADS - 1) / HEADS;
  const int c = blockIdx.x, kh = blockIdx.y / parts, first = blockIdx.y % parts * HEADS, b = blockIdx.z;
  const int heads = min(HEADS, ratio - first), vh0 = kh * ratio + first;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int s0 = seq_start[b], n = seq_start[b + 1] - s0;
  if (c * kCh >= n) return;
  const int nc = min(kCh, n - c * kCh), m0 = s0 + c * kCh;
  float* out = scratch + ((size_t)((s0 - seq_start[0]) / kCh + b + c) * nv + vh0) * kChunkFloats;  // U0, W, P, lg of head vh0

  const float* rows = qkv + (size_t)m0 * conv_dim;
  const float* v_rows = rows + (size_t)2 * nk * kDk + (size_t)vh0 * kDv;
  rows_async_128(Qs, rows + (size_t)kh * kDk, conv_dim, nc, tid, kThreads);
  rows_async_128(Ks, rows + (size_t)nk * kDk + (size_t)kh * kDk, conv_dim, nc, tid, kThreads);
  cp_async_commit();
  if constexpr (kStageV) {
    for (int i = tid; i < heads * kCh * 32; i += kThreads) {
      const int h = i / (kCh * 32), r = i / 32 % kCh, c4 = i % 32;
      cp_async16(Vs + (size_t)(h * kCh + r) * kDv + 4 * c4, v_rows + (size_t)(r < nc ? r : 0) * conv_dim + h * kDv + 4 * c4, r < nc);
    }
  }
  cp_async_commit();
  // Gates: a warp per head, two tokens per lane; lg = inclusive sum of the log decays, added token by token. (A tree would give
  // neighbouring sums that were rounded in different orders: behind sums of 10^6 the factor e^(lg_i - lg_j) of two tokens that
  // hardly decay came out as e^(1/16) instead of 1. The 64 additions run under the copies above.)
  if (warp < heads) {
    float be[2] = {0.0f, 0.0f}, la[2] = {0.0f, 0.0f};
    const int vh = vh0 + warp;
#pragma unroll
    for (int e = 0; e < 2; ++e)
      if (2 * lane + e < nc) token_gates(ab, m0 + 2 * lane + e, nv, vh, A[vh], dt_bias[vh], be[e], la[e]);
    float run = 0.0f, lg0 = 0.0f, lg1 = 0.0f;
#pragma unroll
    for (int i = 0; i < 32; ++i) {
      const float first_of = run + __shfl_sync(0xffffffffu, la[0], i);
      run = first_of + __shfl_sync(0xffffffffu, la[1], i);
      if (lane == i) {
        lg0 = first_of;
        lg1 = run;
      }
    }
    const int at = warp * kCh + 2 * lane;
    beta_s[at] = be[0];
    beta_s[at + 1] = be[1];
    lg_s[at] = lg0;
    lg_s[at + 1] = lg1;
    bg_s[at] = be[0] * expf(lg0);
    bg_s[at + 1] = be[1] * expf(lg1);
    float* lgg = out + (size_t)warp * kChunkFloats + 2 * kCh * 128 + kCh * kCh;
    lgg[2 * lane] = lg0;
    lgg[2 * lane + 1] = lg1;
  }
  cp_async_wait<1>();
  __syncthreads();

  // ---- G = K K^T and Q K^T, lower triangles: thread = rows {2 ty, 2 ty + 1} x columns {tx + 16 jj} up to the row's 16-block ----
  // three heads, 24 groups: the longest rows are a group's only ones, the shortest follow the next shortest
  for (int ty = HEADS == 3 ? 31 - (tid >> 4) : tid >> 4, tx = tid & 15; ty >= 0 && ty < 32; ty += HEADS == 3 ? (ty >= 16 ? -32 : -8) : kThreads / 16) {
    float ag[2][4], ap[2][4];
#pragma unroll
    for (int i = 0; i < 2; ++i)
#pragma unroll
      for (int jj = 0; jj < 4; ++jj) ag[i][jj] = ap[i][jj] = 0.0f;
    auto products = [&](auto count) {
      constexpr int J = decltype(count)::value;
#pragma unroll 4
      for (int kk = 0; kk < 128; kk += 4) {
        float4 ak[2], aq[2], bk[J];
#pragma unroll
        for (int i = 0; i < 2; ++i) {
          ak[i] = *reinterpret_cast<const float4*>(Ks + (2 * ty + i) * kLd + kk);
          aq[i] = *reinterpret_cast<const float4*>(Qs + (2 * ty + i) * kLd + kk);
        }
#pragma unroll
        for (int jj = 0; jj < J; ++jj) bk[jj] = *reinterpret_cast<const float4*>(Ks + (tx + 16 * jj) * kLd + kk);
#pragma unroll
        for (int i = 0; i < 2; ++i)
#pragma unroll
          for (int jj = 0; jj < J; ++jj) {
            ag[i][jj] += ak[i].x * bk[jj].x + ak[i].y * bk[jj].y + ak[i].z * bk[jj].z + ak[i].w * bk[jj].w;
            ap[i][jj] += aq[i].x * bk[jj].x + aq[i].y * bk[jj].y + aq[i].z * bk[jj].z + aq[i].w * bk[jj].w;
          }
      }
    };
    switch (ty >> 3) {  // a warp's two ty share it
      case 0: products(std::integral_constant<int, 1>{}); break;
      case 1: products(std::integral_constant<int, 2>{}); break;
      case 2: products(std::integral_constant<int, 3>{}); break;
      default: products(std::integral_constant<int, 4>{}); break;
    }
#pragma unroll
    for (int h = 0; h < HEADS; ++h) {
      if (h >= heads) break;
      const float* lg = lg_s + h * kCh;
      float* Ah = As + h * kCh * kLdP;
      float* Pg = out + (size_t)h * kChunkFloats + 2 * kCh * 128;
#pragma unroll
      for (int i = 0; i < 2; ++i)
#pragma unroll
        for (int jj = 0; jj < 4; ++jj) {
          const int r = 2 * ty + i, col = tx + 16 * jj;
          const float e = col <= r ? expf(lg[r] - lg[col]) : 0.0f;
          Ah[r * kLdP + col] = col < r ? beta_s[h * kCh + r] * e * ag[i][jj] : 0.0f;
          Pg[r * kCh + col] = e * ap[i][jj];
        }
    }
  }
  cp_async_wait<0>();
  __syncthreads();

  // ---- forward substitution (I + A) X = RHS: columns of [diag(beta) V | diag(beta e^lg) K] ----
  if constexpr (HEADS > 1) {
    // A thread has the same column of both halves, which share the reads of A's rows from shared memory. By blocks of sixteen rows
    // in one rolled loop: a block is solved, stored and taken out of the rows behind it, whose sums so far move down by a block
    // (all 64 rows of two columns unrolled are 80 KB of code and slower than a column per thread).
    constexpr int kB = 16;
    const int h = warp >> 2, col = tid & 127;
    if (h >= heads) return;
    const float* Ab = As + h * kCh * kLdP;
    float* dst = out + (size_t)h * kChunkFloats + col;
    float sum[2][kCh - kB], x[2][kB];  // of the rows behind the block, of its own
#pragma unroll
    for (int e = 0; e < 2; ++e) {
#pragma unroll
      for (int i = 0; i < kCh - kB; ++i) sum[e][i] = 0.0f;
#pragma unroll
      for (int i = 0; i < kB; ++i) x[e][i] = 0.0f;
    }
#pragma unroll 1
    for (int b0 = 0; b0 < kCh; b0 += kB, Ab += kB * kLdP + kB) {
#pragma unroll
      for (int i = 0; i < kB; ++i) {
        const int r = h * kCh + b0 + i;
        x[0][i] = beta_s[r] * Vs[(size_t)r * kDv + col] - x[0][i];
        x[1][i] = bg_s[r] * Ks[(b0 + i) * kLd + col] - x[1][i];
      }
#pragma unroll
      for (int i = 1; i < kB; ++i) {
        float c[2][4] = {};  // four chains: the row's sum is not one serial dependency
#pragma unroll
        for (int j0 = 0; j0 < i; j0 += 4) {
          const float4 a4 = *reinterpret_cast<const float4*>(Ab + i * kLdP + j0);  // entries at j >= i are zero
          const float a[4] = {a4.x, a4.y, a4.z, a4.w};
#pragma unroll
          for (int q = 0; q < 4; ++q)
#pragma unroll
            for (int e = 0; e < 2; ++e)
              if (j0 + q < i) c[e][q] += a[q] * x[e][j0 + q];
        }
#pragma unroll
        for (int e = 0; e < 2; ++e) x[e][i] -= (c[e][0] + c[e][1]) + (c[e][2] + c[e][3]);
      }
#pragma unroll
      for (int i = 0; i < kB; ++i) {
        dst[(b0 + i) * 128] = x[0][i];
        dst[(kCh + b0 + i) * 128] = x[1][i];
      }
#pragma unroll
      for (int n = 0; n < (kCh - kB) / kB; ++n) {
        if (b0 + kB * (n + 1) >= kCh) break;
#pragma unroll
        for (int i = 0; i < kB; ++i)
#pragma unroll
          for (int j0 = 0; j0 < kB; j0 += 4) {
            const float4 a4 = *reinterpret_cast<const float4*>(Ab + (kB * (n + 1) + i) * kLdP + j0);
#pragma unroll
            for (int e = 0; e < 2; ++e) {
              float& s = sum[e][kB * n + i];
              s += a4.x * x[e][j0];
              s += a4.y * x[e][j0 + 1];
              s += a4.z * x[e][j0 + 2];
              s += a4.w * x[e][j0 + 3];
            }
          }
      }
#pragma unroll
      for (int e = 0; e < 2; ++e) {
#pragma unroll
        for (int i = 0; i < kB; ++i) x[e][i] = sum[e][i];
#pragma unroll
        for (int i = 0; i < kCh - 2 * kB; ++i) sum[e][i] = sum[e][i + kB];
      }
    }
  } else if (tid < 256) {  // one column per thread
    const int col = tid;
    const float* Ah = As;
    float x[kCh];
    if (col < 128) {
#pragma unroll
      for (int i = 0; i < kCh; ++i) x[i] = i < nc ? beta_s[i] * v_rows[(size_t)i * conv_dim + col] : 0.0f;
    } else {
#pragma unroll
      for (int i = 0; i < kCh; ++i) x[i] = bg_s[i] * Ks[i * kLd + col - 128];
    }
#pragma unroll
    for (int i = 1; i < kCh; ++i) {
      float c0 = 0.0f, c1 = 0.0f, c2 = 0.0f, c3 = 0.0f;  // four chains: the row's sum is not one serial dependency
#pragma unroll
      for (int j0 = 0; j0 < i; j0 += 4) {
        const float4 a4 = *reinterpret_cast<const float4*>(Ah + i * kLdP + j0);  // entries at j >= i are zero
        c0 += a4.x * x[j0];
        if (j0 + 1 < i) c1 += a4.y * x[j0 + 1];
        if (j0 + 2 < i) c2 += a4.z * x[j0 + 2];
        if (j0 + 3 < i) c3 += a4.w * x[j0 + 3];
      }
      x[i] -= (c0 + c1) + (c2 + c3);
    }
    float* dst = out + (col < 128 ? col : kCh * 128 + col - 128);
#pragma unroll
    for (int i = 0; i < kCh; ++i) dst[i * 128] = x[i];
  }
}

constexpr int kScanSmemBytes = (128 * kLd + 4 * kCh * kLd + kCh * kLdP + 3 * kCh) * 4;

// VSPLIT = 1: one CTA per (v head, sequence) updates all 128 state rows and finishes the output (gated RMSNorm)
// itself. VSPLIT = 2: two CTAs per head, 64 state rows each (the rows are independent given k, q, beta, decay); the
// un-normalised outputs go to scratch and gdn_norm_gate_kernel finishes them, because the norm runs over all 128
// outputs of a token. The split doubles the CTAs of the sequential part when a step has few (head, sequence) pairs.
template <int VSPLIT>
__global__ void __launch_bounds__(kChunkThreads, 1) gdn_chunk_scan_kernel(
    const float* __restrict__ qkv, int conv_dim, const __nv_bfloat16* __restrict__ z, int ld_z,
    const float* __restrict__ norm_w, float eps, __nv_bfloat16* __restrict__ out, int layer, int num_layers, int nk,
    int nv, float* __restrict__ recurrent, const int* __restrict__ seq_start, const int* __restrict__ seq_slot,
    const float* __restrict__ scratch, float* __restrict__ o_scratch) {
  pdl_wait();               // everything written by earlier kernels of the stream is visible from here on
  pdl_launch_dependents();  // the next kernel may be scheduled now; it holds its own dependent work back the same way
  constexpr int NV = kDv / VSPLIT;  // state rows (v) of this CTA
  constexpr int TV = 4 / VSPLIT;    // v per thread in the [tokens][v] products: v = lane + 32 jj
  extern __shared__ float scan_sm[];
  float* Ss = scan_sm;               // [NV v][kLd]
  float* Ws = Ss + NV * kLd;         // [64][kLd]
  float* Qs = Ws + kCh * kLd;
  float* Kd = Qs + kCh * kLd;        // K rows
  float* Us = Kd + kCh * kLd;        // U0, then U: [64][kLd], NV columns used
  float* Ps = Us + kCh * kLd;        // [64][kLdP]
  float* lg_s = Ps + kCh * kLdP;
  float* eg_s = lg_s + kCh;          // e^{lg_t}
  float* kd_s = eg_s + kCh;          // e^{lg_C - lg_j}
  const int vh = blockIdx.x / VSPLIT, vbase = (blockIdx.x % VSPLIT) * NV, b = blockIdx.y;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int s0 = seq_start[b], n = seq_start[b + 1] - s0;
  if (n <= 0) return;
  const int kh = vh / (nv / nk);
  float* S = recurrent + ((((size_t)seq_slot[b] * num_layers + layer) * nv + vh) * kDv + vbase) * kDk;
  for (int i = tid; i < NV * 32; i += kChunkThreads)
    *reinterpret_cast<float4*>(Ss + (i >> 5) * kLd + 4 * (i & 31)) = *reinterpret_cast<const float4*>(S + (size_t)i * 4);
  const int chunks = (n + kCh - 1) / kCh;
  float nw[TV];
#pragma unroll
  for (int jj = 0; jj < TV; ++jj) nw[jj] = norm_w[vbase + lane + 32 * jj];

  for (int c = 0; c < chunks; ++c) {
    const int nc = min(kCh, n - c * kCh), m0 = s0 + c * kCh;
    const float* in = scratch + ((size_t)((s0 - seq_start[0]) / kCh + b + c) * nv + vh) * kChunkFloats;
    __syncthreads();  // the previous chunk's state update (or the initial state load) is complete
    if (tid < kCh) {
      const float lg = in[2 * kCh * 128 + kCh * kCh + tid], lgc = in[2 * kCh * 128 + kCh * kCh + kCh - 1];
      lg_s[tid] = lg;
      eg_s[tid] = expf(lg);
      kd_s[tid] = expf(lgc - lg);
    }
    __syncthreads();
    const float* rows = qkv + (size_t)m0 * conv_dim;
    // group 1: what the two state products need (W, Q, U0); group 2: P and K, which land while those run
    rows_async_128(Ws, in + kCh * 128, 128, kCh, tid);
    rows_async_128(Qs, rows + (size_t)kh * kDk, conv_dim, nc, tid);
    for (int i = tid; i < kCh * (NV / 4); i += kChunkThreads) {
      const int r = i / (NV / 4), c4 = i % (NV / 4);
      cp_async16(Us + r * kLd + 4 * c4, in + (size_t)r * 128 + vbase + 4 * c4, true);
    }
    cp_async_commit();
    rows_async_128(Kd, rows + (size_t)nk * kDk + (size_t)kh * kDk, conv_dim, nc, tid);
    for (int i = tid; i < kCh * 16; i += kChunkThreads)
      cp_async16(Ps + (i >> 4) * kLdP + 4 * (i & 15), in + 2 * kCh * 128 + (size_t)i * 4, true);
    cp_async_commit();
    cp_async_wait<1>();
    __syncthreads();

    // [64 tokens][NV v] products: threads 0-255 compute X = W S0^T, threads 256-511 Y = Q S0^T at the same time.
    // Thread tile 8 tokens (8 gw + i) x TV v (lane + 32 jj): with TV = 4, 12 shared-memory reads feed 128 FMAs, which
    // keeps the products FMA-bound instead of shared-memory-bound.
    const int grp = warp >> 3, gw = warp & 7;  // grp 0: X / upper half of P U, grp 1: Y / lower half + output
    const int t0 = 8 * gw;
    float acc[8][TV];
#pragma unroll
    for (int i = 0; i < 8; ++i)
#pragma unroll
      for (int jj = 0; jj < TV; ++jj) acc[i][jj] = 0.0f;
    {
      const float* Am = grp == 0 ? Ws : Qs;
#pragma unroll 2
      for (int kk = 0; kk < 128; kk += 4) {
        float4 bv[TV];
#pragma unroll
        for (int jj = 0; jj < TV; ++jj) bv[jj] = *reinterpret_cast<const float4*>(Ss + (lane + 32 * jj) * kLd + kk);
#pragma unroll
        for (int i = 0; i < 8; ++i) {
          const float4 av = *reinterpret_cast<const float4*>(Am + (t0 + i) * kLd + kk);
#pragma unroll
          for (int jj = 0; jj < TV; ++jj)
            acc[i][jj] += av.x * bv[jj].x + av.y * bv[jj].y + av.z * bv[jj].z + av.w * bv[jj].w;
        }
      }
    }
    if (grp == 0) {  // (a) U = U0 - X
#pragma unroll
      for (int i = 0; i < 8; ++i)
#pragma unroll
        for (int jj = 0; jj < TV; ++jj) Us[(t0 + i) * kLd + lane + 32 * jj] -= acc[i][jj];
    } else {         // (b) Y scaled by e^{lg_t}
#pragma unroll
      for (int i = 0; i < 8; ++i)
#pragma unroll
        for (int jj = 0; jj < TV; ++jj) acc[i][jj] *= eg_s[t0 + i];
    }
    cp_async_wait<0>();
    __syncthreads();  // U complete; nobody reads W any more; P and K have landed

    // ---- (c) O = Y + P U. P is lower triangular: tokens 8 gw .. 8 gw + 7 need j < 8 gw + 8; the two thread groups
    // split that range (group 1 continues on top of Y, group 0 starts from zero and hands its part over through
    // the W buffer).
    {
      const int j_end = 8 * gw + 8;
      const int j_mid = (j_end / 2) & ~3;
      const int ja = grp == 0 ? j_mid : 0, jb = grp == 0 ? j_end : j_mid;
      if (grp == 0) {
#pragma unroll
        for (int i = 0; i < 8; ++i)
#pragma unroll
          for (int jj = 0; jj < TV; ++jj) acc[i][jj] = 0.0f;
      }
      for (int j = ja; j < jb; j += 4) {
        float uv[4][TV];
#pragma unroll
        for (int q = 0; q < 4; ++q)
#pragma unroll
          for (int jj = 0; jj < TV; ++jj) uv[q][jj] = Us[(j + q) * kLd + lane + 32 * jj];
#pragma unroll
        for (int i = 0; i < 8; ++i) {
          const float4 pv = *reinterpret_cast<const float4*>(Ps + (t0 + i) * kLdP + j);
#pragma unroll
          for (int jj = 0; jj < TV; ++jj)
            acc[i][jj] += pv.x * uv[0][jj] + pv.y * uv[1][jj] + pv.z * uv[2][jj] + pv.w * uv[3][jj];
        }
      }
      if (grp == 0) {
#pragma unroll
        for (int i = 0; i < 8; ++i)
#pragma unroll
          for (int jj = 0; jj < TV; ++jj) Ws[(t0 + i) * kLd + lane + 32 * jj] = acc[i][jj];
      }
    }
    __syncthreads();  // group 0's part of P U is in the W buffer; every read of S0 is done
    if (grp == 1) {
#pragma unroll
      for (int i = 0; i < 8; ++i) {
#pragma unroll
        for (int jj = 0; jj < TV; ++jj) acc[i][jj] += Ws[(t0 + i) * kLd + lane + 32 * jj];
        const int t = t0 + i;
        const size_t m = (size_t)(m0 + t);
        if constexpr (VSPLIT == 1) {
          // gated RMSNorm over the 128 outputs of each token (a warp holds whole tokens)
          float sq = 0.0f;
#pragma unroll
          for (int jj = 0; jj < TV; ++jj) sq += acc[i][jj] * acc[i][jj];
          const float ss = warp_sum(sq);
          if (t < nc) {
            const float r = 1.0f / sqrtf(ss / float(kDv) + eps);
#pragma unroll
            for (int jj = 0; jj < TV; ++jj) {
              const int d = lane + 32 * jj;
              const float zz = __bfloat162float(z[m * ld_z + (size_t)vh * kDv + d]);
              out[m * nv * kDv + (size_t)vh * kDv + d] = __float2bfloat16_rn(acc[i][jj] * r * nw[jj] * silu_f(zz));
            }
          }
        } else if (t < nc) {
#pragma unroll
          for (int jj = 0; jj < TV; ++jj)
            o_scratch[(m - seq_start[0]) * nv * kDv + (size_t)vh * kDv + vbase + lane + 32 * jj] = acc[i][jj];
        }
      }
    }

    // ---- (d) S = e^{lg_C} S0 + U^T diag(e^{lg_C - lg}) K: thread tile v = TV vq + i, k = 4 ko + {0..3} and 64 + 4 ko + {0..3}
    {
      const int vq = tid >> 4, ko = tid & 15;
      float sacc[TV][8];
#pragma unroll
      for (int i = 0; i < TV; ++i)
#pragma unroll
        for (int e = 0; e < 8; ++e) sacc[i][e] = 0.0f;
#pragma unroll 4
      for (int j = 0; j < kCh; ++j) {
        const float kdj = kd_s[j];  // e^{lg_C - lg_j}: the decay from token j to the end of the chunk
        float uu[TV];
#pragma unroll
        for (int i = 0; i < TV; ++i) uu[i] = Us[j * kLd + TV * vq + i] * kdj;
        const float4 k0 = *reinterpret_cast<const float4*>(Kd + j * kLd + 4 * ko);
        const float4 k1 = *reinterpret_cast<const float4*>(Kd + j * kLd + 64 + 4 * ko);
        const float kk8[8] = {k0.x, k0.y, k0.z, k0.w, k1.x, k1.y, k1.z, k1.w};
#pragma unroll
        for (int i = 0; i < TV; ++i)
#pragma unroll
          for (int e = 0; e < 8; ++e) sacc[i][e] += uu[i] * kk8[e];
      }
      const float gC = eg_s[kCh - 1];
#pragma unroll
      for (int i = 0; i < TV; ++i) {
        float* r0 = Ss + (TV * vq + i) * kLd + 4 * ko;
        float4 a = *reinterpret_cast<float4*>(r0), bq = *reinterpret_cast<float4*>(r0 + 64);
        a.x = gC * a.x + sacc[i][0];
        a.y = gC * a.y + sacc[i][1];
        a.z = gC * a.z + sacc[i][2];
        a.w = gC * a.w + sacc[i][3];
        bq.x = gC * bq.x + sacc[i][4];
        bq.y = gC * bq.y + sacc[i][5];
        bq.z = gC * bq.z + sacc[i][6];
        bq.w = gC * bq.w + sacc[i][7];
        *reinterpret_cast<float4*>(r0) = a;
        *reinterpret_cast<float4*>(r0 + 64) = bq;
      }
    }
  }
  __syncthreads();
  for (int i = tid; i < NV * 32; i += kChunkThreads)
    *reinterpret_cast<float4*>(S + (size_t)i * 4) = *reinterpret_cast<const float4*>(Ss + (i >> 5) * kLd + 4 * (i & 31));
}

// ---------------------------------------------------------------------------------------------------
// The same scan with the per-chunk products on the 5th-generation tensor cores: one CTA per (v head, sequence), the decay
// factors, the preparation kernel's U0 / W / P and the state layout those of gdn_chunk_scan_kernel, which stays as the fp32
// CUDA-core form of the operator. Every fp32 factor x is cut into three bf16 terms x = hi + mid + lo of eight mantissa bits
// each (exact) and a product is six MMAs, smallest terms first: what is dropped is at most 2^-21 of the product (mid lo + lo mid,
// each up to 2^-22, always toward zero), and fp32's range of exponents stays. Error of state and outputs against float64, runs of
// 1531 and 900 tokens: 1.9e-7 and 6.5e-7 (fp32 scan 1.4e-7 and 6.4e-7; pairs of TF32 on mma.sync, the form before, 4.7e-7 and 7.5e-7),
// with decays of at most 1 % a token 4.7e-7 and 1.0e-6 (1.9e-7 and 2.2e-7; 9.2e-7 and 1.7e-6). (One TF32 product per term moved outputs
// that are small through cancellation by more than the operator's tolerance.)
//   The state is the A operand, in tensor memory: 128 rows (v) = 128 lanes. With e_t = e^{lg_t}, d_t = e^{lg_C - lg_t}
//   (1) [Y | X] = S0 [e Q | W]^T      128 v x 128 tokens, k = 128; Q and W rows K-major in shared memory
//       U = U0^T - X                  into tensor memory, the A operand of
//   (2) D = U (d K)                   128 v x 128 k, k = 64 tokens; K as it lies, dk contiguous (MN-major)
//   (3) Y += U P^T                    128 v x 64 tokens
//       S = e_C S0 + D                in registers (a thread: one row, 32 columns), back into tensor memory as three terms
// D lies over X, which has been read by then: 192 columns of results + 192 of the state + 96 of U. Sixteen warps turn results into
// the next operand in tensor memory, half of it at a time so that the product starts on the first half; seven cut Q, W, K and P
// of the chunks to come into terms; one issues the MMAs, copies U0 a chunk ahead and asks for the other inputs of the next chunk.
// Rolled loops where nothing is gained by more: with everything unrolled the code was 109 KB and a chunk took 13,000 cycles.
// The gated norm of the outputs is a kernel of its own: here its reads and writes held up everybody's shared memory accesses.
// Bound by the serial work on a chunk, 11,000 cycles: (1) 48 MMAs of 64 cycles, U, (2) 24 of 64, (3) 24 of 60 (their issue),
// half of S, and by the seven warps' loads. 512 tokens of 48 heads, both without norm and gate: 90 us with TF32 on mma.sync, 64 us
// now (50 warm); 1531 tokens in three sequences, whole mixer: 744 and 618 us.
// One CTA per (v head, sequence) however few there are, where the form before had two: 16 heads of one sequence, whole mixer, 64
// tokens 66.6 and 66.3 us, 1024 tokens 285 and 220, 1531 tokens 396 and 299.
// ---------------------------------------------------------------------------------------------------
constexpr int kScanStateWarps = 16, kScanLoadWarps = 7, kScanMmaWarp = kScanStateWarps + kScanLoadWarps, kScanThreads = (kScanMmaWarp + 1) * 32;
constexpr int kScanWq = 0, kScanWqTerm = 2 * 128 * 128, kScanWqSlice = 128 * 128;  // per term two slices of 64 k: [Q 64 | W 64][128 bytes]
constexpr int kScanK = kScanWq + 3 * kScanWqTerm, kScanKTerm = 2 * kCh * 128;      // per term two chunks of 64 dk: [64 tokens][128 bytes]
constexpr int kScanP = kScanK + 3 * kScanKTerm, kScanPTerm = kCh * 128;            // per term [64 tokens][64 earlier tokens]
constexpr int kScanU0 = kScanP + 3 * kScanPTerm, kScanU0Bytes = kCh * kDv * 4;       // as the preparation kernel left it
constexpr int kScanBar = kScanU0 + kScanU0Bytes;
constexpr int kScanUmmaSmem = 1024 + kScanBar + 128;
static_assert(kScanUmmaSmem <= 227 * 1024, "shared memory");
constexpr uint32_t kScanTmY = 0, kScanTmX = 64, kScanTmD = 64, kScanTmS = 192, kScanTmU = 384;  // tensor memory columns

// two neighbours as packed bf16 terms (the first one in the low half); truncation leaves an exact remainder each time
struct Terms {
  uint32_t hi, mid, lo;
};
__device__ __forceinline__ void less_top(uint32_t& a, uint32_t& b) {  // both minus their upper sixteen bits, one two-lane FMA
  asm("{\n\t.reg .b64 x, t, m;\n\t.reg .b32 ta, tb;\n\t"
      "mov.b64 x, {%0, %1};\n\tand.b32 ta, %0, 0xffff0000;\n\tand.b32 tb, %1, 0xffff0000;\n\tmov.b64 t, {ta, tb};\n\t"
      "mov.b64 m, 0xbf800000bf800000;\n\tfma.rn.f32x2 x, t, m, x;\n\tmov.b64 {%0, %1}, x;\n\t}"
      : "+r"(a), "+r"(b));
}
__device__ __forceinline__ Terms split3(float x, float y) {
  uint32_t a = __float_as_uint(x), b = __float_as_uint(y);
  Terms t;
  t.hi = __byte_perm(a, b, 0x7632);
  less_top(a, b);
  t.mid = __byte_perm(a, b, 0x7632);
  less_top(a, b);
  t.lo = __byte_perm(a, b, 0x7632);
  return t;
}
// four neighbours to the same place of the three terms of an operand
__device__ __forceinline__ void store_terms(uint8_t* dst, int term_bytes, const float4& v) {
  const Terms a = split3(v.x, v.y), b = split3(v.z, v.w);
  *reinterpret_cast<uint2*>(dst) = make_uint2(a.hi, b.hi);
  *reinterpret_cast<uint2*>(dst + term_bytes) = make_uint2(a.mid, b.mid);
  *reinterpret_cast<uint2*>(dst + 2 * term_bytes) = make_uint2(a.lo, b.lo);
}
// N MMAs over 16 N of the contraction: A = tensor memory columns a_tmem + 8 i, B = descriptors b_desc + i * STEP (16-byte units;
// the address field cannot carry). The first one overwrites the accumulator unless `accumulate`. Converged warp.
template <int N, int STEP>
__device__ __forceinline__ void umma_bf16_ta(uint32_t d_tmem, uint32_t a_tmem, uint64_t b_desc, uint32_t idesc, uint32_t accumulate) {
  static_assert(N == 2 || N == 4);
  if constexpr (N == 4) {
    asm volatile(
        "{\n\t.reg .pred p, t, leader;\n\t.reg .b32 a1, a2, a3;\n\t.reg .b64 b1, b2, b3;\n\t"
        "elect.sync _|leader, 0xffffffff;\n\t"
        "setp.ne.b32 p, %4, 0;\n\t"
        "setp.eq.b32 t, %4, %4;\n\t"
        "add.u32 a1, %1, 8;\n\tadd.u32 a2, %1, 16;\n\tadd.u32 a3, %1, 24;\n\t"
        "add.u64 b1, %2, %5;\n\tadd.u64 b2, %2, %6;\n\tadd.u64 b3, %2, %7;\n\t"
        "@leader tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p;\n\t"
        "@leader tcgen05.mma.cta_group::1.kind::f16 [%0], [a1], b1, %3, t;\n\t"
        "@leader tcgen05.mma.cta_group::1.kind::f16 [%0], [a2], b2, %3, t;\n\t"
        "@leader tcgen05.mma.cta_group::1.kind::f16 [%0], [a3], b3, %3, t;\n\t}"
        ::"r"(d_tmem), "r"(a_tmem), "l"(b_desc), "r"(idesc), "r"(accumulate), "n"(STEP), "n"(2 * STEP), "n"(3 * STEP)
        : "memory");
  } else {
    asm volatile(
        "{\n\t.reg .pred p, t, leader;\n\t.reg .b32 a1;\n\t.reg .b64 b1;\n\t"
        "elect.sync _|leader, 0xffffffff;\n\t"
        "setp.ne.b32 p, %4, 0;\n\t"
        "setp.eq.b32 t, %4, %4;\n\t"
        "add.u32 a1, %1, 8;\n\t"
        "add.u64 b1, %2, %5;\n\t"
        "@leader tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p;\n\t"
        "@leader tcgen05.mma.cta_group::1.kind::f16 [%0], [a1], b1, %3, t;\n\t}"
        ::"r"(d_tmem), "r"(a_tmem), "l"(b_desc), "r"(idesc), "r"(accumulate), "n"(STEP)
        : "memory");
  }
}

// Past L1: with what 204 KB of shared memory leave of it, loads that take room there waited for it (13,000 cycles a chunk, not 10,800).
__device__ __forceinline__ float4 ld_once(const float* p) {
  float4 v;
  asm volatile("ld.global.L1::no_allocate.v4.f32 {%0,%1,%2,%3}, [%4];" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "l"(p));
  return v;
}
__global__ void __launch_bounds__(kScanThreads, 1) gdn_chunk_scan_umma_kernel(
    const float* __restrict__ qkv, int conv_dim, int layer, int num_layers, int nk, int nv, float* __restrict__ recurrent,
    const int* __restrict__ seq_start, const int* __restrict__ seq_slot, const float* __restrict__ scratch, float* __restrict__ o_scratch) {
  extern __shared__ uint8_t scan_raw[];
  uint8_t* smem = scan_raw + ((1024 - (smem_u32(scan_raw) & 1023)) & 1023);
  uint64_t* done = reinterpret_cast<uint64_t*>(smem + kScanBar);  // [3]: products (1), (2), (3)
  uint64_t *s_ready = done + 3, *u_ready = done + 5;              // [2] operands in tensor memory, halves of the contraction
  uint64_t *wq_full = done + 7, *kp_full = done + 8;              // operands in shared memory
  uint64_t* u0_full = done + 9;
  uint64_t* drained = done + 10;  // products that the issuing warp itself waits for
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(done + 11);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);
  volatile int* not_finite = abort_flag + 1;  // 1 + the last chunk with an update U that is not finite
  const int vh = blockIdx.x, b = blockIdx.y, kh = vh / (nv / nk);
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  if (tid == 0) {
    for (int i = 0; i < 3; ++i) mbar_init(&done[i], 1);
    for (int i = 0; i < 4; ++i) mbar_init(&s_ready[i], kScanStateWarps);
    mbar_init(wq_full, kScanLoadWarps);
    mbar_init(kp_full, kScanLoadWarps);
    mbar_init(u0_full, 1);
    mbar_init(drained, 1);
    *abort_flag = 0;
    *not_finite = 0;
    mbar_fence_init();
  }
  if (warp == kScanMmaWarp) tmem_alloc(tmem_slot, 512);
  pdl_wait();               // everything written by earlier kernels of the stream is visible from here on
  pdl_launch_dependents();  // the next kernel may be scheduled now; it holds its own dependent work back the same way
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = *tmem_slot;
  const int s0 = seq_start[b], n = seq_start[b + 1] - s0, chunks = (n + kCh - 1) / kCh;
  const float* in0 = scratch + ((size_t)((s0 - seq_start[0]) / kCh + b) * nv + vh) * kChunkFloats;  // U0, W, P, lg of the first chunk
  const size_t in_step = (size_t)nv * kChunkFloats;
  constexpr int kLgAt = 2 * kCh * 128 + kCh * kCh;
  bool alive = true;  // false: a wait ran out; the role goes through its loop without waiting, computing or storing
  // every barrier completes once per chunk
  auto wait = [&](uint64_t* bar, int c, unsigned site) {
    bool there = !alive;
#pragma unroll 1
    for (uint32_t i = 0; i < kSpinLimit && !there; ++i) {
      there = mbar_try_wait(bar, uint32_t(c) & 1u);
      if (!there && *abort_flag) break;
    }
    if (!there) {
      report_error(site);
      *abort_flag = 1;
    }
    alive = __all_sync(0xffffffffu, alive && there);
  };

  if (warp == kScanMmaWarp) {
    constexpr uint32_t kIdesc = (1u << 4) | (1u << 7) | (1u << 10) | (uint32_t(128 >> 4) << 24);  // bf16, fp32 sums, 128 rows
    constexpr uint32_t kIdesc1 = kIdesc | (uint32_t(128 >> 3) << 17), kIdesc2 = kIdesc1 | (1u << 16), kIdesc3 = kIdesc | (uint32_t(kCh >> 3) << 17);
    // terms of A and B, smallest products first; rolled loops: unrolled, this warp's code alone was 35 KB
    auto term_a = [](int i) { return (0x001102u >> (4 * i)) & 15u; };  // lo hi mid mid hi hi
    auto term_b = [](int i) { return (0x010120u >> (4 * i)) & 15u; };  // hi lo mid hi mid hi
    const uint64_t wq = smem_desc_sw128(smem_u32(smem + kScanWq)), kd = smem_desc_sw128_mn(smem_u32(smem + kScanK), kCh * 128),
                   pd = smem_desc_sw128(smem_u32(smem + kScanP));
    const uint64_t policy = policy_evict_first();
    int requested = 0, drains = 0;
    auto drain = [&](unsigned site) {
      umma_commit(drained);
      const bool there = mbar_wait(drained, uint32_t(drains++) & 1u, site);
      if (!there) *abort_flag = 1;
      alive = __all_sync(0xffffffffu, alive && there);
    };
    auto request_u0 = [&](int c) {  // one copy, a chunk ahead of its use
      ++requested;
      if (lane == 0) {
        mbar_expect_tx(u0_full, kScanU0Bytes);
        bulk_g2s(smem + kScanU0, in0 + c * in_step, kScanU0Bytes, u0_full, policy);
      }
      __syncwarp();
    };
    // the rest of a chunk's input, a line per lane: what it costs is not the bytes but the first touch of their pages
    auto prefetch = [&](int c) {
      const float* in = in0 + c * in_step + kCh * 128;
      const int nc = min(kCh, n - c * kCh);
      const float* rows = qkv + (size_t)(s0 + c * kCh) * conv_dim + (size_t)kh * kDk;
#pragma unroll 4
      for (int i = lane; i < (kCh * 128 + kCh * kCh) / 32; i += 32) asm volatile("prefetch.global.L2 [%0];" ::"l"(in + 32 * i));
#pragma unroll 4
      for (int i = lane; i < 8 * nc; i += 32)
        asm volatile("prefetch.global.L2 [%0];" ::"l"(rows + (size_t)(i >> 3) * conv_dim + (i & 4 ? nk * kDk : 0) + 32 * (i & 3)));
    };
    if (chunks > 0) request_u0(0);
#pragma unroll 1
    for (int c = 0; c < chunks; ++c) {
      wait(wq_full, c, 0x411);
#pragma unroll 1
      for (uint32_t h = 0; h < 2; ++h) {
        wait(&s_ready[h], c, 0x412);
        if (!alive) continue;
        tc_fence_after();
#pragma unroll 1
        for (uint32_t i = 0; i < 6; ++i)
          umma_bf16_ta<4, 2>(tmem + kScanTmY, tmem + kScanTmS + 64 * term_a(i) + 32 * h,
                             wq + uint64_t((kScanWqTerm >> 4) * term_b(i) + (kScanWqSlice >> 4) * h), kIdesc1, i | h);
      }
      if (alive) umma_commit(&done[0]);
      if (c + 1 < chunks) prefetch(c + 1);
      wait(kp_full, c, 0x413);
#pragma unroll 1
      for (uint32_t h = 0; h < 2; ++h) {
        wait(&u_ready[h], c, 0x414);
        if (!alive) continue;
        tc_fence_after();
#pragma unroll 1
        for (uint32_t i = 0; i < 6; ++i)
          umma_bf16_ta<2, 128>(tmem + kScanTmD, tmem + kScanTmU + 32 * term_a(i) + 16 * h,
                               kd + uint64_t((kScanKTerm >> 4) * term_b(i) + 256 * h), kIdesc2, i | h);
      }
      if (alive) {
        if (c + 1 < chunks) request_u0(c + 1);
        umma_commit(&done[1]);
        if (*not_finite != c + 1) {
#pragma unroll 1
          for (uint32_t i = 0; i < 6; ++i)
            umma_bf16_ta<4, 2>(tmem + kScanTmY, tmem + kScanTmU + 32 * term_a(i), pd + uint64_t((kScanPTerm >> 4) * term_b(i)), kIdesc3, 1u);
        } else {
          // P is zero above its diagonal, but zero times what is not finite is NaN: sixteen tokens of U at a time, into the outputs
          // from theirs on alone, so that a bad row spoils no token ahead of its block of sixteen. Products of different widths
          // may overtake each other, hence the waits.
#pragma unroll 1
          for (uint32_t e = 0; e < 24 && alive; ++e) {
            const uint32_t k = e / 6, i = e % 6;
            umma_bf16_ts(tmem + kScanTmY + 16 * k, tmem + kScanTmU + 32 * term_a(i) + 8 * k,
                         pd + uint64_t((kScanPTerm >> 4) * term_b(i) + 130 * k), kIdesc3 - (k << 18), 1u);
            if (i == 5) drain(0x41e);
          }
        }
        if (alive) umma_commit(&done[2]);
      }
    }
    if (!alive) {  // given up: the copy and the products that may be in flight end before shared and tensor memory go to another CTA
      if (requested > 0) mbar_wait(u0_full, uint32_t(requested - 1) & 1u, 0x41b);
      drain(0x41d);
    }
  } else if (warp < kScanStateWarps && chunks > 0) {
    // ---- U and the state: a thread = one row; of each half of the 64 tokens and of the 128 dk, its part is 8 tokens and 16 dk ----
    const int quarter = warp & 3, part = warp >> 2, v = 32 * quarter + lane;
    const uint32_t lanes = tmem + (uint32_t(32 * quarter) << 16);
    float* S_g = recurrent + (((size_t)seq_slot[b] * num_layers + layer) * nv + vh) * kDv * kDk;
    float* o_g = o_scratch + ((size_t)(s0 - seq_start[0]) * nv + vh) * kDv + v;
    // the state comes and goes through shared memory (where K and P go later, Q and W went): a thread's pieces of a row, straight
    // from global memory, are 32 lines an instruction
    float *S_in = reinterpret_cast<float*>(smem + kScanK), *S_out = reinterpret_cast<float*>(smem + kScanWq);
    static_assert(128 * kLd * 4 <= kScanU0 - kScanK && 128 * kLd * 4 <= kScanK - kScanWq, "state rows in shared memory");
#pragma unroll 8
    for (int i = tid; i < 128 * 32; i += kScanStateWarps * 32) cp_async16(S_in + (i >> 5) * kLd + 4 * (i & 31), S_g + (size_t)i * 4, true);
    cp_async_commit();
    cp_async_wait<0>();
    named_bar_sync(1, kScanStateWarps * 32);
    float S[32];  // [half][own columns]
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      const float4 x = *reinterpret_cast<const float4*>(S_in + v * kLd + 64 * (i / 4) + 16 * part + 4 * (i % 4));
      S[4 * i] = x.x;
      S[4 * i + 1] = x.y;
      S[4 * i + 2] = x.z;
      S[4 * i + 3] = x.w;
    }
    // eight neighbours of the row into columns col .. col + 3 of the three terms of an operand
    auto eight_to_tmem = [&](uint32_t col, uint32_t term_cols, const float* x) {
      uint32_t hi[4], mid[4], lo[4];
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const Terms t = split3(x[2 * i], x[2 * i + 1]);
        hi[i] = t.hi;
        mid[i] = t.mid;
        lo[i] = t.lo;
      }
      tmem_st4(lanes + col, hi);
      tmem_st4(lanes + col + term_cols, mid);
      tmem_st4(lanes + col + 2 * term_cols, lo);
    };
    auto arrive = [&](uint64_t* bar) {  // the warp's stores to and loads from tensor memory are complete
      tmem_wait_st();
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(bar);
    };
    const float* u0_sm = reinterpret_cast<const float*>(smem + kScanU0) + v;
#pragma unroll
    for (int h = 0; h < 2; ++h) {
#pragma unroll
      for (int e = 0; e < 2; ++e) eight_to_tmem(kScanTmS + uint32_t(32 * h + 8 * part + 4 * e), 64, S + 16 * h + 8 * e);
      arrive(&s_ready[h]);
    }
#pragma unroll 1
    for (int c = 0; c < chunks; ++c) {
      const bool more = c + 1 < chunks;
      const int nc = alive ? min(kCh, n - c * kCh) : 0;
      const float eC = expf(in0[c * in_step + kLgAt + kCh - 1]);
      wait(u0_full, c, 0x418);
      float u[16];
#pragma unroll
      for (int i = 0; i < 16; ++i) u[i] = u0_sm[(32 * (i / 8) + 8 * part + i % 8) * kDv];
      wait(&done[0], c, 0x415);
      tc_fence_after();
      float zero[2] = {};  // NaN where an update is not finite
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        uint32_t x[8];
        tmem_ld8(lanes + kScanTmX + uint32_t(32 * h + 8 * part), x);
#pragma unroll
        for (int i = 0; i < 8; ++i) {
          u[8 * h + i] -= __uint_as_float(x[i]);
          zero[h] = fmaf(u[8 * h + i], 0.0f, zero[h]);
        }
      }
      if (zero[0] + zero[1] != 0.0f) *not_finite = c + 1;
      __syncwarp();  // together for the stores to tensor memory
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        eight_to_tmem(kScanTmU + uint32_t(16 * h + 4 * part), 32, u + 8 * h);
        arrive(&u_ready[h]);
      }
      wait(&done[1], c, 0x416);
      tc_fence_after();
      uint32_t y[16];
#pragma unroll
      for (int h = 0; h < 2; ++h) {
#pragma unroll
        for (int e = 0; e < 2; ++e) {
          uint32_t d[8];
          tmem_ld8(lanes + kScanTmD + uint32_t(64 * h + 16 * part + 8 * e), d);
#pragma unroll
          for (int i = 0; i < 8; ++i) S[16 * h + 8 * e + i] = eC * S[16 * h + 8 * e + i] + __uint_as_float(d[i]);
          if (more) eight_to_tmem(kScanTmS + uint32_t(32 * h + 8 * part + 4 * e), 64, S + 16 * h + 8 * e);
        }
        if (h == 0) {  // the next product (1) overwrites the outputs and the first half of D
          wait(&done[2], c, 0x417);
          tc_fence_after();
          tmem_ld16(lanes + kScanTmY + uint32_t(16 * part), y);
        }
        if (more) arrive(&s_ready[h]);
      }
#pragma unroll
      for (int i = 0; i < 16; ++i) {  // after the arrivals, which would wait for the stores to leave
        const int t = 16 * part + i;
        if (t < nc) o_g[(size_t)(c * kCh + t) * nv * kDv] = __uint_as_float(y[i]);
      }
    }
#pragma unroll
    for (int i = 0; i < 8; ++i)
      *reinterpret_cast<float4*>(S_out + v * kLd + 64 * (i / 4) + 16 * part + 4 * (i % 4)) =
          make_float4(S[4 * i], S[4 * i + 1], S[4 * i + 2], S[4 * i + 3]);
    named_bar_sync(1, kScanStateWarps * 32);
    if (alive) {
#pragma unroll 8
      for (int i = tid; i < 128 * 32; i += kScanStateWarps * 32)
        *reinterpret_cast<float4*>(S_g + (size_t)i * 4) = *reinterpret_cast<const float4*>(S_out + (i >> 5) * kLd + 4 * (i & 31));
    }
  } else if (warp >= kScanStateWarps && chunks > 0) {
    // ---- operands in shared memory: a warp takes every seventh row, five rows of each matrix at a time ----
    constexpr int kBatch = 5;
    const int first = warp - kScanStateWarps;
    const uint32_t swz = uint32_t(lane & 1) * 8, piece = uint32_t(lane & 15) >> 1;  // 8 bytes of a 128-byte row: its 16-byte piece, swizzled by the row
    auto place = [&](int row) { return uint32_t(row) * 128 + ((piece ^ uint32_t(row & 7)) << 4) + swz; };
    const float* q0 = qkv + (size_t)s0 * conv_dim + (size_t)kh * kDk + 4 * lane;
    auto scaled = [](const float4& x, float s) { return make_float4(s * x.x, s * x.y, s * x.z, s * x.w); };
    auto arrive = [&](uint64_t* bar) {
      fence_async_smem();
      __syncwarp();
      if (lane == 0) mbar_arrive(bar);
    };
    auto stage_wq = [&](int c) {
      const float* in = in0 + c * in_step;
      const int nc = min(kCh, n - c * kCh);
      uint8_t* dst = smem + kScanWq + (lane >> 4) * kScanWqSlice;
#pragma unroll 1
      for (int t0 = first; t0 < kCh; t0 += kBatch * kScanLoadWarps) {
        float4 q[kBatch], w[kBatch];
        float lg[kBatch];
#pragma unroll
        for (int i = 0; i < kBatch; ++i) {
          const int t = t0 + i * kScanLoadWarps;
          q[i] = t < nc ? ld_once(q0 + (size_t)(c * kCh + t) * conv_dim) : make_float4(0, 0, 0, 0);
          w[i] = ld_once(in + kCh * 128 + min(t, kCh - 1) * 128 + 4 * lane);
          lg[i] = in[kLgAt + min(t, kCh - 1)];
        }
        if (t0 == first && c > 0) wait(&u_ready[1], c - 1, 0x419);
#pragma unroll
        for (int i = 0; i < kBatch; ++i) {
          const int t = t0 + i * kScanLoadWarps;
          if (t < kCh) {
            store_terms(dst + place(t), kScanWqTerm, scaled(q[i], expf(lg[i])));
            store_terms(dst + place(kCh + t), kScanWqTerm, w[i]);
          }
        }
      }
      arrive(wq_full);
    };
    auto stage_kp = [&](int c) {
      const float* in = in0 + c * in_step;
      const int nc = min(kCh, n - c * kCh);
      const float lgC = in[kLgAt + kCh - 1];
      uint8_t* dst = smem + kScanK + (lane >> 4) * (kCh * 128);
#pragma unroll 1
      for (int t0 = first; t0 < kCh; t0 += kBatch * kScanLoadWarps) {
        float4 k[kBatch], p[kBatch];
        float lg[kBatch];
#pragma unroll
        for (int i = 0; i < kBatch; ++i) {  // of P two rows at a time: the first batch is all of it
          const int t = t0 + i * kScanLoadWarps;
          k[i] = t < nc ? ld_once(q0 + (size_t)(c * kCh + t) * conv_dim + (size_t)nk * kDk) : make_float4(0, 0, 0, 0);
          lg[i] = in[kLgAt + min(t, kCh - 1)];
          if (t < kCh / 2) p[i] = ld_once(in + 2 * kCh * 128 + t * 128 + 4 * lane);
        }
        if (t0 == first) {  // the state has been read from there, or the last chunk's products are complete
          if (c > 0) wait(&done[2], c - 1, 0x41a);
          else wait(&s_ready[1], 0, 0x41c);
        }
#pragma unroll
        for (int i = 0; i < kBatch; ++i) {
          const int t = t0 + i * kScanLoadWarps;
          if (t < kCh) store_terms(dst + place(t), kScanKTerm, scaled(k[i], expf(lgC - lg[i])));
          if (t < kCh / 2) store_terms(smem + kScanP + place(2 * t + (lane >> 4)), kScanPTerm, p[i]);
        }
      }
      arrive(kp_full);
    };
    static_assert(kBatch * kScanLoadWarps >= kCh / 2, "P goes with the first batch");
#pragma unroll 1
    for (int c = 0; c <= chunks; ++c) {
      if (c > 0) stage_kp(c - 1);
      if (c < chunks) stage_wq(c);
    }
  }
  tc_fence_before();
  __syncthreads();
  if (warp == kScanMmaWarp) tmem_dealloc(tmem, 512);
}

// Gated RMSNorm of the scans' outputs: a warp takes two (token, v head) pairs, all their loads first. VEC: four neighbouring
// values per lane (gates and results at 8-byte boundaries), else every 32nd, any alignment.
// Bound by its bytes (o fp32, z and the result bf16).
constexpr int kGateWarps = 8, kGateItems = 2;
template <bool VEC>
__global__ void __launch_bounds__(kGateWarps * 32) gdn_norm_gate_kernel(const float* __restrict__ o,
                                                                        const __nv_bfloat16* __restrict__ z, int ld_z,
                                                                        const float* __restrict__ norm_w, float eps,
                                                                        __nv_bfloat16* __restrict__ out, const int* __restrict__ seq_start,
                                                                        int nv, int items) {
  pdl_wait();
  pdl_launch_dependents();
  const int row0 = seq_start[0];  // of the step's arrays; o starts with the batch's first row
  const int first = (blockIdx.x * kGateWarps + (threadIdx.x >> 5)) * kGateItems, lane = threadIdx.x & 31;
  auto at = [&](int j) { return VEC ? 4 * lane + j : lane + 32 * j; };
  float v[kGateItems][4], zz[kGateItems][4], nw[4];
#pragma unroll
  for (int i = 0; i < kGateItems; ++i) {
    const int item = min(first + i, items - 1), m = item / nv, vh = item - m * nv;
    const float* src = o + (size_t)item * kDv;
    const __nv_bfloat16* gate = z + (size_t)(row0 + m) * ld_z + (size_t)vh * kDv;
    if constexpr (VEC) {
      const float4 x = *reinterpret_cast<const float4*>(src + 4 * lane);
      const uint2 y = *reinterpret_cast<const uint2*>(gate + 4 * lane);
      v[i][0] = x.x;
      v[i][1] = x.y;
      v[i][2] = x.z;
      v[i][3] = x.w;
      zz[i][0] = __uint_as_float(y.x << 16);
      zz[i][1] = __uint_as_float(y.x & 0xffff0000u);
      zz[i][2] = __uint_as_float(y.y << 16);
      zz[i][3] = __uint_as_float(y.y & 0xffff0000u);
    } else {
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        v[i][j] = src[at(j)];
        zz[i][j] = __bfloat162float(gate[at(j)]);
      }
    }
  }
#pragma unroll
  for (int j = 0; j < 4; ++j) nw[j] = norm_w[at(j)];
#pragma unroll
  for (int i = 0; i < kGateItems; ++i) {
    const float ss = warp_sum((v[i][0] * v[i][0] + v[i][1] * v[i][1]) + (v[i][2] * v[i][2] + v[i][3] * v[i][3]));
    const float r = 1.0f / sqrtf(ss / float(kDv) + eps);
    if (first + i >= items) return;
    __nv_bfloat16* dst = out + ((size_t)row0 * nv + first + i) * kDv;
    __nv_bfloat162 y[2];
    y[0] = __floats2bfloat162_rn(v[i][0] * r * nw[0] * silu_f(zz[i][0]), v[i][1] * r * nw[1] * silu_f(zz[i][1]));
    y[1] = __floats2bfloat162_rn(v[i][2] * r * nw[2] * silu_f(zz[i][2]), v[i][3] * r * nw[3] * silu_f(zz[i][3]));
    if constexpr (VEC) {
      *reinterpret_cast<uint2*>(dst + 4 * lane) = *reinterpret_cast<const uint2*>(y);
    } else {
      dst[at(0)] = y[0].x;
      dst[at(1)] = y[0].y;
      dst[at(2)] = y[1].x;
      dst[at(3)] = y[1].y;
    }
  }
}

}  // namespace

int g_chunk_scan_tensor_cores = 1;

Q38_REGISTER_ERROR_WORD();

}  // namespace q38

using namespace q38;

extern "C" int q38_gdn_ab(const q38_bf16* xbf, int m, int hidden, const q38_bf16* w_ab, int rows,
                          const float* partials_in, float eps, float* ab_out, void* stream) {
  if (m == 0) return Q38_OK;
  Q38_REQUIRE(xbf && w_ab && ab_out, "gdn_ab: null argument");
  Q38_REQUIRE(m > 0 && hidden > 0 && hidden % 128 == 0 && rows > 0, "gdn_ab: m %d hidden %d rows %d", m, hidden, rows);
  const int tile = m > 256 ? 2 : 1;
  (void)launch_kernel(tile == 2 ? gdn_ab_kernel<2, 2> : gdn_ab_kernel<1, 1>,
                      dim3((rows + 8 * tile - 1) / (8 * tile), (m + 16 * tile - 1) / (16 * tile)), dim3(kAbWarps * 32), 0,
                      as_stream(stream), reinterpret_cast<const __nv_bfloat16*>(xbf), m, hidden,
                      reinterpret_cast<const __nv_bfloat16*>(w_ab), rows, partials_in, eps, ab_out);
  Q38_LAUNCH_OK("gdn_ab_kernel");
  return Q38_OK;
}

extern "C" int q38_gdn_conv(const q38_gdn_conv_params* p, const q38_gdn_dims* d, const q38_batch_desc* batch,
                            const q38_gdn_state_desc* st, void* stream) {
  Q38_REQUIRE(p && d && batch && st, "gdn_conv: null argument");
  if (batch->num_tokens == 0) return Q38_OK;
  Q38_REQUIRE(d->conv_dim == (2 * d->num_k_heads + d->num_v_heads) * 128, "gdn_conv: conv_dim %d", d->conv_dim);
  Q38_REQUIRE(p->proj && p->conv_w && p->qkv && st->conv, "gdn_conv: null pointer");
  const cudaStream_t s = as_stream(stream);
  const __nv_bfloat16* proj = reinterpret_cast<const __nv_bfloat16*>(p->proj);
  __nv_bfloat16* cs = reinterpret_cast<__nv_bfloat16*>(st->conv);
  // decode batches (one token per sequence) roll the conv state inside the conv kernel; longer runs need the second
  // kernel, because the first three tokens of a run all read the old taps
  const int roll = batch->max_tokens_per_seq == 1 ? 1 : 0;
  const bool many = batch->num_tokens >= 256 && !roll;  // tokens per warp: one for latency, kConvBlock from 256 tokens on
  const bool each = roll && batch->num_tokens == batch->num_seqs;
  const bool vectors = d->ld_proj % 4 == 0 && (reinterpret_cast<uintptr_t>(p->proj) | reinterpret_cast<uintptr_t>(cs)) % 8 == 0 &&
                       reinterpret_cast<uintptr_t>(p->qkv) % 16 == 0;
  if (vectors) {
    const int per_cta = kConvWarps * (many ? kConvBlock : 1);
    (void)launch_kernel(many ? gdn_conv_vec_kernel<kConvBlock> : gdn_conv_vec_kernel<1>,
                        dim3(d->conv_dim / 128, (batch->num_tokens + per_cta - 1) / per_cta), dim3(kConvWarps * 32), 0, s, proj,
                        d->ld_proj, p->conv_w, p->qkv, d->conv_dim, d->num_k_heads * 128, p->gdn_layer, st->num_gdn_layers, cs,
                        batch->seq_start, batch->seq_slot, batch->tok_seq, batch->num_tokens, roll, each ? 1 : 0);
    Q38_LAUNCH_OK("gdn_conv_vec_kernel");
  } else if (many) {  // any alignment
    (void)launch_kernel(gdn_conv_block_kernel, dim3(d->conv_dim / 128, (batch->num_tokens + kConvWindow - 1) / kConvWindow),
                        dim3(128), 0, s, proj, d->ld_proj, p->conv_w, p->qkv, d->conv_dim, d->num_k_heads * 128,
                        p->gdn_layer, st->num_gdn_layers, static_cast<const __nv_bfloat16*>(cs), batch->seq_start,
                        batch->seq_slot, batch->tok_seq, batch->num_tokens);
    Q38_LAUNCH_OK("gdn_conv_block_kernel");
  } else {
    const int per_cta = batch->num_tokens >= 256 ? 8 : 1;
    (void)launch_kernel(gdn_conv_kernel, dim3(d->conv_dim / 128, (batch->num_tokens + per_cta - 1) / per_cta),
                        dim3(128), 0, s, proj, d->ld_proj, p->conv_w, p->qkv, d->conv_dim, d->num_k_heads * 128,
                        p->gdn_layer, st->num_gdn_layers, cs, batch->seq_start, batch->seq_slot, batch->tok_seq, roll,
                        batch->num_tokens, per_cta, each ? 1 : 0);
    Q38_LAUNCH_OK("gdn_conv_kernel");
  }
  if (roll) return Q38_OK;
  (void)launch_kernel(gdn_conv_state_kernel, dim3(d->conv_dim / 128, batch->num_seqs), dim3(128), 0, s, 
      proj, d->ld_proj, d->conv_dim, p->gdn_layer, st->num_gdn_layers, cs, batch->seq_start, batch->seq_slot);
  Q38_LAUNCH_OK("gdn_conv_state_kernel");
  return Q38_OK;
}

extern "C" int q38_gdn_recurrence(const q38_gdn_recurrence_params* p, const q38_gdn_dims* d,
                                  const q38_batch_desc* batch, const q38_gdn_state_desc* st, void* stream) {
  Q38_REQUIRE(p && d && batch && st, "gdn_recurrence: null argument");
  if (batch->num_tokens == 0) return Q38_OK;
  Q38_REQUIRE(d->num_k_heads > 0 && d->num_v_heads % d->num_k_heads == 0, "gdn_recurrence: head ratio");
  Q38_REQUIRE(p->qkv && p->ab && p->A && p->dt_bias && p->z && p->norm_w && p->out && st->recurrent,
              "gdn_recurrence: null pointer");
  if (batch->max_tokens_per_seq == 1) {
    static const cudaError_t attr = cudaFuncSetAttribute(gdn_recurrence_decode_kernel,
                                                         cudaFuncAttributeMaxDynamicSharedMemorySize, kDecSmemBytes);
    Q38_CUDA_OK(attr);
    Q38_REQUIRE(d->conv_dim % 4 == 0 && p->ld_z % 8 == 0 && reinterpret_cast<uintptr_t>(p->qkv) % 16 == 0 &&
                    reinterpret_cast<uintptr_t>(p->z) % 16 == 0 && reinterpret_cast<uintptr_t>(st->recurrent) % 16 == 0,
                "gdn_recurrence: rows of qkv, z and the state must be 16-byte aligned");
    const int items = batch->num_seqs * d->num_v_heads;
    (void)launch_kernel(gdn_recurrence_decode_kernel, dim3(std::min(num_sms(), items)), dim3(kDecThreads), kDecSmemBytes, as_stream(stream), 
        p->qkv, d->conv_dim, p->ab, p->A, p->dt_bias, reinterpret_cast<const __nv_bfloat16*>(p->z), p->ld_z, p->norm_w,
        p->eps, reinterpret_cast<__nv_bfloat16*>(p->out), p->gdn_layer, st->num_gdn_layers, d->num_k_heads,
        d->num_v_heads, st->recurrent, batch->seq_start, batch->seq_slot, batch->num_seqs);
    Q38_LAUNCH_OK("gdn_recurrence_decode_kernel");
    return Q38_OK;
  }
  (void)launch_kernel(gdn_recurrence_kernel, dim3(d->num_v_heads, batch->num_seqs), dim3(kRecWarps * 32), 0, as_stream(stream), 
      p->qkv, d->conv_dim, p->ab, p->A, p->dt_bias, reinterpret_cast<const __nv_bfloat16*>(p->z), p->ld_z, p->norm_w,
      p->eps, reinterpret_cast<__nv_bfloat16*>(p->out), p->gdn_layer, st->num_gdn_layers, d->num_k_heads,
      d->num_v_heads, st->recurrent, batch->seq_start, batch->seq_slot);
  Q38_LAUNCH_OK("gdn_recurrence_kernel");
  return Q38_OK;
}

extern "C" void q38_gdn_set_chunk_scan_tensor_cores(int on) { q38::g_chunk_scan_tensor_cores = on != 0; }

extern "C" size_t q38_gdn_chunk_scratch_floats(int max_tokens, int max_seqs, int num_v_heads) {
  // per-chunk U0 / W / P / lg for every chunk slot, then one [tokens][v heads * 128] fp32 row block for the split scan
  return (size_t)(max_tokens / kCh + max_seqs) * (size_t)num_v_heads * kChunkFloats +
         (size_t)max_tokens * (size_t)num_v_heads * kDv;
}

extern "C" int q38_gdn_recurrence_chunked(const q38_gdn_recurrence_params* p, const q38_gdn_dims* d,
                                          const q38_batch_desc* batch, const q38_gdn_state_desc* st, float* scratch,
                                          size_t scratch_floats, void* stream) {
  Q38_REQUIRE(p && d && batch && st, "gdn_recurrence_chunked: null argument");
  if (batch->num_tokens == 0) return Q38_OK;
  Q38_REQUIRE(d->num_k_heads > 0 && d->num_v_heads % d->num_k_heads == 0, "gdn_recurrence_chunked: head ratio");
  Q38_REQUIRE(p->qkv && p->ab && p->A && p->dt_bias && p->z && p->norm_w && p->out && st->recurrent && scratch,
              "gdn_recurrence_chunked: null pointer");
  Q38_REQUIRE(d->conv_dim % 4 == 0 && reinterpret_cast<uintptr_t>(p->qkv) % 16 == 0 &&
                  reinterpret_cast<uintptr_t>(scratch) % 16 == 0 && reinterpret_cast<uintptr_t>(st->recurrent) % 16 == 0,
              "gdn_recurrence_chunked: qkv rows, scratch and state must be 16-byte aligned");
  Q38_REQUIRE(batch->max_tokens_per_seq >= 1, "gdn_recurrence_chunked: max_tokens_per_seq %d", batch->max_tokens_per_seq);
  const size_t need = q38_gdn_chunk_scratch_floats(batch->num_tokens, batch->num_seqs, d->num_v_heads);
  Q38_REQUIRE(scratch_floats >= need, "gdn_recurrence_chunked: scratch of %zu floats, %zu needed", scratch_floats, need);
  static const cudaError_t attr1[4] = {
      cudaFuncSetAttribute(gdn_chunk_prep_kernel<1, 256>, cudaFuncAttributeMaxDynamicSharedMemorySize, prep_smem_bytes(1)),
      cudaFuncSetAttribute(gdn_chunk_prep_kernel<1, 512>, cudaFuncAttributeMaxDynamicSharedMemorySize, prep_smem_bytes(1)),
      cudaFuncSetAttribute(gdn_chunk_prep_kernel<2, 256>, cudaFuncAttributeMaxDynamicSharedMemorySize, prep_smem_bytes(2)),
      cudaFuncSetAttribute(gdn_chunk_prep_kernel<3, 384>, cudaFuncAttributeMaxDynamicSharedMemorySize, prep_smem_bytes(3))};
  for (const cudaError_t e : attr1) Q38_CUDA_OK(e);
  static const cudaError_t attr2 =
      cudaFuncSetAttribute(gdn_chunk_scan_kernel<1>, cudaFuncAttributeMaxDynamicSharedMemorySize, kScanSmemBytes);
  static const cudaError_t attr3 =
      cudaFuncSetAttribute(gdn_chunk_scan_kernel<2>, cudaFuncAttributeMaxDynamicSharedMemorySize, kScanSmemBytes);
  static const cudaError_t attr4 =
      cudaFuncSetAttribute(gdn_chunk_scan_umma_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kScanUmmaSmem);
  Q38_CUDA_OK(attr2);
  Q38_CUDA_OK(attr3);
  Q38_CUDA_OK(attr4);
  const cudaStream_t s = as_stream(stream);
  const int max_chunks = (batch->max_tokens_per_seq + kCh - 1) / kCh;
  // several value heads per CTA unless that leaves SMs idle (two CTAs of one head fit an SM, with 256 threads each; with an SM
  // to itself a CTA has 512 for the products: 130 tokens of 48 heads, whole mixer 146 -> 138 us)
  const int ratio = d->num_v_heads / d->num_k_heads;
  const long long singles = (long long)max_chunks * batch->num_seqs * d->num_v_heads;
  const int heads = ratio == 1 || singles <= 2 * num_sms() ? 1 : ratio % 2 == 0 ? 2 : 3;
  auto prep = [&](auto kernel, int threads) {
    (void)launch_kernel(kernel, dim3(max_chunks, d->num_k_heads * ((ratio + heads - 1) / heads), batch->num_seqs),
                        dim3(threads), prep_smem_bytes(heads), s, p->qkv, d->conv_dim, p->ab, p->A, p->dt_bias,
                        d->num_k_heads, d->num_v_heads, batch->seq_start, scratch);
  };
  if (heads == 3) prep(gdn_chunk_prep_kernel<3, 384>, 384);
  else if (heads == 2) prep(gdn_chunk_prep_kernel<2, 256>, 256);
  else if (singles > num_sms()) prep(gdn_chunk_prep_kernel<1, 256>, 256);
  else prep(gdn_chunk_prep_kernel<1, 512>, 512);
  Q38_LAUNCH_OK("gdn_chunk_prep_kernel");
  const __nv_bfloat16* zp = reinterpret_cast<const __nv_bfloat16*>(p->z);
  __nv_bfloat16* outp = reinterpret_cast<__nv_bfloat16*>(p->out);
  float* o_scratch = scratch + (size_t)(batch->num_tokens / kCh + batch->num_seqs) * (size_t)d->num_v_heads * kChunkFloats;
  auto norm_gate = [&]() -> int {
    const int items = batch->num_tokens * d->num_v_heads;
    const bool vec = p->ld_z % 4 == 0 && (reinterpret_cast<uintptr_t>(p->z) | reinterpret_cast<uintptr_t>(p->out)) % 8 == 0;
    const int per_cta = kGateWarps * kGateItems;
    (void)launch_kernel(vec ? gdn_norm_gate_kernel<true> : gdn_norm_gate_kernel<false>, dim3((items + per_cta - 1) / per_cta),
                        dim3(kGateWarps * 32), 0, s, o_scratch, zp, p->ld_z, p->norm_w, p->eps, outp, batch->seq_start, d->num_v_heads, items);
    Q38_LAUNCH_OK("gdn_norm_gate_kernel");
    return Q38_OK;
  };
  if (g_chunk_scan_tensor_cores != 0) {
    (void)launch_kernel(gdn_chunk_scan_umma_kernel, dim3(d->num_v_heads, batch->num_seqs), dim3(kScanThreads), kScanUmmaSmem, s,
                        p->qkv, d->conv_dim, p->gdn_layer, st->num_gdn_layers, d->num_k_heads, d->num_v_heads, st->recurrent,
                        batch->seq_start, batch->seq_slot, scratch, o_scratch);
    Q38_LAUNCH_OK("gdn_chunk_scan_umma_kernel");
    return norm_gate();
  }
  // fp32: one CTA per (v head, sequence); with few of them, two CTAs share a head's state rows
  const bool split = 2 * d->num_v_heads * batch->num_seqs <= num_sms();
  (void)launch_kernel(split ? gdn_chunk_scan_kernel<2> : gdn_chunk_scan_kernel<1>, dim3((split ? 2 : 1) * d->num_v_heads, batch->num_seqs),
                      dim3(kChunkThreads), kScanSmemBytes, s, p->qkv, d->conv_dim, zp, p->ld_z, p->norm_w, p->eps, outp,
                      p->gdn_layer, st->num_gdn_layers, d->num_k_heads, d->num_v_heads, st->recurrent, batch->seq_start,
                      batch->seq_slot, scratch, o_scratch);
  Q38_LAUNCH_OK("gdn_chunk_scan_kernel");
  return split ? norm_gate() : Q38_OK;
}
