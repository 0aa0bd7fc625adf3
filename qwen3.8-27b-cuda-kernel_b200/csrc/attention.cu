// Full-attention layers: fused q/k-norm + partial RoPE + KV quantise + paged append, split-KV GQA
// flash-decoding with the merge + sigmoid output gate, and chunked-prefill causal attention over the
// paged int8 / bf16 KV cache.
//
// Replaces kernels::qk_norm_rope_append, attention_decode(+_splits) and attention_prefill of the
// reference (src/kernels/kernels.h:140-179; src/kernels/qk_norm_rope.cu, attention_decode.cu,
// attention_prefill.cu). Page layout per (layer, page): K [kv_head][64][256], V same, then (int8) fp16
// scales K [kv_head][64][4], V same (reference docs/FORMAT.md 3.1).
#include <algorithm>
#include <climits>
#include <cmath>
#include <type_traits>

#include "common.cuh"
#include "host_util.h"
#include "tcgen05.cuh"

namespace q38 {
namespace {

constexpr int kHd = Q38_HEAD_DIM;
constexpr int kPage = Q38_PAGE_TOKENS;

struct KvView {
  uint8_t* pool;
  int int8;
  int kv_heads;
  int num_pages;
  size_t page_bytes;
  size_t layer_stride;
  const int* block_table;
  int max_pages_per_seq;

  __device__ __forceinline__ size_t elem() const { return int8 ? 1 : 2; }
  __device__ __forceinline__ size_t k_off(int head, int tok) const { return ((size_t)head * kPage + tok) * kHd * elem(); }
  __device__ __forceinline__ size_t v_off(int head, int tok) const {
    return (size_t)kv_heads * kPage * kHd * elem() + k_off(head, tok);
  }
  __device__ __forceinline__ size_t ks_off(int head, int tok) const {
    return 2 * (size_t)kv_heads * kPage * kHd + ((size_t)head * kPage + tok) * 8;
  }
  __device__ __forceinline__ size_t vs_off(int head, int tok) const {
    return ks_off(head, tok) + (size_t)kv_heads * kPage * 8;
  }
  // base of the (layer, page) block holding position `pos` of `slot`; nullptr if the table entry is invalid
  __device__ __forceinline__ uint8_t* page_of(int layer, int slot, int pos) const {
    const int page = block_table[(size_t)slot * max_pages_per_seq + pos / kPage];
    if (page < 0 || page >= num_pages) return nullptr;
    return pool + (size_t)layer * layer_stride + (size_t)page * page_bytes;
  }
};

KvView make_view(const q38_kv_cache_desc& d) {
  KvView v;
  v.pool = d.pool;
  v.int8 = d.dtype == Q38_KV_INT8;
  v.kv_heads = d.kv_heads;
  v.num_pages = d.num_pages;
  v.page_bytes = d.page_bytes;
  v.layer_stride = d.layer_stride;
  v.block_table = d.block_table;
  v.max_pages_per_seq = d.max_pages_per_seq;
  return v;
}

struct RopeTable {
  float inv_freq[32];  // evaluated on the host exactly as the CPU oracle does (src/ref/ops.cpp:104)
};

// ---------------------------------------------------------------------------------------------------
// qk_norm_rope_append: one CTA per token, one warp per head (nq query heads, nkv key heads, nkv value
// heads); a lane owns 8 consecutive dims. Rounding points (reference src/kernels/qk_norm_rope.cu:38-89,
// oracle src/ref/ops.cpp:79-142): q -> fp16; K (after norm + RoPE) and V (raw) -> int8 with one fp16
// scale = amax / 127 per 64 dims, q = clamp(rint(x / scale), +-127); or bf16.
// ---------------------------------------------------------------------------------------------------
__global__ void __launch_bounds__(1024) qk_norm_rope_kernel(const __nv_bfloat16* __restrict__ proj, int ld_proj,
                                                            const float* __restrict__ q_norm,
                                                            const float* __restrict__ k_norm, float eps, int nq, int nkv,
                                                            __half* __restrict__ q_out, int layer,
                                                            const __grid_constant__ RopeTable rope,
                                                            const int* __restrict__ tok_pos,
                                                            const int* __restrict__ tok_seq,
                                                            const int* __restrict__ seq_slot, KvView kv) {
  pdl_wait();               // everything written by earlier kernels of the stream is visible from here on
  pdl_launch_dependents();  // the next kernel may be scheduled now; it holds its own dependent work back the same way
  const int m = blockIdx.x, warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  // The token's 32 angles are the same for every head: one warp evaluates their cosines and sines (each head's warp for itself,
  // eight lanes at a time, they were most of the kernel: 24 us for 512 tokens of 24 + 4 heads).
  __shared__ float2 trig[32];
  const int pos = tok_pos[m];
  if (warp == 0) {
    const float angle = float(pos) * rope.inv_freq[lane];
    trig[lane] = make_float2(cosf(angle), sinf(angle));
  }
  __syncthreads();
  if (warp >= nq + 2 * nkv) return;
  const bool is_q = warp < nq, is_k = !is_q && warp < nq + nkv;
  const int head = is_q ? warp : is_k ? warp - nq : warp - nq - nkv;
  const size_t col = is_q ? (size_t)head * kHd : is_k ? (size_t)(2 * nq + head) * kHd : (size_t)(2 * nq + nkv + head) * kHd;
  const uint4 raw = *reinterpret_cast<const uint4*>(proj + (size_t)m * ld_proj + col + 8 * lane);
  const __nv_bfloat162* rp = reinterpret_cast<const __nv_bfloat162*>(&raw);
  float x[8];
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    x[2 * i] = __low2float(rp[i]);
    x[2 * i + 1] = __high2float(rp[i]);
  }
  if (is_q || is_k) {
    float ss = 0.0f;
#pragma unroll
    for (int i = 0; i < 8; ++i) ss += x[i] * x[i];
    ss = warp_sum(ss);
    const float r = 1.0f / sqrtf(ss / float(kHd) + eps);
    const float* w = (is_q ? q_norm : k_norm) + 8 * lane;
#pragma unroll
    for (int i = 0; i < 8; ++i) x[i] = x[i] * r * w[i];
    // partial RoPE on dims (i, i + 32), i < 32: lanes 0-3 hold dims 0..31, lanes 4-7 hold dims 32..63
    float other[8];
#pragma unroll
    for (int i = 0; i < 8; ++i) other[i] = __shfl_xor_sync(0xffffffffu, x[i], 4);
    if (lane < 8) {
      const bool low = lane < 4;
#pragma unroll
      for (int i = 0; i < 8; ++i) {
        const float c = trig[8 * (lane & 3) + i].x, s = trig[8 * (lane & 3) + i].y;
        // low half: x1 c - x2 s ; high half: x2 c + x1 s
        x[i] = low ? x[i] * c - other[i] * s : x[i] * c + other[i] * s;
      }
    }
  }
  if (is_q) {
    __half2 h[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) h[i] = __floats2half2_rn(x[2 * i], x[2 * i + 1]);
    *reinterpret_cast<uint4*>(q_out + ((size_t)m * nq + head) * kHd + 8 * lane) = *reinterpret_cast<uint4*>(h);
    return;
  }
  const int slot = seq_slot[tok_seq[m]];
  uint8_t* page = kv.page_of(layer, slot, pos);
  if (page == nullptr) {
    report_error(0x201);
    return;
  }
  const int tok = pos % kPage;
  if (kv.int8) {
    float amax = 0.0f;
#pragma unroll
    for (int i = 0; i < 8; ++i) amax = fmaxf(amax, fabsf(x[i]));
    // one scale per 64 dims = 8 lanes
#pragma unroll
    for (int o = 4; o > 0; o >>= 1) amax = fmaxf(amax, __shfl_xor_sync(0xffffffffu, amax, o));
    const __half sh = __float2half_rn(amax / 127.0f);
    const float scale = __half2float(sh);
    uint32_t packed[2] = {0u, 0u};
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      float q = 0.0f;
      if (scale > 0.0f) q = fminf(fmaxf(rintf(x[i] / scale), -127.0f), 127.0f);
      packed[i >> 2] |= (uint32_t(int(q)) & 255u) << (8 * (i & 3));
    }
    uint8_t* dst = page + (is_k ? kv.k_off(head, tok) : kv.v_off(head, tok)) + 8 * lane;
    *reinterpret_cast<uint2*>(dst) = make_uint2(packed[0], packed[1]);
    if ((lane & 7) == 0) {
      uint8_t* sdst = page + (is_k ? kv.ks_off(head, tok) : kv.vs_off(head, tok)) + 2 * (lane >> 3);
      *reinterpret_cast<__half*>(sdst) = sh;
    }
  } else {
    __nv_bfloat162 b[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) b[i] = __floats2bfloat162_rn(x[2 * i], x[2 * i + 1]);
    uint8_t* dst = page + (is_k ? kv.k_off(head, tok) : kv.v_off(head, tok)) + 16 * lane;
    *reinterpret_cast<uint4*>(dst) = *reinterpret_cast<uint4*>(b);
  }
}

// ---------------------------------------------------------------------------------------------------
// Token attention (generic path): one CTA per (split, kv head, row). A row is one query token with its
// causal length L; the GROUP query heads of the kv head share every K/V byte read. Warps stride over
// the keys of the split, a lane owns 8 dims; online softmax in the log2 domain; the warps' states are
// merged through shared memory. With num_splits == 1 the CTA normalises, applies the sigmoid gate and
// writes bf16 itself; otherwise it writes (acc[256], m, l) per head to the scratch for the merge kernel.
// Serves decode (row = sequence, L = pos0 + 1) and, as the first prefill implementation, every prompt
// token of a chunk (row = token, L = pos + 1).
// ---------------------------------------------------------------------------------------------------
constexpr int kAttnWarps = 4;
constexpr float kLog2e = 1.4426950408889634f;

template <int GROUP, bool INT8>
__global__ void __launch_bounds__(kAttnWarps * 32) attn_token_kernel(
    const __half* __restrict__ q, const __nv_bfloat16* __restrict__ gate, int ld_gate, __nv_bfloat16* __restrict__ out,
    int nq, int layer, float* __restrict__ scratch, int max_splits, int num_splits, int decode_rows,
    const int* __restrict__ seq_start, const int* __restrict__ seq_slot, const int* __restrict__ seq_pos0,
    const int* __restrict__ tok_pos, const int* __restrict__ tok_seq, KvView kv) {
  pdl_wait();               // everything written by earlier kernels of the stream is visible from here on
  pdl_launch_dependents();  // the next kernel may be scheduled now; it holds its own dependent work back the same way
  const int split = blockIdx.x, kvh = blockIdx.y, row = blockIdx.z;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  int m, slot, L;
  if (decode_rows) {
    m = seq_start[row];
    slot = seq_slot[row];
    L = seq_pos0[row] + 1;
  } else {
    m = row;
    slot = seq_slot[tok_seq[row]];
    L = tok_pos[row] + 1;
  }
  // keys of this split (whole pages except possibly the last)
  const int pages = (L + kPage - 1) / kPage;
  const int pages_per_split = (pages + num_splits - 1) / num_splits;
  const int t0 = min(L, split * pages_per_split * kPage), t1 = min(L, (split + 1) * pages_per_split * kPage);

  float qv[GROUP][8];
#pragma unroll
  for (int h = 0; h < GROUP; ++h) {
    const uint4 raw = *reinterpret_cast<const uint4*>(q + ((size_t)m * nq + kvh * GROUP + h) * kHd + 8 * lane);
    const __half2* hp = reinterpret_cast<const __half2*>(&raw);
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const float2 f = __half22float2(hp[i]);
      qv[h][2 * i] = f.x * (kLog2e / 16.0f);  // 1 / sqrt(256), log2 domain
      qv[h][2 * i + 1] = f.y * (kLog2e / 16.0f);
    }
  }
  float mx[GROUP], l[GROUP], acc[GROUP][8];
#pragma unroll
  for (int h = 0; h < GROUP; ++h) {
    mx[h] = -INFINITY;
    l[h] = 0.0f;
#pragma unroll
    for (int i = 0; i < 8; ++i) acc[h][i] = 0.0f;
  }

  for (int t = t0 + warp; t < t1; t += kAttnWarps) {
    const uint8_t* page = kv.page_of(layer, slot, t);
    if (page == nullptr) {
      report_error(0x202);
      break;
    }
    const int tok = t % kPage;
    float kx[8], vx[8];
    if constexpr (INT8) {
      const uint2 kr = *reinterpret_cast<const uint2*>(page + kv.k_off(kvh, tok) + 8 * lane);
      const uint2 vr = *reinterpret_cast<const uint2*>(page + kv.v_off(kvh, tok) + 8 * lane);
      const float ks = __half2float(*reinterpret_cast<const __half*>(page + kv.ks_off(kvh, tok) + 2 * (lane >> 3)));
      const float vs = __half2float(*reinterpret_cast<const __half*>(page + kv.vs_off(kvh, tok) + 2 * (lane >> 3)));
      const uint32_t kw[2] = {kr.x, kr.y}, vw[2] = {vr.x, vr.y};
#pragma unroll
      for (int i = 0; i < 8; ++i) {
        kx[i] = float(int8_t(kw[i >> 2] >> (8 * (i & 3)))) * ks;
        vx[i] = float(int8_t(vw[i >> 2] >> (8 * (i & 3)))) * vs;
      }
    } else {
      const uint4 kr = *reinterpret_cast<const uint4*>(page + kv.k_off(kvh, tok) + 16 * lane);
      const uint4 vr = *reinterpret_cast<const uint4*>(page + kv.v_off(kvh, tok) + 16 * lane);
      const __nv_bfloat162* kp = reinterpret_cast<const __nv_bfloat162*>(&kr);
      const __nv_bfloat162* vp = reinterpret_cast<const __nv_bfloat162*>(&vr);
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        kx[2 * i] = __low2float(kp[i]);
        kx[2 * i + 1] = __high2float(kp[i]);
        vx[2 * i] = __low2float(vp[i]);
        vx[2 * i + 1] = __high2float(vp[i]);
      }
    }
#pragma unroll
    for (int h = 0; h < GROUP; ++h) {
      float s = 0.0f;
#pragma unroll
      for (int i = 0; i < 8; ++i) s += qv[h][i] * kx[i];
      s = warp_sum(s);
      const float mn = fmaxf(mx[h], s);
      const float corr = exp2f(mx[h] - mn), p = exp2f(s - mn);
      mx[h] = mn;
      l[h] = l[h] * corr + p;
#pragma unroll
      for (int i = 0; i < 8; ++i) acc[h][i] = acc[h][i] * corr + p * vx[i];
    }
  }

  // merge the warps' states: shared [warp][GROUP][256 + 2]
  __shared__ float sm_acc[kAttnWarps][GROUP][kHd];
  __shared__ float sm_ml[kAttnWarps][GROUP][2];
#pragma unroll
  for (int h = 0; h < GROUP; ++h) {
#pragma unroll
    for (int i = 0; i < 8; ++i) sm_acc[warp][h][8 * lane + i] = acc[h][i];
    if (lane == 0) {
      sm_ml[warp][h][0] = mx[h];
      sm_ml[warp][h][1] = l[h];
    }
  }
  __syncthreads();
  for (int idx = threadIdx.x; idx < GROUP * kHd; idx += kAttnWarps * 32) {
    const int h = idx / kHd, d = idx % kHd;
    float mm = -INFINITY;
#pragma unroll
    for (int w = 0; w < kAttnWarps; ++w) mm = fmaxf(mm, sm_ml[w][h][0]);
    float ll = 0.0f, a = 0.0f;
#pragma unroll
    for (int w = 0; w < kAttnWarps; ++w) {
      const float mw = sm_ml[w][h][0];
      const float c = mw == -INFINITY ? 0.0f : exp2f(mw - mm);
      ll += sm_ml[w][h][1] * c;
      a += sm_acc[w][h][d] * c;
    }
    const int qh = kvh * GROUP + h;
    if (num_splits == 1) {
      const float g = __bfloat162float(gate[(size_t)m * ld_gate + (size_t)qh * kHd + d]);
      out[(size_t)m * nq * kHd + (size_t)qh * kHd + d] = __float2bfloat16_rn(a / ll * sigmoid_f(g));
    } else {
      float* dst = scratch + (((size_t)row * nq + qh) * max_splits + split) * (kHd + 2);
      dst[d] = a;
      if (d == 0) {
        dst[kHd] = mm;
        dst[kHd + 1] = ll;
      }
    }
  }
}

// ---------------------------------------------------------------------------------------------------
#ifndef Q38_ATTN_MIN_PAGES_PER_SPLIT
#define Q38_ATTN_MIN_PAGES_PER_SPLIT 8
#endif
constexpr int kMinPagesPerSplit = Q38_ATTN_MIN_PAGES_PER_SPLIT;  // 64-token pages

// Decode attention over int8 KV on tensor cores: one CTA per (split, kv head, sequence), two CTAs per SM.
//   * a producer lane walks the sequence's block-table row and brings one (page, kv head) per stage with four
//     1-D bulk copies: K 16 KB, V 16 KB and their two 512-byte scale rows are each contiguous in the page;
//   * each of the 4 consumer warps owns 16 of the page's 64 tokens. S = K Q^T runs as m16n8k16 f16 MMAs with the
//     tokens as rows and the (<= 8) query heads of the kv head as the 8 columns; the int8 bytes become exact
//     fp16 integers in registers (byte permute into 0x64xx = 1024 + x, minus 1152), and the per-(token, 64-dim)
//     K scale multiplies each 64-dim partial sum in fp32. The order of dims inside an MMA k-step is permuted
//     so that a lane reads 16 contiguous bytes per token (Q fragments use the same permutation);
//   * online softmax in the log2 domain on the accumulator fragments; P is scaled by the V scales, cast to
//     fp16 and transposed in registers (movmatrix) to become the B operand of O^T = V^T P^T, whose A operand
//     pairs two tokens of one dim (bytes of two V rows permuted together);
//   * the warps' (m, l, O) are merged through shared memory; a single split finishes in place (normalise,
//     sigmoid gate, bf16), otherwise the state goes to the scratch for attn_merge_kernel.
// K/V bytes are read from HBM exactly once per GQA group (reference design point: attention_decode.cu).
// ---------------------------------------------------------------------------------------------------
constexpr int kMmaWarps = 4;
constexpr int kMmaThreads = (kMmaWarps + 1) * 32;
constexpr int kMmaStages = 3;
constexpr int kStageK = 0, kStageV = 16384, kStageKs = 32768, kStageVs = 33280, kStageBytes = 33792;
constexpr int kMmaSmem = kMmaStages * kStageBytes + 256;

__device__ __forceinline__ void mma_f16_16816(float (&d)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3,
                                              uint32_t b0, uint32_t b1) {
  asm volatile(
      "mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
      : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
      : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}
__device__ __forceinline__ uint32_t movmatrix_trans(uint32_t a) {
  uint32_t d;
  asm volatile("movmatrix.sync.aligned.m8n8.trans.b16 %0, %1;" : "=r"(d) : "r"(a));
  return d;
}
// two biased bytes (x + 128) of one word -> half2 (x0, x1)
template <int SEL>
__device__ __forceinline__ uint32_t bytes_to_half2(uint32_t w) {
  const uint32_t h = __byte_perm(w, 0x64646464u, SEL);
  const __half2 r = __hsub2(*reinterpret_cast<const __half2*>(&h), __half2half2(__ushort_as_half(0x6480)));
  return *reinterpret_cast<const uint32_t*>(&r);
}
// the four bytes of two words, interleaved: half2 (wa.byte i, wb.byte i), i = 0..3
__device__ __forceinline__ void byte_pairs_to_half2(uint32_t wa, uint32_t wb, uint32_t (&h)[4]) {
  const uint32_t lo = __byte_perm(wa, wb, 0x5140), hi = __byte_perm(wa, wb, 0x7362);
  h[0] = bytes_to_half2<0x4140>(lo);
  h[1] = bytes_to_half2<0x4342>(lo);
  h[2] = bytes_to_half2<0x4140>(hi);
  h[3] = bytes_to_half2<0x4342>(hi);
}

__global__ void __launch_bounds__(kMmaThreads, 2) attn_decode_mma_kernel(
    const __half* __restrict__ q, const __nv_bfloat16* __restrict__ gate, int ld_gate, __nv_bfloat16* __restrict__ out,
    int nq, int group, int layer, float* __restrict__ scratch, int max_splits, int num_splits, int decode_rows,
    const int* __restrict__ seq_start, const int* __restrict__ seq_slot, const int* __restrict__ seq_pos0,
    const int* __restrict__ tok_pos, const int* __restrict__ tok_seq, KvView kv) {
  pdl_wait();               // everything written by earlier kernels of the stream is visible from here on
  pdl_launch_dependents();  // the next kernel may be scheduled now; it holds its own dependent work back the same way
  extern __shared__ __align__(128) uint8_t dsm[];
  uint64_t* full = reinterpret_cast<uint64_t*>(dsm + kMmaStages * kStageBytes);
  uint64_t* empty = full + kMmaStages;
  volatile int* abort_flag = reinterpret_cast<volatile int*>(empty + kMmaStages);
  const int split = blockIdx.x, kvh = blockIdx.y, row = blockIdx.z;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  // a row is a sequence's single new token (decode) or one prompt token of a chunk with its causal length (prefill)
  const int m = decode_rows ? seq_start[row] : row;
  const int slot = decode_rows ? seq_slot[row] : seq_slot[tok_seq[row]];
  const int L = (decode_rows ? seq_pos0[row] : tok_pos[row]) + 1;
  const int pages = (L + kPage - 1) / kPage;
  // a split takes at least kMinPagesPerSplit pages: a short sequence of a ragged batch uses fewer of the launch's
  // splits (the others leave at once) instead of paying a CTA's fixed cost for one or two pages
  const int pages_per_split = max(kMinPagesPerSplit, (pages + num_splits - 1) / num_splits);
  const int p0 = min(pages, split * pages_per_split), p1 = min(pages, (split + 1) * pages_per_split);
  if (p0 >= p1 && num_splits > 1) {  // a split beyond this sequence's pages: an empty state for the merge, nothing else
    if (tid < group) {
      float* dst = scratch + (((size_t)row * nq + (size_t)kvh * group + tid) * max_splits + split) * (kHd + 2);
      dst[kHd] = -INFINITY;
      dst[kHd + 1] = 0.0f;
    }
    return;
  }
  if (tid == 0) {
    for (int s = 0; s < kMmaStages; ++s) {
      mbar_init(&full[s], 1);
      mbar_init(&empty[s], kMmaWarps);
    }
    *abort_flag = 0;
    mbar_fence_init();
  }
  __syncthreads();

  if (warp == kMmaWarps) {
    if (lane == 0) {
      // decode reads every page once; the prompt tokens of a chunk re-read each other's pages out of L2
      const uint64_t pol = decode_rows ? policy_evict_first() : policy_evict_normal();
      const int* table = kv.block_table + (size_t)slot * kv.max_pages_per_seq;
      for (int p = p0, it = 0; p < p1; ++p, ++it) {
        const int s = it % kMmaStages;
        if (*abort_flag || !mbar_wait(&empty[s], ((it / kMmaStages) & 1) ^ 1, 0x211)) {
          *abort_flag = 1;
          break;
        }
        const int page = table[p];
        if (page < 0 || page >= kv.num_pages) {
          report_error(0x212);
          *abort_flag = 1;
          break;
        }
        const uint8_t* base = kv.pool + (size_t)layer * kv.layer_stride + (size_t)page * kv.page_bytes;
        uint8_t* st = dsm + (size_t)s * kStageBytes;
        mbar_expect_tx(&full[s], 2 * 16384 + 2 * 512);
        bulk_g2s(st + kStageK, base + kv.k_off(kvh, 0), 16384, &full[s], pol);
        bulk_g2s(st + kStageV, base + kv.v_off(kvh, 0), 16384, &full[s], pol);
        bulk_g2s(st + kStageKs, base + kv.ks_off(kvh, 0), 512, &full[s], pol);
        bulk_g2s(st + kStageVs, base + kv.vs_off(kvh, 0), 512, &full[s], pol);
      }
    }
    return;
  }

  const int g = lane >> 2, t = lane & 3;
  // Q fragments: head g of the group, dims 64 grp + 16 t + 4 s + {0..3}
  uint32_t qf[4][4][2];
  {
    const bool live = g < group;
    const __half* qrow = q + ((size_t)m * nq + (size_t)kvh * group + (live ? g : 0)) * kHd;
#pragma unroll
    for (int grp = 0; grp < 4; ++grp)
#pragma unroll
      for (int s = 0; s < 4; ++s) {
        const uint2 v = *reinterpret_cast<const uint2*>(qrow + 64 * grp + 16 * t + 4 * s);
        qf[grp][s][0] = live ? v.x : 0u;
        qf[grp][s][1] = live ? v.y : 0u;
      }
  }
  float o[16][4];
#pragma unroll
  for (int T = 0; T < 16; ++T)
#pragma unroll
    for (int c = 0; c < 4; ++c) o[T][c] = 0.0f;
  float m0 = -INFINITY, m1 = -INFINITY, l0 = 0.0f, l1 = 0.0f;  // heads 2t and 2t + 1
  constexpr float kScale = kLog2e / 16.0f;

  for (int p = p0, it = 0; p < p1; ++p, ++it) {
    const int s = it % kMmaStages;
    bool ok = !*abort_flag && mbar_wait(&full[s], (it / kMmaStages) & 1, 0x213);
    ok = __all_sync(0xffffffffu, ok);
    if (!ok) *abort_flag = 1;
    const int tok0 = 16 * warp, tbase = p * kPage + tok0;
    if (ok && tbase < L) {
      const uint8_t* st = dsm + (size_t)s * kStageBytes;
      const uint8_t* Ks = st + kStageK + (size_t)tok0 * kHd;
      const uint8_t* Vs = st + kStageV + (size_t)tok0 * kHd;
      const __half* Ksc = reinterpret_cast<const __half*>(st + kStageKs) + tok0 * 4;
      const __half* Vsc = reinterpret_cast<const __half*>(st + kStageVs) + tok0 * 4;
      // ---- S = K Q^T ----
      float sacc[4] = {0.0f, 0.0f, 0.0f, 0.0f};
#pragma unroll
      for (int grp = 0; grp < 4; ++grp) {
        const uint4 ka = *reinterpret_cast<const uint4*>(Ks + g * kHd + 64 * grp + 16 * t);
        const uint4 kb = *reinterpret_cast<const uint4*>(Ks + (g + 8) * kHd + 64 * grp + 16 * t);
        const uint32_t wa[4] = {ka.x ^ 0x80808080u, ka.y ^ 0x80808080u, ka.z ^ 0x80808080u, ka.w ^ 0x80808080u};
        const uint32_t wb[4] = {kb.x ^ 0x80808080u, kb.y ^ 0x80808080u, kb.z ^ 0x80808080u, kb.w ^ 0x80808080u};
        float d[4] = {0.0f, 0.0f, 0.0f, 0.0f};
#pragma unroll
        for (int ss = 0; ss < 4; ++ss)
          mma_f16_16816(d, bytes_to_half2<0x4140>(wa[ss]), bytes_to_half2<0x4140>(wb[ss]),
                        bytes_to_half2<0x4342>(wa[ss]), bytes_to_half2<0x4342>(wb[ss]), qf[grp][ss][0], qf[grp][ss][1]);
        const float ksa = __half2float(Ksc[g * 4 + grp]), ksb = __half2float(Ksc[(g + 8) * 4 + grp]);
        sacc[0] += ksa * d[0];
        sacc[1] += ksa * d[1];
        sacc[2] += ksb * d[2];
        sacc[3] += ksb * d[3];
      }
      // ---- online softmax over the block's 16 tokens ----
      const bool va = tbase + g < L, vb = tbase + g + 8 < L;
      const float s0 = va ? sacc[0] * kScale : -INFINITY, s1 = va ? sacc[1] * kScale : -INFINITY;
      const float s2 = vb ? sacc[2] * kScale : -INFINITY, s3 = vb ? sacc[3] * kScale : -INFINITY;
      float bm0 = fmaxf(s0, s2), bm1 = fmaxf(s1, s3);
#pragma unroll
      for (int off = 4; off < 32; off <<= 1) {
        bm0 = fmaxf(bm0, __shfl_xor_sync(0xffffffffu, bm0, off));
        bm1 = fmaxf(bm1, __shfl_xor_sync(0xffffffffu, bm1, off));
      }
      const float mn0 = fmaxf(m0, bm0), mn1 = fmaxf(m1, bm1);
      const float c0 = exp2f(m0 - mn0), c1 = exp2f(m1 - mn1);
      const float pr0 = exp2f(s0 - mn0), pr1 = exp2f(s1 - mn1), pr2 = exp2f(s2 - mn0), pr3 = exp2f(s3 - mn1);
      float ls0 = pr0 + pr2, ls1 = pr1 + pr3;
#pragma unroll
      for (int off = 4; off < 32; off <<= 1) {
        ls0 += __shfl_xor_sync(0xffffffffu, ls0, off);
        ls1 += __shfl_xor_sync(0xffffffffu, ls1, off);
      }
      m0 = mn0;
      m1 = mn1;
      l0 = l0 * c0 + ls0;
      l1 = l1 * c1 + ls1;
      if (__any_sync(0xffffffffu, c0 != 1.0f || c1 != 1.0f)) {  // (a maximum moved: rarely, after the first pages)
#pragma unroll
        for (int T = 0; T < 16; ++T) {
          o[T][0] *= c0;
          o[T][1] *= c1;
          o[T][2] *= c0;
          o[T][3] *= c1;
        }
      }
      // ---- O^T += V^T P^T ----
#pragma unroll
      for (int grp = 0; grp < 4; ++grp) {
        const float vsa = __half2float(Vsc[g * 4 + grp]), vsb = __half2float(Vsc[(g + 8) * 4 + grp]);
        const __half2 pa = __floats2half2_rn(pr0 * vsa, pr1 * vsa), pb = __floats2half2_rn(pr2 * vsb, pr3 * vsb);
        const uint32_t b0 = movmatrix_trans(*reinterpret_cast<const uint32_t*>(&pa));
        const uint32_t b1 = movmatrix_trans(*reinterpret_cast<const uint32_t*>(&pb));
#pragma unroll
        for (int jj = 0; jj < 2; ++jj) {
          const int J = 2 * grp + jj;
          const uint8_t* vp = Vs + 32 * J + 4 * g;
          const uint32_t w0 = *reinterpret_cast<const uint32_t*>(vp + (2 * t) * kHd) ^ 0x80808080u;
          const uint32_t w1 = *reinterpret_cast<const uint32_t*>(vp + (2 * t + 1) * kHd) ^ 0x80808080u;
          const uint32_t w2 = *reinterpret_cast<const uint32_t*>(vp + (2 * t + 8) * kHd) ^ 0x80808080u;
          const uint32_t w3 = *reinterpret_cast<const uint32_t*>(vp + (2 * t + 9) * kHd) ^ 0x80808080u;
          uint32_t ha[4], hb[4];
          byte_pairs_to_half2(w0, w1, ha);
          byte_pairs_to_half2(w2, w3, hb);
          mma_f16_16816(o[2 * J], ha[0], ha[1], hb[0], hb[1], b0, b1);
          mma_f16_16816(o[2 * J + 1], ha[2], ha[3], hb[2], hb[3], b0, b1);
        }
      }
    }
    __syncwarp();
    if (lane == 0) mbar_arrive(&empty[s]);
  }

  // ---- merge the four warps (shared memory aliases the drained stages) ----
  named_bar_sync(1, kMmaWarps * 32);
  float* sm_acc = reinterpret_cast<float*>(dsm);                       // [warp][8 heads][256]
  float* sm_ml = sm_acc + kMmaWarps * 8 * kHd;                         // [warp][8 heads][2]
#pragma unroll
  for (int T = 0; T < 16; ++T)
#pragma unroll
    for (int c = 0; c < 4; ++c) {
      const int dim = 32 * (T >> 1) + 4 * g + 2 * (T & 1) + (c >> 1);
      const int head = 2 * t + (c & 1);
      sm_acc[((size_t)warp * 8 + head) * kHd + dim] = o[T][c];
    }
  if (g == 0) {
    sm_ml[(warp * 8 + 2 * t) * 2] = m0;
    sm_ml[(warp * 8 + 2 * t) * 2 + 1] = l0;
    sm_ml[(warp * 8 + 2 * t + 1) * 2] = m1;
    sm_ml[(warp * 8 + 2 * t + 1) * 2 + 1] = l1;
  }
  named_bar_sync(1, kMmaWarps * 32);
  for (int idx = tid; idx < group * kHd; idx += kMmaWarps * 32) {
    const int h = idx / kHd, d = idx % kHd;
    float mm = -INFINITY;
#pragma unroll
    for (int w = 0; w < kMmaWarps; ++w) mm = fmaxf(mm, sm_ml[(w * 8 + h) * 2]);
    float ll = 0.0f, acc = 0.0f;
#pragma unroll
    for (int w = 0; w < kMmaWarps; ++w) {
      const float mw = sm_ml[(w * 8 + h) * 2];
      const float c = mw == -INFINITY ? 0.0f : exp2f(mw - mm);
      ll += sm_ml[(w * 8 + h) * 2 + 1] * c;
      acc += sm_acc[((size_t)w * 8 + h) * kHd + d] * c;
    }
    const int qh = kvh * group + h;
    if (num_splits == 1) {
      const float gt = __bfloat162float(gate[(size_t)m * ld_gate + (size_t)qh * kHd + d]);
      out[(size_t)m * nq * kHd + (size_t)qh * kHd + d] = __float2bfloat16_rn(acc / ll * sigmoid_f(gt));
    } else {
      float* dst = scratch + (((size_t)row * nq + qh) * max_splits + split) * (kHd + 2);
      dst[d] = acc;
      if (d == 0) {
        dst[kHd] = mm;
        dst[kHd + 1] = ll;
      }
    }
  }
}

// ---------------------------------------------------------------------------------------------------
// Chunked-prefill attention over int8 or bf16 pages on the 5th-generation tensor cores.
// Replaces the reference's attention_prefill kernel (src/kernels/attention_prefill.cu:154-313).
//
// One CTA per (KV split, kv head, tile of `tq` consecutive prompt tokens of one sequence). The tile's rows are its
// (token, query head of the kv head's group) pairs, at most 128 = one row per TMEM lane; keys go by in blocks of 128.
//   warps 0-3    softmax: a thread owns a row. Scores come from TMEM (two passes: maximum, then exponentials), P goes
//                back over the scores as packed fp16, the A operand of the value product. Online softmax in the log2
//                domain; the reference maximum of a row moves only when a score exceeds it by more than kLazy powers
//                of two (P is then at most 2^kLazy, the same relative precision in fp16), so the 128 x 256 fp32 output
//                accumulator in TMEM is rescaled a few times per tile, not per block.
//   warps 4-11   bring the keys and values in, once per tile, into a ring of 16 KB slots in the 128-byte swizzle: int8 from the
//                staged bytes of two pages -> fp16(int8) * fp16(scale of its key and 64-dim group) (the rounding of the
//                reference's prefill kernel), bf16 by 16-byte copies, four slots ahead, -> fp16 in place.
//   warp 13      int8: copies a group's bytes and scales (contiguous in a page) into staging, a group ahead.
//   warp 12      issues the MMAs: S(i) = Q K^T (M 128, N 128 keys, four slots of 64 dims), then O += P(i-1) V(i-1) (N 256
//                dims, four slots of 32 keys, V as it lies in the page: dims contiguous, an MN-major operand), so the
//                softmax of a block runs under the products of its neighbours.
// TMEM: O in columns 0-255, two score buffers of 128 columns behind it. Keys beyond a row's position are masked; positions
// nobody has written yet are loaded as zeros.
// A tile cuts its blocks evenly over at most `num_splits` CTAs: over `wave_splits`, which run at once, in pieces of at least
// kMinBlocksIdle blocks, over more only in pieces of at least kMinBlocksPerSplit; a tile with a single
// live split normalises, applies the sigmoid output gate and writes bf16 itself (and marks its rows as finished for the merge
// by a negative row sum); otherwise the (O, m, l) states go to the scratch for attn_merge_kernel.
//
// Bound by shared memory: per block of 128 keys 448 KB go through it (raw bytes in and out, converted tiles in, operands of
// the MMAs out), 3500 cycles at 128 bytes a cycle, and the raw reads collide in pairs; the tensor pipe asks 2048. It takes about 4800,
// the rest waits along staging, conversion, scores and softmax (512 tokens behind 32 K, with the merge, 702 and 618 us). Whole mixer of
// 512 tokens behind 32 K tokens of int8, 24 / 4 heads: 826 us with 16-byte copies by the converting warps, 764 us now; behind
// 16 K: 487 and 441 us; bf16 behind 16 K, one piece of code for K and V instead of four: 597 and 510 us.
// ---------------------------------------------------------------------------------------------------
constexpr int kPfRows = 128;
constexpr int kPfBlock = 128;                  // keys per block: two pages
constexpr int kPfSoftmaxWarps = 4, kPfLoadWarps = 8;
constexpr int kPfMmaWarp = kPfSoftmaxWarps + kPfLoadWarps;
constexpr int kPfFetchWarp = kPfMmaWarp + 1, kPfThreads = (kPfFetchWarp + 1) * 32;
constexpr int kPfMaxSlots = 10, kPfSlotBytes = 16384;
constexpr int kPfQBytes = kPfRows * kHd * 2;
constexpr int kPfRingOff = kPfQBytes;
constexpr int kPfBarOff = kPfRingOff + kPfMaxSlots * kPfSlotBytes;
constexpr int kPfMlOff = kPfBarOff + 256;      // [128][2] floats
constexpr int kPfSmem = 1024 + kPfMlOff + kPfRows * 8;
constexpr int kPfOStride = kHd + 4;            // floats per staged output row (aliases Q and the ring)
static_assert(kPfRows * kPfOStride * 4 <= kPfBarOff, "output staging");
static_assert(kPfSmem <= 227 * 1024, "shared memory budget");
constexpr int kPfTmemCols = 512, kPfSCol = 256;
constexpr float kLazy = 8.0f;
// Fewest blocks of a split. A split's fixed cost (query staging, TMEM, its share of the merge) is that of about eight blocks, so
// where splits have to wait for SMs they are no shorter than twice that. SMs that would have nothing to do otherwise cost
// nothing: splits of the first wave go down to two blocks (one or three: the same or slower). 512 tokens behind 2048, 3 / 1
// heads (13 tiles of 17 to 20 blocks): 68 us with at least sixteen blocks, 31 us now; 64 tokens behind 4096, 24 / 4: 69 and 38 us.
constexpr int kMinBlocksPerSplit = 16, kMinBlocksIdle = 2;

// D += A B^T with A in tensor memory (packed fp16, eight columns per k16 step) and B in shared memory; converged warp.
__device__ __forceinline__ void umma_f16_ta(uint32_t d_tmem, uint32_t a_tmem, uint64_t b_desc, uint32_t idesc, uint32_t accumulate) {
  asm volatile(
      "{\n\t.reg .pred p, leader;\n\t"
      "elect.sync _|leader, 0xffffffff;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "@leader tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p;\n\t}"
      ::"r"(d_tmem), "r"(a_tmem), "l"(b_desc), "r"(idesc), "r"(accumulate)
      : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
__device__ __forceinline__ float ex2(float x) {
  float y;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}
// two fp32 lanes of one instruction
__device__ __forceinline__ uint64_t pack2(uint32_t a, uint32_t b) {
  uint64_t d;
  asm("mov.b64 %0, {%1, %2};" : "=l"(d) : "r"(a), "r"(b));
  return d;
}
__device__ __forceinline__ void unpack2(uint64_t v, float& a, float& b) { asm("mov.b64 {%0, %1}, %2;" : "=f"(a), "=f"(b) : "l"(v)); }
__device__ __forceinline__ uint64_t fma2(uint64_t a, uint64_t b, uint64_t c) {
  uint64_t d;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(d) : "l"(a), "l"(b), "l"(c));
  return d;
}
__device__ __forceinline__ uint64_t add2(uint64_t a, uint64_t b) {
  uint64_t d;
  asm("add.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
  return d;
}
__device__ __forceinline__ uint32_t half2_bits(__half2 h) { return *reinterpret_cast<uint32_t*>(&h); }

// 16 int8 values -> 16 fp16 values times `scale`: chunks of eight
__device__ __forceinline__ void dequant16_to_half(const uint4& raw, __half scale, uint4& c0, uint4& c1) {
  const __half2 sc = __half2half2(scale);
  const uint32_t w[4] = {raw.x ^ 0x80808080u, raw.y ^ 0x80808080u, raw.z ^ 0x80808080u, raw.w ^ 0x80808080u};
  uint32_t outw[8];
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const uint32_t lo = bytes_to_half2<0x4140>(w[i]), hi = bytes_to_half2<0x4342>(w[i]);
    outw[2 * i] = half2_bits(__hmul2(*reinterpret_cast<const __half2*>(&lo), sc));
    outw[2 * i + 1] = half2_bits(__hmul2(*reinterpret_cast<const __half2*>(&hi), sc));
  }
  c0 = make_uint4(outw[0], outw[1], outw[2], outw[3]);
  c1 = make_uint4(outw[4], outw[5], outw[6], outw[7]);
}

// 8 bf16 values (16 bytes) -> 8 fp16 values (exact for every magnitude an fp16 holds; K and V rows are O(1))
__device__ __forceinline__ uint4 bf16x8_to_half(const uint4& raw) {
  const uint32_t w[4] = {raw.x, raw.y, raw.z, raw.w};
  uint32_t o[4];
#pragma unroll
  for (int i = 0; i < 4; ++i)
    o[i] = half2_bits(__floats2half2_rn(__uint_as_float(w[i] << 16), __uint_as_float(w[i] & 0xffff0000u)));
  return make_uint4(o[0], o[1], o[2], o[3]);
}

template <bool kInt8>
__global__ void __launch_bounds__(kPfThreads, 1) attn_prefill_umma_kernel(
    const __half* __restrict__ q, const __nv_bfloat16* __restrict__ gate, int ld_gate, __nv_bfloat16* __restrict__ out,
    int nq, int group, int layer, int tq, int tiles_per_seq, float* __restrict__ scratch, int max_splits, int num_splits,
    int wave_splits, const int* __restrict__ seq_start, const int* __restrict__ seq_slot, const int* __restrict__ seq_pos0, KvView kv) {
  pdl_wait();               // everything written by earlier kernels of the stream is visible from here on
  pdl_launch_dependents();  // the next kernel may be scheduled now; it holds its own dependent work back the same way
  extern __shared__ uint8_t pf_raw[];
  uint8_t* smem = pf_raw + ((1024 - (smem_u32(pf_raw) & 1023)) & 1023);
  // int8: eight slots and 32 KB of staging for the raw bytes; bf16: ten slots
  constexpr int kSlots = kInt8 ? 8 : 10, kRingOff = kPfRingOff;
  uint8_t* ring = smem + kRingOff;
  uint64_t* full = reinterpret_cast<uint64_t*>(smem + kPfBarOff);
  uint64_t* empty = full + kSlots;
  uint64_t* s_full = empty + kSlots;   // [2]
  uint64_t* p_full = s_full + 2;         // [2]
  uint64_t* pv_done = p_full + 2;        // [2]: consecutive blocks in turn, so that no wait can be two completions behind
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(pv_done + 2);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);
  uint64_t *raw_full = pv_done + 4, *raw_empty = raw_full + 1;  // int8: the staging of a group's bytes
  int* raw_keys = reinterpret_cast<int*>(raw_empty + 1);        // [2] its keys that count, per page
  float* ml = reinterpret_cast<float*>(smem + kPfMlOff);
  static_assert((2 * kSlots + 10) * 8 + 8 <= 256, "barrier area");

  const int split = blockIdx.x, kvh = blockIdx.y;
  const int b = blockIdx.z / tiles_per_seq, ti = blockIdx.z % tiles_per_seq;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int s_first = seq_start[b], n_seq = seq_start[b + 1] - s_first;
  const int i0 = ti * tq;
  if (i0 >= n_seq) return;                       // this sequence's chunk has fewer tiles
  const int nt = min(tq, n_seq - i0);            // tokens of the tile
  const int rows = nt * group;                   // (token, head) rows, <= 128
  const int m0 = s_first + i0;                   // first token row of the tile in the step's arrays
  const int pos0 = seq_pos0[b] + i0;             // its position; row r sees keys 0 .. pos0 + r / group
  const int slot_id = seq_slot[b];
  const int L = pos0 + nt;
  const int blocks = (L + kPfBlock - 1) / kPfBlock;
  const int long_splits = min(num_splits, max(1, blocks / kMinBlocksPerSplit));
  const int per = min(max(kMinBlocksIdle, (blocks + wave_splits - 1) / wave_splits), (blocks + long_splits - 1) / long_splits);
  const bool alone = blocks <= per;
  const int b0 = min(blocks, split * per), nb = min(blocks, (split + 1) * per) - b0;
  if (nb <= 0) {  // (only with several splits) nothing to do here: empty states for the merge
    if (!alone)
      for (int r = tid; r < rows; r += kPfThreads) {
        float* dst = scratch + (((size_t)(m0 + r / group) * nq + (size_t)kvh * group + r % group) * max_splits + split) * (kHd + 2);
        dst[kHd] = -INFINITY;
        dst[kHd + 1] = 0.0f;
      }
    return;
  }
  if (tid == 0) {
    for (int s = 0; s < kSlots; ++s) {
      mbar_init(&full[s], kPfLoadWarps / 4);
      mbar_init(&empty[s], 1);
    }
    for (int s = 0; s < 2; ++s) {
      mbar_init(&s_full[s], 1);
      mbar_init(&p_full[s], kPfSoftmaxWarps);
      mbar_init(&pv_done[s], 1);
    }
    mbar_init(raw_full, 1);
    mbar_init(raw_empty, kPfLoadWarps);
    *abort_flag = 0;
    mbar_fence_init();
  }
  if (warp == kPfMmaWarp) tmem_alloc(tmem_slot, kPfTmemCols);
  // the tile's query rows (fp16) as a K-major operand in the 128-byte swizzle, zero rows beyond the tile
#pragma unroll 5
  for (int i = tid; i < kPfRows * (kHd / 8); i += kPfThreads) {
    const int r = i / (kHd / 8), c = i % (kHd / 8);
    uint4 v = make_uint4(0u, 0u, 0u, 0u);
    if (r < rows)
      v = *reinterpret_cast<const uint4*>(q + ((size_t)(m0 + r / group) * nq + (size_t)kvh * group + r % group) * kHd + 8 * c);
    *reinterpret_cast<uint4*>(smem + (c >> 3) * (kPfRows * 128) + r * 128 + (((c & 7) ^ (r & 7)) << 4)) = v;
  }
  fence_async_smem();
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = *tmem_slot;

  // Slots run in the order K(0) K(1) V(0) K(2) V(1) ... K(nb-1) V(nb-2) V(nb-1), four of each: the order of the MMAs.
  if (warp == kPfMmaWarp) {
    constexpr uint32_t kIdescS = (1u << 4) | (uint32_t(kPfBlock >> 3) << 17) | (uint32_t(128 >> 4) << 24);
    constexpr uint32_t kIdescV = (1u << 4) | (1u << 16) | (uint32_t(kHd >> 3) << 17) | (uint32_t(128 >> 4) << 24);
    const uint64_t qd = smem_desc_sw128(smem_u32(smem));
    const uint32_t ring_u = smem_u32(ring);
    int slot = 0;
    uint32_t par = 0;
    bool alive = true;
    auto next_slot = [&]() {
      if (++slot == kSlots) {
        slot = 0;
        par ^= 1u;
      }
    };
#pragma unroll 1
    for (int i = 0; i <= nb && alive; ++i) {
      if (i < nb) {
        const uint32_t d = tmem + uint32_t(kPfSCol + (i & 1) * kPfBlock);
#pragma unroll 1
        for (int sub = 0; sub < 4 && alive; ++sub) {
          alive = __all_sync(0xffffffffu, wait_flag(&full[slot], par, abort_flag, 0x231));
          if (!alive) break;
          tc_fence_after();
          const uint64_t kd = smem_desc_sw128(ring_u + uint32_t(slot * kPfSlotBytes));
#pragma unroll
          for (int ks = 0; ks < 4; ++ks)
            umma_bf16(d, qd + uint64_t((sub * kPfRows * 128 + ks * 32) >> 4), kd + uint64_t((ks * 32) >> 4), kIdescS,
                      uint32_t(sub | ks));
          umma_commit(&empty[slot]);
          next_slot();
        }
        if (alive) umma_commit(&s_full[i & 1]);
      }
      if (i > 0 && alive) {
        const int j = i - 1;
        alive = __all_sync(0xffffffffu, wait_flag(&p_full[j & 1], uint32_t(j >> 1) & 1u, abort_flag, 0x232));
        if (!alive) break;
        tc_fence_after();
        const uint32_t pa = tmem + uint32_t(kPfSCol + (j & 1) * kPfBlock);
#pragma unroll 1
        for (int sub = 0; sub < 4 && alive; ++sub) {
          alive = __all_sync(0xffffffffu, wait_flag(&full[slot], par, abort_flag, 0x233));
          if (!alive) break;
          tc_fence_after();
          const uint64_t vd = smem_desc_sw128_mn(ring_u + uint32_t(slot * kPfSlotBytes), 4096);
#pragma unroll
          for (int ks = 0; ks < 2; ++ks)
            umma_f16_ta(tmem, pa + uint32_t(sub * 16 + ks * 8), vd + uint64_t((ks * 2048) >> 4), kIdescV,
                        uint32_t(j | sub | ks));
          umma_commit(&empty[slot]);
          next_slot();
        }
        if (alive) umma_commit(&pv_done[j & 1]);
      }
    }
  } else if (warp >= kPfSoftmaxWarps) {
    // ------------------------------ keys and values ------------------------------
    // A slot is [128 keys][64 dims] of K or, of V, four [32 keys][64 dims] side by side. Four teams of two warps; team t makes
    // slot t of every group of four, so that a thread has eight (bf16: sixteen) independent units of 16 bytes in hand: the
    // conversion is bound by latency and instruction count, and with all eight warps on every slot a slot took 800 cycles.
    // int8: a group's bytes and scales are four contiguous runs (two pages, one kv head). The fetch warp copies them into staging
    // in one piece each, as soon as all teams have the last group's in registers. (With cp.async by the teams, 64 bytes of a row
    // at a time, and the scales by plain loads, half of a team's 2,700 cycles a slot went into issuing them.)
    // bf16: units come by cp.async, a group ahead, into the slot itself and are converted in place; only their thread reads them.
    constexpr int kLanesPerRow = kInt8 ? 4 : 8;          // threads that make up the 64 dims of a row
    constexpr int kStep = 64 / kLanesPerRow;             // rows a team covers at once
    constexpr int kUnits = kPfBlock / kStep;             // per thread and slot
    constexpr int kVRows = 32 / kStep;                   // units per 64 dims of a V slot
    constexpr int kRow = kHd * (kInt8 ? 1 : 2), kPart = kRow / 4;  // bytes of a row, of its 64 dims
    constexpr int kNone = INT_MIN;
    uint8_t* const staging = smem + kRingOff + kSlots * kPfSlotBytes;  // int8: [2 pages][64 keys][256]
    const __half* const scales = reinterpret_cast<const __half*>(ml);  // int8: [2 pages][64 keys][4]; the rows' maxima come later
    const int* table = kv.block_table + (size_t)slot_id * kv.max_pages_per_seq;
    const int pages = (L + kPage - 1) / kPage;
    const uint8_t* pool = kv.pool + (size_t)layer * kv.layer_stride;
    auto entry = [&](int p) { return p < pages ? table[p] : kNone; };
    auto page_at = [&](int page) -> const uint8_t* {  // nullptr: beyond the tile's keys, or an invalid entry
      if (page < 0 || page >= kv.num_pages) {
        if (page != kNone) report_error(0x222);
        return nullptr;
      }
      return pool + (size_t)page * kv.page_bytes;
    };
    // groups g = 0 .. 2 nb - 1 in slot order: g == 0: K(0); odd g: K((g + 1) / 2), but the last one is V(nb - 1); even g > 0: V(g / 2 - 1)
    const int groups = 2 * nb;
    auto is_v_group = [&](int g) { return (g > 0 && (g & 1) == 0) || g == groups - 1; };
    // pages of the block of the next V group and of the last K group; table entries of the K group after that
    const uint8_t *k0 = nullptr, *k1 = nullptr, *v0 = nullptr, *v1 = nullptr;
    int k_blk = b0, v_blk = b0, e0 = kNone, e1 = kNone;
    auto first_group = [&]() {
      k0 = v0 = page_at(entry(2 * b0));
      k1 = v1 = page_at(entry(2 * b0 + 1));
      if (nb > 1) {
        e0 = entry(2 * b0 + 2);
        e1 = entry(2 * b0 + 3);
      }
    };
    auto next_group = [&](int g) {  // from group g to the one behind it
      if (is_v_group(g)) {  // the next V group belongs to the block whose K group came last
        v0 = k0;
        v1 = k1;
        v_blk = k_blk;
      }
      if (g + 1 < groups && !is_v_group(g + 1)) {
        ++k_blk;
        k0 = page_at(e0);
        k1 = page_at(e1);
        const bool another = k_blk + 1 < b0 + nb;
        e0 = another ? entry(2 * k_blk + 2) : kNone;
        e1 = another ? entry(2 * k_blk + 3) : kNone;
      }
    };
    bool alive = true;
    if (warp == kPfFetchWarp) {
      if constexpr (kInt8) {
        const uint64_t policy = policy_evict_normal();
        int issued = 0;
        first_group();
#pragma unroll 1
        for (int g = 0; g < groups; ++g) {
          const bool v = is_v_group(g);
          const int blk = v ? v_blk : k_blk;
          if (alive && g > 0) alive = wait_flag(raw_empty, uint32_t(g - 1) & 1u, abort_flag, 0x239);
          alive = __all_sync(0xffffffffu, alive);
          if (!alive) break;
          if (lane == 0) {
            const uint8_t* pg[2] = {v ? v0 : k0, v ? v1 : k1};
            int keys[2];
#pragma unroll
            for (int e = 0; e < 2; ++e) raw_keys[e] = keys[e] = pg[e] ? max(0, min(kPage, L - (2 * blk + e) * kPage)) : 0;
            mbar_expect_tx(raw_full, uint32_t((keys[0] > 0) + (keys[1] > 0)) * uint32_t(kPage * (kRow + 8)));
#pragma unroll
            for (int e = 0; e < 2; ++e) {
              if (keys[e] == 0) continue;
              bulk_g2s(staging + e * kPage * kRow, pg[e] + (v ? kv.v_off(kvh, 0) : kv.k_off(kvh, 0)), kPage * kRow, raw_full, policy);
              bulk_g2s(reinterpret_cast<uint8_t*>(ml) + e * kPage * 8, pg[e] + (v ? kv.vs_off(kvh, 0) : kv.ks_off(kvh, 0)), kPage * 8, raw_full, policy);
            }
          }
          __syncwarp();
          ++issued;
          next_group(g);
        }
        if (!alive && issued > 0) mbar_wait(raw_full, uint32_t(issued - 1) & 1u, 0x23b);  // given up: its copies may be in flight
      }
    } else {
      const int lt = tid - kPfSoftmaxWarps * 32;
      const int team = lt / 64, lrow = lt % 64 / kLanesPerRow, lch = lt % kLanesPerRow;
      // The thread's place in a slot: row and first chunk, swizzled (its rows are multiples of eight apart). The eight threads
      // of a store phase write even and odd rows' chunks (int8) or one row (bf16): distinct banks.
      const uint32_t x0 = uint32_t(lrow * 128) + uint32_t(((kInt8 ? 2 * lch : lch) ^ (lrow & 7)) << 4);
      [[maybe_unused]] const int second = (x0 & 16u) ? -16 : 16;  // from a unit's first chunk to its second
      // unit r of either kind goes r * kStep * 128 bytes behind the thread's place (a V part of 64 dims has kVRows * kStep = 32 rows)
      constexpr int kPlace = kStep * 128;
      static_assert(kVRows * kPlace == 4096);
      const int v_row = 32 * (team & 1) + lrow;  // the thread's first row of V in its page
      int slot = team;
      uint32_t par = 1;
      auto advance = [&](int& s, uint32_t& p) {
        s += 4;
        if (s >= kSlots) {
          s -= kSlots;
          p ^= 1u;
        }
      };
      if constexpr (kInt8) {
        const uint8_t* const k_at = staging + lrow * kRow + team * kPart + 16 * lch;
        const uint8_t* const v_at = staging + (team >= 2 ? kPage * kRow : 0) + v_row * kRow + 16 * lch;
        const __half* const ks_at = scales + 4 * lrow + team;
        const __half* const vs_at = scales + (team >= 2 ? kPage * 4 : 0) + 4 * v_row;
#pragma unroll 1
        for (int g = 0; g < groups; ++g) {
          const bool v = is_v_group(g);
          if (alive) alive = wait_flag(raw_full, uint32_t(g) & 1u, abort_flag, 0x23a);
          uint4 raw[kUnits];
          __half scale[kUnits];
          const uint8_t* src = v ? v_at : k_at;
          const __half* ssrc = v ? vs_at : ks_at;
#pragma unroll
          for (int r = 0; r < kUnits; ++r) {
            raw[r] = *reinterpret_cast<const uint4*>(src + (v ? (r % kVRows) * (kStep * kRow) + (r / kVRows) * kPart : r * (kStep * kRow)));
            scale[r] = ssrc[v ? (r % kVRows) * (kStep * 4) + r / kVRows : r * (kStep * 4)];
          }
          const int n0 = raw_keys[0], n1 = raw_keys[1];
          if (n0 + n1 < kPfBlock) {  // what nobody has written yet stays out: zeros
#pragma unroll
            for (int r = 0; r < kUnits; ++r) {
              const int key = v ? v_row + r % kVRows * kStep : r * kStep % kPage + lrow, n = (v ? team >= 2 : r * kStep >= kPage) ? n1 : n0;
              if (key >= n) {
                raw[r] = make_uint4(0u, 0u, 0u, 0u);
                scale[r] = __ushort_as_half(0);
              }
            }
          }
          __syncwarp();
          if (lane == 0) mbar_arrive(raw_empty);
          if (alive) alive = wait_flag(&empty[slot], par, abort_flag, 0x234);
          if (alive) {
            uint8_t* dst = ring + slot * kPfSlotBytes + x0;
#pragma unroll
            for (int r = 0; r < kUnits; ++r) {
              uint4 c0, c1;
              dequant16_to_half(raw[r], scale[r], c0, c1);
              uint8_t* d = dst + r * kPlace;
              *reinterpret_cast<uint4*>(d) = c0;
              *reinterpret_cast<uint4*>(d + second) = c1;
            }
          }
          fence_async_smem();
          __syncwarp();
          if (lane == 0) mbar_arrive(&full[slot]);
          advance(slot, par);
        }
      } else {
        const size_t k_off = kv.k_off(kvh, 0) + (size_t)lrow * kRow + team * kPart + 16 * lch;
        const size_t v_off = kv.v_off(kvh, 0) + (size_t)v_row * kRow + 16 * lch;
        // Requests the team's slot of block `blk` with pages pg0 and pg1 to dst. One piece of code for K and V: the units' offsets
        // are selected, not branched on (four copies of it, K and V behind K and V, made 137 KB of code, and a fifth of the
        // warps' time went into waiting for instructions).
        auto fetch = [&](bool v, int blk, const uint8_t* pg0, const uint8_t* pg1, uint8_t* dst) {
          const bool whole = (blk + 1) * kPfBlock <= L && pg0 != nullptr && pg1 != nullptr;
          const uint8_t *a = v && team >= 2 ? pg1 : pg0, *b = v && team < 2 ? pg0 : pg1;  // pages of the first and second half of the units
          const size_t off = v ? v_off : k_off;
          const int key0 = blk * kPfBlock + (v ? 32 * team : 0) + lrow;
#pragma unroll
          for (int r = 0; r < kUnits; ++r) {
            const uint8_t* pg = r < kUnits / 2 ? a : b;
            const bool real = whole || (pg != nullptr && key0 + (v ? r % kVRows : r) * kStep < L);  // what nobody has written yet stays out: zeros
            const uint8_t* src = real ? pg + off + (v ? (r % kVRows) * (kStep * kRow) + (r / kVRows) * kPart : (r * kStep % kPage) * kRow) : pool;
            asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(smem_u32(dst + r * kPlace)), "l"(src), "r"(real ? 16 : 0)
                         : "memory");
          }
        };
        first_group();
        fetch(false, b0, k0, k1, ring + slot * kPfSlotBytes + x0);  // every slot's first use is free
        cp_async_commit();
#pragma unroll 1
        for (int g = 0; g < groups; ++g) {
          const bool more = g + 1 < groups, nv = more && is_v_group(g + 1);
          next_group(g);
          uint8_t* dst = ring + slot * kPfSlotBytes + x0;
          int next = slot;
          uint32_t next_par = par;
          advance(next, next_par);
          if (more) {
            if (alive) alive = wait_flag(&empty[next], next_par, abort_flag, 0x234);
            if (alive) fetch(nv, nv ? v_blk : k_blk, nv ? v0 : k0, nv ? v1 : k1, ring + next * kPfSlotBytes + x0);
          }
          cp_async_commit();
          asm volatile("cp.async.wait_group 1;" ::: "memory");
#pragma unroll
          for (int r = 0; r < kUnits; ++r) {
            uint4* d = reinterpret_cast<uint4*>(dst + r * kPlace);
            *d = bf16x8_to_half(*d);
          }
          fence_async_smem();
          __syncwarp();
          if (lane == 0) mbar_arrive(&full[slot]);
          slot = next;
          par = next_par;
        }
        asm volatile("cp.async.wait_group 0;" ::: "memory");
      }
    }
  } else {
    // ------------------------------ softmax: thread = row ------------------------------
    const int r = tid;
    const int pos = r < rows ? pos0 + r / group : -1;  // last key position the row may see (-1: padding row)
    const int warp_first = pos0 + (32 * warp) / group;  // smallest position among the warp's rows
    const uint32_t lanes = uint32_t(32 * warp) << 16;
    float mref = -INFINITY, l = 0.0f;
    constexpr float kScale = kLog2e / 16.0f;
    bool alive = true;
#pragma unroll 1
    for (int i = 0; i < nb; ++i) {
      if (alive && i >= 2) alive = wait_flag(&pv_done[i & 1], uint32_t((i - 2) >> 1) & 1u, abort_flag, 0x235);  // it precedes S(i)
      if (alive) alive = wait_flag(&s_full[i & 1], uint32_t(i >> 1) & 1u, abort_flag, 0x236);
      alive = __all_sync(0xffffffffu, alive);
      if (!alive) break;
      tc_fence_after();
      const uint32_t st = tmem + lanes + uint32_t(kPfSCol + (i & 1) * kPfBlock);
      const int kbase = (b0 + i) * kPfBlock;
      const bool need_mask = kbase + kPfBlock - 1 > warp_first;
      const int seen = pos - kbase;  // keys 0 .. seen of the block
      // 64 scores at a time: half as many round trips to tensor memory as with 32
      float mx0 = -INFINITY, mx1 = -INFINITY;
#pragma unroll 1
      for (int c = 0; c < 4; c += 2) {
        uint32_t s[2][32];
        tmem_ld32(st + uint32_t(32 * c), s[0]);
        tmem_ld32(st + uint32_t(32 * c + 32), s[1]);
        tmem_wait_ld(s[0], s[1]);
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          if (need_mask) {
#pragma unroll
            for (int e = 0; e < 32; ++e)
              if (32 * (c + h) + e > seen) s[h][e] = 0xff800000u;
          }
#pragma unroll
          for (int e = 0; e < 32; e += 4) {
            mx0 = fmaxf(fmaxf(mx0, __uint_as_float(s[h][e])), __uint_as_float(s[h][e + 1]));
            mx1 = fmaxf(fmaxf(mx1, __uint_as_float(s[h][e + 2])), __uint_as_float(s[h][e + 3]));
          }
        }
      }
      const float mb = fmaxf(mx0, mx1) * kScale;
      float corr = 1.0f;
      if (mb > mref + kLazy) {  // (the row's first keys: mref is -inf, the factor 0)
        corr = ex2(mref - mb);
        mref = mb;
      }
      l *= corr;
      if (i > 0 && __any_sync(0xffffffffu, corr != 1.0f)) {  // rescale the accumulator once PV(i - 1) is in it
        alive = __all_sync(0xffffffffu, wait_flag(&pv_done[(i - 1) & 1], uint32_t((i - 1) >> 1) & 1u, abort_flag, 0x237));
        if (!alive) break;
        tc_fence_after();
#pragma unroll 1
        for (int c = 0; c < kHd; c += 32) {
          uint32_t o[32];
          tmem_ld32(tmem + lanes + uint32_t(c), o);
          tmem_wait_ld(o);
#pragma unroll
          for (int e = 0; e < 32; ++e) o[e] = __float_as_uint(__uint_as_float(o[e]) * corr);
          tmem_st32(tmem + lanes + uint32_t(c), o);
        }
      }
      const float ref = mref == -INFINITY ? 0.0f : mref;  // no inf - inf
      const uint64_t scale2 = pack2(__float_as_uint(kScale), __float_as_uint(kScale));
      const uint64_t ref2 = pack2(__float_as_uint(-ref), __float_as_uint(-ref));
      uint64_t sum2 = 0;
#pragma unroll 1
      for (int c = 0; c < 4; c += 2) {
        uint32_t s[2][32];
        tmem_ld32(st + uint32_t(32 * c), s[0]);
        tmem_ld32(st + uint32_t(32 * c + 32), s[1]);
        tmem_wait_ld(s[0], s[1]);
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          uint32_t p[16];
          if (need_mask) {
#pragma unroll
            for (int e = 0; e < 32; ++e)
              if (32 * (c + h) + e > seen) s[h][e] = 0xff800000u;
          }
#pragma unroll
          for (int e = 0; e < 16; ++e) {
            float e0, e1;
            unpack2(fma2(pack2(s[h][2 * e], s[h][2 * e + 1]), scale2, ref2), e0, e1);
            e0 = ex2(e0);
            e1 = ex2(e1);
            sum2 = add2(sum2, pack2(__float_as_uint(e0), __float_as_uint(e1)));
            p[e] = half2_bits(__floats2half2_rn(e0, e1));
          }
          tmem_st16(st + uint32_t(16 * (c + h)), p);  // over score columns that have been read
        }
      }
      float ls0, ls1;
      unpack2(sum2, ls0, ls1);
      l += ls0 + ls1;
      tmem_wait_st();
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(&p_full[i & 1]);
    }
    // ---- finish: the accumulator through shared memory (queries and ring are drained) for coalesced gates and stores ----
    if (alive) alive = wait_flag(&pv_done[(nb - 1) & 1], uint32_t((nb - 1) >> 1) & 1u, abort_flag, 0x238);
    alive = __all_sync(0xffffffffu, alive);
    if (alive) {
      tc_fence_after();
      float* os = reinterpret_cast<float*>(smem) + (size_t)r * kPfOStride;
      const float inv = alone && l > 0.0f ? 1.0f / l : 1.0f;
#pragma unroll 1
      for (int c = 0; c < kHd; c += 32) {
        uint32_t o[32];
        tmem_ld32(tmem + lanes + uint32_t(c), o);
        tmem_wait_ld(o);
#pragma unroll
        for (int e = 0; e < 32; e += 4)
          *reinterpret_cast<float4*>(os + c + e) =
              make_float4(__uint_as_float(o[e]) * inv, __uint_as_float(o[e + 1]) * inv, __uint_as_float(o[e + 2]) * inv,
                          __uint_as_float(o[e + 3]) * inv);
      }
      ml[2 * r] = mref;
      ml[2 * r + 1] = l;
      tc_fence_before();
    }
  }
  __syncthreads();
  if (warp == kPfMmaWarp) {
    tc_fence_after();
    tmem_dealloc(tmem, kPfTmemCols);
  }
  if (*abort_flag) return;
  // A row per warp and turn. States leave eight bytes a lane, whole sectors (a lane's 32 bytes at a time wrote every sector four
  // times: some 80 cycles a row); finished rows take their gates four rows ahead of their use.
  constexpr int kRowStep = kPfThreads / 32, kRowsAhead = 4;
  auto row_of = [&](int r) { return reinterpret_cast<const float*>(smem) + (size_t)r * kPfOStride; };
  if (!alone) {
    for (int r = warp; r < rows; r += kRowStep) {
      const float* os = row_of(r) + 2 * lane;
      float* dst = scratch + (((size_t)(m0 + r / group) * nq + (size_t)kvh * group + r % group) * max_splits + split) * (kHd + 2);
#pragma unroll
      for (int i = 0; i < 4; ++i)
        *reinterpret_cast<float2*>(dst + 2 * lane + 64 * i) = *reinterpret_cast<const float2*>(os + 64 * i);
      if (lane < 2) dst[kHd + lane] = ml[2 * r + lane];
    }
    return;
  }
  for (int r0 = warp; r0 < rows; r0 += kRowStep * kRowsAhead) {
    uint2 graw[kRowsAhead][2];  // dims 4 lane and 128 + 4 lane
#pragma unroll
    for (int u = 0; u < kRowsAhead; ++u) {
      const int r = min(r0 + u * kRowStep, rows - 1);
      const __nv_bfloat16* gp = gate + (size_t)(m0 + r / group) * ld_gate + (size_t)(kvh * group + r % group) * kHd + 4 * lane;
      graw[u][0] = *reinterpret_cast<const uint2*>(gp);
      graw[u][1] = *reinterpret_cast<const uint2*>(gp + 128);
    }
#pragma unroll
    for (int u = 0; u < kRowsAhead; ++u) {
      const int r = r0 + u * kRowStep;
      if (r >= rows) break;
      const size_t at = (size_t)(m0 + r / group) * nq + (size_t)kvh * group + r % group;
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        const float4 x = *reinterpret_cast<const float4*>(row_of(r) + 128 * h + 4 * lane);
        const float2 g0 = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&graw[u][h].x));
        const float2 g1 = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&graw[u][h].y));
        __nv_bfloat162 res[2];
        res[0] = __floats2bfloat162_rn(x.x * sigmoid_f(g0.x), x.y * sigmoid_f(g0.y));
        res[1] = __floats2bfloat162_rn(x.z * sigmoid_f(g1.x), x.w * sigmoid_f(g1.y));
        *reinterpret_cast<uint2*>(out + at * kHd + 128 * h + 4 * lane) = *reinterpret_cast<uint2*>(res);
      }
      if (num_splits > 1 && lane == 0) scratch[(at * max_splits + split) * (kHd + 2) + kHd + 1] = -1.0f;  // finished: nothing left for the merge
    }
  }
}

// Merge of the splits + normalisation + sigmoid gate -> bf16 (reference attention_decode.cu:241-257). PARTS warps per (row, query
// head), a lane owns 8 / PARTS dims; a prefill row that its only live split has finished (negative row sum) is left alone.
// Bound by round trips to L2: 4 * PARTS accumulator rows are on their way at a time, added in the order of the splits. Few rows,
// and so up to 64 splits of each, take eight warps (bf16 cache, one sequence of 24 heads at 2048 tokens: attention and merge 36 us
// with a warp per head and a split at a time, 20 us now).
constexpr int kMergeWarps = 8;
template <int PARTS>
__global__ void __launch_bounds__(kMergeWarps * 32) attn_merge_kernel(const float* __restrict__ scratch, int max_splits,
                                                                      int num_splits, const __nv_bfloat16* __restrict__ gate,
                                                                      int ld_gate, __nv_bfloat16* __restrict__ out, int nq,
                                                                      int items, const int* __restrict__ seq_start) {
  pdl_wait();               // everything written by earlier kernels of the stream is visible from here on
  pdl_launch_dependents();  // the next kernel may be scheduled now; it holds its own dependent work back the same way
  constexpr int kDims = 8 / PARTS, kAtOnce = 4 * PARTS;
  const int unit = blockIdx.x * kMergeWarps + (threadIdx.x >> 5), lane = threadIdx.x & 31;
  const int item = unit / PARTS, d0 = unit % PARTS * (32 * kDims) + lane;
  if (item >= items) return;
  const int row = item / nq, qh = item - row * nq;
  const int m = seq_start ? seq_start[row] : row;  // decode: a sequence's token row; prefill tiles: the token row itself
  const float* base = scratch + (size_t)item * max_splits * (kHd + 2);
  // the splits' (m, l) a lane each; an empty split's accumulator row was never written
  const float first_sum = base[kHd + 1];
  float mm = -INFINITY;
  for (int s = lane; s < num_splits; s += 32) mm = fmaxf(mm, base[(size_t)s * (kHd + 2) + kHd]);
  if (first_sum < 0.0f) return;
  mm = warp_max(mm);
  float ll = 0.0f, a[kDims], g[kDims];
#pragma unroll
  for (int i = 0; i < kDims; ++i) {
    a[i] = 0.0f;
    g[i] = __bfloat162float(gate[(size_t)m * ld_gate + (size_t)qh * kHd + d0 + 32 * i]);
  }
  for (int s0 = 0; s0 < num_splits; s0 += 32) {
    const int s = s0 + lane;
    const float ms = s < num_splits ? base[(size_t)s * (kHd + 2) + kHd] : -INFINITY;
    const float c = ms == -INFINITY ? 0.0f : exp2f(ms - mm);
    if (ms != -INFINITY) ll += base[(size_t)s * (kHd + 2) + kHd + 1] * c;
    for (unsigned live = __ballot_sync(0xffffffffu, ms != -INFINITY); live;) {
      float p[kAtOnce][kDims], cj[kAtOnce];
#pragma unroll
      for (int u = 0; u < kAtOnce; ++u) {
        const int j = live ? __ffs(live) - 1 : -1;  // -1: no further split, nothing added
        live &= live - 1;
        cj[u] = __shfl_sync(0xffffffffu, c, j & 31);
        if (j < 0) cj[u] = 0.0f;
#pragma unroll
        for (int i = 0; i < kDims; ++i) p[u][i] = j >= 0 ? base[(size_t)(s0 + j) * (kHd + 2) + d0 + 32 * i] : 0.0f;
      }
#pragma unroll
      for (int u = 0; u < kAtOnce; ++u)
#pragma unroll
        for (int i = 0; i < kDims; ++i) a[i] += p[u][i] * cj[u];
    }
  }
  ll = warp_sum(ll);
  __nv_bfloat16* o = out + ((size_t)m * nq + qh) * kHd + d0;
#pragma unroll
  for (int i = 0; i < kDims; ++i) o[32 * i] = __float2bfloat16_rn(a[i] / ll * sigmoid_f(g[i]));
}

// Warps per (row, query head): at most four rounds of loads, and eight where there are few of them.
void launch_merge(int rows, cudaStream_t s, const float* scratch, int max_splits, int splits, const __nv_bfloat16* gate,
                  int ld_gate, __nv_bfloat16* out, int nq, const int* seq_start) {
  const int items = rows * nq;
  const int parts = items <= 2 * num_sms() ? 8 : splits <= 16 ? 1 : splits <= 32 ? 2 : 4;
  const int per_cta = kMergeWarps / parts;
  (void)launch_kernel(parts == 8 ? attn_merge_kernel<8> : parts == 4 ? attn_merge_kernel<4> : parts == 2 ? attn_merge_kernel<2> : attn_merge_kernel<1>,
                      dim3((items + per_cta - 1) / per_cta), dim3(kMergeWarps * 32), 0, s, scratch,
                      max_splits, splits, gate, ld_gate, out, nq, items, seq_start);
}

template <int GROUP>
int launch_token_attention(const q38_attention_params& p, const q38_batch_desc& b, const q38_kv_cache_desc& kvd,
                           bool decode, int splits, cudaStream_t s) {
  const KvView kv = make_view(kvd);
  const int rows = decode ? b.num_seqs : b.num_tokens;
  const dim3 grid(splits, p.num_kv_heads, rows);
  const __half* q = reinterpret_cast<const __half*>(p.q);
  const __nv_bfloat16* gate = reinterpret_cast<const __nv_bfloat16*>(p.gate);
  __nv_bfloat16* out = reinterpret_cast<__nv_bfloat16*>(p.out);
  if (kv.int8)
    (void)launch_kernel(attn_token_kernel<GROUP, true>, dim3(grid), dim3(kAttnWarps * 32), 0, s, 
        q, gate, p.ld_gate, out, p.num_q_heads, p.attn_layer, p.split_scratch, p.max_splits, splits, decode ? 1 : 0,
        b.seq_start, b.seq_slot, b.seq_pos0, b.tok_pos, b.tok_seq, kv);
  else
    (void)launch_kernel(attn_token_kernel<GROUP, false>, dim3(grid), dim3(kAttnWarps * 32), 0, s, 
        q, gate, p.ld_gate, out, p.num_q_heads, p.attn_layer, p.split_scratch, p.max_splits, splits, decode ? 1 : 0,
        b.seq_start, b.seq_slot, b.seq_pos0, b.tok_pos, b.tok_seq, kv);
  Q38_LAUNCH_OK("attn_token_kernel");
  if (splits > 1) {
    launch_merge(rows, s, p.split_scratch, p.max_splits, splits, gate, p.ld_gate, out, p.num_q_heads, b.seq_start);
    Q38_LAUNCH_OK("attn_merge_kernel");
  }
  return Q38_OK;
}

int dispatch_group(int group, const q38_attention_params& p, const q38_batch_desc& b, const q38_kv_cache_desc& kv,
                   bool decode, int splits, cudaStream_t s) {
  switch (group) {
    case 1: return launch_token_attention<1>(p, b, kv, decode, splits, s);
    case 2: return launch_token_attention<2>(p, b, kv, decode, splits, s);
    case 3: return launch_token_attention<3>(p, b, kv, decode, splits, s);
    case 4: return launch_token_attention<4>(p, b, kv, decode, splits, s);
    case 5: return launch_token_attention<5>(p, b, kv, decode, splits, s);
    case 6: return launch_token_attention<6>(p, b, kv, decode, splits, s);
    case 7: return launch_token_attention<7>(p, b, kv, decode, splits, s);
    case 8: return launch_token_attention<8>(p, b, kv, decode, splits, s);
    default: set_error("attention: GQA group %d is not implemented (1..8)", group); return Q38_ERR_INVALID;
  }
}

int check_attention(const q38_attention_params* p, const q38_batch_desc* b, const q38_kv_cache_desc* kv) {
  Q38_REQUIRE(p && b && kv, "attention: null argument");
  Q38_REQUIRE(p->q && p->gate && p->out, "attention: null pointer");
  Q38_REQUIRE(p->num_kv_heads > 0 && p->num_q_heads % p->num_kv_heads == 0, "attention: heads %d / %d",
              p->num_q_heads, p->num_kv_heads);
  Q38_REQUIRE(kv->kv_heads == p->num_kv_heads, "attention: kv head count mismatch");
  Q38_REQUIRE(kv->pool && kv->block_table && kv->max_pages_per_seq > 0, "attention: kv cache descriptor");
  return Q38_OK;
}

}  // namespace

Q38_REGISTER_ERROR_WORD();

}  // namespace q38

using namespace q38;

extern "C" int q38_qk_norm_rope_append(const q38_qk_norm_rope_params* p, const q38_batch_desc* batch,
                                       const q38_kv_cache_desc* kv, void* stream) {
  Q38_REQUIRE(p && batch && kv, "qk_norm_rope_append: null argument");
  if (batch->num_tokens == 0) return Q38_OK;
  const int warps = p->num_q_heads + 2 * p->num_kv_heads;
  Q38_REQUIRE(warps > 0 && warps <= 32, "qk_norm_rope_append: %d heads per token exceed one CTA", warps);
  Q38_REQUIRE(kv->kv_heads == p->num_kv_heads, "qk_norm_rope_append: kv head count mismatch");
  Q38_REQUIRE(p->ld_proj % 8 == 0, "qk_norm_rope_append: ld_proj must be a multiple of 8");
  RopeTable rope;
  for (int i = 0; i < 32; ++i) rope.inv_freq[i] = 1.0f / std::pow(float(p->rope_theta), float(2 * i) / 64.0f);
  (void)launch_kernel(qk_norm_rope_kernel, dim3(batch->num_tokens), dim3(warps * 32), 0, as_stream(stream), 
      reinterpret_cast<const __nv_bfloat16*>(p->proj), p->ld_proj, p->q_norm, p->k_norm, p->eps, p->num_q_heads,
      p->num_kv_heads, reinterpret_cast<__half*>(p->q_out), p->attn_layer, rope, batch->tok_pos, batch->tok_seq,
      batch->seq_slot, make_view(*kv));
  Q38_LAUNCH_OK("qk_norm_rope_kernel");
  return Q38_OK;
}

// Split count of the decode launcher. Context lengths of a ragged batch differ by orders of magnitude and the count is
// fixed per captured graph, so it is chosen for balance, not for occupancy: about sixteen work items per SM, so
// that the longest sequence's share per CTA is small against the whole step; splits beyond a short sequence's
// pages cost one early-exiting CTA each.
extern "C" int q38_attention_decode_splits(int batch_seqs, int kv_heads, int num_sms, int max_splits) {
  const int ctas = batch_seqs * kv_heads;
  if (ctas <= 0) return 1;
  int s = (16 * num_sms + ctas - 1) / ctas;
  if (s < 1) s = 1;
  if (s > max_splits) s = max_splits;
  if (s > 256) s = 256;
  return s;
}

extern "C" int q38_attention_decode(const q38_attention_params* p, const q38_batch_desc* batch,
                                    const q38_kv_cache_desc* kv, void* stream) {
  const int rc = check_attention(p, batch, kv);
  if (rc != Q38_OK) return rc;
  if (batch->num_seqs == 0) return Q38_OK;
  Q38_REQUIRE(batch->num_tokens == batch->num_seqs, "attention_decode: one token per sequence expected");
  int splits = q38_attention_decode_splits(batch->num_seqs, p->num_kv_heads, num_sms(), p->max_splits);
  if (!p->split_scratch) splits = 1;
  const int group = p->num_q_heads / p->num_kv_heads;
  if (kv->dtype != Q38_KV_INT8) return dispatch_group(group, *p, *batch, *kv, true, splits, as_stream(stream));
  Q38_REQUIRE(group >= 1 && group <= 8, "attention: GQA group %d is not implemented (1..8)", group);
  static const cudaError_t attr =
      cudaFuncSetAttribute(attn_decode_mma_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kMmaSmem);
  Q38_CUDA_OK(attr);
  const cudaStream_t s = as_stream(stream);
  const __nv_bfloat16* gate = reinterpret_cast<const __nv_bfloat16*>(p->gate);
  __nv_bfloat16* out = reinterpret_cast<__nv_bfloat16*>(p->out);
  (void)launch_kernel(attn_decode_mma_kernel, dim3(splits, p->num_kv_heads, batch->num_seqs), dim3(kMmaThreads), kMmaSmem, s, 
      reinterpret_cast<const __half*>(p->q), gate, p->ld_gate, out, p->num_q_heads, group, p->attn_layer,
      p->split_scratch, p->max_splits, splits, 1, batch->seq_start, batch->seq_slot, batch->seq_pos0, batch->tok_pos,
      batch->tok_seq, make_view(*kv));
  Q38_LAUNCH_OK("attn_decode_mma_kernel");
  if (splits > 1) {
    launch_merge(batch->num_seqs, s, p->split_scratch, p->max_splits, splits, gate, p->ld_gate, out, p->num_q_heads,
                 batch->seq_start);
    Q38_LAUNCH_OK("attn_merge_kernel");
  }
  return Q38_OK;
}

extern "C" int q38_attention_prefill(const q38_attention_params* p, const q38_batch_desc* batch,
                                     const q38_kv_cache_desc* kv, void* stream) {
  const int rc = check_attention(p, batch, kv);
  if (rc != Q38_OK) return rc;
  if (batch->num_tokens == 0) return Q38_OK;
  const int group = p->num_q_heads / p->num_kv_heads;
  const bool int8 = kv->dtype == Q38_KV_INT8;
  if (batch->max_tokens_per_seq > 1 && group >= 1 && group <= kPfRows) {
    // chunks of more than one token: the query-tiled kernel. With few tiles for the GPU (one long request, or a
    // tensor-parallel rank with one kv head) the keys are cut over several CTAs per tile when the caller's scratch
    // (laid out [token][q head][max_splits][258]) allows it.
    static const cudaError_t attr_pf =
        cudaFuncSetAttribute(attn_prefill_umma_kernel<true>, cudaFuncAttributeMaxDynamicSharedMemorySize, kPfSmem);
    static const cudaError_t attr_pf16 =
        cudaFuncSetAttribute(attn_prefill_umma_kernel<false>, cudaFuncAttributeMaxDynamicSharedMemorySize, kPfSmem);
    Q38_CUDA_OK(attr_pf);
    Q38_CUDA_OK(attr_pf16);
    const int tq = kPfRows / group;
    const int tiles_per_seq = (batch->max_tokens_per_seq + tq - 1) / tq;
    const int tiles = (batch->num_tokens + tq - 1) / tq + batch->num_seqs;  // upper bound of the live tiles
    int splits = 1, wave_splits = 1;
    if (p->split_scratch && p->max_splits > 1 && p->scratch_rows >= batch->num_tokens) {
      // The cut that gives every CTA the fewest keys per wave of CTAs: s / ceil(tiles * kv heads * s / SMs) is largest
      // (thirteen tiles of one kv head: eleven cuts fill one wave of 143 CTAs, sixteen would need two waves of longer
      // tails). One sequence: the tile count is exact; otherwise it is the upper bound above. Up to three waves (a
      // hundred tiles: four cuts run in 3 / 4 of the time of one). The kernel itself uses fewer cuts for short contexts.
      const int live = (batch->num_seqs == 1 ? tiles_per_seq : tiles) * p->num_kv_heads;
      const int sms = num_sms(), cap = std::min(p->max_splits, 16);
      double best = 0.0;
      for (int c = 1; c <= cap; ++c) {
        const int waves = (live * c + sms - 1) / sms;
        if (waves > 3) break;
        if (waves == 1) wave_splits = c;
        const double gain = double(c) / waves;
        if (gain > best * (waves == 1 ? 1.0 : 1.1)) {  // a further wave must pay for its share of the merge
          best = gain;
          splits = c;
        }
      }
    }
    const cudaStream_t s = as_stream(stream);
    const __nv_bfloat16* gate = reinterpret_cast<const __nv_bfloat16*>(p->gate);
    __nv_bfloat16* out = reinterpret_cast<__nv_bfloat16*>(p->out);
    (void)launch_kernel(int8 ? attn_prefill_umma_kernel<true> : attn_prefill_umma_kernel<false>,
                        dim3(splits, p->num_kv_heads, batch->num_seqs * tiles_per_seq), dim3(kPfThreads), kPfSmem, s,
                        reinterpret_cast<const __half*>(p->q), gate, p->ld_gate, out, p->num_q_heads, group, p->attn_layer,
                        tq, tiles_per_seq, p->split_scratch, p->max_splits, splits, wave_splits, batch->seq_start, batch->seq_slot,
                        batch->seq_pos0, make_view(*kv));
    Q38_LAUNCH_OK("attn_prefill_umma_kernel");
    if (splits > 1) {
      launch_merge(batch->num_tokens, s, p->split_scratch, p->max_splits, splits, gate, p->ld_gate, out, p->num_q_heads, nullptr);
      Q38_LAUNCH_OK("attn_merge_kernel");
    }
    return Q38_OK;
  }
  if (!int8) return dispatch_group(group, *p, *batch, *kv, false, 1, as_stream(stream));
  // single-token chunks: the decode kernel, one CTA per (kv head, token)
  Q38_REQUIRE(group >= 1 && group <= 8, "attention: GQA group %d is not implemented (1..8)", group);
  static const cudaError_t attr =
      cudaFuncSetAttribute(attn_decode_mma_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kMmaSmem);
  Q38_CUDA_OK(attr);
  (void)launch_kernel(attn_decode_mma_kernel, dim3(1, p->num_kv_heads, batch->num_tokens), dim3(kMmaThreads), kMmaSmem, as_stream(stream), 
      reinterpret_cast<const __half*>(p->q), reinterpret_cast<const __nv_bfloat16*>(p->gate), p->ld_gate,
      reinterpret_cast<__nv_bfloat16*>(p->out), p->num_q_heads, group, p->attn_layer, p->split_scratch, p->max_splits, 1,
      0, batch->seq_start, batch->seq_slot, batch->seq_pos0, batch->tok_pos, batch->tok_seq, make_view(*kv));
  Q38_LAUNCH_OK("attn_decode_mma_kernel");
  return Q38_OK;
}
