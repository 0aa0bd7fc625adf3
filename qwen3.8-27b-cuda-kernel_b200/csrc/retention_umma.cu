// Retention of prefill runs with heads of 128 x 128 on the 5th-generation tensor cores (see retention.cu for the operator). The
// run is cut into chunks of 128 tokens, and everything but the sum of the states is parallel over (chunk, head):
//   angles   cos and sin of every (token, dimension pair), once for all heads
//   chunk    D_c = sum_j decay^(n-1-j) k_j v_j^T       128 dk x 128 v per (chunk, head)
//   sum      S_c = state ahead of chunk c, c = 0, 1, ...: S' = decay^n S + D_c; elementwise, fp32
//   output   o_i = decay^(i+1) S_c^T q_i + sum_(j <= i) decay^(i-j) (q_i . k_j) v_j, its norm and output gate
// Every fp32 factor goes into an MMA as two bf16 terms hi + lo (16 mantissa bits; v is bf16 as it stands): three products where
// both factors have two, two where one does; sums are fp32, smallest terms first.
// Scratch: D_c of a whole chunk lies in `o` where the chunk's rows are, of a run's last, shorter chunk in `qk`; S_c, as the hi and lo
// operand tiles that the output kernel copies into shared memory in one piece, and the angles lie in `qk`.
// Bound by the conversions to terms (chunk, output) and by the D and S traffic (64 KB each per chunk and head). 2048 tokens of 32
// heads 194 us with one walk over the chunks (mma.sync), rotation and gate apart, 90 us with approximate gates (4, 24, 13 and 50);
// whole mixer 477 us, 387 and, with gates by expf and a division as in retention.cu, 393 now.
#include <algorithm>

#include "act.cuh"
#include "retention_umma.h"
#include "tcgen05.cuh"

namespace q38 {
Q38_REGISTER_ERROR_WORD();
namespace {

using bf16 = __nv_bfloat16;
constexpr int kDim = 128, kTok = 128, kHalf = kDim / 2;
constexpr int kPow = Q38_RETENTION_CHUNK;                // longest power in the table of decays
constexpr size_t kTileBytes = size_t(kDim) * kDim * 4;   // D fp32; S as hi + lo
constexpr int kSlice = kTok * 128;                       // [128 rows][64 columns bf16], 128-byte swizzle

// places in `qk`, from the batch's first row on: S of every chunk slot, D of every run's last chunk, angles
struct Scratch {
  uint8_t* base;
  int heads, slots, seqs;
  __device__ Scratch(const q38_retention_params& p, const q38_batch_desc& b)
      : base(static_cast<uint8_t*>(p.qk) + (size_t)b.seq_start[0] * p.heads * 4 * kDim * 2), heads(p.heads),
        slots(b.num_tokens / kTok + b.num_seqs), seqs(b.num_seqs) {}
  __device__ uint8_t* state(int slot, int h) const { return base + ((size_t)slot * heads + h) * kTileBytes; }
  __device__ float* last(int seq, int h) const { return reinterpret_cast<float*>(base + ((size_t)(slots + seq) * heads + h) * kTileBytes); }
  __device__ float2* angles() const { return reinterpret_cast<float2*>(base + (size_t)(slots + seqs) * heads * kTileBytes); }
};
inline size_t scratch_bytes(int tokens, int seqs, int heads) {
  return (size_t(tokens / kTok + seqs) + size_t(seqs)) * size_t(heads) * kTileBytes + size_t(tokens) * kHalf * sizeof(float2);
}
// D of chunk c (its first row `row` in the step's arrays)
__device__ __forceinline__ float* chunk_sum(const q38_retention_params& p, const Scratch& sc, int seq, int h, int row, int n) {
  return n == kTok ? p.o + ((size_t)row * p.heads + (size_t)h * kTok) * kDim : sc.last(seq, h);
}
// decay^i, i <= 128
__device__ __forceinline__ float decay_to(const float* pw, int i) { return i <= kPow ? pw[i] : pw[kPow] * pw[i - kPow]; }

__device__ __forceinline__ uint32_t pack2(float a, float b) {
  const __nv_bfloat162 p = __floats2bfloat162_rn(a, b);
  return *reinterpret_cast<const uint32_t*>(&p);
}
// two neighbours as hi and lo terms
__device__ __forceinline__ void split2(float a, float b, uint32_t& hi, uint32_t& lo) {
  hi = pack2(a, b);
  lo = pack2(a - __uint_as_float(hi << 16), b - __uint_as_float(hi & 0xffff0000u));
}
// Past L1, of which little is left beside the tiles in shared memory.
__device__ __forceinline__ uint2 ld_once8(const void* p) {
  uint2 v;
  asm volatile("ld.global.L1::no_allocate.v2.u32 {%0,%1}, [%2];" : "=r"(v.x), "=r"(v.y) : "l"(p));
  return v;
}
__device__ __forceinline__ float4 ld_once16(const void* p) {
  float4 v;
  asm volatile("ld.global.L1::no_allocate.v4.f32 {%0,%1,%2,%3}, [%4];" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "l"(p));
  return v;
}
__device__ __forceinline__ void cp_async16(void* dst, const void* src, bool real) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(smem_u32(dst)), "l"(src), "r"(real ? 16 : 0) : "memory");
}

// A row's eight dimensions of this lane, 4 t .. + 3 and 64 + 4 t .. + 3 (t = lane % 16), before and after the rotation.
struct Pairs {
  uint2 lower, upper;
};
struct Turn {
  float4 a, b;  // (cos, sin) of dimensions 4 t, + 1 and + 2, + 3
};
__device__ __forceinline__ Pairs load_pairs(const bf16* head, int t) { return {ld_once8(head + 4 * t), ld_once8(head + kHalf + 4 * t)}; }
__device__ __forceinline__ Turn load_turn(const float2* row, int t) { return {ld_once16(row + 4 * t), ld_once16(row + 4 * t + 2)}; }
// ... turned, times `f`, into row r of the hi and lo operand tiles (two slices of 64 dimensions each)
__device__ __forceinline__ void store_turned(uint8_t* hi_tile, uint8_t* lo_tile, int r, int t, const Pairs& x, const Turn& w, float f) {
  const float c[4] = {w.a.x, w.a.z, w.b.x, w.b.z}, s[4] = {w.a.y, w.a.w, w.b.y, w.b.w};
  const uint32_t lw[2] = {x.lower.x, x.lower.y}, uw[2] = {x.upper.x, x.upper.y};
  float lo_half[4], up_half[4];
#pragma unroll
  for (int e = 0; e < 4; ++e) {
    const float a = __uint_as_float(e & 1 ? lw[e / 2] & 0xffff0000u : lw[e / 2] << 16);
    const float b = __uint_as_float(e & 1 ? uw[e / 2] & 0xffff0000u : uw[e / 2] << 16);
    lo_half[e] = (a * c[e] - b * s[e]) * f;
    up_half[e] = (b * c[e] + a * s[e]) * f;
  }
  const uint32_t at = uint32_t(r) * 128 + ((uint32_t(t >> 1) ^ uint32_t(r & 7)) << 4) + uint32_t(t & 1) * 8;
  uint2 h, l;
  split2(lo_half[0], lo_half[1], h.x, l.x);
  split2(lo_half[2], lo_half[3], h.y, l.y);
  *reinterpret_cast<uint2*>(hi_tile + at) = h;
  *reinterpret_cast<uint2*>(lo_tile + at) = l;
  split2(up_half[0], up_half[1], h.x, l.x);
  split2(up_half[2], up_half[3], h.y, l.y);
  *reinterpret_cast<uint2*>(hi_tile + kSlice + at) = h;
  *reinterpret_cast<uint2*>(lo_tile + kSlice + at) = l;
}
// 16-byte piece of a value tile: row r, piece c of 16
__device__ __forceinline__ uint32_t value_place(int r, int c) {
  return uint32_t(c >> 3) * kSlice + uint32_t(r) * 128 + ((uint32_t(c & 7) ^ uint32_t(r & 7)) << 4);
}

// ---- angles -------------------------------------------------------------------------------------------------------------------
__global__ void __launch_bounds__(256) retention_angles_kernel(q38_retention_params p, q38_batch_desc b) {
  pdl_wait();
  pdl_launch_dependents();
  const int i = blockIdx.x * 256 + threadIdx.x, row = i / kHalf, d = i % kHalf;
  if (row >= b.num_tokens) return;
  // formed and reduced in double precision
  const double turns = double(b.tok_pos[row]) * p.inv_freq[d] * 0.15915494309189535;
  float sn, cs;
  sincosf(float((turns - rint(turns)) * 6.283185307179586), &sn, &cs);
  Scratch(p, b).angles()[i] = make_float2(cs, sn);
}

constexpr uint32_t kIdesc = (1u << 4) | (1u << 7) | (1u << 10) | (uint32_t(128 >> 3) << 17) | (uint32_t(128 >> 4) << 24);
constexpr uint32_t kMnA = 1u << 15, kMnB = 1u << 16;

// ---- D of a chunk ----------------------------------------------------------------------------------------------------------------
constexpr int kSumThreads = 256;
constexpr int kSumV = 4 * kSlice, kSumBar = kSumV + 2 * kSlice, kSumPw = kSumBar + 32, kSumSmem = 1024 + kSumPw + (kTok + 1) * 4;

__global__ void __launch_bounds__(kSumThreads, 2) retention_chunk_sum_kernel(q38_retention_params p, q38_batch_desc b) {
  extern __shared__ uint8_t sum_raw[];
  uint8_t* smem = sum_raw + ((1024 - (smem_u32(sum_raw) & 1023)) & 1023);
  uint64_t* done = reinterpret_cast<uint64_t*>(smem + kSumBar);
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(done + 1);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);
  float* pw = reinterpret_cast<float*>(smem + kSumPw);
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, t = lane & 15;
  const int c = blockIdx.x, h = blockIdx.y, seq = blockIdx.z;
  if (tid == 0) {
    mbar_init(done, 1);
    *abort_flag = 0;
    mbar_fence_init();
  }
  for (int i = tid; i <= kTok; i += kSumThreads) pw[i] = decay_to(p.decay_pow + h * (kPow + 1), i);
  pdl_wait();
  pdl_launch_dependents();
  const int start = b.seq_start[seq], n = min(kTok, b.seq_start[seq + 1] - start - c * kTok);
  if (n <= 0) return;
  if (warp == 0) tmem_alloc(tmem_slot, 128);
  const Scratch sc(p, b);
  const int row0 = start + c * kTok;
  const bf16* proj = static_cast<const bf16*>(p.proj) + (size_t)row0 * p.ld_proj;
  const bf16 *k_rows = proj + (size_t)(p.heads + h) * kDim, *v_rows = proj + (size_t)(2 * p.heads + h) * kDim;
  const float2* angles = sc.angles() + (size_t)(row0 - b.seq_start[0]) * kHalf;
  for (int i = tid; i < kTok * 16; i += kSumThreads) {
    const int r = i >> 4, piece = i & 15;
    cp_async16(smem + kSumV + value_place(r, piece), v_rows + (size_t)min(r, n - 1) * p.ld_proj + 8 * piece, r < n);
  }
  asm volatile("cp.async.commit_group;" ::: "memory");
  __syncthreads();  // decays
  {  // keys: a warp takes two rows at a time, sixteen in all, every read in flight
    Pairs x[8];
    Turn w[8];
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      const int r = min(n - 1, 16 * i + 2 * warp + (lane >> 4));
      x[i] = load_pairs(k_rows + (size_t)r * p.ld_proj, t);
      w[i] = load_turn(angles + (size_t)r * kHalf, t);
    }
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      const int r = 16 * i + 2 * warp + (lane >> 4);
      if (r >= n) x[i] = Pairs{};  // beyond the run: zeros
      store_turned(smem, smem + 2 * kSlice, r, t, x[i], w[i], r < n ? p.k_scale * pw[n - 1 - r] : 0.0f);
    }
  }
  asm volatile("cp.async.wait_group 0;" ::: "memory");
  fence_async_smem();
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = *tmem_slot;
  if (warp == 0) {  // D^T [v][dk] = V^T K: lanes = v, so that the stores below are whole rows
    const uint64_t vd = smem_desc_sw128_mn(smem_u32(smem + kSumV), kSlice), kd = smem_desc_sw128_mn(smem_u32(smem), kSlice);
#pragma unroll 1
    for (int i = 0; i < 16; ++i)  // lo terms, then hi
      umma_bf16(tmem, vd + uint64_t((i & 7) * 128), kd + uint64_t((i < 8 ? 2 * kSlice >> 4 : 0) + (i & 7) * 128), kIdesc | kMnA | kMnB, uint32_t(i));
    umma_commit(done);
  }
  __syncwarp();
  const bool alive = __all_sync(0xffffffffu, wait_flag(done, 0, abort_flag, 0x501));
  tc_fence_after();
  if (alive) {
    const int quarter = warp & 3, half = warp >> 2, v = 32 * quarter + lane;
    float* dst = chunk_sum(p, sc, seq, h, row0, n) + v;
#pragma unroll 1
    for (int g = 0; g < 4; ++g) {
      uint32_t d[16];
      tmem_ld16(tmem + (uint32_t(32 * quarter) << 16) + uint32_t(64 * half + 16 * g), d);
#pragma unroll
      for (int i = 0; i < 16; ++i) dst[(size_t)(64 * half + 16 * g + i) * kDim] = __uint_as_float(d[i]);
    }
  }
  tc_fence_before();
  __syncthreads();
  if (warp == 0) tmem_dealloc(tmem, 128);
}

// ---- states ahead of the chunks ------------------------------------------------------------------------------------------------------
// a thread: four neighbouring columns of one row of a head's state, all chunks of a run, eight D in flight
__global__ void __launch_bounds__(256) retention_state_sum_kernel(q38_retention_params p, q38_batch_desc b, q38_recurrent_state_desc st) {
  pdl_wait();
  pdl_launch_dependents();
  const int h = blockIdx.y, seq = blockIdx.z, i = blockIdx.x * 256 + threadIdx.x, d = i >> 5, v = 4 * (i & 31);
  const int start = b.seq_start[seq], count = b.seq_start[seq + 1] - start, chunks = (count + kTok - 1) / kTok;
  if (count <= 0) return;
  const Scratch sc(p, b);
  const int slot0 = (start - b.seq_start[0]) / kTok + seq;
  float4* state = reinterpret_cast<float4*>(st.state + (size_t)b.seq_slot[seq] * st.slot_bytes) + (size_t)h * (kDim * kDim / 4) + i;
  float4 s = b.seq_pos0[seq] > 0 ? *state : make_float4(0, 0, 0, 0);
  const float* pw = p.decay_pow + h * (kPow + 1);
  const float whole = decay_to(pw, kTok), rest = decay_to(pw, count - (chunks - 1) * kTok);
  const uint32_t at = uint32_t(v >> 6) * kSlice + uint32_t(d) * 128 + ((uint32_t(v & 63) >> 3 ^ uint32_t(d & 7)) << 4) + uint32_t(v & 4) * 2;
  constexpr int kAhead = 8;
  for (int c0 = 0; c0 < chunks; c0 += kAhead) {
    float4 x[kAhead];
#pragma unroll
    for (int e = 0; e < kAhead; ++e) {
      const int c = min(c0 + e, chunks - 1), n = min(kTok, count - c * kTok);
      x[e] = reinterpret_cast<const float4*>(chunk_sum(p, sc, seq, h, start + c * kTok, n))[i];
    }
#pragma unroll
    for (int e = 0; e < kAhead; ++e) {
      const int c = c0 + e;
      if (c >= chunks) break;
      uint2 hi, lo;
      split2(s.x, s.y, hi.x, lo.x);
      split2(s.z, s.w, hi.y, lo.y);
      uint8_t* tile = sc.state(slot0 + c, h) + at;
      *reinterpret_cast<uint2*>(tile) = hi;
      *reinterpret_cast<uint2*>(tile + 2 * kSlice) = lo;
      const float f = c + 1 < chunks ? whole : rest;
      s.x = f * s.x + x[e].x;
      s.y = f * s.y + x[e].y;
      s.z = f * s.z + x[e].z;
      s.w = f * s.w + x[e].w;
    }
  }
  *state = s;
}

// ---- outputs ---------------------------------------------------------------------------------------------------------------------------
// Persistent CTAs over (chunk slot, head). Eleven warps make the K, Q and V operands of the next item, each as soon as the last
// product with the one before is complete, while eight turn the scores of this one into weights (through tensor memory) and finish
// its outputs, a thread per row and half of the columns; one issues. What takes long are reads of global memory (3,000 cycles beside
// 225 KB of shared memory): all of a warp's are requested ahead of the wait for the buffer. (Q and K together by seven warps in two
// rounds, gates four at a time: 16,000 cycles an item.)
constexpr int kEpiWarps = 8, kConvWarps = 11, kMmaWarp = kEpiWarps + kConvWarps, kOutThreads = (kMmaWarp + 1) * 32;
constexpr int kOutQ = 0, kOutK = 4 * kSlice, kOutS = 8 * kSlice, kOutV = 12 * kSlice, kOutBar = 14 * kSlice;  // Q, K, S: hi, lo of two slices
constexpr int kOutSs = kOutBar + 128, kOutPw = kOutSs + 2 * kTok * 4, kOutSmem = 1024 + kOutPw + (kTok + 1) * 4;
static_assert(kOutSmem <= 227 * 1024, "shared memory");
constexpr uint32_t kTmScore = 0, kTmD1 = 128, kTmD2 = 256, kTmP = 384;  // tensor memory columns; P: hi, lo of 64

// Sum of squares of a row's outputs in its half of the columns. `lanes`: the warp's rows in tensor memory, `mine`: decay^(row + 1).
__device__ __forceinline__ float sum_squares(uint32_t lanes, int half, float mine) {
  float ss = 0.0f;
#pragma unroll
  for (int g = 0; g < 8; ++g) {
    uint32_t d1[8], d2[8];
    tmem_ld8(lanes + kTmD1 + uint32_t(64 * half + 8 * g), d1);
    tmem_ld8(lanes + kTmD2 + uint32_t(64 * half + 8 * g), d2);
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      const float o = mine * __uint_as_float(d1[i]) + __uint_as_float(d2[i]);
      ss += o * o;
    }
  }
  return ss;
}
// Eight columns of a row's outputs, normalised and gated.
__device__ __forceinline__ void gated_outputs(uint32_t lanes, int half, int g, float mine, float rs, const uint4& gate, bool store, uint4* dst) {
  const uint32_t two[4] = {gate.x, gate.y, gate.z, gate.w};
  uint32_t d1[8], d2[8];
  tmem_ld8(lanes + kTmD1 + uint32_t(64 * half + 8 * g), d1);
  tmem_ld8(lanes + kTmD2 + uint32_t(64 * half + 8 * g), d2);
  uint32_t y[4];
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const float a = (mine * __uint_as_float(d1[2 * i]) + __uint_as_float(d2[2 * i])) * rs;
    const float c = (mine * __uint_as_float(d1[2 * i + 1]) + __uint_as_float(d2[2 * i + 1])) * rs;
    y[i] = pack2(a * silu_f(__uint_as_float(two[i] << 16)), c * silu_f(__uint_as_float(two[i] & 0xffff0000u)));
  }
  if (store) dst[g] = make_uint4(y[0], y[1], y[2], y[3]);
  __syncwarp();  // divisions and stores of single lanes are over: the next loads from tensor memory are the whole warp's
}
// A weight of zero times a value that is not finite is NaN: a bad value row spoils the rows ahead of it in D2 too. Here their sums
// are formed again over their own and earlier tokens alone, from the weights in tensor memory, and the outputs from them. Called by
// the two warps of a quarter of the rows; seldom, hence with code and registers of its own (in place 4 % of a whole mixer, here nothing that shows).
__device__ __noinline__ void outputs_again(uint32_t lanes, int half, int r, float mine, const bf16* v_rows, int ld, int n, float* ss_sm, float eps,
                                           const uint4* gate, bool store, uint4* dst) {
  const int bar = 2 + r / 32;
  named_bar_sync(bar, 64);  // both warps have read the old sums
#pragma unroll 1
  for (int g = 0; g < 8; ++g) {
    uint32_t d2[8];
    tmem_ld8(lanes + kTmD2 + uint32_t(64 * half + 8 * g), d2);
    float zero = 0.0f, sum[8] = {};
#pragma unroll
    for (int i = 0; i < 8; ++i) zero = fmaf(__uint_as_float(d2[i]), 0.0f, zero);
    if (!__any_sync(0xffffffffu, zero != 0.0f)) continue;
#pragma unroll 1
    for (int j0 = 0; j0 < kTok; j0 += 16) {
      uint32_t hi[8], lo[8];
      tmem_ld8(lanes + kTmP + uint32_t(j0 / 2), hi);
      tmem_ld8(lanes + kTmP + uint32_t(64 + j0 / 2), lo);
#pragma unroll
      for (int e = 0; e < 16; ++e) {
        const uint4 v = *reinterpret_cast<const uint4*>(v_rows + (size_t)min(j0 + e, n - 1) * ld + 8 * g);
        const uint32_t vw[4] = {v.x, v.y, v.z, v.w}, h = hi[e / 2], l = lo[e / 2];
        const float w = e & 1 ? __uint_as_float(h & 0xffff0000u) + __uint_as_float(l & 0xffff0000u) : __uint_as_float(h << 16) + __uint_as_float(l << 16);
#pragma unroll
        for (int i = 0; i < 8; ++i) {
          const float x = sum[i] + w * __uint_as_float(i & 1 ? vw[i / 2] & 0xffff0000u : vw[i / 2] << 16);
          sum[i] = j0 + e <= r ? x : sum[i];
        }
      }
    }
#pragma unroll
    for (int i = 0; i < 8; ++i) d2[i] = zero != 0.0f ? __float_as_uint(sum[i]) : d2[i];
    tmem_st8(lanes + kTmD2 + uint32_t(64 * half + 8 * g), d2);
  }
  tmem_wait_st();
  ss_sm[half * kTok + r] = sum_squares(lanes, half, mine);
  named_bar_sync(bar, 64);
  const float rs = 1.0f / sqrtf((ss_sm[r] + ss_sm[kTok + r]) / float(kDim) + eps);
#pragma unroll 1
  for (int g = 0; g < 8; ++g) gated_outputs(lanes, half, g, mine, rs, gate[g], store, dst);
}

__global__ void __launch_bounds__(kOutThreads, 1) retention_output_kernel(q38_retention_params p, q38_batch_desc b) {
  extern __shared__ uint8_t out_raw[];
  uint8_t* smem = out_raw + ((1024 - (smem_u32(out_raw) & 1023)) & 1023);
  uint64_t* bar = reinterpret_cast<uint64_t*>(smem + kOutBar);
  uint64_t *k_full = bar, *v_full = bar + 1, *s_full = bar + 2, *q_full = bar + 8;  // operands in shared memory
  uint64_t *score_done = bar + 3, *state_done = bar + 4, *out_done = bar + 5;   // products Q K^T, Q S, P V
  uint64_t *p_full = bar + 6, *d_empty = bar + 7;                               // weights in tensor memory; results read
  uint64_t* drained = bar + 9;                                                  // products of a CTA that gave up
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bar + 10);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);
  float *ss_sm = reinterpret_cast<float*>(smem + kOutSs), *pw = reinterpret_cast<float*>(smem + kOutPw);
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  if (tid == 0) {
    mbar_init(k_full, kConvWarps);
    mbar_init(q_full, kConvWarps);
    mbar_init(v_full, kConvWarps);
    for (int i = 2; i < 6; ++i) mbar_init(&bar[i], 1);
    mbar_init(p_full, kEpiWarps);
    mbar_init(d_empty, kEpiWarps);
    mbar_init(drained, 1);
    *abort_flag = 0;
    mbar_fence_init();
  }
  if (warp == kMmaWarp) tmem_alloc(tmem_slot, 512);
  pdl_wait();
  pdl_launch_dependents();
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = *tmem_slot;
  const Scratch sc(p, b);
  const int items = sc.slots * p.heads, base = b.seq_start[0];
  bool alive = true;  // false: a wait ran out; the role goes through its loop without waiting, computing or storing
  auto wait = [&](uint64_t* at, int it, unsigned site) {  // every barrier completes once per item
    bool there = !alive;
#pragma unroll 1
    for (uint32_t i = 0; i < kSpinLimit && !there; ++i) {
      there = mbar_try_wait(at, uint32_t(it) & 1u);
      if (!there && *abort_flag) break;
    }
    if (!there) {
      report_error(site);
      *abort_flag = 1;
    }
    alive = __all_sync(0xffffffffu, alive && there);
  };
  // run and rows of a chunk slot; false where the slot is not in use
  int row0 = 0, n = 0;
  auto locate = [&](int slot) {
#pragma unroll 1
    for (int q = 0; q < b.num_seqs; ++q) {
      const int start = b.seq_start[q], count = b.seq_start[q + 1] - start, c = slot - ((start - base) / kTok + q);
      if (c >= 0 && c * kTok < count) {
        row0 = start + c * kTok;
        n = min(kTok, count - c * kTok);
        return true;
      }
    }
    return false;
  };
  int it = 0;
  if (warp == kMmaWarp) {
    const uint64_t q = smem_desc_sw128(smem_u32(smem + kOutQ)), k = smem_desc_sw128(smem_u32(smem + kOutK));
    const uint64_t s = smem_desc_sw128_mn(smem_u32(smem + kOutS), kSlice), v = smem_desc_sw128_mn(smem_u32(smem + kOutV), kSlice);
    const uint64_t policy = policy_evict_first();
    constexpr uint32_t kLoTile = 2 * kSlice >> 4;
    int requested = 0;
    auto request_state = [&](int item) {
      requested += alive ? 1 : 0;
      if (lane == 0 && alive) {
        mbar_expect_tx(s_full, uint32_t(kTileBytes));
        bulk_g2s(smem + kOutS, sc.state(item / p.heads, item % p.heads), uint32_t(kTileBytes), s_full, policy);
      }
      __syncwarp();
    };
    int next = blockIdx.x;
    auto advance = [&]() {  // the next item in use
      while (next < items && !locate(next / p.heads)) next += gridDim.x;
      return next < items;
    };
    bool more = advance();
    if (more) request_state(next);
#pragma unroll 1
    for (; more; ++it) {
      next += gridDim.x;
      more = advance();
      wait(k_full, it, 0x511);
      wait(q_full, it, 0x51b);
      if (alive) {
        tc_fence_after();
#pragma unroll 1
        for (int i = 0; i < 24; ++i) {  // lo hi, hi lo, hi hi; two slices of four steps
          const uint32_t at = uint32_t((i >> 2 & 1) * (kSlice >> 4) + (i & 3) * 2);
          umma_bf16(tmem + kTmScore, q + uint64_t(at + (i < 8 ? kLoTile : 0u)), k + uint64_t(at + (i >= 8 && i < 16 ? kLoTile : 0u)), kIdesc, uint32_t(i));
        }
        umma_commit(score_done);
      }
      wait(s_full, it, 0x512);
      if (it > 0) wait(d_empty, it - 1, 0x513);
      if (alive) {
        tc_fence_after();
#pragma unroll 1
        for (int i = 0; i < 24; ++i) {
          const uint32_t at = uint32_t((i >> 2 & 1) * (kSlice >> 4) + (i & 3) * 2);
          umma_bf16(tmem + kTmD1, q + uint64_t(at + (i < 8 ? kLoTile : 0u)), s + uint64_t((i & 7) * 128 + (i >= 8 && i < 16 ? kLoTile : 0u)),
                    kIdesc | kMnB, uint32_t(i));
        }
        umma_commit(state_done);
      }
      wait(v_full, it, 0x514);
      wait(p_full, it, 0x515);
      if (alive) {
        tc_fence_after();
#pragma unroll 1
        for (int i = 0; i < 16; ++i)
          umma_bf16_ts(tmem + kTmD2, tmem + kTmP + uint32_t((i < 8 ? 64 : 0) + (i & 7) * 8), v + uint64_t((i & 7) * 128), kIdesc | kMnB, uint32_t(i));
        umma_commit(out_done);
      }
      wait(state_done, it, 0x516);
      if (more) request_state(next);
    }
    if (!alive) {  // given up: the copy and the products that may be in flight end before shared and tensor memory go to another CTA
      if (requested > 0) mbar_wait(s_full, uint32_t(requested - 1) & 1u, 0x51c);
      umma_commit(drained);
      mbar_wait(drained, 0, 0x51d);
      __syncwarp();
    }
  } else if (warp >= kEpiWarps) {
    const int first = warp - kEpiWarps, t = lane & 15;
    constexpr int kRows = (kTok / 2 + kConvWarps - 1) / kConvWarps;  // of a warp, two at a time
    auto row = [&](int i) { return 2 * (i * kConvWarps + first) + (lane >> 4); };
    auto release_values = [&]() {
      asm volatile("cp.async.wait_group 0;" ::: "memory");
      fence_async_smem();
      __syncwarp();
      if (lane == 0) mbar_arrive(v_full);
    };
#pragma unroll 1
    for (int item = blockIdx.x; item < items; item += gridDim.x) {
      if (!locate(item / p.heads)) continue;
      const int h = item % p.heads;
      const bf16* proj = static_cast<const bf16*>(p.proj) + (size_t)row0 * p.ld_proj + (size_t)h * kDim;
      const float2* angles = sc.angles() + (size_t)(row0 - base) * kHalf;
#pragma unroll 1
      for (int m = 0; m < 2; ++m) {  // K, then Q
        Pairs x[kRows];
        Turn w[kRows];
        const bf16* src = proj + (m == 0 ? (size_t)p.heads * kDim : 0);
#pragma unroll
        for (int i = 0; i < kRows; ++i) {
          const int r = min(row(i), n - 1);  // beyond the run: the last row's, masked or not stored
          x[i] = load_pairs(src + (size_t)r * p.ld_proj, t);
          w[i] = load_turn(angles + (size_t)r * kHalf, t);
        }
        if (it > 0) {
          if (m == 0) release_values();  // the last item's
          wait(m == 0 ? score_done : state_done, it - 1, 0x517);
        }
        uint8_t* dst = smem + (m == 0 ? kOutK : kOutQ);
        const float f = m == 0 ? p.k_scale : 1.0f;
#pragma unroll
        for (int i = 0; i < kRows; ++i)
          if (row(i) < kTok) store_turned(dst, dst + 2 * kSlice, row(i), t, x[i], w[i], f);
        fence_async_smem();
        __syncwarp();
        if (lane == 0) mbar_arrive(m == 0 ? k_full : q_full);
      }
      if (it > 0) wait(out_done, it - 1, 0x518);
      const bf16* v_rows = proj + (size_t)2 * p.heads * kDim;
      for (int i = first * 32 + lane; i < kTok * 16; i += kConvWarps * 32) {
        const int r = i >> 4, piece = i & 15;
        cp_async16(smem + kOutV + value_place(r, piece), v_rows + (size_t)min(r, n - 1) * p.ld_proj + 8 * piece, r < n);
      }
      asm volatile("cp.async.commit_group;" ::: "memory");
      ++it;
    }
    if (it > 0) release_values();
  } else {
    const int quarter = warp & 3, half = warp >> 2, r = 32 * quarter + lane;  // the thread's row and its half of the columns
    const uint32_t lanes = tmem + (uint32_t(32 * quarter) << 16);
#pragma unroll 1
    for (int item = blockIdx.x; item < items; item += gridDim.x) {
      if (!locate(item / p.heads)) continue;
      const int h = item % p.heads;
      if (tid <= kTok) pw[tid] = decay_to(p.decay_pow + h * (kPow + 1), tid);
      named_bar_sync(1, kEpiWarps * 32);
      wait(score_done, it, 0x519);
      tc_fence_after();
#pragma unroll 1
      for (int g = 0; g < 4; ++g) {
        const int j0 = 64 * half + 16 * g;
        uint32_t s[16], hi[8], lo[8];
        tmem_ld16(lanes + kTmScore + uint32_t(j0), s);
#pragma unroll
        for (int i = 0; i < 8; ++i) {
          float w[2];
#pragma unroll
          for (int e = 0; e < 2; ++e) {
            const int back = r - j0 - 2 * i - e;
            w[e] = back < 0 ? 0.0f : __uint_as_float(s[2 * i + e]) * pw[max(back, 0)];
          }
          split2(w[0], w[1], hi[i], lo[i]);
        }
        tmem_st8(lanes + kTmP + uint32_t(j0 / 2), hi);
        tmem_st8(lanes + kTmP + uint32_t(64 + j0 / 2), lo);
      }
      tmem_wait_st();
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(p_full);
      const float mine = pw[r + 1];
      const bool live = r < n;
      const size_t at = (size_t)(row0 + min(r, n - 1));
      const uint4* gate = reinterpret_cast<const uint4*>(static_cast<const bf16*>(p.proj) + at * p.ld_proj +
                                                         (size_t)(3 * p.heads + h) * kDim + 64 * half);
      uint4* dst = reinterpret_cast<uint4*>(static_cast<bf16*>(p.out) + at * p.ld_out + (size_t)h * kDim + 64 * half);
      uint4 gw[8];
#pragma unroll
      for (int g = 0; g < 8; ++g) gw[g] = gate[g];
      wait(out_done, it, 0x51a);
      tc_fence_after();
      ss_sm[half * kTok + r] = sum_squares(lanes, half, mine);
      named_bar_sync(1, kEpiWarps * 32);
      const float squares = ss_sm[r] + ss_sm[kTok + r], rs = 1.0f / sqrtf(squares / float(kDim) + p.eps);
#pragma unroll
      for (int g = 0; g < 8; ++g) gated_outputs(lanes, half, g, mine, rs, gw[g], live && alive, dst);
      if (__any_sync(0xffffffffu, !(squares < INFINITY)))  // the same for both halves, given up or not: they meet in there
        outputs_again(lanes, half, r, mine, static_cast<const bf16*>(p.proj) + (size_t)row0 * p.ld_proj + (size_t)(2 * p.heads + h) * kDim + 64 * half,
                      p.ld_proj, n, ss_sm, p.eps, gate, live && alive, dst);
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(d_empty);
      ++it;
    }
  }
  tc_fence_before();
  __syncthreads();
  if (warp == kMmaWarp) tmem_dealloc(tmem, 512);
}

}  // namespace

// The scratch of a call is that of retention.cu's kernels: it holds two states per run and one per 128 tokens from about 256
// tokens a run on (heads / (heads - 1) of that). Shorter runs go to those kernels for want of scratch, not for their speed: 264
// tokens of 32 heads in one run, whole mixer, 114 us there and 111 here, 300 of 16 heads 69 and 65, 512 of 32 heads 146 and 128.
bool retention_umma_fits(const q38_retention_params& p, const q38_batch_desc& b, const q38_recurrent_state_desc& st) {
  const auto aligned = [](const void* q, size_t a) { return reinterpret_cast<uintptr_t>(q) % a == 0; };
  return p.act == Q38_ACT_BF16 && p.dim == kDim && p.vdim == kDim && p.rot_dims == kDim && p.qk && p.o && p.ld_proj % 8 == 0 &&
         p.ld_out % 8 == 0 && aligned(p.proj, 16) && aligned(p.out, 16) && aligned(p.qk, 16) && aligned(p.o, 16) && aligned(st.state, 16) &&
         st.slot_bytes % 16 == 0 && scratch_bytes(b.num_tokens, b.num_seqs, p.heads) <= q38_retention_qk_bytes(b.num_tokens, p.heads, p.dim, p.act);
}

int retention_umma(const q38_retention_params& p, const q38_batch_desc& b, const q38_recurrent_state_desc& st, cudaStream_t s) {
  static const cudaError_t attrs[2] = {
      cudaFuncSetAttribute(retention_chunk_sum_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kSumSmem),
      cudaFuncSetAttribute(retention_output_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kOutSmem)};
  for (const cudaError_t e : attrs) Q38_CUDA_OK(e);
  (void)launch_kernel(retention_angles_kernel, dim3((b.num_tokens * kHalf + 255) / 256), dim3(256), 0, s, p, b);
  Q38_LAUNCH_OK("retention_angles_kernel");
  (void)launch_kernel(retention_chunk_sum_kernel, dim3((b.max_tokens_per_seq + kTok - 1) / kTok, p.heads, b.num_seqs), dim3(kSumThreads), kSumSmem, s,
                      p, b);
  Q38_LAUNCH_OK("retention_chunk_sum_kernel");
  (void)launch_kernel(retention_state_sum_kernel, dim3(kDim * kDim / 4 / 256, p.heads, b.num_seqs), dim3(256), 0, s, p, b, st);
  Q38_LAUNCH_OK("retention_state_sum_kernel");
  const long long items = (long long)(b.num_tokens / kTok + b.num_seqs) * p.heads;
  (void)launch_kernel(retention_output_kernel, dim3(unsigned(std::min<long long>(num_sms(), items))), dim3(kOutThreads), kOutSmem, s, p, b);
  Q38_LAUNCH_OK("retention_output_kernel");
  return Q38_OK;
}

}  // namespace q38
