// Embedding gather, ragged-batch packing, sampling and scoring kernels of the step.
#include <cooperative_groups.h>

#include "common.cuh"
#include "host_util.h"

namespace q38 {
namespace {

// ---------------------------------------------------------------------------------------------------
// embed: residual[m] = table[tokens[m]] widened to fp32, bf16 copy, sum of squares per 128 columns.
// Replaces kernels::embed (reference src/kernels/kernels.h:131-134, src/kernels/embed.cu:13-43).
// One CTA per token; a warp owns whole 128-column blocks (4 columns per lane) so each partial is one
// warp reduction. The table may live in mapped pinned host memory (plain loads work for both).
// ---------------------------------------------------------------------------------------------------
__global__ void __launch_bounds__(256) embed_kernel(const __nv_bfloat16* __restrict__ table,
                                                    const int32_t* __restrict__ tokens, int hidden,
                                                    float* __restrict__ residual, __nv_bfloat16* __restrict__ xbf,
                                                    float* __restrict__ partials) {
  pdl_wait();               // everything written by earlier kernels of the stream is visible from here on
  pdl_launch_dependents();  // the next kernel may be scheduled now; it holds its own dependent work back the same way
  const int m = blockIdx.x, lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const __nv_bfloat16* row = table + (size_t)tokens[m] * hidden;
  const int blocks = hidden / 128;
  for (int b = warp; b < blocks; b += blockDim.x >> 5) {
    const int col = b * 128 + 4 * lane;
    const uint2 raw = *reinterpret_cast<const uint2*>(row + col);
    const __nv_bfloat162 p0 = *reinterpret_cast<const __nv_bfloat162*>(&raw.x);
    const __nv_bfloat162 p1 = *reinterpret_cast<const __nv_bfloat162*>(&raw.y);
    const float4 v = make_float4(__low2float(p0), __high2float(p0), __low2float(p1), __high2float(p1));
    *reinterpret_cast<float4*>(residual + (size_t)m * hidden + col) = v;
    *reinterpret_cast<uint2*>(xbf + (size_t)m * hidden + col) = raw;
    const float ss = warp_sum(v.x * v.x + v.y * v.y + v.z * v.z + v.w * v.w);
    if (lane == 0) partials[(size_t)m * blocks + b] = ss;
  }
}

// ---------------------------------------------------------------------------------------------------
// residual_update: the Residual GEMM epilogue as an op of its own, for tensor-parallel runs in which the
// row-parallel projection's partial products are summed over the ranks before they may enter the residual:
// residual += delta; xbf = bf16(residual); partials[m][col / 128] = sum of residual^2 over the 128 columns.
// One warp per (token, 128-column block), as embed_kernel.
// ---------------------------------------------------------------------------------------------------
__global__ void __launch_bounds__(256) residual_update_kernel(const float* __restrict__ delta, int hidden,
                                                              float* __restrict__ residual,
                                                              __nv_bfloat16* __restrict__ xbf,
                                                              float* __restrict__ partials) {
  pdl_wait();
  pdl_launch_dependents();
  const int m = blockIdx.x, lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int blocks = hidden / 128;
  for (int b = warp; b < blocks; b += blockDim.x >> 5) {
    const size_t at = (size_t)m * hidden + b * 128 + 4 * lane;
    const float4 d = *reinterpret_cast<const float4*>(delta + at);
    float4 r = *reinterpret_cast<const float4*>(residual + at);
    r.x += d.x;
    r.y += d.y;
    r.z += d.z;
    r.w += d.w;
    *reinterpret_cast<float4*>(residual + at) = r;
    const __nv_bfloat162 p0 = __floats2bfloat162_rn(r.x, r.y), p1 = __floats2bfloat162_rn(r.z, r.w);
    uint2 packed;
    packed.x = *reinterpret_cast<const uint32_t*>(&p0);
    packed.y = *reinterpret_cast<const uint32_t*>(&p1);
    *reinterpret_cast<uint2*>(xbf + at) = packed;
    const float ss = warp_sum(r.x * r.x + r.y * r.y + r.z * r.z + r.w * r.w);
    if (lane == 0) partials[(size_t)m * blocks + b] = ss;
  }
}

// ---------------------------------------------------------------------------------------------------
// pack_ragged: per-sequence (count, pos0) -> seq_start (exclusive scan), tok_pos, tok_seq.
// One CTA; the scan is a shared-memory Hillis-Steele over up to 1024 sequences per pass.
// ---------------------------------------------------------------------------------------------------
__global__ void __launch_bounds__(1024) pack_ragged_kernel(const int* __restrict__ seq_count,
                                                           const int* __restrict__ seq_pos0, int num_seqs,
                                                           int num_tokens, int* __restrict__ seq_start,
                                                           int* __restrict__ tok_pos, int* __restrict__ tok_seq) {
  pdl_wait();               // everything written by earlier kernels of the stream is visible from here on
  pdl_launch_dependents();  // the next kernel may be scheduled now; it holds its own dependent work back the same way
  __shared__ int scan[1024];
  __shared__ int carry;
  const int tid = threadIdx.x;
  if (tid == 0) carry = 0;
  __syncthreads();
  for (int base = 0; base < num_seqs; base += 1024) {
    const int b = base + tid;
    const int cnt = b < num_seqs ? seq_count[b] : 0;
    scan[tid] = cnt;
    __syncthreads();
    for (int o = 1; o < 1024; o <<= 1) {
      const int add = tid >= o ? scan[tid - o] : 0;
      __syncthreads();
      scan[tid] += add;
      __syncthreads();
    }
    const int start = carry + scan[tid] - cnt;
    if (b < num_seqs) seq_start[b] = start;
    __syncthreads();
    if (tid == 1023) carry += scan[1023];
    __syncthreads();
  }
  if (tid == 0) seq_start[num_seqs] = carry;
  __syncthreads();
  // expansion: one warp per sequence, lanes stride over its tokens
  const int lane = tid & 31, warp = tid >> 5;
  for (int b = warp; b < num_seqs; b += 32) {
    const int s = seq_start[b], n = seq_count[b], p0 = seq_pos0[b];
    for (int i = lane; i < n; i += 32) {
      if (s + i < num_tokens) {
        tok_pos[s + i] = p0 + i;
        tok_seq[s + i] = b;
      }
    }
  }
}

// ---------------------------------------------------------------------------------------------------
// sampling (reference src/kernels/kernels.h:233-256, src/kernels/sampling.cu:137-310). Definition reproduced here: repetition / presence penalties applied once per distinct token of
// the slot's history; temperature <= 0 -> argmax with the lowest id among ties (log-prob reported as
// 0); otherwise top-k keeps every logit >= the k-th largest, min-p keeps l >= max + T log(min_p),
// top-p keeps the smallest set of largest logits whose mass reaches top_p of the kept mass, and the
// token is drawn by inverse CDF in index order. All masses are integers in 2^-40 fixed point, so the
// draw is a pure function of (logits, params, seed, step).
//
// Where this departs from the reference kernel: the reference takes exp((l - max) / T) from the special-function
// unit (__expf) and the min-p bound from logf, whose bit patterns belong to one GPU generation and to no CPU. Here
// both come from fixed_mass(), a sequence of IEEE single / double operations with explicit roundings (no contraction,
// no library call), so a host restatement of this file gives the same integer masses, the same thresholds and
// therefore the same token for every (logits, params, seed, step). The min-p bound is the smallest logit whose mass
// reaches min_p * 2^40, found by bisection over the ordered float keys.
//
// Work split. A row is read by a cluster of 1 ... 8 CTAs (kernels.h's contract allocates nothing, so what the CTAs
// exchange lies in their shared memories); a warp owns one contiguous part of the row and reads it 16 bytes per lane.
// Masses are integers, so neither the split nor the order of a sum changes a result. With 0 < top_k <= kFastTopK (the
// engine's default is 20) the row is read twice: the first pass finds the maximum and, per CTA, the top_k-th largest
// of its threads' maxima - at least top_k logits are no smaller, so the largest of those bounds is a floor below which
// nothing is kept - and the second sums the masses and lists the few logits above the floor; rank 0 settles top-k,
// min-p, top-p and the draw on that list. Everything else, and a list that overflows (ties), takes radix_threshold.
// What bounds it: the double-precision polynomial of the masses (14 FMAs per logit) and two reads of the row from L2.
// 64 rows of 248,320 logits with the default sampling: 3330 us with one CTA per row and four radix passes per filter
// (64-bit shared atomics on a handful of bins), 60 us here (67 with branches and double conversions in the masses and a key and an
// index kept per logit in the first pass); one row 3280 -> 31 us; greedy, 64 rows, 12.3 -> 10.0 us.
// top_p without top_k, 64 rows: 3287 -> 273 us.
// ---------------------------------------------------------------------------------------------------
constexpr int kSampleThreads = 512, kSampleWarps = kSampleThreads / 32;
constexpr int kFastTopK = 256;         // the floor needs top_k thread maxima in a CTA
constexpr int kOwnList = 1024;         // listed logits of a CTA, and of all of them together
constexpr int kAllList = 2048;
constexpr int kHistCopies = 8;         // lanes of a warp that meet in one bin take different copies of it

struct SampleShared {
  union {
    uint32_t seen[(256 * 1024) / 32];
    struct {
      unsigned long long mass[kAllList];
      uint32_t key[kAllList];
      int index[kAllList];
    } all;
    struct {
      uint32_t lo[256 * kHistCopies], hi[256 * kHistCopies];
    } hist;
  };
  uint32_t own_key[kOwnList];
  int own_index[kOwnList];
  unsigned long long digit_sum[256];  // of the row
  unsigned long long warp_u64[2][kSampleWarps];
  float warp_f[kSampleWarps];
  int warp_i[kSampleWarps];
  // read by the other CTAs of the cluster
  unsigned long long own_digit[256];  // of this CTA's part of the row
  float cta_best;
  int cta_best_index;
  uint32_t cta_floor;
  int own_count;
  unsigned long long cta_kept, cta_all;
  uint32_t pick_prefix;
  unsigned long long pick_above;
  uint32_t pick_key;
};

__device__ __forceinline__ uint32_t order_key(float x) {
  uint32_t u = __float_as_uint(x);
  asm("" : "+r"(u));  // an integer from here on: u | 0x80000000 as -|x| would make 0x7fffffff of a NaN, the key of -0
  return (u & 0x80000000u) ? ~u : (u | 0x80000000u);
}

__device__ __forceinline__ uint64_t mix64(uint64_t x) {
  x += 0x9E3779B97F4A7C15ull;
  x = (x ^ (x >> 30)) * 0xBF58476D1CE4E5B9ull;
  x = (x ^ (x >> 27)) * 0x94D049BB133111EBull;
  return x ^ (x >> 31);
}

// 2^40 * exp((l - max) * inv_t), truncated, in operations that round the same way on every IEEE machine:
// x = fl32(fl32(l - max) * inv_t); y = fl64(x * log2 e); n = floor(y + 1/2); f = y - n (exact); 2^f by a degree-13
// Taylor polynomial in Horner form with fused multiply-adds; the scaling by 2^(n + 40) is exact.
// Without branches and without conversions of doubles: adding 1.5 * 2^52
// rounded down leaves floor(y + 1/2) in the low word, the power of two goes into the exponent of the polynomial, and adding 2^52
// rounded toward zero leaves the truncated integer in the mantissa.
__device__ __forceinline__ unsigned long long fixed_mass(float l, float max_logit, float inv_t) {
  const float x = __fmul_rn(__fsub_rn(l, max_logit), inv_t);
  const double y = __dmul_rn(double(x), 1.4426950408889634);
  const double r = __dadd_rd(__dadd_rn(y, 0.5), 6755399441055744.0);
  const double n = __dsub_rn(r, 6755399441055744.0);
  const double f = __dsub_rn(y, n);
  double p = 1.3691488853904128e-12;
  p = fma(p, f, 2.5678435993488206e-11);
  p = fma(p, f, 4.4455382718708116e-10);
  p = fma(p, f, 7.054911620801123e-09);
  p = fma(p, f, 1.01780860092397e-07);
  p = fma(p, f, 1.321548679014431e-06);
  p = fma(p, f, 1.5252733804059841e-05);
  p = fma(p, f, 0.0001540353039338161);
  p = fma(p, f, 0.0013333558146428443);
  p = fma(p, f, 0.009618129107628477);
  p = fma(p, f, 0.05550410866482158);
  p = fma(p, f, 0.24022650695910072);
  p = fma(p, f, 0.6931471805599453);
  p = fma(p, f, 1.0);
  const uint32_t e = uint32_t(__double2loint(r)) + 40u;  // -24 .. 40 for y in (-64, 0]
  const double v = __hiloint2double(int(uint32_t(__double2hiint(p)) + (e << 20)), __double2loint(p));
  const unsigned long long whole = (unsigned long long)__double_as_longlong(__dadd_rz(v, 4503599627370496.0)) & ((1ull << 52) - 1);
  // y <= -64: below 2^-24 of one fixed-point unit (also NaN and -inf); y > 0: l above the maximum cannot happen
  return y > 0.0 ? 1ull << 40 : y > -64.0 ? whole : 0ull;
}

__device__ __forceinline__ float key_to_float(uint32_t key) {
  return __uint_as_float((key & 0x80000000u) ? (key & 0x7fffffffu) : ~key);
}

// Smallest ordered key whose logit keeps a mass of at least min_p * 2^40 (bisection between -FLT_MAX and the maximum).
__device__ uint32_t min_p_key(float max_logit, float inv_t, float min_p) {
  const unsigned long long cut = (unsigned long long)__dmul_rn(double(min_p), 1099511627776.0);
  uint32_t lo = 0x00800000u;  // key of -FLT_MAX
  uint32_t hi = (__float_as_uint(max_logit) & 0x80000000u) ? ~__float_as_uint(max_logit)
                                                           : (__float_as_uint(max_logit) | 0x80000000u);
  if (hi < lo) return hi;
  while (lo < hi) {
    const uint32_t mid = lo + ((hi - lo) >> 1);
    if (fixed_mass(key_to_float(mid), max_logit, inv_t) >= cut) hi = mid;
    else lo = mid + 1u;
  }
  return hi;
}

// Also orders global and shared memory among the CTAs of a row (one CTA by itself has the cheaper barrier).
__device__ __forceinline__ void cluster_barrier(int cluster) {
  if (cluster == 1) __syncthreads();
  else asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}
template <typename T>
__device__ __forceinline__ const T* of_rank(const T* p, int rank) {
  return cooperative_groups::this_cluster().map_shared_rank(const_cast<T*>(p), rank);
}

__device__ __forceinline__ unsigned long long warp_sum_u64(unsigned long long v) {
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}

// The calling warp's part [lo, hi) of a row, visited in steps of 128 logits, four consecutive ones per lane:
// f(index, logit) for each, ascending per lane. Four loads are in flight per lane. In the steps of unaligned rows and the last ones of
// the others there are two, and one piece of code, unless FOUR: where f is short the loads are what takes long (greedy, 64 rows of
// 248,319 logits, unaligned: 17.4 us with two, 13.9 with four), else the code is (top-p alone, 64 rows: 253 us with two, 257 with four).
struct RowPart {
  const float* row;
  int lo, hi;
  bool vec;  // the row starts on a 16-byte boundary (the parts do: they start at multiples of 128)
  __device__ __forceinline__ float4 load(int i) const {
    float4 v;
    if (vec && i + 3 < hi) return *reinterpret_cast<const float4*>(row + i);
    v.x = i < hi ? row[i] : 0.0f;
    v.y = i + 1 < hi ? row[i + 1] : 0.0f;
    v.z = i + 2 < hi ? row[i + 2] : 0.0f;
    v.w = i + 3 < hi ? row[i + 3] : 0.0f;
    return v;
  }
  template <bool FOUR = false, typename F>
  __device__ __forceinline__ void each(int lane, F f) const {
    constexpr int kAhead = 4;
    int i0 = lo + 4 * lane;
    if (vec)
      for (; i0 + 128 * (kAhead - 1) + 3 < hi; i0 += 128 * kAhead) {
        float4 v[kAhead];
#pragma unroll
        for (int u = 0; u < kAhead; ++u) v[u] = *reinterpret_cast<const float4*>(row + i0 + 128 * u);
#pragma unroll
        for (int u = 0; u < kAhead; ++u) {
          f(i0 + 128 * u, v[u].x);
          f(i0 + 128 * u + 1, v[u].y);
          f(i0 + 128 * u + 2, v[u].z);
          f(i0 + 128 * u + 3, v[u].w);
        }
      }
    if constexpr (FOUR) {
      for (; i0 < hi; i0 += 128 * kAhead) {
        float4 v[kAhead];
#pragma unroll
        for (int u = 0; u < kAhead; ++u)
          if (i0 + 128 * u < hi) v[u] = load(i0 + 128 * u);
#pragma unroll
        for (int u = 0; u < kAhead; ++u) {
          const int i = i0 + 128 * u;
          if (i < hi) f(i, v[u].x);
          if (i + 1 < hi) f(i + 1, v[u].y);
          if (i + 2 < hi) f(i + 2, v[u].z);
          if (i + 3 < hi) f(i + 3, v[u].w);
        }
      }
      return;
    }
    float4 v = i0 < hi ? load(i0) : make_float4(0, 0, 0, 0);
#pragma unroll 1
    for (; i0 < hi; i0 += 128) {
      const float4 next = i0 + 128 < hi ? load(i0 + 128) : make_float4(0, 0, 0, 0);
      f(i0, v.x);
      if (i0 + 1 < hi) f(i0 + 1, v.y);
      if (i0 + 2 < hi) f(i0 + 2, v.z);
      if (i0 + 3 < hi) f(i0 + 3, v.w);
      v = next;
    }
  }
};

// Radix select over the ordered keys of the candidates of all CTAs: finds the largest key K with
// weight(keys >= K) >= target, 8 bits per pass. `weigh(l)` is 1 for top-k, the fixed-point mass for top-p.
template <typename W>
__device__ uint32_t radix_threshold(const RowPart& part, uint32_t floor_key, unsigned long long target, int cluster,
                                    SampleShared& sm, W weigh) {
  const int tid = threadIdx.x, lane = tid & 31;
  uint32_t prefix = 0u, mask = 0u;
  unsigned long long above = 0ull;
  for (int shift = 24; shift >= 0; shift -= 8) {
    for (int i = tid; i < 256 * kHistCopies; i += kSampleThreads) sm.hist.lo[i] = sm.hist.hi[i] = 0u;
    __syncthreads();
    part.each(lane, [&](int, float l) {
      const uint32_t key = order_key(l);
      if (key < floor_key || (key & mask) != prefix) return;
      const unsigned long long w = weigh(l);
      if (w == 0ull) return;
      const int at = int((key >> shift) & 255u) * kHistCopies + (lane & (kHistCopies - 1));
      // a 64-bit sum in two words: the thread whose addition wraps the low word carries into the high one
      const uint32_t add = uint32_t(w), old = atomicAdd(&sm.hist.lo[at], add);
      const uint32_t up = uint32_t(w >> 32) + (old + add < old ? 1u : 0u);
      if (up) atomicAdd(&sm.hist.hi[at], up);
    });
    // The copies meet in their own CTA first: a digit is then one word per CTA, neighbouring threads read neighbouring words of the
    // other CTAs (reading all copies there, eight words apart, took 140 us a pass for 16 clusters of eight).
    __syncthreads();
    if (tid < 256) {
      unsigned long long own = 0ull;
#pragma unroll
      for (int c = 0; c < kHistCopies; ++c)
        own += (static_cast<unsigned long long>(sm.hist.hi[tid * kHistCopies + c]) << 32) + sm.hist.lo[tid * kHistCopies + c];
      sm.own_digit[tid] = own;
    }
    cluster_barrier(cluster);
    if (tid < 256) {
      unsigned long long sum = 0ull;
      for (int r = 0; r < cluster; ++r) sum += of_rank(&sm, r)->own_digit[tid];
      sm.digit_sum[tid] = sum;
    }
    __syncthreads();
    if (tid < 32) {  // lane 0 holds the eight largest digits; the highest digit at which the running sum meets the target
      unsigned long long own = 0ull;
      for (int j = 0; j < 8; ++j) own += sm.digit_sum[255 - 8 * lane - j];
      unsigned long long incl = own;
      for (int o = 1; o < 32; o <<= 1) {
        const unsigned long long y = __shfl_up_sync(0xffffffffu, incl, o);
        if (lane >= o) incl += y;
      }
      const uint32_t meets = __ballot_sync(0xffffffffu, above + incl >= target);
      const int first = meets ? __ffs(int(meets)) - 1 : 31;  // none: digit 0
      if (lane == first) {
        unsigned long long cum = above + incl - own;
        int d = 255 - 8 * lane;
        for (const int end = max(d - 7, 1); d >= end; --d) {
          if (cum + sm.digit_sum[d] >= target) break;
          cum += sm.digit_sum[d];
        }
        sm.pick_prefix = prefix | (uint32_t(max(d, 0)) << shift);
        sm.pick_above = cum;
      }
    }
    cluster_barrier(cluster);  // the digits' sums have been read by everybody; the pick is visible in the CTA
    prefix = sm.pick_prefix;
    above = sm.pick_above;
    mask |= 255u << shift;
  }
  return prefix;
}

// The draw's point of the kept mass: an integer below `total` (which is not zero), a function of seed and step.
__device__ __forceinline__ unsigned long long draw_point(uint64_t seed, int step, unsigned long long total) {
  const uint64_t r = mix64(seed ^ (0xD1B54A32D192ED03ull * uint64_t(step + 1)));
  const double u01 = __dmul_rn(double(r >> 11), 1.0 / 9007199254740992.0);
  const unsigned long long u = (unsigned long long)__dmul_rn(u01, double(total));
  return u >= total ? total - 1ull : u;  // double(total) may round up beyond 2^53: the draw stays inside the kept mass
}

__global__ void __launch_bounds__(kSampleThreads, 2) sample_kernel(q38_sampling_args a, int cluster) {
  pdl_wait();               // everything written by earlier kernels of the stream is visible from here on
  pdl_launch_dependents();  // the next kernel may be scheduled now; it holds its own dependent work back the same way
  __shared__ SampleShared sm;
  const int b = blockIdx.x / cluster, rank = blockIdx.x % cluster;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const q38_sampling_params_dev prm = a.params[b];
  float* logits = a.logits + (size_t)b * a.ld;
  const int V = a.vocab;
  const int slot = a.row_slot ? a.row_slot[b] : b;

  auto commit = [&](int tok, float logprob) {
    a.tokens_out[b] = tok;
    if (a.logprob_out) a.logprob_out[b] = logprob;
    if (a.history) {
      const int len = a.history_len[slot];
      a.history[(size_t)slot * a.history_cap + (len % a.history_cap)] = tok;
      a.history_len[slot] = len + 1;
    }
  };
  auto log_share = [](unsigned long long mass, unsigned long long all) {
    const double p = double(mass) / double(all > 0 ? all : 1ull);
    return float(log(p > 0.0 ? p : 1e-300));
  };

  if ((prm.presence_penalty != 0.0f || prm.repetition_penalty != 1.0f) && a.history) {
    if (rank == 0) {
      for (int i = tid; i < (V + 31) / 32; i += kSampleThreads) sm.seen[i] = 0u;
      __syncthreads();
      const int n = min(a.history_len[slot], a.history_cap);
      const int32_t* hist = a.history + (size_t)slot * a.history_cap;
      for (int i = tid; i < n; i += kSampleThreads) {
        const int t = hist[i];
        if (t < 0 || t >= V) continue;
        const uint32_t bit = 1u << (t & 31);
        if (atomicOr(&sm.seen[t >> 5], bit) & bit) continue;
        float l = logits[t];
        if (prm.repetition_penalty != 1.0f)
          l = l > 0.0f ? __fdiv_rn(l, prm.repetition_penalty) : __fmul_rn(l, prm.repetition_penalty);
        logits[t] = __fsub_rn(l, prm.presence_penalty);  // explicit roundings: no multiply-subtract contraction
      }
    }
    cluster_barrier(cluster);
  }

  RowPart part;
  {
    const int parts = cluster * kSampleWarps, size = ((V + parts - 1) / parts + 127) / 128 * 128;
    part.row = logits;
    part.lo = min(V, (rank * kSampleWarps + warp) * size);
    part.hi = min(V, part.lo + size);
    part.vec = (reinterpret_cast<uintptr_t>(logits) & 15) == 0;
  }

  // maximum with the lowest index among ties (without an index where it is not asked for), the key of every thread's maximum (of
  // logits that are numbers: a lower bound of its largest key, which is all that the floor needs)
  const bool few = prm.temperature > 0.0f && prm.top_k > 0 && prm.top_k < V && prm.top_k <= kFastTopK;
  float best = -INFINITY;
  int best_i = 0x7fffffff;
  uint32_t top_key = 0u;
  auto keep_best = [&](int i, float l) {
    if (l > best) {
      best = l;
      best_i = i;
    }
  };
  if (few) {  // the maximum alone: one instruction per logit
    part.each(lane, [&](int, float l) { best = fmaxf(best, l); });
    if (best == 0.0f) {  // the first of its zeros decides the sign
      best = -INFINITY;
      part.each(lane, keep_best);
    }
    top_key = best > -INFINITY ? order_key(best) : 0u;
  } else {
    part.each<true>(lane, keep_best);
  }
  for (int o = 16; o > 0; o >>= 1) {
    const float ov = __shfl_xor_sync(0xffffffffu, best, o);
    const int oi = __shfl_xor_sync(0xffffffffu, best_i, o);
    if (ov > best || (ov == best && oi < best_i)) {
      best = ov;
      best_i = oi;
    }
  }
  if (lane == 0) {
    sm.warp_f[warp] = best;
    sm.warp_i[warp] = best_i;
  }
  uint32_t floor_key = 0u;
  if (few)  // the top_k-th largest of the threads' keys, rounded down to its upper 20 bits
    for (int bit = 31; bit >= 12; --bit) {
      const uint32_t cand = floor_key | (1u << bit);
      if (__syncthreads_count(top_key >= cand) >= prm.top_k) floor_key = cand;
    }
  __syncthreads();
  if (tid == 0) {
    for (int w = 1; w < kSampleWarps; ++w) {
      const float ov = sm.warp_f[w];
      const int oi = sm.warp_i[w];
      if (ov > best || (ov == best && oi < best_i)) {
        best = ov;
        best_i = oi;
      }
    }
    sm.cta_best = best;
    sm.cta_best_index = best_i;
    sm.cta_floor = floor_key;
    sm.own_count = 0;
  }
  cluster_barrier(cluster);
  best = -INFINITY;
  best_i = 0x7fffffff;
  for (int r = 0; r < cluster; ++r) {
    const SampleShared* other = of_rank(&sm, r);
    const float ov = other->cta_best;
    const int oi = other->cta_best_index;
    if (ov > best || (ov == best && oi < best_i)) {
      best = ov;
      best_i = oi;
    }
    floor_key = max(floor_key, other->cta_floor);
  }
  if (prm.temperature <= 0.0f) {
    if (rank == 0 && tid == 0) commit(best_i < V ? best_i : 0, 0.0f);
    cluster_barrier(cluster);  // no CTA leaves while its shared memory is being read
    return;
  }
  const float M = best;
  const float inv_t = __fdiv_rn(1.0f, prm.temperature);
  auto mass = [&](float l) -> unsigned long long { return fixed_mass(l, M, inv_t); };
  // A row whose kept logits are all NaN or -inf takes its maximum, one without a number above -inf token 0. Called by one warp, so
  // seldom that the index is looked up here (not all ways to M keep it).
  auto commit_best = [&](unsigned long long all) {
    int first = V;
    for (int i = lane; i < V && first == V && M > -INFINITY; i += 32)
      if (logits[i] == M) first = i;
    first = __reduce_min_sync(0xffffffffu, first);
    if (lane == 0) commit(first < V ? first : 0, log_share(all > 0ull ? 1ull << 40 : 0ull, all));
  };
  const int step = a.step ? a.step[b] : 0;

  if (few) {
    unsigned long long sum = 0ull;
    const float floor_l = key_to_float(floor_key);
    part.each(lane, [&](int i, float l) {
      sum += mass(l);
      if (l < floor_l) return;  // (a NaN goes on: its key decides)
      const uint32_t key = order_key(l);
      if (key >= floor_key) {
        const int at = atomicAdd(&sm.own_count, 1);
        if (at < kOwnList) {
          sm.own_key[at] = key;
          sm.own_index[at] = i;
        }
      }
    });
    sum = warp_sum_u64(sum);
    if (lane == 0) sm.warp_u64[0][warp] = sum;
    __syncthreads();
    if (tid == 0) {
      unsigned long long total = 0ull;
      for (int w = 0; w < kSampleWarps; ++w) total += sm.warp_u64[0][w];
      sm.cta_all = total;
    }
    cluster_barrier(cluster);
    int n = 0;
    bool fits = true;
    unsigned long long all_sum = 0ull;
    for (int r = 0; r < cluster; ++r) {
      const SampleShared* other = of_rank(&sm, r);
      n += other->own_count;
      fits = fits && other->own_count <= kOwnList;
      all_sum += other->cta_all;
    }
    if (fits && n <= kAllList) {
      if (rank == 0) {
        for (int r = 0, at = 0; r < cluster; ++r) {
          const SampleShared* other = of_rank(&sm, r);
          const int count = other->own_count;
          for (int i = tid; i < count; i += kSampleThreads) {
            const uint32_t key = other->own_key[i];
            sm.all.key[at + i] = key;
            sm.all.index[at + i] = other->own_index[i];
            sm.all.mass[at + i] = mass(key_to_float(key));
          }
          at += count;
        }
        if (tid == 0) sm.pick_key = 0u;
        __syncthreads();
        // top-k: the key with fewer than top_k keys above it and at least top_k not below it
        for (int i = tid; i < n; i += kSampleThreads) {
          const uint32_t key = sm.all.key[i];
          int more = 0, same = 0;
          for (int j = 0; j < n; ++j) {
            more += sm.all.key[j] > key ? 1 : 0;
            same += sm.all.key[j] == key ? 1 : 0;
          }
          if (more < prm.top_k && more + same >= prm.top_k) sm.pick_key = key;
        }
        __syncthreads();
        uint32_t thresh = sm.pick_key;
        if (prm.min_p > 0.0f) thresh = max(thresh, min_p_key(M, inv_t, prm.min_p));
        unsigned long long kept = 0ull;
        for (int j = 0; j < n; ++j)
          if (sm.all.key[j] >= thresh) kept += sm.all.mass[j];
        __syncthreads();
        if (tid == 0) sm.pick_key = 0u;
        __syncthreads();
        if (prm.top_p < 1.0f) {  // the largest key at which the mass of the keys not below it reaches the target
          const unsigned long long part_of = (unsigned long long)__dmul_rn(double(prm.top_p), double(kept));
          const unsigned long long target = part_of > 0 ? part_of : 1ull;
          for (int i = tid; i < n; i += kSampleThreads) {
            const uint32_t key = sm.all.key[i];
            if (key < thresh) continue;
            unsigned long long from = 0ull;
            for (int j = 0; j < n; ++j)
              if (sm.all.key[j] >= key) from += sm.all.mass[j];
            if (from >= target) atomicMax(&sm.pick_key, key);
          }
          __syncthreads();
          thresh = max(thresh, sm.pick_key);
          kept = 0ull;
          for (int j = 0; j < n; ++j)
            if (sm.all.key[j] >= thresh) kept += sm.all.mass[j];
        }
        if (kept > 0ull) {  // inverse CDF in index order
          const unsigned long long u = draw_point(prm.seed, step, kept);
          for (int i = tid; i < n; i += kSampleThreads) {
            if (sm.all.key[i] < thresh) continue;
            const int index = sm.all.index[i];
            unsigned long long before = 0ull;
            for (int j = 0; j < n; ++j)
              if (sm.all.key[j] >= thresh && sm.all.index[j] < index) before += sm.all.mass[j];
            if (u >= before && u < before + sm.all.mass[i]) commit(index, log_share(sm.all.mass[i], all_sum));
          }
        } else if (warp == 0) {
          commit_best(all_sum);
        }
      }
      cluster_barrier(cluster);
      return;
    }
    cluster_barrier(cluster);  // the counts have been read; the lists' memory becomes the histogram
  }

  // the general path: thresholds by radix selection over the whole row
  uint32_t thresh = 0u;
  if (prm.top_k > 0 && prm.top_k < V)
    thresh = radix_threshold(part, 0u, (unsigned long long)prm.top_k, cluster, sm, [](float) { return 1ull; });
  if (prm.min_p > 0.0f) thresh = max(thresh, min_p_key(M, inv_t, prm.min_p));
  // masses of the warps' parts: kept ones, all of them
  auto sums = [&](unsigned long long& kept, unsigned long long& all_sum) {
    unsigned long long own = 0ull, all = 0ull;
    part.each(lane, [&](int, float l) {
      const unsigned long long w = mass(l);
      all += w;
      if (order_key(l) >= thresh) own += w;
    });
    own = warp_sum_u64(own);
    all = warp_sum_u64(all);
    if (lane == 0) {
      sm.warp_u64[0][warp] = own;
      sm.warp_u64[1][warp] = all;
    }
    __syncthreads();
    if (tid == 0) {
      unsigned long long k = 0ull, t = 0ull;
      for (int w = 0; w < kSampleWarps; ++w) {
        k += sm.warp_u64[0][w];
        t += sm.warp_u64[1][w];
      }
      sm.cta_kept = k;
      sm.cta_all = t;
    }
    cluster_barrier(cluster);
    kept = all_sum = 0ull;
    for (int r = 0; r < cluster; ++r) {
      kept += of_rank(&sm, r)->cta_kept;
      all_sum += of_rank(&sm, r)->cta_all;
    }
  };
  unsigned long long kept, all_sum;
  sums(kept, all_sum);
  if (prm.top_p < 1.0f) {
    const unsigned long long target = (unsigned long long)__dmul_rn(double(prm.top_p), double(kept));
    // (its first barrier also lets everybody read the sums before the next ones)
    thresh = max(thresh, radix_threshold(part, thresh, target > 0 ? target : 1ull, cluster, sm, mass));
    sums(kept, all_sum);
  }

  // inverse CDF in index order: the parts follow one another by rank and warp; one warp holds the drawn point
  if (kept > 0ull) {
    const unsigned long long u = draw_point(prm.seed, step, kept);
    unsigned long long cum = 0ull;
    for (int r = 0; r < rank; ++r) cum += of_rank(&sm, r)->cta_kept;
    for (int w = 0; w < warp; ++w) cum += sm.warp_u64[0][w];
    if (u >= cum && u < cum + sm.warp_u64[0][warp]) {
      for (int i0 = part.lo; i0 < part.hi; i0 += 128) {
        const int i = i0 + 4 * lane;
        const float4 v = part.load(i);
        const float l[4] = {v.x, v.y, v.z, v.w};
        unsigned long long w[4], own = 0ull;
#pragma unroll
        for (int e = 0; e < 4; ++e) {
          w[e] = i + e < part.hi && order_key(l[e]) >= thresh ? mass(l[e]) : 0ull;
          own += w[e];
        }
        unsigned long long incl = own;
        for (int o = 1; o < 32; o <<= 1) {
          const unsigned long long y = __shfl_up_sync(0xffffffffu, incl, o);
          if (lane >= o) incl += y;
        }
        const unsigned long long end = cum + __shfl_sync(0xffffffffu, incl, 31);
        if (u < end) {
          unsigned long long at = cum + incl - own;
          if (u >= at && u < at + own) {
            int e = 0;
            while (e < 3 && u >= at + w[e]) at += w[e++];
            commit(i + e, log_share(w[e], all_sum));
          }
          break;
        }
        cum = end;
      }
    }
  } else if (rank == 0 && warp == 0) {
    commit_best(all_sum);
  }
  cluster_barrier(cluster);  // no CTA leaves while its shared memory is being read
}

// out[r] = log softmax(logits[r])[targets[r]], sums in double
// (reference src/kernels/kernels.h:258-260, src/kernels/sampling.cu:312-339).
__global__ void __launch_bounds__(256) target_logprob_kernel(const float* __restrict__ logits, int ld, int vocab,
                                                             const int32_t* __restrict__ targets,
                                                             float* __restrict__ out) {
  pdl_wait();               // everything written by earlier kernels of the stream is visible from here on
  pdl_launch_dependents();  // the next kernel may be scheduled now; it holds its own dependent work back the same way
  __shared__ float red_f[8];
  __shared__ double red_d[8];
  const int r = blockIdx.x, tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const float* row = logits + (size_t)r * ld;
  float mx = -INFINITY;
  for (int i = tid; i < vocab; i += 256) mx = fmaxf(mx, row[i]);
  mx = warp_max(mx);
  if (lane == 0) red_f[warp] = mx;
  __syncthreads();
  mx = red_f[0];
  for (int w = 1; w < 8; ++w) mx = fmaxf(mx, red_f[w]);
  double sum = 0.0;
  for (int i = tid; i < vocab; i += 256) sum += exp(double(row[i] - mx));
  for (int o = 16; o > 0; o >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, o);
  if (lane == 0) red_d[warp] = sum;
  __syncthreads();
  if (tid == 0) {
    double total = 0.0;
    for (int w = 0; w < 8; ++w) total += red_d[w];
    const int t = targets[r];
    out[r] = (t >= 0 && t < vocab) ? float(double(row[t] - mx) - log(total)) : 0.0f;
  }
}

}  // namespace

Q38_REGISTER_ERROR_WORD();
unsigned int* misc_error_address() { return tu_error_address(); }

}  // namespace q38

namespace q38 {
namespace {
// Rows `rows[i]` of the step's normalised-input arrays (bf16 hidden row + its norm partial sums) packed into
// rows i = 0..n-1: the LM-head input of the sequences that sample in a ragged step.
__global__ void __launch_bounds__(256) gather_rows_kernel(const __nv_bfloat16* __restrict__ x,
                                                          const float* __restrict__ partials,
                                                          const int* __restrict__ rows, int hidden, int blocks,
                                                          __nv_bfloat16* __restrict__ x_out,
                                                          float* __restrict__ partials_out) {
  pdl_wait();
  pdl_launch_dependents();
  const int i = blockIdx.x, src = rows[i];
  const uint4* from = reinterpret_cast<const uint4*>(x + (size_t)src * hidden);
  uint4* to = reinterpret_cast<uint4*>(x_out + (size_t)i * hidden);
  for (int c = threadIdx.x; c < hidden / 8; c += blockDim.x) to[c] = from[c];
  for (int c = threadIdx.x; c < blocks; c += blockDim.x) partials_out[(size_t)i * blocks + c] = partials[(size_t)src * blocks + c];
}
}  // namespace
}  // namespace q38

using namespace q38;

extern "C" int q38_gather_rows(const q38_bf16* x, const float* partials, const int* rows, int n, int hidden,
                               q38_bf16* x_out, float* partials_out, void* stream) {
  if (n == 0) return Q38_OK;
  Q38_REQUIRE(x && partials && rows && x_out && partials_out, "gather_rows: null argument");
  Q38_REQUIRE(n > 0 && hidden > 0 && hidden % 128 == 0, "gather_rows: n %d hidden %d", n, hidden);
  (void)launch_kernel(gather_rows_kernel, dim3(n), dim3(256), 0, as_stream(stream),
                      reinterpret_cast<const __nv_bfloat16*>(x), partials, rows, hidden, hidden / 128,
                      reinterpret_cast<__nv_bfloat16*>(x_out), partials_out);
  Q38_LAUNCH_OK("gather_rows_kernel");
  return Q38_OK;
}

extern "C" int q38_embed(const q38_bf16* table, const int32_t* tokens, int m, int hidden, float* residual,
                         q38_bf16* xbf, float* partials, void* stream) {
  if (m == 0) return Q38_OK;
  Q38_REQUIRE(table && tokens && residual && xbf && partials, "embed: null argument");
  Q38_REQUIRE(m > 0 && hidden > 0 && hidden % 128 == 0, "embed: m %d hidden %d", m, hidden);
  (void)launch_kernel(embed_kernel, dim3(m), dim3(256), 0, as_stream(stream), reinterpret_cast<const __nv_bfloat16*>(table), tokens, hidden,
                                                 residual, reinterpret_cast<__nv_bfloat16*>(xbf), partials);
  Q38_LAUNCH_OK("embed_kernel");
  return Q38_OK;
}

extern "C" int q38_residual_update(const float* delta, int m, int hidden, float* residual, q38_bf16* xbf,
                                   float* partials, void* stream) {
  if (m == 0) return Q38_OK;
  Q38_REQUIRE(delta && residual && xbf && partials, "residual_update: null argument");
  Q38_REQUIRE(m > 0 && hidden > 0 && hidden % 128 == 0, "residual_update: m %d hidden %d", m, hidden);
  (void)launch_kernel(residual_update_kernel, dim3(m), dim3(256), 0, as_stream(stream), delta, hidden, residual,
                      reinterpret_cast<__nv_bfloat16*>(xbf), partials);
  Q38_LAUNCH_OK("residual_update_kernel");
  return Q38_OK;
}

extern "C" int q38_pack_ragged(const int* seq_count, const int* seq_pos0, int num_seqs, int num_tokens,
                               int* seq_start, int* tok_pos, int* tok_seq, void* stream) {
  if (num_seqs == 0) return Q38_OK;
  Q38_REQUIRE(seq_count && seq_pos0 && seq_start && tok_pos && tok_seq, "pack_ragged: null argument");
  Q38_REQUIRE(num_seqs > 0 && num_tokens >= 0, "pack_ragged: sizes");
  (void)launch_kernel(pack_ragged_kernel, dim3(1), dim3(1024), 0, as_stream(stream), seq_count, seq_pos0, num_seqs, num_tokens, seq_start,
                                                        tok_pos, tok_seq);
  Q38_LAUNCH_OK("pack_ragged_kernel");
  return Q38_OK;
}

extern "C" int q38_sample(const q38_sampling_args* a, int batch, void* stream) {
  Q38_REQUIRE(a, "sample: null argument");
  Q38_REQUIRE(a->vocab > 0 && a->vocab <= 256 * 1024, "sample: vocab size %d", a->vocab);
  if (batch == 0) return Q38_OK;
  Q38_REQUIRE(a->logits && a->params && a->tokens_out, "sample: null pointer");
  // Two CTAs fit an SM: the largest cluster with which all rows still run at once, and not so many CTAs that a warp's
  // part of a small vocabulary is below one step of 128 logits.
  // More rows than SMs and long ones: halves of rows where they share the SMs out more evenly (200 rows on 148 SMs: two rows or
  // three halves on the busiest; 248,320 logits without a filter 320 and 257 us, 512 rows 577 and 482; 512 short rows, 32,000
  // logits with the default sampling: 64 and 81 us).
  int cluster = 8;
  const int sms = num_sms();
  while (cluster > 1 && (batch * cluster > 2 * sms || a->vocab < cluster * kSampleWarps * 128)) cluster /= 2;
  if (cluster == 1 && a->vocab >= 128 * 1024 && (2 * batch + sms - 1) / sms < 2 * ((batch + sms - 1) / sms)) cluster = 2;
  (void)launch_cluster_kernel(sample_kernel, dim3(unsigned(batch * cluster)), dim3(kSampleThreads), cluster, size_t(0), as_stream(stream), *a,
                              cluster);
  Q38_LAUNCH_OK("sample_kernel");
  return Q38_OK;
}

extern "C" int q38_target_logprobs(const float* logits, int ld, int vocab, const int32_t* targets, int rows,
                                   float* out, void* stream) {
  if (rows == 0) return Q38_OK;
  Q38_REQUIRE(logits && targets && out && vocab > 0, "target_logprobs: arguments");
  (void)launch_kernel(target_logprob_kernel, dim3(rows), dim3(256), 0, as_stream(stream), logits, ld, vocab, targets, out);
  Q38_LAUNCH_OK("target_logprob_kernel");
  return Q38_OK;
}
