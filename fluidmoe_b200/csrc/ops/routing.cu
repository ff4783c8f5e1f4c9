// Router kernels: top-k + softmax, the padded-capacity plan and the dropless plan.  All three turn
// [T, E] logits or [T, k] choices into a few small arrays; they sit between two GEMMs of every MoE
// layer with nothing to overlap, so what counts is their latency, not their bandwidth.
#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <math.h>
#include <stdint.h>
#include <stdio.h>

#include "../include/fm_ops.h"
#include "router_wgrad.h"

extern "C" void fm_set_error(const char* msg);

namespace fm {

// --------------------------------------------------------------------------------------------
// Top-k over experts, then softmax over the k winners (fp32).  Ties go to the lower expert index.
// One warp per token, NV logits per lane (E <= 32 * NV) in registers; a round is one warp maximum of
// the order-preserving integer image of the logits and one warp minimum of the indices that hold it.
// One thread per token (below) reads its row k times with a stride of E floats between lanes.
// 8192 tokens, 64 experts, k = 8: 82 us -> 4.6 us; 4096 tokens, 8 experts, k = 2: 5.0 us -> 3.2 us.
// --------------------------------------------------------------------------------------------
template <int NV>
__global__ void __launch_bounds__(256)
topk_softmax_warp_kernel(const float* __restrict__ logits, long long* __restrict__ idx_out,
                         float* __restrict__ prob_out, int T, int E, int k) {
  const int lane = threadIdx.x & 31;
  const int t = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
  if (t >= T) return;                       // whole warps leave together
  const float* l = logits + (long long)t * E;
  uint32_t key[NV];
  bool nan = false;
#pragma unroll
  for (int q = 0; q < NV; ++q) {
    const int e = q * 32 + lane;
    key[q] = 0;                             // below every number: not a candidate
    if (e < E) {
      const float v = l[e];
      nan |= isnan(v);
      const uint32_t b = __float_as_uint(v + 0.0f);     // -0 and +0 tie
      key[q] = (b & 0x80000000u) ? ~b : (b | 0x80000000u);
    }
  }
  long long* io = idx_out + (long long)t * k;
  float* po = prob_out + (long long)t * k;
  if (__any_sync(0xffffffffu, nan)) {
    // Comparisons with NaN are false, so the serial rule depends on where it stands: a NaN is taken
    // exactly when it is the first candidate left.  Rare; one lane applies the rule as it is.
    if (lane == 0) {
      float vals[16];
      int ids[16];
      for (int j = 0; j < k; ++j) {
        float best = -INFINITY;
        int bi = -1;
        for (int e = 0; e < E; ++e) {
          bool taken = false;
          for (int q = 0; q < j; ++q) taken |= (ids[q] == e);
          if (!taken && (l[e] > best || bi < 0)) {
            best = l[e];
            bi = e;
          }
        }
        vals[j] = best;
        ids[j] = bi;
      }
      float s = 0.f;
      for (int j = 0; j < k; ++j) s += __expf(vals[j] - vals[0]);
      for (int j = 0; j < k; ++j) {
        io[j] = ids[j];
        po[j] = __expf(vals[j] - vals[0]) / s;
      }
    }
    return;
  }
  float m = 0.f, s = 0.f, mine = 0.f;
  int my_id = 0;
  for (int j = 0; j < k; ++j) {
    uint32_t best = key[0];
#pragma unroll
    for (int q = 1; q < NV; ++q) best = max(best, key[q]);
    best = __reduce_max_sync(0xffffffffu, best);
    uint32_t at = 0xffffffffu;
#pragma unroll
    for (int q = NV - 1; q >= 0; --q)
      if (key[q] == best) at = q * 32 + lane;
    at = __reduce_min_sync(0xffffffffu, at);
#pragma unroll
    for (int q = 0; q < NV; ++q)
      if (at == (uint32_t)(q * 32 + lane)) key[q] = 0;
    const float v = __uint_as_float((best & 0x80000000u) ? (best & 0x7fffffffu) : ~best);
    if (j == 0) m = v;
    const float ex = __expf(v - m);
    s += ex;
    if (lane == j) {
      mine = ex;
      my_id = (int)at;
    }
  }
  if (lane < k) {
    io[lane] = my_id;
    po[lane] = mine / s;
  }
}

// One thread per token: more than 256 experts, or so many tokens with so few experts that a warp each is the
// longer way (see fm_topk_softmax).
__global__ void topk_softmax_kernel(const float* __restrict__ logits, long long* __restrict__ idx_out,
                                    float* __restrict__ prob_out, int T, int E, int k) {
  const int t = blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= T) return;
  const float* l = logits + (long long)t * E;
  float vals[16];
  int ids[16];
  for (int j = 0; j < k; ++j) {
    float best = -INFINITY;
    int bi = -1;
    for (int e = 0; e < E; ++e) {
      const float v = l[e];
      bool taken = false;
      for (int q = 0; q < j; ++q) taken |= (ids[q] == e);
      if (!taken && (v > best || bi < 0)) {
        best = v;
        bi = e;
      }
    }
    vals[j] = best;
    ids[j] = bi;
  }
  float m = vals[0], s = 0.f;
  for (int j = 0; j < k; ++j) s += __expf(vals[j] - m);
  for (int j = 0; j < k; ++j) {
    idx_out[(long long)t * k + j] = ids[j];
    prob_out[(long long)t * k + j] = __expf(vals[j] - m) / s;
  }
}

constexpr int kPlanThreads = 1024;
constexpr int kPlanWarps = kPlanThreads / 32;
constexpr int kPlanFewThreads = 128, kPlanFewTokens = 512;   // up to so many tokens, so many threads

// Exclusive prefix of `v` over the CTA and the total; `smem` holds kWarps values.
template <class V, int kWarps = kPlanWarps>
__device__ __forceinline__ V block_excl_scan(V v, V* total, V* smem) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  V x = v;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const V y = __shfl_up_sync(0xffffffffu, x, o);
    if (lane >= o) x += y;
  }
  __syncthreads();
  if (lane == 31) smem[warp] = x;
  __syncthreads();
  if (warp == 0) {
    V w = lane < kWarps ? smem[lane] : V(0);
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const V y = __shfl_up_sync(0xffffffffu, w, o);
      if (lane >= o) w += y;
    }
    if (lane < kWarps) smem[lane] = w;   // inclusive warp totals
  }
  __syncthreads();
  const V base = warp == 0 ? V(0) : smem[warp - 1];
  *total = smem[kWarps - 1];
  return base + x - v;
}

// --------------------------------------------------------------------------------------------
// Routing plan for fixed (padded) capacity.  One CTA per expert:
//   1. collect the tokens routed to the expert (their probability and which choice they are) in
//      shared memory, one pass over the choices;
//   2. if there are more than `cap`, find the cap-th largest probability, four bits of it at a time
//      (probabilities are not negative, so the unsigned order of the bits is the numeric order), and
//      keep ties in ascending token order;
//   3. assign slots: kept tokens, plus the first (cap - kept) tokens that are NOT routed to this
//      expert as padding (probability 0), all in ascending token order.  A thread owns consecutive
//      tokens, so that two scans over the CTA order all of them.
// Outputs have static shapes; nothing is read back by the host.  Bound by latency (one pass
// over T * k choices, about 20 CTA barriers): reading the choices again for every pass of the select and
// scanning 512 tokens at a time took 57 us at 4096 tokens, 8 experts, k = 2 and 180 us at 8192 tokens, 64
// experts, k = 8; this form takes 23 and 30.
// --------------------------------------------------------------------------------------------
// Tokens of one CTA's row lie 32 to a line of 33 words: threads that own 8 (16, ...) consecutive tokens
// each would otherwise meet in the same banks.
__host__ __device__ __forceinline__ int plan_pos(int t) { return t + (t >> 5); }
constexpr int kPlanLoads = 8;      // choices a thread has in flight while it collects
constexpr int kPlanSmemMax = 200 * 1024;
__host__ __device__ __forceinline__ size_t plan_smem_bytes(int T) { return (size_t)(plan_pos(T) + 1) * 5 + 16; }

// A row of few tokens takes few threads, since it waits for little but the barriers: 1024 and 128 threads, us: 64 tokens, 8
// experts, 13.1 and 8.4; 256 11.0 and 7.9; 512 11.0 and 9.0, with 64 experts and k = 8 13.1 and 12.5.
template <int kThreads>
__global__ void __launch_bounds__(kThreads)
moe_plan_kernel(const long long* __restrict__ top_idx, const float* __restrict__ top_probs, int T,
                int k, int E, int cap, long long* __restrict__ sorted_indices,
                float* __restrict__ slot_probs, int* __restrict__ slot_of_token,
                int* __restrict__ routed_per_expert, int* __restrict__ tokens_per_expert) {
  constexpr int kWarps = kThreads / 32;
  extern __shared__ uint32_t bits_s[];                       // [plan_pos(T) + 1] probability bits
  uint8_t* const choice_s = reinterpret_cast<uint8_t*>(bits_s + plan_pos(T) + 1);   // 255: not routed here
  __shared__ unsigned long long scan_s[kWarps];
  __shared__ uint32_t digit_s[2][kWarps][9];             // rows of 9: lane l reads row l without conflicts
  const int e = blockIdx.x;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;

  // ---- 1. collect ----
  for (int i = tid; i < plan_pos(T) + 1; i += kThreads) choice_s[i] = 255;
  __syncthreads();
  // Index and probability are loaded together: a probability fetched only for a hit would put one
  // memory latency after another, since nearly every warp has a hit in every step.
  const int n = T * k;
  int hits = 0;
  for (int i0 = tid; i0 < n; i0 += kThreads * kPlanLoads) {
    int ex[kPlanLoads];
    float pr[kPlanLoads];
#pragma unroll
    for (int q = 0; q < kPlanLoads; ++q) {
      const int i = min(i0 + q * kThreads, n - 1);
      ex[q] = (int)top_idx[i];
      pr[q] = top_probs[i];
    }
#pragma unroll
    for (int q = 0; q < kPlanLoads; ++q) {
      const int i = i0 + q * kThreads;
      if (i < n && ex[q] == e) {
        const int t = (int)((unsigned)i / (unsigned)k);
        choice_s[plan_pos(t)] = (uint8_t)(i - t * k);
        bits_s[plan_pos(t)] = __float_as_uint(pr[q]);
        ++hits;
      }
    }
  }
  __syncthreads();
  const int per = (T + kThreads - 1) / kThreads;
  const int lo = min(T, tid * per), hi = min(T, lo + per);

  // tokens of this expert
  int count = 0;
  for (int t = lo; t < hi; ++t) count += choice_s[plan_pos(t)] != 255 ? 1 : 0;
  count = __reduce_add_sync(0xffffffffu, count);
  hits = __reduce_add_sync(0xffffffffu, hits);
  if (lane == 0) {
    digit_s[0][warp][0] = count;
    digit_s[0][warp][1] = hits;
  }
  __syncthreads();
  count = __reduce_add_sync(0xffffffffu, lane < kWarps ? digit_s[0][lane][0] : 0u);
  if ((int)__reduce_add_sync(0xffffffffu, lane < kWarps ? digit_s[0][lane][1] : 0u) != count) {
    // Some token names this expert twice (a replayed routing may): its first choice counts, and the
    // pass above kept either.  The others have no slot.
    for (int t = lo; t < hi; ++t) {
      if (choice_s[plan_pos(t)] == 255) continue;
      int j = 0;
      while ((int)top_idx[(long long)t * k + j] != e) ++j;
      choice_s[plan_pos(t)] = (uint8_t)j;
      bits_s[plan_pos(t)] = __float_as_uint(top_probs[(long long)t * k + j]);
      for (++j; j < k; ++j)
        if ((int)top_idx[(long long)t * k + j] == e) slot_of_token[(long long)t * k + j] = -1;
    }
  }
  const int kept_total = min(count, cap);

  // ---- 2. threshold (only when tokens must be dropped) ----
  uint32_t thr = 0;      // keep bits > thr, plus `quota` tokens with bits == thr
  int quota = 0;
  const bool drop = count > cap;
  if (drop) {
    int want = cap;      // rank, from the top, of the threshold among the tokens that share its prefix
    uint32_t mask = 0;
    for (int shift = 28; shift >= 0; shift -= 4) {
      // this thread's tokens by digit: sixteen counters of 8 bits (a thread owns at most 39 tokens)
      unsigned long long c0 = 0, c1 = 0;
      for (int t = lo; t < hi; ++t) {
        const uint32_t b = bits_s[plan_pos(t)];
        if (choice_s[plan_pos(t)] != 255 && (b & mask) == thr) {
          const int d = (b >> shift) & 15;
          const unsigned long long one = 1ull << ((d & 7) * 8);
          if (d < 8) c0 += one;
          else c1 += one;
        }
      }
      // widened to 16 bits (fewer than 65536 tokens): word 4h + 2o + w counts digits 8h + 4w + o and the next but one
      uint32_t w[8];
#pragma unroll
      for (int h = 0; h < 2; ++h)
#pragma unroll
        for (int o = 0; o < 2; ++o) {
          const unsigned long long x = ((h ? c1 : c0) >> (8 * o)) & 0x00ff00ff00ff00ffull;
          w[4 * h + 2 * o] = (uint32_t)x;
          w[4 * h + 2 * o + 1] = (uint32_t)(x >> 32);
        }
#pragma unroll
      for (int i = 0; i < 8; ++i) w[i] = __reduce_add_sync(0xffffffffu, w[i]);
      const int buf = (shift >> 2) & 1;      // two buffers: one barrier a round (the count above used buffer 0)
      if (lane == 0) {
#pragma unroll
        for (int i = 0; i < 8; ++i) digit_s[buf][warp][i] = w[i];
      }
      __syncthreads();
#pragma unroll
      for (int i = 0; i < 8; ++i) w[i] = __reduce_add_sync(0xffffffffu, lane < kWarps ? digit_s[buf][lane][i] : 0u);
      int digit = 0, in_digit = 0;
      bool found = false;
#pragma unroll
      for (int d = 15; d >= 0; --d) {
        const int c = (w[4 * (d >> 3) + 2 * (d & 1) + ((d >> 2) & 1)] >> (16 * ((d >> 1) & 1))) & 0xffff;
        if (!found) {
          if (c >= want) {
            found = true;
            digit = d;
            in_digit = c;
          } else {
            want -= c;
          }
        }
      }
      thr |= (uint32_t)digit << shift;
      mask |= 15u << shift;
      if (in_digit == want) break;      // every token with this prefix stays
    }
    quota = want;
  }

  // ---- 3. ordered slot assignment ----
  int ties = 0, unrouted = 0;
  for (int t = lo; t < hi; ++t) {
    const bool routed = choice_s[plan_pos(t)] != 255;
    ties += (drop && routed && bits_s[plan_pos(t)] == thr) ? 1 : 0;
    unrouted += routed ? 0 : 1;
  }
  unsigned long long total;
  const unsigned long long before =
      block_excl_scan<unsigned long long, kWarps>(((unsigned long long)ties << 32) | (unsigned)unrouted, &total, scan_s);
  const int ties0 = (int)(before >> 32), unrouted0 = (int)(before & 0xffffffffu);
  const int pad_budget = cap - kept_total;
  auto walk = [&](auto&& visit) {
    int tr = ties0, ur = unrouted0;
    for (int t = lo; t < hi; ++t) {
      const bool routed = choice_s[plan_pos(t)] != 255;
      const uint32_t b = bits_s[plan_pos(t)];
      bool kept = false, pad = false;
      if (routed) {
        if (!drop || b > thr) kept = true;
        else if (b == thr) kept = tr++ < quota;
      } else {
        pad = ur++ < pad_budget;
      }
      visit(t, routed, kept, pad, b);
    }
  };
  int selected = 0;
  walk([&](int, bool, bool kept, bool pad, uint32_t) { selected += (kept || pad) ? 1 : 0; });
  int pos = (int)block_excl_scan<unsigned long long, kWarps>((unsigned long long)selected, &total, scan_s);
  walk([&](int t, bool routed, bool kept, bool pad, uint32_t b) {
    if ((kept || pad) && pos < cap) {
      const long long slot = (long long)e * cap + pos;
      sorted_indices[slot] = t;
      slot_probs[slot] = kept ? __uint_as_float(b) : 0.f;
      if (kept) slot_of_token[(long long)t * k + choice_s[plan_pos(t)]] = (int)slot;
      ++pos;
    }
    if (routed && !kept) slot_of_token[(long long)t * k + choice_s[plan_pos(t)]] = -1;
  });
  if (tid == 0) {
    routed_per_expert[e] = kept_total;
    if (tokens_per_expert != nullptr) tokens_per_expert[e] = cap;
  }
}

// Token counts whose row does not fit in shared memory (more than about 40 thousand): the choices are
// read again for every pass, the select counts with shared-memory atomics, and the slots are assigned
// kPlanThreads tokens at a time.
__global__ void __launch_bounds__(kPlanThreads)
moe_plan_large_kernel(const long long* __restrict__ top_idx, const float* __restrict__ top_probs, int T,
                      int k, int E, int cap, long long* __restrict__ sorted_indices,
                      float* __restrict__ slot_probs, int* __restrict__ slot_of_token,
                      int* __restrict__ routed_per_expert, int* __restrict__ tokens_per_expert) {
  __shared__ int hist[256];
  __shared__ int scan_s[kPlanWarps];
  __shared__ int sh_count, sh_prefix, sh_quota;
  const int e = blockIdx.x;
  const int tid = threadIdx.x;

  auto lookup = [&](int t, int& j_out) -> float {
    for (int j = 0; j < k; ++j)
      if ((int)top_idx[(long long)t * k + j] == e) {
        j_out = j;
        return top_probs[(long long)t * k + j];
      }
    j_out = -1;
    return 0.f;
  };

  // ---- 1. count ----
  if (tid == 0) sh_count = 0;
  __syncthreads();
  int local = 0;
  for (int t = tid; t < T; t += kPlanThreads) {
    int j;
    lookup(t, j);
    local += j >= 0;
  }
  atomicAdd(&sh_count, local);
  __syncthreads();
  const int count = sh_count;
  const int kept_total = min(count, cap);

  // ---- 2. threshold by radix select (only when tokens must be dropped) ----
  uint32_t thr_bits = 0;   // keep prob > thr, plus `quota` tokens with prob == thr
  int quota = 0;
  if (count > cap) {
    uint32_t prefix = 0, mask = 0;
    int want = cap;  // rank (1-based, from the top) of the threshold element
    for (int shift = 24; shift >= 0; shift -= 8) {
      for (int i = tid; i < 256; i += kPlanThreads) hist[i] = 0;
      __syncthreads();
      for (int t = tid; t < T; t += kPlanThreads) {
        int j;
        const float pr = lookup(t, j);
        if (j < 0) continue;
        const uint32_t b = __float_as_uint(pr);
        if ((b & mask) == prefix) atomicAdd(&hist[(b >> shift) & 255], 1);
      }
      __syncthreads();
      if (tid == 0) {
        int acc = 0, bin = 255;
        for (; bin >= 0; --bin) {
          if (acc + hist[bin] >= want) break;
          acc += hist[bin];
        }
        sh_prefix = bin;
        sh_quota = want - acc;  // rank of the threshold inside the chosen bin
      }
      __syncthreads();
      prefix |= (uint32_t)sh_prefix << shift;
      mask |= 255u << shift;
      want = sh_quota;
      __syncthreads();
    }
    thr_bits = prefix;
    quota = want;  // number of elements equal to the threshold that are kept
  }

  // ---- 3. ordered slot assignment ----
  int ties_seen = 0, sel_seen = 0, nonrouted_seen = 0;
  const int pad_budget = cap - kept_total;
  for (int t0 = 0; t0 < T; t0 += kPlanThreads) {
    const int t = t0 + tid;
    int j = -1;
    float pr = 0.f;
    bool valid = t < T;
    if (valid) pr = lookup(t, j);
    const bool routed = valid && j >= 0;
    const uint32_t b = __float_as_uint(pr);
    const bool above = routed && (count <= cap || b > thr_bits);
    const bool tie = routed && count > cap && b == thr_bits;
    int tot;
    const int tie_rank = block_excl_scan<int>(tie ? 1 : 0, &tot, scan_s) + ties_seen;
    ties_seen += tot;
    const bool kept = above || (tie && tie_rank < quota);
    const bool nonrouted = valid && !routed;
    const int nr_rank = block_excl_scan<int>(nonrouted ? 1 : 0, &tot, scan_s) + nonrouted_seen;
    nonrouted_seen += tot;
    const bool selected = kept || (nonrouted && nr_rank < pad_budget);
    const int pos = block_excl_scan<int>(selected ? 1 : 0, &tot, scan_s) + sel_seen;
    sel_seen += tot;
    if (selected && pos < cap) {
      const long long slot = (long long)e * cap + pos;
      sorted_indices[slot] = t;
      slot_probs[slot] = kept ? pr : 0.f;
      if (kept) slot_of_token[(long long)t * k + j] = (int)slot;
    }
    if (routed && !kept) slot_of_token[(long long)t * k + j] = -1;
    if (routed)
      for (int i = j + 1; i < k; ++i)      // a token that names this expert again has no slot for it
        if ((int)top_idx[(long long)t * k + i] == e) slot_of_token[(long long)t * k + i] = -1;
  }
  if (tid == 0) {
    routed_per_expert[e] = kept_total;
    if (tokens_per_expert != nullptr) tokens_per_expert[e] = cap;
  }
}

// --------------------------------------------------------------------------------------------
// Dropless plan of one rank: rows of an expert-major buffer of which expert e owns
// [offs[e], offs[e] + pad64(counts[e])), offs the running sum of the padded counts, the (token,
// choice) pairs of an expert in the order of their flat index.  Nothing is read by the host: the
// buffer is sized for the worst case (pairs + 63 * E rows) and the grouped GEMMs take offs and the
// padded counts from device memory.  A row that pads an expert to a multiple of 64 gets token -1 (the
// gather writes zeros there, the weight-gradient GEMM contracts in 64-row blocks), a row behind the
// last expert -2 (the gather leaves it alone, nobody reads it).
// Two launches, one CTA per expert in each: the first counts the expert's pairs, the second knows
// every count and therefore every start, and places the pairs.  No atomics, so the order is fixed.
// 8192 tokens, 64 experts, k = 6: 5 + 20 us; sorting on the device and building the row table on the host
// took 120 us of kernels and 1.8 ms during which the GPU waited for the host.
// --------------------------------------------------------------------------------------------
constexpr int kDropRows = 8;                          // pairs of a lane per step, 32 apart: coalesced
constexpr int kDropWarp = 32 * kDropRows;             // consecutive pairs of a warp per step
constexpr int kDropStep = kPlanWarps * kDropWarp;

__global__ void __launch_bounds__(kPlanThreads)
dropless_count_kernel(const long long* __restrict__ top_idx, int n, int* __restrict__ counts) {
  __shared__ int count_s[kPlanWarps];
  const int e = blockIdx.x, lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  int c = 0;
#pragma unroll 8
  for (int i = threadIdx.x; i < n; i += kPlanThreads) c += (int)top_idx[i] == e ? 1 : 0;
  c = __reduce_add_sync(0xffffffffu, c);
  if (lane == 0) count_s[warp] = c;
  __syncthreads();
  if (warp == 0) {
    c = __reduce_add_sync(0xffffffffu, count_s[lane]);
    if (lane == 0) counts[e] = c;
  }
}

__global__ void __launch_bounds__(kPlanThreads)
dropless_place_kernel(const long long* __restrict__ top_idx, const float* __restrict__ top_probs, int n,
                      int k, int E, const int* __restrict__ counts, int* __restrict__ group_rows,
                      int* __restrict__ group_offs, long long* __restrict__ row_token,
                      float* __restrict__ row_prob, int* __restrict__ slot_of_token, int rows_max) {
  __shared__ int scan_s[kPlanWarps];
  __shared__ int step_s[2][kPlanWarps];
  __shared__ int start_s, total_s;
  const int e = blockIdx.x, tid = threadIdx.x;
  // running sum of the padded counts (E <= kPlanThreads)
  {
    const int mine = tid < E ? (counts[tid] + 63) & ~63 : 0;
    int total;
    const int before = block_excl_scan<int>(mine, &total, scan_s);
    if (tid == e) start_s = before;
    if (tid == 0) total_s = total;
    if (e == 0 && tid < E) {
      group_rows[tid] = mine;
      group_offs[tid] = before;
    }
    __syncthreads();
  }
  const int start = start_s, lane = tid & 31, warp = tid >> 5;
  int seen = 0, buf = 0;
  for (int b = 0; b < n; b += kDropStep, buf ^= 1) {
    const int i0 = b + warp * kDropWarp + lane;
    int ex[kDropRows];
    float pr[kDropRows];      // with the index: fetched for hits only it would wait for it each time
#pragma unroll
    for (int q = 0; q < kDropRows; ++q) {
      const int i = min(i0 + 32 * q, n - 1);
      ex[q] = (int)top_idx[i];
      pr[q] = top_probs[i];
    }
    unsigned hits[kDropRows];
    int mine = 0;
#pragma unroll
    for (int q = 0; q < kDropRows; ++q) {
      hits[q] = __ballot_sync(0xffffffffu, i0 + 32 * q < n && ex[q] == e);
      mine += __popc(hits[q]);
    }
    if (lane == 0) step_s[buf][warp] = mine;      // two buffers: one barrier a step
    __syncthreads();
    const int w = step_s[buf][lane];
    int row = start + seen + __reduce_add_sync(0xffffffffu, lane < warp ? w : 0);
    seen += __reduce_add_sync(0xffffffffu, w);
#pragma unroll
    for (int q = 0; q < kDropRows; ++q) {
      if (hits[q] >> lane & 1u) {
        const int i = i0 + 32 * q, r = row + __popc(hits[q] & ((1u << lane) - 1u));
        row_token[r] = (unsigned)i / (unsigned)k;
        row_prob[r] = pr[q];
        slot_of_token[i] = r;
      }
      row += __popc(hits[q]);
    }
  }
  for (int r = start + seen + tid; r < start + ((seen + 63) & ~63); r += kPlanThreads) {
    row_token[r] = -1;
    row_prob[r] = 0.f;
  }
  for (long long r = total_s + (long long)e * kPlanThreads + tid; r < rows_max; r += (long long)E * kPlanThreads) {
    row_token[r] = -2;
    row_prob[r] = 0.f;
  }
}

// --------------------------------------------------------------------------------------------
// Router weight gradient dW[h, e] = sum_t x[t, h] * dlogits[t, e], x in bf16, everything else fp32, where the
// tensor core does not do it (router_wgrad.cu: few tokens or columns, rows that TMA does not take).  A CTA owns 1024
// columns of x (a thread four neighbours), EB experts and a share of the tokens; the gradients of the
// logits are the same for all threads and come from shared memory four at a time.  The shares are summed in
// a fixed order by a second kernel.  Against a conversion of x to fp32 and a library product, with a third of the
// error: 1024 x 4096, 8 experts, 15.3 us; 512 x 2048, 64 experts, 17.4.
// --------------------------------------------------------------------------------------------
constexpr int kRouterThreads = 256, kRouterTokens = 32;

template <int EB>
__global__ void __launch_bounds__(kRouterThreads, 2)
router_wgrad_kernel(const __nv_bfloat16* __restrict__ x, const float* __restrict__ dl, float* __restrict__ partial,
                    int T, int H, int E, int per_split) {
  constexpr int kAhead = 8;      // rows of x in flight
  __shared__ __align__(16) float dl_s[kRouterTokens][EB];
  const int h = blockIdx.x * 4 * kRouterThreads + 4 * threadIdx.x;
  const int e0 = blockIdx.y * EB;
  const int t_end = min(T, (int)(blockIdx.z + 1) * per_split);
  float acc[4][EB];
#pragma unroll
  for (int q = 0; q < 4; ++q)
#pragma unroll
    for (int e = 0; e < EB; ++e) acc[q][e] = 0.f;
  for (int t0 = blockIdx.z * per_split; t0 < t_end; t0 += kRouterTokens) {
    const int nt = min(kRouterTokens, t_end - t0);
    __syncthreads();
    for (int i = threadIdx.x; i < kRouterTokens * EB; i += kRouterThreads) {
      const int t = i / EB, e = e0 + i % EB;
      dl_s[t][i % EB] = (t < nt && e < E) ? dl[(long long)(t0 + t) * E + e] : 0.f;
    }
    __syncthreads();
    if (h < H) {
      const __nv_bfloat16* xr = x + (long long)t0 * H + h;
      for (int t = 0; t < nt; t += kAhead) {
        uint2 w[kAhead];
#pragma unroll
        for (int u = 0; u < kAhead; ++u)
          w[u] = t + u < nt ? *reinterpret_cast<const uint2*>(xr + (long long)(t + u) * H) : make_uint2(0, 0);
#pragma unroll
        for (int u = 0; u < kAhead; ++u) {
          if (t + u >= nt) break;
          const float xv[4] = {__uint_as_float(w[u].x << 16), __uint_as_float(w[u].x & 0xffff0000u),
                               __uint_as_float(w[u].y << 16), __uint_as_float(w[u].y & 0xffff0000u)};
#pragma unroll
          for (int e = 0; e < EB; e += 4) {
            const float4 d = *reinterpret_cast<const float4*>(&dl_s[t + u][e]);
#pragma unroll
            for (int q = 0; q < 4; ++q) {
              acc[q][e] = fmaf(xv[q], d.x, acc[q][e]);
              acc[q][e + 1] = fmaf(xv[q], d.y, acc[q][e + 1]);
              acc[q][e + 2] = fmaf(xv[q], d.z, acc[q][e + 2]);
              acc[q][e + 3] = fmaf(xv[q], d.w, acc[q][e + 3]);
            }
          }
        }
      }
    }
  }
  if (h >= H) return;
  float* out = partial + ((long long)blockIdx.z * H + h) * E + e0;
#pragma unroll
  for (int q = 0; q < 4; ++q)
#pragma unroll
    for (int e = 0; e < EB; e += 4) {
      if (e0 + e + 4 <= E && E % 4 == 0) {
        *reinterpret_cast<float4*>(out + (long long)q * E + e) =
            make_float4(acc[q][e], acc[q][e + 1], acc[q][e + 2], acc[q][e + 3]);
      } else {
#pragma unroll
        for (int i = 0; i < 4; ++i)
          if (e0 + e + i < E) out[(long long)q * E + e + i] = acc[q][e + i];
      }
    }
}

__global__ void __launch_bounds__(256)
router_wgrad_reduce_kernel(const float* __restrict__ partial, float* __restrict__ dw, int splits, long long n) {
  const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  float s = 0.f;
#pragma unroll 8
  for (int q = 0; q < splits; ++q) s += partial[q * n + i];
  dw[i] = s;
}

}  // namespace fm

static int check_launch(const char* what) {
  cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) {
    char buf[256];
    snprintf(buf, sizeof(buf), "%s: %s", what, cudaGetErrorString(e));
    fm_set_error(buf);
    return (int)e;
  }
  return 0;
}

static int router_eb(int E) { return E <= 8 ? 8 : 16; }

// Shares of the tokens, as the kernel makes them that takes x: of many tokens the tensor core makes few.  Left with those,
// rows on 8 bytes took 335 us for 8192 x 4096 x 8 instead of 36, and sums of as many tokens added up their roundings.
extern "C" int fm_router_wgrad_splits(int T, int H, int E, int x_on_16) {
  if (x_on_16 && fm::router_wgrad_mma_applies(T, H, E)) return fm::router_wgrad_mma_splits(T, H, E);
  const int eb = router_eb(E);
  const int tiles = ((H + 4 * fm::kRouterThreads - 1) / (4 * fm::kRouterThreads)) * ((E + eb - 1) / eb);
  int splits = (2 * 148) / tiles;                                         // two CTAs an SM
  const int most = (T + fm::kRouterTokens - 1) / fm::kRouterTokens;       // and a step's tokens for each
  if (splits > most) splits = most;
  return splits < 1 ? 1 : splits;
}

extern "C" int fm_router_wgrad(const void* x, const float* dlogits, float* partial, float* dw, int T, int H, int E,
                               int* status, cudaStream_t s) {
  if (T < 1 || E < 1 || H < 4 || H % 4 != 0 || (reinterpret_cast<uintptr_t>(x) & 7)) {
    fm_set_error("router_wgrad: a multiple of four columns, 8-byte aligned");
    return -1;
  }
  const int on_16 = (reinterpret_cast<uintptr_t>(x) & 15) == 0;
  const int splits = fm_router_wgrad_splits(T, H, E, on_16), eb = router_eb(E);
  int rc;
  if (on_16 && fm::router_wgrad_mma_applies(T, H, E)) {
    rc = fm::router_wgrad_mma(x, dlogits, partial, T, H, E, status, s);
  } else {
    const int per = (T + splits - 1) / splits;
    const dim3 grid((H + 4 * fm::kRouterThreads - 1) / (4 * fm::kRouterThreads), (E + eb - 1) / eb, splits);
    auto launch = [&](auto kernel) {
      kernel<<<grid, fm::kRouterThreads, 0, s>>>((const __nv_bfloat16*)x, dlogits, partial, T, H, E, per);
    };
    if (eb == 8) launch(fm::router_wgrad_kernel<8>);
    else launch(fm::router_wgrad_kernel<16>);
    rc = check_launch("router_wgrad");
  }
  if (rc) return rc;
  const long long n = (long long)H * E;
  fm::router_wgrad_reduce_kernel<<<(unsigned)((n + 255) / 256), 256, 0, s>>>(partial, dw, splits, n);
  return check_launch("router_wgrad_reduce");
}

extern "C" int fm_topk_softmax(const float* logits, long long* idx, float* probs, int T, int E,
                               int k, cudaStream_t s) {
  if (k > 16 || k > E) {
    fm_set_error("topk_softmax: k must be at most 16 and at most the number of experts");
    return -1;
  }
  const int grid = (T + 7) / 8;
  // A warp per token costs the same for every E up to 32 and grows with T, a thread per token costs E * k
  // comparisons in a row whatever T is, as long as the tokens find room side by side.  Warp and thread, us: 16384
  // tokens, 8 experts, k = 2, 3.9 and 3.3, k = 4 4.8 and 5.8; 65536 tokens, 8 experts, k = 2, 10.6 and 4.3, k = 8 19.9
  // and 17.5; 16 experts, k = 2, 10.6 and 8.3, k = 4 13.4 and 15.2.
  const bool threads = E > 256 || (E <= 16 && (long long)E * k * 1024 <= T && E * k <= (E <= 8 ? 64 : 32));
  if (threads) fm::topk_softmax_kernel<<<(T + 127) / 128, 128, 0, s>>>(logits, idx, probs, T, E, k);
  else if (E <= 32) fm::topk_softmax_warp_kernel<1><<<grid, 256, 0, s>>>(logits, idx, probs, T, E, k);
  else if (E <= 64) fm::topk_softmax_warp_kernel<2><<<grid, 256, 0, s>>>(logits, idx, probs, T, E, k);
  else if (E <= 128) fm::topk_softmax_warp_kernel<4><<<grid, 256, 0, s>>>(logits, idx, probs, T, E, k);
  else fm::topk_softmax_warp_kernel<8><<<grid, 256, 0, s>>>(logits, idx, probs, T, E, k);
  return check_launch("topk_softmax");
}

extern "C" int fm_moe_plan(const long long* top_idx, const float* top_probs, int T, int k, int E,
                           int cap, long long* sorted_indices, float* slot_probs, int* slot_of_token,
                           int* routed_per_expert, int* tokens_per_expert, cudaStream_t s) {
  if (k > 16 || cap > T) {
    fm_set_error("moe_plan: k must be at most 16 and the capacity at most the number of tokens");
    return -1;
  }
  const size_t smem = fm::plan_smem_bytes(T);
  if (smem <= fm::kPlanSmemMax) {
    // set on every such call: the limit belongs to the current device
    if (smem > 48 * 1024 && cudaFuncSetAttribute(fm::moe_plan_kernel<fm::kPlanThreads>,
                                                 cudaFuncAttributeMaxDynamicSharedMemorySize,
                                                 fm::kPlanSmemMax) != cudaSuccess)
      return check_launch("moe_plan");
    if (T <= fm::kPlanFewTokens)
      fm::moe_plan_kernel<fm::kPlanFewThreads><<<E, fm::kPlanFewThreads, smem, s>>>(
          top_idx, top_probs, T, k, E, cap, sorted_indices, slot_probs, slot_of_token, routed_per_expert,
          tokens_per_expert);
    else
      fm::moe_plan_kernel<fm::kPlanThreads><<<E, fm::kPlanThreads, smem, s>>>(
          top_idx, top_probs, T, k, E, cap, sorted_indices, slot_probs, slot_of_token, routed_per_expert,
          tokens_per_expert);
  } else {
    fm::moe_plan_large_kernel<<<E, fm::kPlanThreads, 0, s>>>(top_idx, top_probs, T, k, E, cap, sorted_indices,
                                                            slot_probs, slot_of_token, routed_per_expert,
                                                            tokens_per_expert);
  }
  return check_launch("moe_plan");
}

extern "C" int fm_dropless_plan_local(const long long* top_idx, const float* top_probs, int T, int k, int E,
                                      int rows_max, int* counts, int* group_rows, int* group_offs,
                                      long long* row_token, float* row_prob, int* slot_of_token,
                                      cudaStream_t s) {
  const long long n = (long long)T * k;
  if (T < 1 || k < 1 || E < 1 || E > fm::kPlanThreads || n + 63ll * E > 2147483647ll - fm::kDropStep ||
      rows_max < n + 63ll * E) {
    fm_set_error("dropless_plan_local: at most 1024 experts, and room for every pair plus 63 rows per expert");
    return -1;
  }
  fm::dropless_count_kernel<<<E, fm::kPlanThreads, 0, s>>>(top_idx, (int)n, counts);
  int rc = check_launch("dropless_count");
  if (rc) return rc;
  fm::dropless_place_kernel<<<E, fm::kPlanThreads, 0, s>>>(top_idx, top_probs, (int)n, k, E, counts, group_rows,
                                                          group_offs, row_token, row_prob, slot_of_token, rows_max);
  return check_launch("dropless_place");
}
