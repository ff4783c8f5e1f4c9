// GEMM for few rows per group: C[rows_g, N] = A[rows_g, K] * B_g with at most 32 rows in a group (in part 64).
//
// A pass over few tokens reads every weight for a handful of rows, so it is bound by memory.  The tiled GEMM loads 128
// rows of A beside 128 columns of B, of which nearly all rows are other groups': half of its ring and of its copy engine's
// time goes to them, and the tensor core multiplies 256 x 256 tiles for 16 rows (65 % busy, at a power that lowers
// the clock).  Here the product is turned round: the weights are the 128-row operand and 32 (64) tokens the
// other, so that nine tenths of the ring are weights (six stages of 32 KB or eleven of 16) and an MMA takes 65 cycles for
// 4 KB of weights, a third of the time in which they can arrive.
// The k blocks of all tiles lie in one sequence that is cut into equal parts, one per CTA: 896 tiles over 148 SMs would
// otherwise take seven rounds for 6.05, 256 tiles two for 1.73.  A tile that two or more CTAs share is summed in
// fp32 by the last of them to arrive, in the order of its parts (no CTA waits for another).
// Reading weights at 6.1 TB/s, 0.93 of the measured copy rate, for 8 groups of 16 rows, 4096 -> 2 x 14336 (360 -> 307 us);
// 5.4 TB/s for 14336 -> 4096 (181 -> 174), whose rows of 8 KB are cut into pieces of 512 bytes.  The pass over 64 tokens
// of a Mixtral-sized MoE, which the power of the wide products had slowed besides: 703 -> 503 us.
// The same product as the tiled GEMM's with store or activation epilogue; the counterpart in the reference are its per-expert
// products (fluid/moe/forward.py:217-352).
#include <cuda_bf16.h>
#include <string.h>

#include <mutex>

#include "../include/fm_smem.h"
#include "../include/fm_tmap.h"
#include "../include/sm100_ptx.cuh"
#include "../include/stream_table.h"
#include "act_math.cuh"
#include "gemm_few.h"

extern "C" void fm_set_error(const char* msg);

namespace fm {

constexpr int kFewThreads = 192;      // producer, MMA issuer, four epilogue warps (one per TMEM lane quarter)
constexpr int kFewCols = 128;         // weight columns of a tile (of each half, where there is a gate)
constexpr int kFewBK = 64;
constexpr int kFewRows = 32;           // rows of a group, the N extent of the products; twice that in a second form
constexpr int kFewRows2 = 2 * kFewRows;
constexpr int kFewMinBlocks = 16;     // k blocks of a CTA, at least, where tiles are shared
constexpr int kFewMaxCtas = 148;
constexpr int kFewCounters = 4 * kFewMaxCtas;
constexpr int kFewSets = 64;          // counter sets used in rotation
constexpr int kKernelIdGemmFew = 3;
constexpr int kFewSmemMax = 227 * 1024;

// What a tile is and what happens to it: 128 columns stored, 256 columns stored, 128 (or 2 x 128) columns through the
// activation.  The activation is a template parameter because its code is unrolled over sixteen rows.
enum FewKind { kFewNarrow, kFewWide, kFewGelu, kFewSilu, kFewNone, kFewSwiglu };
constexpr bool few_two(int kind) { return kind == kFewWide || kind == kFewSwiglu; }
constexpr bool few_act(int kind) { return kind >= kFewGelu; }

struct FewArgs {
  int groups, N, nk, ntn;             // output columns, k blocks, tiles along N
  int rows, total_rows;               // rows of a group unless they end before; rows of all
  int w_group_stride;                 // rows of the flattened weights between groups
  int n_half;                         // columns between the two halves of a tile
  void* C;
  long long ldc;
  int out_fp32;
  float alpha;
  __nv_bfloat16* pre_out;
  long long ld_pre;
  const float* probs;
  float* partial;                     // null: tiles are not shared
  int* counters;                      // [CTA][lane quarter]: parts that have arrived of the tile that the CTA begins
  int* counters_reset;                // the set that a later launch will use
  unsigned long long timeout_ns;
  int* status;
};

// Which k blocks of the sequence a CTA does: equal parts, or whole tiles where none is shared.
struct FewShare {
  long long units, tiles;
  int nk, ctas, shared;
  __device__ explicit FewShare(const FewArgs& a)
      : units((long long)a.groups * a.ntn * a.nk), tiles((long long)a.groups * a.ntn), nk(a.nk), ctas(gridDim.x),
        shared(a.partial != nullptr) {}
  __device__ __forceinline__ long long begin(int c) const {
    return shared ? units * c / ctas : tiles * c / ctas * nk;
  }
  // The CTA that does unit u (shared tiles only).
  __device__ __forceinline__ int owner(long long u) const {
    int c = (int)((u * ctas) / units);
    while (begin(c + 1) <= u) ++c;
    while (begin(c) > u) --c;
    return c;
  }
};

template <int kKind, int NT>
constexpr int few_stage_bytes() {
  return (few_two(kKind) ? 2 : 1) * kFewCols * kFewBK * 2 + NT * kFewBK * 2;
}
template <int kKind, int NT>
constexpr int few_stages() {
  return (kFewSmemMax - 1024 - 512) / few_stage_bytes<kKind, NT>();
}
template <int kKind, int NT>
constexpr int few_smem() {
  return few_stages<kKind, NT>() * few_stage_bytes<kKind, NT>() + 1024 + 512;
}

template <int kKind, bool kMn, int NT>
__global__ void __launch_bounds__(kFewThreads, 1)
gemm_few_kernel(const __grid_constant__ CUtensorMap tma_w, const __grid_constant__ CUtensorMap tma_x, const FewArgs a) {
  constexpr int W_BYTES = kFewCols * kFewBK * 2;
  constexpr int HALVES = few_two(kKind) ? 2 : 1;
  constexpr int TILE_N = kKind == kFewWide ? 2 * kFewCols : kFewCols;   // output columns
  constexpr int STAGE = few_stage_bytes<kKind, NT>();
  constexpr int NSTAGE = few_stages<kKind, NT>();
  constexpr uint32_t TMEM_COLS = 2 * NT * HALVES;     // two accumulators: 64 to 256 columns
  extern __shared__ uint8_t smem_few[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_few) + 1023) & ~uintptr_t(1023));
  uint64_t* bars = reinterpret_cast<uint64_t*>(smem + NSTAGE * STAGE);
  uint64_t* full = bars;
  uint64_t* empty = bars + NSTAGE;
  uint64_t* tfull = bars + 2 * NSTAGE;
  uint64_t* tempty = tfull + 2;
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(tempty + 2);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);
  static_assert((2 * NSTAGE + 4) * 8 + 8 <= 512, "barriers");

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  if (threadIdx.x == 0) {
    for (int s = 0; s < NSTAGE; ++s) {
      mbar_init(&full[s], 1);
      mbar_init(&empty[s], 1);
    }
    for (int i = 0; i < 2; ++i) {
      mbar_init(&tfull[i], 1);
      mbar_init(&tempty[i], 4);
    }
    *abort_flag = 0;
    mbar_fence_init();
    tma_prefetch_desc(&tma_w);
    tma_prefetch_desc(&tma_x);
  }
  if (a.counters_reset != nullptr && blockIdx.x == 0)
    for (int i = threadIdx.x; i < kFewCounters; i += kFewThreads) a.counters_reset[i] = 0;
  if (warp == 1) {
    tmem_alloc(tmem_slot, TMEM_COLS);
    tmem_relinquish();
  }
  tc_fence_before_sync();
  __syncthreads();
  tc_fence_after_sync();
  const uint32_t tmem_base = *tmem_slot;
  const uint64_t timeout = a.timeout_ns;
  const FewShare share(a);
  const int cta = blockIdx.x;
  const long long u0 = share.begin(cta), u1 = share.begin(cta + 1);
  auto wait_all = [&](uint64_t* bar, uint32_t parity, int what) {
    if (__all_sync(0xffffffffu, mbar_wait(bar, parity, timeout, abort_flag))) return true;
    if (lane == 0) report_status(a.status, kStatusMbarTimeout, kKernelIdGemmFew, what, 0, 0);
    return false;
  };

  if (warp == 0) {
    int stage = 0;
    uint32_t phase = 1;
    bool ok = true;
    for (long long u = u0; ok && u < u1;) {
      const long long tile = u / a.nk;
      const int kb0 = (int)(u - tile * a.nk), kb1 = (int)min((long long)a.nk, kb0 + (u1 - u));
      const int g = (int)(tile / a.ntn), n = (int)(tile - (long long)g * a.ntn) * TILE_N, wrow = g * a.w_group_stride;
      for (int kb = kb0; kb < kb1; ++kb) {
        if (!(ok = wait_all(&empty[stage], phase, 100 + stage))) break;
        if (elect_one()) {
          uint8_t* s = smem + stage * STAGE;
          const int k0 = kb * kFewBK;
          mbar_expect_tx(&full[stage], STAGE);
#pragma unroll
          for (int h = 0; h < HALVES; ++h) {
            const int nh = n + (h ? a.n_half : 0);
            if constexpr (kMn) {
              tma_load_2d(s + h * W_BYTES, &tma_w, &full[stage], nh, wrow + k0);
              tma_load_2d(s + h * W_BYTES + W_BYTES / 2, &tma_w, &full[stage], nh + 64, wrow + k0);
            } else {
              tma_load_2d(s + h * W_BYTES, &tma_w, &full[stage], k0, wrow + nh);
            }
          }
          tma_load_2d(s + HALVES * W_BYTES, &tma_x, &full[stage], k0, g * a.rows);
        }
        __syncwarp();
        if (++stage == NSTAGE) {
          stage = 0;
          phase ^= 1;
        }
      }
      u += kb1 - kb0;
    }
  } else if (warp == 1) {
    constexpr uint32_t idesc = umma_idesc_bf16(128, NT, kMn, false);
    constexpr int kSteps = kFewBK / 16;
    constexpr uint32_t kDescHi = umma_desc_hi(1024), kStageAdd = STAGE >> 4, kHalfAdd = W_BYTES >> 4;
    uint32_t w_lo[kSteps], x_lo[kSteps];      // low descriptor words of the k steps of stage 0
    {
      const uint32_t w0 = smem_u32(smem), x0 = w0 + HALVES * W_BYTES;
#pragma unroll
      for (int k = 0; k < kSteps; ++k) {
        w_lo[k] = kMn ? umma_desc_lo(w0 + k * 2048, W_BYTES / 2) : umma_desc_lo(w0 + k * 32, 0);
        x_lo[k] = umma_desc_lo(x0 + k * 32, 0);
      }
    }
    int stage = 0;
    uint32_t phase = 0, acc_phase = 1;
    int acc = 0;
    bool ok = true;
    for (long long u = u0; ok && u < u1;) {
      const int kb0 = (int)(u % a.nk), kb1 = (int)min((long long)a.nk, kb0 + (u1 - u));
      if (!(ok = wait_all(&tempty[acc], acc_phase, 200 + acc))) break;
      tc_fence_after_sync();
      const uint32_t d = tmem_base + acc * NT * HALVES;
      for (int kb = kb0; kb < kb1; ++kb) {
        if (!(ok = wait_all(&full[stage], phase, 300 + stage))) break;
        tc_fence_after_sync();
        if (elect_one()) {
          const uint32_t sadd = stage * kStageAdd;
#pragma unroll
          for (int h = 0; h < HALVES; ++h) {
            umma_bf16(d + h * NT, umma_desc_join(w_lo[0] + sadd + h * kHalfAdd, kDescHi),
                      umma_desc_join(x_lo[0] + sadd, kDescHi), idesc, kb > kb0 ? 1u : 0u);
#pragma unroll
            for (int k = 1; k < kSteps; ++k)
              umma_bf16_acc(d + h * NT, umma_desc_join(w_lo[k] + sadd + h * kHalfAdd, kDescHi),
                            umma_desc_join(x_lo[k] + sadd, kDescHi), idesc);
          }
          umma_commit(&empty[stage]);
        }
        __syncwarp();
        if (++stage == NSTAGE) {
          stage = 0;
          phase ^= 1;
        }
      }
      if (!ok) break;
      if (elect_one()) umma_commit(&tfull[acc]);
      __syncwarp();
      if (++acc == 2) {
        acc = 0;
        acc_phase ^= 1;
      }
      u += kb1 - kb0;
    }
  } else {
    // A lane holds one weight column and all tokens of the tile.
    const int q = warp & 3;
    const uint32_t lane_addr = (uint32_t)(q * 32) << 16;
    int acc = 0;
    uint32_t acc_phase = 0;
    constexpr int kPart = kFewCols * NT * HALVES;     // floats of a part
    for (long long u = u0; u < u1;) {
      const long long tile = u / a.nk;
      const int kb0 = (int)(u - tile * a.nk), kb1 = (int)min((long long)a.nk, kb0 + (u1 - u));
      u += kb1 - kb0;
      const int g = (int)(tile / a.ntn);
      if (!wait_all(&tfull[acc], acc_phase, 400 + acc)) break;
      tc_fence_after_sync();
      const int col = q * 32 + lane, n = (int)(tile - (long long)g * a.ntn) * TILE_N + col;
      const long long row0 = (long long)g * a.rows;
      const int rows = (int)min((long long)a.rows, a.total_rows - row0);
      const uint32_t t_acc = tmem_base + lane_addr + acc * NT * HALVES;
      // Sixteen rows of the tile at a time: the loops over them stay rolled, so that the code stays small.
      auto load = [&](int i0, float (&v)[HALVES][16]) {
#pragma unroll
        for (int h = 0; h < HALVES; ++h) tmem_ld_32x16(t_acc + h * NT + i0, v[h]);
        tmem_ld_wait();
      };
      auto release = [&]() {
        tc_fence_before_sync();
        __syncwarp();
        if (lane == 0) mbar_arrive(&tempty[acc]);
      };
      auto finish = [&](int i0, const float (&v)[HALVES][16]) {
        const float pr = few_act(kKind) && a.probs != nullptr && (lane & 15) + i0 < rows ?
                             a.probs[row0 + i0 + (lane & 15)] : 1.0f;
#pragma unroll
        for (int i = 0; i < 16; ++i) {
          const float p = few_act(kKind) ? __shfl_sync(0xffffffffu, pr, i) : 1.0f;
          if (i0 + i >= rows) continue;
          const long long row = row0 + i0 + i;
          if constexpr (!few_act(kKind)) {
#pragma unroll
            for (int h = 0; h < HALVES; ++h) {
              if (n + h * kFewCols >= a.N) continue;
              const float x = v[h][i] * a.alpha;
              const long long at = row * a.ldc + n + h * kFewCols;
              if (a.out_fp32) reinterpret_cast<float*>(a.C)[at] = x;
              else reinterpret_cast<__nv_bfloat16*>(a.C)[at] = __float2bfloat16(x);
            }
          } else if (n < a.N) {
            if (a.pre_out != nullptr) {
              a.pre_out[row * a.ld_pre + n] = __float2bfloat16(v[0][i]);
              if constexpr (HALVES == 2) a.pre_out[row * a.ld_pre + a.n_half + n] = __float2bfloat16(v[1][i]);
            }
            float y;
            if constexpr (kKind == kFewSwiglu) y = silu_f(v[0][i]) * v[HALVES - 1][i] * p;
            else y = (kKind == kFewGelu ? gelu_f(v[0][i]) : kKind == kFewSilu ? silu_f(v[0][i]) : v[0][i]) * p;
            reinterpret_cast<__nv_bfloat16*>(a.C)[row * a.ldc + n] = __float2bfloat16(y);
          }
        }
      };
      if (kb1 - kb0 == a.nk) {
#pragma unroll 1
        for (int i0 = 0; i0 < rows; i0 += 16) {
          float v[HALVES][16];
          load(i0, v);
          finish(i0, v);
        }
        release();
      } else {
        // One of several parts.  A CTA has at most two: a tile that an earlier CTA began (slot 2c) and one that it
        // begins and a later CTA ends (slot 2c + 1).  Each warp's columns are counted and summed by themselves.
        float* mine = a.partial + (long long)(2 * cta + (kb0 > 0 ? 0 : 1)) * kPart + col;
#pragma unroll 1
        for (int i0 = 0; i0 < rows; i0 += 16) {
          float v[HALVES][16];
          load(i0, v);
#pragma unroll
          for (int h = 0; h < HALVES; ++h)
#pragma unroll
            for (int i = 0; i < 16; ++i)
              if (i0 + i < rows) mine[(h * NT + i0 + i) * kFewCols] = v[h][i];
        }
        release();
        const int first = share.owner(tile * a.nk), last = share.owner((tile + 1) * a.nk - 1);
        __threadfence();
        __syncwarp();
        int before = 0;
        if (lane == 0) before = atomicAdd(a.counters + first * 4 + q, 1);
        if (__shfl_sync(0xffffffffu, before, 0) == last - first) {
          __threadfence();
#pragma unroll 1
          for (int i0 = 0; i0 < rows; i0 += 16) {
            float v[HALVES][16];
#pragma unroll
            for (int h = 0; h < HALVES; ++h)
#pragma unroll
              for (int i = 0; i < 16; ++i) v[h][i] = 0.f;
#pragma unroll 2
            for (int c = first; c <= last; ++c) {
              const float* part = a.partial + (long long)(2 * c + (c == first ? 1 : 0)) * kPart + i0 * kFewCols + col;
#pragma unroll
              for (int h = 0; h < HALVES; ++h)
#pragma unroll
                for (int i = 0; i < 16; ++i)
                  if (i0 + i < rows) v[h][i] += __ldcg(part + (h * NT + i) * kFewCols);
            }
            finish(i0, v);
          }
        }
      }
      if (++acc == 2) {
        acc = 0;
        acc_phase ^= 1;
      }
    }
  }

  if (*abort_flag) {
    // copies in flight land before the CTA's shared memory is handed back (error path only)
    const uint64_t t0 = global_timer_ns();
    while (global_timer_ns() - t0 < 200000ull) __nanosleep(1000);
  }
  tc_fence_before_sync();
  __syncthreads();
  if (warp == 1) {
    tc_fence_after_sync();
    tmem_dealloc(tmem_base, TMEM_COLS);
  }
}

// ----------------------------------------------------------------------------------------
// host side
// ----------------------------------------------------------------------------------------
// At most 32 rows in every group, a plain store or an activation.  Where the line lies (us, tiled GEMM and this one, weights
// cold): 8 groups, 4096 -> 2 x 14336 SwiGLU, 4 rows 355 and 302, 16 360 and 309, 32 364 and 317; 14336 -> 4096, 16 rows 181
// and 172; 64 groups of 8, 2048 -> 1024 GELU 79 and 70; one of 32, 512 -> 1024 15.4 and 12.4.  With 64 rows (and tiles for
// them) 371 and 332, but 14336 -> 4096 186 and 205, 64 groups 2048 -> 1024 80 and 90, 4096 -> 6144 34 and 45: the rows' part
// of the ring and of the epilogue grows while the tiled GEMM's stays.  Sizes in device memory come padded to 64 rows and go
// the other way for that reason.
// A narrow product of one group, such as the router's logits, takes chunks of 32 rows in the place of groups: few tiles with
// a long contraction, which the tiled GEMM leaves to a CTA for 128 rows each.  Tiled and this, us: 64 rows 4096 -> 8 25.3 and
// 18.7; 256 25.3 and 20.7; 1024 25.3 and 25.3; 2048 25.3 and 29.9; 512 rows 2048 -> 64 15.6 and 13.1; 1531 17.1 and
// 13.0; 8192 17.2 and 21.2; 2048 rows 1024 -> 8 11.0 and 15.1.
static bool few_chunks(const FmGemmDesc* d) {
  return d->uniform_rows > kFewRows && d->num_groups == 1 && d->epi == FM_EPI_STORE && d->N <= kFewCols && d->K >= 2048 &&
         (long long)((d->uniform_rows + kFewRows - 1) / kFewRows) * ((d->K + kFewBK - 1) / kFewBK) < 2048;
}
// Up to 64 rows a group besides: always with an activation, whose products are the wide ones, and stored from several
// groups unless the contraction is long.  Tiled and this, us: 8 groups 4096 -> 2 x 14336 of 40 rows 373 and 320, of 64 376
// and 330; 64 groups 2048 -> 1024 89 and 73, 83 and 78; stored, 64 groups 1024 -> 2048 77 and 68, 77 and 70; 16 groups
// 6400 -> 4096 183 and 168, 181 and 180; 8 groups 14336 -> 4096 184 and 196, 196 and 215; 1 group 2048 -> 6144 23.6 and
// 24.6, 23.6 and 28.7.
static bool few_rows2(const FmGemmDesc* d) {
  return d->uniform_rows <= kFewRows2 && (d->epi == FM_EPI_ACT || (d->num_groups > 1 && d->K <= 8192));
}
bool gemm_few_applies(const FmGemmDesc* d) {
  if (d->mode != 0 || d->a_mn || d->group_rows != nullptr || d->group_offs != nullptr || d->group_b != nullptr ||
      d->gate_flags != nullptr || d->n_rotate || d->k_rotate || d->num_groups <= 0 || d->K <= 0 || d->N <= 0 ||
      !d->cta_pair || d->uniform_rows <= 0 || (d->uniform_rows > kFewRows && !few_chunks(d) && !few_rows2(d)))
    return false;
  if (d->epi == FM_EPI_STORE)
    return !d->accumulate && d->residual == nullptr && d->alpha_dev == nullptr && !d->gated;
  return d->epi == FM_EPI_ACT;
}

static int few_kind(const FmGemmDesc* d) {
  if (d->epi == FM_EPI_STORE) return d->N > kFewCols ? kFewWide : kFewNarrow;
  if (d->gated) return kFewSwiglu;
  return d->act_kind == FM_ACT_GELU ? kFewGelu : d->act_kind == FM_ACT_SILU ? kFewSilu : kFewNone;
}

static int few_tile_cols(const FmGemmDesc* d) { return few_kind(d) == kFewWide ? 2 * kFewCols : kFewCols; }
static int few_ctas(const FmGemmDesc* d) {
  const int n = sm_count() < kFewMaxCtas ? sm_count() : kFewMaxCtas;
  return d->max_ctas > 0 && d->max_ctas < n ? d->max_ctas : n;
}
static long long few_tiles(const FmGemmDesc* d) {
  const long long groups = few_chunks(d) ? (d->uniform_rows + kFewRows - 1) / kFewRows : d->num_groups;
  return groups * ((d->N + few_tile_cols(d) - 1) / few_tile_cols(d));
}
// Whether tiles are shared.  The sum of a shared tile's parts costs about 7 us behind its last block (a store, a fence, a
// counter and a load of each part), in which a CTA's share of the memory rate moves ten blocks of 36 KB or eighteen of 20.
static bool few_shares(const FmGemmDesc* d) {
  const long long nk = (d->K + kFewBK - 1) / kFewBK, tiles = few_tiles(d), ctas = few_ctas(d);
  const long long equal = (tiles * nk + ctas - 1) / ctas;
  return (equal > kFewMinBlocks ? equal : kFewMinBlocks) + (few_two(few_kind(d)) ? 10 : 18) <
         (tiles + ctas - 1) / ctas * nk;
}

static long long few_partial_bytes(const FmGemmDesc* d) {
  return 2ll * kFewMaxCtas * kFewCols * (few_chunks(d) || d->uniform_rows <= kFewRows ? kFewRows : kFewRows2) * (few_two(few_kind(d)) ? 2 : 1) * 4;
}
long long gemm_few_workspace(const FmGemmDesc* d) {
  if (!gemm_few_applies(d) || !few_shares(d)) return 0;
  return few_partial_bytes(d) + kFewCounters * (long long)sizeof(int);
}

// Counters of the shared tiles, one group of sets for a stream: launches on a stream run one after another and use the sets
// in rotation; a launch clears the set that comes up half a rotation later.  Where the stream has none (under capture, and
// beyond the streams that the table knows) the counters lie in the workspace and a node of their own clears them (2 us).
class FewCounters {
 public:
  int *use = nullptr, *reset = nullptr;
  bool take(cudaStream_t stream, int* own) {
    StreamTable<Sets>& t = table();
    std::lock_guard<std::mutex> lock(t.mu);
    Sets* s = nullptr;
    if (!t.find(stream, &s)) return false;
    if (s != nullptr && s->p == nullptr) s->p = fresh(stream);
    if (s != nullptr && s->p != nullptr) {
      const unsigned i = s->next++ % kFewSets;
      use = s->p + i * kFewCounters;
      reset = s->p + (i + kFewSets / 2) % kFewSets * kFewCounters;
      return true;
    }
    use = own;
    if (cudaMemsetAsync(own, 0, kFewCounters * sizeof(int), stream) == cudaSuccess) return true;
    (void)cudaGetLastError();
    return false;
  }
  // The launch that was to clear a set did not run.
  void unused(cudaStream_t stream) {
    if (reset != nullptr) (void)cudaMemsetAsync(reset, 0, kFewCounters * sizeof(int), stream);
  }

 private:
  struct Sets {
    int* p = nullptr;
    unsigned next = 0;
  };
  static StreamTable<Sets>& table() {
    static StreamTable<Sets> t;
    return t;
  }
  static int* fresh(cudaStream_t stream) {
    const size_t bytes = (size_t)kFewSets * kFewCounters * sizeof(int);
    int* p = nullptr;
    cudaStreamCaptureMode mode = cudaStreamCaptureModeRelaxed;   // another thread may be capturing
    (void)cudaThreadExchangeStreamCaptureMode(&mode);
    cudaError_t e = cudaMalloc(&p, bytes);
    (void)cudaThreadExchangeStreamCaptureMode(&mode);
    if (e == cudaSuccess && (e = cudaMemsetAsync(p, 0, bytes, stream)) != cudaSuccess) cudaFree(p);
    if (e == cudaSuccess) return p;
    (void)cudaGetLastError();
    return nullptr;
  }
};

template <int kKind, bool kMn, int NT>
static int few_launch(const CUtensorMap& tw, const CUtensorMap& tx, const FewArgs& a, int grid, cudaStream_t stream) {
  auto kern = gemm_few_kernel<kKind, kMn, NT>;
  constexpr int smem = few_smem<kKind, NT>();
  static std::atomic<unsigned long long> configured{0};
  cudaError_t e = allow_smem(reinterpret_cast<const void*>(kern), smem, configured);
  if (e == cudaSuccess) {
    kern<<<grid, kFewThreads, smem, stream>>>(tw, tx, a);
    e = cudaGetLastError();
  }
  if (e != cudaSuccess) {
    fm_set_error(cudaGetErrorString(e));
    return (int)e;
  }
  return 0;
}

template <int kKind>
static int few_dispatch(const CUtensorMap& tw, const CUtensorMap& tx, const FewArgs& a, bool kn, int grid, cudaStream_t s) {
  if (a.rows <= kFewRows)
    return kn ? few_launch<kKind, true, kFewRows>(tw, tx, a, grid, s) : few_launch<kKind, false, kFewRows>(tw, tx, a, grid, s);
  return kn ? few_launch<kKind, true, kFewRows2>(tw, tx, a, grid, s) : few_launch<kKind, false, kFewRows2>(tw, tx, a, grid, s);
}

int gemm_few_launch(const FmGemmDesc* d, cudaStream_t stream) {
  const int kind = few_kind(d), tile_n = few_tile_cols(d);
  const bool act = d->epi == FM_EPI_ACT;
  const bool kn = d->b_mn != 0, chunks = few_chunks(d);
  CUtensorMap tw, tx;
  if (!make_tmap(&tw, d->B, d->b_inner, d->b_outer, d->ldb, kn ? 64 : 128) ||
      !make_tmap(&tx, d->A, d->a_inner, d->a_outer, d->lda, chunks || d->uniform_rows <= kFewRows ? kFewRows : kFewRows2))
    return -3;
  FewArgs a;
  memset(&a, 0, sizeof(a));
  a.groups = chunks ? (d->uniform_rows + kFewRows - 1) / kFewRows : d->num_groups;
  a.N = d->N;
  a.nk = (d->K + kFewBK - 1) / kFewBK;
  a.ntn = (d->N + tile_n - 1) / tile_n;
  // narrow products of one group: chunks of rows in the place of groups, all with the same weights
  a.rows = chunks ? kFewRows : d->uniform_rows;
  // no more than A has: the last groups may be cut, or empty, as with the tiled GEMM's stores
  const long long all_rows = (long long)(chunks ? 1 : d->num_groups) * d->uniform_rows;
  a.total_rows = (int)(all_rows < d->a_outer ? all_rows : d->a_outer);
  a.w_group_stride = chunks ? 0 : d->b_group_stride;
  a.n_half = kind == kFewWide ? kFewCols : d->n_half;
  a.C = act ? d->act_out : d->C;
  a.ldc = act ? d->ld_act : d->ldc;
  a.out_fp32 = !act && d->out_fp32;
  a.alpha = d->alpha == 0.f ? 1.0f : d->alpha;
  a.pre_out = reinterpret_cast<__nv_bfloat16*>(d->pre_out);
  a.ld_pre = d->ld_pre;
  a.probs = act ? d->probs : nullptr;
  a.timeout_ns = d->timeout_ns ? d->timeout_ns : 4000000000ull;
  a.status = d->status;
  const long long tiles = few_tiles(d), ctas = few_ctas(d);
  long long grid = tiles < ctas ? tiles : ctas;
  FewCounters counters;
  if (few_shares(d) && d->workspace != nullptr && d->workspace_bytes >= gemm_few_workspace(d) &&
      (reinterpret_cast<uintptr_t>(d->workspace) & 15) == 0 &&
      counters.take(stream, reinterpret_cast<int*>(static_cast<char*>(d->workspace) + few_partial_bytes(d)))) {
    a.counters = counters.use;
    a.counters_reset = counters.reset;
    a.partial = reinterpret_cast<float*>(d->workspace);
    grid = (tiles * a.nk + kFewMinBlocks - 1) / kFewMinBlocks;
    if (grid > ctas) grid = ctas;
  }
  int rc = 0;
  switch (kind) {
    case kFewNarrow: rc = few_dispatch<kFewNarrow>(tw, tx, a, kn, (int)grid, stream); break;
    case kFewWide: rc = few_dispatch<kFewWide>(tw, tx, a, kn, (int)grid, stream); break;
    case kFewGelu: rc = few_dispatch<kFewGelu>(tw, tx, a, kn, (int)grid, stream); break;
    case kFewSilu: rc = few_dispatch<kFewSilu>(tw, tx, a, kn, (int)grid, stream); break;
    case kFewNone: rc = few_dispatch<kFewNone>(tw, tx, a, kn, (int)grid, stream); break;
    default: rc = few_dispatch<kFewSwiglu>(tw, tx, a, kn, (int)grid, stream);
  }
  if (rc != 0) counters.unused(stream);
  return rc;
}

}  // namespace fm

extern "C" long long fm_gemm_workspace(const FmGemmDesc* d) { return fm::gemm_few_workspace(d); }
