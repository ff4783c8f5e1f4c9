// Router weight gradient dW[h, e] = sum_t x[t, h] * dlogits[t, e] on the tensor core: x in bf16, everything else in
// 32 bits.
//
// On the fp32 pipe 8192 x 2048 x 64 takes 31 us at best, and took 80.  An fp32 gradient is exactly the sum of three bf16
// numbers (8 + 8 + 8 bits), and a product of two bf16 numbers is exact in fp32, so three bf16 products give every bit
// that one fp32 product gives.  What the tensor core does otherwise is to add: it cuts sums off where the fp32 pipe
// rounds them, which shows in sums of one sign.  Its sums are therefore kept short, two of 32 tokens for the leading part and one
// of 64 for the two small ones, and added up in registers.  Against 64-bit sums, relative, 1536 to 8192 tokens, 512 to 4096
// columns, 8 to 64 experts: terms of both signs 8.3e-8 to 1.3e-7 (fp32 pipe 1.6e-7 to 3.1e-7), of one sign 5.5e-8 to 1.0e-7
// (8.5e-8 to 2.5e-7).  With one sum of 64 tokens for the leading part too, terms of one sign were off by up to 1.4 times as
// much as on the fp32 pipe; the time is the same.
// A CTA owns 128 columns of x (the M of the product; x is read by TMA as it lies, token-major), up to 64 experts and a
// share of the tokens.  Eight warps cut the gradients of 64 tokens into their parts and write them in the layout of the
// product's other operand, four add up finished sums, so that the tensor core has the next block meanwhile.  The
// shares of the tokens are summed in a fixed order by a second kernel.
// Both kernels, fp32 pipe and this, us: 8192 x 2048 x 64 95 and 29.7; x 128 173 and 44; 8192 x 1024 x 160 115 and 38;
// 4096 x 2048 x 16 34 and 19.5; 4096 x 4096 x 8 29.7 and 23.6; 16384 x 4096 x 8 69 and 58; 2048 x 1024 x 8 19.3 and 15.1.
#include <cuda_bf16.h>

#include <algorithm>

#include "../include/fm_tmap.h"
#include "../include/sm100_ptx.cuh"
#include "router_wgrad.h"

extern "C" void fm_set_error(const char* msg);

namespace fm {

constexpr int kRwThreads = 448;       // producer, MMA issuer, two groups of four splitting warps, four summing warps
constexpr int kRwRows = 128, kRwCols = 64, kRwTokens = 64, kRwStages = 4, kRwParts = 3;
constexpr int kRwBoxBytes = 64 * 64 * 2;                                   // 64 tokens of 64 columns or experts
constexpr int kRwStageBytes = (kRwRows / 64 + kRwParts) * kRwBoxBytes;
constexpr int kRwSmem = kRwStages * kRwStageBytes + 1024 + 256;
constexpr int kRwChains = 2;          // accumulators of the leading part: sums of 32 tokens each
constexpr int kRwAccCols = (kRwChains + 1) * kRwCols, kRwTmemCols = 512;   // twice 192, allocated by powers of two
constexpr int kKernelIdRouterWgrad = 4;

// Eight gradients as three bf16 vectors.  Truncation keeps every part finite; what is not finite is all in the first.
__device__ __forceinline__ void rw_split(const float (&v)[8], uint4 (&part)[kRwParts]) {
  uint32_t w[kRwParts][8];
#pragma unroll
  for (int i = 0; i < 8; ++i) {
    const uint32_t b = __float_as_uint(v[i]);
    const bool finite = (b & 0x7f800000u) != 0x7f800000u;
    const uint32_t hi = b & 0xffff0000u;
    const float r1 = v[i] - __uint_as_float(hi);            // exact: 16 bits are left
    const uint32_t mid = __float_as_uint(r1) & 0xffff0000u;
    const float r2 = r1 - __uint_as_float(mid);             // exact: 8 bits are left
    w[0][i] = finite || (b & 0x007fffffu) == 0 ? hi >> 16 : 0x7fc0u;
    w[1][i] = finite ? mid >> 16 : 0u;
    w[2][i] = finite ? __float_as_uint(r2) >> 16 : 0u;
  }
#pragma unroll
  for (int p = 0; p < kRwParts; ++p)
    part[p] = make_uint4(w[p][0] | w[p][1] << 16, w[p][2] | w[p][3] << 16, w[p][4] | w[p][5] << 16,
                         w[p][6] | w[p][7] << 16);
}

__global__ void __launch_bounds__(kRwThreads, 1)
router_wgrad_mma_kernel(const __grid_constant__ CUtensorMap tma_x, const float* __restrict__ dl,
                        float* __restrict__ partial, int T, int H, int E, int per_split, int vec,
                        unsigned long long timeout, int* status) {
  extern __shared__ uint8_t smem_rw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_rw) + 1023) & ~uintptr_t(1023));
  uint64_t* full = reinterpret_cast<uint64_t*>(smem + kRwStages * kRwStageBytes);
  uint64_t* empty = full + kRwStages;
  uint64_t* tfull = empty + kRwStages;
  uint64_t* tempty = tfull + 2;
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(tempty + 2);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);
  static_assert((2 * kRwStages + 4) * 8 + 8 <= 256, "barriers");

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  if (threadIdx.x == 0) {
    for (int s = 0; s < kRwStages; ++s) {
      mbar_init(&full[s], 1 + 4);
      mbar_init(&empty[s], 1);
    }
    for (int i = 0; i < 2; ++i) {
      mbar_init(&tfull[i], 1);
      mbar_init(&tempty[i], 4);
    }
    *abort_flag = 0;
    mbar_fence_init();
    tma_prefetch_desc(&tma_x);
  }
  if (warp == 1) {
    tmem_alloc(tmem_slot, kRwTmemCols);
    tmem_relinquish();
  }
  tc_fence_before_sync();
  __syncthreads();
  tc_fence_after_sync();
  const uint32_t tmem_base = *tmem_slot;
  const int h0 = blockIdx.x * kRwRows, e0 = blockIdx.y * kRwCols;
  const int t0 = blockIdx.z * per_split, t_end = min(T, t0 + per_split);
  const int nb = (t_end - t0 + kRwTokens - 1) / kRwTokens;
  const int cols = min(kRwCols, (E - e0 + 15) & ~15);         // experts in the product, a multiple of its step
  auto wait_all = [&](uint64_t* bar, uint32_t parity, int what) {
    if (__all_sync(0xffffffffu, mbar_wait(bar, parity, timeout, abort_flag))) return true;
    if (lane == 0) report_status(status, kStatusMbarTimeout, kKernelIdRouterWgrad, what, 0, 0);
    return false;
  };

  if (warp == 0) {
    for (int j = 0; j < nb; ++j) {
      const int st = j % kRwStages;
      if (!wait_all(&empty[st], ((j / kRwStages) & 1) ^ 1, 100 + st)) break;
      if (elect_one()) {
        uint8_t* s = smem + st * kRwStageBytes;
        mbar_expect_tx(&full[st], 2 * kRwBoxBytes);
        tma_load_2d(s, &tma_x, &full[st], h0, t0 + j * kRwTokens);
        tma_load_2d(s + kRwBoxBytes, &tma_x, &full[st], h0 + 64, t0 + j * kRwTokens);
      }
      __syncwarp();
    }
  } else if (warp == 1) {
    const uint32_t idesc = umma_idesc_bf16(kRwRows, cols, true, true);
    constexpr uint32_t kDescHi = umma_desc_hi(1024);
    for (int j = 0; j < nb; ++j) {
      const int st = j % kRwStages, acc = j & 1;
      if (!wait_all(&tempty[acc], ((j >> 1) & 1) ^ 1, 200 + acc)) break;
      if (!wait_all(&full[st], (j / kRwStages) & 1, 300 + st)) break;
      tc_fence_after_sync();
      if (elect_one()) {
        const uint32_t x0 = smem_u32(smem + st * kRwStageBytes), g0 = x0 + 2 * kRwBoxBytes;
        const uint32_t lead = tmem_base + acc * kRwAccCols, rest = lead + kRwChains * kRwCols;
        constexpr int kChain = kRwTokens / 16 / kRwChains;       // products of a chain
#pragma unroll
        for (int k = 0; k < kRwTokens / 16; ++k) {
          const uint64_t x = umma_desc_join(umma_desc_lo(x0 + k * 2048, kRwBoxBytes), kDescHi);
#pragma unroll
          for (int p = 0; p < kRwParts; ++p)
            umma_bf16(p == 0 ? lead + k / kChain * kRwCols : rest, x,
                      umma_desc_join(umma_desc_lo(g0 + p * kRwBoxBytes + k * 2048, kRwBoxBytes), kDescHi), idesc,
                      (p == 0 ? k % kChain > 0 : k > 0 || p == 2) ? 1u : 0u);
        }
        umma_commit(&empty[st]);
        umma_commit(&tfull[acc]);
      }
      __syncwarp();
    }
  } else if (warp < 10) {
    // Two groups take the blocks in turn; 16-byte chunks (eight experts of a token), token by token, fetched two blocks
    // ahead.
    constexpr int kChunks = kRwTokens * kRwCols / 8 / 128;
    const int group = (warp - 2) >> 2, i0 = (threadIdx.x - 64) & 127, per_token = cols / 8, n = kRwTokens * per_token;
    float v[kChunks][8];
    auto fetch = [&](int j) {
#pragma unroll
      for (int r = 0; r < kChunks; ++r) {
        const int i = i0 + r * 128, tok = i / per_token, e = e0 + (i - tok * per_token) * 8;
        const int t = t0 + j * kRwTokens + tok;
        const bool row = i < n && j < nb && t < t_end;
        const float* src = dl + (long long)t * E + e;
        if (row && vec && e + 8 <= E) {
          const float4 a = *reinterpret_cast<const float4*>(src), b = *reinterpret_cast<const float4*>(src + 4);
          v[r][0] = a.x; v[r][1] = a.y; v[r][2] = a.z; v[r][3] = a.w;
          v[r][4] = b.x; v[r][5] = b.y; v[r][6] = b.z; v[r][7] = b.w;
        } else {
#pragma unroll
          for (int c = 0; c < 8; ++c) v[r][c] = row && e + c < E ? src[c] : 0.f;
        }
      }
    };
    fetch(group);
    for (int j = group; j < nb; j += 2) {
      const int st = j % kRwStages;
      if (!wait_all(&empty[st], ((j / kRwStages) & 1) ^ 1, 400 + st)) break;
      uint8_t* g = smem + st * kRwStageBytes + 2 * kRwBoxBytes;
#pragma unroll
      for (int r = 0; r < kChunks; ++r) {
        const int i = i0 + r * 128, tok = i / per_token, c = i - tok * per_token;
        if (i >= n) continue;
        uint4 part[kRwParts];
        rw_split(v[r], part);
#pragma unroll
        for (int p = 0; p < kRwParts; ++p)
          *reinterpret_cast<uint4*>(g + p * kRwBoxBytes + tok * 128 + ((c ^ (tok & 7)) << 4)) = part[p];
      }
      fence_proxy_async_smem();
      __syncwarp();
      if (lane == 0) mbar_arrive(&full[st]);
      fetch(j + 2);
    }
  } else {
    // a lane holds one column of x and all experts of the tile
    const int q = warp & 3;
    const uint32_t lane_addr = (uint32_t)(q * 32) << 16;
    float sum[kRwCols];
#pragma unroll
    for (int e = 0; e < kRwCols; ++e) sum[e] = 0.f;
    for (int j = 0; j < nb; ++j) {
      const int acc = j & 1;
      if (!wait_all(&tfull[acc], (j >> 1) & 1, 500 + acc)) break;
      tc_fence_after_sync();
#pragma unroll
      for (int c = 0; c < kRwCols / 16; ++c) {
        if (c * 16 >= cols) continue;
        const uint32_t t = tmem_base + lane_addr + acc * kRwAccCols + c * 16;
        float a[kRwChains][16], b[16];
#pragma unroll
        for (int i = 0; i < kRwChains; ++i) tmem_ld_32x16(t + i * kRwCols, a[i]);
        tmem_ld_32x16(t + kRwChains * kRwCols, b);
        tmem_ld_wait();
#pragma unroll
        for (int e = 0; e < 16; ++e) {
          // an infinity in x meets the zeros of the small parts: the leading sum alone tells
          const float lead = a[0][e] + a[1][e];
          sum[c * 16 + e] += fabsf(lead) < INFINITY ? lead + b[e] : lead;
        }
      }
      tc_fence_before_sync();
      __syncwarp();
      if (lane == 0) mbar_arrive(&tempty[acc]);
    }
    const int h = h0 + q * 32 + lane;
    if (h < H) {
      float* out = partial + ((long long)blockIdx.z * H + h) * E + e0;
#pragma unroll
      for (int e = 0; e < kRwCols; e += 4) {
        if (E % 4 == 0) {
          if (e0 + e < E) *reinterpret_cast<float4*>(out + e) = make_float4(sum[e], sum[e + 1], sum[e + 2], sum[e + 3]);
        } else {
#pragma unroll
          for (int i = 0; i < 4; ++i)
            if (e0 + e + i < E) out[e + i] = sum[e + i];
        }
      }
    }
  }

  if (*abort_flag) {
    // copies in flight land before the CTA's shared memory is handed back (error path only)
    const uint64_t w0 = global_timer_ns();
    while (global_timer_ns() - w0 < 200000ull) __nanosleep(1000);
  }
  tc_fence_before_sync();
  __syncthreads();
  if (warp == 1) {
    tc_fence_after_sync();
    tmem_dealloc(tmem_base, kRwTmemCols);
  }
}

static int rw_tiles(int H, int E) { return ((H + kRwRows - 1) / kRwRows) * ((E + kRwCols - 1) / kRwCols); }
static int rw_per_split(int T, int H, int E) {
  // One round of CTAs; but a lane adds up the blocks of a share one after another, so two shares at the least and no share
  // of more than 4096 tokens.
  const int splits = std::max({148 / rw_tiles(H, E), 2, (T + 4095) / 4096});
  const int per = (T + splits - 1) / splits;
  return (per + kRwTokens - 1) / kRwTokens * kRwTokens;
}

// From 1536 tokens on: below that the fp32 pipe rounds few sums (one sign, 512 x 2048 x 64: 6.5e-8) and there is little to
// gain (17.4 and 15.1 us).  Up to 256 columns the fp32 pipe has more and shorter shares (one sign, 4096 x 128 x 128: 9.9e-8 and
// 1.3e-7).  No more tiles than SMs, and rows that TMA takes.
bool router_wgrad_mma_applies(int T, int H, int E) {
  return H % 8 == 0 && H > 2 * kRwRows && rw_tiles(H, E) <= 148 && T >= 1536;
}
int router_wgrad_mma_splits(int T, int H, int E) {
  const int per = rw_per_split(T, H, E);
  return (T + per - 1) / per;
}

int router_wgrad_mma(const void* x, const float* dlogits, float* partial, int T, int H, int E, int* status,
                     cudaStream_t s) {
  CUtensorMap tx;
  const cuuint64_t dims[2] = {(cuuint64_t)H, (cuuint64_t)T}, strides[1] = {(cuuint64_t)H * 2};
  const cuuint32_t box[2] = {64, kRwTokens};
  if (encode_tiled(&tx, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, x, dims, strides, box, CU_TENSOR_MAP_SWIZZLE_128B,
                   CU_TENSOR_MAP_L2_PROMOTION_L2_256B) != CUDA_SUCCESS) {
    fm_set_error("router_wgrad: cuTensorMapEncodeTiled failed");
    return -3;
  }
  // set on every call: the limit belongs to the current device
  cudaError_t e = cudaFuncSetAttribute(router_wgrad_mma_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kRwSmem);
  if (e == cudaSuccess) {
    const int vec = E % 4 == 0 && (reinterpret_cast<uintptr_t>(dlogits) & 15) == 0;
    const dim3 grid((H + kRwRows - 1) / kRwRows, (E + kRwCols - 1) / kRwCols, router_wgrad_mma_splits(T, H, E));
    router_wgrad_mma_kernel<<<grid, kRwThreads, kRwSmem, s>>>(tx, dlogits, partial, T, H, E, rw_per_split(T, H, E), vec,
                                                              4000000000ull, status);
    e = cudaGetLastError();
  }
  if (e == cudaSuccess) return 0;
  fm_set_error(cudaGetErrorString(e));
  return (int)e;
}

}  // namespace fm
