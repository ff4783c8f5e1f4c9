// Epilogues and host launcher of the tcgen05 GEMM (see gemm_sm100.cuh for the main loop).
#include <math.h>
#include <stdio.h>
#include <stdlib.h>
#include <string.h>

#include <mutex>

#include "../include/fm_api.h"
#include "../include/fm_smem.h"
#include "../include/fm_tmap.h"
#include "../include/stream_table.h"
#include "act_math.cuh"
#include "gemm_few.h"
#include "gemm_sm100.cuh"

namespace fm {

// ----------------------------------------------------------------------------------------
// helpers
// ----------------------------------------------------------------------------------------
template <int K>
struct Kind {
  static constexpr int value = K;
};
// Activation and derivative at once: the error function (sigmoid) is evaluated once for both.
template <int kKind>
__device__ __forceinline__ void act_dact(float x, float& y, float& dy) {
  if constexpr (kKind == FM_ACT_GELU) {
    const float cdf = 0.5f * (1.0f + erff(x * 0.70710678118654752f));
    y = x * cdf;
    dy = cdf + x * (0.3989422804014327f * __expf(-0.5f * x * x));
  } else if constexpr (kKind == FM_ACT_SILU) {
    const float s = sigmoid_f(x);
    y = x * s;
    dy = s * (1.0f + x * (1.0f - s));
  } else {
    y = x;
    dy = 1.0f;
  }
}

__device__ __forceinline__ void load_acc(uint32_t taddr, float* v, bool zero) {
  if (zero) {
#pragma unroll
    for (int i = 0; i < 32; ++i) v[i] = 0.f;
    return;
  }
  uint32_t r[32];
  tmem_ld_32x32(taddr, r);
  tmem_ld_wait();
#pragma unroll
  for (int i = 0; i < 32; ++i) v[i] = __uint_as_float(r[i]);
}

// Store 32 consecutive values of one row as bf16.  `ncols` = columns that exist (<= 32).
__device__ __forceinline__ void store_row_bf16(__nv_bfloat16* dst, const float* v, int ncols) {
  if (ncols >= 32 && (reinterpret_cast<uintptr_t>(dst) & 15) == 0) {
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      uint4 p;
      p.x = pack_bf16x2(v[8 * i + 0], v[8 * i + 1]);
      p.y = pack_bf16x2(v[8 * i + 2], v[8 * i + 3]);
      p.z = pack_bf16x2(v[8 * i + 4], v[8 * i + 5]);
      p.w = pack_bf16x2(v[8 * i + 6], v[8 * i + 7]);
      reinterpret_cast<uint4*>(dst)[i] = p;
    }
  } else {
    for (int i = 0; i < 32 && i < ncols; ++i) dst[i] = __float2bfloat16(v[i]);
  }
}
__device__ __forceinline__ void load_row_bf16(const __nv_bfloat16* src, float* v, int ncols) {
  if (ncols >= 32 && (reinterpret_cast<uintptr_t>(src) & 15) == 0) {
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const uint4 p = reinterpret_cast<const uint4*>(src)[i];
      const uint32_t w[4] = {p.x, p.y, p.z, p.w};
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const __nv_bfloat162 b = *reinterpret_cast<const __nv_bfloat162*>(&w[j]);
        v[8 * i + 2 * j] = __low2float(b);
        v[8 * i + 2 * j + 1] = __high2float(b);
      }
    }
  } else {
    for (int i = 0; i < 32; ++i) v[i] = i < ncols ? __bfloat162float(src[i]) : 0.f;
  }
}

// ----------------------------------------------------------------------------------------
// Coalesced epilogue stores.  After tcgen05.ld every lane holds 32 consecutive columns of ONE
// row, so a direct store makes each warp instruction touch 32 different rows.  Instead the
// warp writes its 32 x 32 block to a shared-memory stage and reads it back so that a
// group of lanes covers one row segment contiguously: every global store instruction then
// writes whole 32-byte sectors (fp32: 8 lanes x 16 B per row, 4 rows per instruction; bf16:
// 4 lanes x 16 B per row, 8 rows per instruction).
// ----------------------------------------------------------------------------------------
// Row `row` of the stage, four floats from column `col` on: rows of 32 floats, their 16-byte chunks swizzled by the row,
// which keeps both ways of walking the block free of bank conflicts without padding.
__device__ __forceinline__ float4* stage_at(float* stg, int row, int col) {
  return reinterpret_cast<float4*>(stg + row * 32 + (((col >> 2) ^ (row & 7)) << 2));
}
__device__ __forceinline__ const float4* stage_at(const float* stg, int row, int col) {
  return stage_at(const_cast<float*>(stg), row, col);
}

__device__ __forceinline__ void stage_put(float* stg, int lane, const float* v) {
  __syncwarp();
#pragma unroll
  for (int i = 0; i < 8; ++i)
    *stage_at(stg, lane, 4 * i) =
        make_float4(v[4 * i], v[4 * i + 1], v[4 * i + 2], v[4 * i + 3]);
  __syncwarp();
}
// The inverse: rows were filled cooperatively, every lane takes its own row back.
__device__ __forceinline__ void stage_get(const float* stg, int lane, float* v) {
  __syncwarp();
#pragma unroll
  for (int i = 0; i < 8; ++i) {
    const float4 x = *stage_at(stg, lane, 4 * i);
    v[4 * i] = x.x; v[4 * i + 1] = x.y; v[4 * i + 2] = x.z; v[4 * i + 3] = x.w;
  }
  __syncwarp();
}

// bf16 rows at base + rr * ld (rr = 0..rows_ok-1), 32 columns each; base 16-byte aligned, ld % 8 == 0.
__device__ __forceinline__ void staged_store_bf16(float* stg, int lane, const float* v, int rows_ok,
                                                  __nv_bfloat16* base, long long ld) {
  stage_put(stg, lane, v);
  const int sub = lane >> 2, c8 = (lane & 3) * 8;
#pragma unroll
  for (int pass = 0; pass < 4; ++pass) {
    const int rr = pass * 8 + sub;
    if (rr < rows_ok) {
      const float4 a = *stage_at(stg, rr, c8);
      const float4 b = *stage_at(stg, rr, c8 + 4);
      uint4 p;
      p.x = pack_bf16x2(a.x, a.y); p.y = pack_bf16x2(a.z, a.w);
      p.z = pack_bf16x2(b.x, b.y); p.w = pack_bf16x2(b.z, b.w);
      *reinterpret_cast<uint4*>(base + rr * ld + c8) = p;
    }
  }
}
// Same with an arbitrary destination per row: `my_row_ptr` is the destination of THIS lane's
// row (null = skip); the other lanes fetch it with a shuffle.
__device__ __forceinline__ void staged_store_bf16_scatter(float* stg, int lane, const float* v,
                                                          __nv_bfloat16* my_row_ptr) {
  stage_put(stg, lane, v);
  const int sub = lane >> 2, c8 = (lane & 3) * 8;
  const unsigned long long mine = reinterpret_cast<unsigned long long>(my_row_ptr);
#pragma unroll
  for (int pass = 0; pass < 4; ++pass) {
    const int rr = pass * 8 + sub;
    __nv_bfloat16* dst = reinterpret_cast<__nv_bfloat16*>(__shfl_sync(0xffffffffu, mine, rr));
    if (dst != nullptr) {
      const float4 a = *stage_at(stg, rr, c8);
      const float4 b = *stage_at(stg, rr, c8 + 4);
      uint4 p;
      p.x = pack_bf16x2(a.x, a.y); p.y = pack_bf16x2(a.z, a.w);
      p.z = pack_bf16x2(b.x, b.y); p.w = pack_bf16x2(b.z, b.w);
      *reinterpret_cast<uint4*>(dst + c8) = p;
    }
  }
}
// fp32 rows, optional accumulate; base 16-byte aligned, ld % 4 == 0.
__device__ __forceinline__ void staged_store_f32(float* stg, int lane, const float* v, int rows_ok,
                                                 float* base, long long ld, bool accumulate) {
  stage_put(stg, lane, v);
  const int sub = lane >> 3, c4 = (lane & 7) * 4;
#pragma unroll
  for (int pass = 0; pass < 8; ++pass) {
    const int rr = pass * 4 + sub;
    if (rr < rows_ok) {
      float4 x = *stage_at(stg, rr, c4);
      float4* dst = reinterpret_cast<float4*>(base + rr * ld + c4);
      if (accumulate) {
        const float4 o = *dst;
        x.x += o.x; x.y += o.y; x.z += o.z; x.w += o.w;
      }
      *dst = x;
    }
  }
}
// Coalesced load of 32 bf16 rows x 32 columns into the stage; every lane then reads its row.
__device__ __forceinline__ void staged_load_bf16(float* stg, int lane, float* v, int rows_ok,
                                                 const __nv_bfloat16* base, long long ld) {
  __syncwarp();
  const int sub = lane >> 2, c8 = (lane & 3) * 8;
#pragma unroll
  for (int pass = 0; pass < 4; ++pass) {
    const int rr = pass * 8 + sub;
    float4 a = make_float4(0.f, 0.f, 0.f, 0.f), b = a;
    if (rr < rows_ok) {
      const uint4 p = *reinterpret_cast<const uint4*>(base + rr * ld + c8);
      const __nv_bfloat162 p0 = *reinterpret_cast<const __nv_bfloat162*>(&p.x);
      const __nv_bfloat162 p1 = *reinterpret_cast<const __nv_bfloat162*>(&p.y);
      const __nv_bfloat162 p2 = *reinterpret_cast<const __nv_bfloat162*>(&p.z);
      const __nv_bfloat162 p3 = *reinterpret_cast<const __nv_bfloat162*>(&p.w);
      a = make_float4(__low2float(p0), __high2float(p0), __low2float(p1), __high2float(p1));
      b = make_float4(__low2float(p2), __high2float(p2), __low2float(p3), __high2float(p3));
    }
    *stage_at(stg, rr, c8) = a;
    *stage_at(stg, rr, c8 + 4) = b;
  }
  stage_get(stg, lane, v);
}
__device__ __forceinline__ bool aligned16(const void* p) {
  return (reinterpret_cast<uintptr_t>(p) & 15) == 0;
}

// ----------------------------------------------------------------------------------------
// Bulk tensor stores.  A warp writes whole boxes of 32 rows x 128 bytes (32 fp32 or 64 bf16 columns) into
// its staging area, one row per lane, in the 128-byte swizzle (16-byte chunk c of row r lies at chunk
// c ^ (r & 7), which also keeps the stores free of bank conflicts), and one lane hands the box to the copy
// engine.  Against stores from registers this takes the second trip through shared memory and the store
// instructions out of the epilogue: with 8 lanes x 16 bytes per row they kept the path from the SM to L2
// busy 79 % of the time at 7 bytes a cycle (weight gradients, 256 KB per output tile).
// Against the stores from registers: weight gradient of 8 experts, 1024 rows, 4096 x 28672, 1.87 -> 1.70 ms; of 64
// experts, 2048 x 1024, 294 -> 244 us; 64 experts' FC2 and FC1 input gradient 265 -> 215 us; 4096 x 6144 x 4096
// dense 158 -> 146 us.
// ----------------------------------------------------------------------------------------
struct BoxStore {
  uint8_t* stg;
  int lane;
  // Nothing that an earlier tile handed over is still being read.
  __device__ __forceinline__ BoxStore(float* s, int l) : stg(reinterpret_cast<uint8_t*>(s)), lane(l) {
    if (lane == 0) bulk_wait_group_read<0>();
    __syncwarp();
  }
  // The box, once the copy engine has read what was last in it.
  __device__ __forceinline__ uint8_t* next() const {
    if (lane == 0) bulk_wait_group_read<0>();
    __syncwarp();
    return stg;
  }
  __device__ __forceinline__ void put(uint8_t* box, int chunk, uint4 v) const {
    *reinterpret_cast<uint4*>(box + lane * 128 + ((chunk ^ (lane & 7)) << 4)) = v;
  }
  __device__ __forceinline__ void put_f32(uint8_t* box, const float* v) const {
#pragma unroll
    for (int i = 0; i < 8; ++i)
      put(box, i, make_uint4(__float_as_uint(v[4 * i]), __float_as_uint(v[4 * i + 1]), __float_as_uint(v[4 * i + 2]),
                             __float_as_uint(v[4 * i + 3])));
  }
  // 32 columns of a bf16 box: half 0 or 1.
  __device__ __forceinline__ void put_bf16(uint8_t* box, int half, const float* v) const {
#pragma unroll
    for (int i = 0; i < 4; ++i)
      put(box, half * 4 + i, make_uint4(pack_bf16x2(v[8 * i], v[8 * i + 1]), pack_bf16x2(v[8 * i + 2], v[8 * i + 3]),
                                        pack_bf16x2(v[8 * i + 4], v[8 * i + 5]),
                                        pack_bf16x2(v[8 * i + 6], v[8 * i + 7])));
  }
  __device__ __forceinline__ void send(const CUtensorMap* m, const uint8_t* box, int col, int row, int group) const {
    fence_proxy_async_smem();
    __syncwarp();
    if (lane == 0) {
      tma_store_3d(m, box, col, row, group);
      bulk_commit_group();
    }
  }
};

// Phase of the barrier of block k's set in the epilogues that update whole blocks in place, two sets of boxes in
// turn.  With four blocks a tile (BN 256) each set is filled twice, so every tile starts at phase 0; with two (BN 128)
// once, so the phase turns with the tiles that the warp has done this way (`fills`).
// Tiles of 128 columns by boxes against the path through registers: GELU gradient of 32768 rows, 64 -> 128 columns, 32.7 ->
// 19.6 us, 2048 -> 128 57 -> 43; AdamW of 14336 x 128, 4096 rows, 42 -> 36.
template <int kBlocks>
__device__ __forceinline__ uint32_t box_parity(int k, uint32_t fills) {
  static_assert(kBlocks == 2 || kBlocks == 4, "tiles of 128 or 256 columns");
  return kBlocks == 4 ? (k >> 1) & 1 : fills & 1;
}

// ----------------------------------------------------------------------------------------
// Epilogue 0: plain store (bf16 or fp32, optional accumulate; the fp32-accumulate form is the
// weight-gradient epilogue that adds straight into a flat gradient buffer).
// ----------------------------------------------------------------------------------------
struct EpiStore {
  void* C;
  long long ldc;
  long long group_stride;
  int out_fp32;
  int accumulate;
  float alpha;
  int boxes;          // C can be written with bulk tensor stores: map 0 is C as [group][row][column]
  const float* alpha_dev;
  const __nv_bfloat16* residual;   // what a bf16 result is added to: another array, or C itself
  long long ld_residual;

  template <int BN>
  __device__ __forceinline__ void run(const Tile& t, const GemmArgs& a, uint32_t taddr, int r,
                                      bool zero, int chalf, float* stg, const CUtensorMap* maps, uint64_t* wbar,
                                      volatile int* abort_flag, int kernel_id, uint32_t& fills) const {
    const int lane = r & 31;
    const long long row = a.mode == 0 ? (long long)t.row_base + t.m0 + r : (long long)t.m0 + r;
    const long long row0 = row - lane;   // first row of this warp
    const long long goff = a.mode == 0 ? 0 : (long long)t.g * group_stride;
    const bool row_ok = r < t.rows_valid;
    const int rows_ok = max(0, min(32, t.rows_valid - (r - lane)));
    const float alpha = alpha_dev != nullptr ? this->alpha * *alpha_dev : this->alpha;
    if (boxes) {
      // All 32 rows exist, or the boxes would reach into the next group's rows; columns past N are cut
      // off by the tensor map.
      BoxStore bs(stg, lane);
      if (rows_ok == 32) {
        const int z = a.mode == 0 ? 0 : t.g;
        constexpr int kStep = BN / 64;      // 32-column blocks of this warp: 4 or 2
        if (out_fp32) {
#pragma unroll 1
          for (int c = chalf * kStep; c < (chalf + 1) * kStep; ++c) {
            const int col = t.n_tile * BN + c * 32;
            if (col >= a.N) break;
            float v[32];
            load_acc(taddr + c * 32, v, zero);
            if (alpha != 1.0f) {
#pragma unroll
              for (int i = 0; i < 32; ++i) v[i] *= alpha;
            }
            uint8_t* box = bs.next();
            bs.put_f32(box, v);
            bs.send(maps, box, col, (int)row0, z);
          }
        } else {
#pragma unroll 1
          for (int c = chalf * kStep; c < (chalf + 1) * kStep; c += 2) {
            const int col = t.n_tile * BN + c * 32;
            if (col >= a.N) break;
            if (residual != nullptr && col + 64 <= a.N) {
              // the stage that turns the rows of the residual over to the lanes is the box itself, so the sums wait
              // in registers until both halves have been read
              uint32_t w[32];
              uint8_t* box = bs.next();
#pragma unroll
              for (int h = 0; h < 2; ++h) {
                float v[32], p[32];
                staged_load_bf16(stg, lane, p, 32, residual + row0 * ld_residual + col + 32 * h, ld_residual);
                load_acc(taddr + (c + h) * 32, v, zero);
#pragma unroll
                for (int i = 0; i < 16; ++i)
                  w[16 * h + i] = pack_bf16x2(fmaf(v[2 * i], alpha, p[2 * i]), fmaf(v[2 * i + 1], alpha, p[2 * i + 1]));
              }
              __syncwarp();
#pragma unroll
              for (int i = 0; i < 8; ++i) bs.put(box, i, make_uint4(w[4 * i], w[4 * i + 1], w[4 * i + 2], w[4 * i + 3]));
              bs.send(maps, box, col, (int)row0, z);
              continue;
            }
            uint8_t* box = bs.next();
#pragma unroll
            for (int h = 0; h < 2; ++h) {
              float v[32];
              load_acc(taddr + (c + h) * 32, v, zero);
              if (alpha != 1.0f) {
#pragma unroll
                for (int i = 0; i < 32; ++i) v[i] *= alpha;
              }
              if (residual != nullptr) {
                // the last columns of the matrix
                float p[32];
                const int nc = min(32, a.N - col - 32 * h);
                if (nc > 0) {
                  load_row_bf16(residual + row * ld_residual + col + 32 * h, p, nc);
#pragma unroll
                  for (int i = 0; i < 32; ++i) v[i] += p[i];
                }
              }
              bs.put_bf16(box, h, v);
            }
            bs.send(maps, box, col, (int)row0, z);
          }
        }
        return;
      }
    }
#pragma unroll 1
    for (int c = chalf * (BN / 64); c < (chalf + 1) * (BN / 64); ++c) {
      const int col = t.n_tile * BN + c * 32;
      if (col >= a.N) break;
      float v[32];
      load_acc(taddr + c * 32, v, zero);
      if (rows_ok == 0) continue;
      const int ncols = min(32, a.N - col);
      if (alpha != 1.0f) {
#pragma unroll
        for (int i = 0; i < 32; ++i) v[i] *= alpha;
      }
      if (out_fp32) {
        float* base = reinterpret_cast<float*>(C) + goff + row0 * ldc + col;
        if (ncols == 32 && (ldc & 3) == 0 && aligned16(base)) {
          staged_store_f32(stg, lane, v, rows_ok, base, ldc, accumulate != 0);
        } else if (row_ok) {
          float* dst = base + (long long)lane * ldc;
          for (int i = 0; i < ncols; ++i) dst[i] = accumulate ? dst[i] + v[i] : v[i];
        }
      } else {
        __nv_bfloat16* base = reinterpret_cast<__nv_bfloat16*>(C) + goff + row0 * ldc + col;
        const __nv_bfloat16* src = accumulate ? base : residual ? residual + row0 * ld_residual + col : nullptr;
        const long long ldr = accumulate ? ldc : ld_residual;
        if (ncols == 32 && (ldc & 7) == 0 && aligned16(base) &&
            (src == nullptr || ((ldr & 7) == 0 && aligned16(src)))) {
          if (src != nullptr) {
            float p[32];
            staged_load_bf16(stg, lane, p, rows_ok, src, ldr);
#pragma unroll
            for (int i = 0; i < 32; ++i) v[i] += p[i];
          }
          staged_store_bf16(stg, lane, v, rows_ok, base, ldc);
        } else if (row_ok) {
          __nv_bfloat16* dst = base + (long long)lane * ldc;
          if (src != nullptr) {
            float p[32];
            load_row_bf16(src + (long long)lane * ldr, p, ncols);
#pragma unroll
            for (int i = 0; i < 32; ++i) v[i] += p[i];
          }
          store_row_bf16(dst, v, ncols);
        }
      }
    }
  }
  __device__ __forceinline__ void tile_done(const Tile&, const GemmArgs&, int) const {}
};

// Store one 32 x 32 block of bf16 rows (consecutive rows, leading dimension ld), coalesced when
// the block is full-width and aligned, per-row otherwise.
__device__ __forceinline__ void put_block_bf16(float* stg, int lane, const float* v, int rows_ok,
                                               bool row_ok, __nv_bfloat16* base, long long ld, int ncols) {
  if (ncols == 32 && (ld & 7) == 0 && aligned16(base))
    staged_store_bf16(stg, lane, v, rows_ok, base, ld);
  else if (row_ok)
    store_row_bf16(base + (long long)lane * ld, v, ncols);
}
__device__ __forceinline__ void get_block_bf16(float* stg, int lane, float* v, int rows_ok, bool row_ok,
                                               const __nv_bfloat16* base, long long ld, int ncols) {
  if (ncols == 32 && (ld & 7) == 0 && aligned16(base)) {
    staged_load_bf16(stg, lane, v, rows_ok, base, ld);
  } else if (row_ok) {
    load_row_bf16(base + (long long)lane * ld, v, ncols);
  } else {
#pragma unroll
    for (int i = 0; i < 32; ++i) v[i] = 0.f;
  }
}

// ----------------------------------------------------------------------------------------
// Epilogue 5: optimizer in the weight-gradient epilogue.  The accumulator tile IS the gradient
// of the matching tile of a bf16 parameter; instead of storing it, the epilogue reads the
// parameter and its two bf16 Adam moments, applies the AdamW update and writes the three back
// (12 bytes of traffic per element instead of a 4-byte gradient store here plus a 16-byte
// optimizer pass later).  Only valid when the gradient is complete after this GEMM: a single
// micro-batch per step and no data-parallel reduction of this parameter.
// 12 bytes an element, which the copy rate would move in 1.7 ms for 8 x 4096 x 28672; it takes 2.66 (4.2 TB/s).  With
// loads and stores from registers the eight epilogue warps spent their time on the way to L2 (requests 56 % busy,
// a third of the stalls `lg_throttle`) and on a trip of the accumulator through shared memory; through boxes, with
// one pipeline stage less, 8 experts of 1024 rows take 3.70 -> 2.69 ms for 4096 x 28672 and 1.78 -> 1.32 ms for
// 14336 x 4096.
// Parameter and moments are not fetched into L2 ahead of the boxes: a tile ahead on every SM is 58 MB of lines on their
// way, which pushed each other and the operands out (8 x 4096 x 7168: 2.38 GB read for 1.59, without 1.73); 2.81 -> 2.66 ms and 1.38 -> 1.29 without,
// the activation's gradient, which did the same, 765 -> 720, 292 -> 267 and 288 -> 251 us for the sizes below.
// ----------------------------------------------------------------------------------------
struct EpiAdam {
  __nv_bfloat16* P;
  __nv_bfloat16* Mo;
  __nv_bfloat16* Vo;
  long long ld;
  long long group_stride;
  float alpha;   // gradient scale
  float lr, beta1, beta2, eps, weight_decay, rbc1, rbc2;

  // One AdamW step on 8 consecutive elements held as bf16 pairs.  The epilogue has only eight
  // warps per SM to hide latency with, so the square root and the division use the hardware
  // approximations (2 ulp; parameter and moments are rounded to bf16 right after).
  static __device__ __forceinline__ float sqrt_approx(float x) {
    float y;
    asm("sqrt.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
  }
  static __device__ __forceinline__ float rcp_approx(float x) {
    float y;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
  }
  // The arithmetic runs on packed fp32 pairs (fma.rn.f32x2 and friends, one issue slot per two elements): the eight
  // epilogue warps hide little latency, so fewer instructions in their chains are what the arithmetic can give.
  __device__ __forceinline__ void update8(const float* gg, uint4& pw, uint4& pm, uint4& pv) const {
    uint32_t* ww = reinterpret_cast<uint32_t*>(&pw);
    uint32_t* wm = reinterpret_cast<uint32_t*>(&pm);
    uint32_t* wv = reinterpret_cast<uint32_t*>(&pv);
    const float c1 = (1.f - beta1) * alpha, c2 = (1.f - beta2) * alpha * alpha;
    const float step_m = lr * rbc1, decay = 1.f - lr * weight_decay;
    const float2 kB1 = make_float2(beta1, beta1), kB2 = make_float2(beta2, beta2);
    const float2 kC1 = make_float2(c1, c1), kC2 = make_float2(c2, c2);
    const float2 kR2 = make_float2(rbc2, rbc2), kEps = make_float2(eps, eps);
    const float2 kNs = make_float2(-step_m, -step_m), kDec = make_float2(decay, decay);
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      // bf16 -> fp32 is a 16-bit shift of the bit pattern
      float2 w2 = make_float2(__uint_as_float(ww[q] << 16), __uint_as_float(ww[q] & 0xffff0000u));
      float2 m2 = make_float2(__uint_as_float(wm[q] << 16), __uint_as_float(wm[q] & 0xffff0000u));
      float2 v2 = make_float2(__uint_as_float(wv[q] << 16), __uint_as_float(wv[q] & 0xffff0000u));
      const float2 g2 = make_float2(gg[2 * q], gg[2 * q + 1]);
      m2 = __ffma2_rn(kB1, m2, __fmul2_rn(kC1, g2));
      v2 = __ffma2_rn(kB2, v2, __fmul2_rn(kC2, __fmul2_rn(g2, g2)));
      float2 s2 = __fmul2_rn(v2, kR2);
      s2.x = sqrt_approx(s2.x);
      s2.y = sqrt_approx(s2.y);
      s2 = __fadd2_rn(s2, kEps);
      const float2 r2 = make_float2(rcp_approx(s2.x), rcp_approx(s2.y));
      w2 = __ffma2_rn(__fmul2_rn(kNs, m2), r2, __fmul2_rn(kDec, w2));
      ww[q] = pack_bf16x2(w2.x, w2.y);
      wm[q] = pack_bf16x2(m2.x, m2.y);
      wv[q] = pack_bf16x2(v2.x, v2.y);
    }
  }

  int boxes;     // parameter and moments (maps 0 to 2) can be moved by bulk tensor copies

  // Whole blocks (32 rows, all of this warp's columns inside the matrix) are updated in shared memory: boxes
  // of 32 rows x 32 columns of the three arrays are copied in, read and written back one row per lane,
  // which is the accumulator's own layout, and copied out.  Two sets of boxes alternate: a set is refilled
  // while the other is updated.  The 64-byte swizzle (chunk c of row r at c ^ (r >> 1 & 3)) keeps the
  // 16-byte accesses of eight lanes in different banks.
  static constexpr int kBox = 32 * 64;
  static constexpr int kWarpBytes = 2 * 3 * kBox;
  template <int BN>
  __device__ __forceinline__ bool whole(const Tile& t, const GemmArgs& a, int r, int chalf) const {
    return boxes && t.rows_valid - (r & ~31) >= 32 && t.n_tile * BN + (chalf + 1) * (BN / 2) <= a.N;
  }
  __device__ __forceinline__ void load_set(const CUtensorMap* maps, uint8_t* set, uint64_t* bar, int col, int row,
                                           int g) const {
    mbar_expect_tx(bar, 3 * kBox);
#pragma unroll
    for (int i = 0; i < 3; ++i) tma_load_3d(set + i * kBox, maps + i, bar, col, row, g);
  }
  template <int BN>
  __device__ __forceinline__ void fetch(const Tile& t, const GemmArgs& a, int r, int chalf, float* stg,
                                        const CUtensorMap* maps, uint64_t* wbar) const {
    if (!whole<BN>(t, a, r, chalf)) return;
    fence_proxy_async_smem();         // what this warp stored in its area by other means is done
    __syncwarp();
    if ((r & 31) == 0) {
      bulk_wait_group_read<0>();      // the last tile's boxes have left
      const int row0 = (a.mode == 0 ? t.row_base : 0) + t.m0 + r;
      const int col = t.n_tile * BN + chalf * (BN / 2);
      uint8_t* sets = reinterpret_cast<uint8_t*>(stg);
#pragma unroll
      for (int i = 0; i < 2; ++i)
        load_set(maps, sets + i * 3 * kBox, wbar + i, col + 32 * i, row0, a.mode == 0 ? 0 : t.g);
    }
    __syncwarp();
  }

  template <int BN>
  __device__ __forceinline__ void run(const Tile& t, const GemmArgs& a, uint32_t taddr, int r,
                                      bool zero, int chalf, float* stg, const CUtensorMap* maps, uint64_t* wbar,
                                      volatile int* abort_flag, int kernel_id, uint32_t& fills) const {
    constexpr int NB = BN / 64;          // 32-column blocks handled by this warp
    const int lane = r & 31;
    const long long row = a.mode == 0 ? (long long)t.row_base + t.m0 + r : (long long)t.m0 + r;
    const long long row0 = row - lane;
    const long long goff = a.mode == 0 ? 0 : (long long)t.g * group_stride;
    const bool row_ok = r < t.rows_valid;
    const int rows_ok = max(0, min(32, t.rows_valid - (r - lane)));
    const int sub = lane >> 2, c8 = (lane & 3) * 8;
    const int c_begin = chalf * NB;
    const long long off0 = goff + row0 * ld + (long long)t.n_tile * BN;
    if (whole<BN>(t, a, r, chalf)) {
      uint8_t* const sets = reinterpret_cast<uint8_t*>(stg);
      const int z = a.mode == 0 ? 0 : t.g;
      const int swz = (lane >> 1) & 3;
#pragma unroll 1
      for (int k = 0; k < NB; ++k) {
        const int col = t.n_tile * BN + (c_begin + k) * 32;
        uint8_t* const set = sets + (k & 1) * 3 * kBox;
        float g[32];
        load_acc(taddr + (c_begin + k) * 32, g, zero);
        if (lane == 0 && k > 0 && k + 1 < NB) {
          // the set of the block before has left: refill it for the block after this one
          bulk_wait_group_read<0>();
          load_set(maps, sets + ((k + 1) & 1) * 3 * kBox, wbar + ((k + 1) & 1), col + 32, (int)row0, z);
        }
        __syncwarp();
        if (!mbar_wait(wbar + (k & 1), box_parity<BN / 64>(k, fills), a.timeout_ns, abort_flag)) {
          if (lane == 0) report_status(a.status, kStatusMbarTimeout, kernel_id, 500 + k, 0, 0);
          return;
        }
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          uint4* const at = reinterpret_cast<uint4*>(set + lane * 64 + ((j ^ swz) << 4));
          uint4 w = at[0], m = at[kBox / 16], v = at[2 * kBox / 16];
          update8(g + 8 * j, w, m, v);
          at[0] = w;
          at[kBox / 16] = m;
          at[2 * kBox / 16] = v;
        }
        fence_proxy_async_smem();
        __syncwarp();
        if (lane == 0) {
#pragma unroll
          for (int i = 0; i < 3; ++i) tma_store_3d(maps + i, set + i * kBox, col, (int)row0, z);
          bulk_commit_group();
        }
      }
      __syncwarp();
      ++fills;
      return;
    }
    if (boxes) {
      if (lane == 0) bulk_wait_group_read<0>();     // the stage below shares the area with the boxes
      __syncwarp();
    }
    // coalesced path: whole 32-column blocks, 16-byte aligned rows (4 lanes x 16 bytes per row)
    const bool vec_ok = (ld & 7) == 0 && aligned16(P + off0) && aligned16(Mo + off0) && aligned16(Vo + off0);
#pragma unroll 1
    for (int k = 0; k < NB; ++k) {
      const int c = c_begin + k;
      const int col = t.n_tile * BN + c * 32;
      if (col >= a.N) break;
      const int ncols = min(32, a.N - col);
      const long long off = off0 + c * 32;
      const bool fast = vec_ok && ncols == 32;
      // parameter and moments do not depend on the accumulator: issue their loads first
      uint4 b[12];
      if (fast && rows_ok == 32) {
#pragma unroll
        for (int pass = 0; pass < 4; ++pass) {
          const long long o = off + (long long)(pass * 8 + sub) * ld + c8;
          b[pass * 3 + 0] = *reinterpret_cast<const uint4*>(P + o);
          b[pass * 3 + 1] = *reinterpret_cast<const uint4*>(Mo + o);
          b[pass * 3 + 2] = *reinterpret_cast<const uint4*>(Vo + o);
        }
      } else if (fast) {
#pragma unroll
        for (int pass = 0; pass < 4; ++pass) {
          const int rr = pass * 8 + sub;
          if (rr < rows_ok) {
            const long long o = off + (long long)rr * ld + c8;
            b[pass * 3 + 0] = *reinterpret_cast<const uint4*>(P + o);
            b[pass * 3 + 1] = *reinterpret_cast<const uint4*>(Mo + o);
            b[pass * 3 + 2] = *reinterpret_cast<const uint4*>(Vo + o);
          }
        }
      }
      float g[32];
      load_acc(taddr + c * 32, g, zero);
      if (rows_ok == 0) continue;
      if (fast && rows_ok == 32) {
        // all rows valid (the common case): branch-free, so that the 32 independent update chains
        // of the four passes can be interleaved by the scheduler
        stage_put(stg, lane, g);
        float gg[4][8];
#pragma unroll
        for (int pass = 0; pass < 4; ++pass) {
          const int rr = pass * 8 + sub;
          const float4 ga = *stage_at(stg, rr, c8);
          const float4 gb = *stage_at(stg, rr, c8 + 4);
          gg[pass][0] = ga.x; gg[pass][1] = ga.y; gg[pass][2] = ga.z; gg[pass][3] = ga.w;
          gg[pass][4] = gb.x; gg[pass][5] = gb.y; gg[pass][6] = gb.z; gg[pass][7] = gb.w;
        }
#pragma unroll
        for (int pass = 0; pass < 4; ++pass) update8(gg[pass], b[pass * 3 + 0], b[pass * 3 + 1], b[pass * 3 + 2]);
#pragma unroll
        for (int pass = 0; pass < 4; ++pass) {
          const long long o = off + (long long)(pass * 8 + sub) * ld + c8;
          *reinterpret_cast<uint4*>(Mo + o) = b[pass * 3 + 1];
          *reinterpret_cast<uint4*>(Vo + o) = b[pass * 3 + 2];
          *reinterpret_cast<uint4*>(P + o) = b[pass * 3 + 0];
        }
        __syncwarp();
      } else if (fast) {
        stage_put(stg, lane, g);
#pragma unroll
        for (int pass = 0; pass < 4; ++pass) {
          const int rr = pass * 8 + sub;
          if (rr < rows_ok) {
            const long long o = off + (long long)rr * ld + c8;
            const float4 ga = *stage_at(stg, rr, c8);
            const float4 gb = *stage_at(stg, rr, c8 + 4);
            const float gg[8] = {ga.x, ga.y, ga.z, ga.w, gb.x, gb.y, gb.z, gb.w};
            update8(gg, b[pass * 3 + 0], b[pass * 3 + 1], b[pass * 3 + 2]);
            *reinterpret_cast<uint4*>(Mo + o) = b[pass * 3 + 1];
            *reinterpret_cast<uint4*>(Vo + o) = b[pass * 3 + 2];
            *reinterpret_cast<uint4*>(P + o) = b[pass * 3 + 0];
          }
        }
        __syncwarp();
      } else if (row_ok) {
        const long long o = off + (long long)lane * ld;
        for (int i = 0; i < ncols; ++i) {
          const float gi = g[i] * alpha;
          float wi = __bfloat162float(P[o + i]);
          const float mi = beta1 * __bfloat162float(Mo[o + i]) + (1.f - beta1) * gi;
          const float vi = beta2 * __bfloat162float(Vo[o + i]) + (1.f - beta2) * gi * gi;
          wi -= lr * ((mi * rbc1) / (sqrtf(vi * rbc2) + eps) + weight_decay * wi);
          Mo[o + i] = __float2bfloat16(mi);
          Vo[o + i] = __float2bfloat16(vi);
          P[o + i] = __float2bfloat16(wi);
        }
      }
    }
  }
  __device__ __forceinline__ void tile_done(const Tile&, const GemmArgs&, int) const {}
};

// ----------------------------------------------------------------------------------------
// Epilogue 1: activation x routing probability (forward FC1).  Non-gated: out = act(x) * p.
// Gated (SwiGLU): the tile holds 128 gate columns then 128 up columns; out = silu(g) * u * p.
// Optionally keeps the pre-activation for the backward pass.
// Reference semantics: fluid/moe/forward.py:231-238,299,317 (probability applied between the
// activation and FC2).
// ----------------------------------------------------------------------------------------
struct EpiAct {
  __nv_bfloat16* act_out;
  long long ld_act;
  __nv_bfloat16* pre_out;
  long long ld_pre;
  const float* probs;
  int act_kind;
  int boxes;     // pre-activation (map 0, where it is kept) and activation (map 1) can be written by bulk stores

  // Whole tiles: one row per lane as the accumulator comes, packed into boxes of 64 columns.
  template <int BN>
  __device__ __forceinline__ void run(const Tile& t, const GemmArgs& a, uint32_t taddr, int r,
                                      bool zero, int chalf, float* stg, const CUtensorMap* maps, uint64_t* wbar,
                                      volatile int* abort_flag, int kernel_id, uint32_t& fills) const {
    const int lane = r & 31;
    const long long row = (long long)t.row_base + t.m0 + r;
    const long long row0 = row - lane;
    const bool row_ok = r < t.rows_valid;
    const int rows_ok = max(0, min(32, t.rows_valid - (r - lane)));
    const float p = (row_ok && probs) ? probs[row] : 1.0f;
    const int span = (a.gated ? BN / 2 : BN) / 2;      // output columns of this warp
    if (boxes && rows_ok == 32 && t.n_tile * 2 * span + (chalf + 1) * span <= a.N) {
      BoxStore bs(stg, lane);
      const int c0 = chalf * (span / 32), col0 = t.n_tile * 2 * span + chalf * span;
#pragma unroll 1
      for (int c = c0; c < c0 + span / 32; c += 2) {
        const int col = col0 + (c - c0) * 32;
        float v[32];
        if (a.gated) {
          // three boxes and room for one: the halves are fetched again for the activation
          if (pre_out != nullptr) {
#pragma unroll
            for (int half = 0; half < 2; ++half) {
              uint8_t* box = bs.next();
#pragma unroll
              for (int h = 0; h < 2; ++h) {
                load_acc(taddr + half * (BN / 2) + (c + h) * 32, v, zero);
                bs.put_bf16(box, h, v);
              }
              bs.send(maps, box, half * a.n_half + col, (int)row0, 0);
            }
          }
          uint8_t* box = bs.next();
#pragma unroll
          for (int h = 0; h < 2; ++h) {
            float u[32];
            load_acc(taddr + (c + h) * 32, v, zero);
            load_acc(taddr + BN / 2 + (c + h) * 32, u, zero);
#pragma unroll
            for (int i = 0; i < 32; ++i) v[i] = silu_f(v[i]) * u[i] * p;
            bs.put_bf16(box, h, v);
          }
          bs.send(maps + 1, box, col, (int)row0, 0);
        } else {
          // The pre-activation is handed over before the activation is evaluated, so that its store is under way
          // during the arithmetic; the block is fetched again for it.
          if (pre_out != nullptr) {
            uint8_t* box = bs.next();
#pragma unroll
            for (int h = 0; h < 2; ++h) {
              load_acc(taddr + (c + h) * 32, v, zero);
              bs.put_bf16(box, h, v);
            }
            bs.send(maps, box, col, (int)row0, 0);
          }
          uint8_t* abox = bs.next();
#pragma unroll
          for (int h = 0; h < 2; ++h) {
            load_acc(taddr + (c + h) * 32, v, zero);
#pragma unroll
            for (int i = 0; i < 32; ++i) v[i] = act_f(act_kind, v[i]) * p;
            bs.put_bf16(abox, h, v);
          }
          bs.send(maps + 1, abox, col, (int)row0, 0);
        }
      }
      return;
    }
    if (boxes) {
      if (lane == 0) bulk_wait_group_read<0>();     // the stage below shares the area with the boxes
      __syncwarp();
    }
    if (a.gated) {
      const int c_first = chalf * (BN / 128), c_last = (chalf + 1) * (BN / 128);
#pragma unroll 1
      for (int c = c_first; c < c_last; ++c) {
        const int col = t.n_tile * (BN / 2) + c * 32;
        if (col >= a.N) break;
        float g[32], u[32];
        load_acc(taddr + c * 32, g, zero);
        load_acc(taddr + BN / 2 + c * 32, u, zero);
        if (rows_ok == 0) continue;
        const int ncols = min(32, a.N - col);
        if (pre_out) {
          put_block_bf16(stg, lane, g, rows_ok, row_ok, pre_out + row0 * ld_pre + col, ld_pre, ncols);
          put_block_bf16(stg, lane, u, rows_ok, row_ok, pre_out + row0 * ld_pre + a.n_half + col, ld_pre, ncols);
        }
#pragma unroll
        for (int i = 0; i < 32; ++i) g[i] = silu_f(g[i]) * u[i] * p;
        put_block_bf16(stg, lane, g, rows_ok, row_ok, act_out + row0 * ld_act + col, ld_act, ncols);
      }
    } else {
      const int c_first = chalf * (BN / 64), c_last = (chalf + 1) * (BN / 64);
#pragma unroll 1
      for (int c = c_first; c < c_last; ++c) {
        const int col = t.n_tile * BN + c * 32;
        if (col >= a.N) break;
        float v[32];
        load_acc(taddr + c * 32, v, zero);
        if (rows_ok == 0) continue;
        const int ncols = min(32, a.N - col);
        if (pre_out) put_block_bf16(stg, lane, v, rows_ok, row_ok, pre_out + row0 * ld_pre + col, ld_pre, ncols);
#pragma unroll
        for (int i = 0; i < 32; ++i) v[i] = act_f(act_kind, v[i]) * p;
        put_block_bf16(stg, lane, v, rows_ok, row_ok, act_out + row0 * ld_act + col, ld_act, ncols);
      }
    }
  }
  __device__ __forceinline__ void tile_done(const Tile&, const GemmArgs&, int) const {}
};

// ----------------------------------------------------------------------------------------
// Epilogue 3: backward of (act x prob), fused after dActW = dY * W2^T.
//   a = act(pre); dprob_partial[row, n_tile, half] = sum_cols(acc * a); dpre = acc * p * act'(pre)
//   gated: a = silu(g) * u; dg = acc * p * u * silu'(g); du = acc * p * silu(g)
// Partial sums per N tile and per column half (two epilogue warps share a row) keep the
// probability gradient deterministic (no atomics): dprobs_partial is [rows, n_tiles, 2].
// Reference math: fluid/moe/backward.py:341-356,1046-1061.
// ----------------------------------------------------------------------------------------
struct EpiDAct {
  const __nv_bfloat16* pre_in;
  long long ld_pre_in;
  __nv_bfloat16* dpre;
  long long ld_dpre;
  const float* probs;
  float* dprobs_partial;  // [rows, n_tiles, 2]
  int n_tiles;
  int act_kind;
  int gated;   // activation is SwiGLU: pre_in / dpre hold [gate | up] halves `n_half` apart
  int n_half;
  int boxes;   // pre-activation (map 0) and its gradient (map 1) can be moved by bulk tensor copies

  // Whole blocks: boxes of 32 rows x 32 columns of the pre-activation (gate and up) are copied in, turned
  // into the gradient in place one row per lane, which is the accumulator's own layout, and copied out.  Two
  // sets of boxes alternate, as in the optimizer epilogue.
  // Against loads and stores from registers around a trip of the accumulator through shared memory:
  // SwiGLU 8 x 1024 rows, 4096 -> 14336, 0.80 -> 0.78 ms; 64 x 768 rows, 2048 -> 1408, 316 -> 292 us; GELU 64 x
  // 1024 rows, 2048 -> 1024, 300 -> 269 us (437 with the error function evaluated twice).
  static constexpr int kBox = 32 * 64;
  static constexpr int kWarpBytes = 2 * 2 * kBox;
  template <int BN>
  __device__ __forceinline__ bool whole(const Tile& t, const GemmArgs& a, int r, int chalf) const {
    return boxes && t.rows_valid - (r & ~31) >= 32 && t.n_tile * BN + (chalf + 1) * (BN / 2) <= a.N;
  }
  __device__ __forceinline__ void load_set(const CUtensorMap* maps, uint8_t* set, uint64_t* bar, int col,
                                           int row) const {
    const int n = gated ? 2 : 1;
    mbar_expect_tx(bar, n * kBox);
    for (int i = 0; i < n; ++i) tma_load_3d(set + i * kBox, maps, bar, col + i * n_half, row, 0);
  }
  template <int BN>
  __device__ __forceinline__ void fetch(const Tile& t, const GemmArgs& a, int r, int chalf, float* stg,
                                        const CUtensorMap* maps, uint64_t* wbar) const {
    if (!whole<BN>(t, a, r, chalf)) return;
    fence_proxy_async_smem();         // what this warp stored in its area by other means is done
    __syncwarp();
    if ((r & 31) == 0) {
      bulk_wait_group_read<0>();      // the last tile's boxes have left
      const int col = t.n_tile * BN + chalf * (BN / 2);
      uint8_t* sets = reinterpret_cast<uint8_t*>(stg);
#pragma unroll
      for (int i = 0; i < 2; ++i) load_set(maps, sets + i * 2 * kBox, wbar + i, col + 32 * i, t.row_base + t.m0 + r);
    }
    __syncwarp();
  }

  template <int BN>
  __device__ __forceinline__ void run(const Tile& t, const GemmArgs& a, uint32_t taddr, int r,
                                      bool zero, int chalf, float* stg, const CUtensorMap* maps, uint64_t* wbar,
                                      volatile int* abort_flag, int kernel_id, uint32_t& fills) const {
    const int lane = r & 31;
    const long long row = (long long)t.row_base + t.m0 + r;
    const long long row0 = row - lane;
    const bool row_ok = r < t.rows_valid;
    const int rows_ok = max(0, min(32, t.rows_valid - (r - lane)));
    const float p = (row_ok && probs) ? probs[row] : 1.0f;
    float dp = 0.f;
    const int c_first = chalf * (BN / 64), c_last = (chalf + 1) * (BN / 64);
    if (whole<BN>(t, a, r, chalf)) {
      uint8_t* const sets = reinterpret_cast<uint8_t*>(stg);
      const int swz = (lane >> 1) & 3;
      const int boxes_of_set = gated ? 2 : 1;
      float d4[4] = {0.f, 0.f, 0.f, 0.f};      // four partial sums of the row
#pragma unroll 1
      for (int k = 0; k < BN / 64; ++k) {
        const int col = t.n_tile * BN + (c_first + k) * 32;
        uint8_t* const set = sets + (k & 1) * 2 * kBox;
        float v[32];
        load_acc(taddr + (c_first + k) * 32, v, zero);
        if (lane == 0 && k > 0 && k + 1 < BN / 64) {
          // the set of the block before has left: refill it for the block after this one
          bulk_wait_group_read<0>();
          load_set(maps, sets + ((k + 1) & 1) * 2 * kBox, wbar + ((k + 1) & 1), col + 32, (int)row0);
        }
        __syncwarp();
        if (!mbar_wait(wbar + (k & 1), box_parity<BN / 64>(k, fills), a.timeout_ns, abort_flag)) {
          if (lane == 0) report_status(a.status, kStatusMbarTimeout, kernel_id, 510 + k, 0, 0);
          return;
        }
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          uint4* const at = reinterpret_cast<uint4*>(set + lane * 64 + ((j ^ swz) << 4));
          const uint4 rg = at[0];
          const uint32_t wg[4] = {rg.x, rg.y, rg.z, rg.w};
          float og[8], ou[8];
          if (gated) {
            const uint4 ru = at[kBox / 16];
            const uint32_t wu[4] = {ru.x, ru.y, ru.z, ru.w};
#pragma unroll
            for (int i = 0; i < 8; ++i) {
              // bf16 -> fp32 is a 16-bit shift of the bit pattern
              const float gi = __uint_as_float((i & 1) ? (wg[i >> 1] & 0xffff0000u) : (wg[i >> 1] << 16));
              const float ui = __uint_as_float((i & 1) ? (wu[i >> 1] & 0xffff0000u) : (wu[i >> 1] << 16));
              const float x = v[8 * j + i];
              const float sg = sigmoid_f(gi);          // one sigmoid serves silu and its derivative
              const float sl = gi * sg;
              d4[i & 3] += x * sl * ui;
              const float da = x * p;
              og[i] = da * ui * (sg * (1.0f + gi * (1.0f - sg)));
              ou[i] = da * sl;
            }
            at[kBox / 16] = make_uint4(pack_bf16x2(ou[0], ou[1]), pack_bf16x2(ou[2], ou[3]), pack_bf16x2(ou[4], ou[5]),
                                       pack_bf16x2(ou[6], ou[7]));
          } else {
            auto plain = [&](auto kind) {
#pragma unroll
              for (int i = 0; i < 8; ++i) {
                const float xi = __uint_as_float((i & 1) ? (wg[i >> 1] & 0xffff0000u) : (wg[i >> 1] << 16));
                const float x = v[8 * j + i];
                float y, dy;
                act_dact<decltype(kind)::value>(xi, y, dy);
                d4[i & 3] += x * y;
                og[i] = x * p * dy;
              }
            };
            if (act_kind == FM_ACT_GELU) plain(Kind<FM_ACT_GELU>{});
            else if (act_kind == FM_ACT_SILU) plain(Kind<FM_ACT_SILU>{});
            else plain(Kind<FM_ACT_NONE>{});
          }
          at[0] = make_uint4(pack_bf16x2(og[0], og[1]), pack_bf16x2(og[2], og[3]), pack_bf16x2(og[4], og[5]),
                             pack_bf16x2(og[6], og[7]));
        }
        fence_proxy_async_smem();
        __syncwarp();
        if (lane == 0) {
          for (int i = 0; i < boxes_of_set; ++i)
            tma_store_3d(maps + 1, set + i * kBox, col + i * n_half, (int)row0, 0);
          bulk_commit_group();
        }
      }
      __syncwarp();
      ++fills;
      dp = (d4[0] + d4[1]) + (d4[2] + d4[3]);
      if (dprobs_partial) dprobs_partial[(row * n_tiles + t.n_tile) * 2 + chalf] = dp;
      return;
    }
    if (boxes) {
      if (lane == 0) bulk_wait_group_read<0>();     // the stage below shares the area with the boxes
      __syncwarp();
    }
#pragma unroll 1
    for (int c = c_first; c < c_last; ++c) {
      const int col = t.n_tile * BN + c * 32;
      if (col >= a.N) break;
      float v[32];
      load_acc(taddr + c * 32, v, zero);
      if (rows_ok == 0) continue;
      const int ncols = min(32, a.N - col);
      if (gated) {
        float g[32], u[32];
        get_block_bf16(stg, lane, g, rows_ok, row_ok, pre_in + row0 * ld_pre_in + col, ld_pre_in, ncols);
        get_block_bf16(stg, lane, u, rows_ok, row_ok, pre_in + row0 * ld_pre_in + n_half + col, ld_pre_in, ncols);
#pragma unroll
        for (int i = 0; i < 32; ++i) {
          const float sg = sigmoid_f(g[i]);          // one sigmoid serves silu and its derivative
          const float s = g[i] * sg;
          dp += v[i] * s * u[i];
          const float da = v[i] * p;
          g[i] = da * u[i] * (sg * (1.0f + g[i] * (1.0f - sg)));
          u[i] = da * s;
        }
        put_block_bf16(stg, lane, g, rows_ok, row_ok, dpre + row0 * ld_dpre + col, ld_dpre, ncols);
        put_block_bf16(stg, lane, u, rows_ok, row_ok, dpre + row0 * ld_dpre + n_half + col, ld_dpre, ncols);
      } else {
        float x[32];
        get_block_bf16(stg, lane, x, rows_ok, row_ok, pre_in + row0 * ld_pre_in + col, ld_pre_in, ncols);
#pragma unroll
        for (int i = 0; i < 32; ++i) {
          dp += v[i] * act_f(act_kind, x[i]);
          x[i] = v[i] * p * dact_f(act_kind, x[i]);
        }
        put_block_bf16(stg, lane, x, rows_ok, row_ok, dpre + row0 * ld_dpre + col, ld_dpre, ncols);
      }
    }
    if (row_ok && dprobs_partial) dprobs_partial[(row * n_tiles + t.n_tile) * 2 + chalf] = dp;
  }
  __device__ __forceinline__ void tile_done(const Tile&, const GemmArgs&, int) const {}
};

// ----------------------------------------------------------------------------------------
// Epilogue 2: scatter rows to their owners (FC2 + combine).  Row R of the result is written
// as bf16 to dst_base[dst_rank[R]] + dst_row[R] * ld_dst, which may be another GPU's buffer
// mapped over NVLink (plain 16-byte peer stores, 64 contiguous bytes per row per instruction
// group).  After a tile, each destination's arrival counter grows by the number of rows the
// tile sent it; the owner waits until its counter equals rows_expected * n_tiles * 2 (each of
// the two epilogue warps that share a row reports its half).  Replaces the combine all-to-all
// rounds of fluid/moe/forward.py:903-948.
// ----------------------------------------------------------------------------------------
struct EpiScatter {
  __nv_bfloat16* const* dst_base;
  const int* dst_rank;
  const int* dst_row;
  long long ld_dst;
  int* const* dst_flags;  // per destination rank: pointer to the counter this rank bumps
  int num_ranks;
  // One fp32 per row that rides along (the routing-probability gradient on the way back to the
  // token owner, which the reference sends through a separate small all-to-all,
  // fluid/layer/transformer.py:526-538): stored by the first column tile's first warp group,
  // before the release that publishes the row.
  const float* row_aux;
  float* const* row_aux_dst;

  template <int BN>
  __device__ __forceinline__ void run(const Tile& t, const GemmArgs& a, uint32_t taddr, int r,
                                      bool zero, int chalf, float* stg, const CUtensorMap* maps, uint64_t* wbar,
                                      volatile int* abort_flag, int kernel_id, uint32_t& fills) const {
    const int lane = r & 31;
    const long long row = (long long)t.row_base + t.m0 + r;
    const bool row_ok = r < t.rows_valid;
    int rank = -1;
    long long drow = 0;
    if (row_ok) {
      rank = dst_rank[row];
      drow = dst_row[row];
    }
    if (row_aux != nullptr && t.n_tile == 0 && chalf == 0 && rank >= 0)
      row_aux_dst[rank][drow] = row_aux[row];
    __nv_bfloat16* base = rank >= 0 ? dst_base[rank] + drow * ld_dst : nullptr;
    const bool fast = (ld_dst & 7) == 0 &&
                      __all_sync(0xffffffffu, base == nullptr || aligned16(base));
#pragma unroll 1
    for (int c = chalf * (BN / 64); c < (chalf + 1) * (BN / 64); ++c) {
      const int col = t.n_tile * BN + c * 32;
      if (col >= a.N) break;
      float v[32];
      load_acc(taddr + c * 32, v, zero);
      const int ncols = min(32, a.N - col);
      if (fast && ncols == 32 && (col & 7) == 0) {
        staged_store_bf16_scatter(stg, lane, v, base ? base + col : nullptr);
      } else if (base != nullptr) {
        store_row_bf16(base + col, v, ncols);
      }
    }
    if (dst_flags != nullptr) __threadfence_system();
  }
  // Called by every epilogue thread after the tile's stores; `r` is the thread's row in the
  // tile.  Each warp aggregates its 32 rows by destination, so no cross-warp barrier is needed.
  __device__ __forceinline__ void tile_done(const Tile& t, const GemmArgs& a, int r) const {
    if (dst_flags == nullptr) return;
    const long long row = (long long)t.row_base + t.m0 + r;
    const int rank = r < t.rows_valid ? dst_rank[row] : -1;
    __syncwarp();
    const unsigned peers = __match_any_sync(0xffffffffu, rank);
    const int leader = __ffs(peers) - 1;
    if ((int)(threadIdx.x & 31) == leader && rank >= 0)
      flag_release_add(dst_flags[rank], __popc(peers));
  }
};

// ----------------------------------------------------------------------------------------
// Epilogue 4: scatter COLUMN blocks to their owners (QKV projection + SP->HP exchange, and
// out-projection input gradient + SP->HP).  Columns [p*cpr, (p+1)*cpr) of every result row
// belong to rank p; they are stored as bf16 into rank p's buffer at row (dst_row_offset + row),
// column (col - p*cpr), leading dimension dst_ld -- the position the all-to-all would have put
// them (fluid/core/comm.py:162-209).  Each warp adds the rows it delivered, once per 32-column
// chunk, to the destination's counter for this source; the owner waits for
// rows * (cpr / 32) per source.
// ----------------------------------------------------------------------------------------
struct EpiColScatter {
  __nv_bfloat16* const* dst_base;
  int cols_per_rank;
  long long dst_ld;
  long long dst_row_offset;
  int* const* dst_flags;

  template <int BN>
  __device__ __forceinline__ void run(const Tile& t, const GemmArgs& a, uint32_t taddr, int r,
                                      bool zero, int chalf, float* stg, const CUtensorMap* maps, uint64_t* wbar,
                                      volatile int* abort_flag, int kernel_id, uint32_t& fills) const {
    const int lane = r & 31;
    const long long row0 = (long long)t.row_base + t.m0 + (r - lane);
    const bool row_ok = r < t.rows_valid;
    const int rows_ok = max(0, min(32, t.rows_valid - (r - lane)));
    int pend_rank = -1, pend_cnt = 0;
#pragma unroll 1
    for (int c = chalf * (BN / 64); c < (chalf + 1) * (BN / 64); ++c) {
      const int col = t.n_tile * BN + c * 32;
      if (col >= a.N) break;
      float v[32];
      load_acc(taddr + c * 32, v, zero);
      if (rows_ok == 0) continue;
      const int rank = col / cols_per_rank;
      const int cin = col - rank * cols_per_rank;
      __nv_bfloat16* base = dst_base[rank] + (dst_row_offset + row0) * dst_ld + cin;
      put_block_bf16(stg, lane, v, rows_ok, row_ok, base, dst_ld, min(32, a.N - col));
      if (rank != pend_rank) {
        if (pend_cnt > 0 && dst_flags != nullptr) {
          __threadfence_system();
          __syncwarp();
          if (lane == 0) flag_release_add(dst_flags[pend_rank], pend_cnt);
        }
        pend_rank = rank;
        pend_cnt = 0;
      }
      pend_cnt += rows_ok;
    }
    if (pend_cnt > 0 && dst_flags != nullptr) {
      __threadfence_system();
      __syncwarp();
      if (lane == 0) flag_release_add(dst_flags[pend_rank], pend_cnt);
    }
  }
  __device__ __forceinline__ void tile_done(const Tile&, const GemmArgs&, int) const {}
};

// ----------------------------------------------------------------------------------------
// host side
// ----------------------------------------------------------------------------------------
}  // namespace fm
extern "C" void fm_set_error(const char* msg);
namespace fm {
static void set_err(const char* msg) { fm_set_error(msg); }

// 2-D bf16 tensor map, 128-byte swizzle, box = {64 inner, box_outer}.
bool make_tmap(CUtensorMap* m, const void* ptr, long long inner, long long outer,
                      long long ld, int box_outer) {
  if ((reinterpret_cast<uintptr_t>(ptr) & 15) || ((ld * 2) & 15)) {
    set_err("TMA operand must be 16-byte aligned with a 16-byte-multiple row stride");
    return false;
  }
  cuuint64_t dims[2] = {(cuuint64_t)inner, (cuuint64_t)outer};
  cuuint64_t strides[1] = {(cuuint64_t)ld * 2};
  cuuint32_t box[2] = {64, (cuuint32_t)box_outer};
  const CUresult r = encode_tiled(m, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, ptr, dims, strides, box,
                                  CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B);
  if (r != CUDA_SUCCESS) {
    char buf[256];
    snprintf(buf, sizeof(buf), "cuTensorMapEncodeTiled failed: %d (inner=%lld outer=%lld ld=%lld)",
             (int)r, inner, outer, ld);
    set_err(buf);
    return false;
  }
  return true;
}

// 3-D view of an MN-major operand stored [outer, inner] (inner contiguous, a multiple of 64):
// dims {64, outer, inner / 64}; one box {64, 64 k-rows, nblk} lands as nblk slabs of [64 k][64 mn].
static bool make_tmap_mn3d(CUtensorMap* m, const void* ptr, long long inner, long long outer,
                           long long ld, int nblk) {
  cuuint64_t dims[3] = {64, (cuuint64_t)outer, (cuuint64_t)(inner / 64)};
  cuuint64_t strides[2] = {(cuuint64_t)ld * 2, 128};
  cuuint32_t box[3] = {64, 64, (cuuint32_t)nblk};
  const CUresult r = encode_tiled(m, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 3, ptr, dims, strides, box,
                                  CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B);
  if (r != CUDA_SUCCESS) {
    char buf[256];
    snprintf(buf, sizeof(buf), "cuTensorMapEncodeTiled (3-D) failed: %d (inner=%lld outer=%lld ld=%lld)",
             (int)r, inner, outer, ld);
    set_err(buf);
    return false;
  }
  return true;
}

// Tensor map of an epilogue output [groups][rows][cols] (row stride `ld`, group stride `gs` elements) with
// boxes of 32 rows x 128 (or 64) bytes in the swizzle of that width.  False when the addresses or strides do not
// allow it (16-byte rule).
static bool make_out_map(CUtensorMap* m, const void* ptr, bool fp32, long long cols, long long rows, long long ld,
                         long long groups, long long gs, int row_bytes = 128,
                         CUtensorMapL2promotion promotion = CU_TENSOR_MAP_L2_PROMOTION_NONE) {
  const long long es = fp32 ? 4 : 2;
  if (groups <= 1) {
    groups = 1;
    gs = (rows * ld + 7) / 8 * 8;      // never stepped
  }
  if (ptr == nullptr || (reinterpret_cast<uintptr_t>(ptr) & 15) || (ld * es) % 16 || (gs * es) % 16 ||
      cols <= 0 || rows <= 0 || ld <= 0 || gs <= 0 || rows >= (1ll << 31) || ld * es >= (1ll << 40) ||
      gs * es >= (1ll << 40))
    return false;
  cuuint64_t dims[3] = {(cuuint64_t)cols, (cuuint64_t)rows, (cuuint64_t)groups};
  cuuint64_t strides[2] = {(cuuint64_t)(ld * es), (cuuint64_t)(gs * es)};
  cuuint32_t box[3] = {(cuuint32_t)(row_bytes / es), 32, 1};
  return encode_tiled(m, fp32 ? CU_TENSOR_MAP_DATA_TYPE_FLOAT32 : CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 3, ptr, dims, strides,
                      box, row_bytes == 64 ? CU_TENSOR_MAP_SWIZZLE_64B : CU_TENSOR_MAP_SWIZZLE_128B,
                      promotion) == CUDA_SUCCESS;
}

int sm_count() {
  static int n = 0;
  if (n == 0) {
    int dev = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev);
  }
  return n;
}

template <bool A_MN, bool B_MN, int BN, class Epi, class Gate>
static int launch_one(const CUtensorMap& ta, const CUtensorMap& tb, const GemmArgs& args,
                      const Epi& epi, const Gate& gate, const OutMaps& maps, int grid, cudaStream_t stream) {
  auto kern = gemm_sm100_kernel<A_MN, B_MN, BN, Epi, Gate>;
  constexpr int smem = gemm_smem_bytes<BN, Epi>();
  static std::atomic<unsigned long long> configured{0};
  cudaError_t e = allow_smem(reinterpret_cast<const void*>(kern), smem, configured);
  if (e != cudaSuccess) {
    set_err(cudaGetErrorString(e));
    return (int)e;
  }
  kern<<<grid, kGemmThreads, smem, stream>>>(ta, tb, args, epi, gate, maps);
  e = cudaGetLastError();
  if (e != cudaSuccess) {
    set_err(cudaGetErrorString(e));
    return (int)e;
  }
  return 0;
}

// Workspace of the dynamic tile order, one for a stream: launches on one stream run one
// after another, so they can share claim counters (used in rotation; a launch zeroes the counter
// that comes up half a rotation later) and the log (entries carry the launch's epoch).  A stream
// that is being captured into a graph keeps the static order, because a replay would repeat the
// epoch of the capture, and so do streams beyond those that the table knows.
struct SchedWorkspace {
  int* ctrs = nullptr;
  unsigned long long* log = nullptr;
  size_t log_entries = 0;
  unsigned int epoch = 0;
};
constexpr int kSchedCounters = 64;

static bool sched_dynamic_enabled() {
  static int on = -1;
  if (on < 0) {
    const char* e = getenv("FLUIDMOE_GEMM_DYNAMIC_TILES");
    on = (e == nullptr || e[0] != '0') ? 1 : 0;
  }
  return on == 1;
}

// Fills the scheduler fields of `args` for a launch of `pairs` CTA pairs over at most `tiles`
// tiles; leaves them empty (static order) when the dynamic order is off or cannot be used.
static void sched_prepare(GemmArgs& args, int pairs, long long tiles, cudaStream_t stream) {
  args.sched_ctr = nullptr;
  args.sched_ctr_reset = nullptr;
  args.sched_log = nullptr;
  args.sched_cap = 0;
  args.sched_epoch = 0;
  if (!sched_dynamic_enabled() || tiles <= pairs || tiles > (1ll << 24)) return;
  static StreamTable<SchedWorkspace> table;
  std::lock_guard<std::mutex> lock(table.mu);
  SchedWorkspace* state = nullptr;
  if (!table.find(stream, &state) || state == nullptr) return;
  SchedWorkspace& ws = *state;
  if (ws.ctrs == nullptr) {
    if (cudaMalloc(&ws.ctrs, kSchedCounters * sizeof(int)) != cudaSuccess) {
      (void)cudaGetLastError();
      ws.ctrs = nullptr;
      return;
    }
    cudaMemsetAsync(ws.ctrs, 0, kSchedCounters * sizeof(int), stream);
  }
  // A pair can claim every tile but the other pairs' first ones, and one claim past the end.
  const size_t cap_per_pair = (size_t)(tiles + 2);
  const size_t need = cap_per_pair * (size_t)pairs;
  if (need * sizeof(unsigned long long) > ((size_t)64 << 20)) return;   // very many tiles: static order
  if (need > ws.log_entries) {
    // The old log may still be read by a launch in flight on this stream: it is not freed (logs
    // only grow a few times, while the largest problem of a model is met for the first time).
    unsigned long long* fresh = nullptr;
    if (cudaMalloc(&fresh, need * sizeof(unsigned long long)) != cudaSuccess) {
      (void)cudaGetLastError();
      return;
    }
    cudaMemsetAsync(fresh, 0, need * sizeof(unsigned long long), stream);
    ws.log = fresh;
    ws.log_entries = need;
  }
  if (++ws.epoch == 0) ws.epoch = 1;
  args.sched_ctr = ws.ctrs + ws.epoch % kSchedCounters;
  args.sched_ctr_reset = ws.ctrs + (ws.epoch + kSchedCounters / 2) % kSchedCounters;
  args.sched_log = ws.log;
  args.sched_cap = (int)cap_per_pair;
  args.sched_epoch = ws.epoch;
}

template <bool A_MN, bool B_MN, class Epi, class Gate>
static int launch_pair(const CUtensorMap& ta, const CUtensorMap& tb, const GemmArgs& args_in,
                       const Epi& epi, const Gate& gate, const OutMaps& maps, int grid, cudaStream_t stream) {
  auto kern = gemm2_sm100_kernel<A_MN, B_MN, Epi, Gate>;
  constexpr int smem = gemm2_smem_bytes<Epi>();
  static std::atomic<unsigned long long> configured{0};
  cudaError_t e = allow_smem(reinterpret_cast<const void*>(kern), smem, configured);
  if (e != cudaSuccess) {
    set_err(cudaGetErrorString(e));
    return (int)e;
  }
  // The kernel is persistent: never launch more pairs than can be resident at once (pairs must
  // sit on two SMs of one GPC, so this can be fewer than SMs / 2).
  static int max_pairs = 0;
  if (max_pairs == 0) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(sm_count() & ~1);
    cfg.blockDim = dim3(kGemmThreads);
    cfg.dynamicSmemBytes = smem;
    cudaLaunchAttribute attr;
    attr.id = cudaLaunchAttributeClusterDimension;
    attr.val.clusterDim.x = 2;
    attr.val.clusterDim.y = 1;
    attr.val.clusterDim.z = 1;
    cfg.attrs = &attr;
    cfg.numAttrs = 1;
    int n = 0;
    if (cudaOccupancyMaxActiveClusters(&n, kern, &cfg) != cudaSuccess || n <= 0) {
      (void)cudaGetLastError();
      n = sm_count() / 2 - 2;
    }
    max_pairs = n;
  }
  grid &= ~1;   // whole CTA pairs
  if (grid > 2 * max_pairs) grid = 2 * max_pairs;
  if (grid < 2) grid = 2;
  GemmArgs args = args_in;
  sched_prepare(args, grid / 2, args_in.sched_cap, stream);   // sched_cap arrives as the tile bound
  kern<<<grid, kGemmThreads, smem, stream>>>(ta, tb, args, epi, gate, maps);
  e = cudaGetLastError();
  if (e != cudaSuccess) {
    set_err(cudaGetErrorString(e));
    return (int)e;
  }
  return 0;
}

template <class Epi, class Gate>
static int dispatch_shape(const FmGemmDesc* d, const CUtensorMap& ta, const CUtensorMap& tb,
                          const GemmArgs& args, const Epi& epi, const Gate& gate, const OutMaps& maps, int grid,
                          cudaStream_t s) {
  const bool amn = d->a_mn != 0, bmn = d->b_mn != 0;
  if (d->cta_pair && d->bn == 256) {
    if (!amn && !bmn) return launch_pair<false, false>(ta, tb, args, epi, gate, maps, grid, s);
    if (!amn && bmn) return launch_pair<false, true>(ta, tb, args, epi, gate, maps, grid, s);
    if (amn && bmn) return launch_pair<true, true>(ta, tb, args, epi, gate, maps, grid, s);
  }
  if (d->bn == 256) {
    if (!amn && !bmn) return launch_one<false, false, 256>(ta, tb, args, epi, gate, maps, grid, s);
    if (!amn && bmn) return launch_one<false, true, 256>(ta, tb, args, epi, gate, maps, grid, s);
    if (amn && bmn) return launch_one<true, true, 256>(ta, tb, args, epi, gate, maps, grid, s);
  } else if (d->bn == 128) {
    if (!amn && !bmn) return launch_one<false, false, 128>(ta, tb, args, epi, gate, maps, grid, s);
    if (!amn && bmn) return launch_one<false, true, 128>(ta, tb, args, epi, gate, maps, grid, s);
    if (amn && bmn) return launch_one<true, true, 128>(ta, tb, args, epi, gate, maps, grid, s);
  }
  set_err("unsupported operand-major / tile combination");
  return -2;
}

// Stored products (sizes known here, no gate) of few tiles leave the CTA pairs and their 256 x 256 tiles.
// Where tiles of 128 x 128 go round once, one a CTA: pairs would leave most SMs idle.  Pairs, single CTAs with 128 x 256 and
// with 128 x 128, us: 2048 x 1024, K = 1024 18.4, 16.4 and 14.3, K = 4096 32.8, 32.8 and 28.7, K = 8192 51.2, 57.3
// and 45.1; 512 x 512 x 512 14.3, 12.3 and 12.3; 256 x 1024, K = 2048 20.5, 20.5 and 18.4.  In two rounds they lose, since the operands of a
// small tile take as long as those of a large one: 2560 x 1024, K = 1024 18.4, 16.4 and 18.4, K = 4096 32.8, 32.8 and 45.1.
// Short contractions in up to two rounds of pairs take single CTAs with 128 x 256, which start 2 us sooner than a pair:
// 2048 x 3072, K = 512 20.4 and 16.4, K = 1024 24.6 and 22.5; 4096 x 2304 20.5 and 18.4, 24.6 and 24.6; beyond, 4096 x 3072, K = 1024 30.7
// and 30.7, with K = 2048 47.1 and 49.2.
static void small_shape(FmGemmDesc* d) {
  if (!d->cta_pair || d->bn != 256 || d->epi != FM_EPI_STORE || d->gated || d->group_rows != nullptr ||
      d->group_offs != nullptr || d->group_b != nullptr || d->gate_flags != nullptr || d->n_rotate || d->k_rotate)
    return;
  const long long rows = d->mode == 1 ? d->M : d->uniform_rows, k = d->mode == 1 ? d->uniform_rows : d->K;
  if (rows <= 0) return;
  const int ctas = d->max_ctas > 0 && d->max_ctas < sm_count() ? d->max_ctas : sm_count();
  auto tiles = [&](int m, int n) { return d->num_groups * ((rows + m - 1) / m) * ((d->N + n - 1) / n); };
  if (tiles(128, 128) <= ctas) d->bn = 128;
  else if (k <= 1024 && tiles(256, 256) <= ctas && d->max_ctas <= 0) d->cta_pair = 0;
}

template <class Epi>
static int dispatch_gate(const FmGemmDesc* d, const CUtensorMap& ta, const CUtensorMap& tb,
                         const GemmArgs& args, const Epi& epi, const OutMaps& maps, int grid, cudaStream_t s) {
  if (d->gate_flags != nullptr && d->gate_k_blocks_per_src > 0) {
    GateKSource g{d->gate_flags, d->gate_k_blocks_per_src, d->gate_blocks_per_group,
                  d->gate_expected > 0 ? d->gate_expected : 1};
    return dispatch_shape(d, ta, tb, args, epi, g, maps, grid, s);
  }
  if (d->gate_flags != nullptr) {
    GateRowBlockFlags g{d->gate_flags, d->gate_group_base, d->gate_blocks_per_group,
                        d->gate_expected};
    return dispatch_shape(d, ta, tb, args, epi, g, maps, grid, s);
  }
  return dispatch_shape(d, ta, tb, args, epi, GateNone{}, maps, grid, s);
}

}  // namespace fm


extern "C" int fm_gemm_launch(const FmGemmDesc* d, cudaStream_t stream) {
  using namespace fm;
  if (d->bn != 128 && d->bn != 256) {
    set_err("bn must be 128 or 256");
    return -1;
  }
  if (d->gated && d->bn != 256) {
    set_err("gated tiles need bn == 256");
    return -1;
  }
  if (d->mode == 1 && !(d->a_mn && d->b_mn)) {
    set_err("grouped-K mode needs both operands stored [rows, M] / [rows, N]");
    return -1;
  }
  if (d->gated && d->n_half % 8 != 0) {
    set_err("gated layout needs the up half to start at a multiple of 8 columns");
    return -1;
  }
  if (d->mode == 0 && d->K % 8 != 0) {
    set_err("K must be a multiple of 8");
    return -1;
  }
  if (d->mode == 0 && d->num_groups > 1 && d->K % kBK != 0) {
    set_err("grouped GEMM needs K to be a multiple of 64");
    return -1;
  }
  if (gemm_few_applies(d)) return gemm_few_launch(d, stream);
  FmGemmDesc by_size = *d;
  small_shape(&by_size);
  d = &by_size;
  CUtensorMap ta, tb;
  // One 3-D box per MN-major tile when every tile starts on a 64-element boundary of a
  // 64-multiple inner extent; otherwise 64-wide 2-D boxes.
  const bool a3 = d->a_mn && d->a_inner % 64 == 0 && (d->mode == 1 || d->group_offs == nullptr) &&
                  (d->mode == 1 || d->uniform_rows % 64 == 0);
  const bool b3 = d->b_mn && d->b_inner % 64 == 0 && (!d->gated || d->n_half % 64 == 0);
  const bool mn3d = (!d->a_mn || a3) && (!d->b_mn || b3) && (d->a_mn || d->b_mn) &&
                    ((uintptr_t)d->A % 16 == 0) && ((uintptr_t)d->B % 16 == 0) && d->lda % 8 == 0 &&
                    d->ldb % 8 == 0;
  // The CTA-pair kernel fetches MN-major operands only through 3-D boxes.
  FmGemmDesc dd = *d;
  if (dd.cta_pair && (dd.bn != 256 || ((dd.a_mn || dd.b_mn) && !mn3d) || (dd.mode == 0 && dd.a_mn)))
    dd.cta_pair = 0;
  d = &dd;
  // A: K-major -> box {64 k, 128 rows}; MN-major -> box {64 rows, 64 k}
  if (d->a_mn && mn3d) {
    if (!make_tmap_mn3d(&ta, d->A, d->a_inner, d->a_outer, d->lda, kBM / 64)) return -3;
  } else if (!make_tmap(&ta, d->A, d->a_inner, d->a_outer, d->lda, d->a_mn ? 64 : 128)) {
    return -3;
  }
  // B: K-major -> box {64 k, 128 n}; MN-major -> box {64 n, 64 k}
  if (d->b_mn && mn3d) {
    if (!make_tmap_mn3d(&tb, d->B, d->b_inner, d->b_outer, d->ldb,
                        (d->gated || d->cta_pair) ? d->bn / 128 : d->bn / 64))
      return -3;
  } else if (!make_tmap(&tb, d->B, d->b_inner, d->b_outer, d->ldb, d->b_mn ? 64 : 128)) {
    return -3;
  }

  GemmArgs args;
  memset(&args, 0, sizeof(args));
  args.mode = d->mode;
  args.num_groups = d->num_groups;
  args.M = d->M;
  args.N = d->N;
  args.K = d->K;
  args.uniform_rows = d->uniform_rows;
  args.group_rows = d->group_rows;
  args.group_offs = d->group_offs;
  args.group_b = d->group_b;
  args.b_group_stride = d->b_group_stride;
  args.gated = d->gated;
  args.n_half = d->n_half;
  args.swizzle_m = d->swizzle_m;
  args.mn3d = mn3d ? 1 : 0;
  args.n_rotate = d->n_rotate;
  args.k_rotate = d->k_rotate;
  args.timeout_ns = d->timeout_ns ? d->timeout_ns : 4000000000ull;
  args.status = d->status;
  args.wait_ns = d->wait_ns;

  int grid = sm_count();
  if (d->max_ctas > 0 && d->max_ctas < grid) grid = d->max_ctas;
  // Do not launch more CTAs than tiles when the tile count is known on the host.
  {
    const int npt = d->gated ? d->bn / 2 : d->bn;
    const long long nt = (d->N + npt - 1) / npt;
    const int tm = d->cta_pair ? 2 * kBM : kBM;
    if (d->group_rows == nullptr) {
      const long long mt = d->mode == 0 ? (d->uniform_rows + tm - 1) / tm : (d->M + tm - 1) / tm;
      const long long tiles = nt * mt * d->num_groups * (d->cta_pair ? 2 : 1);
      if (tiles < grid) grid = (int)(tiles > 0 ? tiles : 1);
    }
    // Upper bound of the tile count for the dynamic tile order of the CTA-pair kernel (the launcher
    // replaces it by the log's row length).  With row counts in device memory the rows of A bound it.
    long long bound;
    if (d->mode == 1)
      bound = nt * ((d->M + tm - 1) / tm) * d->num_groups;
    else if (d->group_rows == nullptr)
      bound = nt * ((d->uniform_rows + tm - 1) / tm) * d->num_groups;
    else
      bound = nt * (d->a_outer / tm + d->num_groups);
    args.sched_cap = (int)(bound < (1ll << 30) ? bound : 0);
  }

  OutMaps maps;
  memset(&maps, 0, sizeof(maps));
  switch (d->epi) {
    case FM_EPI_STORE: {
      EpiStore e{d->C, d->ldc, d->c_group_stride, d->out_fp32, d->accumulate,
                 d->alpha == 0.f ? 1.0f : d->alpha, 0, d->alpha_dev,
                 reinterpret_cast<const __nv_bfloat16*>(d->residual), d->ld_residual};
      if (d->residual != nullptr && (d->out_fp32 || d->accumulate || d->mode != 0)) {
        set_err("a residual goes with a bf16 result that does not accumulate");
        return -1;
      }
      if (d->accumulate && !d->out_fp32 && d->mode == 0) {
        e.accumulate = 0;
        e.residual = reinterpret_cast<const __nv_bfloat16*>(d->C);
        e.ld_residual = d->ldc;
      }
      // Other sums that a store accumulates into are read first and keep the stores from registers; so does a
      // residual off 16 bytes.
      if (!e.accumulate &&
          (e.residual == nullptr || (e.ld_residual % 8 == 0 && (reinterpret_cast<uintptr_t>(e.residual) & 15) == 0)))
        e.boxes = make_out_map(&maps.m[0], d->C, d->out_fp32 != 0, d->N,
                               d->mode == 0 ? (d->a_mn ? d->a_inner : d->a_outer) : d->M, d->ldc,
                               d->mode == 0 ? 1 : d->num_groups, d->c_group_stride);
      return dispatch_gate(d, ta, tb, args, e, maps, grid, stream);
    }
    case FM_EPI_ACT: {
      EpiAct e{reinterpret_cast<__nv_bfloat16*>(d->act_out), d->ld_act,
               reinterpret_cast<__nv_bfloat16*>(d->pre_out), d->ld_pre, d->probs, d->act_kind, 0};
      const long long rows = d->a_mn ? d->a_inner : d->a_outer;
      // a copy starts on 16 bytes: the up half at a multiple of 8 columns
      e.boxes = (!d->gated || d->n_half % 8 == 0) &&
                make_out_map(&maps.m[1], d->act_out, false, d->N, rows, d->ld_act, 1, 0) &&
                (d->pre_out == nullptr ||
                 make_out_map(&maps.m[0], d->pre_out, false, d->gated ? d->n_half + d->N : d->N, rows, d->ld_pre, 1, 0));
      return dispatch_gate(d, ta, tb, args, e, maps, grid, stream);
    }
    case FM_EPI_DACT: {
      const int nt = (d->N + d->bn - 1) / d->bn;
      EpiDAct e{reinterpret_cast<const __nv_bfloat16*>(d->pre_in), d->ld_pre_in,
                reinterpret_cast<__nv_bfloat16*>(d->C), d->ldc, d->probs, d->dprobs, nt,
                d->act_kind, d->gated, d->n_half, 0};
      const long long rows = d->a_mn ? d->a_inner : d->a_outer, cols = d->gated ? d->n_half + d->N : d->N;
      // a copy starts on 16 bytes: the up half at a multiple of 8 columns
      e.boxes = (!d->gated || d->n_half % 8 == 0) &&
                make_out_map(&maps.m[0], d->pre_in, false, cols, rows, d->ld_pre_in, 1, 0, 64) &&
                make_out_map(&maps.m[1], d->C, false, cols, rows, d->ldc, 1, 0, 64);
      args.gated = 0;  // here `gated` describes the activation, not the layout of B
      return dispatch_gate(d, ta, tb, args, e, maps, grid, stream);
    }
    case FM_EPI_SCATTER: {
      EpiScatter e{reinterpret_cast<__nv_bfloat16* const*>(d->dst_base), d->dst_rank, d->dst_row,
                   d->ld_dst, d->dst_flags, d->num_ranks, d->row_aux, d->row_aux_dst};
      return dispatch_gate(d, ta, tb, args, e, maps, grid, stream);
    }
    case FM_EPI_COLSCATTER: {
      if (d->cols_per_rank <= 0 || d->cols_per_rank % 32 != 0) {
        set_err("column scatter needs cols_per_rank to be a positive multiple of 32");
        return -1;
      }
      EpiColScatter e{reinterpret_cast<__nv_bfloat16* const*>(d->dst_base), d->cols_per_rank, d->ld_dst,
                      d->dst_row_offset, d->dst_flags};
      return dispatch_gate(d, ta, tb, args, e, maps, grid, stream);
    }
    case FM_EPI_ADAM: {
      if (d->adam_p == nullptr || d->adam_m == nullptr || d->adam_v == nullptr) {
        set_err("optimizer epilogue needs parameter and moment pointers");
        return -1;
      }
      EpiAdam e{reinterpret_cast<__nv_bfloat16*>(d->adam_p), reinterpret_cast<__nv_bfloat16*>(d->adam_m),
                reinterpret_cast<__nv_bfloat16*>(d->adam_v), d->ldc, d->c_group_stride,
                d->alpha == 0.f ? 1.0f : d->alpha, d->adam_lr, d->adam_beta1, d->adam_beta2, d->adam_eps,
                d->adam_wd, d->adam_rbc1, d->adam_rbc2, 1};
      void* const arrays[3] = {d->adam_p, d->adam_m, d->adam_v};
      // The boxes of a row's 512 bytes follow one another, 64 bytes each; memory is read 256 at a time (none against 256,
      // 8 x 4096 x 28672 2590 and 2526 us, 64 x 2048 x 2816 1011 and 960, 8 x 14336 x 4096 the same).
      for (int i = 0; i < 3; ++i)
        if (!make_out_map(&maps.m[i], arrays[i], false, d->N, d->M, d->ldc, d->num_groups, d->c_group_stride, 64,
                          CU_TENSOR_MAP_L2_PROMOTION_L2_256B))
          e.boxes = 0;
      return dispatch_shape(d, ta, tb, args, e, GateNone{}, maps, grid, stream);
    }
    default:
      set_err("unknown epilogue");
      return -1;
  }
}
