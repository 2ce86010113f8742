// Direct store of a train gradient: 32 consecutive accumulator columns of one output row, scaled, cast to
// the parameter dtype and written (or added) to the row-major result.  Used where no other CTA adds to
// the same tile, so that neither the fp32 workspace nor the scaling pass over it is needed.
#pragma once
#include <cuda_bf16.h>
#include <stdint.h>

#include "sm100_ptx.cuh"

namespace gb {

// `vec`: rows start on 16-byte boundaries, so whole groups of 32 columns go out as 16-byte stores (one row a lane;
// store_grad_block32 is the form for the rest)
__device__ __forceinline__ void store_grad_row32(void* out, int is_f32, int accumulate, float scale, long long at,
                                                 const uint32_t (&r)[32], int ncol, bool vec) {
  if (is_f32) {
    float* o = static_cast<float*>(out) + at;
    if (vec && ncol >= 32 && !accumulate) {
#pragma unroll
      for (int j = 0; j < 32; j += 4)
        *reinterpret_cast<float4*>(o + j) = make_float4(__uint_as_float(r[j]) * scale, __uint_as_float(r[j + 1]) * scale,
                                                        __uint_as_float(r[j + 2]) * scale, __uint_as_float(r[j + 3]) * scale);
    } else {
#pragma unroll
      for (int j = 0; j < 32; ++j)
        if (j < ncol) o[j] = __uint_as_float(r[j]) * scale + (accumulate ? o[j] : 0.f);
    }
  } else {
    __nv_bfloat16* o = static_cast<__nv_bfloat16*>(out) + at;
    if (vec && ncol >= 32 && !accumulate) {
#pragma unroll
      for (int j = 0; j < 32; j += 8) {
        uint32_t w[4];
#pragma unroll
        for (int e = 0; e < 4; ++e) {
          const __nv_bfloat162 h = __floats2bfloat162_rn(__uint_as_float(r[j + 2 * e]) * scale, __uint_as_float(r[j + 2 * e + 1]) * scale);
          w[e] = *reinterpret_cast<const uint32_t*>(&h);
        }
        *reinterpret_cast<uint4*>(o + j) = make_uint4(w[0], w[1], w[2], w[3]);
      }
    } else {
#pragma unroll
      for (int j = 0; j < 32; ++j)
        if (j < ncol) o[j] = __float2bfloat16_rn(__uint_as_float(r[j]) * scale + (accumulate ? __bfloat162float(o[j]) : 0.f));
    }
  }
}

// The 32 x 32 block of a warp (lane r holds row r) where single rows cannot go out as whole 16-byte pieces: turned in
// shared memory (`box`: 32 x 32 floats of the warp's own, columns rotated by the row against bank conflicts),
// a store of the warp then covers neighbouring columns of one row.  With a row per lane every store touched 32 rows:
// 15 x 51 tokens of 141 -> 64 in bf16 took 18 us for half a microsecond of work.
__device__ __forceinline__ void store_grad_block32(void* out, int is_f32, int accumulate, float scale, long long row0_at,
                                                   long long ld, const uint32_t (&r)[32], int nrow, int ncol, float* box) {
  const int lane = threadIdx.x & 31;
  __syncwarp();
#pragma unroll
  for (int j = 0; j < 32; ++j) box[lane * 32 + ((j + lane) & 31)] = __uint_as_float(r[j]);
  __syncwarp();
  if (lane < ncol) {
#pragma unroll 8
    for (int row = 0; row < 32; ++row) {
      if (row >= nrow) break;
      const float v = box[row * 32 + ((lane + row) & 31)] * scale;
      const long long at = row0_at + row * ld + lane;
      if (is_f32) {
        float* o = static_cast<float*>(out) + at;
        *o = accumulate ? v + *o : v;
      } else {
        __nv_bfloat16* o = static_cast<__nv_bfloat16*>(out) + at;
        *o = __float2bfloat16_rn(accumulate ? v + __bfloat162float(*o) : v);
      }
    }
  }
}

// A 128 x 256 fp32 accumulator tile through two swizzled [128][32] boxes of shared memory that the copy engine writes out
// at row y0 of `tm` (make_tmap_f32_store_2d), by the four epilogue warps (128 threads, named barrier 2).  Rows of a tile
// lie 1 KB apart: 32-byte stores, a row a lane, reached L2 as 2.9 million requests of one sector (24 + 5 samples
// of 768 x 1000) and took the load/store unit half of the kernel's time.  `boxes` counts the boxes handed over so far.
__device__ __forceinline__ void store_tile_f32(const CUtensorMap* tm, uint8_t* store_box, uint32_t t_acc, int y0, uint32_t& boxes) {
  constexpr int kBoxBytes = 128 * 32 * 4;
  const int row = static_cast<int>(threadIdx.x);
#pragma unroll 1
  for (int c0 = 0; c0 < 256; c0 += 32, ++boxes) {
    uint32_t r[32];
    tmem_ld32(t_acc + c0, r);
    tmem_ld_wait();
    uint8_t* box = store_box + (boxes & 1) * kBoxBytes;
    // the store that read this buffer two boxes ago has finished reading it
    if (threadIdx.x == 0) bulk_wait_group_read<1>();
    named_bar_sync(2, 128);
#pragma unroll
    for (int ch = 0; ch < 8; ++ch)
      st_shared_v4(box + row * 128 + ((ch ^ (row & 7)) << 4), r[4 * ch], r[4 * ch + 1], r[4 * ch + 2], r[4 * ch + 3]);
    fence_proxy_async_smem();
    named_bar_sync(2, 128);
    if (threadIdx.x == 0) {
      tma_store_2d(tm, box, c0, y0);
      bulk_commit_group();
    }
  }
}

// Split-K factor of a train-gradient pass with the shortest critical path, in units of one row block
// of one tile (about 0.28 us on both kernels): ceil(units / workers) rounds of (row blocks per split + a
// fixed cost per unit for the accumulator hand-over and the epilogue).  Splitting also pays for zeroing
// the fp32 workspace and for the scaling pass: two launches (5 us) and ten bytes per weight element
// at 5 TB/s; one split stores the result itself.  Fixed costs, measured: `add_cost` with red.add
// into the workspace, a quarter of it with plain stores.
// The tensor core's accumulator truncates, so the error grows with the rows one split covers.  A bf16
// result does not show it; a float32 result does (4096 rows of 768 x 768, bf16 operands: 4.2e-6 off the
// 64-bit result in one split, 4.5e-7 in ten), so there the merge is not counted against splitting.
inline int pick_k_splits(long long tiles, int workers, int kb, int add_cost, double weight_elems, bool f32_result) {
  int splits = 1;
  double best = static_cast<double>((tiles + workers - 1) / workers) * (kb + (f32_result ? add_cost : add_cost / 4));
  const double merge = f32_result ? 0. : (5.0 + weight_elems * 10.0 / 5e6) / 0.28;
  for (int s = 2; s <= 64 && s <= kb; ++s) {
    const double cost = static_cast<double>((tiles * s + workers - 1) / workers) * ((kb + s - 1) / s + add_cost) + merge;
    if (cost < best) { best = cost; splits = s; }
  }
  return splits;
}

}  // namespace gb
