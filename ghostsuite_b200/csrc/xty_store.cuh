// Direct store of a train gradient: an accumulator tile, scaled, cast to the parameter dtype and written (or added)
// to the row-major result.  Used where no other CTA adds to the same tile, so that neither the fp32 workspace
// nor the scaling pass over it is needed.
#pragma once
#include <cuda_bf16.h>
#include <stdint.h>

#include "sm100_ptx.cuh"

namespace gb {

// A matrix that a GEMM with one split writes itself
struct GradOut {
  void* out;               // [rows, cols], row-major
  int rows, cols;
  int is_f32, accumulate;
  int vec;                 // rows start on 16-byte boundaries
  float scale;
};

// Elements of the block at `base` that lie in rows [0, nrow), this lane's of columns [0, ncol): `value(row)` reads what was staged,
// loads of eight rows go out together.
template <typename T, typename V>
__device__ __forceinline__ void store_grad_columns(T* base, long long ld, int nrow, int col, int ncol, V&& value) {
  T* o = base + col;
#pragma unroll 1
  for (int r0 = 0; r0 < 32; r0 += 8) {
    T v[8];
#pragma unroll
    for (int i = 0; i < 8; ++i) v[i] = value(r0 + i);
#pragma unroll
    for (int i = 0; i < 8; ++i, o += ld)
      if (r0 + i < nrow && col < ncol) *o = v[i];
  }
}

// A warp's 32 rows (from `m0` on) of a 256-column accumulator tile (from column `n0` of the result on): scaled, cast and written, or
// added, to the result.  Blocks of 128 bytes a row (64 columns in bf16, 32 in float32) are turned in shared memory (`box`, 4 KB of the warp's
// own, 16-byte chunk c of row r at r * 128 + ((c ^ (r & 7)) << 4)), so that a store of the warp covers whole lines of four rows, or one
// row's neighbouring columns where rows begin anywhere.
// These stores are what bounds a call of few token rows.  With a row a lane (16-byte stores to 32 rows, aligned rows) and a
// loop that waited for each row's value before its store (others), 364 rows of 3392 x 1488
// (bf16) took 20.5 us and 3389 x 1484 49.5; 16.4 and 20.5 so.
__device__ __forceinline__ void store_grad_rows(const GradOut& g, uint32_t t_acc, int m0, int n0, uint8_t* box) {
  const int lane = threadIdx.x & 31;
  const int nrow = g.rows - m0 < 32 ? g.rows - m0 : 32;
  if (nrow <= 0) return;
  const long long ld = g.cols;
  uint8_t* mine = box + lane * 128;
  const int turn = lane & 7;
  auto chunk = [&](int row, int c) { return box + row * 128 + ((c ^ (row & 7)) << 4); };
  // whole chunks: eight lanes a row
  auto store_chunks = [&](uint8_t* base, int ncol_bytes) {
    const int c = lane & 7;
    uint4 v[8];
#pragma unroll
    for (int i = 0; i < 8; ++i) v[i] = *reinterpret_cast<const uint4*>(chunk(4 * i + (lane >> 3), c));
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      const int row = 4 * i + (lane >> 3);
      if (row < nrow && c * 16 < ncol_bytes) *reinterpret_cast<uint4*>(base + row * ld * (g.is_f32 ? 4 : 2) + c * 16) = v[i];
    }
  };
  if (g.is_f32 || g.accumulate) {
#pragma unroll 1
    for (int c0 = 0; c0 < 256 && n0 + c0 < g.cols; c0 += 32) {
      const int ncol = g.cols - n0 - c0 < 32 ? g.cols - n0 - c0 : 32;
      uint32_t r[32];
      tmem_ld32(t_acc + c0, r);
      tmem_ld_wait();
      __syncwarp();                        // the block before has been read
#pragma unroll
      for (int c = 0; c < 8; ++c) {
        float4 w;
        w.x = __uint_as_float(r[4 * c]) * g.scale; w.y = __uint_as_float(r[4 * c + 1]) * g.scale;
        w.z = __uint_as_float(r[4 * c + 2]) * g.scale; w.w = __uint_as_float(r[4 * c + 3]) * g.scale;
        *reinterpret_cast<float4*>(mine + ((c ^ turn) << 4)) = w;
      }
      __syncwarp();
      const long long at = m0 * ld + n0 + c0;
      auto staged = [&](int row) { return *reinterpret_cast<const float*>(chunk(row, lane >> 2) + (lane & 3) * 4); };
      auto there = [&](int row) { return row < nrow && lane < ncol; };
      if (g.is_f32) {
        float* base = static_cast<float*>(g.out) + at;
        if (g.accumulate)
          store_grad_columns(base, ld, nrow, lane, ncol, [&](int row) { return there(row) ? staged(row) + base[row * ld + lane] : 0.f; });
        else if (g.vec)
          store_chunks(reinterpret_cast<uint8_t*>(base), ncol * 4);
        else
          store_grad_columns(base, ld, nrow, lane, ncol, staged);
      } else {
        __nv_bfloat16* base = static_cast<__nv_bfloat16*>(g.out) + at;
        store_grad_columns(base, ld, nrow, lane, ncol, [&](int row) {
          return __float2bfloat16_rn(there(row) ? staged(row) + __bfloat162float(base[row * ld + lane]) : 0.f);
        });
      }
    }
    return;
  }
#pragma unroll 1
  for (int c0 = 0; c0 < 256 && n0 + c0 < g.cols; c0 += 64) {
    const int ncol = g.cols - n0 - c0 < 64 ? g.cols - n0 - c0 : 64;
    uint32_t r[2][32];
    tmem_ld32(t_acc + c0, r[0]);
    tmem_ld32(t_acc + c0 + 32, r[1]);
    tmem_ld_wait();
    __syncwarp();                          // the block before has been read
#pragma unroll
    for (int c = 0; c < 8; ++c) {
      uint32_t w[4];
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        const int j = 8 * (c & 3) + 2 * e;
        const __nv_bfloat162 h = __floats2bfloat162_rn(__uint_as_float(r[c >> 2][j]) * g.scale, __uint_as_float(r[c >> 2][j + 1]) * g.scale);
        w[e] = *reinterpret_cast<const uint32_t*>(&h);
      }
      st_shared_v4(mine + ((c ^ turn) << 4), w[0], w[1], w[2], w[3]);
    }
    __syncwarp();
    __nv_bfloat16* base = static_cast<__nv_bfloat16*>(g.out) + m0 * ld + n0 + c0;
    if (g.vec) {
      store_chunks(reinterpret_cast<uint8_t*>(base), ncol * 2);
    } else {
#pragma unroll
      for (int h = 0; h < 2; ++h)
        store_grad_columns(base, ld, nrow, lane + 32 * h, ncol, [&](int row) {
          return *reinterpret_cast<const __nv_bfloat16*>(chunk(row, 4 * h + (lane >> 3)) + (lane & 7) * 2);
        });
    }
  }
}

// The same rows added to the fp32 workspace of a result that several CTAs share: whole lines of four rows a store, rows of `ld` (a
// multiple of four), from a 16-byte boundary where the caller's workspace begins on one.  (A row a lane: 8192 rows of 256 x 256 bf16 23.6 us,
// 768 x 768 float32 43.4; 19.5 and 37.9 so.)  A result of up to 48 rows has one or two warps of a tile at work, and the way through shared
// memory is longer than it saves: those go a row a lane (bf16 results, us, lines and a row a lane: 6000 token rows of 16 x 4096 14.5 and 13.4,
// 33 x 4096 15.1 and 13.8, 40 x 4096 15.2 and 14.3, 16384 of 40 x 1024 13.2 and 13.5; of 64 x 1024 13.6 and 15.1, of 96 x 1024 14.1 and 16.8).
__device__ __forceinline__ void add_grad_rows(float* ws, long long ld, int rows, int cols, uint32_t t_acc, int m0, int n0, uint8_t* box) {
  const int lane = threadIdx.x & 31, c = lane & 7;
  const int nrow = rows - m0 < 32 ? rows - m0 : 32;
  if (nrow <= 0) return;
  const bool aligned = (reinterpret_cast<uintptr_t>(ws) & 15) == 0;
  // zeros behind the last column, up to the row's end
  auto add4 = [](float* at, float x, float y, float z, float w) {
    asm volatile("red.global.v4.f32.add [%0], {%1, %2, %3, %4};" ::"l"(at), "f"(x), "f"(y), "f"(z), "f"(w) : "memory");
  };
  if (rows <= 48 && aligned) {
    float* at = ws + (m0 + lane) * ld + n0;
#pragma unroll 1
    for (int c0 = 0; c0 < 256 && n0 + c0 < cols; c0 += 32) {
      uint32_t r[32];
      tmem_ld32(t_acc + c0, r);
      tmem_ld_wait();
      if (lane < nrow) {
#pragma unroll
        for (int q = 0; q < 8; ++q)
          if (n0 + c0 + 4 * q < cols)
            add4(at + c0 + 4 * q, __uint_as_float(r[4 * q]), __uint_as_float(r[4 * q + 1]), __uint_as_float(r[4 * q + 2]), __uint_as_float(r[4 * q + 3]));
      }
    }
    return;
  }
#pragma unroll 1
  for (int c0 = 0; c0 < 256 && n0 + c0 < cols; c0 += 64) {
    uint32_t r[2][32];
    tmem_ld32(t_acc + c0, r[0]);
    tmem_ld32(t_acc + c0 + 32, r[1]);
    tmem_ld_wait();
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      __syncwarp();                        // the block before has been read
#pragma unroll
      for (int q = 0; q < 8; ++q)
        st_shared_v4(box + lane * 128 + ((q ^ c) << 4), r[h][4 * q], r[h][4 * q + 1], r[h][4 * q + 2], r[h][4 * q + 3]);
      __syncwarp();
      float4 v[8];
#pragma unroll
      for (int i = 0; i < 8; ++i) {
        const int row = 4 * i + (lane >> 3);
        v[i] = *reinterpret_cast<const float4*>(box + row * 128 + ((c ^ (row & 7)) << 4));
      }
      const int col = n0 + c0 + 32 * h + 4 * c;
      float* at = ws + (m0 + (lane >> 3)) * ld + col;
#pragma unroll
      for (int i = 0; i < 8; ++i, at += 4 * ld) {
        if (4 * i + (lane >> 3) >= nrow || col >= cols) continue;
        if (aligned) {
          add4(at, v[i].x, v[i].y, v[i].z, v[i].w);
        } else {
          const float e[4] = {v[i].x, v[i].y, v[i].z, v[i].w};
#pragma unroll
          for (int j = 0; j < 4; ++j) asm volatile("red.global.add.f32 [%0], %1;" ::"l"(at + j), "f"(e[j]) : "memory");
        }
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

}  // namespace gb
