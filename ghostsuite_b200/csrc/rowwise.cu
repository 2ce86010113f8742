// Bandwidth-bound kernels of the ghost hot path: dtype cast / bf16 split, per-sample column sums
// (bias terms) and per-sample LayerNorm gradients.  All of them stream their inputs once with
// 16-byte coalesced loads and reduce with warp shuffles / shared memory.
#include "common.cuh"
#include "sm100_ptx.cuh"

namespace gb {

__device__ __forceinline__ float warp_sum(float v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}

// 8 consecutive elements -> fp32
template <typename T> struct Vec8;
template <> struct Vec8<__nv_bfloat16> {
  static __device__ __forceinline__ void load(const __nv_bfloat16* p, float (&x)[8]) {
    const uint4 w = *reinterpret_cast<const uint4*>(p);
    const uint32_t ww[4] = {w.x, w.y, w.z, w.w};
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      x[2 * e] = __uint_as_float(ww[e] << 16);
      x[2 * e + 1] = __uint_as_float(ww[e] & 0xffff0000u);
    }
  }
};
template <> struct Vec8<float> {
  static __device__ __forceinline__ void load(const float* p, float (&x)[8]) {
    const float4 a = *reinterpret_cast<const float4*>(p);
    const float4 b = *reinterpret_cast<const float4*>(p + 4);
    x[0] = a.x; x[1] = a.y; x[2] = a.z; x[3] = a.w;
    x[4] = b.x; x[5] = b.y; x[6] = b.z; x[7] = b.w;
  }
};
// One value of every CTA of the cluster, added up in rank order
__device__ __forceinline__ float cluster_sum(const float* mine, int ranks) {
  float v = 0.f;
  for (int r = 0; r < ranks; ++r) v += ld_cluster_f32(map_to_cta(smem_u32(mine), r));
  return v;
}

template <typename T> __device__ __forceinline__ float to_f32(T v);
template <> __device__ __forceinline__ float to_f32<float>(float v) { return v; }
template <> __device__ __forceinline__ float to_f32<__nv_bfloat16>(__nv_bfloat16 v) { return __bfloat162float(v); }

// ------------------------------------------------------------------------------------------
// cast / split.  dst is bf16 with `parts` copies of the (zero-padded) source laid out either
// side by side along columns (col_stack) or one below the other inside each sample (row_stack).
// part kinds: 0 = bf16(x) ("hi"), 1 = bf16(x - hi) ("lo").
// ------------------------------------------------------------------------------------------
struct CastParams {
  const void* src;
  __nv_bfloat16* dst;
  long long samples, T;     // rows = samples * T
  int cols, cpad;           // cpad = padded column count of one part
  long long ld_src, ld_dst;
  int parts;
  int kind[3];
  int row_stack;            // 0: parts side by side; 1: parts stacked along rows within a sample
  unsigned blocks;          // of the launch
};
struct CastPair { CastParams job[2]; };

// Bound by HBM once the index arithmetic is in 32 bits (I: unsigned wherever the element groups and rows fit)
// and hi and lo parts are made once an element: 64-bit divisions were most of its instructions (both
// operands of 29 samples of 197 x (768, 1000) float32: 18.8 us before, 14.4 now).
template <typename T, typename I>
__device__ __forceinline__ void cast_rows(const CastParams& p, unsigned block) {
  const I cvec = static_cast<I>(p.cpad / 8);
  const I total = static_cast<I>(p.samples * p.T) * cvec;
  const bool stacked = p.row_stack && p.parts > 1;
  const long long stride = stacked ? p.T * p.ld_dst : p.cpad;
  for (I i = block * static_cast<I>(blockDim.x) + threadIdx.x; i < total; i += p.blocks * static_cast<I>(blockDim.x)) {
    const I row = i / cvec;
    const int c0 = static_cast<int>(i - row * cvec) * 8;
    float x[8];
    const T* src = static_cast<const T*>(p.src) + static_cast<long long>(row) * p.ld_src + c0;
    if (c0 + 8 <= p.cols && (reinterpret_cast<uintptr_t>(src) & 15u) == 0) {
      Vec8<T>::load(src, x);
    } else {
#pragma unroll
      for (int j = 0; j < 8; ++j) x[j] = (c0 + j < p.cols) ? to_f32<T>(src[j]) : 0.f;
    }
    uint32_t hw[4], lw[4];               // the values as bf16, and what that leaves of them
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      const __nv_bfloat162 hi = __floats2bfloat162_rn(x[2 * e], x[2 * e + 1]);
      const __nv_bfloat162 lo = __floats2bfloat162_rn(x[2 * e] - __bfloat162float(hi.x), x[2 * e + 1] - __bfloat162float(hi.y));
      hw[e] = *reinterpret_cast<const uint32_t*>(&hi);
      lw[e] = *reinterpret_cast<const uint32_t*>(&lo);
    }
    // sample s of `parts` blocks of T rows: row + s * (parts - 1) * T
    const long long at = stacked ? row + static_cast<long long>(row / static_cast<I>(p.T)) * (p.parts - 1) * p.T : row;
    __nv_bfloat16* dst = p.dst + at * p.ld_dst + c0;
#pragma unroll
    for (int part = 0; part < 3; ++part) {
      if (part >= p.parts) break;
      const bool low = p.kind[part] == 1;
      *reinterpret_cast<uint4*>(dst + part * stride) =
          make_uint4(low ? lw[0] : hw[0], low ? lw[1] : hw[1], low ? lw[2] : hw[2], low ? lw[3] : hw[3]);
    }
  }
}
template <typename T, typename I>
__global__ void cast_split_kernel(const CastParams p) {
  stream_order();
  cast_rows<T, I>(p, blockIdx.x);
}
// bf16 rows of two operands, padded, in one launch.  A warp takes 256 neighbouring columns: the panels of split_pair_kernel
// below, two rows of 128 to a warp, touch more lines a load where rows lie off 16-byte boundaries (15 x 1220 tokens
// of 64 -> 13119, a hook: 506 us with them, 445 so; 171 x 1984 of 64 -> 133 125 and 105).
template <typename I>
__global__ void cast_pair_kernel(const CastPair p) {
  stream_order();
  const bool second = blockIdx.x >= p.job[0].blocks;
  cast_rows<__nv_bfloat16, I>(p.job[second ? 1 : 0], blockIdx.x - (second ? p.job[0].blocks : 0u));
}

// Both operands of a token-contracted GEMM in one launch: rows zero-padded to ld (a multiple of 64) columns, as the
// values alone (PARTS = 1; bf16 rows whose sums are not asked for go through cast_pair_kernel) or as values and residuals, [samples, 2, T, ld] or [2, samples * T, ld].  A block takes a panel of 128 columns of
// some rows, a thread eight columns of every 16th row, two rows in flight.  Where the column sums of an operand are
// wanted the rows are one sample's, or a chunk of it whose sums meet in a cluster or are added to zeros, and they cost no second pass.
// Bound by HBM and, on small layers, by the round trip of one round of loads: 8 x 2048 rows of (1024, 2048) float32 at
// 5.5 TB/s, 29 x 197 of (768, 1000) with their sums 17 us from cold caches, 14 with the operands in L2 (two launches of
// cast_split_kernel with three parts 17.4, and 8.5 for the sums in a pass of their own).
static constexpr int kSplitCols = 128, kSplitLanes = 16;       // columns and row lanes of a block
struct SplitJob {
  const void* src;
  __nv_bfloat16* dst;
  float* sums;             // [samples, cols] or null
  int is_f32, cols, ld, panels;
  int vec;                 // rows on 16-byte boundaries
  long long rows, per;     // all rows; rows of a block
  int chunks;              // blocks that share a sample (sums only)
  int ranks;               // they are a cluster of so many, which adds up the sums, or 1: the sums are added to zeros
  long long blocks;        // in the grid: with those that fill the last cluster
  long long used;
};
struct SplitParams {
  SplitJob job[2];
  long long T;             // rows of a sample
  long long part_rows;     // rows of a part: T, or those of all samples
};

template <typename E, int PARTS, bool VEC>
__device__ __forceinline__ void split_rows(const SplitJob& j, long long T, long long r0, long long r1, int c0, float (&sum)[8]) {
  constexpr int R = 2;                   // rows in flight of a thread
  const bool inside = c0 + 8 <= j.cols;
  const long long first = r0 + (threadIdx.x / (kSplitCols / 8));
  int left = r1 - first > 0 ? static_cast<int>(r1 - first) : 0;          // a block has far fewer than 2^31 rows
  const E* src = static_cast<const E*>(j.src) + first * j.cols + c0;
  // sample s of two parts of T rows: row + s * T.  The sample of this thread's first row, then step by step.
  long long sample = 0;
  if (PARTS == 2) sample = j.rows < (1ll << 32) ? static_cast<unsigned>(first) / static_cast<unsigned>(T) : first / T;
  long long in_sample = T - (first - sample * T);                        // rows of it from here on
  __nv_bfloat16* dst = j.dst + (first + (PARTS == 2 ? sample * T : 0)) * j.ld + c0;
  const long long row_src = static_cast<long long>(kSplitLanes) * j.cols, row_dst = static_cast<long long>(kSplitLanes) * j.ld, lo = T * j.ld;
  for (; left > 0; left -= R * kSplitLanes) {
    float x[R][8];
#pragma unroll
    for (int q = 0; q < R; ++q, src += row_src) {
#pragma unroll
      for (int e = 0; e < 8; ++e) x[q][e] = 0.f;
      if (kSplitLanes * q < left) {
        if (VEC && inside) {
          Vec8<E>::load(src, x[q]);
        } else {
#pragma unroll
          for (int e = 0; e < 8; ++e)
            if (c0 + e < j.cols) x[q][e] = to_f32<E>(src[e]);
        }
      }
    }
#pragma unroll
    for (int e = 0; e < 8; ++e) sum[e] += x[0][e] + x[1][e];
#pragma unroll
    for (int q = 0; q < R; ++q) {
      uint32_t hw[4], lw[4];             // the values as bf16, and what that leaves of them
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        const float a = x[q][2 * e], b = x[q][2 * e + 1];
        const __nv_bfloat162 hi = __floats2bfloat162_rn(a, b);
        const __nv_bfloat162 lv = __floats2bfloat162_rn(a - __bfloat162float(hi.x), b - __bfloat162float(hi.y));
        hw[e] = *reinterpret_cast<const uint32_t*>(&hi);
        lw[e] = *reinterpret_cast<const uint32_t*>(&lv);
      }
      if (kSplitLanes * q < left) {
        *reinterpret_cast<uint4*>(dst) = make_uint4(hw[0], hw[1], hw[2], hw[3]);
        if (PARTS == 2) *reinterpret_cast<uint4*>(dst + lo) = make_uint4(lw[0], lw[1], lw[2], lw[3]);
      }
      dst += row_dst;
      if (PARTS == 2) {
        in_sample -= kSplitLanes;
        while (in_sample <= 0) { in_sample += T; dst += lo; }
      }
    }
  }
}

template <int PARTS>
__global__ void __launch_bounds__(256, 4) split_pair_kernel(const SplitParams p) {
  __shared__ float red[8][kSplitCols];
  stream_order();
  const bool second = blockIdx.x >= p.job[0].blocks;
  const SplitJob& j = p.job[second ? 1 : 0];
  const unsigned at = blockIdx.x - (second ? static_cast<unsigned>(p.job[0].blocks) : 0u);
  if (at >= j.used) return;
  // a cluster's blocks are the chunks of one sample and panel; otherwise neighbouring blocks read along the rows
  unsigned chunk = 0, panel = at % j.panels, rest = at / j.panels;
  if (j.ranks > 1) {
    chunk = at % j.ranks;
    panel = at / j.ranks % j.panels;
    rest = at / j.ranks / j.panels;
  } else if (j.sums) {
    chunk = rest % j.chunks;
    rest /= j.chunks;
  }
  const int oct = threadIdx.x % (kSplitCols / 8), c0 = static_cast<int>(panel) * kSplitCols + oct * 8;
  long long sample = 0, r0 = rest * j.per, r1 = j.rows;
  if (j.sums) {
    sample = rest;
    r0 = sample * p.T + chunk * j.per;
    r1 = (sample + 1) * p.T;
  }
  if (r0 + j.per < r1) r1 = r0 + j.per;
  float sum[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
  if (c0 < j.ld) {
    if (j.is_f32 && j.vec) split_rows<float, PARTS, true>(j, p.part_rows, r0, r1, c0, sum);
    else if (j.is_f32) split_rows<float, PARTS, false>(j, p.part_rows, r0, r1, c0, sum);
    else if (j.vec) split_rows<__nv_bfloat16, PARTS, true>(j, p.part_rows, r0, r1, c0, sum);
    else split_rows<__nv_bfloat16, PARTS, false>(j, p.part_rows, r0, r1, c0, sum);
  }
  if (!j.sums) return;
#pragma unroll
  for (int e = 0; e < 8; ++e) sum[e] += __shfl_xor_sync(0xffffffffu, sum[e], 16);
  if ((threadIdx.x & 31) < 16)
#pragma unroll
    for (int e = 0; e < 8; ++e) red[threadIdx.x >> 5][oct * 8 + e] = sum[e];
  __syncthreads();
  const int t = threadIdx.x, c = static_cast<int>(panel) * kSplitCols + t;
  float v = 0.f;
  if (t < kSplitCols)
    v = ((red[0][t] + red[1][t]) + (red[2][t] + red[3][t])) + ((red[4][t] + red[5][t]) + (red[6][t] + red[7][t]));
  float* out = j.sums + sample * j.cols + c;
  if (j.ranks > 1) {
    if (t < kSplitCols) red[0][t] = v;             // read above by this thread alone
    cluster_sync_all();
    if (chunk == 0 && t < kSplitCols && c < j.cols) *out = cluster_sum(&red[0][t], j.ranks);
    cluster_sync_all();                            // no CTA leaves while another reads its sums
  } else if (t < kSplitCols && c < j.cols) {
    if (j.chunks == 1) *out = v;
    else atomicAdd(out, v);
  }
}

// ------------------------------------------------------------------------------------------
// per-sample column sums: out[n, c] = sum_t G[n, t, c], of one split or of several that are a cluster; others add theirs to zeros
// ------------------------------------------------------------------------------------------
template <typename T>
__global__ void colsum_kernel(const T* G, long long Tn, int cols, long long ld,
                              float* __restrict__ out, int t_splits, int clustered) {
  // block: 32 column vectors (256 columns) x 8 row lanes
  __shared__ float red[8][256 + 8];
  stream_order();
  const int n = blockIdx.z;
  const int split = blockIdx.y;
  const int cx = threadIdx.x & 31, ry = threadIdx.x >> 5;
  const int c0 = (blockIdx.x * 32 + cx) * 8;
  const long long per = (Tn + t_splits - 1) / t_splits;
  const long long t0 = split * per;
  const long long t1 = (t0 + per < Tn) ? t0 + per : Tn;
  float acc[8];
#pragma unroll
  for (int j = 0; j < 8; ++j) acc[j] = 0.f;
  const bool vec_ok = (c0 + 8 <= cols) && (ld % 8 == 0) &&
                      ((reinterpret_cast<uintptr_t>(G + static_cast<long long>(n) * Tn * ld + c0) & 15u) == 0);
  if (c0 < cols) {
    const T* base = G + static_cast<long long>(n) * Tn * ld + c0;
    long long t = t0 + ry;
    if (vec_ok) {
      // four independent 16-byte loads in flight per thread
      for (; t + 24 < t1; t += 32) {
        float x0[8], x1[8], x2[8], x3[8];
        Vec8<T>::load(base + t * ld, x0);
        Vec8<T>::load(base + (t + 8) * ld, x1);
        Vec8<T>::load(base + (t + 16) * ld, x2);
        Vec8<T>::load(base + (t + 24) * ld, x3);
#pragma unroll
        for (int j = 0; j < 8; ++j) acc[j] += (x0[j] + x1[j]) + (x2[j] + x3[j]);
      }
    }
    for (; t < t1; t += 8) {
      float x[8];
      if (vec_ok) {
        Vec8<T>::load(base + t * ld, x);
      } else {
#pragma unroll
        for (int j = 0; j < 8; ++j) x[j] = (c0 + j < cols) ? to_f32<T>(base[t * ld + j]) : 0.f;
      }
#pragma unroll
      for (int j = 0; j < 8; ++j) acc[j] += x[j];
    }
  }
#pragma unroll
  for (int j = 0; j < 8; ++j) red[ry][cx * 8 + j] = acc[j];
  __syncthreads();
  const int c = threadIdx.x;   // 256 threads, one column each
  float s = 0.f;
#pragma unroll
  for (int r = 0; r < 8; ++r) s += red[r][c];
  const int col = blockIdx.x * 256 + c;
  if (clustered) {                        // the splits are a cluster: no zeros to add to
    red[0][c] = s;                        // read above by this thread alone
    cluster_sync_all();
    if (split == 0 && col < cols) out[static_cast<long long>(n) * cols + col] = cluster_sum(&red[0][c], t_splits);
    cluster_sync_all();                   // no CTA leaves while another reads its sums
    return;
  }
  if (col < cols) {
    float* dst = out + static_cast<long long>(n) * cols + col;
    if (t_splits > 1) atomicAdd(dst, s); else *dst = s;
  }
}

// ------------------------------------------------------------------------------------------
// LayerNorm per-sample gradients, one warp per token row, F <= 256 * NCHUNK, F % 8 == 0.
//   gw[n, f] += sum_t G[n,t,f] * xhat[n,t,f],   gb[n, f] += sum_t G[n,t,f]
// ------------------------------------------------------------------------------------------
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N> __device__ __forceinline__ void cp_async_wait() {
  asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory");
}

// Two float32 operations an instruction, each rounded as the single one is
__device__ __forceinline__ float2 add2(float2 a, float2 b) {
  float2 d;
  asm("{\n\t.reg .b64 x, y;\n\tmov.b64 x, {%2, %3};\n\tmov.b64 y, {%4, %5};\n\tadd.rn.f32x2 x, x, y;\n\tmov.b64 {%0, %1}, x;\n\t}"
      : "=f"(d.x), "=f"(d.y) : "f"(a.x), "f"(a.y), "f"(b.x), "f"(b.y));
  return d;
}
__device__ __forceinline__ float2 mul2(float2 a, float2 b) {
  float2 d;
  asm("{\n\t.reg .b64 x, y;\n\tmov.b64 x, {%2, %3};\n\tmov.b64 y, {%4, %5};\n\tmul.rn.f32x2 x, x, y;\n\tmov.b64 {%0, %1}, x;\n\t}"
      : "=f"(d.x), "=f"(d.y) : "f"(a.x), "f"(a.y), "f"(b.x), "f"(b.y));
  return d;
}
__device__ __forceinline__ float2 fma2(float2 a, float2 b, float2 c) {
  float2 d;
  asm("{\n\t.reg .b64 x, y, z;\n\tmov.b64 x, {%2, %3};\n\tmov.b64 y, {%4, %5};\n\tmov.b64 z, {%6, %7};\n\tfma.rn.f32x2 x, x, y, z;\n\t"
      "mov.b64 {%0, %1}, x;\n\t}"
      : "=f"(d.x), "=f"(d.y) : "f"(a.x), "f"(a.y), "f"(b.x), "f"(b.y), "f"(c.x), "f"(c.y));
  return d;
}

// Each warp streams its token rows through a private three-slot ring in shared memory filled with
// cp.async: the loads of the next two rows are in flight while the current row goes through its two
// dependent shuffle reductions.  A lane reads back exactly the 16-byte pieces it copied itself, so
// the ring needs no synchronisation beyond cp.async.wait_group.
//
// Bound by issue slots before HBM: 388 instructions a row of 768 bf16 features kept the schedulers 60 % busy at
// 4.35 TB/s.  So features go in pairs (f32x2), and a width that fills the lanes (FULL: F = 256 NCHUNK) has no tests:
// 40 x 1024 rows went from 30.1 to 24.2 us (5.2 TB/s) with a part of them in L2; from cold caches they take 30.4.
constexpr int kLnSlots = 3;

template <typename T, int NCHUNK, bool FULL>
__global__ void __launch_bounds__(256, NCHUNK <= 3 ? 2 : 1)
layernorm_persample_kernel(const T* A, const T* G, long long Tn, int F,
                           float eps, float* __restrict__ gw, float* __restrict__ gb,
                           float* __restrict__ part, int t_splits, int rms) {
  stream_order();
  extern __shared__ __align__(16) unsigned char sm_raw[];   // rings [8 warps][3][2][F] of T, then [8][2][F] floats
  float* sm = reinterpret_cast<float*>(sm_raw);
  const int n = blockIdx.y, split = blockIdx.x;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  T* ring = reinterpret_cast<T*>(sm_raw) + static_cast<size_t>(warp) * kLnSlots * 2 * F;
  const long long per = (Tn + t_splits - 1) / t_splits;
  const long long t0 = split * per;
  const long long t1 = (t0 + per < Tn) ? t0 + per : Tn;
  float2 aw[NCHUNK][4], ab[NCHUNK][4];
#pragma unroll
  for (int i = 0; i < NCHUNK; ++i)
#pragma unroll
    for (int j = 0; j < 4; ++j) aw[i][j] = ab[i][j] = make_float2(0.f, 0.f);
  const float invF = 1.f / static_cast<float>(F);
  auto inside = [&](int i) { return FULL || (i * 32 + lane) * 8 < F; };

  long long t = t0 + warp, ahead = t;                  // row at work, row to fetch next
  const T *pa = A + (static_cast<long long>(n) * Tn + t) * F + lane * 8, *pg = G + (pa - A);
  const uint32_t ring0 = static_cast<uint32_t>(__cvta_generic_to_shared(ring + lane * 8)), slot_bytes = 2 * F * sizeof(T);
  const uint32_t row_bytes = F * sizeof(T);
  auto issue = [&](int slot) {
    if (ahead < t1) {
      const uint32_t dst = ring0 + slot * slot_bytes;
#pragma unroll
      for (int i = 0; i < NCHUNK; ++i) {
        if (inside(i)) {
#pragma unroll
          for (int b = 0; b < static_cast<int>(8 * sizeof(T)); b += 16) {
            const int at = i * 256 * static_cast<int>(sizeof(T)) + b;
            asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst + at), "l"(reinterpret_cast<const unsigned char*>(pa) + at) : "memory");
            asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst + row_bytes + at), "l"(reinterpret_cast<const unsigned char*>(pg) + at) : "memory");
          }
        }
      }
    }
    cp_async_commit();      // an empty group keeps the group count uniform at the tail
    ahead += 8;
    pa += 8ll * F;
    pg += 8ll * F;
  };

  issue(0);
  issue(1);
  int slot = 0;
  for (; t < t1; t += 8) {
    issue(slot == 0 ? 2 : slot - 1);
    cp_async_wait<kLnSlots - 1>();
    const T* sa = ring + static_cast<size_t>(slot) * 2 * F;
    const T* sg = sa + F;
    slot = (slot + 1 == kLnSlots) ? 0 : slot + 1;
    float2 x[NCHUNK][4], g[NCHUNK][4];
    auto load = [&](const T* row, int i, float2 (&v)[4]) {
      float e[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
      if (inside(i)) Vec8<T>::load(row + (i * 32 + lane) * 8, e);
#pragma unroll
      for (int j = 0; j < 4; ++j) v[j] = make_float2(e[2 * j], e[2 * j + 1]);
    };
    float2 s = make_float2(0.f, 0.f);
#pragma unroll
    for (int i = 0; i < NCHUNK; ++i) load(sa, i, x[i]);
#pragma unroll
    for (int i = 0; i < NCHUNK; ++i) load(sg, i, g[i]);
    float mean = 0.f;                                  // RMS norm: no centring
    if (!rms) {
#pragma unroll
      for (int i = 0; i < NCHUNK; ++i) s = add2(s, add2(add2(x[i][0], x[i][1]), add2(x[i][2], x[i][3])));
      mean = warp_sum(s.x + s.y) * invF;
    }
    const float2 centre = make_float2(-mean, -mean);
    float2 q = make_float2(0.f, 0.f);
#pragma unroll
    for (int i = 0; i < NCHUNK; ++i) {
      if (inside(i)) {
#pragma unroll
        for (int j = 0; j < 4; ++j) { x[i][j] = add2(x[i][j], centre); q = fma2(x[i][j], x[i][j], q); }
      }
    }
    const float rstd = rsqrtf(warp_sum(q.x + q.y) * invF + eps);
    const float2 scale = make_float2(rstd, rstd);
#pragma unroll
    for (int i = 0; i < NCHUNK; ++i)
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        aw[i][j] = fma2(g[i][j], mul2(x[i][j], scale), aw[i][j]);
        ab[i][j] = add2(ab[i][j], g[i][j]);
      }
  }
  cp_async_wait<0>();
  __syncthreads();          // the rings are reused as the cross-warp reduction scratch
  float* mine = sm + static_cast<size_t>(warp) * 2 * F;
#pragma unroll
  for (int i = 0; i < NCHUNK; ++i) {
    const int f = (i * 32 + lane) * 8;
    if (f < F) {
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        *reinterpret_cast<float2*>(mine + f + 2 * j) = aw[i][j];
        *reinterpret_cast<float2*>(mine + F + f + 2 * j) = ab[i][j];
      }
    }
  }
  __syncthreads();
  for (int f = threadIdx.x; f < 2 * F; f += blockDim.x) {
    float v = 0.f;
#pragma unroll
    for (int w = 0; w < 8; ++w) v += sm[static_cast<size_t>(w) * 2 * F + f];
    if (t_splits > 1) {
      part[(static_cast<long long>(split) * gridDim.y + n) * 2 * F + f] = v;
    } else if (f < F) {
      gw[static_cast<long long>(n) * F + f] = v;
    } else {
      gb[static_cast<long long>(n) * F + f - F] = v;
    }
  }
}

// second stage: sum the per-split partials in a fixed order (deterministic)
__global__ void layernorm_reduce_kernel(const float* part, int N, int F, int t_splits,
                                        float* __restrict__ gw, float* __restrict__ gb) {
  stream_order();
  const long long total = static_cast<long long>(N) * 2 * F;
  for (long long i = blockIdx.x * static_cast<long long>(blockDim.x) + threadIdx.x; i < total;
       i += static_cast<long long>(gridDim.x) * blockDim.x) {
    float v = 0.f;
    for (int s = 0; s < t_splits; ++s) v += part[static_cast<long long>(s) * total + i];
    const int n = static_cast<int>(i / (2 * F)), f = static_cast<int>(i % (2 * F));
    if (f < F) gw[static_cast<long long>(n) * F + f] = v;
    else gb[static_cast<long long>(n) * F + f - F] = v;
  }
}

// A thread's PT features of a row as they are loaded: pieces of eight, or every THREADS-th.  They are converted in a second
// step: behind its bounds check a conversion makes each load of a group of rows wait for the one before (RMS hooks
// of 6 + 2 x 1024 rows in bf16, us: F = 4096 60 and 52, 8192 94.5 and 82.5, 4097 109 and 92).
template <typename T, bool VEC, int PT> struct NormRaw {
  using Bits = typename std::conditional<sizeof(T) == 2, unsigned short, float>::type;
  static constexpr int kWords = static_cast<int>(sizeof(T)) / 2;       // 16-byte words of eight features
  uint4 v[VEC ? PT / 8 * kWords : 1];
  Bits e[VEC ? 1 : PT];
  template <int THREADS> __device__ __forceinline__ void load(const T* row, int F) {
    if constexpr (VEC) {
#pragma unroll
      for (int c = 0; c < PT / 8; ++c) {
        const int f = (c * THREADS + static_cast<int>(threadIdx.x)) * 8;
#pragma unroll
        for (int w = 0; w < kWords; ++w) {
          v[c * kWords + w] = make_uint4(0u, 0u, 0u, 0u);
          if (f < F) v[c * kWords + w] = reinterpret_cast<const uint4*>(row + f)[w];
        }
      }
    } else {
#pragma unroll
      for (int c = 0; c < PT; ++c) {
        const int f = c * THREADS + static_cast<int>(threadIdx.x);
        e[c] = 0;
        if (f < F) e[c] = reinterpret_cast<const Bits*>(row)[f];
      }
    }
  }
  __device__ __forceinline__ void values(float (&x)[PT]) const {
    if constexpr (VEC) {
#pragma unroll
      for (int c = 0; c < PT / 8; ++c) {
        if constexpr (sizeof(T) == 2) {
          const uint32_t w[4] = {v[c].x, v[c].y, v[c].z, v[c].w};
#pragma unroll
          for (int j = 0; j < 4; ++j) {
            x[c * 8 + 2 * j] = __uint_as_float(w[j] << 16);
            x[c * 8 + 2 * j + 1] = __uint_as_float(w[j] & 0xffff0000u);
          }
        } else {
#pragma unroll
          for (int h = 0; h < 2; ++h) {
            const uint4 w = v[2 * c + h];
            x[c * 8 + 4 * h] = __uint_as_float(w.x); x[c * 8 + 4 * h + 1] = __uint_as_float(w.y);
            x[c * 8 + 4 * h + 2] = __uint_as_float(w.z); x[c * 8 + 4 * h + 3] = __uint_as_float(w.w);
          }
        }
      }
    } else {
#pragma unroll
      for (int c = 0; c < PT; ++c) {
        if constexpr (sizeof(T) == 2) x[c] = __uint_as_float(static_cast<uint32_t>(e[c]) << 16);
        else x[c] = e[c];
      }
    }
  }
};

// F beyond the warp-per-row kernel (above 1024, or no multiple of eight) up to 8192: a block owns the whole
// width, a thread PT features of it (pieces of eight, or every THREADS-th feature when rows are not
// 16-byte aligned), and R = 32 / PT rows (whole ones) go through the two reductions together, so their loads are in
// flight at once and one barrier serves R rows.  The gradients of a thread's features stay in registers.
// Bound by the latency of a group of rows (loads, two reductions) more than by HBM: 3 to 4 TB/s.  The
// block-per-row kernel below reads every row three times in single elements and meets at four
// barriers per row; whole LayerNorm hook, 24 samples of 1024 rows of bf16: F = 4096 803 -> 138 us, F = 2048
// 380 -> 97, F = 731 173 -> 60; RMS norm, 12 x 1024 rows of F = 8192: 1179 -> 138.
template <typename T, bool VEC, int PT, int THREADS>
__global__ void __launch_bounds__(THREADS, THREADS <= 256 ? 2 : 1)
norm_wide_kernel(const T* A, const T* G, long long Tn, int F, float eps, float* __restrict__ gw,
                 float* __restrict__ gb, float* __restrict__ part, int t_splits, int rms) {
  constexpr int R = 32 / PT, W = THREADS / 32;
  // Rows added up in registers before they join the totals: one chain over all rows of a split had 1.7 times the
  // error of the kernel before (4096 rows of 8192 in nine splits: 3.9e-7 against 2.3e-7; 1.5e-7 now).
  constexpr int kChain = 32;
  __shared__ float red[2][R][W];
  stream_order();
  extern __shared__ float s_total[];     // [2][PT][THREADS]: a thread's own totals, where they cost no registers
  const int n = blockIdx.y, split = blockIdx.x;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const long long per = (Tn + t_splits - 1) / t_splits;
  const long long t0 = split * per;
  const long long t1 = (t0 + per < Tn) ? t0 + per : Tn;
  const float invF = 1.f / static_cast<float>(F);
  auto feature = [&](int e) -> int {
    return VEC ? (e / 8) * THREADS * 8 + static_cast<int>(threadIdx.x) * 8 + e % 8 : e * THREADS + static_cast<int>(threadIdx.x);
  };
  int buf = 0;
  // sums of one value per row over the block; the buffers alternate, so one barrier is enough
  auto block_sum = [&](float (&s)[R]) {
#pragma unroll
    for (int r = 0; r < R; ++r) s[r] = warp_sum(s[r]);
    if (lane == 0)
#pragma unroll
      for (int r = 0; r < R; ++r) red[buf][r][warp] = s[r];
    __syncthreads();
#pragma unroll
    for (int r = 0; r < R; ++r) {
      s[r] = 0.f;
#pragma unroll
      for (int w = 0; w < W; ++w) s[r] += red[buf][r][w];
    }
    buf ^= 1;
  };
  float aw[PT], ab[PT];
#pragma unroll
  for (int e = 0; e < PT; ++e) { aw[e] = 0.f; ab[e] = 0.f; }
  bool first = true;
  auto to_total = [&]() {
#pragma unroll
    for (int e = 0; e < PT; ++e) {
      float* w = s_total + e * THREADS + threadIdx.x;
      float* b = w + PT * THREADS;
      *w = first ? aw[e] : *w + aw[e];
      *b = first ? ab[e] : *b + ab[e];
      aw[e] = 0.f;
      ab[e] = 0.f;
    }
    first = false;
  };
  int chain = 0;
  for (long long t = t0; t < t1; t += R) {
    float x[R][PT], g[R][PT], s[R];
    auto at = [&](int r) { return (static_cast<long long>(n) * Tn + (t + r < t1 ? t + r : t)) * F; };
    if constexpr (!VEC && PT == 4) {     // eight rows of four features: converted at once, 1 % faster (40 + 8 x 1024 x 1001 bf16 83.3 and 84.5 us)
#pragma unroll
      for (int r = 0; r < R; ++r)
#pragma unroll
        for (int o = 0; o < 2; ++o)
#pragma unroll
          for (int e = 0; e < PT; ++e) (o ? g : x)[r][e] = feature(e) < F ? to_f32<T>(((o ? G : A) + at(r))[feature(e)]) : 0.f;
    } else {
      NormRaw<T, VEC, PT> ra[R], rg[R];
#pragma unroll
      for (int r = 0; r < R; ++r) {
        ra[r].template load<THREADS>(A + at(r), F);
        rg[r].template load<THREADS>(G + at(r), F);
      }
#pragma unroll
      for (int r = 0; r < R; ++r) { ra[r].values(x[r]); rg[r].values(g[r]); }
    }
    if (!rms) {                          // RMS norm: no centring
#pragma unroll
      for (int r = 0; r < R; ++r) {
        s[r] = 0.f;
#pragma unroll
        for (int e = 0; e < PT; ++e) s[r] += x[r][e];
      }
      block_sum(s);
#pragma unroll
      for (int r = 0; r < R; ++r)
#pragma unroll
        for (int e = 0; e < PT; ++e) x[r][e] = feature(e) < F ? x[r][e] - s[r] * invF : 0.f;
    }
#pragma unroll
    for (int r = 0; r < R; ++r) {
      s[r] = 0.f;
#pragma unroll
      for (int e = 0; e < PT; ++e) s[r] += x[r][e] * x[r][e];
    }
    block_sum(s);
#pragma unroll
    for (int r = 0; r < R; ++r) {
      if (t + r >= t1) break;
      const float rstd = rsqrtf(s[r] * invF + eps);
#pragma unroll
      for (int e = 0; e < PT; ++e) {
        aw[e] = fmaf(g[r][e], x[r][e] * rstd, aw[e]);
        ab[e] += g[r][e];
      }
    }
    if ((chain += R) >= kChain) { to_total(); chain = 0; }
  }
  if (!first) {
    to_total();
#pragma unroll
    for (int e = 0; e < PT; ++e) {
      aw[e] = s_total[e * THREADS + threadIdx.x];
      ab[e] = s_total[(PT + e) * THREADS + threadIdx.x];
    }
  }
#pragma unroll
  for (int e = 0; e < PT; ++e) {
    const int f = feature(e);
    if (f >= F) continue;
    if (t_splits > 1) {
      float* dst = part + (static_cast<long long>(split) * gridDim.y + n) * 2 * F;
      dst[f] = aw[e];
      dst[F + f] = ab[e];
    } else {
      gw[static_cast<long long>(n) * F + f] = aw[e];
      gb[static_cast<long long>(n) * F + f] = ab[e];
    }
  }
}

// F above 8192: one block per (sample, split); rows handled one at a time by the whole block
template <typename T>
__global__ void __launch_bounds__(256)
layernorm_persample_generic_kernel(const T* __restrict__ A, const T* __restrict__ G, long long Tn, int F,
                                   float eps, float* __restrict__ gw, float* __restrict__ gb, int t_splits,
                                   int rms) {
  extern __shared__ float sm[];   // [2][F] + 32
  float* s_gw = sm;
  float* s_gb = sm + F;
  float* s_red = sm + 2 * F;
  const int n = blockIdx.y, split = blockIdx.x;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  for (int i = threadIdx.x; i < 2 * F; i += blockDim.x) sm[i] = 0.f;
  const long long per = (Tn + t_splits - 1) / t_splits;
  const long long t0 = split * per;
  const long long t1 = (t0 + per < Tn) ? t0 + per : Tn;
  const float invF = 1.f / static_cast<float>(F);
  for (long long t = t0; t < t1; ++t) {
    const T* a = A + (static_cast<long long>(n) * Tn + t) * F;
    const T* g = G + (static_cast<long long>(n) * Tn + t) * F;
    float s = 0.f;
    for (int f = threadIdx.x; f < F; f += blockDim.x) s += to_f32<T>(a[f]);
    s = warp_sum(s);
    __syncthreads();
    if (lane == 0) s_red[warp] = s;
    __syncthreads();
    float tot = 0.f;
    for (int w = 0; w < 8; ++w) tot += s_red[w];
    const float mean = rms ? 0.f : tot * invF;
    float q = 0.f;
    for (int f = threadIdx.x; f < F; f += blockDim.x) { const float dlt = to_f32<T>(a[f]) - mean; q += dlt * dlt; }
    q = warp_sum(q);
    __syncthreads();
    if (lane == 0) s_red[warp] = q;
    __syncthreads();
    tot = 0.f;
    for (int w = 0; w < 8; ++w) tot += s_red[w];
    const float rstd = rsqrtf(tot * invF + eps);
    for (int f = threadIdx.x; f < F; f += blockDim.x) {
      const float gv = to_f32<T>(g[f]);
      s_gw[f] += gv * (to_f32<T>(a[f]) - mean) * rstd;   // each f is owned by one thread
      s_gb[f] += gv;
    }
  }
  __syncthreads();
  for (int f = threadIdx.x; f < F; f += blockDim.x) {
    const long long o = static_cast<long long>(n) * F + f;
    if (t_splits > 1) { atomicAdd(&gw[o], s_gw[f]); atomicAdd(&gb[o], s_gb[f]); }
    else { gw[o] = s_gw[f]; gb[o] = s_gb[f]; }
  }
}

}  // namespace gb

using namespace gb;

static unsigned cast_blocks(long long octets, const DeviceState* ds) {
  const long long blocks = (octets + 255) / 256, most = ds->sm_count * 16;
  return static_cast<unsigned>(blocks < most ? blocks : most);
}
// element groups and rows fit 32 bits, a grid stride further too
static bool cast_narrow(const CastParams& p) {
  return p.samples * p.T * (p.cpad / 8) < (1ll << 31) && p.samples * p.T < (1ll << 31);
}

extern "C" int ghost_cast_split_bf16(const void* src, int src_is_f32, long long samples, long long T,
                                     int cols, long long ld_src, void* dst, long long ld_dst, int cpad,
                                     int parts, int kind0, int kind1, int kind2, int row_stack,
                                     void* stream) {
  const DeviceState* ds = device_state();
  if (!ds) return GHOST_ERR_DEVICE;
  GB_REQUIRE(src && dst, "ghost_cast_split_bf16: null pointer");
  GB_REQUIRE(samples > 0 && T > 0 && cols > 0, "ghost_cast_split_bf16: empty input");
  GB_REQUIRE(parts >= 1 && parts <= 3, "ghost_cast_split_bf16: parts must be 1..3");
  GB_REQUIRE(cpad % 8 == 0 && cpad >= cols, "ghost_cast_split_bf16: cpad must be a multiple of 8 and >= cols");
  GB_REQUIRE(ld_dst % 8 == 0 && ld_dst >= (row_stack ? cpad : parts * cpad), "ghost_cast_split_bf16: bad destination pitch");
  GB_REQUIRE((reinterpret_cast<uintptr_t>(dst) & 15u) == 0,
             "ghost_cast_split_bf16: destination must be 16-byte aligned");
  const CastParams p = {src, static_cast<__nv_bfloat16*>(dst), samples, T, cols, cpad, ld_src, ld_dst, parts, {kind0, kind1, kind2},
                        row_stack, cast_blocks(samples * T * (cpad / 8), ds)};
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  const unsigned grid = p.blocks;
  if (cast_narrow(p)) {
    if (src_is_f32) GB_CUDA_OK(launch_next(cast_split_kernel<float, unsigned>, dim3(grid), dim3(256), 0, st, p));
    else GB_CUDA_OK(launch_next(cast_split_kernel<__nv_bfloat16, unsigned>, dim3(grid), dim3(256), 0, st, p));
  } else {
    if (src_is_f32) GB_CUDA_OK(launch_next(cast_split_kernel<float, long long>, dim3(grid), dim3(256), 0, st, p));
    else GB_CUDA_OK(launch_next(cast_split_kernel<__nv_bfloat16, long long>, dim3(grid), dim3(256), 0, st, p));
  }
  count_launch();
  return post_launch("cast_split_kernel");
}

// Operands up to this many bytes have their column sums added up by clusters
static constexpr double kClusterBytes = 16e6;

static int pick_splits(long long Tn, long long ctas_without_split, int sm_count, int rows_per_cta_min) {
  long long want = (4ll * sm_count + ctas_without_split - 1) / ctas_without_split;
  long long maxs = (Tn + rows_per_cta_min - 1) / rows_per_cta_min;
  if (want > maxs) want = maxs;
  if (want < 1) want = 1;
  if (want > 65535) want = 65535;
  return static_cast<int>(want);
}

extern "C" int ghost_split_operands(const void* X, int x_is_f32, int x_cols, const void* Y, int y_is_f32, int y_cols, int parts,
                                    long long samples, long long T, int merged, void* X_out, void* Y_out, float* x_sums,
                                    float* y_sums, void* stream) {
  const DeviceState* ds = device_state();
  if (!ds) return GHOST_ERR_DEVICE;
  GB_REQUIRE((X == nullptr) == (X_out == nullptr) && (Y == nullptr) == (Y_out == nullptr) && (X || Y), "ghost_split_operands: null pointer");
  GB_REQUIRE((X || !x_sums) && (Y || !y_sums), "ghost_split_operands: sums of an operand that is not there");
  GB_REQUIRE(samples > 0 && T > 0 && (!X || x_cols > 0) && (!Y || y_cols > 0), "ghost_split_operands: empty dimension");
  GB_REQUIRE(parts == 1 || parts == 2, "ghost_split_operands: one or two parts");
  GB_REQUIRE(((reinterpret_cast<uintptr_t>(X_out) | reinterpret_cast<uintptr_t>(Y_out)) & 15u) == 0,
             "ghost_split_operands: destinations must be 16-byte aligned");
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  if (parts == 1 && !x_sums && !y_sums && !(X && x_is_f32) && !(Y && y_is_f32)) {
    CastPair pair = {};
    auto copy = [&](CastParams& q, const void* src, int cols, void* dst) {
      if (!src) return;
      const int cpad = (cols + 63) / 64 * 64;
      q = CastParams{src, static_cast<__nv_bfloat16*>(dst), samples, T, cols, cpad, cols, cpad, 1, {0, 0, 0}, 1,
                     cast_blocks(samples * T * (cpad / 8), ds)};
    };
    copy(pair.job[0], X, x_cols, X_out);
    copy(pair.job[1], Y, y_cols, Y_out);
    const dim3 grid(pair.job[0].blocks + pair.job[1].blocks);
    if (cast_narrow(pair.job[0]) && cast_narrow(pair.job[1])) GB_CUDA_OK(launch_next(cast_pair_kernel<unsigned>, grid, dim3(256), 0, st, pair));
    else GB_CUDA_OK(launch_next(cast_pair_kernel<long long>, grid, dim3(256), 0, st, pair));
    count_launch();
    return post_launch("cast_pair_kernel");
  }
  SplitParams p = {};
  p.T = T;
  p.part_rows = merged ? samples * T : T;
  auto fill = [&](SplitJob& j, const void* src, int f32, int cols, void* dst, float* sums) {
    j.panels = 1;
    if (!src) return;
    j.src = src;
    j.dst = static_cast<__nv_bfloat16*>(dst);
    j.sums = sums;
    j.is_f32 = f32;
    j.cols = cols;
    j.panels = ceil_div(cols, kSplitCols);
    j.ld = (cols + 63) / 64 * 64;
    j.rows = samples * T;
    j.vec = cols % (f32 ? 4 : 8) == 0 && (reinterpret_cast<uintptr_t>(src) & 15u) == 0;
    // 64 rows to a block (two rounds of loads) while that is a few waves of blocks, more rows beyond it.  Sums: a sample to a
    // block and no atomics where that fills the GPU; up to 512 rows, so that a chain of additions has sixteen at most.
    const long long units = sums ? T : j.rows, each = (sums ? samples : 1) * j.panels, wave = 4ll * ds->sm_count;
    j.per = 64;
    if (sums && each >= wave && T <= 512) j.per = (units + 63) / 64 * 64;
    while (j.per < (sums ? 512 : units) && (units + j.per - 1) / j.per * each > 16 * wave) j.per *= 2;
    j.chunks = static_cast<int>((units + j.per - 1) / j.per);
    j.used = j.blocks = j.chunks * each;
  };
  fill(p.job[0], X, x_is_f32, x_cols, X_out, x_sums);
  fill(p.job[1], Y, y_is_f32, y_cols, Y_out, y_sums);
  // The chunks of a sample add their sums up as a cluster, of up to eight; sums of both operands, or of more chunks, are added
  // to zeros, which take a launch: 3 us or more where the host bounds the hook (10 x 512 of (256, 256) float32 44.9 -> 41.2, 34 x 127
  // of (126, 640) 44.7 -> 40.9).  Large operands keep it: clusters walk down a panel where blocks on their own read along
  // the rows (29 x 197 of (768, 1000), 41 MB: 77.6 against 80.3; 30 x 200 of (500, 700), 29 MB: 47.6 against 50.0).
  const int summed = p.job[0].sums ? 0 : 1;
  const bool both = p.job[0].sums && p.job[1].sums;
  double read = 0.;
  for (const SplitJob& j : p.job) read += j.src ? static_cast<double>(j.rows) * j.cols * (j.is_f32 ? 4 : 2) : 0.;
  const int ranks = !both && read <= kClusterBytes && p.job[summed].sums && p.job[summed].chunks <= 8 ? p.job[summed].chunks : 1;
  for (SplitJob& j : p.job) {
    j.ranks = j.sums ? ranks : 1;
    j.blocks = (j.used + ranks - 1) / ranks * ranks;
    if (j.sums && j.chunks > 1 && ranks == 1)
      if (int rc = clear_ahead(j.sums, sizeof(float) * static_cast<size_t>(samples) * j.cols, st)) return rc;
  }
  const long long blocks = p.job[0].blocks + p.job[1].blocks;
  GB_REQUIRE(blocks < (1ll << 31), "ghost_split_operands: too many rows");
  GB_CUDA_OK(launch_next_cluster(dim3(ranks), parts == 1 ? split_pair_kernel<1> : split_pair_kernel<2>, dim3(static_cast<unsigned>(blocks)),
                                 dim3(256), 0, st, p));
  count_launch();
  return post_launch("split_pair_kernel");
}

extern "C" int ghost_colsum(const void* G, int is_f32, int N, long long T, int cols, long long ld,
                            float* out, void* stream) {
  const DeviceState* ds = device_state();
  if (!ds) return GHOST_ERR_DEVICE;
  GB_REQUIRE(G && out, "ghost_colsum: null pointer");
  GB_REQUIRE(N > 0 && T > 0 && cols > 0 && N <= 65535, "ghost_colsum: bad dimensions");
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  const int cblocks = ceil_div(cols, 256);
  // Up to eight splits are a cluster that adds up their sums (6 x 512 rows of 768 bf16, the hook: 45.1 -> 41.3 us, the host's); more, of
  // longer samples, add to zeros, and so do large operands (6 x 512 of 3072: 50.4 against 51.5).
  const bool small = static_cast<double>(N) * T * cols * (is_f32 ? 4 : 2) <= kClusterBytes;
  int splits = pick_splits(T, static_cast<long long>(cblocks) * N, ds->sm_count, 64);
  if (small && splits > 8 && T <= 8 * 128) splits = 8;
  const int ranks = small && splits <= 8 ? splits : 1;
  if (splits > ranks)
    if (int rc = clear_ahead(out, sizeof(float) * static_cast<size_t>(N) * cols, st)) return rc;
  const dim3 grid(cblocks, splits, N), cluster(1, ranks, 1);
  if (is_f32) GB_CUDA_OK(launch_next_cluster(cluster, colsum_kernel<float>, grid, dim3(256), 0, st, static_cast<const float*>(G), T, cols, ld, out, splits, ranks > 1 ? 1 : 0));
  else GB_CUDA_OK(launch_next_cluster(cluster, colsum_kernel<__nv_bfloat16>, grid, dim3(256), 0, st, static_cast<const __nv_bfloat16*>(G), T, cols, ld, out, splits, ranks > 1 ? 1 : 0));
  count_launch();
  return post_launch("colsum_kernel");
}

static int ln_splits(long long Tn, int N, int resident, int min_rows) {
  long long want = resident / N;           // one wave
  const long long maxs = (Tn + min_rows - 1) / min_rows;
  if (want > maxs) want = maxs;
  if (want < 1) want = 1;
  return static_cast<int>(want);
}

// Rows below which another split costs more than it gives: a warp of the warp-per-row kernel should see eight,
// a block of the wide kernel goes through its rows two to eight at a time.
static constexpr int kLnMinRows = 64, kLnWideMinRows = 8;

extern "C" long long ghost_layernorm_workspace_bytes(int N, long long T, int F) {
  // one wave of at most two CTAs per SM over the N samples: 512 is above any device this runs on
  long long splits = (T + kLnWideMinRows - 1) / kLnWideMinRows;
  const long long wave = N > 0 ? 512 / N : 1;
  if (splits > wave) splits = wave;
  if (splits < 1) splits = 1;
  return splits * N * 2 * F * 4 + 256;
}

template <typename T, bool VEC, int PT, int THREADS>
static int launch_norm_wide_of(dim3 grid, const T* A, const T* G, long long Tn, int F, float eps, float* gw, float* gb, float* ws,
                               int splits, const DeviceState* ds, cudaStream_t st, int rms) {
  constexpr int kSmem = 2 * PT * THREADS * 4;
  static bool attr_set[64] = {};
  if (kSmem > 47 * 1024 && !attr_set[ds->device]) {
    GB_CUDA_OK(cudaFuncSetAttribute(norm_wide_kernel<T, VEC, PT, THREADS>, cudaFuncAttributeMaxDynamicSharedMemorySize, kSmem));
    attr_set[ds->device] = true;
  }
  GB_CUDA_OK(launch_next(norm_wide_kernel<T, VEC, PT, THREADS>, dim3(grid), dim3(THREADS), kSmem, st, A, G, Tn, F, eps, gw, gb, ws, splits, rms));
  return GHOST_OK;
}
template <typename T, bool VEC>
static int launch_norm_wide(dim3 grid, const T* A, const T* G, long long Tn, int F, float eps, float* gw, float* gb, float* ws,
                            int splits, const DeviceState* ds, cudaStream_t st, int rms) {
  // Rows that begin anywhere are loaded element by element, and a feature beyond F costs its instructions all the same (bf16 RMS
  // hooks of 6 + 2 x 1024, with 16 features a thread and as many as the row needs, us: F = 2501 52.4 and 42.4,
  // 3001 54.9 and 47.7, 4097 92 and 72, 5999 106 and 92; float32 4097 84 and 73; 16 features of fewer threads: 4097 93, float32 75).
  // Pieces of eight keep 16 features a thread and take the threads that the row needs, which leaves each more registers for
  // loads in flight (LayerNorm hooks, 256 or 512 threads and as many as needed: bf16 2304 44.7 and 39.6, 4104 84.5 and 69.6,
  // 6144 89.8 and 78, 7000 95.4 and 92.3; float32 5120 97.7 and 84.3; 224 threads for 3456: no difference).
  if constexpr (!VEC) {
    if (F <= 1024) return launch_norm_wide_of<T, false, 4, 256>(grid, A, G, Tn, F, eps, gw, gb, ws, splits, ds, st, rms);
    if (F <= 2048) return launch_norm_wide_of<T, false, 8, 256>(grid, A, G, Tn, F, eps, gw, gb, ws, splits, ds, st, rms);
    if (F <= 2560) return launch_norm_wide_of<T, false, 10, 256>(grid, A, G, Tn, F, eps, gw, gb, ws, splits, ds, st, rms);
    if (F <= 3072) return launch_norm_wide_of<T, false, 12, 256>(grid, A, G, Tn, F, eps, gw, gb, ws, splits, ds, st, rms);
    if (F <= 4096) return launch_norm_wide_of<T, false, 16, 256>(grid, A, G, Tn, F, eps, gw, gb, ws, splits, ds, st, rms);
    if (F <= 5120) return launch_norm_wide_of<T, false, 10, 512>(grid, A, G, Tn, F, eps, gw, gb, ws, splits, ds, st, rms);
    if (F <= 6144) return launch_norm_wide_of<T, false, 12, 512>(grid, A, G, Tn, F, eps, gw, gb, ws, splits, ds, st, rms);
  } else {
    if (F <= 2048) return launch_norm_wide_of<T, true, 8, 256>(grid, A, G, Tn, F, eps, gw, gb, ws, splits, ds, st, rms);
    if (F <= 3072) return launch_norm_wide_of<T, true, 16, 192>(grid, A, G, Tn, F, eps, gw, gb, ws, splits, ds, st, rms);
    if (F <= 4096) return launch_norm_wide_of<T, true, 16, 256>(grid, A, G, Tn, F, eps, gw, gb, ws, splits, ds, st, rms);
    if (F <= 5120) return launch_norm_wide_of<T, true, 16, 320>(grid, A, G, Tn, F, eps, gw, gb, ws, splits, ds, st, rms);
    if (F <= 6144) return launch_norm_wide_of<T, true, 16, 384>(grid, A, G, Tn, F, eps, gw, gb, ws, splits, ds, st, rms);
    if (F <= 7168) return launch_norm_wide_of<T, true, 16, 448>(grid, A, G, Tn, F, eps, gw, gb, ws, splits, ds, st, rms);
  }
  return launch_norm_wide_of<T, VEC, 16, 512>(grid, A, G, Tn, F, eps, gw, gb, ws, splits, ds, st, rms);
}

template <typename T, int NCHUNK, bool FULL>
static int launch_ln_warp(dim3 grid, size_t smem, const T* A, const T* G, long long Tn, int F, float eps, float* gw, float* gb, float* ws,
                          int splits, const DeviceState* ds, cudaStream_t st, int rms) {
  static bool attr_set[64] = {};
  if (!attr_set[ds->device]) {
    GB_CUDA_OK(cudaFuncSetAttribute(layernorm_persample_kernel<T, NCHUNK, FULL>, cudaFuncAttributeMaxDynamicSharedMemorySize, 200 * 1024));
    attr_set[ds->device] = true;
  }
  GB_CUDA_OK(launch_next(layernorm_persample_kernel<T, NCHUNK, FULL>, dim3(grid), dim3(256), smem, st, A, G, Tn, F, eps, gw, gb, ws, splits, rms));
  return GHOST_OK;
}

template <typename T>
static int launch_ln(const T* A, const T* G, int N, long long Tn, int F, float eps, float* gw, float* gb,
                     float* ws, long long ws_bytes, const DeviceState* ds, cudaStream_t st, int rms) {
  const bool aligned = (F % 8 == 0) && ((reinterpret_cast<uintptr_t>(A) & 15u) == 0) && ((reinterpret_cast<uintptr_t>(G) & 15u) == 0);
  const int resident = (F <= 4096 ? 2 : 1) * (ds->sm_count < 256 ? ds->sm_count : 256);
  int splits = ln_splits(Tn, N, resident, aligned && F <= 1024 ? kLnMinRows : kLnWideMinRows);
  const bool room = splits == 1 || (ws && ws_bytes >= static_cast<long long>(splits) * N * 2 * F * 4);
  if (aligned && F <= 1024) GB_REQUIRE(room, "ghost_layernorm_persample: workspace too small");
  if (F <= 8192 && room) {               // the kernel after it needs no workspace
    dim3 grid(splits, N);
    // per-warp cp.async rings (3 slots x (A row + G row)), reused for the cross-warp reduction
    const size_t ring = sizeof(T) * 8 * kLnSlots * 2 * static_cast<size_t>(F);
    const size_t red = sizeof(float) * 8 * 2 * static_cast<size_t>(F);
    const size_t smem = ring > red ? ring : red;
    const int nchunk = aligned ? (F + 255) / 256 : 0;
    int rc = GHOST_OK;
#define GB_LN_LAUNCH(NC)                                                                              \
    rc = F == 256 * NC ? launch_ln_warp<T, NC, true>(grid, smem, A, G, Tn, F, eps, gw, gb, ws, splits, ds, st, rms) \
                       : launch_ln_warp<T, NC, false>(grid, smem, A, G, Tn, F, eps, gw, gb, ws, splits, ds, st, rms)
    switch (nchunk) {
      case 0: rc = launch_norm_wide<T, false>(grid, A, G, Tn, F, eps, gw, gb, ws, splits, ds, st, rms); break;
      case 1: GB_LN_LAUNCH(1); break;
      case 2: GB_LN_LAUNCH(2); break;
      case 3: GB_LN_LAUNCH(3); break;
      case 4: GB_LN_LAUNCH(4); break;
      default: rc = launch_norm_wide<T, true>(grid, A, G, Tn, F, eps, gw, gb, ws, splits, ds, st, rms); break;
    }
    if (rc != GHOST_OK) return rc;
#undef GB_LN_LAUNCH
    count_launch();
    rc = post_launch("layernorm_persample_kernel");
    if (rc != GHOST_OK || splits == 1) return rc;
    const long long total = static_cast<long long>(N) * 2 * F;
    long long blocks = (total + 255) / 256;
    if (blocks > ds->sm_count * 8) blocks = ds->sm_count * 8;
    GB_CUDA_OK(launch_next(layernorm_reduce_kernel, dim3(static_cast<int>(blocks)), dim3(256), 0, st, ws, N, F, splits, gw, gb));
    count_launch();
    return post_launch("layernorm_reduce_kernel");
  }
  splits = pick_splits(Tn, N, ds->sm_count, 32);
  if (splits > 1) {
    GB_CUDA_OK(cudaMemsetAsync(gw, 0, sizeof(float) * static_cast<size_t>(N) * F, st));
    GB_CUDA_OK(cudaMemsetAsync(gb, 0, sizeof(float) * static_cast<size_t>(N) * F, st));
  }
  dim3 grid(splits, N);
  const size_t smem = sizeof(float) * (2 * static_cast<size_t>(F) + 32);
  if (smem > 48 * 1024)
    GB_CUDA_OK(cudaFuncSetAttribute(layernorm_persample_generic_kernel<T>,
                                    cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(smem)));
  layernorm_persample_generic_kernel<T><<<grid, 256, smem, st>>>(A, G, Tn, F, eps, gw, gb, splits, rms);
  count_launch();
  return post_launch("layernorm_persample_generic_kernel");
}

static int norm_persample(const char* who, const void* A, const void* G, int is_f32, int N, long long T, int F,
                          float eps, float* gw, float* gb, void* ws, long long ws_bytes, void* stream, int rms) {
  const DeviceState* ds = device_state();
  if (!ds) return GHOST_ERR_DEVICE;
  GB_REQUIRE(A && G && gw && gb, "%s: null pointer", who);
  GB_REQUIRE(N > 0 && T > 0 && F > 0 && N <= 65535, "%s: bad dimensions", who);
  GB_REQUIRE(F <= 24 * 1024, "%s: normalized size above 24576 is not supported", who);
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  float* w = static_cast<float*>(ws);
  if (is_f32) return launch_ln<float>(static_cast<const float*>(A), static_cast<const float*>(G), N, T, F, eps, gw, gb, w, ws_bytes, ds, st, rms);
  return launch_ln<__nv_bfloat16>(static_cast<const __nv_bfloat16*>(A), static_cast<const __nv_bfloat16*>(G), N, T, F, eps, gw, gb, w, ws_bytes, ds, st, rms);
}

extern "C" int ghost_layernorm_persample(const void* A, const void* G, int is_f32, int N, long long T,
                                         int F, float eps, float* gw, float* gb, void* ws,
                                         long long ws_bytes, void* stream) {
  return norm_persample("ghost_layernorm_persample", A, G, is_f32, N, T, F, eps, gw, gb, ws, ws_bytes, stream, 0);
}

extern "C" int ghost_rmsnorm_persample(const void* A, const void* G, int is_f32, int N, long long T,
                                       int F, float eps, float* gw, float* gsum, void* ws,
                                       long long ws_bytes, void* stream) {
  return norm_persample("ghost_rmsnorm_persample", A, G, is_f32, N, T, F, eps, gw, gsum, ws, ws_bytes, stream, 1);
}
