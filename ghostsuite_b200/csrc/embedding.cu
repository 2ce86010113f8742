// Embedding-table terms of the ghost hot path (index / gather work, HBM- and latency-bound).
//
// embedding_dot:  M[v, b] = sum_{t, s : id_b[t] == id_v[s]} <G_b[t], G_v[s]>
//   The reference scatters the validation rows into a [vocab, d] table and gathers it at the train
//   ids (ghostEngines/supported_layers_grad_samplers_dotprod.py:203-210); here train and validation
//   tokens are bucketed by id and joined id by id, so no [vocab, d] scratch exists, every row is
//   fetched about once, and the result is split per validation sample.
//
// embedding_wgrad: averaged train gradient of the table (:214-235).  Each train bucket is summed in
//   ascending token order in float32, rounded to the table dtype once, then divided by n_train --
//   the arithmetic and the order of the CPU index_add_, so the result is bit-identical to it.
//
// Both results share the buckets (count, allocate, fill): ghost_embedding_pass makes them once.
#include <limits.h>

#include <mutex>

#include "common.cuh"
#include "mma_sync.cuh"
#include "sm100_ptx.cuh"

namespace gb {

__device__ __forceinline__ float ewarp_sum(float v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}
template <typename T> __device__ __forceinline__ float ld_f32(const T* p);
template <> __device__ __forceinline__ float ld_f32<float>(const float* p) { return *p; }
template <> __device__ __forceinline__ float ld_f32<__nv_bfloat16>(const __nv_bfloat16* p) { return __bfloat162float(*p); }
template <typename T> __device__ __forceinline__ float round_to(float x);
template <> __device__ __forceinline__ float round_to<float>(float x) { return x; }
template <> __device__ __forceinline__ float round_to<__nv_bfloat16>(float x) { return __bfloat162float(__float2bfloat16_rn(x)); }
__device__ __forceinline__ void load8(const float* p, float (&x)[8]) {
  const float4 a = *reinterpret_cast<const float4*>(p);
  const float4 b = *reinterpret_cast<const float4*>(p + 4);
  x[0] = a.x; x[1] = a.y; x[2] = a.z; x[3] = a.w; x[4] = b.x; x[5] = b.y; x[6] = b.z; x[7] = b.w;
}
__device__ __forceinline__ void load8(const __nv_bfloat16* p, float (&x)[8]) {
  const uint4 w = *reinterpret_cast<const uint4*>(p);
  const uint32_t ww[4] = {w.x, w.y, w.z, w.w};
#pragma unroll
  for (int e = 0; e < 4; ++e) {
    x[2 * e] = __uint_as_float(ww[e] << 16);
    x[2 * e + 1] = __uint_as_float(ww[e] & 0xffff0000u);
  }
}
__device__ __forceinline__ void store8(float* p, const float (&x)[8]) {
  *reinterpret_cast<float4*>(p) = make_float4(x[0], x[1], x[2], x[3]);
  *reinterpret_cast<float4*>(p + 4) = make_float4(x[4], x[5], x[6], x[7]);
}
__device__ __forceinline__ void store8(__nv_bfloat16* p, const float (&x)[8]) {
  uint32_t w[4];
#pragma unroll
  for (int e = 0; e < 4; ++e) {
    const __nv_bfloat162 h = __floats2bfloat162_rn(x[2 * e], x[2 * e + 1]);
    w[e] = *reinterpret_cast<const uint32_t*>(&h);
  }
  *reinterpret_cast<uint4*>(p) = make_uint4(w[0], w[1], w[2], w[3]);
}
template <typename T> __device__ __forceinline__ T from_f32(float x);
template <> __device__ __forceinline__ float from_f32<float>(float x) { return x; }
template <> __device__ __forceinline__ __nv_bfloat16 from_f32<__nv_bfloat16>(float x) { return __float2bfloat16_rn(x); }

// ---------------------------------------------------------------- dot product, least workspace
// Validation tokens chained per id in a vocab-sized head table; every train token walks the chain of its
// id.  For callers that have no room for the buckets (ghost_embedding_dot_noalloc).
__global__ void emb_chain_val_kernel(const long long* __restrict__ ids_val, long long n_tok, int vocab,
                                     int* __restrict__ head, int* __restrict__ next, int* __restrict__ err) {
  for (long long j = blockIdx.x * static_cast<long long>(blockDim.x) + threadIdx.x; j < n_tok;
       j += static_cast<long long>(gridDim.x) * blockDim.x) {
    const long long id = ids_val[j];
    if (id >= 0 && id < vocab) {
      next[j] = atomicExch(&head[id], static_cast<int>(j));
    } else {            // the reference's index_add_ raises here; skipped and reported through the error word
      next[j] = -1;
      atomicExch(err, kErrBadIndex);
    }
  }
}

// grid (token blocks of one sample, n_train); 8 warps, each walks kTokPerWarp tokens
template <typename T>
__global__ void __launch_bounds__(256)
emb_chain_dot_kernel(const long long* __restrict__ ids, const T* __restrict__ G, int n_train, int n_val,
               long long Tn, int d, int vocab, const int* __restrict__ head,
               const int* __restrict__ next, float scale, float* __restrict__ M, int tok_per_block, int* __restrict__ err) {
  extern __shared__ float s_acc[];   // [n_val]
  const int b = blockIdx.y;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  for (int v = threadIdx.x; v < n_val; v += blockDim.x) s_acc[v] = 0.f;
  __syncthreads();
  const long long t_begin = static_cast<long long>(blockIdx.x) * tok_per_block;
  long long t_end = t_begin + tok_per_block;
  if (t_end > Tn) t_end = Tn;
  const T* Gval = G + static_cast<long long>(n_train) * Tn * d;
  const bool vec = (d % 8 == 0) && ((reinterpret_cast<uintptr_t>(G) & 15u) == 0);
  for (long long t = t_begin + warp; t < t_end; t += 8) {
    const long long id = ids[static_cast<long long>(b) * Tn + t];
    if (id < 0 || id >= vocab) {
      if (lane == 0) atomicExch(err, kErrBadIndex);
      continue;
    }
    int j = head[id];
    const T* row = G + (static_cast<long long>(b) * Tn + t) * d;
    while (j >= 0) {
      const T* vrow = Gval + static_cast<long long>(j) * d;
      float s = 0.f;
      if (vec && sizeof(T) == 2) {
        for (int f = lane * 8; f < d; f += 256) {
          const uint4 x = *reinterpret_cast<const uint4*>(row + f);
          const uint4 y = *reinterpret_cast<const uint4*>(vrow + f);
          const uint32_t xx[4] = {x.x, x.y, x.z, x.w}, yy[4] = {y.x, y.y, y.z, y.w};
#pragma unroll
          for (int e = 0; e < 4; ++e) {
            s = fmaf(__uint_as_float(xx[e] << 16), __uint_as_float(yy[e] << 16), s);
            s = fmaf(__uint_as_float(xx[e] & 0xffff0000u), __uint_as_float(yy[e] & 0xffff0000u), s);
          }
        }
      } else {
        for (int f = lane; f < d; f += 32) s = fmaf(ld_f32<T>(row + f), ld_f32<T>(vrow + f), s);
      }
      s = ewarp_sum(s);
      if (lane == 0) atomicAdd(&s_acc[j / Tn], s);
      j = next[j];
    }
  }
  __syncthreads();
  for (int v = threadIdx.x; v < n_val; v += blockDim.x) {
    const float s = s_acc[v];
    if (s != 0.f) atomicAdd(&M[static_cast<long long>(v) * n_train + b], s * scale);
  }
}

// Shared pieces of the two segment-sum kernels.  A thread owns 8 consecutive features.
template <typename T>
__device__ __forceinline__ void emb_load_row(const T* G, int j, int d, int f, bool vec, float (&x)[8]) {
  const T* row = G + static_cast<long long>(j) * d + f;
  if (vec) {
    if (f < d) {
      load8(row, x);
    } else {
#pragma unroll
      for (int e = 0; e < 8; ++e) x[e] = 0.f;
    }
  } else {
#pragma unroll
    for (int e = 0; e < 8; ++e) x[e] = (f + e < d) ? ld_f32<T>(row + e) : 0.f;
  }
}
// no fma contraction: product and sum are rounded separately, as the reference does
template <typename T>
__device__ __forceinline__ void emb_accumulate(const float (&x)[8], float pre_scale, float (&acc)[8]) {
#pragma unroll
  for (int e = 0; e < 8; ++e) acc[e] = __fadd_rn(acc[e], round_to<T>(__fmul_rn(x[e], pre_scale)));
}
template <typename T>
__device__ __forceinline__ void emb_store_row(T* __restrict__ out, int k, int d, int f, bool vec, const float (&acc)[8],
                                              float divisor, int accumulate) {
  T* dst = out + static_cast<long long>(k) * d + f;
  float o[8];
  // dividing by a power of two and multiplying by its reciprocal are the same rounding of the same number
  const bool pow2 = (__float_as_uint(divisor) & 0x7fffffu) == 0;
  const float inv = 1.f / divisor;
#pragma unroll
  for (int e = 0; e < 8; ++e) {
    o[e] = round_to<T>(pow2 ? __fmul_rn(round_to<T>(acc[e]), inv) : __fdiv_rn(round_to<T>(acc[e]), divisor));
    if (accumulate && f + e < d) o[e] = round_to<T>(__fadd_rn(ld_f32<T>(dst + e), o[e]));
  }
  if (vec) {
    if (f < d) store8(dst, o);
  } else {
#pragma unroll
    for (int e = 0; e < 8; ++e)
      if (f + e < d) dst[e] = from_f32<T>(o[e]);
  }
}

// Eight consecutive features of a row as loaded (16 bytes of bf16, 32 bytes of float32)
template <typename T> struct EmbRaw;
template <> struct EmbRaw<__nv_bfloat16> {
  using type = uint4;
  static __device__ __forceinline__ uint4 load(const __nv_bfloat16* p) { return *reinterpret_cast<const uint4*>(p); }
  static __device__ __forceinline__ uint4 zero() { return make_uint4(0u, 0u, 0u, 0u); }
  static __device__ __forceinline__ void unpack(const uint4& w, float (&x)[8]) {
    const uint32_t ww[4] = {w.x, w.y, w.z, w.w};
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      x[2 * e] = __uint_as_float(ww[e] << 16);
      x[2 * e + 1] = __uint_as_float(ww[e] & 0xffff0000u);
    }
  }
};
struct EmbFloat8 { float4 a, b; };
template <> struct EmbRaw<float> {
  using type = EmbFloat8;
  static __device__ __forceinline__ EmbFloat8 load(const float* p) {
    EmbFloat8 r;
    r.a = *reinterpret_cast<const float4*>(p);
    r.b = *reinterpret_cast<const float4*>(p + 4);
    return r;
  }
  static __device__ __forceinline__ EmbFloat8 zero() {
    EmbFloat8 r;
    r.a = make_float4(0.f, 0.f, 0.f, 0.f);
    r.b = r.a;
    return r;
  }
  static __device__ __forceinline__ void unpack(const EmbFloat8& w, float (&x)[8]) {
    x[0] = w.a.x; x[1] = w.a.y; x[2] = w.a.z; x[3] = w.a.w; x[4] = w.b.x; x[5] = w.b.y; x[6] = w.b.z; x[7] = w.b.w;
  }
};

// ---------------------------------------------------------------- buckets of tokens by id
// Train and validation tokens have indices of their own, both from zero; a scan runs over the train tokens
// and then, from `first_val` on, over the validation tokens.
struct EmbBuckets {
  const long long *ids_b, *ids_v;
  long long n_tok, first_val;           // tokens that take part, train tokens among them
  int vocab;
  int *cnt_b, *cnt_v;                   // [vocab] tokens per id, train / validation (cnt_v null: no dot products)
  int *off_b, *off_v;                   // [vocab] first position of the id's bucket in perm_b / perm_v
  int *rank;                            // [n_tok] position inside the bucket, -1 for an id outside the table
  int *perm_b, *perm_v;
  int *totals;                          // [0] train tokens placed, [1] validation, [2] big rows, [3] items, [4] hot ids, [5] small rows,
                                        // [6, 7] 64-bit count of gradient items handed out, [8] CTAs done with the join, [9] table rows looked over
  int4 *small;                          // (id, offset, tokens) of the rows with 1 to kEmbSmallBucket train tokens
  int *big;                             // ids with more than kEmbSmallBucket train tokens
  int4 *items;                          // join items: (first train position, train rows, first validation position
                                        // or slot, validation rows or -1 for the slot's summed rows)
  int *hot;                             // ids by slot
  long long max_items;
  int hot_threshold, max_parts, want_rows;         // want_rows: the train gradient is wanted, list its rows
  int* err;
};

constexpr int kEmbSmallBucket = 32;      // buckets up to this size are sorted and summed by one warp
constexpr int kEmbHotCap = 256;
constexpr int kEmbTotals = 12;
constexpr int kEmbChunk = 8;             // train rows of a join item
constexpr int kEmbValChunk = 32;         // validation rows of a join item

// Counting hands every token its place in the bucket, so filling needs no second round of atomics.
__device__ __forceinline__ void emb_count_tokens(const EmbBuckets& q, long long first, long long step) {
  for (long long j = first; j < q.n_tok; j += step) {
    const long long id = j < q.first_val ? q.ids_b[j] : q.ids_v[j - q.first_val];
    if (id >= 0 && id < q.vocab) {
      q.rank[j] = atomicAdd((j < q.first_val ? q.cnt_b : q.cnt_v) + id, 1);
    } else {            // the reference's index_add_ raises here; skipped and reported through the error word
      q.rank[j] = -1;
      atomicExch(q.err, kErrBadIndex);
    }
  }
}
// It also clears the sums that the join adds to two launches later, and zero-fills a gradient of odd width.
__global__ void __launch_bounds__(256) emb_count_kernel(const EmbBuckets q, double* __restrict__ M64, long long m_size,
                                                        uint4* __restrict__ zero, long long zero_size) {
  stream_order();
  if (M64 != nullptr)
    for (long long i = blockIdx.x * 256ll + threadIdx.x; i < m_size; i += gridDim.x * 256ll) M64[i] = 0.;
  emb_count_tokens(q, blockIdx.x * 256ll + threadIdx.x, gridDim.x * 256ll);
  const uint4 z = make_uint4(0u, 0u, 0u, 0u);
  for (long long i = blockIdx.x * 256ll + threadIdx.x; i < zero_size; i += gridDim.x * 256ll) zero[i] = z;
}

// Buckets may lie in any order, so a block of ids takes its space with one atomic instead of waiting for
// a scan over the whole table (22 us in one block for 50 k ids, 4.6 us now).  Also listed here: the
// gradient's rows by size, join items, and ids that many validation tokens share (padding, separators).
// Every thread of the block has an id of its own, or none (in).
template <int WARPS>
__device__ __forceinline__ void emb_alloc_ids(const EmbBuckets& q, int id, bool in) {
  __shared__ int s_warp[3][WARPS], s_base[3];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int tokens = in ? q.cnt_b[id] : 0;
  const int n[3] = {tokens, in && q.cnt_v ? q.cnt_v[id] : 0, q.want_rows && tokens > 0 && tokens <= kEmbSmallBucket ? 1 : 0};
  int before[3];
#pragma unroll
  for (int h = 0; h < 3; ++h) {
    int x = n[h];
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int y = __shfl_up_sync(0xffffffffu, x, o);
      if (lane >= o) x += y;
    }
    before[h] = x - n[h];
    if (lane == 31) s_warp[h][warp] = x;
  }
  __syncthreads();
  if (threadIdx.x < 3) {
    int sum = 0;
#pragma unroll
    for (int w = 0; w < WARPS; ++w) { const int c = s_warp[threadIdx.x][w]; s_warp[threadIdx.x][w] = sum; sum += c; }
    s_base[threadIdx.x] = sum ? atomicAdd(q.totals + (threadIdx.x == 2 ? 5 : threadIdx.x), sum) : 0;
  }
  __syncthreads();
  const int off = s_base[0] + s_warp[0][warp] + before[0];
  if (in) q.off_b[id] = off;
  if (n[2]) q.small[s_base[2] + s_warp[2][warp] + before[2]] = make_int4(id, off, tokens, 0);
  if (q.want_rows && n[0] > kEmbSmallBucket) q.big[atomicAdd(q.totals + 2, 1)] = id;
  if (q.cnt_v == nullptr) return;
  const int off_v = s_base[1] + s_warp[1][warp] + before[1];
  if (in) q.off_v[id] = off_v;
  int slot = -1, parts = 0;
  if (n[1] > 0 && n[0] > 0) {
    if (n[1] > q.hot_threshold) {
      slot = atomicAdd(q.totals + 4, 1);
      if (slot < kEmbHotCap) q.hot[slot] = id; else slot = -1;
    }
    parts = slot >= 0 ? 1 : (n[1] + kEmbValChunk - 1) / kEmbValChunk;
    // more hot ids than slots: their long validation lists stay in one item per train chunk
    if (parts > q.max_parts) parts = -1;
  }
  // the items of an id are written by the whole warp: a frequent word has hundreds
  const int count = (n[0] + kEmbChunk - 1) / kEmbChunk * (parts < 0 ? 1 : parts);
  int at = count;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const int y = __shfl_up_sync(0xffffffffu, at, o);
    if (lane >= o) at += y;
  }
  const int warp_items = __shfl_sync(0xffffffffu, at, 31);
  int base = 0;
  if (lane == 0 && warp_items > 0) base = atomicAdd(q.totals + 3, warp_items);
  at += __shfl_sync(0xffffffffu, base, 0) - count;
  for (unsigned todo = __ballot_sync(0xffffffffu, count > 0); todo != 0; todo &= todo - 1) {
    const int who = __ffs(todo) - 1;
    const int w_count = __shfl_sync(0xffffffffu, count, who), w_at = __shfl_sync(0xffffffffu, at, who);
    const int w_parts = __shfl_sync(0xffffffffu, parts, who), w_slot = __shfl_sync(0xffffffffu, slot, who);
    const int w_b = __shfl_sync(0xffffffffu, off, who), w_nb = __shfl_sync(0xffffffffu, n[0], who);
    const int w_v = __shfl_sync(0xffffffffu, off_v, who), w_nv = __shfl_sync(0xffffffffu, n[1], who);
    for (int i = lane; i < w_count; i += 32) {
      const int c = w_parts > 1 ? i / w_parts : i, v = w_parts > 1 ? i % w_parts : 0;
      const int4 rows = w_slot >= 0   ? make_int4(0, 0, w_slot, -1)
                        : w_parts < 0 ? make_int4(0, 0, w_v, w_nv)
                                      : make_int4(0, 0, w_v + v * kEmbValChunk, min(kEmbValChunk, w_nv - v * kEmbValChunk));
      q.items[w_at + i] = make_int4(w_b + c * kEmbChunk, min(kEmbChunk, w_nb - c * kEmbChunk), rows.z, rows.w);
    }
  }
}

__global__ void __launch_bounds__(256) emb_alloc_kernel(const EmbBuckets q) {
  stream_order();
  const int id = blockIdx.x * 256 + threadIdx.x;
  emb_alloc_ids<8>(q, id, id < q.vocab);
}

__device__ __forceinline__ void emb_fill_buckets(const EmbBuckets& q, long long first, long long step) {
  for (long long j = first; j < q.n_tok; j += step) {
    const int r = q.rank[j];
    if (r < 0) continue;
    if (j < q.first_val) q.perm_b[q.off_b[q.ids_b[j]] + r] = static_cast<int>(j);
    else q.perm_v[q.off_v[q.ids_v[j - q.first_val]] + r] = static_cast<int>(j - q.first_val);
  }
}
__global__ void __launch_bounds__(256) emb_fill_kernel(const EmbBuckets q) {
  stream_order();
  emb_fill_buckets(q, blockIdx.x * 256ll + threadIdx.x, gridDim.x * 256ll);
}

// All of it for a small batch in one launch, zeroing included: one cluster with a thread for each token, whose barriers part the
// steps.  Instead of the whole table it looks at the ids that occur: the first token of an id (the first validation token of
// one without train tokens) allocates it, and of the validation counts only those of ids that occur are cleared (the train
// counts all: the gradient's empty rows are found by them).  TOKENS is the largest batch, 4096 or 8192 (emb_one_cluster).
constexpr int kEmbBucketCtas = 8;
template <int TOKENS>
__global__ void __cluster_dims__(kEmbBucketCtas, 1, 1) __launch_bounds__(TOKENS / kEmbBucketCtas)
emb_bucket_kernel(const EmbBuckets q, double* __restrict__ M64, long long m_size) {
  constexpr int kThreads = TOKENS / kEmbBucketCtas;
  stream_order();
  const int j = blockIdx.x * kThreads + threadIdx.x, n_b = static_cast<int>(q.first_val);
  const bool train = j < n_b;
  int id = -1;
  if (j < q.n_tok) {
    const long long x = train ? q.ids_b[j] : q.ids_v[j - n_b];
    if (x >= 0 && x < q.vocab) {
      id = static_cast<int>(x);
      if (q.cnt_v != nullptr) q.cnt_v[id] = 0;
    } else {
      atomicExch(q.err, kErrBadIndex);
    }
  }
  // totals and train counts lie behind each other; with a table of nearly 2^31 rows they are more words than an int counts
  const long long zero = kEmbTotals + static_cast<long long>(q.vocab);
  for (long long i = j; i < zero / 4; i += TOKENS) reinterpret_cast<uint4*>(q.totals)[i] = make_uint4(0u, 0u, 0u, 0u);
  if (j < (zero & 3)) q.totals[(zero & ~3ll) + j] = 0;
  if (M64 != nullptr)
    for (long long i = j; i < m_size; i += TOKENS) M64[i] = 0.;
  cluster_sync_all();
  const int rank = id >= 0 ? atomicAdd((train ? q.cnt_b : q.cnt_v) + id, 1) : -1;
  cluster_sync_all();
  emb_alloc_ids<kThreads / 32>(q, id, rank == 0 && (train || q.cnt_b[id] == 0));
  cluster_sync_all();
  if (id < 0) return;
  if (train) q.perm_b[q.off_b[id] + rank] = j;
  else q.perm_v[q.off_v[id] + rank] = j - n_b;
}

// Tokens of the cluster's kernel that a batch takes, 0: the three kernels behind a cleared table of counts.  The cluster saves
// launches, which bound the host, and looks at no ids that do not occur; it pays by clearing the counts and the sums of the
// matrix from eight SMs, 0.45 TB/s, where the others have the counts cleared at full rate and the sums by a block for
// every 256 tokens.  Bytes of counts and of sums (0: no matrix wanted); three kernels and the cluster, bf16, us:
// * up to 4096 tokens.  Hooks: 8 + 2 x 41 tokens of 320, vocabulary 36761, 38.9 and 31.3; 12 + 4 x 250 of 768, 50304, text ids 51.2
//   and 46.7.  Matrix alone: 34 x 100 of 64, a million ids 24.7 and 24.5, two million 31.3 and 32.8; 2000 + 250 samples of one
//   token, 4 MB of sums, 28.4 and 26.6, 3900 + 130 25.7 and 26.4, 2048 + 2048 64 and 94.  Gradient alone, which saves one launch less
//   and reads the whole table anyway: 34 x 100 of 64, 200000 ids 28.8 and 27.8, 300000 32.3 and 34.0, a million 71.6 and 76.1;
// * up to 8192, with twice the threads: hooks of tables whose gradient is written in less time than the host takes (12 + 4 x 330
//   of 256, 50304: 39.2 and 31.1; 8 + 2 x 512 of 768, the same, 50.7 and 52.4; 16 x 400 of 8, 100000 ids 40.9 and 34.1, 262000 41.1
//   and 41.6).  A result on its own leaves the host time enough (16 x 400 of 8, 100000 ids: matrix 18.7 and 20.4, gradient 24.7
//   and 27.9).
// A thread for two tokens, 16384 of them: 53.9 and 62.
static int emb_one_cluster(long long tokens, double table_bytes, long long counts, long long sums, bool grad) {
  constexpr long long little = 3 << 18;
  if (tokens <= 4096) {
    if (sums == 0) return counts <= little ? 4096 : 0;
    return counts <= 4 << 20 && (tokens <= 2048 || sums <= 2 << 20) ? 4096 : 0;
  }
  return tokens <= 8192 && grad && sums > 0 && table_bytes <= 32e6 && counts + sums <= little ? 8192 : 0;
}

// ---------------------------------------------------------------- dot product: join by id
// R[slot][v] = sum of validation sample v's rows with the hot id of `slot` (float32).  One CTA per (slot,
// sample): the sample's tokens are picked out of the bucket 1024 at a time; a thread adds eight
// features of every groups-th token, four rows in flight, and the groups meet in shared memory.
template <typename T>
__global__ void __launch_bounds__(256)
emb_hot_reduce_kernel(const EmbBuckets q, const T* Gv, long long Tn, int d, int n_val, float* __restrict__ R) {
  stream_order();
  __shared__ int s_tok[1024];
  __shared__ __align__(16) float s_sum[256 * 8];
  __shared__ int s_n;
  const int hot = min(q.totals[4], kEmbHotCap);
  const bool vec = (d % 8 == 0) && ((reinterpret_cast<uintptr_t>(Gv) & 15u) == 0);
  const int per_row = min(256, (d + 7) / 8), groups = 256 / per_row;
  const int grp = threadIdx.x / per_row, fi = threadIdx.x % per_row;
  for (int w = blockIdx.x; w < hot * n_val; w += gridDim.x) {
    const int slot = w / n_val, v = w % n_val;
    const int id = q.hot[slot], cnt = q.cnt_v[id], off = q.off_v[id];
    const long long lo = v * Tn, hi = lo + Tn;
    float* dst = R + static_cast<long long>(w) * d;
    for (int c0 = 0; c0 < cnt; c0 += 1024) {
      __syncthreads();
      if (threadIdx.x == 0) s_n = 0;
      __syncthreads();
      for (int i = c0 + threadIdx.x; i < min(cnt, c0 + 1024); i += 256) {
        const int j = q.perm_v[off + i];
        if (j >= lo && j < hi) s_tok[atomicAdd(&s_n, 1)] = j;
      }
      __syncthreads();
      const int n = s_n;
      for (int f0 = 0; f0 < d; f0 += per_row * 8) {
        const int f = f0 + fi * 8;
        float s[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
        if (grp < groups && f < d) {
#pragma unroll 4
          for (int i = grp; i < n; i += groups) {
            float x[8];
            emb_load_row<T>(Gv, s_tok[i], d, f, vec, x);
#pragma unroll
            for (int e = 0; e < 8; ++e) s[e] += x[e];
          }
        }
        __syncthreads();
#pragma unroll
        for (int e = 0; e < 8; ++e) s_sum[threadIdx.x * 8 + e] = s[e];
        __syncthreads();
        for (int i = threadIdx.x; i < per_row * 8 && f0 + i < d; i += 256) {
          float t = c0 == 0 ? 0.f : dst[f0 + i];
          for (int g = 0; g < groups; ++g) t += s_sum[g * per_row * 8 + i];
          dst[f0 + i] = t;
        }
      }
    }
  }
}

// Eight consecutive contraction elements of one row as bf16x2 words: the values themselves for a bf16 row,
// three parts (8 + 8 + 8 bits of the mantissa) for a float32 row, whose leading six products rebuild the
// float32 product.
template <typename E> struct EmbOct;
template <> struct EmbOct<__nv_bfloat16> {
  static constexpr int kParts = 1;
  uint4 raw;
  uint32_t w[1][4];
  template <bool VEC> __device__ __forceinline__ void load(const __nv_bfloat16* row, int k, int d, bool ok) {
    raw = make_uint4(0u, 0u, 0u, 0u);
    if (!ok) return;
    if (VEC) {
      if (k < d) raw = __ldg(reinterpret_cast<const uint4*>(row + k));
    } else {
      __nv_bfloat16 v[8];
#pragma unroll
      for (int e = 0; e < 8; ++e) v[e] = k + e < d ? row[k + e] : __float2bfloat16_rn(0.f);
      raw = make_uint4(pack_bf16x2(v[0], v[1]), pack_bf16x2(v[2], v[3]), pack_bf16x2(v[4], v[5]), pack_bf16x2(v[6], v[7]));
    }
  }
  __device__ __forceinline__ void split() { w[0][0] = raw.x; w[0][1] = raw.y; w[0][2] = raw.z; w[0][3] = raw.w; }
};
template <> struct EmbOct<float> {
  static constexpr int kParts = 3;
  float v[8];
  uint32_t w[3][4];
  template <bool VEC> __device__ __forceinline__ void load(const float* row, int k, int d, bool ok) {
#pragma unroll
    for (int e = 0; e < 8; ++e) v[e] = 0.f;
    if (!ok) return;
    if (VEC) {
      if (k < d) {
        *reinterpret_cast<float4*>(&v[0]) = __ldg(reinterpret_cast<const float4*>(row + k));
        *reinterpret_cast<float4*>(&v[4]) = __ldg(reinterpret_cast<const float4*>(row + k + 4));
      }
    } else {
#pragma unroll
      for (int e = 0; e < 8; ++e) if (k + e < d) v[e] = __ldg(row + k + e);
    }
  }
  __device__ __forceinline__ void split() {
#pragma unroll
    for (int h = 0; h < 4; ++h) {
      float a = v[2 * h], b = v[2 * h + 1];
#pragma unroll
      for (int p = 0; p < 3; ++p) {
        const __nv_bfloat16 x = __float2bfloat16_rn(a), y = __float2bfloat16_rn(b);
        w[p][h] = pack_bf16x2(x, y);
        a -= __bfloat162float(x);
        b -= __bfloat162float(y);
      }
    }
  }
};

// acc += 16 validation rows x 8 train rows over the whole row length; a lane supplies rows g and g + 8 of
// the first operand, row g of the second, 8 of every 32 columns (the contraction order inside a
// step is permuted alike for both).  The loads of kDepth steps are issued together.
// The tensor core's accumulator truncates, an error that grows with every product added to it, so each
// product starts from zero and the sums are made in float32 registers, in short chains: 1.2e-5 off the
// 64-bit result over 2048 float32 features without that, 3e-8 with it, 6e-8 with multiply-adds on the CUDA
// cores (16 + 8 samples of 512 text tokens; 236 us a hook either way).
template <typename VT, typename BT, bool VEC>
__device__ __forceinline__ void emb_mma_rows(const VT* va, const VT* vb, const BT* tr, bool va_ok, bool vb_ok, bool tr_ok,
                                             int d, int c, float (&acc)[4]) {
  constexpr int kDepth = (sizeof(VT) + 2 * sizeof(BT)) <= 6 ? 4 : 2;
  for (int k0 = c * 8; k0 < (d + 31) / 32 * 32; k0 += 32 * kDepth) {
    EmbOct<VT> a[kDepth], b[kDepth];
    EmbOct<BT> t[kDepth];
#pragma unroll
    for (int s = 0; s < kDepth; ++s) {
      a[s].template load<VEC>(va, k0 + 32 * s, d, va_ok);
      b[s].template load<VEC>(vb, k0 + 32 * s, d, vb_ok);
      t[s].template load<VEC>(tr, k0 + 32 * s, d, tr_ok);
    }
    float group[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
    for (int s = 0; s < kDepth; ++s) {
      a[s].split();
      b[s].split();
      t[s].split();
      float first[4], second[4];
      mma_16816_new(first, a[s].w[0][0], b[s].w[0][0], a[s].w[0][1], b[s].w[0][1], t[s].w[0][0], t[s].w[0][1]);
      mma_16816_new(second, a[s].w[0][2], b[s].w[0][2], a[s].w[0][3], b[s].w[0][3], t[s].w[0][2], t[s].w[0][3]);
#pragma unroll
      for (int e = 0; e < 4; ++e) group[e] += first[e] + second[e];
      if constexpr (EmbOct<VT>::kParts > 1 || EmbOct<BT>::kParts > 1) {
        float low[4] = {0.f, 0.f, 0.f, 0.f};         // everything but the leading parts: 2^-8 of them and less
#pragma unroll
        for (int h = 0; h < 4; h += 2)
#pragma unroll
          for (int p = 0; p < EmbOct<VT>::kParts; ++p)
#pragma unroll
            for (int r = 0; r < EmbOct<BT>::kParts; ++r)
              if (p + r >= 1 && p + r <= 2)
                mma_16816(low, a[s].w[p][h], b[s].w[p][h], a[s].w[p][h + 1], b[s].w[p][h + 1], t[s].w[r][h], t[s].w[r][h + 1]);
#pragma unroll
        for (int e = 0; e < 4; ++e) group[e] += low[e];
      }
    }
#pragma unroll
    for (int e = 0; e < 4; ++e) acc[e] += group[e];
  }
}

// <v, b> of two rows in float32 by one warp
template <typename VT, typename BT>
__device__ __forceinline__ float emb_plain_dot(const VT* v, const BT* b, int d, int lane) {
  float s = 0.f;
  for (int f = lane; f < d; f += 32) s = fmaf(ld_f32<VT>(v + f), ld_f32<BT>(b + f), s);
  return ewarp_sum(s);
}

// The parts of an infinite float32 value are an infinity and NaN, so an entry that is not finite (and ought
// to be infinite, or lies beyond the parts' range) is made again from the rows as they are.  Lane
// (g, c) holds entries (g, 2c), (g, 2c + 1), (g + 8, 2c), (g + 8, 2c + 1); `lv` is its two validation rows.
template <typename VT, typename BT>
__device__ __noinline__ float4 emb_redo(const VT* V, const BT* B, int2 lv, int my_b, unsigned todo, int d, int dk, float4 sums) {
  float acc[4] = {sums.x, sums.y, sums.z, sums.w};
  const int lane = threadIdx.x & 31;
  for (unsigned who_mask = __ballot_sync(0xffffffffu, todo != 0); who_mask != 0; who_mask &= who_mask - 1) {
    const int who = __ffs(who_mask) - 1;
    const unsigned what = __shfl_sync(0xffffffffu, todo, who);
    const int r0 = __shfl_sync(0xffffffffu, lv.x, who), r1 = __shfl_sync(0xffffffffu, lv.y, who);
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      const int b = __shfl_sync(0xffffffffu, my_b, 2 * (who & 3) + (e & 1));
      if (!(what >> e & 1)) continue;
      const float s = emb_plain_dot<VT, BT>(V + static_cast<long long>(e < 2 ? r0 : r1) * d, B + static_cast<long long>(b) * d, dk, lane);
      if (lane == who) acc[e] = s;
    }
  }
  return make_float4(acc[0], acc[1], acc[2], acc[3]);
}

// One join item per warp: up to eight train rows of one id against up to 32 validation rows of it (or, for a
// hot id, one summed row per validation sample), 16 at a time on mma.sync with fragments loaded
// straight from global memory.  Rows come from HBM once; repeats hit L1 / L2.  What bounds it is the
// latency of item -> token lists -> rows, so the kernel keeps registers low, items small (frequent ids
// fall apart into many) and the next item's entry in flight.  Forms before it, for text ids (40 x 1024 tokens
// of 768 bf16 features): a chain walk per train token, 150 us; validation rows in registers and
// products on the CUDA cores, 80 us at eight warps per SM.
// An item's rows arrive over several rounds of loads in a row, 0.7 us each, so a batch with fewer items than warps leaves the
// kernel waiting for the longest: 16 + 4 x 512 text tokens of 2048 float32 features, 32 rounds an item, took 229 us with the
// hook, 168 now (9 + 3 x 333 of 701 67 and 50).  There (CUT) items fall into pieces of a range of features where that shortens
// the rounds that a warp goes through, a piece's indices and sums counted as kEmbJoinAround of them.  Batches
// of more train tokens than four a warp have items enough (at 32 x 1024 the arithmetic alone cost 1.2 us of 99).  With one or two
// validation samples the entries of an item fall on so few scores that their additions wait for each other, and more
// pieces are more additions; bf16 rows that arrive in whole vectors are back before that (5 + 1 x 515 tokens of 768: 66 us in
// pieces, 49 whole; 4 + 2 x 512: 62 and 49; but 36 + 1 x 253 of 1472 float32 45 and 66).
// What it reads (rows, buckets, hot sums) was written before the gradient kernel ahead of it passed its own wait, and so before
// a block of the join came up: read-only for the join's whole life, unlike in the kernels that wait at their start.
constexpr int kEmbJoinAround = 2;
template <typename T, bool VEC, bool CUT>
__global__ void __launch_bounds__(256, 2)
emb_join_kernel(const EmbBuckets q, const T* __restrict__ Gb, const T* __restrict__ Gv, int n_train, int n_val, int Tn, int d,
                const float* __restrict__ R, float scale, double* __restrict__ M64, float* __restrict__ M, long long pitch,
                int local) {
  extern __shared__ float s_M[];         // [n_val, n_train] when `local`
  const int lane = threadIdx.x & 31, g = lane >> 2, c = lane & 3;
  if (local) {
    for (int i = threadIdx.x; i < n_val * n_train; i += 256) s_M[i] = 0.f;
    __syncthreads();
  }
  // Sums over the items of many CTAs: hundreds of float32 additions to one entry cost more accuracy than
  // the products, so they are made in float64 and rounded once.
  auto add = [&](int v, int b, float x) {
    const long long at = static_cast<long long>(v) * n_train + b;
    if (local) atomicAdd(s_M + at, x);
    else atomicAdd(M64 + at, static_cast<double>(x));
  };
  const bool single = n_val == 1 && n_train == 1;
  const int n_items = q.totals[3], stride = gridDim.x * 8;
  int pieces = 1, width = d;
  if (CUT && n_items < 2 * stride && d > 128) {                // every lane weighs one number of pieces (see kEmbJoinAround)
    constexpr int kStep = sizeof(T) == 2 ? 128 : 64;           // features of a round of loads
    const unsigned tried = ((d + lane) / (lane + 1) + 127) / 128 * 128;
    const unsigned rounds = (n_items * ((d + tried - 1) / tried) + stride - 1) / stride;
    const unsigned cost = rounds * (kEmbJoinAround + (tried + kStep - 1) / kStep);
    const unsigned least = __reduce_min_sync(0xffffffffu, cost);
    width = __shfl_sync(0xffffffffu, tried, __ffs(__ballot_sync(0xffffffffu, cost == least)) - 1);
    pieces = (d + width - 1) / width;
  }
  const int n_units = n_items * pieces;
  auto item_of = [&](int u) { return CUT ? u / pieces : u; };
  int unit = blockIdx.x * 8 + (threadIdx.x >> 5);
  int4 item = unit < n_units ? q.items[item_of(unit)] : make_int4(0, 0, 0, 0);
  for (; unit < n_units; unit += stride) {
    const int nb = item.y, at_v = item.z;
    const bool hot = item.w < 0;
    const int cv = hot ? n_val : item.w;
    const int my_b = lane < nb ? q.perm_b[item.x + lane] : 0;
    const int k0 = CUT ? unit % pieces * width : 0, dk = CUT && width < d - k0 ? width : d - k0;
    if (unit + stride < n_units) item = q.items[item_of(unit + stride)];
    const int jb = __shfl_sync(0xffffffffu, my_b, g);
    const bool b_ok = g < nb;
    const int col = my_b / Tn;             // lanes 0..7: train sample of row `lane`
    const int b0 = __shfl_sync(0xffffffffu, col, 2 * c), b1 = __shfl_sync(0xffffffffu, col, 2 * c + 1);
    for (int v0 = 0; v0 < cv; v0 += 16) {
      const int r0 = v0 + g, r1 = v0 + g + 8;
      const bool ok0 = r0 < cv, ok1 = r1 < cv;
      float acc[4] = {0.f, 0.f, 0.f, 0.f};
      int s0 = r0, s1 = r1, j0 = 0, j1 = 0;
      if (hot) {
        const float* base = R + static_cast<long long>(at_v) * n_val * d + k0;
        emb_mma_rows<float, T, VEC>(base + static_cast<long long>(ok0 ? r0 : 0) * d, base + static_cast<long long>(ok1 ? r1 : 0) * d,
                                    Gb + static_cast<long long>(jb) * d + k0, ok0, ok1, b_ok, dk, c, acc);
      } else {
        j0 = ok0 ? q.perm_v[at_v + r0] : 0;
        j1 = ok1 ? q.perm_v[at_v + r1] : 0;
        s0 = j0 / Tn;
        s1 = j1 / Tn;
        emb_mma_rows<T, T, VEC>(Gv + static_cast<long long>(j0) * d + k0, Gv + static_cast<long long>(j1) * d + k0,
                                Gb + static_cast<long long>(jb) * d + k0, ok0, ok1, b_ok, dk, c, acc);
      }
      const bool c0 = 2 * c < nb, c1 = 2 * c + 1 < nb;      // an absent row times an infinite one is no zero
      const unsigned redo = (ok0 && c0 && !isfinite(acc[0]) ? 1u : 0u) | (ok0 && c1 && !isfinite(acc[1]) ? 2u : 0u) |
                            (ok1 && c0 && !isfinite(acc[2]) ? 4u : 0u) | (ok1 && c1 && !isfinite(acc[3]) ? 8u : 0u);
      if (__any_sync(0xffffffffu, redo != 0)) {
        const float4 was = make_float4(acc[0], acc[1], acc[2], acc[3]);
        const float4 is = hot ? emb_redo<float, T>(R + static_cast<long long>(at_v) * n_val * d + k0, Gb + k0, make_int2(s0, s1), my_b,
                                                   redo, d, dk, was)
                              : emb_redo<T, T>(Gv + k0, Gb + k0, make_int2(j0, j1), my_b, redo, d, dk, was);
        acc[0] = is.x; acc[1] = is.y; acc[2] = is.z; acc[3] = is.w;
      }
      if (single) {                        // every entry belongs to the one pair
        float s = ((ok0 && c0 ? acc[0] : 0.f) + (ok0 && c1 ? acc[1] : 0.f)) + ((ok1 && c0 ? acc[2] : 0.f) + (ok1 && c1 ? acc[3] : 0.f));
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
        if (lane == 0) add(0, 0, s);
      } else {
        if (ok0 && c0) add(s0, b0, acc[0]);
        if (ok0 && c1) add(s0, b1, acc[1]);
        if (ok1 && c0) add(s1, b0, acc[2]);
        if (ok1 && c1) add(s1, b1, acc[3]);
      }
    }
  }
  if (local) {
    __syncthreads();
    for (int i = threadIdx.x; i < n_val * n_train; i += 256) {
      const float s = s_M[i];
      if (s != 0.f) atomicAdd(M64 + i, static_cast<double>(s));
    }
    // the last CTA rounds the finished sums
    __shared__ int s_last;
    __threadfence();
    __syncthreads();
    if (threadIdx.x == 0) s_last = atomicAdd(q.totals + 8, 1) == static_cast<int>(gridDim.x) - 1;
    __syncthreads();
    if (s_last) {
      __threadfence();
      for (int i = threadIdx.x; i < n_val * n_train; i += 256)
        M[i / n_train * pitch + i % n_train] = static_cast<float>(__ldcg(M64 + i) * scale);
    }
  }
  // Launched beside the gradient kernel, whose results it does not read; but what follows in the stream
  // waits for this grid only, so it ends no earlier.
  asm volatile("griddepcontrol.wait;" ::: "memory");
}

// The same rounding for a matrix that is too large for one CTA.
__global__ void __launch_bounds__(256) emb_round_kernel(const double* __restrict__ M64, int n_val, int n_train, float scale,
                                                        float* __restrict__ M, long long pitch) {
  const long long size = static_cast<long long>(n_val) * n_train;
  for (long long i = blockIdx.x * 256ll + threadIdx.x; i < size; i += gridDim.x * 256ll)
    M[i / n_train * pitch + i % n_train] = static_cast<float>(M64[i] * scale);
}

// ---------------------------------------------------------------- train gradient
// Both parts below add a row's tokens in ascending order in float32 and round as the reference does.
// Rows that share few tokens (one to kEmbSmallBucket): a warp per listed row and 256 features.  The row's
// tokens are sorted across the warp, loads of kBatch of them are issued before they are added in order.
// Items are handed out kEmbGrab at a time by a counter, the next hand-out fetched while one is worked on:
// static shares left the warps with the rows of 20 to 32 tokens running alone.
constexpr int kEmbGrab = 4;

template <typename T>
__device__ __forceinline__ void emb_small_rows(const EmbBuckets& q, const T* G, int d, float pre_scale,
                                               float divisor, int accumulate, T* __restrict__ out) {
  const int lane = threadIdx.x & 31;
  const bool vec = (d % 8 == 0) && ((reinterpret_cast<uintptr_t>(G) & 15u) == 0) &&
                   ((reinterpret_cast<uintptr_t>(out) & 15u) == 0);
  const int steps = (d + 255) / 256;
  const long long total = static_cast<long long>(q.totals[5]) * steps;
  using Raw = typename EmbRaw<T>::type;
  constexpr int kBatch = sizeof(T) == 2 ? 8 : 4;      // 32 registers of loaded rows for either dtype
  unsigned long long* counter = reinterpret_cast<unsigned long long*>(q.totals + 6);
  auto grab = [&]() -> long long {
    return lane == 0 ? static_cast<long long>(atomicAdd(counter, static_cast<unsigned long long>(kEmbGrab))) : 0;
  };
  long long mine = grab();
  while (true) {
    const long long first = __shfl_sync(0xffffffffu, mine, 0);
    if (first >= total) return;
    mine = grab();
    // (row, step) of the first item by one division, of the others by counting on
    int row = total <= INT_MAX ? static_cast<int>(static_cast<unsigned>(first) / static_cast<unsigned>(steps))
                               : static_cast<int>(first / steps);
    int step = static_cast<int>(first - static_cast<long long>(row) * steps);
    int items = static_cast<int>(first + kEmbGrab < total ? kEmbGrab : total - first);
    int4 entry = q.small[row];
    for (; items > 0; --items) {
      const int k = entry.x, off = entry.y, n = entry.z;
      const int f = step * 256 + lane * 8;
      int tok = lane < n ? q.perm_b[off + lane] : INT_MAX;
      if (++step == steps) {
        step = 0;
        if (++row < q.totals[5]) entry = q.small[row];
      }
      // bitonic sort of the first n keys, ascending
#pragma unroll
      for (int size = 2; size <= 32; size <<= 1) {
        if (size >= 2 * n) break;
#pragma unroll
        for (int stride = size >> 1; stride > 0; stride >>= 1) {
          const int other = __shfl_xor_sync(0xffffffffu, tok, stride);
          const bool up = ((lane & size) == 0), lower = ((lane & stride) == 0);
          tok = (lower == up) ? min(tok, other) : max(tok, other);
        }
      }
      float acc[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
      if (vec) {
        for (int i0 = 0; i0 < n; i0 += kBatch) {
          Raw x[kBatch];
#pragma unroll
          for (int r = 0; r < kBatch; ++r) {
            if (i0 + r >= n) break;
            const int j = __shfl_sync(0xffffffffu, tok, i0 + r);
            x[r] = f < d ? EmbRaw<T>::load(G + static_cast<long long>(j) * d + f) : EmbRaw<T>::zero();
          }
#pragma unroll
          for (int r = 0; r < kBatch; ++r) {
            if (i0 + r >= n) break;
            float xf[8];
            EmbRaw<T>::unpack(x[r], xf);
            emb_accumulate<T>(xf, pre_scale, acc);
          }
        }
      } else {
        for (int i = 0; i < n; ++i) {
          float x[8];
          emb_load_row<T>(G, __shfl_sync(0xffffffffu, tok, i), d, f, false, x);
          emb_accumulate<T>(x, pre_scale, acc);
        }
      }
      emb_store_row<T>(out, k, d, f, vec, acc, divisor, accumulate);
    }
  }
}

// Rows that many tokens share (padding, separators, frequent words).  A CTA takes 256 bytes of one row's
// features (128 bf16, 64 float32).  Ascending order comes from a bit map instead of a sort: the row's
// tokens set bits of a window of 32768 tokens in shared memory, and prefix sums of the words' bit counts
// turn the map into an ordered list.  The sum is sequential per feature (float addition in the CPU's
// order), so its bound is the issue rate of one warp, eight instructions a token; a three-slot ring of
// 32-row stages filled with cp.async keeps the rows arriving at that pace.
constexpr int kEmbGradThreads = 128;
constexpr int kBigWindow = 32768;        // tokens of a bit map: 1024 words, eight per thread
constexpr int kBigList = 2048;           // list entries held at a time
constexpr int kBigStage = 32, kBigSlots = 3;

template <typename T>
__device__ __forceinline__ void emb_big_rows(const EmbBuckets& q, const T* G, int d, int slices, float pre_scale,
                                             float divisor, int accumulate, T* __restrict__ out) {
  constexpr int kFeat = 256 / static_cast<int>(sizeof(T));
  constexpr int kPer = 16 / static_cast<int>(sizeof(T));       // features of a 16-byte piece
  __shared__ unsigned s_map[kBigWindow / 32];
  __shared__ unsigned short s_list[kBigList];
  __shared__ int s_warp[kEmbGradThreads / 32];
  extern __shared__ __align__(16) unsigned char s_dyn[];
  T (*s_ring)[kBigStage][kFeat] = reinterpret_cast<T (*)[kBigStage][kFeat]>(s_dyn);
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int total = q.totals[2];
  const bool vec = (d % 8 == 0) && ((reinterpret_cast<uintptr_t>(G) & 15u) == 0);
  const long long n_train_tok = q.first_val;
  for (long long w = blockIdx.x; w < static_cast<long long>(total) * slices; w += gridDim.x) {
    const int k = q.big[w / slices];
    const int f0 = static_cast<int>(w % slices) * kFeat;
    const int cnt = q.cnt_b[k], off = q.off_b[k];
    const int f = f0 + tid;
    const bool mine = tid < kFeat && f < d;
    float acc = 0.f;
    for (long long win = 0; win < n_train_tok; win += kBigWindow) {
      __syncthreads();
      for (int i = tid; i < kBigWindow / 32; i += kEmbGradThreads) s_map[i] = 0u;
      __syncthreads();
#pragma unroll 4
      for (int i = tid; i < cnt; i += kEmbGradThreads) {
        const long long j = q.perm_b[off + i] - win;
        if (j >= 0 && j < kBigWindow) atomicOr(&s_map[j >> 5], 1u << (j & 31));
      }
      __syncthreads();
      unsigned m[8];
      int own = 0;
#pragma unroll
      for (int e = 0; e < 8; ++e) { m[e] = s_map[tid * 8 + e]; own += __popc(m[e]); }
      int x = own;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const int y = __shfl_up_sync(0xffffffffu, x, o);
        if (lane >= o) x += y;
      }
      if (lane == 31) s_warp[warp] = x;
      __syncthreads();
      int first = x - own, in_window = 0;
#pragma unroll
      for (int v = 0; v < kEmbGradThreads / 32; ++v) {
        if (v < warp) first += s_warp[v];
        in_window += s_warp[v];
      }
      for (int lo = 0; lo < in_window; lo += kBigList) {       // entries [lo, lo + kBigList) of the ordered list
        const int n = min(kBigList, in_window - lo);
        __syncthreads();
        if (first < lo + n && first + own > lo) {
          int at = first - lo;
#pragma unroll
          for (int e = 0; e < 8; ++e) {
            unsigned bits = m[e];
            while (bits) {
              const int bit = __ffs(bits) - 1;
              bits &= bits - 1;
              if (at >= 0 && at < n) s_list[at] = static_cast<unsigned short>((tid * 8 + e) * 32 + bit);
              ++at;
            }
          }
        }
        __syncthreads();
        if (vec) {
          const int n_stages = (n + kBigStage - 1) / kBigStage;
          auto issue = [&](int st) {
            if (st < n_stages) {
#pragma unroll
              for (int e = 0; e < kBigStage * 16 / kEmbGradThreads; ++e) {
                const int c = e * kEmbGradThreads + tid, r = c >> 4, piece = (c & 15) * kPer;
                const int i = st * kBigStage + r;
                if (i < n && f0 + piece < d) {
                  const T* src = G + (win + s_list[i]) * d + f0 + piece;
                  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(static_cast<uint32_t>(
                                   __cvta_generic_to_shared(&s_ring[st % kBigSlots][r][piece]))), "l"(src) : "memory");
                }
              }
            }
            asm volatile("cp.async.commit_group;" ::: "memory");
          };
          for (int st = 0; st < kBigSlots - 1; ++st) issue(st);
          for (int st = 0; st < n_stages; ++st) {
            asm volatile("cp.async.wait_group %0;" ::"n"(kBigSlots - 2) : "memory");
            __syncthreads();              // stage `st` has arrived; slot of stage st - 1 is free
            issue(st + kBigSlots - 1);
            if (mine) {
              const int rows = min(kBigStage, n - st * kBigStage);
              if (rows == kBigStage) {
#pragma unroll 8
                for (int r = 0; r < kBigStage; ++r)
                  acc = __fadd_rn(acc, round_to<T>(__fmul_rn(ld_f32<T>(&s_ring[st % kBigSlots][r][tid]), pre_scale)));
              } else {
                for (int r = 0; r < rows; ++r)
                  acc = __fadd_rn(acc, round_to<T>(__fmul_rn(ld_f32<T>(&s_ring[st % kBigSlots][r][tid]), pre_scale)));
              }
            }
          }
          asm volatile("cp.async.wait_all;" ::: "memory");
        } else if (mine) {
#pragma unroll 4
          for (int i = 0; i < n; ++i)
            acc = __fadd_rn(acc, round_to<T>(__fmul_rn(ld_f32<T>(G + (win + s_list[i]) * d + f), pre_scale)));
        }
      }
    }
    if (mine) {
      T* dst = out + static_cast<long long>(k) * d + f;
      float o = round_to<T>(__fdiv_rn(round_to<T>(acc), divisor));
      if (accumulate) o = round_to<T>(__fadd_rn(ld_f32<T>(dst), o));
      *dst = from_f32<T>(o);
    }
  }
}

// Zeroes the gradient's rows without tokens, `each` (up to 32) ids a warp drawn from a counter.  It runs behind the sums, on the warps
// that find no more of them: the longest row's sum leaves HBM idle for 30 us, and the counting kernel, which zeroed all
// rows ahead of everything else, took 13 us for it on a table of 50304 x 768 bf16.  A draw is at most kEmbZeroBytes of rows: 32 wide
// rows of a small table leave most warps without a draw (3 + 7 x 22 text tokens, table of 18455 x 1664 bf16: a hook of 55 us, 39 with
// four; 9 + 4 x 112 positions, 4096 x 1280 float32: 73 and 40).
constexpr int kEmbZeroBytes = 24 * 1024;
template <typename T>
__device__ void emb_zero_rows(const EmbBuckets& q, int d, int each, T* __restrict__ out) {
  const int lane = threadIdx.x & 31;
  const int pieces = static_cast<int>(d * sizeof(T) / 16);
  const uint4 z = make_uint4(0u, 0u, 0u, 0u);
  while (true) {
    int first = 0;
    if (lane == 0) first = atomicAdd(q.totals + 9, each);
    first = __shfl_sync(0xffffffffu, first, 0);
    if (first >= q.vocab) break;
    const bool empty = lane < each && first + lane < q.vocab && q.cnt_b[first + lane] == 0;
    for (unsigned todo = __ballot_sync(0xffffffffu, empty); todo != 0; todo &= todo - 1) {
      uint4* row = reinterpret_cast<uint4*>(out + static_cast<long long>(first + __ffs(todo) - 1) * d);
      for (int i = lane; i < pieces; i += 32) row[i] = z;
    }
  }
}

// One launch for both: every CTA takes its share of the long rows, whose chains are the longest, and goes on
// with the short ones.  Apart, a launch of each (text ids, 40 x 1024 tokens of 768 bf16 features) took 46 and
// 35 us, mostly with a few warps left per SM; 39 us together, 30 of them the longest rows' chains.
// What bounds it is issue slots and latency, not bandwidth, and the same holds for the join, which is launched beside
// this grid's tail (a programmatic launch: it reads nothing written here); one after the other they took a fifth longer.
template <typename T>
__global__ void __launch_bounds__(kEmbGradThreads, 6)
emb_grad_kernel(const EmbBuckets q, const T* G, int d, int slices, float pre_scale, float divisor,
                int accumulate, int zero_each, T* __restrict__ out) {
  stream_order();                        // from here on the join may start beside this grid's tail
  emb_big_rows<T>(q, G, d, slices, pre_scale, divisor, accumulate, out);
  emb_small_rows<T>(q, G, d, pre_scale, divisor, accumulate, out);
  if (zero_each) emb_zero_rows<T>(q, d, zero_each, out);
}

static inline long long up256(long long x) { return (x + 255) / 256 * 256; }

}  // namespace gb

using namespace gb;

// head [vocab] + next [n_val * T]: the least a caller of ghost_embedding_dot must provide (chain kernels).
extern "C" long long ghost_embedding_dot_workspace_bytes(int n_val, long long T, int vocab) {
  return up256(4ll * vocab) + up256(4ll * n_val * T);
}

// Every id with tokens on both sides splits into train chunks times at most kEmbMaxParts validation parts.
constexpr int kEmbMaxParts = 2;
static long long emb_max_items(long long tb, int vocab) {
  return kEmbMaxParts * (tb / kEmbChunk + (tb < vocab ? tb : vocab) + 1);
}

extern "C" long long ghost_embedding_pass_workspace_bytes(int n_train, int n_val, long long T, int vocab, int d) {
  const long long tb = static_cast<long long>(n_train) * T, tv = static_cast<long long>(n_val) * T;
  return up256(4ll * (2 * static_cast<long long>(vocab) + kEmbTotals)) + 2 * up256(4ll * vocab)     // counts and totals; offsets
         + up256(8ll * n_train * n_val)                                                    // sums of the matrix
         + up256(4ll * (tb + tv)) + up256(4ll * tb) + up256(4ll * tv)                      // rank, perm_b, perm_v
         + up256(4ll * (tb / (kEmbSmallBucket + 1) + 2)) + up256(16ll * emb_max_items(tb, vocab))   // big rows, items
         + up256(4ll * kEmbHotCap) + up256(16ll * (vocab < tb ? vocab : tb)) + up256(4ll * kEmbHotCap * static_cast<long long>(n_val) * d);
}
extern "C" long long ghost_embedding_wgrad_workspace_bytes(int n_train, long long T, int vocab) {
  return ghost_embedding_pass_workspace_bytes(n_train, 0, T, vocab, 0);
}

namespace gb {

template <typename T>
static int emb_pass(const EmbBuckets& q, const T* Gb, const T* Gv, int n_train, int n_val, long long Tn, int d, float scale,
                    float* M, long long pitch, double* M64, float* R, float pre_scale, float divisor, int accumulate, T* out, const DeviceState* ds, cudaStream_t st) {
  int blocks = static_cast<int>((q.n_tok + 255) / 256);
  if (blocks > ds->sm_count * 8) blocks = ds->sm_count * 8;
  // Rows without tokens are zeroed behind the sums where 16-byte stores can, by the counting kernel where the table as a
  // whole takes them (rows of odd widths), or by a memset.
  const long long out_bytes = static_cast<long long>(q.vocab) * d * static_cast<long long>(sizeof(T));
  const bool fill = out != nullptr && !accumulate, aligned = (reinterpret_cast<uintptr_t>(out) & 15u) == 0;
  const bool by_rows = fill && aligned && d * sizeof(T) % 16 == 0 && q.vocab < INT_MAX - (1 << 24);
  const bool quick = fill && !by_rows && aligned && out_bytes % 16 == 0;
  if (fill && !by_rows && !quick) GB_CUDA_OK(cudaMemsetAsync(out, 0, out_bytes, st));
  const int tokens = blocks;
  if (quick) blocks = ds->sm_count * 8;
  const int one = quick ? 0 : emb_one_cluster(q.n_tok, static_cast<double>(out_bytes), 4 * (kEmbTotals + static_cast<long long>(q.vocab)),
                                              M64 != nullptr ? 8ll * n_val * n_train : 0, out != nullptr);
  if (one > 0) {
    GB_CUDA_OK(launch_next(one == 4096 ? emb_bucket_kernel<4096> : emb_bucket_kernel<8192>, dim3(kEmbBucketCtas), dim3(one / kEmbBucketCtas), 0, st,
                           q, M64, static_cast<long long>(n_val) * n_train));
    count_launch();
  } else {
    if (int rc = clear_ahead(q.totals, 4 * (kEmbTotals + static_cast<size_t>(q.vocab) * (M != nullptr ? 2 : 1)), st)) return rc;
    GB_CUDA_OK(launch_next(emb_count_kernel, dim3(blocks), dim3(256), 0, st, q, M64, static_cast<long long>(n_val) * n_train,
                           reinterpret_cast<uint4*>(out), quick ? out_bytes / 16 : 0ll));
    GB_CUDA_OK(launch_next(emb_alloc_kernel, dim3(ceil_div(q.vocab, 256)), dim3(256), 0, st, q));
    GB_CUDA_OK(launch_next(emb_fill_kernel, dim3(tokens), dim3(256), 0, st, q));
    count_launch(3);
  }
  const bool vec = d % 8 == 0 && ((reinterpret_cast<uintptr_t>(Gb) | reinterpret_cast<uintptr_t>(Gv)) & 15u) == 0;
  if (M != nullptr) {
    if (static_cast<long long>(n_val) * Tn > q.hot_threshold) {
      int hb = kEmbHotCap * n_val;
      if (hb > ds->sm_count * 8) hb = ds->sm_count * 8;
      GB_CUDA_OK(launch_next(emb_hot_reduce_kernel<T>, dim3(hb), dim3(256), 0, st, q, Gv, Tn, d, n_val, R));
      count_launch();
    }
  }
  if (out != nullptr) {
    // every row with tokens is a long row's slices or a short row's steps: at least one item per warp
    const long long rows = q.vocab < q.first_val ? q.vocab : q.first_val;      // at most one row per token
    const int slices = ceil_div(d, 256 / static_cast<int>(sizeof(T)));
    const long long most = rows * slices;
    int gb = static_cast<int>(most < ds->sm_count * 6 ? most : ds->sm_count * 6);
    if (by_rows) {                       // warps enough for the empty rows too
      const int zb = ceil_div(q.vocab, kEmbGradThreads), all = ds->sm_count * 6;
      if (gb < zb) gb = zb < all ? zb : all;
    }
    int zero_each = 32;
    while (zero_each > 4 && zero_each * d * sizeof(T) > kEmbZeroBytes) zero_each /= 2;
    constexpr int kBigRing = kBigSlots * kBigStage * 256;
    GB_CUDA_OK(launch_next(emb_grad_kernel<T>, dim3(gb), dim3(kEmbGradThreads), kBigRing, st, q, Gb, d, slices, pre_scale, divisor,
                           accumulate, by_rows ? zero_each : 0, out));
    count_launch();
  }
  if (M != nullptr) {
    // a matrix of up to 16 KB is summed up in shared memory first: few, hot addresses otherwise
    const int local = static_cast<long long>(n_val) * n_train <= 4096 ? 1 : 0;
    const size_t smem = local ? sizeof(float) * n_val * n_train : 0;
    const int Ti = static_cast<int>(Tn);
    const long long most = (q.max_items + 7) / 8;
    const int jb = static_cast<int>(most < ds->sm_count * 2 ? most : ds->sm_count * 2);
    const bool cut = q.first_val <= 4ll * 8 * jb && !(n_val <= 2 && sizeof(T) == 2 && vec);
    const auto join = cut ? vec ? emb_join_kernel<T, true, true> : emb_join_kernel<T, false, true>
                          : vec ? emb_join_kernel<T, true, false> : emb_join_kernel<T, false, false>;
    cudaLaunchAttribute beside = {};
    beside.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    beside.val.programmaticStreamSerializationAllowed = 1;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(jb);
    cfg.blockDim = dim3(256);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = st;
    cfg.attrs = &beside;
    cfg.numAttrs = out != nullptr ? 1 : 0;
    GB_CUDA_OK(cudaLaunchKernelEx(&cfg, join, q, Gb, Gv, n_train, n_val, Ti,
                                  d, static_cast<const float*>(R), scale, M64, M, pitch, local));
    count_launch();
    if (!local) {
      const int rb = ceil_div(static_cast<long long>(n_val) * n_train, 256);
      emb_round_kernel<<<rb < ds->sm_count * 8 ? rb : ds->sm_count * 8, 256, 0, st>>>(M64, n_val, n_train, scale, M, pitch);
      count_launch();
    }
  }
  return post_launch("ghost_embedding_pass");
}

}  // namespace gb

namespace gb {

// Train samples [b0, b0 + n_b) against all validation samples (M non-null), and their gradient (out non-null)
static int emb_pass_group(const long long* ids, const void* G, int is_f32, int n_train, int b0, int n_b, int n_val,
                          long long T, int d, int vocab, float scale, float* M, float pre_scale, float divisor,
                          int accumulate, void* out, void* ws, const DeviceState* ds, cudaStream_t st) {
  const long long tb = static_cast<long long>(n_b) * T, tv = static_cast<long long>(n_val) * T;
  uint8_t* at = static_cast<uint8_t*>(ws);
  auto take = [&](long long bytes) { void* p = at; at += up256(bytes); return p; };
  EmbBuckets q = {};
  q.ids_b = ids + b0 * T;
  q.ids_v = ids + n_train * T;
  q.first_val = tb;
  q.n_tok = tb + tv;
  q.vocab = vocab;
  q.totals = static_cast<int*>(take(4ll * (2 * static_cast<long long>(vocab) + kEmbTotals)));
  q.cnt_b = q.totals + kEmbTotals;
  q.cnt_v = M ? q.cnt_b + vocab : nullptr;
  q.off_b = static_cast<int*>(take(4ll * vocab));
  q.off_v = static_cast<int*>(take(4ll * vocab));
  q.rank = static_cast<int*>(take(4ll * (tb + tv)));
  q.perm_b = static_cast<int*>(take(4ll * tb));
  q.perm_v = static_cast<int*>(take(4ll * tv));
  q.big = static_cast<int*>(take(4ll * (tb / (kEmbSmallBucket + 1) + 2)));
  q.max_items = emb_max_items(tb, vocab);
  q.items = static_cast<int4*>(take(16ll * q.max_items));
  q.hot = static_cast<int*>(take(4ll * kEmbHotCap));
  q.small = static_cast<int4*>(take(16ll * (vocab < tb ? vocab : tb)));
  double* M64 = static_cast<double*>(take(M ? 8ll * n_b * n_val : 0));
  float* R = static_cast<float*>(take(4ll * kEmbHotCap * static_cast<long long>(n_val) * (M ? d : 0)));
  // A hot id costs n_val dot products per train token instead of one per validation token, after a pass over
  // its validation rows; the products are cheap, so that pass pays from a few join items' worth on.
  q.hot_threshold = 2 * n_val > kEmbMaxParts * kEmbValChunk ? 2 * n_val : kEmbMaxParts * kEmbValChunk;
  q.max_parts = kEmbMaxParts;
  q.want_rows = out != nullptr;
  q.err = ds->err_word;
  float* Mg = M ? M + b0 : nullptr;
  if (is_f32) {
    const float* g = static_cast<const float*>(G);
    return emb_pass<float>(q, g + b0 * T * d, g + n_train * T * d, n_b, n_val, T, d, scale, Mg, n_train, M ? M64 : nullptr, R,
                           pre_scale, divisor, accumulate, static_cast<float*>(out), ds, st);
  }
  const __nv_bfloat16* g = static_cast<const __nv_bfloat16*>(G);
  return emb_pass<__nv_bfloat16>(q, g + b0 * T * d, g + n_train * T * d, n_b, n_val, T, d, scale, Mg, n_train, M ? M64 : nullptr, R,
                                 pre_scale, divisor, accumulate, static_cast<__nv_bfloat16*>(out), ds, st);
}

}  // namespace gb

extern "C" int ghost_embedding_pass(const long long* ids, const void* G, int is_f32, int n_train, int n_val, long long T,
                                    int d, int vocab, float scale, float* M_out, float pre_scale, float divisor,
                                    int accumulate, void* grad_out, void* ws, long long ws_bytes, void* stream) {
  const DeviceState* ds = device_state();
  if (!ds) return GHOST_ERR_DEVICE;
  GB_REQUIRE(ids && G && ws && (M_out || grad_out), "ghost_embedding_pass: null pointer");
  GB_REQUIRE(n_train > 0, "No training samples to compute dot product, check batch sizes.");
  GB_REQUIRE(T > 0 && d > 0 && vocab > 0 && (n_val > 0 || M_out == nullptr), "ghost_embedding_pass: bad dimensions");
  if (M_out == nullptr) n_val = 0;
  GB_REQUIRE((static_cast<long long>(n_train) + n_val) * T < INT_MAX, "ghost_embedding_pass: too many tokens");
  GB_REQUIRE(n_val <= 8192, "ghost_embedding_pass: at most 8192 validation samples");
  GB_REQUIRE(grad_out == nullptr || divisor != 0.f, "ghost_embedding_pass: divisor must be non-zero");
  GB_REQUIRE(ws_bytes >= ghost_embedding_pass_workspace_bytes(n_train, n_val, T, vocab, M_out ? d : 0),
             "ghost_embedding_pass: workspace too small");
  return emb_pass_group(ids, G, is_f32, n_train, 0, n_train, n_val, T, d, vocab, scale, M_out, pre_scale, divisor, accumulate,
                        grad_out, ws, ds, static_cast<cudaStream_t>(stream));
}

// Room for the join with the train samples in groups of at least 32 (all of them at once in most batches)
static int emb_dot_group(int n_val) { return n_val > 32 ? n_val : 32; }
extern "C" long long ghost_embedding_dot_workspace_bytes_for(int n_val, long long T, int vocab, int d) {
  return ghost_embedding_pass_workspace_bytes(emb_dot_group(n_val), n_val, T, vocab, d);
}

extern "C" int ghost_embedding_wgrad(const long long* ids, const void* G, int is_f32, int n_train, long long T,
                                     int d, int vocab, float pre_scale, float divisor, int accumulate,
                                     void* out, void* ws, long long ws_bytes, void* stream) {
  GB_REQUIRE(ids && G && out && ws, "ghost_embedding_wgrad: null pointer");
  return ghost_embedding_pass(ids, G, is_f32, n_train, 0, T, d, vocab, 1.f, nullptr, pre_scale, divisor, accumulate, out, ws,
                              ws_bytes, stream);
}

extern "C" int ghost_embedding_dot(const long long* ids, const void* G, int is_f32, int n_train, int n_val,
                                   long long T, int d, int vocab, float scale, float* M_out, void* ws,
                                   long long ws_bytes, void* stream) {
  const DeviceState* ds = device_state();
  if (!ds) return GHOST_ERR_DEVICE;
  GB_REQUIRE(ids && G && M_out && ws, "ghost_embedding_dot: null pointer");
  GB_REQUIRE(n_train > 0, "No training samples to compute dot product, check batch sizes.");
  GB_REQUIRE(n_val > 0 && T > 0 && d > 0 && vocab > 0, "ghost_embedding_dot: bad dimensions");
  GB_REQUIRE(static_cast<long long>(n_val) * T < INT_MAX && n_train <= 65535, "ghost_embedding_dot: too many tokens");
  GB_REQUIRE(n_val <= 8192, "ghost_embedding_dot: at most 8192 validation samples");
  GB_REQUIRE(ws_bytes >= ghost_embedding_dot_workspace_bytes(n_val, T, vocab), "ghost_embedding_dot: workspace too small");
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  // as many train samples at a time as the workspace has room for, in groups of 32 and more
  int group = n_train;
  auto fits = [&](int g) {
    return (static_cast<long long>(g) + n_val) * T < INT_MAX && ws_bytes >= ghost_embedding_pass_workspace_bytes(g, n_val, T, vocab, d);
  };
  while (group > emb_dot_group(n_val) && !fits(group)) group = (group + 1) / 2 > emb_dot_group(n_val) ? (group + 1) / 2 : emb_dot_group(n_val);
  if (fits(group)) {
    for (int b0 = 0; b0 < n_train; b0 += group) {
      const int rc = emb_pass_group(ids, G, is_f32, n_train, b0, n_train - b0 < group ? n_train - b0 : group, n_val, T, d, vocab,
                                    scale, M_out, 1.f, 1.f, 0, nullptr, ws, ds, st);
      if (rc != GHOST_OK) return rc;
    }
    return GHOST_OK;
  }
  int* head = static_cast<int*>(ws);
  int* next = reinterpret_cast<int*>(static_cast<uint8_t*>(ws) + up256(4ll * vocab));
  const long long n_vtok = static_cast<long long>(n_val) * T;
  GB_CUDA_OK(cudaMemsetAsync(head, 0xFF, 4ull * vocab, st));
  GB_CUDA_OK(cudaMemsetAsync(M_out, 0, sizeof(float) * static_cast<size_t>(n_val) * n_train, st));
  int blocks = static_cast<int>((n_vtok + 255) / 256);
  if (blocks > ds->sm_count * 8) blocks = ds->sm_count * 8;
  emb_chain_val_kernel<<<blocks, 256, 0, st>>>(ids + static_cast<long long>(n_train) * T, n_vtok, vocab, head, next, ds->err_word);
  const int tok_per_block = 64;
  dim3 grid(ceil_div(T, tok_per_block), n_train);
  const size_t smem = sizeof(float) * n_val;
  if (is_f32)
    emb_chain_dot_kernel<float><<<grid, 256, smem, st>>>(ids, static_cast<const float*>(G), n_train, n_val, T, d, vocab, head, next, scale, M_out, tok_per_block, ds->err_word);
  else
    emb_chain_dot_kernel<__nv_bfloat16><<<grid, 256, smem, st>>>(ids, static_cast<const __nv_bfloat16*>(G), n_train, n_val, T, d, vocab, head, next, scale, M_out, tok_per_block, ds->err_word);
  count_launch(2);
  return post_launch("emb_chain_dot_kernel");
}

// ------------------------------------------------------------------------------------------------
// Allocation-free variant of ghost_embedding_dot.
//
// Who needs it: callers that are not allowed to obtain device memory when the hook fires.  Two real
// cases: a process whose device memory is owned up front by a fixed-size pool (an inference or
// data-valuation service with a hard memory budget, where a late cudaMalloc can fail or stall every
// stream while the driver synchronises), and code that runs inside another component's critical
// section (an allocator callback, a communication progress thread) where calling back into any
// allocator, torch's included, would deadlock.  Such callers can still hand over their inputs and
// the output matrix, but they have nowhere to get the id-chain tables from.
//
// The tables therefore live in the library image itself: one file-scope __device__ array per GPU
// that loads the library (kEmbStaticBytes, held until the process exits).  Limits follow from its
// size: vocab <= 131072 and n_val * T <= 131072.  Larger problems are rejected; use
// ghost_embedding_dot with a caller-provided workspace for those.
//
// The array's name is a host-side handle, not a device address, so the device address is looked up
// with cudaGetSymbolAddress the first time the entry point runs on a device (with that device
// current) and cached.  That first call should happen before any stream capture begins.  The
// tables keep whatever the previous call left: every call re-initialises the head table and
// rewrites the whole next-table range it uses before reading it.  All calls on one GPU share the
// one array, so two calls whose kernels can overlap (different streams, no ordering) race; keep
// calls to this entry point on one stream or order them with events.
// ------------------------------------------------------------------------------------------------
namespace gb {
constexpr int kEmbStaticMaxVocab = 131072;
constexpr long long kEmbStaticMaxValTokens = 131072;
constexpr long long kEmbStaticBytes = 4ll * kEmbStaticMaxVocab + 4ll * kEmbStaticMaxValTokens;   // 1 MiB
static __device__ __align__(256) unsigned char g_emb_static_scratch[kEmbStaticBytes];

static int emb_static_scratch(void** out) {
  static std::mutex mu;
  static void* ptrs[64] = {};
  int dev = -1;
  GB_CUDA_OK(cudaGetDevice(&dev));
  if (dev < 0 || dev >= 64) return fail(GHOST_ERR_INVALID, "unsupported device ordinal %d", dev);
  std::lock_guard<std::mutex> lock(mu);
  if (!ptrs[dev]) {
    void* p = nullptr;
    // set-up, once per device, with that device current
    GB_CUDA_OK(cudaGetSymbolAddress(&p, g_emb_static_scratch));
    ptrs[dev] = p;
  }
  *out = ptrs[dev];
  return GHOST_OK;
}
}  // namespace gb

extern "C" int ghost_embedding_dot_noalloc(const long long* ids, const void* G, int is_f32, int n_train,
                                           int n_val, long long T, int d, int vocab, float scale,
                                           float* M_out, void* stream) {
  if (!device_state()) return GHOST_ERR_DEVICE;
  GB_REQUIRE(vocab > 0 && vocab <= kEmbStaticMaxVocab,
             "ghost_embedding_dot_noalloc: vocab %d exceeds the built-in scratch (max %d); use "
             "ghost_embedding_dot with a caller workspace", vocab, kEmbStaticMaxVocab);
  GB_REQUIRE(n_val > 0 && T > 0 && static_cast<long long>(n_val) * T <= kEmbStaticMaxValTokens,
             "ghost_embedding_dot_noalloc: n_val * T = %lld exceeds the built-in scratch (max %lld); use "
             "ghost_embedding_dot with a caller workspace", static_cast<long long>(n_val) * T,
             kEmbStaticMaxValTokens);
  void* scratch = nullptr;
  int rc = emb_static_scratch(&scratch);
  if (rc != GHOST_OK) return rc;
  // same kernels as ghost_embedding_dot; the head table is cleared and the used part of the next
  // table rewritten on every call, so stale contents of the shared array are never read
  return ghost_embedding_dot(ids, G, is_f32, n_train, n_val, T, d, vocab, scale, M_out, scratch,
                             kEmbStaticBytes, stream);
}
