// Linear / Conv1D layers with few token rows: dot-product matrix, train gradient and per-sample column
// sums in ONE launch, float32 arithmetic on the CUDA cores straight from the operands.
//
// The tensor-core paths need bf16 operands (two to six conversion launches for float32 layers), zeroed
// outputs, a GEMM whose grid is a handful of tiles, and a scaling pass: eight to twelve launches whose
// fixed costs are ten times the arithmetic when a layer has tens of rows.  Here the blocks of one grid
// share out the three results; nothing is converted, zeroed or written twice.  Layer 1024 -> 1024,
// 64 + 16 samples of one token, float32: 11 launches, 93 us of GPU time before, one of 7 us now.
#include "common.cuh"
#include "launch_rules.h"
#include "sm100_ptx.cuh"

namespace gb {

struct SmallDense {
  const void *A, *B;                    // [N, T, d], [N, T, p]
  int n_train, n_val, T, d, p;
  int in_by_out;                        // weight [d, p] instead of [p, d]
  float* M;                             // [n_val, n_train]
  void* grad;                           // null: not wanted
  int grad_f32;
  float grad_scale;
  float* colsums;                       // [N, p]; null: not wanted
  // blocks [0, gram_blocks): pairs of sample groups, a cluster of `ranks` to each in the SPLIT form; then wgrad_blocks tiles of
  // 64 x 64; then column sums
  int sv, sb, groups_b, gram_blocks;    // samples of a group (validation, train)
  int tiles_n, wgrad_blocks;
  int ranks;
};

// Four consecutive elements as they are loaded, and as numbers.  Two steps, so that the loads of several rows are in flight
// together: with the conversion behind each load's bounds check a step of 1024 bf16 columns took 4.4 us, 1.1 so
// (4 + 12 samples of one token, 108 -> 27072: 123 and 33 us, 109 -> 27072 160 and 35; 4 + 4 x 16 of 64 -> 64 32.8 and 22).
template <typename E, bool VEC> struct SdQuad;
template <bool VEC> struct SdQuad<float, VEC> {
  float4 raw;
  // zero beyond `left`; VEC: row starts are aligned and `left` is a multiple of four
  __device__ __forceinline__ void load(const float* p, int left) {
    if constexpr (VEC) {
      raw = make_float4(0.f, 0.f, 0.f, 0.f);
      if (left > 0) raw = *reinterpret_cast<const float4*>(p);
    } else {
      raw = make_float4(left > 0 ? p[0] : 0.f, left > 1 ? p[1] : 0.f, left > 2 ? p[2] : 0.f, left > 3 ? p[3] : 0.f);
    }
  }
  __device__ __forceinline__ float4 value() const { return raw; }
};
template <> struct SdQuad<__nv_bfloat16, true> {
  uint2 raw;
  __device__ __forceinline__ void load(const __nv_bfloat16* p, int left) {
    raw = make_uint2(0u, 0u);
    if (left > 0) raw = *reinterpret_cast<const uint2*>(p);
  }
  __device__ __forceinline__ float4 value() const {
    return make_float4(__uint_as_float(raw.x << 16), __uint_as_float(raw.x & 0xffff0000u), __uint_as_float(raw.y << 16),
                       __uint_as_float(raw.y & 0xffff0000u));
  }
};
template <> struct SdQuad<__nv_bfloat16, false> {
  unsigned short raw[4];
  __device__ __forceinline__ void load(const __nv_bfloat16* p, int left) {
    const unsigned short* u = reinterpret_cast<const unsigned short*>(p);
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      raw[e] = 0;
      if (left > e) raw[e] = u[e];
    }
  }
  __device__ __forceinline__ float4 value() const {
    return make_float4(__uint_as_float(static_cast<uint32_t>(raw[0]) << 16), __uint_as_float(static_cast<uint32_t>(raw[1]) << 16),
                       __uint_as_float(static_cast<uint32_t>(raw[2]) << 16), __uint_as_float(static_cast<uint32_t>(raw[3]) << 16));
  }
};

static constexpr int kSdV = 8, kSdB = 4;   // validation x train rows of a Gram tile

// The 8 x 4 products of one tile over columns of X [.., K]: eight warps take 128-column units in turn, a
// lane four columns of all twelve rows, so every row is read with full lines and once.  A butterfly
// that halves the number of values with the distance leaves entry `lane` of the tile in every lane.
// SPLIT: `warp` counts over the `warps` of all blocks that share the tile.
template <typename E, bool VEC, bool SPLIT>
__device__ __forceinline__ float sd_gram(const E* X, int K, long long row_v, int rows_v, long long row_b, int rows_b, int warp, int warps,
                                         int lane) {
  float acc[kSdV * kSdB];
#pragma unroll
  for (int e = 0; e < kSdV * kSdB; ++e) acc[e] = 0.f;
  for (int k0 = warp * 128; k0 < K; k0 += SPLIT ? warps * 128 : 1024) {
    const int k = k0 + lane * 4;
    SdQuad<E, VEC> v[kSdV], b[kSdB];
#pragma unroll
    for (int i = 0; i < kSdV; ++i) v[i].load(X + (row_v + (i < rows_v ? i : 0)) * K + k, K - k);
#pragma unroll
    for (int j = 0; j < kSdB; ++j) b[j].load(X + (row_b + (j < rows_b ? j : 0)) * K + k, K - k);
#pragma unroll
    for (int i = 0; i < kSdV; ++i) {
      const float4 x = v[i].value();
#pragma unroll
      for (int j = 0; j < kSdB; ++j) {
        const float4 y = b[j].value();
        float& s = acc[i * kSdB + j];
        s = fmaf(x.x, y.x, s); s = fmaf(x.y, y.y, s); s = fmaf(x.z, y.z, s); s = fmaf(x.w, y.w, s);
      }
    }
  }
#pragma unroll
  for (int o = 16; o >= 1; o >>= 1) {
    const bool up = (lane & o) != 0;
#pragma unroll
    for (int e = 0; e < o; ++e) {
      const float send = up ? acc[e] : acc[e + o], keep = up ? acc[e + o] : acc[e];
      acc[e] = keep + __shfl_xor_sync(0xffffffffu, send, o);
    }
  }
  return acc[0];
}

template <typename E, bool VEC, bool SPLIT>
__global__ void __launch_bounds__(256, 2) dense_small_kernel(const SmallDense q) {
  stream_order();
  __shared__ __align__(16) float sm[2 * 2 * 16 * 64];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const E* A = static_cast<const E*>(q.A);
  const E* B = static_cast<const E*>(q.B);
  int blk = blockIdx.x;

  if (blk < q.gram_blocks) {
    float* red = sm;                     // [operand][warp][32 entries]
    float* part = sm + 512;              // SPLIT: [tile parity][operand][32]: this block's share of the entries
    const int ranks = SPLIT ? q.ranks : 1, rank = SPLIT ? blk % ranks : 0;
    if (SPLIT) blk /= ranks;
    int parity = 0;
    const int v0 = blk / q.groups_b * q.sv, b0 = blk % q.groups_b * q.sb;
    const int nv = min(q.sv, q.n_val - v0), nb = min(q.sb, q.n_train - b0);
    const long long first_v = static_cast<long long>(q.n_train + v0) * q.T, first_b = static_cast<long long>(b0) * q.T;
    const int rows_v = nv * q.T, rows_b = nb * q.T;      // T == 1, or one sample per side, or a few short ones
    float total = 0.f;                   // warp 0: T == 1: entry `lane`; else thread's pair (see below)
    for (int i0 = 0; i0 < rows_v; i0 += kSdV)
      for (int j0 = 0; j0 < rows_b; j0 += kSdB, parity ^= 64) {
        const int rv = min(kSdV, rows_v - i0), rb = min(kSdB, rows_b - j0);
        red[warp * 32 + lane] = sd_gram<E, VEC, SPLIT>(A, q.d, first_v + i0, rv, first_b + j0, rb, rank * 8 + warp, ranks * 8, lane);
        red[256 + warp * 32 + lane] = sd_gram<E, VEC, SPLIT>(B, q.p, first_v + i0, rv, first_b + j0, rb, rank * 8 + warp, ranks * 8, lane);
        __syncthreads();
        if (SPLIT) {                     // rank 0 reads tile k's parts before it arrives at tile k + 1's barrier
          if (warp == 0) {
            float sa = 0.f, sg = 0.f;
#pragma unroll
            for (int w = 0; w < 8; ++w) { sa += red[w * 32 + lane]; sg += red[256 + w * 32 + lane]; }
            part[parity + lane] = sa;
            part[parity + 32 + lane] = sg;
          }
          cluster_sync_all();
        }
        if (warp == 0 && rank == 0) {
          float sa = 0.f, sg = 0.f;
          if (SPLIT) {
            float a[8], g[8];
#pragma unroll
            for (int r = 0; r < 8; ++r)
              if (r < ranks) {
                a[r] = ld_cluster_f32(map_to_cta(smem_u32(part + parity + lane), r));
                g[r] = ld_cluster_f32(map_to_cta(smem_u32(part + parity + 32 + lane), r));
              }
#pragma unroll
            for (int r = 0; r < 8; ++r)
              if (r < ranks) { sa += a[r]; sg += g[r]; }
          } else {
#pragma unroll
            for (int w = 0; w < 8; ++w) { sa += red[w * 32 + lane]; sg += red[256 + w * 32 + lane]; }
          }
          const int i = lane / kSdB, j = lane % kSdB;
          const float prod = i < rv && j < rb ? sa * sg : 0.f;
          if (q.T == 1) {
            total = prod;                // groups are tile-sized: one tile
          } else {                       // pairs (v, b) of the group sum their entries of this tile
            const int mine_v = i0 + i < rows_v ? (i0 + i) / q.T : -1, mine_b = j0 + j < rows_b ? (j0 + j) / q.T : -1;
            for (int pr = 0; pr < nv * nb; ++pr) {
              float s = mine_v == pr / nb && mine_b == pr % nb ? prod : 0.f;
#pragma unroll
              for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
              if (lane == pr) total += s;
            }
          }
        }
        __syncthreads();
      }
    if (SPLIT) cluster_sync_all();       // no block leaves while rank 0 still reads its shared memory
    if (warp == 0 && rank == 0) {
      const int i = q.T == 1 ? lane / kSdB : lane / nb, j = q.T == 1 ? lane % kSdB : lane % nb;
      if (i < nv && j < nb) q.M[static_cast<long long>(v0 + i) * q.n_train + b0 + j] = total;
    }
    return;
  }
  blk -= q.gram_blocks;

  if (blk < q.wgrad_blocks) {            // 64 x 64 outputs, 16 rows per stage, the next stage's loads in flight
    const E* X = q.in_by_out ? A : B;
    const E* Y = q.in_by_out ? B : A;
    const int m = q.in_by_out ? q.d : q.p, n = q.in_by_out ? q.p : q.d;
    const int m0 = blk / q.tiles_n * 64, n0 = blk % q.tiles_n * 64;
    const int rows = q.n_train * q.T;
    float (*xs)[16][64] = reinterpret_cast<float (*)[16][64]>(sm);
    float (*ys)[16][64] = reinterpret_cast<float (*)[16][64]>(sm + 2 * 16 * 64);
    const int lr = threadIdx.x >> 4, lc = (threadIdx.x & 15) * 4;
    const int ty = threadIdx.x >> 4, tx = threadIdx.x & 15;
    float acc[4][4];
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
      for (int j = 0; j < 4; ++j) acc[i][j] = 0.f;
    SdQuad<E, VEC> x, y;
    auto fetch = [&](int r0) {
      const int r = r0 + lr;
      const bool in = r < rows;
      x.load(X + static_cast<long long>(in ? r : 0) * m + m0 + lc, in ? m - m0 - lc : 0);
      y.load(Y + static_cast<long long>(in ? r : 0) * n + n0 + lc, in ? n - n0 - lc : 0);
    };
    fetch(0);
    *reinterpret_cast<float4*>(&xs[0][lr][lc]) = x.value();
    *reinterpret_cast<float4*>(&ys[0][lr][lc]) = y.value();
    __syncthreads();
    int buf = 0;
    for (int r0 = 0; r0 < rows; r0 += 16, buf ^= 1) {
      const bool more = r0 + 16 < rows;
      if (more) fetch(r0 + 16);
#pragma unroll
      for (int k = 0; k < 16; ++k) {
        const float4 a = *reinterpret_cast<const float4*>(&xs[buf][k][ty * 4]);
        const float4 b = *reinterpret_cast<const float4*>(&ys[buf][k][tx * 4]);
        const float av[4] = {a.x, a.y, a.z, a.w}, bv[4] = {b.x, b.y, b.z, b.w};
#pragma unroll
        for (int i = 0; i < 4; ++i)
#pragma unroll
          for (int j = 0; j < 4; ++j) acc[i][j] = fmaf(av[i], bv[j], acc[i][j]);
      }
      if (more) {
        *reinterpret_cast<float4*>(&xs[buf ^ 1][lr][lc]) = x.value();
        *reinterpret_cast<float4*>(&ys[buf ^ 1][lr][lc]) = y.value();
      }
      __syncthreads();
    }
    const bool quad = (n & 3) == 0 && (reinterpret_cast<uintptr_t>(q.grad) & 15u) == 0;
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const int r = m0 + ty * 4 + i, c = n0 + tx * 4;
      if (r >= m || c >= n) continue;
      const long long at = static_cast<long long>(r) * n + c;
      float o[4];
#pragma unroll
      for (int j = 0; j < 4; ++j) o[j] = acc[i][j] * q.grad_scale;
      if (q.grad_f32) {
        float* g = static_cast<float*>(q.grad) + at;
        if (quad) *reinterpret_cast<float4*>(g) = make_float4(o[0], o[1], o[2], o[3]);
        else
#pragma unroll
          for (int j = 0; j < 4; ++j) if (c + j < n) g[j] = o[j];
      } else {
        __nv_bfloat16* g = static_cast<__nv_bfloat16*>(q.grad) + at;
#pragma unroll
        for (int j = 0; j < 4; ++j) if (c + j < n) g[j] = __float2bfloat16_rn(o[j]);
      }
    }
    return;
  }
  blk -= q.wgrad_blocks;

  const int blocks_c = (q.p + 1023) / 1024;
  const int s = blk / blocks_c, c = blk % blocks_c * 1024 + threadIdx.x * 4;
  if (c >= q.p || (SPLIT && (q.colsums == nullptr || s >= q.n_train + q.n_val))) return;      // blocks that fill up the last cluster
  float4 sum = make_float4(0.f, 0.f, 0.f, 0.f);
  const E* row = B + static_cast<long long>(s) * q.T * q.p + c;
#pragma unroll 4
  for (int t = 0; t < q.T; ++t) {
    SdQuad<E, VEC> quad;
    quad.load(row + static_cast<long long>(t) * q.p, q.p - c);
    const float4 x = quad.value();
    sum.x += x.x; sum.y += x.y; sum.z += x.z; sum.w += x.w;
  }
  float* o = q.colsums + static_cast<long long>(s) * q.p + c;
  o[0] = sum.x;
  if (c + 1 < q.p) o[1] = sum.y;
  if (c + 2 < q.p) o[2] = sum.z;
  if (c + 3 < q.p) o[3] = sum.w;
}

}  // namespace gb

using namespace gb;

// The line between this kernel and the tensor-core paths.  Pairs x features is the traffic of the Gram part
// (about one byte of L2 reads each; 2e7 take 5 us), rows x d x p the multiply-adds of the train
// gradient (about 12e12 a second here).  Beyond these the fixed costs it avoids -- some 40 us of
// launches for float32 operands, 20 us for bf16 -- no longer pay for slower arithmetic.  A pair of
// samples is one block, which walks its token tiles in turn (1.5 us each): at most eight of them.
//
// A gradient tile is one block that walks all train rows, 0.045 us each (float32; 0.045 to 0.067 bf16),
// however few the tiles are; the tensor-core paths split the rows.  GPU time of a hook, this kernel
// against the better of them: 64 -> 64 float32, one-token samples, 35 / 34 us at 768 rows, 91 / 37 at 2048,
// 715 / 68 at 16384; 1024 -> 128 45 / 58 us at 1024 rows, 70 / 58 at 1536; with 16 tokens a sample 23 / 21
// at 512, 45 / 23 at 1024; bf16 64 -> 64 23 / 25 us at 512 rows, 45 / 26 at 1024.
extern "C" int ghost_dense_small_fits(int is_f32, int n_train, int n_val, long long T, int d, int p) {
  const double pairs = static_cast<double>(n_train) * T * n_val * T;
  const double train_rows = static_cast<double>(n_train) * T;
  const double macs = train_rows * d * p;
  const double rows = static_cast<double>(n_train + n_val) * T;
  const double chain = !is_f32 || T > 4 ? 512 : 700 + 0.6 * (static_cast<double>(d) + p);
  return T <= 16 && pairs * (static_cast<double>(d) + p) <= 2e7 && macs <= (is_f32 ? 3e8 : 6e7) && rows * p <= 1e8 &&
         train_rows <= chain ? 1 : 0;
}

template <typename E, bool VEC>
static cudaError_t launch_small(const SmallDense& q, unsigned grid, cudaStream_t st) {
  if (q.ranks > 1) return launch_next_cluster(dim3(q.ranks), dense_small_kernel<E, VEC, true>, dim3(grid), dim3(256), 0, st, q);
  return launch_next(dense_small_kernel<E, VEC, false>, dim3(grid), dim3(256), 0, st, q);
}

// Sample groups of a call, and what small_cluster() makes of it
struct SmallGroups { int sv, sb, groups_b; long long gram, wgrad; int ranks; };
static SmallGroups small_groups(int n_train, int n_val, long long T, int d, int p, bool want_grad, const DeviceState* ds) {
  SmallGroups g;
  // groups of whole samples: a tile's worth of one-token samples, fewer longer ones, at least one
  g.sv = T >= kSdV ? 1 : static_cast<int>(kSdV / T);
  g.sb = T >= kSdB ? 1 : static_cast<int>(kSdB / T);
  g.groups_b = ceil_div(n_train, g.sb);
  g.gram = static_cast<long long>(ceil_div(n_val, g.sv)) * g.groups_b;
  g.wgrad = want_grad ? static_cast<long long>(ceil_div(d, 64)) * ceil_div(p, 64) : 0;
  g.ranks = small_cluster(g.gram, (T + kSdV - 1) / kSdV * ((T + kSdB - 1) / kSdB), g.wgrad, n_train * T, d, p, ds->sm_count);
  return g;
}

extern "C" int ghost_dense_small_cluster_size(int n_train, int n_val, long long T, int d, int p, int want_grad) {
  const DeviceState* ds = device_state();
  if (!ds) return GHOST_ERR_DEVICE;
  GB_REQUIRE(n_train > 0 && n_val > 0 && T > 0 && d > 0 && p > 0, "ghost_dense_small_cluster_size: bad size");
  return small_groups(n_train, n_val, T, d, p, want_grad != 0, ds).ranks;
}

extern "C" int ghost_dense_small(const void* A, const void* B, int is_f32, int n_train, int n_val, long long T, int d,
                                 int p, int in_by_out, float* M_out, void* grad_out, int grad_is_f32, float grad_scale,
                                 float* colsum_out, void* stream) {
  const DeviceState* ds = device_state();
  if (!ds) return GHOST_ERR_DEVICE;
  GB_REQUIRE(A && B && M_out, "ghost_dense_small: null pointer");
  GB_REQUIRE(n_train > 0, "No training samples to compute dot product, check batch sizes.");
  GB_REQUIRE(n_val > 0 && T > 0 && d > 0 && p > 0, "ghost_dense_small: empty dimension");
  GB_REQUIRE(ghost_dense_small_fits(is_f32, n_train, n_val, T, d, p), "ghost_dense_small: beyond the sizes this kernel is for");
  SmallDense q = {};
  q.A = A; q.B = B;
  q.n_train = n_train; q.n_val = n_val; q.T = static_cast<int>(T); q.d = d; q.p = p;
  q.in_by_out = in_by_out;
  q.M = M_out;
  q.grad = grad_out; q.grad_f32 = grad_is_f32; q.grad_scale = grad_scale;
  q.colsums = colsum_out;
  const SmallGroups groups = small_groups(n_train, n_val, T, d, p, grad_out != nullptr, ds);
  q.sv = groups.sv; q.sb = groups.sb; q.groups_b = groups.groups_b; q.ranks = groups.ranks;
  q.tiles_n = ceil_div(in_by_out ? p : d, 64);
  const long long gram = groups.gram, wgrad = groups.wgrad;
  const long long col = colsum_out ? static_cast<long long>(n_train + n_val) * ceil_div(p, 1024) : 0;
  GB_REQUIRE(gram + wgrad + col < (1ll << 31), "ghost_dense_small: too many blocks");
  q.gram_blocks = static_cast<int>(gram * q.ranks);
  q.wgrad_blocks = static_cast<int>(wgrad);
  const uintptr_t align = is_f32 ? 15 : 7;
  const bool vec = d % 4 == 0 && p % 4 == 0 && (reinterpret_cast<uintptr_t>(A) & align) == 0 && (reinterpret_cast<uintptr_t>(B) & align) == 0;
  const unsigned grid = static_cast<unsigned>((gram * q.ranks + wgrad + col + q.ranks - 1) / q.ranks * q.ranks);
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  if (is_f32) {
    if (vec) GB_CUDA_OK((launch_small<float, true>(q, grid, st)));
    else GB_CUDA_OK((launch_small<float, false>(q, grid, st)));
  } else {
    if (vec) GB_CUDA_OK((launch_small<__nv_bfloat16, true>(q, grid, st)));
    else GB_CUDA_OK((launch_small<__nv_bfloat16, false>(q, grid, st)));
  }
  count_launch();
  return post_launch("dense_small_kernel");
}
