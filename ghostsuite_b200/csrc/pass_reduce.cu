// End-of-pass reductions.  A backward pass leaves one small job per parameter: the [n_val, n_train]
// Gram of per-sample vectors (bias, LayerNorm, RMS norm), the sum of their train rows, and the column
// sum over the validation samples of every parameter's matrix.  All of them run in one launch whose
// jobs travel as kernel parameters; a second kernel adds the finished matrices of a step up.
#include <string.h>

#include <cooperative_groups.h>
#include <type_traits>

#include "common.cuh"

namespace cg = cooperative_groups;

namespace gb {

// One cluster of eight CTAs per (job, block of 32 train samples).  The vectors are a few hundred
// kilobytes in L2, so what bounds a job is how few SMs fetch them and the latency of each round of
// loads: the eight CTAs split the vector length F; a CTA brings its columns of 32 train and eight
// validation rows into shared memory with full-line copies, all in flight at once, and a lane then
// holds one train sample against eight validation samples.  Partial sums meet in distributed shared
// memory in a fixed order, so results do not depend on timing.  A warp per (validation, train) pair,
// the form before it, fetched every row once per partner; lanes that loaded one row each from global
// memory touched 32 lines per instruction.
static constexpr int kPassCluster = 8;
static constexpr int kPassThreads = 256;
// Columns staged at a time: a CTA's whole share up to kPassMost, so that one round of loads serves it and the sums of
// the train rows come out of the same copy (32 + 8 vectors of 3072: two rounds and a second pass over the
// rows 10.8 us, 9.5 now; of 768: 6.7 and 5.0); no more than the list's longest vector needs, which leaves room for the CTAs of other kernels, and half of
// kPassMost with blocks of sixteen validation rows, and where the launch has more CTAs than three quarters of the SMs, which would wait
// for their memory then (32 + 8 vectors of 8192, one job 22.2 us in halves and 18.4 whole; 24 jobs 25.7 and 49).
static constexpr int kPassMost = 1024;
// Shared memory that keeps a second CTA off the SM.  Two of 111 KB turn all of an SM's memory into shared memory, and the kernel that
// comes up there next has no L1 for its loads: RMS hooks of 6 + 2 x 1024 x 5120 float32 in a row took 104 us, 85.7 in halves, 80.8
// so.  (Rounds of more than 512 with sixteen validation rows, 160 KB and up, do the same alone: 6 + 10 x 512 x 8192 113 us in halves, 126.)
static constexpr int kPassAlone = 118 * 1024;
__host__ __device__ constexpr int pass_pitch(int sub) { return sub + 4; }      // rows 16 bytes apart modulo 128: no bank conflicts
// 32 train rows, then nv validation rows; behind them the warps' partial sums
__host__ __device__ constexpr int pass_smem(int sub, int nv) { return (32 + nv) * pass_pitch(sub) * 4 + 8 * nv * 32 * 4; }
__host__ __device__ constexpr int pass_chunk(int F) { return ((F + kPassCluster - 1) / kPassCluster + 7) / 8 * 8; }

static constexpr double kPassOneMatrix = 1 << 21;     // products of a single matrix that the clusters take

template <int CAP> struct PassJobs { int sub; ghost_pass_job job[CAP]; };      // sub: columns staged at a time, a multiple of 32

__device__ __forceinline__ const float* pass_val_row(const ghost_pass_job& j, int v) {
  return j.Xv == nullptr ? j.X + static_cast<long long>(j.n_train + v) * j.F
                         : j.Xv + static_cast<long long>(v / j.v_per_rank) * j.v_rank_pitch +
                               static_cast<long long>(v % j.v_per_rank) * j.F;
}

// Columns [f, f + width) of `train` train rows from b0 on and `val` validation rows from v0 on into shared memory, from rows 0 and 32 on,
// zero up to the next multiple of four.  Rows that are not there stay what they were: what their lanes make of them is not
// read.  (3 + 1 vectors of 8192: 18.1 us with 36 rows of zeros and two rounds of 512 columns, 10.2 so; 48 jobs of 8 + 2 41 and 27.)
__device__ __forceinline__ void pass_stage(const ghost_pass_job& j, bool vec, int b0, int train, int v0, int val, int f, int width, float* st,
                                           int pitch) {
  const int quads = (width + 3) / 4;
  for (int i = threadIdx.x; i < (train + val) * quads; i += kPassThreads) {
    const int row = i / quads, r = row < train ? row : row - train + 32, q = (i - row * quads) * 4;
    const float* src = row < train ? j.X + static_cast<long long>(b0 + row) * j.F : pass_val_row(j, v0 + row - train);
    float* dst = st + r * pitch + q;
    if (vec) {                    // F is a multiple of four then, and so is every width
      asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(static_cast<uint32_t>(__cvta_generic_to_shared(dst))),
                   "l"(src + f + q) : "memory");
    } else {
      float x[4];
#pragma unroll
      for (int e = 0; e < 4; ++e) x[e] = q + e < width ? src[f + q + e] : 0.f;
      *reinterpret_cast<float4*>(dst) = make_float4(x[0], x[1], x[2], x[3]);
    }
  }
  asm volatile("cp.async.wait_all;" ::: "memory");
}

// sum_out over columns [f0, f1): the clusters of a job take groups of 128 columns in turn, four groups at
// a time; a warp adds every eighth train row, and the eight partial rows meet in shared memory.
template <bool VEC>
__device__ __forceinline__ void pass_row_sums(const ghost_pass_job& j, int f0, int f1, int blk, int n_blk, float* red) {
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  for (int c0 = f0 + blk * 128; c0 < f1; c0 += 4 * 128 * n_blk) {
    float4 acc[4];
#pragma unroll
    for (int g = 0; g < 4; ++g) acc[g] = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll 4
    for (int n = warp; n < j.n_train; n += 8) {
      const float* row = j.X + static_cast<long long>(n) * j.F;
#pragma unroll
      for (int g = 0; g < 4; ++g) {
        const int c = c0 + g * 128 * n_blk + lane * 4;
        if constexpr (VEC) {
          if (c < f1) {
            const float4 x = *reinterpret_cast<const float4*>(row + c);
            acc[g].x += x.x; acc[g].y += x.y; acc[g].z += x.z; acc[g].w += x.w;
          }
        } else {
          if (c < f1) acc[g].x += row[c];
          if (c + 1 < f1) acc[g].y += row[c + 1];
          if (c + 2 < f1) acc[g].z += row[c + 2];
          if (c + 3 < f1) acc[g].w += row[c + 3];
        }
      }
    }
    __syncthreads();                     // whatever used `red` before is done with it
#pragma unroll
    for (int g = 0; g < 4; ++g) *reinterpret_cast<float4*>(red + (warp * 4 + g) * 128 + lane * 4) = acc[g];
    __syncthreads();
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      const int i = h * kPassThreads + threadIdx.x, c = c0 + (i >> 7) * 128 * n_blk + (i & 127);
      if (c >= f1) continue;
      float s = 0.f;
#pragma unroll
      for (int w = 0; w < 8; ++w) s += red[w * 512 + i];
      s *= j.sum_scale;
      if (j.sum_is_f32) static_cast<float*>(j.sum_out)[c] = s;
      else static_cast<__nv_bfloat16*>(j.sum_out)[c] = __float2bfloat16_rn(s);
    }
  }
}

// The same sums, bit for bit, from the staged columns of a block that holds all train rows
// (`train` of them, staged up to the next multiple of eight)
__device__ __forceinline__ void pass_staged_sums(const ghost_pass_job& j, int train, int f, int width, const float* st, int pitch) {
  for (int c = threadIdx.x; c < width; c += kPassThreads) {
    float a[8] = {};
#pragma unroll
    for (int n = 0; n < 32; n += 8)
      if (n < train)
#pragma unroll
        for (int w = 0; w < 8; ++w) a[w] += st[(n + w) * pitch + c];
    float s = 0.f;
#pragma unroll
    for (int w = 0; w < 8; ++w) s += a[w];
    s *= j.sum_scale;
    if (j.sum_is_f32) static_cast<float*>(j.sum_out)[f + c] = s;
    else static_cast<__nv_bfloat16*>(j.sum_out)[f + c] = __float2bfloat16_rn(s);
  }
}

// Sum of eight values in pairs
template <typename F> __device__ __forceinline__ float pass_sum8(F&& v) {
  return ((v(0) + v(1)) + (v(2) + v(3))) + ((v(4) + v(5)) + (v(6) + v(7)));
}

// NV: validation rows that go through a block together, 16 where a job has more than eight.  256 + 32 vectors of 1024 took
// 21 us in four rounds that each brought the train rows again, 16 in two; with eight or fewer, 16 would stage rows of zeros.
template <int CAP, int NV>
__global__ void __cluster_dims__(kPassCluster, 1, 1) __launch_bounds__(kPassThreads)
pass_reduce_kernel(const __grid_constant__ PassJobs<CAP> jobs) {
  extern __shared__ __align__(16) float stage[];       // pass_smem(sub, NV) bytes
  const int pitch = pass_pitch(jobs.sub);
  stream_order();
  __shared__ float part[2][NV][32];      // this CTA's share of F, read by rank 0 of the cluster
  __shared__ float cols[8][32];
  const ghost_pass_job& j = jobs.job[blockIdx.z];
  const int n_blk = (j.n_train + 31) / 32, step = gridDim.y;       // one block each, unless a job has more than a grid
  if (blockIdx.y >= n_blk) return;       // the whole cluster leaves
  const int rank = blockIdx.x;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;

  if (j.X == nullptr) {                  // the matrix exists already: column sums only
    if (rank != 0) return;
    for (int blk = blockIdx.y; blk < n_blk; blk += step) {
      const int b = blk * 32 + lane;
      float s = 0.f;
      if (b < j.n_train)
        for (int v = warp; v < j.n_val; v += 8) s += j.M[static_cast<long long>(v) * j.n_train + b];
      __syncthreads();
      cols[warp][lane] = s;
      __syncthreads();
      if (warp == 0 && b < j.n_train) {
#pragma unroll
        for (int w = 1; w < 8; ++w) s += cols[w][lane];
        j.vec[b] = s;
      }
    }
    return;
  }

  const int F = j.F;
  const int chunk = pass_chunk(F);
  const int f0 = rank * chunk;
  const int f1 = f0 + chunk < F ? f0 + chunk : F;
  const bool vec_x = (F & 3) == 0 && (reinterpret_cast<uintptr_t>(j.X) & 15) == 0;

  // all train rows are in one block and all of this CTA's columns in one round
  const bool staged_sums = j.M != nullptr && j.sum_out != nullptr && n_blk == 1 && chunk <= jobs.sub;
  if (j.M != nullptr) {
    cg::cluster_group cluster = cg::this_cluster();
    const bool vec = vec_x && (j.Xv == nullptr || ((reinterpret_cast<uintptr_t>(j.Xv) & 15) == 0 && (j.v_rank_pitch & 3) == 0));
    int buf = 0;
    for (int blk = blockIdx.y; blk < n_blk; blk += step) {
      const int b = blk * 32 + lane;
      const bool live = b < j.n_train;
      const int train = j.n_train - blk * 32 < 32 ? j.n_train - blk * 32 : 32;
      float col = 0.f;                     // rank 0: this thread's share of vec
      for (int v0 = 0; v0 < j.n_val; v0 += NV, buf ^= 1) {
        float4 acc[NV];                    // a sum per quarter of the columns: short chains, as one warp per pair had
#pragma unroll
        for (int i = 0; i < NV; ++i) acc[i] = make_float4(0.f, 0.f, 0.f, 0.f);
        const int val = j.n_val - v0 < NV ? j.n_val - v0 : NV;
        for (int f = f0; f < f1; f += jobs.sub) {
          const int width = f1 - f < jobs.sub ? f1 - f : jobs.sub;
          __syncthreads();
          if (staged_sums && v0 == 0)        // for the sums below: zeros up to the next multiple of eight rows
            for (int i = threadIdx.x; i < (-train & 7) * pitch; i += kPassThreads) stage[train * pitch + i] = 0.f;
          // one round holds all columns: the train rows are there already
          pass_stage(j, vec, blk * 32, v0 > 0 && chunk <= jobs.sub ? 0 : train, v0, val, f, width, stage, pitch);
          __syncthreads();
          if (staged_sums && v0 == 0) pass_staged_sums(j, train, f, width, stage, pitch);
          auto products = [&](auto some) {     // of the first rows; a test a row costs more than products that are not read (24 jobs of 32 + 8
                                               // vectors of 4096 19.4 us with tests, 16.4 without)
            // two steps of sixteen rows at a time would take 143 registers, which leaves an SM one block: 48 jobs of 53 + 17 vectors of 2560 77 us so, 42
            // with 128; 24 of 11 + 13 x 640 9.4 and 6.0
#pragma unroll (NV == 16 ? 1 : 2)
            for (int q = warp * 4; q < width; q += 32) {
              const float4 x = *reinterpret_cast<const float4*>(stage + lane * pitch + q);
#pragma unroll
              for (int i = 0; i < decltype(some)::value; ++i) {
                const float4 y = *reinterpret_cast<const float4*>(stage + (32 + i) * pitch + q);
                acc[i].x = fmaf(x.x, y.x, acc[i].x); acc[i].y = fmaf(x.y, y.y, acc[i].y);
                acc[i].z = fmaf(x.z, y.z, acc[i].z); acc[i].w = fmaf(x.w, y.w, acc[i].w);
              }
            }
          };
          if (val > NV / 2) products(std::integral_constant<int, NV>());
          else if (val > NV / 4) products(std::integral_constant<int, NV / 2>());
          else products(std::integral_constant<int, NV / 4>());
        }
        float* red = stage + (32 + NV) * pitch;        // [warp][validation row][train lane]
#pragma unroll
        for (int i = 0; i < NV; ++i) red[(warp * NV + i) * 32 + lane] = (acc[i].x + acc[i].y) + (acc[i].z + acc[i].w);
        __syncthreads();
        // thread (warp, lane) now owns pairs (v0 + warp, b), (v0 + 8 + warp, b)
#pragma unroll
        for (int h = 0; h < NV; h += 8)
          part[buf][h + warp][lane] = pass_sum8([&](int w) { return red[(w * NV + h + warp) * 32 + lane]; });
        // one cluster barrier per block: `part` alternates, and rank 0 reads block k's before it
        // arrives at block k + 1's barrier, which every CTA passes before writing that buffer again
        cluster.sync();
        if (rank == 0) {
#pragma unroll
          for (int h = 0; h < NV; h += 8) {
            const float m = j.dot_scale * pass_sum8([&](int r) { return *cluster.map_shared_rank(&part[buf][h + warp][lane], r); });
            if (v0 + h + warp < j.n_val && live) {
              j.M[static_cast<long long>(v0 + h + warp) * j.n_train + b] = m;
              col += m;
            }
          }
        }
      }
      if (rank == 0 && j.vec != nullptr) {
        cols[warp][lane] = col;
        __syncthreads();
        if (warp == 0 && live) j.vec[b] = pass_sum8([&](int w) { return cols[w][lane]; });
      }
      __syncthreads();                   // `cols` and the staged rows are free for the next block
    }
    if (j.sum_out == nullptr || staged_sums) cluster.sync();   // no CTA leaves while rank 0 still reads its shared memory
  }
  if (j.sum_out != nullptr && !staged_sums) {
    const int share = n_blk < step ? n_blk : step;
    if (vec_x) pass_row_sums<true>(j, f0, f1, blockIdx.y, share, stage);
    else pass_row_sums<false>(j, f0, f1, blockIdx.y, share, stage);
    if (j.M != nullptr) cg::this_cluster().sync();
  }
}

// M[v, b] = scale * <X[n_train + v], X[b]> with a warp per pair: for one matrix on its own, whose blocks above
// are too few to fill the GPU once a pair is long or the validation rows are many (a cluster goes through
// them sixteen at a time).  256 x 256 pairs of 768: 47 us in the clusters, 19 here; 256 x 32 of 50257: 308 and 139;
// 16384 x 1 of 1024: 64 and 11; 256 x 128 of 256 19 and 9.  Smaller ones (64 x 64 of 512: 11.6 in the clusters), and every matrix of a batch, stay with the clusters, which fetch a row once.
__global__ void __launch_bounds__(256) small_gram_kernel(const float* X, int n_train, unsigned pairs, int F,
                                                         float scale, float* __restrict__ M) {
  stream_order();
  const unsigned pair = blockIdx.x * 8u + (threadIdx.x >> 5);
  const int lane = threadIdx.x & 31;
  if (pair >= pairs) return;
  const unsigned v = pair / static_cast<unsigned>(n_train);
  const float* xv = X + static_cast<long long>(n_train + v) * F;
  const float* xb = X + static_cast<long long>(pair - v * n_train) * F;
  float even[4] = {0.f, 0.f, 0.f, 0.f}, odd[4] = {0.f, 0.f, 0.f, 0.f};      // short chains: 256 sums a pair
  if ((F & 3) == 0 && (reinterpret_cast<uintptr_t>(X) & 15) == 0) {
    auto add = [&](int f, float (&sum)[4]) {
      const float4 x = reinterpret_cast<const float4*>(xv)[f], y = reinterpret_cast<const float4*>(xb)[f];
      sum[0] = fmaf(x.x, y.x, sum[0]); sum[1] = fmaf(x.y, y.y, sum[1]);
      sum[2] = fmaf(x.z, y.z, sum[2]); sum[3] = fmaf(x.w, y.w, sum[3]);
    };
    const int F4 = F >> 2;
    int f = lane;
#pragma unroll 2
    for (; f + 32 < F4; f += 64) { add(f, even); add(f + 32, odd); }
    if (f < F4) add(f, even);
  } else {
    for (int f0 = lane; f0 < F; f0 += 512) {     // sixteen loads of either row in flight
      float x[16], y[16];
#pragma unroll
      for (int u = 0; u < 16; ++u) {
        const bool in = f0 + u * 32 < F;
        x[u] = in ? xv[f0 + u * 32] : 0.f;
        y[u] = in ? xb[f0 + u * 32] : 0.f;
      }
#pragma unroll
      for (int u = 0; u < 16; ++u) {
        float& sum = (u & 4) ? odd[u & 3] : even[u & 3];
        sum = fmaf(x[u], y[u], sum);
      }
    }
  }
  float s = ((even[0] + even[1]) + (even[2] + even[3])) + ((odd[0] + odd[1]) + (odd[2] + odd[3]));
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
  if (lane == 0) M[pair] = s * scale;
}

// out[c] = (accumulate ? out[c] : 0) + scale * sum over the rows of X[n, c] for one matrix on its own: the
// additions of pass_row_sums in their order (the same bits), with a block per COLS columns instead of the
// blocks that a job's pairs ask for.  4 rows of 1000003: 245 us in the
// batched kernel, 17 here; 256 of 50257: 68 and 16; 16384 of 1024: 626 and 123.
template <int COLS>
__global__ void __launch_bounds__(256) rows_sum_kernel(const float* X, int n_rows, int F, float scale,
                                                       void* __restrict__ out, int out_is_f32, int accumulate) {
  stream_order();
  constexpr int PER = COLS / 32;
  __shared__ float red[8][COLS];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const long long c0 = blockIdx.x * static_cast<long long>(COLS);
  float acc[PER];
#pragma unroll
  for (int g = 0; g < PER; ++g) acc[g] = 0.f;
#pragma unroll 8
  for (int n = warp; n < n_rows; n += 8) {
    const float* row = X + static_cast<long long>(n) * F + c0;
#pragma unroll
    for (int g = 0; g < PER; ++g)
      if (c0 + g * 32 + lane < F) acc[g] += row[g * 32 + lane];
  }
#pragma unroll
  for (int g = 0; g < PER; ++g) red[warp][g * 32 + lane] = acc[g];
  __syncthreads();
  const long long c = c0 + threadIdx.x;
  if (threadIdx.x >= COLS || c >= F) return;
  float s = 0.f;
#pragma unroll
  for (int w = 0; w < 8; ++w) s += red[w][threadIdx.x];
  s *= scale;
  if (out_is_f32) {
    float* o = static_cast<float*>(out) + c;
    *o = accumulate ? s + *o : s;
  } else {
    __nv_bfloat16* o = static_cast<__nv_bfloat16*>(out) + c;
    *o = __float2bfloat16_rn(accumulate ? s + __bfloat162float(*o) : s);
  }
}

template <int CAP, int NV>
static int launch_pass(const ghost_pass_job* jobs, int n, int blocks, const DeviceState* ds, cudaStream_t st) {
  static bool attr_set[64] = {};
  if (!attr_set[ds->device]) {
    GB_CUDA_OK(cudaFuncSetAttribute(pass_reduce_kernel<CAP, NV>, cudaFuncAttributeMaxDynamicSharedMemorySize, pass_smem(kPassMost, NV)));
    attr_set[ds->device] = true;
  }
  PassJobs<CAP> batch;
  memcpy(batch.job, jobs, sizeof(ghost_pass_job) * n);
  int longest = 0;
  for (int i = 0; i < n; ++i)
    if (jobs[i].X != nullptr && jobs[i].F > longest) longest = jobs[i].F;
  const int sub = (pass_chunk(longest) + 31) / 32 * 32;
  // the row sums of longer lists reduce 8 x 4 x 128 partial sums in the same memory
  const int most = NV == 8 && static_cast<long long>(blocks) * n * kPassCluster * 4 <= ds->sm_count * 3ll ? kPassMost : kPassMost / 2;
  batch.sub = sub < 128 ? 128 : sub > most ? most : sub;
  int smem = pass_smem(batch.sub, NV);
  if (batch.sub > kPassMost / 2 && smem < kPassAlone) smem = kPassAlone;
  GB_CUDA_OK(launch_next(pass_reduce_kernel<CAP, NV>, dim3(dim3(kPassCluster, blocks, n)), dim3(kPassThreads), smem, st, batch));
  count_launch();
  return post_launch("pass_reduce_kernel");
}

// total[v, b] = sum_p mats[p][v, b];  vec[b] = sum_v total[v, b].  One CTA per 32 train samples, its
// 32 warps split over eight validation rows and four groups of matrices: a step has one matrix per
// parameter, a few kilobytes each, and the time is the chain of loads per thread.
static constexpr int kSumPointers = 440;   // 3520 bytes of pointers: below the 4 KB every driver takes
struct MatrixList { const float* m[kSumPointers]; };

__global__ void __launch_bounds__(1024)
matrix_sum_kernel(const __grid_constant__ MatrixList list, int n, int n_val, int n_train, int accumulate,
                  float* total, float* vec, const int* err_word, int* err_out) {
  stream_order();
  __shared__ float red[4][8][32];
  __shared__ float cols[8][32];
  const int lane = threadIdx.x & 31, row = (threadIdx.x >> 5) & 7, grp = threadIdx.x >> 8;
  const int b = blockIdx.x * 32 + lane;
  float col = 0.f;
  for (int v0 = 0; v0 < n_val; v0 += 8) {
    const int v = v0 + row;
    const long long at = static_cast<long long>(v) * n_train + b;
    const bool live = v < n_val && b < n_train;
    float s = 0.f;
    if (live) {
#pragma unroll 8
      for (int p = grp; p < n; p += 4) s += list.m[p][at];
    }
    red[grp][row][lane] = s;
    __syncthreads();
    if (grp == 0 && live) {
      s = (red[0][row][lane] + red[1][row][lane]) + (red[2][row][lane] + red[3][row][lane]);
      if (accumulate) s += total[at];
      total[at] = s;
      col += s;
    }
    __syncthreads();
  }
  if (grp == 0) cols[row][lane] = col;
  __syncthreads();
  if (threadIdx.x < 32 && b < n_train) {
    float s = 0.f;
#pragma unroll
    for (int r = 0; r < 8; ++r) s += cols[r][lane];
    vec[b] = s;
  }
  if (err_out != nullptr && blockIdx.x == 0 && threadIdx.x == 0) *err_out = *err_word;
}

}  // namespace gb

using namespace gb;

extern "C" int ghost_pass_reduce(const ghost_pass_job* jobs, int n_jobs, void* stream) {
  const DeviceState* ds = device_state();
  if (!ds) return GHOST_ERR_DEVICE;
  GB_REQUIRE(jobs != nullptr && n_jobs > 0, "ghost_pass_reduce: no jobs");
  for (int i = 0; i < n_jobs; ++i) {
    const ghost_pass_job& j = jobs[i];
    GB_REQUIRE(j.n_train > 0 && j.n_val >= 0 && (j.M == nullptr || j.n_val > 0), "ghost_pass_reduce: job %d has an empty dimension", i);
    if (j.X == nullptr) {
      GB_REQUIRE(j.M != nullptr && j.vec != nullptr, "ghost_pass_reduce: job %d has no input or no output", i);
      continue;
    }
    GB_REQUIRE(j.M != nullptr || j.sum_out != nullptr, "ghost_pass_reduce: job %d has no input or no output", i);
    GB_REQUIRE(j.F > 0, "ghost_pass_reduce: job %d has an empty dimension", i);
    GB_REQUIRE(j.M != nullptr || j.vec == nullptr, "ghost_pass_reduce: job %d wants column sums without a matrix", i);
    GB_REQUIRE(j.Xv == nullptr || (j.v_per_rank > 0 && j.v_rank_pitch >= static_cast<long long>(j.v_per_rank) * j.F),
               "ghost_pass_reduce: job %d has separate validation rows without a valid layout", i);
  }
  // Kernel parameters are copied whole whatever the job count, so short lists take a small block.
  // A few jobs are one layer called on its own; the largest block (24 KB of the 32 KB a launch
  // takes) holds all parameters of a GPT-2-sized model.
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  constexpr int kLarge = 300;
  for (int first = 0; first < n_jobs; first += kLarge) {
    const int n = n_jobs - first < kLarge ? n_jobs - first : kLarge;
    int most = 1;
    for (int i = 0; i < n; ++i) most = jobs[first + i].n_train > most ? jobs[first + i].n_train : most;
    const int blocks = ceil_div(most, 32) < 65535 ? ceil_div(most, 32) : 65535;
    bool many = false;
    for (int i = 0; i < n; ++i) many |= jobs[first + i].M != nullptr && jobs[first + i].X != nullptr && jobs[first + i].n_val > 8;
    const ghost_pass_job* list = jobs + first;
    const int rc = n <= 4    ? many ? launch_pass<4, 16>(list, n, blocks, ds, st) : launch_pass<4, 8>(list, n, blocks, ds, st)
                   : n <= 40 ? many ? launch_pass<40, 16>(list, n, blocks, ds, st) : launch_pass<40, 8>(list, n, blocks, ds, st)
                   : many    ? launch_pass<kLarge, 16>(list, n, blocks, ds, st)
                             : launch_pass<kLarge, 8>(list, n, blocks, ds, st);
    if (rc != GHOST_OK) return rc;
  }
  return GHOST_OK;
}

extern "C" int ghost_small_reduce_batch(const ghost_small_job* jobs, int n_jobs, void* stream) {
  GB_REQUIRE(jobs != nullptr && n_jobs > 0, "ghost_small_reduce_batch: no jobs");
  constexpr int kAtATime = 48;
  ghost_pass_job batch[kAtATime];
  for (int first = 0; first < n_jobs; first += kAtATime) {
    const int n = n_jobs - first < kAtATime ? n_jobs - first : kAtATime;
    for (int i = 0; i < n; ++i) {
      const ghost_small_job& s = jobs[first + i];
      GB_REQUIRE(s.X != nullptr, "ghost_small_reduce_batch: job %d has no input or no output", first + i);
      batch[i] = ghost_pass_job{s.X, s.Xv, s.M, nullptr, s.sum_out, s.v_rank_pitch, s.n_train, s.n_val, s.F,
                                s.v_per_rank, s.sum_is_f32, s.dot_scale, s.sum_scale};
    }
    const int rc = ghost_pass_reduce(batch, n, stream);
    if (rc != GHOST_OK) return rc;
  }
  return GHOST_OK;
}

extern "C" int ghost_small_gram_f32(const float* X, int n_train, int n_val, int F, float scale,
                                    float* M_out, void* stream) {
  GB_REQUIRE(X && M_out, "ghost_small_gram_f32: null pointer");
  GB_REQUIRE(n_train > 0, "No training samples to compute dot product, check batch sizes.");
  GB_REQUIRE(n_val > 0 && F > 0, "ghost_small_gram_f32: bad dimensions");
  const long long pairs = static_cast<long long>(n_train) * n_val;
  if (static_cast<double>(pairs) * F <= kPassOneMatrix) {
    const ghost_pass_job j = {X, nullptr, M_out, nullptr, nullptr, 0, n_train, n_val, F, 0, 1, scale, 1.f};
    return ghost_pass_reduce(&j, 1, stream);
  }
  if (!device_state()) return GHOST_ERR_DEVICE;
  GB_REQUIRE(pairs < (1ll << 32) - 8, "ghost_small_gram_f32: too many pairs");
  GB_CUDA_OK(launch_next(small_gram_kernel, dim3(ceil_div(pairs, 8)), dim3(256), 0, static_cast<cudaStream_t>(stream), X, n_train, static_cast<unsigned>(pairs), F, scale, M_out));
  count_launch();
  return post_launch("small_gram_kernel");
}

extern "C" int ghost_rows_sum(const float* X, int n_rows, int F, float scale, void* out, int out_is_f32,
                              int accumulate, void* stream) {
  const DeviceState* ds = device_state();
  if (!ds) return GHOST_ERR_DEVICE;
  GB_REQUIRE(X && out, "ghost_rows_sum: null pointer");
  GB_REQUIRE(n_rows > 0 && F > 0, "ghost_rows_sum: bad dimensions");
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  // wide blocks read full lines; narrow ones while a row has too few for the GPU
  if (ceil_div(F, 128) >= ds->sm_count)
    GB_CUDA_OK(launch_next(rows_sum_kernel<128>, dim3(ceil_div(F, 128)), dim3(256), 0, st, X, n_rows, F, scale, out, out_is_f32, accumulate));
  else
    GB_CUDA_OK(launch_next(rows_sum_kernel<32>, dim3(ceil_div(F, 32)), dim3(256), 0, st, X, n_rows, F, scale, out, out_is_f32, accumulate));
  count_launch();
  return post_launch("rows_sum_kernel");
}

extern "C" int ghost_matrix_sum(const float* const* mats, int n_mats, int n_val, int n_train, float* total,
                                float* vec, int* err_out, void* stream) {
  const DeviceState* ds = device_state();
  if (!ds) return GHOST_ERR_DEVICE;
  GB_REQUIRE(mats && total && vec, "ghost_matrix_sum: null pointer");
  GB_REQUIRE(n_mats > 0 && n_val > 0 && n_train > 0, "ghost_matrix_sum: empty dimension");
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  for (int first = 0; first < n_mats; first += kSumPointers) {
    const int n = n_mats - first < kSumPointers ? n_mats - first : kSumPointers;
    MatrixList list;
    memcpy(list.m, mats + first, sizeof(float*) * n);
    const bool last = first + n == n_mats;
    GB_CUDA_OK(launch_next(matrix_sum_kernel, dim3(ceil_div(n_train, 32)), dim3(1024), 0, st, list, n, n_val, n_train, first > 0 ? 1 : 0, total, vec,
                                                              ds->err_word, last ? err_out : nullptr));
    count_launch();
    const int rc = post_launch("matrix_sum_kernel");
    if (rc != GHOST_OK) return rc;
  }
  return GHOST_OK;
}
