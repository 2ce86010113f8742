// Similarity of projected gradients: S = scale * P1 P2^T for two blocks of projection rows
// [n, total_proj_dim] (Examples/ghost_gradproj_lm.py:190-196): a few rows, a very long contraction, bound by
// streaming both operands once.  The contraction is split over the CTAs of the grid, up to 64 x 64 scores per CTA.
//
// float operands are split into bf16 hi/lo parts in registers (hi*hi + lo*hi + hi*lo).
#include <cooperative_groups.h>

#include "common.cuh"
#include "mma_sync.cuh"
#include "sm100_ptx.cuh"

namespace cg = cooperative_groups;

namespace gb {

struct SimParams {
  const void* P1;   // [n1, D], row pitch ld1
  const void* P2;   // [n2, D], row pitch ld2
  int n1, n2;
  long long D, ld1, ld2;
  long long per_cta;       // 32-element steps (TMA: stages) of the contraction a CTA covers
  int direct;              // the cluster covers the whole contraction: its sums are the scores
  int vec_s;               // rows of S on 16-byte boundaries
  float scale;
  float* S;         // [n1, ld_s]
  long long ld_s;
  int* err;
};

// The end of a block, from its warps' partial sums part[WK][BM * BN] in shared memory.  The CTAs of a cluster (grid.x) add their
// blocks up through distributed shared memory before one of them touches the scores: with an addition per CTA and score
// the 1.2 million atomics of a 64 x 64 block over 296 CTAs were a quarter of a 20 us call.  A contraction that one cluster
// covers is stored without a zeroed result.
template <int WK, int BM, int BN, int THREADS>
__device__ __forceinline__ void sim_finish(float* part, const SimParams& p) {
  static_assert(BM * BN % 4 == 0 && BN % 4 == 0, "four scores a thread");
  __syncthreads();
  for (int e = threadIdx.x; e < BM * BN; e += THREADS) {
    float v = 0.f;
#pragma unroll
    for (int w = 0; w < WK; ++w) v += part[w * (BM * BN) + e];
    part[e] = v;
  }
  cg::cluster_group cluster = cg::this_cluster();
  const int ranks = static_cast<int>(cluster.num_blocks()), rank = static_cast<int>(cluster.block_rank());
  cluster.sync();
  // four neighbouring scores of a row a thread, dealt to the CTAs of the cluster
  for (int q = rank * THREADS + static_cast<int>(threadIdx.x); q < BM * BN / 4; q += ranks * THREADS) {
    float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll 4
    for (int r = 0; r < ranks; ++r) {
      const float4 x = *reinterpret_cast<const float4*>(cluster.map_shared_rank(&part[4 * q], r));
      v.x += x.x; v.y += x.y; v.z += x.z; v.w += x.w;
    }
    const int i = static_cast<int>(blockIdx.y) * BM + 4 * q / BN, j = static_cast<int>(blockIdx.z) * BN + 4 * q % BN;
    if (i >= p.n1) continue;
    float* dst = p.S + static_cast<long long>(i) * p.ld_s + j;
    const float out[4] = {p.scale * v.x, p.scale * v.y, p.scale * v.z, p.scale * v.w};
    if (p.vec_s && j + 4 <= p.n2) {
      if (p.direct) *reinterpret_cast<float4*>(dst) = make_float4(out[0], out[1], out[2], out[3]);
      else
        asm volatile("red.global.v4.f32.add [%0], {%1, %2, %3, %4};" ::"l"(dst), "f"(out[0]), "f"(out[1]), "f"(out[2]), "f"(out[3])
                     : "memory");
    } else {
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        if (j + e >= p.n2) continue;
        if (p.direct) dst[e] = out[e];
        else atomicAdd(dst + e, out[e]);
      }
    }
  }
  cluster.sync();            // no CTA leaves while another reads its block
}

// Eight consecutive contraction elements of one row: hi parts, and lo parts for float rows
template <typename PT, bool VEC> struct SimOct {
  float v[sizeof(PT) == 4 ? 8 : 1];
  uint4 raw;
  __device__ __forceinline__ void load(const PT* row, long long k, long long d, bool ok) {
    if constexpr (sizeof(PT) == 4) {
      if (VEC) {
        const bool in = ok && k < d;       // D % 8 == 0
        const float4 z = make_float4(0.f, 0.f, 0.f, 0.f);
        *reinterpret_cast<float4*>(&v[0]) = in ? *reinterpret_cast<const float4*>(row + k) : z;
        *reinterpret_cast<float4*>(&v[4]) = in ? *reinterpret_cast<const float4*>(row + k + 4) : z;
      } else {
#pragma unroll
        for (int e = 0; e < 8; ++e) v[e] = ok && k + e < d ? row[k + e] : 0.f;
      }
    } else {
      if (VEC) {
        raw = ok && k < d ? *reinterpret_cast<const uint4*>(row + k) : make_uint4(0u, 0u, 0u, 0u);
      } else {
        __nv_bfloat16 x[8];
#pragma unroll
        for (int e = 0; e < 8; ++e) x[e] = ok && k + e < d ? row[k + e] : __float2bfloat16_rn(0.f);
        raw = make_uint4(pack_bf16x2(x[0], x[1]), pack_bf16x2(x[2], x[3]), pack_bf16x2(x[4], x[5]), pack_bf16x2(x[6], x[7]));
      }
    }
  }
  __device__ __forceinline__ void parts(uint32_t (&hi)[4], uint32_t (&lo)[4]) const {
    if constexpr (sizeof(PT) == 4) {
#pragma unroll
      for (int h = 0; h < 4; ++h) {
        const __nv_bfloat16 x = __float2bfloat16_rn(v[2 * h]), y = __float2bfloat16_rn(v[2 * h + 1]);
        hi[h] = pack_bf16x2(x, y);
        lo[h] = pack_bf16x2(__float2bfloat16_rn(v[2 * h] - __bfloat162float(x)), __float2bfloat16_rn(v[2 * h + 1] - __bfloat162float(y)));
      }
    } else {
      hi[0] = raw.x; hi[1] = raw.y; hi[2] = raw.z; hi[3] = raw.w;
    }
  }
};

// A warp holds a (16 MT) x (8 NT) block of scores for every WK-th step of its CTA's range; WM x WN warps
// tile the CTA's block and WK of them split its range, so operand rows are fetched once per block of up
// to 64 x 64 scores (again from L2 / L1 for the next block and the neighbouring warps) instead of once
// per 16 x 16.  All loads of a 32-element step go out together.
template <typename PT, int MT, int NT, int WM, int WN, bool VEC>
__global__ void __launch_bounds__(256, 2) proj_similarity_kernel(const SimParams p) {
  constexpr int WK = 8 / (WM * WN);
  constexpr int BM = 16 * MT * WM, BN = 8 * NT * WN;
  constexpr bool kSplit = sizeof(PT) == 4;
  __shared__ __align__(16) float part[WK * BM * BN];
  stream_order();
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int g = lane >> 2, c = lane & 3;
  const int wk = warp / (WM * WN), wm = warp % (WM * WN) / WN, wn = warp % WN;
  const int i0 = blockIdx.y * BM + wm * 16 * MT, j0 = blockIdx.z * BN + wn * 8 * NT;
  const PT* A = static_cast<const PT*>(p.P1);
  const PT* B = static_cast<const PT*>(p.P2);
  const PT* ar[2 * MT];
  const PT* br[NT];
#pragma unroll
  for (int m = 0; m < 2 * MT; ++m) ar[m] = A + static_cast<long long>(min(i0 + 8 * m + g, p.n1 - 1)) * p.ld1;
#pragma unroll
  for (int n = 0; n < NT; ++n) br[n] = B + static_cast<long long>(min(j0 + 8 * n + g, p.n2 - 1)) * p.ld2;

  float acc[MT][NT][4];
#pragma unroll
  for (int m = 0; m < MT; ++m)
#pragma unroll
    for (int n = 0; n < NT; ++n)
#pragma unroll
      for (int e = 0; e < 4; ++e) acc[m][n][e] = 0.f;
  const long long s0 = blockIdx.x * p.per_cta, steps = (p.D + 31) / 32;
  const long long s1 = s0 + p.per_cta < steps ? s0 + p.per_cta : steps;
  const bool some = i0 < p.n1 && j0 < p.n2;            // a warp whose whole block lies outside idles
  // few rows per warp: several steps' loads in flight instead of one's
  constexpr int kUnroll = 2 * MT + NT <= 4 ? 4 : 2 * MT + NT <= 6 ? 2 : 1;
#pragma unroll kUnroll
  for (long long s = s0 + wk; some && s < s1; s += WK) {
    const long long k = s * 32 + 8 * c;
    SimOct<PT, VEC> a[2 * MT], b[NT];
#pragma unroll
    for (int m = 0; m < 2 * MT; ++m) a[m].load(ar[m], k, p.D, true);
#pragma unroll
    for (int n = 0; n < NT; ++n) b[n].load(br[n], k, p.D, true);
    uint32_t ah[2 * MT][4], al[2 * MT][4];
#pragma unroll
    for (int m = 0; m < 2 * MT; ++m) a[m].parts(ah[m], al[m]);
#pragma unroll
    for (int n = 0; n < NT; ++n) {
      uint32_t bh[4], bl[4];
      b[n].parts(bh, bl);
#pragma unroll
      for (int m = 0; m < MT; ++m) {
        // The tensor core's accumulator truncates, so it holds one step and the sum over the steps is made
        // here.  16 x 16 scores over 98304 elements: 7.8e-7 -> 4.2e-7 off the 64-bit result (float32), 2.5e-7 ->
        // 0.9e-7 (bf16); 64 x 64 over 2^20: 5.4e-6 -> 3.8e-7 and 149 -> 156 us (float32, bound by the
        // splitting of its operands), 1.8e-6 -> 2.4e-7 and 207 -> 82 us (bf16, was bound by the chain).
        float step[4];
        if constexpr (kSplit) {
          mma_16816_new(step, al[2 * m][0], al[2 * m + 1][0], al[2 * m][1], al[2 * m + 1][1], bh[0], bh[1]);
          mma_16816(step, ah[2 * m][0], ah[2 * m + 1][0], ah[2 * m][1], ah[2 * m + 1][1], bl[0], bl[1]);
          mma_16816(step, al[2 * m][2], al[2 * m + 1][2], al[2 * m][3], al[2 * m + 1][3], bh[2], bh[3]);
          mma_16816(step, ah[2 * m][2], ah[2 * m + 1][2], ah[2 * m][3], ah[2 * m + 1][3], bl[2], bl[3]);
          mma_16816(step, ah[2 * m][0], ah[2 * m + 1][0], ah[2 * m][1], ah[2 * m + 1][1], bh[0], bh[1]);
        } else {
          mma_16816_new(step, ah[2 * m][0], ah[2 * m + 1][0], ah[2 * m][1], ah[2 * m + 1][1], bh[0], bh[1]);
        }
        mma_16816(step, ah[2 * m][2], ah[2 * m + 1][2], ah[2 * m][3], ah[2 * m + 1][3], bh[2], bh[3]);
        add_fragment(acc[m][n], step);
      }
    }
  }
#pragma unroll
  for (int m = 0; m < MT; ++m)
#pragma unroll
    for (int n = 0; n < NT; ++n)
#pragma unroll
      for (int e = 0; e < 4; ++e)
        part[wk * (BM * BN) + (wm * 16 * MT + 16 * m + g + 8 * (e >> 1)) * BN + wn * 8 * NT + 8 * n + 2 * c + (e & 1)] = acc[m][n][e];
  sim_finish<WK, BM, BN, 256>(part, p);
}

// A stage holds PANELS panels of 128 bytes of columns of all rows of a block, each an [BM][128 bytes] and a [BN][128 bytes]
// block in the 128-byte swizzle; the stages fill what the partial sums leave of the shared memory.
template <typename PT, int MT, int NT, int WM, int WN>
struct SimCfg {
  static constexpr int WK = 8 / (WM * WN);                 // warps that split a stage's panels
  static constexpr int BM = 16 * MT * WM, BN = 8 * NT * WN;
  static constexpr int kPanelCols = 128 / static_cast<int>(sizeof(PT));
  static constexpr int PANELS = WK;
  static constexpr int kPanelBytes = (BM + BN) * 128;
  static constexpr int kStageBytes = PANELS * kPanelBytes;
  static constexpr int kRoom = (200 * 1024) / kStageBytes;
  static constexpr int kStages = kRoom < 8 ? kRoom : 8;
  static constexpr int kSmemBytes = kStages * kStageBytes + 1024 + 256;
  static constexpr int kThreads = 288;
  static_assert(WK * BM * BN * 4 <= kStages * kStageBytes, "the partial sums reuse the stages");
};

// Eight consecutive contraction elements of one row as hi parts, and lo parts for float rows
template <typename PT>
__device__ __forceinline__ void sim_parts(const uint8_t* row, int r, int c, int half, uint32_t (&hi)[4], uint32_t (&lo)[4]) {
  if constexpr (sizeof(PT) == 4) {
    float v[8];
    *reinterpret_cast<float4*>(&v[0]) = *reinterpret_cast<const float4*>(row + (((2 * c) ^ r) << 4));
    *reinterpret_cast<float4*>(&v[4]) = *reinterpret_cast<const float4*>(row + (((2 * c + 1) ^ r) << 4));
#pragma unroll
    for (int h = 0; h < 4; ++h) {
      const __nv_bfloat162 x = __floats2bfloat162_rn(v[2 * h], v[2 * h + 1]);
      const __nv_bfloat162 y = __floats2bfloat162_rn(v[2 * h] - __bfloat162float(x.x), v[2 * h + 1] - __bfloat162float(x.y));
      hi[h] = *reinterpret_cast<const uint32_t*>(&x);
      lo[h] = *reinterpret_cast<const uint32_t*>(&y);
    }
  } else {
    const uint4 w = *reinterpret_cast<const uint4*>(row + (((4 * half + c) ^ r) << 4));
    hi[0] = w.x; hi[1] = w.y; hi[2] = w.z; hi[3] = w.w;
  }
}

// The same for rows that TMA can read, once there are many bytes of them: eight warps work on stages that a ninth keeps coming,
// 200 KB of them on their way per SM, where the kernel above has what its registers hold in flight.  64 x 64 rows of 98304 float32:
// 24.2 us with fragments from global memory and an atomic per CTA and score, 18.8 here; of 2^20 bf16 75 and 59.
template <typename PT, int MT, int NT, int WM, int WN>
__global__ void __launch_bounds__(288, 1)
proj_similarity_tma_kernel(const __grid_constant__ CUtensorMap tm_a, const __grid_constant__ CUtensorMap tm_b, const SimParams p) {
  using Cfg = SimCfg<PT, MT, NT, WM, WN>;
  constexpr int WK = Cfg::WK, BM = Cfg::BM, BN = Cfg::BN, P = Cfg::PANELS, kStages = Cfg::kStages;
  constexpr bool kSplit = sizeof(PT) == 4;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  uint64_t* full_bar = reinterpret_cast<uint64_t*>(smem + kStages * Cfg::kStageBytes);
  uint64_t* empty_bar = full_bar + kStages;
  volatile int* abort_flag = reinterpret_cast<volatile int*>(empty_bar + kStages);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const long long panels = (p.D + Cfg::kPanelCols - 1) / Cfg::kPanelCols, stages = (panels + P - 1) / P;
  const long long q0 = blockIdx.x * p.per_cta;
  const long long q1 = q0 + p.per_cta < stages ? q0 + p.per_cta : stages;

  if (threadIdx.x == 0) {
    for (int s = 0; s < kStages; ++s) { mbar_init(&full_bar[s], 1); mbar_init(&empty_bar[s], 8); }
    *abort_flag = 0;
    fence_barrier_init();
  }
  if (warp == 8 && lane == 0) { tma_prefetch_desc(&tm_a); tma_prefetch_desc(&tm_b); }
  __syncthreads();
  stream_order();

  float acc[MT][NT][4];
  if (warp >= 8) {
    int stage = 0; uint32_t phase = 0;
    // a box per panel and operand, one lane each; columns and rows past the end read as zero
    for (long long q = q0; q < q1; ++q) {
      int w = 1;
      if (lane == 0) w = mbar_wait(&empty_bar[stage], phase ^ 1, abort_flag, p.err, 471) ? 1 : 0;
      w = __shfl_sync(0xffffffffu, w, 0);
      if (!w) break;
      if (lane == 0) mbar_arrive_expect_tx(&full_bar[stage], Cfg::kStageBytes);
      __syncwarp();
      if (lane < 2 * P) {
        const int pn = lane >> 1;
        const bool b = lane & 1;
        uint8_t* dst = smem + stage * Cfg::kStageBytes + pn * Cfg::kPanelBytes + (b ? BM * 128 : 0);
        tma_load_2d(dst, b ? &tm_b : &tm_a, &full_bar[stage], static_cast<int>(q * P + pn) * Cfg::kPanelCols,
                    b ? static_cast<int>(blockIdx.z) * BN : static_cast<int>(blockIdx.y) * BM);
      }
      if (++stage == kStages) { stage = 0; phase ^= 1; }
    }
  } else {
    const int g = lane >> 2, c = lane & 3;
    const int wk = warp / (WM * WN), wm = warp % (WM * WN) / WN, wn = warp % WN;
#pragma unroll
    for (int m = 0; m < MT; ++m)
#pragma unroll
      for (int n = 0; n < NT; ++n)
#pragma unroll
        for (int e = 0; e < 4; ++e) acc[m][n][e] = 0.f;
    int stage = 0; uint32_t phase = 0;
    for (long long q = q0; q < q1; ++q) {
      int ok = 1;
      if (lane == 0) ok = mbar_wait(&full_bar[stage], phase, abort_flag, p.err, 171) ? 1 : 0;
      ok = __shfl_sync(0xffffffffu, ok, 0);
      __syncwarp();                    // the shuffle carries the verdict; this orders the stage's bytes for all lanes
      if (!ok) break;
      const uint8_t* a = smem + stage * Cfg::kStageBytes + wk * Cfg::kPanelBytes + (wm * 16 * MT + g) * 128;
      const uint8_t* b = smem + stage * Cfg::kStageBytes + wk * Cfg::kPanelBytes + (BM + wn * 8 * NT + g) * 128;
#pragma unroll
      for (int half = 0; half < (kSplit ? 1 : 2); ++half) {
        uint32_t ah[2 * MT][4], al[2 * MT][4];
#pragma unroll
        for (int m = 0; m < 2 * MT; ++m) sim_parts<PT>(a + m * 1024, g, c, half, ah[m], al[m]);
#pragma unroll
        for (int n = 0; n < NT; ++n) {
          uint32_t bh[4], bl[4];
          sim_parts<PT>(b + n * 1024, g, c, half, bh, bl);
#pragma unroll
          for (int m = 0; m < MT; ++m) {
            // one step of 32 elements in the accumulator, as above
            float step[4];
            if constexpr (kSplit) {
              mma_16816_new(step, al[2 * m][0], al[2 * m + 1][0], al[2 * m][1], al[2 * m + 1][1], bh[0], bh[1]);
              mma_16816(step, ah[2 * m][0], ah[2 * m + 1][0], ah[2 * m][1], ah[2 * m + 1][1], bl[0], bl[1]);
              mma_16816(step, al[2 * m][2], al[2 * m + 1][2], al[2 * m][3], al[2 * m + 1][3], bh[2], bh[3]);
              mma_16816(step, ah[2 * m][2], ah[2 * m + 1][2], ah[2 * m][3], ah[2 * m + 1][3], bl[2], bl[3]);
              mma_16816(step, ah[2 * m][0], ah[2 * m + 1][0], ah[2 * m][1], ah[2 * m + 1][1], bh[0], bh[1]);
            } else {
              mma_16816_new(step, ah[2 * m][0], ah[2 * m + 1][0], ah[2 * m][1], ah[2 * m + 1][1], bh[0], bh[1]);
            }
            mma_16816(step, ah[2 * m][2], ah[2 * m + 1][2], ah[2 * m][3], ah[2 * m + 1][3], bh[2], bh[3]);
            add_fragment(acc[m][n], step);
          }
        }
      }
      __syncwarp();
      if (lane == 0) mbar_arrive(&empty_bar[stage]);     // this warp is done with the stage
      if (++stage == kStages) { stage = 0; phase ^= 1; }
    }
  }

  // the block's partial sums, where the stages were: all of them have been read
  __syncthreads();
  float* part = reinterpret_cast<float*>(smem);            // [WK][BM * BN]
  if (warp < 8) {
    const int g = lane >> 2, c = lane & 3;
    const int wk = warp / (WM * WN), wm = warp % (WM * WN) / WN, wn = warp % WN;
#pragma unroll
    for (int m = 0; m < MT; ++m)
#pragma unroll
      for (int n = 0; n < NT; ++n)
#pragma unroll
        for (int e = 0; e < 4; ++e)
          part[wk * (BM * BN) + (wm * 16 * MT + 16 * m + g + 8 * (e >> 1)) * BN + wn * 8 * NT + 8 * n + 2 * c + (e & 1)] = acc[m][n][e];
  }
  sim_finish<WK, BM, BN, Cfg::kThreads>(part, p);
}

// Grid and cluster of a call: `most` is the largest number of splits worth making of the contraction
struct SimGrid { long long splits; int ranks; };
static SimGrid sim_grid(SimParams& p, int bi, int bj, long long slots, long long most, long long units) {
  long long splits = slots / (static_cast<long long>(bi) * bj);
  if (splits > most) splits = most;
  if (splits < 1) splits = 1;
  // Up to eight splits are one cluster.  Beyond that two to a cluster: GPCs have 18 or 20 SMs, which larger ones do not fill,
  // and the clusters left over take a second round (64 x 64 x 2^20 float32, clusters of four: 222 us, 132 in pairs).
  int ranks = 1;
  if (splits <= 8) { while (ranks < splits) ranks *= 2; }
  else ranks = 2;
  splits = splits <= 8 ? ranks : splits / ranks * ranks;
  p.per_cta = (units + splits - 1) / splits;
  p.direct = splits == ranks;
  p.vec_s = p.ld_s % 4 == 0 && (reinterpret_cast<uintptr_t>(p.S) & 15u) == 0;
  return {splits, ranks};
}

template <typename K, typename... A>
static int sim_launch(K kernel, const SimParams& p, SimGrid g, int bi, int bj, int threads, size_t smem, cudaStream_t st, const A&... args) {
  if (!p.direct)
    GB_CUDA_OK(cudaMemset2DAsync(p.S, static_cast<size_t>(p.ld_s) * 4, 0, static_cast<size_t>(p.n2) * 4, static_cast<size_t>(p.n1), st));
  cudaLaunchConfig_t cfg = {};
  cudaLaunchAttribute attr[2];
  cfg.gridDim = dim3(static_cast<unsigned>(g.splits), static_cast<unsigned>(bi), static_cast<unsigned>(bj));
  cfg.blockDim = dim3(threads, 1, 1);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = st;
  cfg.attrs = attr;
  cfg.numAttrs = early_start(attr, st);
  if (g.ranks > 1) {
    cudaLaunchAttribute& cluster = attr[cfg.numAttrs++];
    cluster.id = cudaLaunchAttributeClusterDimension;
    cluster.val.clusterDim.x = g.ranks;
    cluster.val.clusterDim.y = 1;
    cluster.val.clusterDim.z = 1;
  }
  GB_CUDA_OK(cudaLaunchKernelEx(&cfg, kernel, args...));
  count_launch();
  return post_launch("proj_similarity_kernel");
}

template <typename PT, int MT, int NT, int WM, int WN>
static int launch_similarity(SimParams p, bool vec, const DeviceState* ds, cudaStream_t st) {
  using Cfg = SimCfg<PT, MT, NT, WM, WN>;
  const int bi = ceil_div(p.n1, Cfg::BM), bj = ceil_div(p.n2, Cfg::BN);
  GB_REQUIRE(bi <= 65535 && bj <= 65535, "ghost_projection_similarity: too many rows");
  // Below 16 MB a call is launch, ramp and reduction, and the fragments' kernel is ahead (97 x 8 rows of 9104 bf16: 9.5 us in the
  // ring, 6 there); TMA also wants box coordinates that are ints.
  if (vec && (static_cast<double>(p.n1) + p.n2) * p.D * sizeof(PT) >= 16e6 && p.D < (1ll << 31) - 4096) {
    CUtensorMap ta, tb;
    int rc;
    if ((rc = make_tmap_rows(&ta, p.P1, sizeof(PT), p.n1, p.D, p.ld1, Cfg::BM)) != GHOST_OK) return rc;
    if ((rc = make_tmap_rows(&tb, p.P2, sizeof(PT), p.n2, p.D, p.ld2, Cfg::BN)) != GHOST_OK) return rc;
    static bool attr_set[64] = {};
    if (!attr_set[ds->device]) {
      GB_CUDA_OK(cudaFuncSetAttribute(proj_similarity_tma_kernel<PT, MT, NT, WM, WN>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                      Cfg::kSmemBytes));
      attr_set[ds->device] = true;
    }
    // one CTA per SM, two stages each at least
    const long long stages = (p.D + Cfg::PANELS * Cfg::kPanelCols - 1) / (Cfg::PANELS * Cfg::kPanelCols);
    const SimGrid g = sim_grid(p, bi, bj, ds->sm_count, (stages + 1) / 2, stages);
    return sim_launch(proj_similarity_tma_kernel<PT, MT, NT, WM, WN>, p, g, bi, bj, Cfg::kThreads, Cfg::kSmemBytes, st, ta, tb, p);
  }
  // one wave of two CTAs per SM, but at least eight steps for each of a CTA's WK warps of a block
  const long long steps = (p.D + 31) / 32, least = 8 * Cfg::WK;
  const SimGrid g = sim_grid(p, bi, bj, 2ll * ds->sm_count, (steps + least - 1) / least, steps);
  if (vec) return sim_launch(proj_similarity_kernel<PT, MT, NT, WM, WN, true>, p, g, bi, bj, 256, 0, st, p);
  return sim_launch(proj_similarity_kernel<PT, MT, NT, WM, WN, false>, p, g, bi, bj, 256, 0, st, p);
}

// Block shape with the least time per 32-element step over all blocks, in cycles of an SM: what the rows take to arrive
// (24 bytes a cycle) or the instructions of its warps (three per row and lane to split float32, six or two products
// per 16 x 8 scores), whichever is more.  One 64 x 64 block for everything beyond 16 rows padded 18 x 74 rows to 64 x 128
// (710864 floats: 177 us).
template <typename PT>
static int dispatch_similarity(const SimParams& p, bool vec, const DeviceState* ds, cudaStream_t st) {
  constexpr double kSplitCost = sizeof(PT) == 4 ? 3.5 : 0.5, kProducts = sizeof(PT) == 4 ? 48. : 16.;
  struct Shape { int mt, nt, wm, wn; };
  static constexpr Shape shapes[] = {{1, 1, 1, 1}, {1, 2, 1, 1}, {1, 4, 1, 2}, {2, 4, 1, 1}, {2, 4, 1, 2}, {2, 2, 2, 1}, {2, 4, 2, 2}};
  int best = -1;
  double least = 0.;
  for (int i = 0; i < 7; ++i) {
    const Shape& s = shapes[i];
    const double bi = ceil_div(p.n1, 16 * s.mt * s.wm), bj = ceil_div(p.n2, 8 * s.nt * s.wn);
    if (bi > 65535 || bj > 65535) continue;                  // no grid of such blocks
    const double arrive = (bj * p.n1 + bi * p.n2) * 32. * sizeof(PT) / 24.;
    const double work = bi * bj * s.wm * s.wn * (kSplitCost * (16 * s.mt + 8 * s.nt) + kProducts * s.mt * s.nt) * 1.3 / 4.;
    const double cost = arrive > work ? arrive : work;
    if (best < 0 || cost < least) { least = cost; best = i; }
  }
  switch (best) {
    case 0: return launch_similarity<PT, 1, 1, 1, 1>(p, vec, ds, st);
    case 1: return launch_similarity<PT, 1, 2, 1, 1>(p, vec, ds, st);
    case 2: return launch_similarity<PT, 1, 4, 1, 2>(p, vec, ds, st);
    case 3: return launch_similarity<PT, 2, 4, 1, 1>(p, vec, ds, st);
    case 4: return launch_similarity<PT, 2, 4, 1, 2>(p, vec, ds, st);
    case 5: return launch_similarity<PT, 2, 2, 2, 1>(p, vec, ds, st);
    default: return launch_similarity<PT, 2, 4, 2, 2>(p, vec, ds, st);
  }
}

}  // namespace gb

using namespace gb;

extern "C" int ghost_projection_similarity(const void* P1, const void* P2, int is_f32, int n1, int n2, long long D,
                                           long long ld1, long long ld2, float scale, float* S, long long ld_s,
                                           void* stream) {
  const DeviceState* ds = device_state();
  if (!ds) return GHOST_ERR_DEVICE;
  GB_REQUIRE(P1 && P2 && S, "ghost_projection_similarity: null pointer");
  GB_REQUIRE(n1 > 0 && n2 > 0 && D > 0, "ghost_projection_similarity: empty dimension");
  GB_REQUIRE(ld1 >= D && ld2 >= D && ld_s >= n2, "ghost_projection_similarity: pitch smaller than the row it holds");
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  SimParams p = {};
  p.P1 = P1; p.P2 = P2; p.n1 = n1; p.n2 = n2; p.D = D; p.ld1 = ld1; p.ld2 = ld2; p.scale = scale; p.S = S;
  p.ld_s = ld_s;
  const int esize = is_f32 ? 4 : 2;
  p.err = ds->err_word;
  const bool vec = D % 8 == 0 && (ld1 * esize) % 16 == 0 && (ld2 * esize) % 16 == 0 &&
                   ((reinterpret_cast<uintptr_t>(P1) | reinterpret_cast<uintptr_t>(P2)) & 15u) == 0;
  return is_f32 ? dispatch_similarity<float>(p, vec, ds, st) : dispatch_similarity<__nv_bfloat16>(p, vec, ds, st);
}
