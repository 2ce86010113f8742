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

// The end of a block, from its warps' partial sums part[WK][BM * BN] in shared memory: added to zeroed scores, or stored where no
// other CTA has a share.  kCluster: the CTAs of a cluster (grid.x) cover the contraction and add their blocks up through distributed
// shared memory first.  A form of its own: with the cluster's code in the other one its main loops came out slower as well (37 x 43
// unaligned rows of 927511 float32: 142 us, 132 without).
//
// A thread takes four neighbouring scores of a row where rows of S start on 16-byte boundaries, else one, so that a warp's additions
// cover neighbouring scores either way (four there as well: 4 x 59 rows of 522904 float32 38 us, 31 one by one).
template <int WK, int BM, int BN, int THREADS, bool kCluster>
__device__ __forceinline__ void sim_finish(float* part, const SimParams& p) {
  static_assert(BN % 4 == 0, "four scores a thread");
  __syncthreads();
  const int rows = p.n1 - static_cast<int>(blockIdx.y) * BM, cols = p.n2 - static_cast<int>(blockIdx.z) * BN;      // of this block
  auto at = [&](int e) {
    return p.S + static_cast<long long>(static_cast<int>(blockIdx.y) * BM + e / BN) * p.ld_s + static_cast<int>(blockIdx.z) * BN + e % BN;
  };
  auto out4 = [&](int e, float4 v) {
    v.x *= p.scale; v.y *= p.scale; v.z *= p.scale; v.w *= p.scale;
    if (p.direct) *reinterpret_cast<float4*>(at(e)) = v;
    else asm volatile("red.global.v4.f32.add [%0], {%1, %2, %3, %4};" ::"l"(at(e)), "f"(v.x), "f"(v.y), "f"(v.z), "f"(v.w) : "memory");
  };
  auto out1 = [&](int e, float v) {
    if (p.direct) *at(e) = p.scale * v;
    else atomicAdd(at(e), p.scale * v);
  };
  auto inside = [&](int e) { return e / BN < rows && e % BN < cols; };
  if constexpr (kCluster) {
    for (int e = threadIdx.x; e < BM * BN; e += THREADS) {
      float v = 0.f;
#pragma unroll
      for (int w = 0; w < WK; ++w) v += part[w * (BM * BN) + e];
      part[e] = v;
    }
    cg::cluster_group cluster = cg::this_cluster();
    const int ranks = static_cast<int>(cluster.num_blocks()), rank = static_cast<int>(cluster.block_rank());
    cluster.sync();
    if (p.vec_s) {
      for (int e = 4 * (rank * THREADS + static_cast<int>(threadIdx.x)); e < BM * BN; e += 4 * ranks * THREADS) {
        if (!inside(e)) continue;
        float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll 4
        for (int r = 0; r < ranks; ++r) {
          const float4 x = *reinterpret_cast<const float4*>(cluster.map_shared_rank(&part[e], r));
          v.x += x.x; v.y += x.y; v.z += x.z; v.w += x.w;
        }
        out4(e, v);
      }
    } else {
      for (int e = rank * THREADS + static_cast<int>(threadIdx.x); e < BM * BN; e += ranks * THREADS) {
        if (!inside(e)) continue;
        float v = 0.f;
#pragma unroll 4
        for (int r = 0; r < ranks; ++r) v += *cluster.map_shared_rank(&part[e], r);
        out1(e, v);
      }
    }
    cluster.sync();          // no CTA leaves while another reads its block
  } else if (p.vec_s) {
    for (int e = 4 * static_cast<int>(threadIdx.x); e < BM * BN; e += 4 * THREADS) {
      if (!inside(e)) continue;
      float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
      for (int w = 0; w < WK; ++w) {
        const float4 x = *reinterpret_cast<const float4*>(&part[w * (BM * BN) + e]);
        v.x += x.x; v.y += x.y; v.z += x.z; v.w += x.w;
      }
      out4(e, v);
    }
  } else {
    for (int e = threadIdx.x; e < BM * BN; e += THREADS) {
      if (!inside(e)) continue;
      float v = 0.f;
#pragma unroll
      for (int w = 0; w < WK; ++w) v += part[w * (BM * BN) + e];
      out1(e, v);
    }
  }
}

// Eight consecutive contraction elements of one row: hi parts, and lo parts for float rows.  Elements one by one (not VEC) go
// through the read-only path, which leaves their order to the compiler (97 x 127 rows of 814571 float32: 870 us with ordinary loads, 718
// so): that form is not launched early, and nobody writes its rows while it lives.
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
        for (int e = 0; e < 8; ++e) v[e] = ok && k + e < d ? __ldg(row + k + e) : 0.f;
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
template <typename PT, int MT, int NT, int WM, int WN, bool VEC, bool kCluster>
__global__ void __launch_bounds__(256, 2) proj_similarity_kernel(const SimParams p) {
  constexpr int WK = 8 / (WM * WN);
  constexpr int BM = 16 * MT * WM, BN = 8 * NT * WN;
  constexpr bool kSplit = sizeof(PT) == 4;
  __shared__ __align__(16) float part[WK * BM * BN];
  if constexpr (VEC) stream_order();
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
        // here.  16 x 16 scores of positive rows over 98304 elements: 7.8e-7 -> 4.2e-7 off the 64-bit result (float32), 2.5e-7 ->
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
  sim_finish<WK, BM, BN, 256, kCluster>(part, p);
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
// 200 KB of them on their way per SM, where the kernel above has what its registers hold in flight (times of both: dispatch_similarity).
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
  sim_finish<WK, BM, BN, Cfg::kThreads, false>(part, p);
}

// Warps and blocks of a form of the kernels (their template arguments)
struct SimShape {
  int mt, nt, wm, wn;
  int bm() const { return 16 * mt * wm; }
  int bn() const { return 8 * nt * wn; }
  int wk() const { return 8 / (wm * wn); }
};

// How a call is spread: `splits` CTAs for each of the bi x bj blocks, in clusters of `ranks`
struct SimGrid {
  SimShape shape;
  long long bi, bj, splits, per_cta;     // per_cta: steps (ring: stages) of the contraction
  int ranks;
  bool direct;                           // one cluster covers the contraction: no zeroed result, no additions to it
  bool clear_ahead;                      // the zeros come from a kernel, not from a memset
  double cost;
};

// In a cluster up to eight splits are all of them and their sums the scores (5 x 6 rows of 688 float32 6.2 us with a zeroed result,
// 4.3 without); else each adds to the scores by itself.  More than eight in clusters of two halve those additions, but
// their barriers cost every small call 2 us (9 x 3 rows of 215550 bf16: 10.3 us, 8.3 without), and larger clusters leave SMs idle.
static SimGrid sim_grid(const SimParams& p, const SimShape& s, long long slots, long long units, long long least, bool cluster) {
  SimGrid g = {s, (p.n1 + s.bm() - 1ll) / s.bm(), (p.n2 + s.bn() - 1ll) / s.bn()};
  const long long blocks = g.bi * g.bj, most = (units + least - 1) / least;
  g.splits = slots / blocks < most ? slots / blocks : most;
  if (g.splits < 1) g.splits = 1;
  g.ranks = 1;
  if (cluster) {
    while (g.ranks < g.splits && g.ranks < 8) g.ranks *= 2;
    g.splits = g.ranks;
  }
  g.direct = g.splits == g.ranks;
  g.per_cta = (units + g.splits - 1) / g.splits;
  return g;
}

// What tells the shapes apart, in arbitrary units: rounds of a warp one after the other, each the latency of its loads; what the
// warps of an SM issue in a round (products of a warp's 16 x 8 blocks, loads, eight for one where rows are off vector boundaries); the
// rows that arrive, once per block that needs them; additions to a zeroed result.  In the ring the rows arrive beside the
// work on them.  The constants are fits to all seven shapes at 330 sizes (rows 1 to 128, 256 to 2^20 elements, both types, aligned
// and not): the shape with the least sum is within 2 % of the best one in the mean.
static double sim_cost(const SimParams& p, const SimGrid& g, int esize, bool vec, bool ring, int sms) {
  const SimShape& s = g.shape;
  const double products = (esize == 4 ? 48. : 16.) * s.mt * s.nt;
  const double arrive = (static_cast<double>(g.bj) * p.n1 + static_cast<double>(g.bi) * p.n2) * p.D * esize * 1e-6;
  const double ctas = static_cast<double>(g.bi) * g.bj * g.splits;
  if (ring) {
    const double stages = g.per_cta * (ctas > sms ? ctas / sms : 1.), stage = (s.bm() + s.bn()) * 128. * s.wk();
    const double work = stages * (0.66 + 1.0e-3 * products * (esize == 4 ? 1 : 2) + 2.1e-6 * stage);
    return work > 0.22 * arrive ? work : 0.22 * arrive;
  }
  const double rounds = static_cast<double>((g.per_cta + s.wk() - 1) / s.wk()) * (ctas > 2. * sms ? ctas / (2. * sms) : 1.);
  const double loads = (16. * s.mt + 8. * s.nt) * (vec ? 4.2e-4 * esize / 16. : 1.0e-2);
  return (g.direct ? 0. : 0.91) + rounds * (0.26 + (ctas > sms ? 2. : 1.) * (8.7e-4 * products + loads)) + 8.3e-3 * arrive;
}

template <typename K, typename... A>
static int sim_launch(K kernel, bool early, const SimParams& p, const SimGrid& g, int threads, size_t smem, cudaStream_t st, const A&... args) {
  if (!p.direct && g.clear_ahead && p.ld_s == p.n2) {
    if (int rc = clear_ahead(p.S, sizeof(float) * static_cast<size_t>(p.n1) * p.n2, st)) return rc;
  } else if (!p.direct) {
    GB_CUDA_OK(cudaMemset2DAsync(p.S, static_cast<size_t>(p.ld_s) * 4, 0, static_cast<size_t>(p.n2) * 4, static_cast<size_t>(p.n1), st));
  }
  cudaLaunchConfig_t cfg = {};
  cudaLaunchAttribute attr[2];
  cfg.gridDim = dim3(static_cast<unsigned>(g.splits), static_cast<unsigned>(g.bi), static_cast<unsigned>(g.bj));
  cfg.blockDim = dim3(threads, 1, 1);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = st;
  cfg.attrs = attr;
  cfg.numAttrs = early ? early_start(attr, st) : 0;
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
static int launch_similarity(SimParams p, const SimGrid& g, bool vec, bool ring, const DeviceState* ds, cudaStream_t st) {
  using Cfg = SimCfg<PT, MT, NT, WM, WN>;
  p.per_cta = g.per_cta;
  p.direct = g.direct;
  p.vec_s = p.n2 % 4 == 0 && p.ld_s % 4 == 0 && (reinterpret_cast<uintptr_t>(p.S) & 15u) == 0;
  if (ring) {
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
    return sim_launch(proj_similarity_tma_kernel<PT, MT, NT, WM, WN>, true, p, g, Cfg::kThreads, Cfg::kSmemBytes, st, ta, tb, p);
  }
  if (g.ranks > 1) {
    if (vec) return sim_launch(proj_similarity_kernel<PT, MT, NT, WM, WN, true, true>, true, p, g, 256, 0, st, p);
    return sim_launch(proj_similarity_kernel<PT, MT, NT, WM, WN, false, true>, false, p, g, 256, 0, st, p);
  }
  if (vec) return sim_launch(proj_similarity_kernel<PT, MT, NT, WM, WN, true, false>, true, p, g, 256, 0, st, p);
  return sim_launch(proj_similarity_kernel<PT, MT, NT, WM, WN, false, false>, false, p, g, 256, 0, st, p);
}

// The ring takes aligned rows once there are 16 MB of them, of bf16 128, and more than 16 on either side (TMA also wants box
// coordinates that are ints).  Below that a call is launch, ramp and reduction, and with few rows on one side its stages are mostly
// rows that are not there and its eight warps the bound, where sixteen work on fragments.  In the ring and as fragments, us: float32
// 32 x 32 rows of 98304 12.5 and 20.5, 128 x 128 48 and 74, 64 x 64 of 2^20 133 and 195, 1 x 98 of 895136 117 and 84; bf16 76 x 59
// of 418048 47 and 43, 64 x 64 of 2^20 57 and 77.
template <typename PT>
static int dispatch_similarity(const SimParams& p, bool vec, const DeviceState* ds, cudaStream_t st) {
  static constexpr SimShape shapes[] = {{1, 1, 1, 1}, {1, 2, 1, 1}, {1, 4, 1, 2}, {2, 4, 1, 1}, {2, 4, 1, 2}, {2, 2, 2, 1}, {2, 4, 2, 2}};
  const double bytes = (static_cast<double>(p.n1) + p.n2) * p.D * sizeof(PT);
  const bool ring = vec && p.n1 > 16 && p.n2 > 16 && bytes >= (sizeof(PT) == 4 ? 16e6 : 128e6) && p.D < (1ll << 31) - 4096;
  int best = -1;
  SimGrid grid = {};
  for (int i = 0; i < 14; ++i) {
    const SimShape& s = shapes[i / 2];
    const bool cluster = i % 2 == 0;
    if (ring && cluster) continue;
    constexpr int kPanelCols = 128 / static_cast<int>(sizeof(PT));
    // one CTA per SM of two stages at least, or two CTAs of four steps for each of their warps of a block
    const long long panels = (p.D + kPanelCols - 1) / kPanelCols;
    SimGrid g = ring ? sim_grid(p, s, ds->sm_count, (panels + s.wk() - 1) / s.wk(), 2, false)
                     : sim_grid(p, s, 2ll * ds->sm_count, (p.D + 31) / 32, 4 * s.wk(), cluster);
    if (g.bi > 65535 || g.bj > 65535) continue;              // no grid of such blocks
    g.cost = sim_cost(p, g, sizeof(PT), vec, ring, ds->sm_count);
    if (best < 0 || g.cost < grid.cost) { grid = g; best = i / 2; }
  }
  // A kernel's zeros hide behind the call ahead and cost the host a launch, which a call that comes alone waits for.  Back to back with
  // a memset and with the kernel, and the same alone, us: float32 23 x 17 rows of 300000 16.4 and 13.0, 24.0 and 25.4; 32 x 32 of 98304 10.3
  // and 7.5, 18.4 and 19.8; 64 x 64 16.5 and 15.2, 27.2 and 31; 40 x 40 of 50000 12.4 and 10.0, 22.0 and 22.2; bf16 3 x 57 of
  // 200000 8.7 and 7.3, 17.4 and 18.5.  Below 16 MB it gives no more than it costs: float32 16 x 16 of 98304 8.2 and 7.4, 15.6 and
  // 16.5; 64 x 8 of 50000 8.2 and 7.4, 16.0 and 17.1; bf16 7 x 28 of 153620 10.3 and 10.3, 19.4 and 20.9.
  grid.clear_ahead = bytes >= 16e6;
  switch (best) {
    case 0: return launch_similarity<PT, 1, 1, 1, 1>(p, grid, vec, ring, ds, st);
    case 1: return launch_similarity<PT, 1, 2, 1, 1>(p, grid, vec, ring, ds, st);
    case 2: return launch_similarity<PT, 1, 4, 1, 2>(p, grid, vec, ring, ds, st);
    case 3: return launch_similarity<PT, 2, 4, 1, 1>(p, grid, vec, ring, ds, st);
    case 4: return launch_similarity<PT, 2, 4, 1, 2>(p, grid, vec, ring, ds, st);
    case 5: return launch_similarity<PT, 2, 2, 2, 1>(p, grid, vec, ring, ds, st);
    case 6: return launch_similarity<PT, 2, 4, 2, 2>(p, grid, vec, ring, ds, st);
    default: return fail(GHOST_ERR_INVALID, "ghost_projection_similarity: too many rows");
  }
}

// One bf16 row against many: exact products, float32 sums that are kept apart by lane and element and added up over lanes, warps and
// CTAs in a fixed order.  The tensor core's sums truncate, and where there is one row to share out its chains are long: 1 x 200 rows of
// 512 came out 5.8e-8 off the 64-bit scores (float32 GEMM of the library: 4.3e-8, here 4.3e-8), of 65536 1.3e-7 (6.7e-8, 4.6e-8).
// A warp has four rows, so that the one row's elements are loaded once for four products, and eight loads of theirs are in flight.
// Bound by streaming the rows (1 x 512 of 262144 5.8 TB/s); unaligned ones by their element loads.
struct SimRow {
  const __nv_bfloat16 *one, *many;       // [D], [n, D] with row pitch ld
  int n, warps, ranks;     // warps of a CTA and CTAs of a cluster that share four rows
  long long D, ld;
  float scale;
  float* S;                // score i at S + i * step
  long long step;
};

// Sum of the first n of eight values, n a power of two, in pairs of pairs
template <typename F> __device__ __forceinline__ float row_sum8(int n, F&& v) {
  float x[8];
#pragma unroll
  for (int i = 0; i < 8; ++i) {
    x[i] = 0.f;
    if (i < n) x[i] = v(i);
  }
  return ((x[0] + x[1]) + (x[2] + x[3])) + ((x[4] + x[5]) + (x[6] + x[7]));
}

template <bool VEC>
__global__ void __launch_bounds__(256, 2) proj_row_kernel(const SimRow q) {
  stream_order();
  __shared__ float part[8][4];
  __shared__ float total[4];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int rank = static_cast<int>(blockIdx.x) % q.ranks;
  const long long row0 = 4 * (static_cast<long long>(blockIdx.x / q.ranks) * (8 / q.warps) + warp / q.warps);
  const int share = rank * q.warps + warp % q.warps, shares = q.ranks * q.warps;
  float acc[4][8];
#pragma unroll
  for (int r = 0; r < 4; ++r)
#pragma unroll
    for (int e = 0; e < 8; ++e) acc[r][e] = 0.f;
  if (row0 < q.n) {
    const __nv_bfloat16* y[4];
#pragma unroll
    for (int r = 0; r < 4; ++r) y[r] = q.many + (row0 + r < q.n ? row0 + r : q.n - 1) * q.ld;
    if constexpr (VEC) {                 // D is a multiple of eight
      const long long step = shares * 256ll;
      for (long long k0 = (share * 32 + lane) * 8; k0 < q.D; k0 += 2 * step) {
        uint4 a[2], b[2][4];
#pragma unroll
        for (int i = 0; i < 2; ++i) {
          const long long k = k0 + i * step;
          const bool in = k < q.D;
          a[i] = make_uint4(0u, 0u, 0u, 0u);
          if (in) a[i] = *reinterpret_cast<const uint4*>(q.one + k);
#pragma unroll
          for (int r = 0; r < 4; ++r) {
            b[i][r] = make_uint4(0u, 0u, 0u, 0u);
            if (in) b[i][r] = *reinterpret_cast<const uint4*>(y[r] + k);
          }
        }
#pragma unroll
        for (int i = 0; i < 2; ++i)
#pragma unroll
          for (int r = 0; r < 4; ++r) {
            const uint32_t u[4] = {a[i].x, a[i].y, a[i].z, a[i].w}, v[4] = {b[i][r].x, b[i][r].y, b[i][r].z, b[i][r].w};
#pragma unroll
            for (int e = 0; e < 4; ++e) {
              acc[r][2 * e] = fmaf(__uint_as_float(u[e] << 16), __uint_as_float(v[e] << 16), acc[r][2 * e]);
              acc[r][2 * e + 1] = fmaf(__uint_as_float(u[e] & 0xffff0000u), __uint_as_float(v[e] & 0xffff0000u), acc[r][2 * e + 1]);
            }
          }
      }
    } else {                             // rows that begin anywhere: element by element
      auto bits = [](const __nv_bfloat16* at) { return static_cast<uint32_t>(*reinterpret_cast<const unsigned short*>(at)) << 16; };
      const long long step = shares * 32ll;
      for (long long k0 = share * 32 + lane; k0 < q.D; k0 += 8 * step) {
        uint32_t a[8], b[8][4];
#pragma unroll
        for (int i = 0; i < 8; ++i) {
          const long long k = k0 + i * step;
          const bool in = k < q.D;
          a[i] = 0u;
          if (in) a[i] = bits(q.one + k);
#pragma unroll
          for (int r = 0; r < 4; ++r) {
            b[i][r] = 0u;
            if (in) b[i][r] = bits(y[r] + k);
          }
        }
#pragma unroll
        for (int i = 0; i < 8; ++i)
#pragma unroll
          for (int r = 0; r < 4; ++r) acc[r][i] = fmaf(__uint_as_float(a[i]), __uint_as_float(b[i][r]), acc[r][i]);
      }
    }
  }
  float sum = 0.f;                       // lanes 0 to 3: of row0 + lane
#pragma unroll
  for (int r = 0; r < 4; ++r) {
    float v = ((acc[r][0] + acc[r][1]) + (acc[r][2] + acc[r][3])) + ((acc[r][4] + acc[r][5]) + (acc[r][6] + acc[r][7]));
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    if (lane == r) sum = v;
  }
  if (q.warps > 1) {
    if (lane < 4) part[warp][lane] = sum;
    __syncthreads();
    if (lane < 4) sum = row_sum8(q.warps, [&](int w) { return part[warp / q.warps * q.warps + w][lane]; });
  }
  if (q.ranks > 1) {                     // the CTA's warps share the same rows
    if (threadIdx.x < 4) total[lane] = sum;
    cluster_sync_all();
    if (rank == 0 && threadIdx.x < 4) sum = row_sum8(q.ranks, [&](int r) { return ld_cluster_f32(map_to_cta(smem_u32(&total[lane]), r)); });
    cluster_sync_all();                  // no CTA leaves while another reads its sums
  }
  if (rank == 0 && warp % q.warps == 0 && lane < 4 && row0 + lane < q.n) q.S[(row0 + lane) * q.step] = sum * q.scale;
}

// Warps that share four rows, in CTAs of eight: as many as two CTAs an SM hold while a lane has a piece of eight elements.
static int launch_row(SimRow q, bool vec, const DeviceState* ds, cudaStream_t st) {
  const long long fours = (q.n + 3ll) / 4;
  int shares = 1;
  while (shares < 64 && 2 * shares * fours <= 16ll * ds->sm_count && 2ll * shares * 256 <= q.D) shares *= 2;
  q.warps = shares < 8 ? shares : 8;
  q.ranks = shares / q.warps;
  const int per_cta = 8 / q.warps;
  const unsigned grid = static_cast<unsigned>((fours + per_cta - 1) / per_cta) * q.ranks;
  if (vec) GB_CUDA_OK(launch_next_cluster(dim3(q.ranks), proj_row_kernel<true>, dim3(grid), dim3(256), 0, st, q));
  else GB_CUDA_OK(launch_next_cluster(dim3(q.ranks), proj_row_kernel<false>, dim3(grid), dim3(256), 0, st, q));
  count_launch();
  return post_launch("proj_row_kernel");
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
  // Longer sets against one row, which callers would else send to a float32 product (us, this kernel and the ones below: 1 x 129 rows of 2048
  // 2.4 and 3.6, 1 x 512 of 262144 45.9 and 59.6, 1 x 200 of 1711 4.3 and 6.3; 1 x 200 of 128 2.1 and 1.7, 1 x 65536 of it 12.3 and 6.8).
  if (!is_f32 && (n1 == 1 || n2 == 1) && (n1 > 128 || n2 > 128) && D >= 96) {
    SimRow q = {};
    q.one = static_cast<const __nv_bfloat16*>(n1 == 1 ? P1 : P2);
    q.many = static_cast<const __nv_bfloat16*>(n1 == 1 ? P2 : P1);
    q.n = n1 == 1 ? n2 : n1;
    q.ld = n1 == 1 ? ld2 : ld1;
    q.step = n1 == 1 ? 1 : ld_s;
    q.D = D; q.scale = scale; q.S = S;
    return launch_row(q, vec, ds, st);
  }
  return is_f32 ? dispatch_similarity<float>(p, vec, ds, st) : dispatch_similarity<__nv_bfloat16>(p, vec, ds, st);
}
