// Similarity of projected gradients: S = scale * P1 P2^T for two blocks of projection rows
// [n, total_proj_dim] (Examples/ghost_gradproj_lm.py:190-196): a few rows, a very long
// contraction, bound by streaming both operands once.  The contraction is split over all
// warps of the grid, up to 64 x 64 outputs per CTA, partial sums added with atomics.
//
// float operands are split into bf16 hi/lo parts in registers (hi*hi + lo*hi + hi*lo).
#include "common.cuh"
#include "mma_sync.cuh"

namespace gb {

// ------------------------------------------------------------------------------------------------
// similarity of projection rows
// ------------------------------------------------------------------------------------------------
struct SimParams {
  const void* P1;   // [n1, D], row pitch ld1
  const void* P2;   // [n2, D], row pitch ld2
  int n1, n2;
  long long D, ld1, ld2;
  long long per_cta;       // 32-element steps of the contraction a CTA covers
  float scale;
  float* S;         // [n1, ld_s]
  long long ld_s;
};

// Eight consecutive contraction elements of one row: hi parts, and lo parts for float rows
template <typename PT, bool VEC> struct SimOct {
  float v[sizeof(PT) == 4 ? 8 : 1];
  uint4 raw;
  __device__ __forceinline__ void load(const PT* row, long long k, long long d, bool ok) {
    if constexpr (sizeof(PT) == 4) {
      if (VEC) {
        const bool in = ok && k < d;       // D % 8 == 0
        const float4 z = make_float4(0.f, 0.f, 0.f, 0.f);
        *reinterpret_cast<float4*>(&v[0]) = in ? __ldg(reinterpret_cast<const float4*>(row + k)) : z;
        *reinterpret_cast<float4*>(&v[4]) = in ? __ldg(reinterpret_cast<const float4*>(row + k + 4)) : z;
      } else {
#pragma unroll
        for (int e = 0; e < 8; ++e) v[e] = ok && k + e < d ? __ldg(row + k + e) : 0.f;
      }
    } else {
      if (VEC) {
        raw = ok && k < d ? __ldg(reinterpret_cast<const uint4*>(row + k)) : make_uint4(0u, 0u, 0u, 0u);
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
  __shared__ float part[WK > 1 ? WK : 1][BM * BN / (WK > 1 ? 1 : BM * BN)];
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
  auto add = [&](int i, int j, float v) {
    if (i < p.n1 && j < p.n2) atomicAdd(p.S + static_cast<long long>(i) * p.ld_s + j, p.scale * v);
  };
  if constexpr (WK == 1) {
    if (some) {
#pragma unroll
      for (int m = 0; m < MT; ++m)
#pragma unroll
        for (int n = 0; n < NT; ++n)
#pragma unroll
          for (int e = 0; e < 4; ++e) add(i0 + 16 * m + g + 8 * (e >> 1), j0 + 8 * n + 2 * c + (e & 1), acc[m][n][e]);
    }
  } else {
#pragma unroll
    for (int m = 0; m < MT; ++m)
#pragma unroll
      for (int n = 0; n < NT; ++n)
#pragma unroll
        for (int e = 0; e < 4; ++e)
          part[wk][(wm * 16 * MT + 16 * m + g + 8 * (e >> 1)) * BN + wn * 8 * NT + 8 * n + 2 * c + (e & 1)] = acc[m][n][e];
    __syncthreads();
    for (int e = threadIdx.x; e < BM * BN; e += 256) {
      float v = 0.f;
#pragma unroll
      for (int w = 0; w < WK; ++w) v += part[w][e];
      add(blockIdx.y * BM + e / BN, blockIdx.z * BN + e % BN, v);
    }
  }
}

template <typename PT, int MT, int NT, int WM, int WN>
static int launch_similarity(SimParams p, bool vec, const DeviceState* ds, cudaStream_t st) {
  const int bi = ceil_div(p.n1, 16 * MT * WM), bj = ceil_div(p.n2, 8 * NT * WN);
  GB_REQUIRE(bi <= 65535 && bj <= 65535, "ghost_projection_similarity: too many rows");
  // one wave of two CTAs per SM, but at least eight steps for each of a CTA's WK warps of a block
  const long long steps = (p.D + 31) / 32;
  long long splits = (2ll * ds->sm_count + bi * bj - 1) / (static_cast<long long>(bi) * bj);
  const long long least = 8 * (8 / (WM * WN));
  const long long most = (steps + least - 1) / least;
  if (splits > most) splits = most;
  if (splits < 1) splits = 1;
  p.per_cta = (steps + splits - 1) / splits;
  const dim3 grid(static_cast<unsigned>((steps + p.per_cta - 1) / p.per_cta), static_cast<unsigned>(bi), static_cast<unsigned>(bj));
  if (vec) proj_similarity_kernel<PT, MT, NT, WM, WN, true><<<grid, 256, 0, st>>>(p);
  else proj_similarity_kernel<PT, MT, NT, WM, WN, false><<<grid, 256, 0, st>>>(p);
  count_launch();
  return post_launch("proj_similarity_kernel");
}

// Block shape by row counts: the smallest that holds both sets, up to 64 x 64 scores
template <typename PT>
static int dispatch_similarity(const SimParams& p, bool vec, const DeviceState* ds, cudaStream_t st) {
  if (p.n1 <= 16 && p.n2 <= 8) return launch_similarity<PT, 1, 1, 1, 1>(p, vec, ds, st);
  if (p.n1 <= 16 && p.n2 <= 16) return launch_similarity<PT, 1, 2, 1, 1>(p, vec, ds, st);
  if (p.n1 <= 16) return launch_similarity<PT, 1, 4, 1, 2>(p, vec, ds, st);
  if (p.n1 <= 32 && p.n2 <= 32) return launch_similarity<PT, 2, 4, 1, 1>(p, vec, ds, st);
  if (p.n2 <= 16) return launch_similarity<PT, 2, 2, 2, 1>(p, vec, ds, st);
  return launch_similarity<PT, 2, 4, 2, 2>(p, vec, ds, st);
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
  GB_CUDA_OK(cudaMemset2DAsync(S, static_cast<size_t>(ld_s) * 4, 0, static_cast<size_t>(n2) * 4,
                               static_cast<size_t>(n1), st));
  SimParams p = {};
  p.P1 = P1; p.P2 = P2; p.n1 = n1; p.n2 = n2; p.D = D; p.ld1 = ld1; p.ld2 = ld2; p.scale = scale; p.S = S;
  p.ld_s = ld_s;
  const int esize = is_f32 ? 4 : 2;
  const bool vec = D % 8 == 0 && (ld1 * esize) % 16 == 0 && (ld2 * esize) % 16 == 0 &&
                   ((reinterpret_cast<uintptr_t>(P1) | reinterpret_cast<uintptr_t>(P2)) & 15u) == 0;
  return is_f32 ? dispatch_similarity<float>(p, vec, ds, st) : dispatch_similarity<__nv_bfloat16>(p, vec, ds, st);
}
