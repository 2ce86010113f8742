// Convolution operands as token matrices.  Every output position of a Conv2d is a token whose features are
// the C * kh * kw inputs under the kernel window; conv_tokens_kernel writes them (and, with a 1 x 1 window,
// the [N, p, Ho, Wo] out-grad) straight into the bf16 layouts that the tensor-core paths read -- plain,
// or the hi/lo parts of float32 data side by side or stacked per sample -- in one pass over the input.
#include "common.cuh"

namespace gb {

struct ConvTokens {
  const void* src;                       // [N, C, H, W], dense
  int C, H, W, kh, kw, sy, sx, py, px, dy, dx, Wo;
  long long T;                           // Ho * Wo
  int cols, cpad;                        // C * kh * kw, padded
  __nv_bfloat16* dst;
  long long ld_dst;
  int parts, kind[3], row_stack;
};

template <typename E> __device__ __forceinline__ float ct_f32(E v);
template <> __device__ __forceinline__ float ct_f32<float>(float v) { return v; }
template <> __device__ __forceinline__ float ct_f32<__nv_bfloat16>(__nv_bfloat16 v) { return __bfloat162float(v); }

// A 64-token x 64-feature tile per block, turned in shared memory: lanes run over tokens for the loads
// (adjacent positions of one input row) and over features for the stores (128 bytes of an output
// row).  Bound by issue slots: the divisions that find a feature's channel and window position are made once
// a block (once a lane and feature they were half of all instructions: 52 us for the operands of 80
// samples of 64 x 16 x 16 with a 3 x 3 window and 128 outputs, float32; 24.6 now), and hi and lo parts
// once an element.  The library unfold before it ran one launch per sample and two more passes: 575 us.
template <typename E>
__global__ void __launch_bounds__(256) conv_tokens_kernel(const ConvTokens q) {
  stream_order();
  __shared__ float tile[64][65];
  __shared__ long long s_off[64];        // of a feature: channel and window position as an offset into the sample
  __shared__ int2 s_ij[64];              // and the position alone; far outside for the padding features
  constexpr int kFar = -(1 << 30);
  const unsigned t0 = blockIdx.x * 64u;  // tokens of a sample fit an int
  const int f0 = blockIdx.y * 64;
  const long long n = blockIdx.z;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const unsigned tokens = static_cast<unsigned>(q.T);
  const E* src = static_cast<const E*>(q.src) + n * q.C * q.H * q.W;
  if (threadIdx.x < 64) {
    const int f = f0 + threadIdx.x, window = q.kh * q.kw;
    const int c = f / window, w = f % window;
    const int i = w / q.kw * q.dy, j = w % q.kw * q.dx;
    s_off[threadIdx.x] = (static_cast<long long>(c) * q.H + i) * q.W + j;
    s_ij[threadIdx.x] = make_int2(f < q.cols ? i : kFar, j);
  }
  int y0[2], x0[2];
  long long base[2];
#pragma unroll
  for (int h = 0; h < 2; ++h) {
    const unsigned t = t0 + h * 32 + lane;
    const int oy = static_cast<int>(t / static_cast<unsigned>(q.Wo)), ox = static_cast<int>(t % static_cast<unsigned>(q.Wo));
    y0[h] = t < tokens ? oy * q.sy - q.py : kFar;
    x0[h] = ox * q.sx - q.px;
    base[h] = static_cast<long long>(y0[h]) * q.W + x0[h];
  }
  __syncthreads();
#pragma unroll
  for (int r = 0; r < 8; ++r) {
    const int2 ij = s_ij[warp * 8 + r];
    const long long off = s_off[warp * 8 + r];
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      const bool in = static_cast<unsigned>(y0[h] + ij.x) < static_cast<unsigned>(q.H) &&
                      static_cast<unsigned>(x0[h] + ij.y) < static_cast<unsigned>(q.W);
      tile[warp * 8 + r][h * 32 + lane] = in ? ct_f32<E>(src[base[h] + off]) : 0.f;
    }
  }
  __syncthreads();
#pragma unroll
  for (int h = 0; h < 2; ++h) {
    const int u = h * 256 + threadIdx.x;
    const int tl = u >> 3, fl = (u & 7) * 8;
    const unsigned t = t0 + tl;
    if (t >= tokens || f0 + fl >= q.cpad) continue;
    uint32_t hw[4], lw[4];               // the values as bf16, and what that leaves of them
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      const float va = tile[fl + 2 * e][tl], vb = tile[fl + 2 * e + 1][tl];
      const __nv_bfloat162 hi = __floats2bfloat162_rn(va, vb);
      const __nv_bfloat162 lo = __floats2bfloat162_rn(va - __bfloat162float(hi.x), vb - __bfloat162float(hi.y));
      hw[e] = *reinterpret_cast<const uint32_t*>(&hi);
      lw[e] = *reinterpret_cast<const uint32_t*>(&lo);
    }
    const long long stride = q.row_stack == 2 ? gridDim.z * q.T * q.ld_dst : q.row_stack ? q.T * q.ld_dst : q.cpad;
    __nv_bfloat16* dst = q.dst + (q.row_stack == 1 ? n * q.parts * q.T + t : n * q.T + t) * q.ld_dst + f0 + fl;
#pragma unroll
    for (int part = 0; part < 3; ++part) {
      if (part >= q.parts) break;
      const bool low = q.kind[part] == 1;
      *reinterpret_cast<uint4*>(dst + part * stride) =
          make_uint4(low ? lw[0] : hw[0], low ? lw[1] : hw[1], low ? lw[2] : hw[2], low ? lw[3] : hw[3]);
    }
  }
}

// out[r] = sum of row r of a dense [rows, len] matrix: per-sample, per-channel sums of an NCHW out-grad.
// One warp per row; the rows are contiguous, so the loads are.
template <typename E>
__global__ void __launch_bounds__(256) row_sums_kernel(const E* __restrict__ x, long long rows, long long len, float* __restrict__ out) {
  stream_order();
  const long long r = blockIdx.x * 8ll + (threadIdx.x >> 5);
  if (r >= rows) return;
  float s = 0.f;
#pragma unroll 4
  for (long long i = threadIdx.x & 31; i < len; i += 32) s += ct_f32<E>(x[r * len + i]);
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
  if ((threadIdx.x & 31) == 0) out[r] = s;
}

}  // namespace gb

using namespace gb;

extern "C" int ghost_conv_tokens_bf16(const void* src, int src_is_f32, long long samples, int C, int H, int W, int kh, int kw,
                                      int sy, int sx, int py, int px, int dy, int dx, void* dst, long long ld_dst, int cpad,
                                      int parts, int kind0, int kind1, int kind2, int row_stack, void* stream) {
  const DeviceState* ds = device_state();
  if (!ds) return GHOST_ERR_DEVICE;
  GB_REQUIRE(src && dst, "ghost_conv_tokens_bf16: null pointer");
  GB_REQUIRE(samples > 0 && samples <= 65535 && C > 0 && H > 0 && W > 0 && kh > 0 && kw > 0 && sy > 0 && sx > 0 && py >= 0 &&
                 px >= 0 && dy > 0 && dx > 0, "ghost_conv_tokens_bf16: bad geometry");
  const int Ho = (H + 2 * py - dy * (kh - 1) - 1) / sy + 1, Wo = (W + 2 * px - dx * (kw - 1) - 1) / sx + 1;
  GB_REQUIRE(H + 2 * py > dy * (kh - 1) && W + 2 * px > dx * (kw - 1), "ghost_conv_tokens_bf16: the window is larger than the padded input");
  const long long cols = static_cast<long long>(C) * kh * kw;
  GB_REQUIRE(cols <= 64ll * 65535 && cpad <= 64 * 65535, "ghost_conv_tokens_bf16: too many features per token");
  GB_REQUIRE(static_cast<long long>(Ho) * Wo < (1ll << 31) - 64, "ghost_conv_tokens_bf16: too many output positions");
  GB_REQUIRE(parts >= 1 && parts <= 3, "ghost_conv_tokens_bf16: parts must be 1..3");
  GB_REQUIRE(cpad % 8 == 0 && cpad >= cols && ld_dst % 8 == 0 && ld_dst >= (row_stack ? cpad : parts * cpad) &&
                 (reinterpret_cast<uintptr_t>(dst) & 15u) == 0, "ghost_conv_tokens_bf16: bad destination layout");
  ConvTokens q = {};
  q.src = src;
  q.C = C; q.H = H; q.W = W; q.kh = kh; q.kw = kw; q.sy = sy; q.sx = sx; q.py = py; q.px = px; q.dy = dy; q.dx = dx;
  q.Wo = Wo;
  q.T = static_cast<long long>(Ho) * Wo;
  q.cols = static_cast<int>(cols);
  q.cpad = cpad;
  q.dst = static_cast<__nv_bfloat16*>(dst);
  q.ld_dst = ld_dst;
  q.parts = parts;
  q.kind[0] = kind0; q.kind[1] = kind1; q.kind[2] = kind2;
  q.row_stack = row_stack;
  const dim3 grid(ceil_div(q.T, 64), ceil_div(cpad, 64), static_cast<unsigned>(samples));
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  if (src_is_f32) GB_CUDA_OK(launch_next(conv_tokens_kernel<float>, dim3(grid), dim3(256), 0, st, q));
  else GB_CUDA_OK(launch_next(conv_tokens_kernel<__nv_bfloat16>, dim3(grid), dim3(256), 0, st, q));
  count_launch();
  return post_launch("conv_tokens_kernel");
}

extern "C" int ghost_row_sums(const void* x, int is_f32, long long rows, long long len, float* out, void* stream) {
  const DeviceState* ds = device_state();
  if (!ds) return GHOST_ERR_DEVICE;
  GB_REQUIRE(x && out && rows > 0 && len > 0 && rows < (1ll << 33), "ghost_row_sums: bad arguments");
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  const unsigned grid = static_cast<unsigned>((rows + 7) / 8);
  if (is_f32) GB_CUDA_OK(launch_next(row_sums_kernel<float>, dim3(grid), dim3(256), 0, st, static_cast<const float*>(x), rows, len, out));
  else GB_CUDA_OK(launch_next(row_sums_kernel<__nv_bfloat16>, dim3(grid), dim3(256), 0, st, static_cast<const __nv_bfloat16*>(x), rows, len, out));
  count_launch();
  return post_launch("row_sums_kernel");
}
