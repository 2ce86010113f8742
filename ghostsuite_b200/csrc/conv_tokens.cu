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
// row).  Bound by the stores, which are kh * kw * parts times the input.  The library unfold before it
// ran one launch per sample and produced [features, tokens], transposed and split by two more passes:
// 575 us for 80 samples of 64 x 16 x 16 with a 3 x 3 window, against 19 us.
template <typename E>
__global__ void __launch_bounds__(256) conv_tokens_kernel(const ConvTokens q) {
  __shared__ float tile[64][65];
  const long long t0 = blockIdx.x * 64ll;
  const int f0 = blockIdx.y * 64;
  const long long n = blockIdx.z;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const E* src = static_cast<const E*>(q.src) + n * q.C * q.H * q.W;
  int y0[2], x0[2];
  bool ok[2];
#pragma unroll
  for (int h = 0; h < 2; ++h) {
    const long long t = t0 + h * 32 + lane;
    ok[h] = t < q.T;
    const int oy = static_cast<int>(ok[h] ? t / q.Wo : 0), ox = static_cast<int>(ok[h] ? t % q.Wo : 0);
    y0[h] = oy * q.sy - q.py;
    x0[h] = ox * q.sx - q.px;
  }
  const int window = q.kh * q.kw;
#pragma unroll
  for (int r = 0; r < 8; ++r) {
    const int f = f0 + warp * 8 + r;
    const int c = f / window, w = f % window;
    const int i = w / q.kw * q.dy, j = w % q.kw * q.dx;
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      const int y = y0[h] + i, x = x0[h] + j;
      const bool in = f < q.cols && ok[h] && y >= 0 && y < q.H && x >= 0 && x < q.W;
      tile[warp * 8 + r][h * 32 + lane] = in ? ct_f32<E>(src[(static_cast<long long>(c) * q.H + y) * q.W + x]) : 0.f;
    }
  }
  __syncthreads();
#pragma unroll
  for (int h = 0; h < 2; ++h) {
    const int u = h * 256 + threadIdx.x;
    const int tl = u >> 3, fl = (u & 7) * 8;
    const long long t = t0 + tl;
    if (t >= q.T || f0 + fl >= q.cpad) continue;
    float v[8];
#pragma unroll
    for (int e = 0; e < 8; ++e) v[e] = tile[fl + e][tl];
    for (int part = 0; part < q.parts; ++part) {
      uint32_t w[4];
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        __nv_bfloat16 a = __float2bfloat16_rn(v[2 * e]), b = __float2bfloat16_rn(v[2 * e + 1]);
        if (q.kind[part] == 1) {
          a = __float2bfloat16_rn(v[2 * e] - __bfloat162float(a));
          b = __float2bfloat16_rn(v[2 * e + 1] - __bfloat162float(b));
        }
        w[e] = static_cast<uint32_t>(__bfloat16_as_ushort(a)) | (static_cast<uint32_t>(__bfloat16_as_ushort(b)) << 16);
      }
      const long long at = q.row_stack ? ((n * q.parts + part) * q.T + t) * q.ld_dst + f0 + fl
                                       : (n * q.T + t) * q.ld_dst + static_cast<long long>(part) * q.cpad + f0 + fl;
      *reinterpret_cast<uint4*>(q.dst + at) = make_uint4(w[0], w[1], w[2], w[3]);
    }
  }
}

// out[r] = sum of row r of a dense [rows, len] matrix: per-sample, per-channel sums of an NCHW out-grad.
// One warp per row; the rows are contiguous, so the loads are.
template <typename E>
__global__ void __launch_bounds__(256) row_sums_kernel(const E* __restrict__ x, long long rows, long long len, float* __restrict__ out) {
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
  GB_REQUIRE(cols <= (1 << 22), "ghost_conv_tokens_bf16: too many features per token");
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
  if (src_is_f32) conv_tokens_kernel<float><<<grid, 256, 0, st>>>(q);
  else conv_tokens_kernel<__nv_bfloat16><<<grid, 256, 0, st>>>(q);
  count_launch();
  return post_launch("conv_tokens_kernel");
}

extern "C" int ghost_row_sums(const void* x, int is_f32, long long rows, long long len, float* out, void* stream) {
  const DeviceState* ds = device_state();
  if (!ds) return GHOST_ERR_DEVICE;
  GB_REQUIRE(x && out && rows > 0 && len > 0 && rows < (1ll << 33), "ghost_row_sums: bad arguments");
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  const unsigned grid = static_cast<unsigned>((rows + 7) / 8);
  if (is_f32) row_sums_kernel<float><<<grid, 256, 0, st>>>(static_cast<const float*>(x), rows, len, out);
  else row_sums_kernel<__nv_bfloat16><<<grid, 256, 0, st>>>(static_cast<const __nv_bfloat16*>(x), rows, len, out);
  count_launch();
  return post_launch("row_sums_kernel");
}
