// Convolution operands as token matrices.  Every output position of a Conv2d is a token whose features are
// the C * kh * kw inputs under the kernel window; conv_tokens_kernel writes them (and, with a 1 x 1 window,
// the [N, p, Ho, Wo] out-grad) straight into the bf16 layouts that the tensor-core paths read -- plain,
// or the hi/lo parts of float32 data side by side or stacked per sample -- in one pass over the input.
#include <type_traits>

#include "common.cuh"

namespace gb {

struct ConvTokens {
  const void* src;                       // [N, C, H, W], dense
  int f32;
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

// Both operands of a layer, or one
struct ConvPair {
  ConvTokens q[2];
  int blocks[3];                         // rows of blocks of the first operand, of both, and with the row sums behind them
  float* sums;                           // sums over the positions of the second operand's channels, [samples, C]
};

// A 64-token x 64-feature tile per block.  Lanes run over tokens for the loads (adjacent positions of one input row); a
// warp's eight features of a token are 16 bytes of either part, which are split in registers and go through
// shared memory for stores of 128 bytes of an output row.  Bound by issue slots, so the divisions that find a feature's channel
// and window position are made once a block and offsets are 32 bits wide where a sample allows (WIDE: it does not).
// Operands of 80 samples of 64 x 16 x 16 with a 3 x 3 window and 128 outputs, float32, with the sums of the latter:
// 20 us in one launch (the hook 57); three launches, values turned in shared memory one at a time, took 30 (65), and the
// library unfold, a launch per sample and two more passes, 575.
template <typename E, bool WIDE>
__device__ __forceinline__ void conv_tile(const ConvTokens& q, unsigned t0, int f0, long long n, long long samples,
                                          uint4 (*piece)[64 * 8], long long* s_off, int2* s_ij) {
  using Off = std::conditional_t<WIDE, long long, int>;
  constexpr int kFar = -(1 << 30);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const unsigned tokens = static_cast<unsigned>(q.T);
  const E* src = static_cast<const E*>(q.src) + n * q.C * q.H * q.W;
  if (threadIdx.x < 64) {
    const int f = f0 + threadIdx.x, window = q.kh * q.kw;
    const int c = f / window, w = f % window;
    const int i = w / q.kw * q.dy, j = w % q.kw * q.dx;
    s_off[threadIdx.x] = (static_cast<long long>(c) * q.H + i) * q.W + j;
    s_ij[threadIdx.x] = make_int2(f < q.cols ? i : kFar, j);     // far outside for the padding features
  }
  int y0[2], x0[2];
  Off base[2];
#pragma unroll
  for (int h = 0; h < 2; ++h) {
    const unsigned t = t0 + h * 32 + lane;
    const int oy = static_cast<int>(t / static_cast<unsigned>(q.Wo)), ox = static_cast<int>(t % static_cast<unsigned>(q.Wo));
    const int row = t < tokens ? oy * q.sy - q.py : 0;
    y0[h] = t < tokens ? row : kFar;
    x0[h] = ox * q.sx - q.px;
    base[h] = static_cast<Off>(row) * q.W + x0[h];
  }
  __syncthreads();
  float v[2][8];
#pragma unroll
  for (int r = 0; r < 8; ++r) {
    const int2 ij = s_ij[warp * 8 + r];
    const Off off = static_cast<Off>(s_off[warp * 8 + r]);
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      const bool in = static_cast<unsigned>(y0[h] + ij.x) < static_cast<unsigned>(q.H) &&
                      static_cast<unsigned>(x0[h] + ij.y) < static_cast<unsigned>(q.W);
      v[h][r] = in ? ct_f32<E>(src[base[h] + off]) : 0.f;
    }
  }
#pragma unroll
  for (int h = 0; h < 2; ++h) {
    uint32_t hw[4], lw[4];               // the values as bf16, and what that leaves of them
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      const float va = v[h][2 * e], vb = v[h][2 * e + 1];
      const __nv_bfloat162 hi = __floats2bfloat162_rn(va, vb);
      const __nv_bfloat162 lo = __floats2bfloat162_rn(va - __bfloat162float(hi.x), vb - __bfloat162float(hi.y));
      hw[e] = *reinterpret_cast<const uint32_t*>(&hi);
      lw[e] = *reinterpret_cast<const uint32_t*>(&lo);
    }
    const int at = (h * 32 + lane) * 8 + (warp ^ (lane & 7));
    piece[0][at] = make_uint4(hw[0], hw[1], hw[2], hw[3]);
    piece[1][at] = make_uint4(lw[0], lw[1], lw[2], lw[3]);
  }
  __syncthreads();
  const long long stride = q.row_stack == 2 ? samples * q.T * q.ld_dst : q.row_stack ? q.T * q.ld_dst : q.cpad;
#pragma unroll
  for (int h = 0; h < 2; ++h) {
    const int u = h * 256 + threadIdx.x;
    const int tl = u >> 3, fl = (u & 7) * 8;
    const unsigned t = t0 + tl;
    if (t >= tokens || f0 + fl >= q.cpad) continue;
    __nv_bfloat16* dst = q.dst + (q.row_stack == 1 ? n * q.parts * q.T + t : n * q.T + t) * q.ld_dst + f0 + fl;
#pragma unroll
    for (int part = 0; part < 3; ++part) {
      if (part >= q.parts) break;
      *reinterpret_cast<uint4*>(dst + part * stride) = piece[q.kind[part] == 1][tl * 8 + ((u & 7) ^ (tl & 7))];
    }
  }
}

template <typename E> __device__ __forceinline__ void row_sum(const E* x, long long r, long long len, float* __restrict__ out) {
  float s = 0.f;
#pragma unroll 4
  for (long long i = threadIdx.x & 31; i < len; i += 32) s += ct_f32<E>(x[r * len + i]);
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
  if ((threadIdx.x & 31) == 0) out[r] = s;
}

template <bool WIDE>
__global__ void __launch_bounds__(256) conv_tokens_kernel(const __grid_constant__ ConvPair p) {
  stream_order();
  __shared__ __align__(16) uint4 piece[2][64 * 8];
  __shared__ long long s_off[64];        // of a feature: channel and window position as an offset into the sample
  __shared__ int2 s_ij[64];              // and the position alone
  const long long n = blockIdx.z;
  const int y = blockIdx.y;
  if (y >= p.blocks[1]) {                // a warp per channel of the second operand
    const ConvTokens& q = p.q[1];
    const long long c = (static_cast<long long>(y - p.blocks[1]) * gridDim.x + blockIdx.x) * 8 + (threadIdx.x >> 5);
    if (c >= q.C) return;
    if (q.f32) row_sum(static_cast<const float*>(q.src), n * q.C + c, q.T, p.sums);
    else row_sum(static_cast<const __nv_bfloat16*>(q.src), n * q.C + c, q.T, p.sums);
    return;
  }
  const ConvTokens& q = p.q[y >= p.blocks[0]];
  const int f0 = (y >= p.blocks[0] ? y - p.blocks[0] : y) * 64;
  if (q.f32) conv_tile<float, WIDE>(q, blockIdx.x * 64u, f0, n, gridDim.z, piece, s_off, s_ij);
  else conv_tile<__nv_bfloat16, WIDE>(q, blockIdx.x * 64u, f0, n, gridDim.z, piece, s_off, s_ij);
}

// out[r] = sum of row r of a dense [rows, len] matrix: per-sample, per-channel sums of an NCHW out-grad.
// One warp per row; the rows are contiguous, so the loads are.
template <typename E>
__global__ void __launch_bounds__(256) row_sums_kernel(const E* x, long long rows, long long len, float* __restrict__ out) {
  stream_order();
  const long long r = blockIdx.x * 8ll + (threadIdx.x >> 5);
  if (r < rows) row_sum(x, r, len, out);
}

// Operand `q` from the entry points' arguments, `dst` with its layout
static int conv_operand(ConvTokens& q, const void* src, int src_is_f32, long long samples, int C, int H, int W, int kh, int kw,
                        int sy, int sx, int py, int px, int dy, int dx, void* dst, long long ld_dst, int cpad, int parts,
                        int row_stack) {
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
  q.src = src;
  q.f32 = src_is_f32;
  q.C = C; q.H = H; q.W = W; q.kh = kh; q.kw = kw; q.sy = sy; q.sx = sx; q.py = py; q.px = px; q.dy = dy; q.dx = dx;
  q.Wo = Wo;
  q.T = static_cast<long long>(Ho) * Wo;
  q.cols = static_cast<int>(cols);
  q.cpad = cpad;
  q.dst = static_cast<__nv_bfloat16*>(dst);
  q.ld_dst = ld_dst;
  q.parts = parts;
  q.row_stack = row_stack;
  return GHOST_OK;
}

// Offsets and positions of a sample, the padding around it included, fit 32 bits
static bool conv_narrow(const ConvTokens& q) {
  const long long rows = static_cast<long long>(q.H) + 2 * q.py, width = static_cast<long long>(q.W) + 2 * q.px;
  return (static_cast<long long>(q.C) + 1) * rows * width < (1ll << 30);
}

static int launch_conv_tokens(const ConvPair& p, bool wide, long long samples, cudaStream_t st) {
  const dim3 grid(ceil_div(p.q[0].T, 64), p.blocks[2], static_cast<unsigned>(samples));
  if (wide) GB_CUDA_OK(launch_next(conv_tokens_kernel<true>, grid, dim3(256), 0, st, p));
  else GB_CUDA_OK(launch_next(conv_tokens_kernel<false>, grid, dim3(256), 0, st, p));
  count_launch();
  return post_launch("conv_tokens_kernel");
}

}  // namespace gb

using namespace gb;

extern "C" int ghost_conv_tokens_bf16(const void* src, int src_is_f32, long long samples, int C, int H, int W, int kh, int kw,
                                      int sy, int sx, int py, int px, int dy, int dx, void* dst, long long ld_dst, int cpad,
                                      int parts, int kind0, int kind1, int kind2, int row_stack, void* stream) {
  const DeviceState* ds = device_state();
  if (!ds) return GHOST_ERR_DEVICE;
  ConvPair p = {};
  const int rc = conv_operand(p.q[0], src, src_is_f32, samples, C, H, W, kh, kw, sy, sx, py, px, dy, dx, dst, ld_dst, cpad, parts, row_stack);
  if (rc != GHOST_OK) return rc;
  p.q[0].kind[0] = kind0; p.q[0].kind[1] = kind1; p.q[0].kind[2] = kind2;
  p.blocks[0] = p.blocks[1] = p.blocks[2] = ceil_div(cpad, 64);
  return launch_conv_tokens(p, !conv_narrow(p.q[0]), samples, static_cast<cudaStream_t>(stream));
}

extern "C" int ghost_conv_operands(const void* A, int a_is_f32, const void* B, int b_is_f32, long long samples, int C, int H, int W,
                                   int kh, int kw, int sy, int sx, int py, int px, int dy, int dx, int p_out, int Ho, int Wo,
                                   int parts, int merged, void* A_out, void* B_out, float* b_sums, void* stream) {
  const DeviceState* ds = device_state();
  if (!ds) return GHOST_ERR_DEVICE;
  GB_REQUIRE(parts == 1 || parts == 2, "ghost_conv_operands: one or two parts");
  GB_REQUIRE(p_out > 0 && p_out <= 64 * 65535 && C > 0 && kh > 0 && kw > 0 && static_cast<long long>(C) * kh * kw <= 64ll * 65535,
             "ghost_conv_operands: too many features per token");
  ConvPair p = {};
  const int pad_a = (C * kh * kw + 63) / 64 * 64, pad_b = (p_out + 63) / 64 * 64, stack = merged ? 2 : 1;
  int rc = conv_operand(p.q[0], A, a_is_f32, samples, C, H, W, kh, kw, sy, sx, py, px, dy, dx, A_out, pad_a, pad_a, parts, stack);
  if (rc == GHOST_OK) rc = conv_operand(p.q[1], B, b_is_f32, samples, p_out, Ho, Wo, 1, 1, 1, 1, 0, 0, 1, 1, B_out, pad_b, pad_b, parts, stack);
  if (rc != GHOST_OK) return rc;
  GB_REQUIRE(p.q[0].T == p.q[1].T && p.q[0].Wo == Wo, "ghost_conv_operands: the out-grad is not this convolution's output size");
  p.q[0].kind[1] = p.q[1].kind[1] = 1;
  const long long tiles = ceil_div(p.q[0].T, 64);
  const long long rows = b_sums ? (ceil_div(p_out, 8) + tiles - 1) / tiles : 0;
  p.blocks[0] = pad_a / 64;
  p.blocks[1] = p.blocks[0] + pad_b / 64;
  p.blocks[2] = p.blocks[1] + static_cast<int>(rows);
  p.sums = b_sums;
  const bool wide = !conv_narrow(p.q[0]) || !conv_narrow(p.q[1]);
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  if (p.blocks[2] <= 65535) return launch_conv_tokens(p, wide, samples, st);
  // more blocks of features than a grid has rows: an operand a launch
  ConvPair one = p;
  one.blocks[1] = one.blocks[2] = one.blocks[0];
  if ((rc = launch_conv_tokens(one, wide, samples, st)) != GHOST_OK) return rc;
  one.q[0] = p.q[1];
  one.blocks[0] = one.blocks[1] = one.blocks[2] = pad_b / 64;
  if ((rc = launch_conv_tokens(one, wide, samples, st)) != GHOST_OK || !b_sums) return rc;
  return ghost_row_sums(B, b_is_f32, samples * p_out, p.q[1].T, b_sums, stream);
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
