// tile_dot: second half of the per-sample-gradient path.
//
// xty_gemm (kEpiStoreTiles) leaves the per-sample weight-gradient tiles of the validation samples
// (V) and of a group of train samples (W) in a workspace, tile-major: [tile][sample][32768].  V and W
// may be one buffer holding all samples (train first) or two buffers; either way they are described
// by 3-D tensor maps [tiles, samples, 32768] plus a first-validation-sample offset.  This kernel streams both once and produces
//     M[v, b]  += scale * sum_k V[v][k] * W[b][k]        (Frobenius products, reference :135)
//     sum[k]   (+)= sum_b W[b][k]                        (the train gradient, reference :168)
//
// HBM-bound by design, so it is built as a copy pipeline: one producer thread feeds a ring of
// shared-memory stages with TMA (one box of validation rows and one of train rows per stage: float32 8, 16 or 32
// train rows, 256 elements wide, bf16 16 or 32 of 512); the compute warps consume them.  Each CTA owns a contiguous range of stages:
// the train-gradient sum is a plain read-modify-write (deterministic, no atomics); the dot
// products are reduced inside the CTA and added to M once per CTA and block.
//
// bf16 tiles (tile_dot_mma_kernel): the stage is loaded as eight 128-byte-swizzled 64-element
// panels per operand, and both contractions run on the tensor cores through mma.sync
// (m16n8k16, fp32 accumulate) fed by ldmatrix: the dot products as W[16 train x 16 k] x
// V[16 k x 8 val], the train-gradient sum as mask[16 x 16 train] x W[16 train x 8 k] (a
// transposed ldmatrix of the same rows).  A warp owns 32 (or 64) neighbouring elements of the stage's 512.  With the
// arithmetic off the CUDA cores the kernel is bound by the stream, and up to 32 validation rows
// share one pass over the train rows.
//
// fp32 tiles (tile_dot_f32_kernel): the same split of a stage over the warps, with the products on the
// CUDA cores (exact fp32 products).
#include "common.cuh"
#include "sm100_ptx.cuh"

namespace gb {

constexpr int kTileElems = 128 * 256;
constexpr int kTdCols = 256;            // elements per stage row

struct TileDotParams {
  long long stages;           // bf16: tiles * (32768 / 512); fp32: m_cols * n_tiles_n rows of 256 elements
  long long stages_per_cta;
  int n_val, n_grp;           // validation samples, train samples in this group
  int v_off;                  // index of the first validation sample inside V's sample dimension
  int v_per_rank;             // > 0: V is [ranks][tiles][v_per_rank][32768] (bf16 kernel only), v_off = 0
  int b0, n_train;            // first train sample of the group, total train samples (M row pitch)
  float scale;
  float* M;                   // [n_val, n_train]
  float* sum;                 // [tiles * 32768] fp32 or null
  int sum_init;               // 1: this group overwrites sum, 0: it accumulates
  // direct output of the train gradient (single-group case): out[r, c] (= or +=) out_scale * sum.  With `sum` too (bf16 tiles) the
  // blocks of train rows before the last one add up there, and the last one rounds to `out` once
  void* out;                  // [m_cols, n_cols] row-major in the parameter dtype, or null
  int out_is_f32, out_accumulate;
  int m_cols, n_cols, n_tiles_n;
  float out_scale;
  int* err;
};

// two float32 in one register pair: sum, and product added to a third
__device__ __forceinline__ uint64_t td_add2(uint64_t a, uint64_t b) {
  uint64_t d;
  asm("add.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
  return d;
}
__device__ __forceinline__ void td_fma2(uint64_t& acc, uint64_t a, uint64_t b) {
  asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(acc) : "l"(a), "l"(b));
}
__device__ __forceinline__ float2 td_unpack(uint64_t v) {
  float2 f;
  asm("mov.b64 {%0, %1}, %2;" : "=f"(f.x), "=f"(f.y) : "l"(v));
  return f;
}
__device__ __forceinline__ ulonglong2 td_load4(uint32_t addr) {      // four floats of shared memory
  ulonglong2 v;
  asm volatile("ld.shared.v2.b64 {%0, %1}, [%2];" : "=l"(v.x), "=l"(v.y) : "r"(addr));
  return v;
}

// Stage of the fp32 kernel: 256 elements of every row, as eight 128-byte-swizzled panels of 32.  VR validation rows and
// 8 KB train rows go through together.
template <int VR, int KB>
struct TdF32Cfg {
  static constexpr int kTrainRows = 8 * KB;
  static constexpr int kPanels = kTdCols / 32;
  static constexpr int kWarpRows = VR == 16 ? 8 : 4;         // validation rows of a warp
  static constexpr int kWarpPanels = VR / kWarpRows;         // and its panels of a stage
  static constexpr int kValBytes = kPanels * VR * 128;
  static constexpr int kStageBytes = kValBytes + kPanels * kTrainRows * 128;     // 12 to 48 KB
  // Two CTAs per SM: with one CTA's eight warps the schedulers have two warps each to hide a stage's chain of loads,
  // products and shuffles behind.  Sixteen validation rows a pass take the registers of both: with four rows a warp
  // the train rows would be read from shared memory four times (64 + 16 x 512 x (1024 -> 1024): 90.7 against 89.2 us, 17.4
  // against 14.6 for 64 + 16 of 128 x 576).
  static constexpr int kCtas = VR == 16 ? 1 : 2;
  static constexpr int kStages = kCtas == 1 || kStageBytes <= 24 * 1024 ? 4 : 2;
  static constexpr int kRedBytes = 8 * kTrainRows * kWarpRows * 4;               // per-warp partial dot blocks
  static constexpr int kSmemBytes = kStages * kStageBytes + kRedBytes + 1024 + 256;
};

// VR validation rows x 8 KB train rows per pass.  A warp owns one or two panels of a stage and four or eight of the validation
// rows; lane (g, q) holds train rows g, g + 8, ... and elements 8q .. 8q + 7 of a panel, so the swizzle puts the eight 16-byte
// reads of a quarter-warp into different banks, the column sums are seven shuffles, and the warps run through
// the ring on their own: no barrier among them until the block is done.  Stages follow the rows of
// the weight, so rows that only pad the last tile are not read.  Train rows past the group read as zero (the
// tensor map ends with the group), so nothing is masked.
//
// What bounds it: reads of shared memory (53 % of its cycles; a quarter-warp that shares a row still takes one) and, on small
// layers, the latency of a handful of stages.  Two elements an instruction (f32x2), the stage's place counted on
// and no masks make it 390 instructions a warp and stage where there were 618; the sum that a later block of train rows adds to is fetched
// ahead of the wait.  Before and now, L2 warm: 24 + 5 samples of 768 x 1000 26.9 -> 23.7 us (91 MB), 31 + 3 of 640 x 126 10.0 -> 7.1,
// 3 + 1 of 468 x 128 8.3 -> 5.1, 40 + 13 of 512 x 512 29.9 -> 27.3, 64 + 16 of 1024 x 1024 103 -> 89.  Tried: tf32 products of values in two
// parts on the tensor cores take 19.9 us for the first, but its sums are cut short and the dot products' error
// against 64 bits grew by 8e-8 of 1.26e-6; one CTA per SM with eight validation rows a warp 25.2.
template <int VR, int KB>
__global__ void __launch_bounds__(288, TdF32Cfg<VR, KB>::kCtas)
tile_dot_f32_kernel(const __grid_constant__ CUtensorMap tm_v, const __grid_constant__ CUtensorMap tm_w,
                    const TileDotParams p) {
  using Cfg = TdF32Cfg<VR, KB>;
  constexpr int kStages = Cfg::kStages, TR = Cfg::kTrainRows, WR = Cfg::kWarpRows, WP = Cfg::kWarpPanels;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  float* s_red = reinterpret_cast<float*>(smem + kStages * Cfg::kStageBytes);            // [8 warps][WR][TR]
  uint64_t* bars = reinterpret_cast<uint64_t*>(smem + kStages * Cfg::kStageBytes + Cfg::kRedBytes);
  uint64_t* full_bar = bars;
  uint64_t* empty_bar = bars + kStages;
  volatile int* abort_flag = reinterpret_cast<volatile int*>(bars + 2 * kStages);

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const long long s_begin = static_cast<long long>(blockIdx.x) * p.stages_per_cta;
  const long long s_end = (s_begin + p.stages_per_cta < p.stages) ? s_begin + p.stages_per_cta : p.stages;
  // row of the weight and 256-column block of the first stage; the following ones are counted on (a 64-bit division a stage
  // was a third of a warp's instructions)
  const int r_begin = static_cast<int>(s_begin / p.n_tiles_n), tn_begin = static_cast<int>(s_begin % p.n_tiles_n);

  if (threadIdx.x == 0) {
    for (int s = 0; s < kStages; ++s) { mbar_init(&full_bar[s], 1); mbar_init(&empty_bar[s], 8); }
    *abort_flag = 0;
    fence_barrier_init();
  }
  if (warp == 8 && lane == 0) { tma_prefetch_desc(&tm_v); tma_prefetch_desc(&tm_w); }
  __syncthreads();
  stream_order();

  if (warp == 8) {
    // ---------------------------------------------------------------- TMA producer
    if (lane == 0) {
      int stage = 0; uint32_t phase = 0; bool ok = true;
      for (int j0 = 0; j0 < p.n_grp && ok; j0 += TR)
        for (int v0 = 0; v0 < p.n_val && ok; v0 += VR) {
          int r = r_begin, tn = tn_begin;
          for (long long s = s_begin; s < s_end; ++s) {
            if (!mbar_wait(&empty_bar[stage], phase ^ 1, abort_flag, p.err, 431)) { ok = false; break; }
            uint8_t* st = smem + stage * Cfg::kStageBytes;
            const int tile = (r >> 7) * p.n_tiles_n + tn, panel = (r & 127) * Cfg::kPanels;
            mbar_arrive_expect_tx(&full_bar[stage], Cfg::kStageBytes);
            tma_load_4d(st, &tm_v, &full_bar[stage], 0, p.v_off + v0, panel, tile);
            tma_load_4d(st + Cfg::kValBytes, &tm_w, &full_bar[stage], 0, j0, panel, tile);
            if (++stage == kStages) { stage = 0; phase ^= 1; }
            if (++tn == p.n_tiles_n) { tn = 0; ++r; }
          }
        }
    }
    return;
  }

  // ------------------------------------------------------------------ compute warps 0-7
  const int g = lane >> 2, q = lane & 3;
  const int rows_of = warp / (8 / WP), row0 = rows_of * WR, panel0 = warp % (8 / WP) * WP;
  // the panel whose column sums this warp takes, and the element of the stage whose sum ends up in this lane (see the
  // butterfly below)
  const int sum_panel = panel0 + rows_of;
  const int mine = sum_panel * 32 + q * 8 + ((lane >> 4) & 1) * 4 + ((lane >> 3) & 1) * 2 + ((lane >> 2) & 1);
  // Places of this lane's 16-byte chunks 2q and 2q + 1 in the rows of a panel: chunk ^ (row mod 8), which goes by the address, so
  // panels of four rows fill half of the swizzle's 1024-byte period.  Everything else is an immediate.
  const uint32_t s_stage = smem_u32(smem);
  const uint32_t w_at[2] = {static_cast<uint32_t>(g * 128 + (((2 * q) ^ g) << 4)), static_cast<uint32_t>(g * 128 + (((2 * q + 1) ^ g) << 4))};
  const int q_row = (2 * q) ^ (((VR == 4 ? 4 * warp : row0)) & 4);
  uint32_t v_at[WR / 2];
#pragma unroll
  for (int m = 0; m < WR / 2; ++m) v_at[m] = static_cast<uint32_t>(row0 * 128 + ((q_row ^ (2 * m)) << 4));
  int stage = 0; uint32_t phase = 0;
  bool alive = true;
  for (int j0 = 0; j0 < p.n_grp && alive; j0 += TR) {
    for (int v0 = 0; v0 < p.n_val && alive; v0 += VR) {
      uint64_t acc[WR][KB];              // elements of even and odd index apart
#pragma unroll
      for (int i = 0; i < WR; ++i)
#pragma unroll
        for (int k = 0; k < KB; ++k) acc[i][k] = 0;
      const bool do_sum = (v0 == 0) && (p.sum != nullptr || p.out != nullptr);
      const bool onto = p.out != nullptr ? p.out_accumulate || j0 > 0 : !(p.sum_init && j0 == 0);
      int r = r_begin, tn = tn_begin;
#pragma unroll 1
      for (long long s = s_begin; s < s_end; ++s) {
        // the sum that this stage's is added to is fetched ahead of the wait
        const bool stored = do_sum && (p.out == nullptr || tn * 256 + mine < p.n_cols);
        const long long at = p.out != nullptr ? static_cast<long long>(r) * p.n_cols + tn * 256 + mine
                                              : (static_cast<long long>(r >> 7) * p.n_tiles_n + tn) * kTileElems + (r & 127) * kTdCols + mine;
        float old = 0.f;
        if (stored && onto)
          old = p.out == nullptr ? p.sum[at] : p.out_is_f32 ? static_cast<const float*>(p.out)[at] : __bfloat162float(static_cast<const __nv_bfloat16*>(p.out)[at]);
        int ok = 1;
        if (lane == 0) ok = mbar_wait(&full_bar[stage], phase, abort_flag, p.err, 132) ? 1 : 0;
        ok = __shfl_sync(0xffffffffu, ok, 0);
        __syncwarp();                    // the shuffle carries the verdict; this orders the stage's bytes for all lanes
        if (!ok) { alive = false; break; }
        const uint32_t vbuf = s_stage + stage * Cfg::kStageBytes + panel0 * (VR * 128);
        const uint32_t wbuf = s_stage + stage * Cfg::kStageBytes + Cfg::kValBytes + panel0 * (TR * 128);
        uint64_t sum2[4];
#pragma unroll (WP < 4 ? WP : 1)
        for (int pn = 0; pn < WP; ++pn) {
#pragma unroll
          for (int c = 0; c < 2; ++c) {
            ulonglong2 w[KB];
#pragma unroll
            for (int k = 0; k < KB; ++k) w[k] = td_load4(wbuf + pn * (TR * 128) + w_at[c] + k * 1024);
            if (WP == 1 || pn == rows_of) {
              sum2[2 * c] = w[0].x;
              sum2[2 * c + 1] = w[0].y;
#pragma unroll
              for (int k = 1; k < KB; ++k) {
                sum2[2 * c] = td_add2(sum2[2 * c], w[k].x);
                sum2[2 * c + 1] = td_add2(sum2[2 * c + 1], w[k].y);
              }
            }
#pragma unroll
            for (int i = 0; i < WR; ++i) {
              const ulonglong2 v = td_load4(vbuf + pn * (VR * 128) + v_at[i >> 1] + i * 128 + (((i & 1) ^ c) << 4));
#pragma unroll
              for (int k = 0; k < KB; ++k) {
                td_fma2(acc[i][k], v.x, w[k].x);
                td_fma2(acc[i][k], v.y, w[k].y);
              }
            }
          }
        }
        __syncwarp();
        if (lane == 0) mbar_arrive(&empty_bar[stage]);     // this warp is done with the stage
        if (++stage == kStages) { stage = 0; phase ^= 1; }
        if (do_sum) {
          // the lane's train rows are added up; now over the eight lanes g: a
          // butterfly that halves the elements with every step leaves one in each lane
          float sum[8];
#pragma unroll
          for (int x = 0; x < 4; ++x) {
            const float2 f = td_unpack(sum2[x]);
            sum[2 * x] = f.x;
            sum[2 * x + 1] = f.y;
          }
#pragma unroll
          for (int h = 4; h >= 1; h >>= 1) {
            const bool up = (lane & (h * 4)) != 0;
#pragma unroll
            for (int x = 0; x < h; ++x) {
              const float send = up ? sum[x] : sum[x + h], keep = up ? sum[x + h] : sum[x];
              sum[x] = keep + __shfl_xor_sync(0xffffffffu, send, h * 4);
            }
          }
          if (stored) {
            if (p.out == nullptr) p.sum[at] = sum[0] + old;
            else if (p.out_is_f32) static_cast<float*>(p.out)[at] = sum[0] * p.out_scale + old;
            else static_cast<__nv_bfloat16*>(p.out)[at] = __float2bfloat16_rn(sum[0] * p.out_scale + old);
          }
        }
        if (++tn == p.n_tiles_n) { tn = 0; ++r; }
      }
      // the only CTA-wide agreement: every compute warp gets here once per block, aborted or not
      if (!named_bar_and(1, 256, alive)) { alive = false; break; }
      // reduce the block over the four lanes q, then over the warps that share its rows; one atomic per (v, b) and CTA
      float* part = s_red + warp * (TR * WR);
#pragma unroll
      for (int i = 0; i < WR; ++i) {
        float a[KB];
#pragma unroll
        for (int k = 0; k < KB; ++k) {
          const float2 f = td_unpack(acc[i][k]);
          a[k] = f.x + f.y;
        }
        if constexpr (KB == 4) {
#pragma unroll
          for (int h = 2; h >= 1; h >>= 1) {
            const bool up = (lane & h) != 0;
#pragma unroll
            for (int k = 0; k < h; ++k) {
              const float send = up ? a[k] : a[k + h], keep = up ? a[k + h] : a[k];
              a[k] = keep + __shfl_xor_sync(0xffffffffu, send, h);
            }
          }
          part[i * TR + q * 8 + g] = a[0];       // lane q is left with k = q
        } else {
#pragma unroll
          for (int k = 0; k < KB; ++k) {
            a[k] += __shfl_xor_sync(0xffffffffu, a[k], 1);
            a[k] += __shfl_xor_sync(0xffffffffu, a[k], 2);
            if (q == k) part[i * TR + k * 8 + g] = a[k];
          }
        }
      }
      named_bar_sync(2, 256);
      for (int idx = threadIdx.x; idx < TR * VR; idx += 256) {
        const int b = idx % TR, v = idx / TR;
        const float* from = s_red + v / WR * (8 / WP) * (TR * WR) + v % WR * TR + b;
        float t = 0.f;
#pragma unroll
        for (int w = 0; w < 8 / WP; ++w) t += from[w * (TR * WR)];
        if (v0 + v < p.n_val && j0 + b < p.n_grp && t != 0.f)
          atomicAdd(&p.M[static_cast<long long>(v0 + v) * p.n_train + p.b0 + j0 + b], t * p.scale);
      }
      named_bar_sync(2, 256);
    }
  }
}

// ------------------------------------------------------------------------------------------------
// bf16 tiles on mma.sync
// ------------------------------------------------------------------------------------------------
__device__ __forceinline__ void ldsm_x4(uint32_t addr, uint32_t (&r)[4]) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0, %1, %2, %3}, [%4];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(addr));
}
__device__ __forceinline__ void ldsm_x4_trans(uint32_t addr, uint32_t (&r)[4]) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0, %1, %2, %3}, [%4];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(addr));
}
__device__ __forceinline__ void mma_bf16_16816(float (&d)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
  asm volatile(
      "mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, "
      "{%0, %1, %2, %3};"
      : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
      : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}

// Elements per stage row of the bf16 kernel.  Every warp pays a barrier wait per stage, so a stage
// is made as wide as the shared memory allows: 512 elements = 32 or 64 per warp = two or four k-steps.
constexpr int kMmaCols = 512;

// NVT: 8-row validation blocks per stage (1, 2 or 4); MT: 16-row train blocks per stage (2, or 1
// when the group has at most 16 train samples: a data-parallel rank's share of the batch -- the
// stage then holds and the warps then work on half as many rows)
template <int NVT, int MT = 2>
struct TdMmaCfg {
  static constexpr int kTrainRows = 16 * MT;
  static constexpr int kValRows = 8 * NVT;
  // Sixteen compute warps: a warp's stage is a chain of a barrier wait, two rounds of ldmatrix, dependent products and the store
  // of its sums, and with eight of them the schedulers issued in 27 % of their cycles, most of the rest waiting
  // for fixed latencies.  Of 32 validation rows there is enough to do for eight, and the sixteen would
  // have to add up their blocks in rounds (233 + 17 samples of one tile: 21 against 40 us).
  static constexpr int kWarps = NVT == 4 ? 8 : 16;
  static constexpr int kPanels = kMmaCols / 64;                              // 64-element panels per stage row
  static constexpr int kWarpChunks = kMmaCols / 8 / kWarps;                    // 16-byte chunks per warp and stage
  static constexpr int kWarpKSteps = kWarpChunks / 2;
  static constexpr int kValBytes = kPanels * kValRows * 128;
  static constexpr int kStageBytes = kValBytes + kPanels * kTrainRows * 128;     // 40 / 48 / 64 KB at MT = 2
  static constexpr int kStages = NVT == 1 ? 4 : 3;
  static constexpr int kRedBytes = 8 * kTrainRows * kValRows * 4;            // partial dot blocks, of one or two warps each
  // (validation row, train row) of a block; the permutation puts a warp's stores into different banks
  static __device__ __forceinline__ int red_at(int v, int b) { return v * kTrainRows + (b ^ ((((v >> 1) & 3) << 3) & (kTrainRows - 1))); }
  static constexpr int kSmemBytes = kStages * kStageBytes + kRedBytes + 1024 + 256;
};

template <int NVT, int MT>
__global__ void __launch_bounds__((TdMmaCfg<NVT, MT>::kWarps + 1) * 32, 1)
tile_dot_mma_kernel(const __grid_constant__ CUtensorMap tm_v, const __grid_constant__ CUtensorMap tm_w,
                    const TileDotParams p) {
  using Cfg = TdMmaCfg<NVT, MT>;
  constexpr int kStages = Cfg::kStages, VR = Cfg::kValRows, TR = Cfg::kTrainRows, kWarps = Cfg::kWarps;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  float* s_red = reinterpret_cast<float*>(smem + kStages * Cfg::kStageBytes);            // [8][VR][TR]
  uint64_t* bars = reinterpret_cast<uint64_t*>(smem + kStages * Cfg::kStageBytes + Cfg::kRedBytes);
  uint64_t* full_bar = bars;
  uint64_t* empty_bar = bars + kStages;
  volatile int* abort_flag = reinterpret_cast<volatile int*>(bars + 2 * kStages);

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const long long s_begin = static_cast<long long>(blockIdx.x) * p.stages_per_cta;
  const long long s_end = (s_begin + p.stages_per_cta < p.stages) ? s_begin + p.stages_per_cta : p.stages;
  constexpr int kStagesPerTile = kTileElems / kMmaCols;   // 64
  constexpr int KS = Cfg::kWarpKSteps, CW = Cfg::kWarpChunks;
  const int tm_begin = static_cast<int>(s_begin / kStagesPerTile / p.n_tiles_n), tn_begin = static_cast<int>(s_begin / kStagesPerTile % p.n_tiles_n);

  if (threadIdx.x == 0) {
    for (int s = 0; s < kStages; ++s) { mbar_init(&full_bar[s], 1); mbar_init(&empty_bar[s], kWarps); }
    *abort_flag = 0;
    fence_barrier_init();
  }
  if (warp == kWarps && lane == 0) { tma_prefetch_desc(&tm_v); tma_prefetch_desc(&tm_w); }
  __syncthreads();
  stream_order();

  if (warp == kWarps) {
    // ---------------------------------------------------------------- TMA producer
    if (lane == 0) {
      int stage = 0; uint32_t phase = 0; bool ok = true;
      for (int j0 = 0; j0 < p.n_grp && ok; j0 += TR)
        for (int v0 = 0; v0 < p.n_val && ok; v0 += VR)
          for (long long s = s_begin; s < s_end; ++s) {
            if (!mbar_wait(&empty_bar[stage], phase ^ 1, abort_flag, p.err, 431)) { ok = false; break; }
            uint8_t* st = smem + stage * Cfg::kStageBytes;
            const int tile = static_cast<int>(s / kStagesPerTile);
            const int panel = static_cast<int>(s % kStagesPerTile) * Cfg::kPanels;   // 64-element panels
            mbar_arrive_expect_tx(&full_bar[stage], Cfg::kStageBytes);
            if (p.v_per_rank > 0)
              tma_load_5d(st, &tm_v, &full_bar[stage], 0, v0 % p.v_per_rank, v0 / p.v_per_rank, panel, tile);
            else
              tma_load_4d(st, &tm_v, &full_bar[stage], 0, p.v_off + v0, panel, tile);
            tma_load_4d(st + Cfg::kValBytes, &tm_w, &full_bar[stage], 0, j0, panel, tile);
            if (++stage == kStages) { stage = 0; phase ^= 1; }
          }
    }
    return;
  }

  // ------------------------------------------------------------------ compute warps
  // This warp's slice of a stage: CW 16-byte chunks (KS k-steps) starting at chunk c0 of panel pn.
  const int pn = (warp * CW) / 8, c0 = (warp * CW) % 8;
  const int g = lane >> 2, q = lane & 3;
  // ldmatrix lane addresses inside a stage (panel rows are 128 bytes, chunk index XOR (row & 7))
  uint32_t a_off[MT][KS];    // W as the A operand: [m-tile][k-step]
#pragma unroll
  for (int mt = 0; mt < MT; ++mt)
#pragma unroll
    for (int ks = 0; ks < KS; ++ks) {
      const int row = mt * 16 + (lane & 15), chunk = c0 + 2 * ks + (lane >> 4);
      a_off[mt][ks] = Cfg::kValBytes + pn * (TR * 128) + row * 128 + ((chunk ^ (row & 7)) << 4);
    }
  uint32_t b_off[NVT][KS / 2];   // V as the B operand: [n-tile][pair of k-steps], one x4 each
#pragma unroll
  for (int nt = 0; nt < NVT; ++nt)
#pragma unroll
    for (int h = 0; h < KS / 2; ++h) {
      const int row = nt * 8 + (lane & 7), chunk = c0 + 4 * h + (lane >> 3);
      b_off[nt][h] = pn * (VR * 128) + row * 128 + ((chunk ^ (row & 7)) << 4);
    }
  uint32_t t_off[CW];        // W transposed, for the column sums: [8-element group], rows = lane
  const int trow = lane & (TR - 1);      // with 16 train rows lanes 16-31 repeat rows 0-15 (their matrices are not used)
#pragma unroll
  for (int j = 0; j < CW; ++j)
    t_off[j] = Cfg::kValBytes + pn * (TR * 128) + trow * 128 + (((c0 + j) ^ (trow & 7)) << 4);

  int stage = 0; uint32_t phase = 0;
  bool alive = true;
  for (int j0 = 0; j0 < p.n_grp && alive; j0 += TR) {
    // A operand of the column-sum MMA: 1.0 where the train row (the k index) belongs to the group
    uint32_t mask_a[2][4];
#pragma unroll
    for (int kr = 0; kr < 2; ++kr) {
      const int k_lo = j0 + kr * 16 + q * 2, k_hi = k_lo + 8;
      const uint32_t lo = (k_lo < p.n_grp ? 0x3F80u : 0u) | (k_lo + 1 < p.n_grp ? 0x3F800000u : 0u);
      const uint32_t hi = (k_hi < p.n_grp ? 0x3F80u : 0u) | (k_hi + 1 < p.n_grp ? 0x3F800000u : 0u);
      mask_a[kr][0] = lo; mask_a[kr][1] = lo; mask_a[kr][2] = hi; mask_a[kr][3] = hi;
    }
    for (int v0 = 0; v0 < p.n_val && alive; v0 += VR) {
      float acc[MT][NVT][4];
#pragma unroll
      for (int mt = 0; mt < MT; ++mt)
#pragma unroll
        for (int nt = 0; nt < NVT; ++nt)
#pragma unroll
          for (int e = 0; e < 4; ++e) acc[mt][nt][e] = 0.f;
      const bool do_sum = (v0 == 0) && (p.sum != nullptr || p.out != nullptr);
      // stage inside its 128 x 256 tile, and that tile's place
      int in_tile = static_cast<int>(s_begin % kStagesPerTile), tm = tm_begin, tn = tn_begin;
#pragma unroll 1
      for (long long s = s_begin; s < s_end; ++s) {
        // the warps run through the ring independently of one another; lane 0 waits for the warp
        int ok = 1;
        if (lane == 0) ok = mbar_wait(&full_bar[stage], phase, abort_flag, p.err, 132) ? 1 : 0;
        ok = __shfl_sync(0xffffffffu, ok, 0);
        __syncwarp();                    // the shuffle carries the verdict; this orders the stage's bytes for all lanes
        if (!ok) { alive = false; break; }
        const uint32_t st = smem_u32(smem + stage * Cfg::kStageBytes);
        uint32_t a[MT][KS][4];
#pragma unroll
        for (int mt = 0; mt < MT; ++mt)
#pragma unroll
          for (int ks = 0; ks < KS; ++ks) ldsm_x4(st + a_off[mt][ks], a[mt][ks]);
#pragma unroll
        for (int nt = 0; nt < NVT; ++nt)
#pragma unroll
          for (int h = 0; h < KS / 2; ++h) {
            uint32_t b[4];
            ldsm_x4(st + b_off[nt][h], b);
#pragma unroll
            for (int mt = 0; mt < MT; ++mt) {
              mma_bf16_16816(acc[mt][nt], a[mt][2 * h], b[0], b[1]);
              mma_bf16_16816(acc[mt][nt], a[mt][2 * h + 1], b[2], b[3]);
            }
          }
        float t0 = 0.f, t1 = 0.f;
        if (do_sum) {
          // every row of the column-sum accumulator holds the sums of 8 elements of this warp's
          // slice; lane (g, q), g < CW, keeps elements 8g + 2q, 8g + 2q + 1 of its 32 or 64
#pragma unroll
          for (int j = 0; j < CW; ++j) {
            uint32_t t[4];
            float cs[4] = {0.f, 0.f, 0.f, 0.f};
            ldsm_x4_trans(st + t_off[j], t);
            mma_bf16_16816(cs, mask_a[0], t[0], t[1]);
            if (MT == 2) mma_bf16_16816(cs, mask_a[1], t[2], t[3]);
            if (g == j) { t0 = cs[0]; t1 = cs[1]; }
          }
        }
        __syncwarp();
        if (lane == 0) mbar_arrive(&empty_bar[stage]);     // this warp is done with the stage
        if (++stage == kStages) { stage = 0; phase ^= 1; }
        if (do_sum && g < CW) {
          const int e0 = warp * (CW * 8) + g * 8 + q * 2;    // element inside the stage
          float2* at = reinterpret_cast<float2*>(p.sum + s * kMmaCols + e0);
          if (p.sum != nullptr && !(p.sum_init && j0 == 0)) {
            const float2 old = *at;
            t0 += old.x;
            t1 += old.y;
          }
          if (p.out != nullptr && (p.sum == nullptr || j0 + TR >= p.n_grp)) {
            // one stage is kMmaCols / 256 row segments (256 columns each) of one 128 x 256 tile
            const int r = tm * 128 + in_tile * (kMmaCols / 256) + (e0 >> 8);
            const int c = tn * 256 + (e0 & 255);
            if (r < p.m_cols && c < p.n_cols) {
              const long long o = static_cast<long long>(r) * p.n_cols + c;
              const bool rmw = p.out_accumulate || (p.sum == nullptr && j0 > 0);
              const bool pair = (c + 1 < p.n_cols) && ((p.n_cols & 1) == 0);     // o is even then
              t0 *= p.out_scale; t1 *= p.out_scale;
              if (p.out_is_f32) {
                float* dst = static_cast<float*>(p.out) + o;
                if (pair) {
                  float2 v = make_float2(t0, t1);
                  if (rmw) { const float2 old = *reinterpret_cast<const float2*>(dst); v.x += old.x; v.y += old.y; }
                  *reinterpret_cast<float2*>(dst) = v;
                } else {
                  dst[0] = rmw ? dst[0] + t0 : t0;
                  if (c + 1 < p.n_cols) dst[1] = rmw ? dst[1] + t1 : t1;
                }
              } else {
                __nv_bfloat16* dst = static_cast<__nv_bfloat16*>(p.out) + o;
                if (pair) {
                  if (rmw) {
                    const __nv_bfloat162 old = *reinterpret_cast<const __nv_bfloat162*>(dst);
                    t0 += __bfloat162float(old.x); t1 += __bfloat162float(old.y);
                  }
                  *reinterpret_cast<__nv_bfloat162*>(dst) = __floats2bfloat162_rn(t0, t1);
                } else {
                  dst[0] = __float2bfloat16_rn(rmw ? __bfloat162float(dst[0]) + t0 : t0);
                  if (c + 1 < p.n_cols) dst[1] = __float2bfloat16_rn(rmw ? __bfloat162float(dst[1]) + t1 : t1);
                }
              }
            }
          } else {
            *at = make_float2(t0, t1);
          }
        }
        if (++in_tile == kStagesPerTile) {
          in_tile = 0;
          if (++tn == p.n_tiles_n) { tn = 0; ++tm; }
        }
      }
      // the only CTA-wide agreement: every compute warp gets here once per block, aborted or not
      if (!named_bar_and(1, kWarps * 32, alive)) { alive = false; break; }
      // reduce the per-warp [TR train x VR val] partial blocks, one atomic per (v, b) and CTA; two warps may share a slot
      float* mine = s_red + (warp & 7) * (TR * VR);
#pragma unroll
      for (int turn = 0; turn < kWarps / 8; ++turn) {
        if ((warp >> 3) == turn) {
#pragma unroll
          for (int mt = 0; mt < MT; ++mt)
#pragma unroll
            for (int nt = 0; nt < NVT; ++nt)
#pragma unroll
              for (int e = 0; e < 4; ++e) {
                float* slot = mine + Cfg::red_at(nt * 8 + q * 2 + (e & 1), mt * 16 + g + (e >> 1) * 8);
                *slot = turn ? *slot + acc[mt][nt][e] : acc[mt][nt][e];
              }
        }
        named_bar_sync(2, kWarps * 32);
      }
      for (int idx = threadIdx.x; idx < TR * VR; idx += kWarps * 32) {
        float t = 0.f;
#pragma unroll
        for (int w = 0; w < 8; ++w) t += s_red[w * (TR * VR) + Cfg::red_at(idx / TR, idx % TR)];
        const int b = j0 + idx % TR, v = v0 + idx / TR;
        if (v < p.n_val && b < p.n_grp && t != 0.f)
          atomicAdd(&p.M[static_cast<long long>(v) * p.n_train + p.b0 + b], t * p.scale);
      }
      named_bar_sync(2, kWarps * 32);
    }
  }
}

// out[r, c] (= or +=) scale * sum[tile(r, c)][r % 128][c % 256], cast to the parameter dtype
template <typename OutT>
__global__ void tile_sum_finalize_kernel(const float* sum, int n_tiles_n, OutT* __restrict__ out,
                                         int rows, int cols, float scale, int accumulate) {
  stream_order();
  const long long n = static_cast<long long>(rows) * cols;
  for (long long i = blockIdx.x * static_cast<long long>(blockDim.x) + threadIdx.x; i < n;
       i += static_cast<long long>(gridDim.x) * blockDim.x) {
    const int r = static_cast<int>(i / cols), c = static_cast<int>(i % cols);
    const long long tile = static_cast<long long>(r >> 7) * n_tiles_n + (c >> 8);
    float v = sum[tile * kTileElems + (r & 127) * 256 + (c & 255)] * scale;
    if (accumulate) v += static_cast<float>(out[i]);
    out[i] = static_cast<OutT>(v);
  }
}

template <int VR, int KB>
static int launch_tile_dot_f32_t(const void* V, int v_samples, const void* W, int w_samples, long long tiles,
                                 TileDotParams& p, const DeviceState* ds, cudaStream_t st) {
  using Cfg = TdF32Cfg<VR, KB>;
  CUtensorMap tv, tw;
  int rc;
  if ((rc = make_tmap_f32_tiles(&tv, V, tiles, v_samples, v_samples, VR)) != GHOST_OK) return rc;
  if ((rc = make_tmap_f32_tiles(&tw, W, tiles, w_samples, p.n_grp, Cfg::kTrainRows)) != GHOST_OK) return rc;
  static bool attr_set[64] = {};
  if (!attr_set[ds->device]) {
    GB_CUDA_OK(cudaFuncSetAttribute(tile_dot_f32_kernel<VR, KB>, cudaFuncAttributeMaxDynamicSharedMemorySize, Cfg::kSmemBytes));
    attr_set[ds->device] = true;
  }
  long long ctas = static_cast<long long>(ds->sm_count) * Cfg::kCtas;
  if (ctas > p.stages) ctas = p.stages;
  p.stages_per_cta = (p.stages + ctas - 1) / ctas;
  ctas = (p.stages + p.stages_per_cta - 1) / p.stages_per_cta;
  GB_CUDA_OK(launch_next(tile_dot_f32_kernel<VR, KB>, dim3(static_cast<int>(ctas)), dim3(288), Cfg::kSmemBytes, st, tv, tw, p));
  count_launch();
  return post_launch("tile_dot_f32_kernel");
}

// A stage holds as many train rows as the group has, up to the next 8, 16 or 32, and validation rows up to the next 4, 8 or 16:
// the rest would be zeros that are fetched and multiplied (3 + 1 samples of 468 x 128 with 8 + 32 rows: 8.3 us, 5.1).
template <int VR>
static int launch_tile_dot_f32(const void* V, int v_samples, const void* W, int w_samples, long long tiles,
                               TileDotParams& p, const DeviceState* ds, cudaStream_t st) {
  if (p.n_grp <= 8) return launch_tile_dot_f32_t<VR, 1>(V, v_samples, W, w_samples, tiles, p, ds, st);
  if (p.n_grp <= 16) return launch_tile_dot_f32_t<VR, 2>(V, v_samples, W, w_samples, tiles, p, ds, st);
  return launch_tile_dot_f32_t<VR, 4>(V, v_samples, W, w_samples, tiles, p, ds, st);
}

template <int NVT, int MT>
static int launch_tile_dot_mma_t(const void* V, int v_samples, const void* W, int w_samples, long long tiles,
                                 TileDotParams& p, const DeviceState* ds, cudaStream_t st) {
  using Cfg = TdMmaCfg<NVT, MT>;
  CUtensorMap tv, tw;
  int rc;
  // [tiles][samples][32768] seen as [tiles][512 panels][samples][64]: one box = the stage's 8 panels
  if (p.v_per_rank > 0)
    rc = make_tmap_bf16_gathered_tiles(&tv, V, v_samples / p.v_per_rank, tiles, p.v_per_rank, Cfg::kValRows, Cfg::kPanels);
  else
    rc = make_tmap_bf16_blocks(&tv, V, tiles, v_samples, kTileElems, kTileElems, Cfg::kValRows, Cfg::kPanels);
  if (rc != GHOST_OK) return rc;
  if ((rc = make_tmap_bf16_blocks(&tw, W, tiles, w_samples, kTileElems, kTileElems, Cfg::kTrainRows, Cfg::kPanels)) != GHOST_OK)
    return rc;
  static bool attr_set[64] = {};
  if (!attr_set[ds->device]) {
    GB_CUDA_OK(cudaFuncSetAttribute(tile_dot_mma_kernel<NVT, MT>, cudaFuncAttributeMaxDynamicSharedMemorySize, Cfg::kSmemBytes));
    attr_set[ds->device] = true;
  }
  long long ctas = ds->sm_count;
  if (ctas > p.stages) ctas = p.stages;
  p.stages_per_cta = (p.stages + ctas - 1) / ctas;
  ctas = (p.stages + p.stages_per_cta - 1) / p.stages_per_cta;
  GB_CUDA_OK(launch_next(tile_dot_mma_kernel<NVT, MT>, dim3(static_cast<int>(ctas)), dim3((Cfg::kWarps + 1) * 32), Cfg::kSmemBytes, st, tv, tw, p));
  count_launch();
  return post_launch("tile_dot_mma_kernel");
}

template <int NVT>
static int launch_tile_dot_mma(const void* V, int v_samples, const void* W, int w_samples, long long tiles,
                               TileDotParams& p, const DeviceState* ds, cudaStream_t st) {
  if (p.n_grp <= 16) return launch_tile_dot_mma_t<NVT, 1>(V, v_samples, W, w_samples, tiles, p, ds, st);
  return launch_tile_dot_mma_t<NVT, 2>(V, v_samples, W, w_samples, tiles, p, ds, st);
}

// V: [tiles][v_samples][32768] with the validation samples at index v_off..v_off+n_val-1;
// W: [tiles][w_samples][32768] with the group's train samples at index 0..n_grp-1.
// v_per_rank > 0: V holds validation samples only, as an all-gather over ranks leaves them,
// [v_samples / v_per_rank ranks][tiles][v_per_rank][32768] (bf16).
int launch_tile_dot(const void* V, int v_samples, int v_off, const void* W, int w_samples, int is_f32,
                    long long tiles, int n_val, int n_grp, int b0, int n_train, float scale, float* M,
                    float* sum, int sum_init, void* out, int out_is_f32, int out_accumulate, int m_cols,
                    int n_cols, int n_tiles_n, float out_scale, const DeviceState* ds, cudaStream_t st,
                    int v_per_rank) {
  TileDotParams p;
  p.v_off = v_off;
  p.v_per_rank = v_per_rank;
  p.out = out; p.out_is_f32 = out_is_f32; p.out_accumulate = out_accumulate;
  p.m_cols = m_cols; p.n_cols = n_cols; p.n_tiles_n = n_tiles_n; p.out_scale = out_scale;
  p.stages = is_f32 ? static_cast<long long>(m_cols) * n_tiles_n : tiles * (kTileElems / kMmaCols);
  p.stages_per_cta = 0;
  p.n_val = n_val; p.n_grp = n_grp; p.b0 = b0; p.n_train = n_train;
  p.scale = scale; p.M = M; p.sum = sum; p.sum_init = sum_init;
  p.err = ds->err_word;
  if (is_f32 && n_val <= 4) return launch_tile_dot_f32<4>(V, v_samples, W, w_samples, tiles, p, ds, st);
  if (is_f32 && n_val <= 8) return launch_tile_dot_f32<8>(V, v_samples, W, w_samples, tiles, p, ds, st);
  if (is_f32) return launch_tile_dot_f32<16>(V, v_samples, W, w_samples, tiles, p, ds, st);
  if (n_val <= 8) return launch_tile_dot_mma<1>(V, v_samples, W, w_samples, tiles, p, ds, st);
  if (n_val <= 16) return launch_tile_dot_mma<2>(V, v_samples, W, w_samples, tiles, p, ds, st);
  return launch_tile_dot_mma<4>(V, v_samples, W, w_samples, tiles, p, ds, st);
}

int launch_tile_sum_finalize(const float* sum, int n_tiles_n, void* out, int out_is_f32, int rows, int cols,
                             float scale, int accumulate, const DeviceState* ds, cudaStream_t st) {
  const long long n = static_cast<long long>(rows) * cols;
  long long blocks = (n + 255) / 256;
  if (blocks > ds->sm_count * 8) blocks = ds->sm_count * 8;
  if (out_is_f32)
    GB_CUDA_OK(launch_next(tile_sum_finalize_kernel<float>, dim3(static_cast<int>(blocks)), dim3(256), 0, st, sum, n_tiles_n, static_cast<float*>(out), rows, cols, scale, accumulate));
  else
    GB_CUDA_OK(launch_next(tile_sum_finalize_kernel<__nv_bfloat16>, dim3(static_cast<int>(blocks)), dim3(256), 0, st, sum, n_tiles_n, static_cast<__nv_bfloat16*>(out), rows, cols, scale, accumulate));
  count_launch();
  return post_launch("tile_sum_finalize_kernel");
}

}  // namespace gb
