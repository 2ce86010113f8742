// ghost_gram: the fused "ghost" dot-product kernel for Linear / Conv1D weights.
//
//   M[v, b] = sum_{t in sample b} sum_{s in sample v} (A_t . A_s) * (G_t . G_s)
//
// which is the Frobenius product of the per-sample weight gradients of train sample b and
// validation sample v (replaces the two GEMMs, the Hadamard product and the reductions of
// ghostEngines/supported_layers_grad_samplers_dotprod.py:119-130 and :416-437).  Train tokens are
// the M dimension, validation tokens the N dimension, and there are two contraction dimensions:
// d_in for the activation Gram and d_out for the output-gradient Gram.  Both 128 x BN Gram tiles
// are accumulated in tensor memory by tcgen05.mma, multiplied element-wise and reduced by the
// epilogue warps straight out of TMEM; the Gram matrices never exist in HBM.
//
// CTA layout (192 threads, persistent over tiles):
//   warps 0-3  epilogue: tcgen05.ld both accumulators, Hadamard, segmented reduce, atomicAdd to M
//   warp  4    TMA producer (one elected lane)
//   warp  5    TMEM allocator + MMA issuer (one elected lane)
// Pipeline: kStages shared-memory stages (train tile 128xBK + val tile BNxBK bf16 in 64-element atoms, 128B swizzle),
// full/empty mbarriers per stage, acc_full/acc_empty mbarriers per accumulator buffer.
#include <atomic>

#include "common.cuh"
#include "gram_operands.cuh"
#include "launch_rules.h"
#include "sm100_ptx.cuh"

namespace gb {

struct GramParams {
  long long rows_t;   // n_train * T
  long long rows_v;   // n_val * T
  long long T;
  int n_train, n_val;
  int ka, kg;         // contraction lengths (elements) of the activation / out-grad operands
  int m_tiles, n_tiles;
  int ranks;          // CTAs that share a tile
  int round_mode;     // 0: fp32 product of fp32 Grams; 1: round Grams and product to bf16
  float scale;
  float* M;           // [n_val, n_train]
  int* err;
};

// PARTS = 2: float32 rows as two bf16 parts, three products per K step into the same accumulator; a stage holds both
// parts of 64 K elements.  (Parts stacked along K, three per operand, fetched the values twice.)
template <int BN, int PARTS>
struct GramCfg {
  static constexpr int BM = 128;
  static constexpr int kAtomK = 64;                        // K elements of one 128-byte swizzle atom
  // K elements per stage.  BN = 128: two atoms per operand (64 KB stages), so the issuing thread
  // does one barrier round trip per eight MMAs; BN = 256 keeps one atom (48 KB stages), two would
  // leave room for two stages only.
  static constexpr int BK = (BN == 256 || PARTS == 2) ? 64 : 128;
  static constexpr int kStageBytes = (BM + BN) * BK * 2 * PARTS;
  static constexpr int kStages = (BN == 256) ? 4 : 3;
  static constexpr int kAccBufs = 512 / (2 * BN);          // 1 (BN=256) or 2 (BN=128)
  static constexpr int kSmemBytes = kStages * kStageBytes + 1024 /*align*/ + 256 /*barriers*/;
};

// Adds the sums of a warp's 32 rows for validation sample v, one addition per train sample among them: lane l takes in lane l + o
// while that is a row of the same sample (rows are ascending).  A share of the columns is a sixteenth or less of a tile, so a row a lane
// adds as many times more often to the same few sums: with one addition per row, where a warp holds two samples, 12 + 6 x 83 bf16 tokens
// of 1792 + 64 took 22.8 us in four CTAs a tile, 15.3 alone and 13.8 so; 6 + 4 x 111 of 1344 + 798 25.4, 17.5 and 17.3.
struct GramRows {
  int b;                   // this lane's train sample, -1: none
  uint32_t same;           // bit i: lane + 2^i has it too
  bool first;              // of the sample's lanes
  __device__ __forceinline__ GramRows(const GramParams& p, long long row) {
    const int lane = threadIdx.x & 31;
    b = row < p.rows_t ? static_cast<int>(row / p.T) : -1;
    same = 0;
#pragma unroll
    for (int i = 0; i < 5; ++i) {
      const int other = __shfl_down_sync(0xffffffffu, b, 1 << i);
      same |= static_cast<uint32_t>(lane + (1 << i) < 32 && other == b) << i;
    }
    const int before = __shfl_up_sync(0xffffffffu, b, 1);
    first = b >= 0 && (lane == 0 || before != b);
  }
  __device__ __forceinline__ void flush(const GramParams& p, float val, int v) const {
    if (v >= p.n_val) return;
#pragma unroll
    for (int i = 0; i < 5; ++i) {
      const float other = __shfl_down_sync(0xffffffffu, val, 1 << i);
      if (same >> i & 1) val += other;
    }
    if (first) atomicAdd(&p.M[static_cast<long long>(v) * p.n_train + b], val * p.scale);
  }
};

__device__ __forceinline__ float gram_product(const GramParams& p, float x, float y) {
  return p.round_mode == 0 ? x * y : bf16_round(bf16_round(x) * bf16_round(y));
}

// Four columns of an accumulator, summed in rank order over the CTAs of `mask`; the loads of all eight go out together
__device__ __forceinline__ float4 gram_cluster_sum(const uint8_t* at, uint32_t mask) {
  float4 v[8], sum = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
  for (int r = 0; r < 8; ++r)
    if (mask >> r & 1) v[r] = ld_cluster_v4(map_to_cta(smem_u32(at), r));
#pragma unroll
  for (int r = 0; r < 8; ++r)
    if (mask >> r & 1) { sum.x += v[r].x; sum.y += v[r].y; sum.z += v[r].z; sum.w += v[r].w; }
  return sum;
}

// The columns of share `part` of `parts` of a tile whose partial accumulators lie in the cluster's shared memory ([column / 4][row][4] floats,
// the activations' accumulator before the gradients'); a row a thread,
// at which `smem` points.
template <int BM, int BN>
__device__ __forceinline__ void gram_split(const GramParams& p, const uint8_t* smem, uint32_t has_a, uint32_t has_g, int part, int parts,
                                           long long row, long long n0) {
  const GramRows rows(p, row);
  const int quads = static_cast<int>((p.rows_v - n0 < BN ? p.rows_v - n0 : BN) + 3) / 4;
  const int q0 = quads * part / parts, q1 = quads * (part + 1) / parts;
  if (q0 == q1) return;
  int v = static_cast<int>((n0 + 4 * q0) / p.T);
  long long boundary = static_cast<long long>(v + 1) * p.T - n0;       // tile-relative column
  float sum = 0.f;
  for (int q = q0; q < q1; ++q) {
    const float4 a = gram_cluster_sum(smem + q * BM * 16, has_a);
    const float4 g = gram_cluster_sum(smem + (BN / 4 + q) * BM * 16, has_g);
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      if (4 * q + e == boundary) {
        rows.flush(p, sum, v++);
        sum = 0.f;
        boundary += p.T;
      }
      sum += gram_product(p, e == 0 ? a.x : e == 1 ? a.y : e == 2 ? a.z : a.w, e == 0 ? g.x : e == 1 ? g.y : e == 2 ? g.z : g.w);
    }
  }
  rows.flush(p, sum, v);
}

// In a cluster the partial accumulators are laid out, fetched and multiplied by sixteen warps: with four, whose loads from
// the other CTAs' shared memory wait on one another, it took 2 us longer.
constexpr int gram_threads(bool split) { return split ? 512 : 192; }

// SPLIT: a cluster shares a tile.  Its CTAs take equal runs of the K steps of both operands, lay their partial accumulators out in
// the shared memory that the stages leave free, and each sums, multiplies and reduces its share of the columns over
// the cluster (gram_split).  A tile alone is bound by what one SM has in flight, 0.53 us a step of 128 K elements whatever
// the rest of the GPU does (0.61 a step of 64 in two parts): 4 + 2 x 64 tokens of 768 -> 20000 are two tiles, 97.3 us on two CTAs and
// 27.6 on sixteen; float32 216 and 52.  The sums of the partial accumulators are rounded, where the tensor core's truncate.
template <int BN, int PARTS, bool SPLIT>
__global__ void __launch_bounds__(gram_threads(SPLIT), 1)
ghost_gram_kernel(const __grid_constant__ CUtensorMap tm_at, const __grid_constant__ CUtensorMap tm_av,
                  const __grid_constant__ CUtensorMap tm_gt, const __grid_constant__ CUtensorMap tm_gv,
                  const GramParams p) {
  using Cfg = GramCfg<BN, PARTS>;
  static_assert(PARTS == 1 || BN == 128, "two parts of wider tiles leave two stages");
  static_assert(!SPLIT || 2 * 128 * BN * 4 <= Cfg::kStages * Cfg::kStageBytes, "partial accumulators lie in the stages");
  constexpr int BM = Cfg::BM, BK = Cfg::BK, kStages = Cfg::kStages, kAccBufs = Cfg::kAccBufs;

  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  uint64_t* bars = reinterpret_cast<uint64_t*>(smem + kStages * Cfg::kStageBytes);
  uint64_t* full_bar = bars;                         // [kStages]
  uint64_t* empty_bar = bars + kStages;              // [kStages]
  uint64_t* acc_full = bars + 2 * kStages;           // [kAccBufs]
  uint64_t* acc_empty = acc_full + kAccBufs;         // [kAccBufs]
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(acc_empty + kAccBufs);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);

  const int warp = threadIdx.x >> 5;
  const int lane = threadIdx.x & 31;
  const int num_tiles = p.m_tiles * p.n_tiles;
  // Tiles are walked in bands of kBandM train tiles: inside a band the train index runs fastest, so
  // the ~148 tiles in flight at any time cover a near-square (train x val) patch and every operand
  // slice is fetched from HBM about once per patch and then shared through the L2.
  constexpr int kBandM = 16;
  auto tile_coords = [&](int tile, int& tm, int& tn) {
    const int band = tile / (kBandM * p.n_tiles);
    const int first = band * kBandM;
    const int rows = (p.m_tiles - first < kBandM) ? p.m_tiles - first : kBandM;
    const int local = tile - band * kBandM * p.n_tiles;
    tm = first + local % rows;
    tn = local / rows;
  };
  const int kb_a = (p.ka + BK - 1) / BK;
  const int kb_total = kb_a + (p.kg + BK - 1) / BK;
  const int ranks = SPLIT ? p.ranks : 1;                   // CTAs of a tile
  const int rank = SPLIT ? static_cast<int>(cluster_ctarank()) : 0;
  auto k_first = [&](int r) { return SPLIT ? static_cast<int>(static_cast<long long>(kb_total) * r / ranks) : r * kb_total; };
  const int kb0 = k_first(rank), kb1 = k_first(rank + 1);
  const int tile0 = SPLIT ? blockIdx.x / ranks : blockIdx.x, tile_step = SPLIT ? num_tiles : gridDim.x;    // a cluster has one tile

  if (threadIdx.x == 0) {
    for (int s = 0; s < kStages; ++s) {
      mbar_init(&full_bar[s], 1);
      mbar_init(&empty_bar[s], 1);
    }
    for (int a = 0; a < kAccBufs; ++a) {
      mbar_init(&acc_full[a], 1);
      mbar_init(&acc_empty[a], 4);   // one arrival per epilogue warp
    }
    *abort_flag = 0;
    fence_barrier_init();
  }
  if (warp == 5) {
    tmem_alloc(tmem_slot, 512);
    tmem_relinquish();
  }
  if (warp == 4 && lane == 0) {
    tma_prefetch_desc(&tm_at);
    tma_prefetch_desc(&tm_av);
    tma_prefetch_desc(&tm_gt);
    tma_prefetch_desc(&tm_gv);
  }
  tc_fence_before_sync();
  __syncthreads();
  tc_fence_after_sync();
  const uint32_t tmem_base = *tmem_slot;
  stream_order();

  if (warp == 4) {
    // ------------------------------------------------------------------ TMA producer
    if (lane == 0) {
      int stage = 0;
      uint32_t phase = 0;
      bool ok = true;
      for (int tile = tile0; tile < num_tiles && ok; tile += tile_step) {
        int tm, tn;
        tile_coords(tile, tm, tn);
        const int m0 = tm * BM;
        const int n0 = tn * BN;
        for (int kb = kb0; kb < kb1; ++kb) {
          if (!mbar_wait(&empty_bar[stage], phase ^ 1, abort_flag, p.err, 401)) { ok = false; break; }
          uint8_t* st = smem + stage * Cfg::kStageBytes;
          mbar_arrive_expect_tx(&full_bar[stage], Cfg::kStageBytes);
          // stage layout: train atoms, then validation atoms; an atom past the end of K is
          // zero-filled by the bounds check
          const CUtensorMap* mt = (kb < kb_a) ? &tm_at : &tm_gt;
          const CUtensorMap* mv = (kb < kb_a) ? &tm_av : &tm_gv;
          const int k0 = ((kb < kb_a) ? kb : kb - kb_a) * BK;
          if constexpr (PARTS == 2) {
            tma_load_3d(st, mt, &full_bar[stage], k0, m0, 0);
            tma_load_3d(st + BM * BK * 4, mv, &full_bar[stage], k0, n0, 0);
          }
#pragma unroll
          for (int a = 0; a < (PARTS == 2 ? 0 : BK / Cfg::kAtomK); ++a) {
            tma_load_2d(st + a * (BM * Cfg::kAtomK * 2), mt, &full_bar[stage], k0 + a * Cfg::kAtomK, m0);
            tma_load_2d(st + BM * BK * 2 + a * (BN * Cfg::kAtomK * 2), mv, &full_bar[stage],
                        k0 + a * Cfg::kAtomK, n0);
          }
          if (++stage == kStages) { stage = 0; phase ^= 1; }
        }
      }
    }
  } else if (warp == 5) {
    // ------------------------------------------------------------------ MMA issuer
    if (lane == 0) {
      constexpr uint32_t idesc = make_idesc_bf16(BM, BN, 0, 0);
      int stage = 0;
      uint32_t phase = 0;
      int acc = 0;
      uint32_t acc_phase = 0;
      bool ok = true;
      for (int tile = tile0; tile < num_tiles && ok; tile += tile_step) {
        if (!mbar_wait(&acc_empty[acc], acc_phase ^ 1, abort_flag, p.err, 502)) { ok = false; break; }
        tc_fence_after_sync();
        const uint32_t d_a = tmem_base + acc * (2 * BN);
        const uint32_t d_g = d_a + BN;
        for (int kb = kb0; kb < kb1; ++kb) {
          if (!mbar_wait(&full_bar[stage], phase, abort_flag, p.err, 503)) { ok = false; break; }
          tc_fence_after_sync();
          const uint32_t sa = smem_u32(smem + stage * Cfg::kStageBytes);
          const bool first = (kb == kb0) || (kb == kb_a);
          const uint32_t dst = (kb < kb_a) ? d_a : d_g;
#pragma unroll
          for (int a = 0; a < BK / Cfg::kAtomK; ++a) {
            const uint64_t adesc = make_smem_desc_sw128(sa + a * (BM * Cfg::kAtomK * 2), 16, 1024);
            const uint64_t bdesc = make_smem_desc_sw128(sa + BM * BK * 2 * PARTS + a * (BN * Cfg::kAtomK * 2), 16, 1024);
#pragma unroll
            for (int k = 0; k < Cfg::kAtomK / 16; ++k) {
              const uint32_t add = (first && a == 0 && k == 0) ? 0u : 1u;
              if constexpr (PARTS == 2) {      // residual parts lie behind the values
                umma_bf16(dst, adesc + 2 * k + BM * BK * 2 / 16, bdesc + 2 * k, idesc, add);
                umma_bf16(dst, adesc + 2 * k, bdesc + 2 * k + BN * BK * 2 / 16, idesc, 1u);
                umma_bf16(dst, adesc + 2 * k, bdesc + 2 * k, idesc, 1u);
              } else {
                umma_bf16(dst, adesc + 2 * k, bdesc + 2 * k, idesc, add);
              }
            }
          }
          umma_commit(&empty_bar[stage]);   // frees the stage once these MMAs have read it
          if (++stage == kStages) { stage = 0; phase ^= 1; }
        }
        if (ok) umma_commit(&acc_full[acc]);
        if (++acc == kAccBufs) { acc = 0; acc_phase ^= 1; }
      }
    }
  } else if constexpr (SPLIT) {
    if (warp < 4) mbar_wait_warp(&acc_full[0], 0, abort_flag, p.err, 104);
  } else {
    // ------------------------------------------------------------------ epilogue (warps 0-3)
    int acc = 0;
    uint32_t acc_phase = 0;
    const uint32_t lane_base = static_cast<uint32_t>(warp * 32) << 16;
    for (int tile = blockIdx.x; tile < num_tiles; tile += gridDim.x) {
      int tm, tn;
      tile_coords(tile, tm, tn);
      const long long m0 = static_cast<long long>(tm) * BM;
      const long long n0 = static_cast<long long>(tn) * BN;
      if (!mbar_wait_warp(&acc_full[acc], acc_phase, abort_flag, p.err, 104)) break;
      tc_fence_after_sync();

      const long long row = m0 + threadIdx.x;
      const bool row_ok = row < p.rows_t;
      const int b = row_ok ? static_cast<int>(row / p.T) : -1;
      // rows are ascending, so the warp covers one train sample iff its first and last rows agree
      const int b_first = __shfl_sync(0xffffffffu, b, 0);
      const int b_last = __shfl_sync(0xffffffffu, b, 31);
      const bool warp_uniform = (b_first == b_last) && (b_first >= 0);

      int cur_v = static_cast<int>(n0 / p.T);
      long long boundary = static_cast<long long>(cur_v + 1) * p.T - n0;   // tile-relative column
      float sum = 0.f;
      const uint32_t t_a = tmem_base + lane_base + acc * (2 * BN);
      const uint32_t t_g = t_a + BN;

      // (Not GramRows: 15 + 2 x 47 tokens of 64 + 192 bf16 9.4 us so, 9.6 with a structure in place of what a lambda captures; sums per
      // sample of the warp cost small T up to 0.9 us.)
      auto flush = [&](float val, int v) {
        if (v >= p.n_val) return;
        val *= p.scale;
        if (warp_uniform) {
#pragma unroll
          for (int o = 16; o > 0; o >>= 1) val += __shfl_xor_sync(0xffffffffu, val, o);
          if (lane == 0) atomicAdd(&p.M[static_cast<long long>(v) * p.n_train + b_first], val);
        } else if (row_ok) {
          atomicAdd(&p.M[static_cast<long long>(v) * p.n_train + b], val);
        }
      };

#pragma unroll 1
      for (int c0 = 0; c0 < BN; c0 += 32) {
        uint32_t ra[32], rg[32];
        tmem_ld32(t_a + c0, ra);
        tmem_ld32(t_g + c0, rg);
        tmem_ld_wait();
        if (c0 + 32 <= boundary) {
          if (p.round_mode == 0) {
#pragma unroll
            for (int j = 0; j < 32; ++j) sum = fmaf(__uint_as_float(ra[j]), __uint_as_float(rg[j]), sum);
          } else {
#pragma unroll
            for (int j = 0; j < 32; ++j)
              sum += bf16_round(bf16_round(__uint_as_float(ra[j])) * bf16_round(__uint_as_float(rg[j])));
          }
        } else {
#pragma unroll
          for (int j = 0; j < 32; ++j) {
            if (c0 + j == boundary) {
              flush(sum, cur_v);
              sum = 0.f;
              ++cur_v;
              boundary += p.T;
            }
            sum += gram_product(p, __uint_as_float(ra[j]), __uint_as_float(rg[j]));
          }
        }
      }
      // every TMEM read of this tile is done: hand the accumulator back before the atomics
      tc_fence_before_sync();
      __syncwarp();
      if (lane == 0) mbar_arrive(&acc_empty[acc]);
      flush(sum, cur_v);
      if (++acc == kAccBufs) { acc = 0; acc_phase ^= 1; }
    }
  }

  if constexpr (SPLIT) {
    __syncthreads();                                       // the accumulators are complete, the stages free
    tc_fence_after_sync();
    int tm, tn;
    tile_coords(tile0, tm, tn);
    const int row = threadIdx.x & 127, grp = threadIdx.x >> 7;         // a lane of tensor memory is read by warps of its quarter
    const long long m0 = static_cast<long long>(tm) * BM, n0 = static_cast<long long>(tn) * BN;
    if (*abort_flag == 0) {
      const uint32_t t_acc = tmem_base + (static_cast<uint32_t>(row & 96) << 16);
#pragma unroll 1
      for (int c0 = grp * 32; c0 < 2 * BN; c0 += 128) {    // the activations' accumulator, then the gradients'
        if ((c0 < BN ? kb0 >= kb_a : kb1 <= kb_a) || (c0 & (BN - 1)) >= p.rows_v - n0) continue;
        uint32_t r[32];
        tmem_ld32(t_acc + c0, r);
        tmem_ld_wait();
#pragma unroll
        for (int q = 0; q < 8; ++q)
          st_shared_v4(smem + ((c0 / 4 + q) * BM + row) * 16, r[4 * q], r[4 * q + 1], r[4 * q + 2], r[4 * q + 3]);
      }
    }
    tc_fence_before_sync();
    cluster_sync_all();
    uint32_t has_a = 0, has_g = 0;                         // CTAs with a partial of either accumulator
    for (int r = 0; r < ranks; ++r) {
      has_a |= static_cast<uint32_t>(k_first(r) < kb_a) << r;
      has_g |= static_cast<uint32_t>(k_first(r + 1) > kb_a) << r;
    }
    gram_split<BM, BN>(p, smem + row * 16, has_a, has_g, rank * 4 + grp, ranks * 4, m0 + row, n0);
    cluster_sync_all();                                    // no CTA leaves while another still reads its shared memory
  }

  // ------------------------------------------------------------------ teardown
  tc_fence_before_sync();
  __syncthreads();
  if (warp == 5) {
    tc_fence_after_sync();
    tmem_dealloc(tmem_base, 512);
  }
}

static int gram_map(CUtensorMap* t, const GramOperands& o, const void* base, long long rows, int k, long long ld, int box_rows) {
  return o.parts == 2 ? make_tmap_bf16_part_rows(t, base, o.part_rows, rows, ld, box_rows)
                      : make_tmap_bf16_2d(t, base, rows, k, ld, box_rows);
}
int gram_maps(CUtensorMap (&t)[4], const GramOperands& o, long long rows_t, long long rows_v, int box_t, int box_v) {
  int rc;
  if ((rc = gram_map(&t[0], o, o.a_t, rows_t, o.ka, o.ld_at, box_t)) != GHOST_OK) return rc;
  if ((rc = gram_map(&t[1], o, o.a_v, rows_v, o.ka, o.ld_av, box_v)) != GHOST_OK) return rc;
  if ((rc = gram_map(&t[2], o, o.g_t, rows_t, o.kg, o.ld_gt, box_t)) != GHOST_OK) return rc;
  return gram_map(&t[3], o, o.g_v, rows_v, o.kg, o.ld_gv, box_v);
}

template <int BN, int PARTS, bool SPLIT>
static int gram_smem_attr(const DeviceState* ds) {
  static bool attr_set[64] = {};
  if (!attr_set[ds->device]) {
    GB_CUDA_OK(cudaFuncSetAttribute(ghost_gram_kernel<BN, PARTS, SPLIT>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                    GramCfg<BN, PARTS>::kSmemBytes));
    attr_set[ds->device] = true;
  }
  return GHOST_OK;
}

// Clusters of `ranks` CTAs that the device holds at a time (the driver's count, asked once per device and size), or 0
template <int PARTS>
static int gram_resident(int ranks, const DeviceState* ds) {
  static std::atomic<int> known[64][9];      // count + 1; several threads may find the same
  std::atomic<int>& slot = known[ds->device][ranks];
  int n = slot.load(std::memory_order_relaxed);
  if (n == 0) {
    cudaLaunchConfig_t cfg = {};
    cudaLaunchAttribute attr;
    attr.id = cudaLaunchAttributeClusterDimension;
    attr.val.clusterDim.x = ranks;
    attr.val.clusterDim.y = attr.val.clusterDim.z = 1;
    cfg.gridDim = dim3(ranks, 1, 1);
    cfg.blockDim = dim3(gram_threads(true), 1, 1);
    cfg.dynamicSmemBytes = GramCfg<128, PARTS>::kSmemBytes;
    cfg.attrs = &attr;
    cfg.numAttrs = 1;
    int count = 0;
    if (gram_smem_attr<128, PARTS, true>(ds) != GHOST_OK ||
        cudaOccupancyMaxActiveClusters(&count, ghost_gram_kernel<128, PARTS, true>, &cfg) != cudaSuccess) {
      (void)cudaGetLastError();
      return 0;                              // no cluster for this call; the next one asks again
    }
    n = count + 1;
    slot.store(n, std::memory_order_relaxed);
  }
  return n - 1;
}

// CTAs that share a tile of 128 x 128
template <int PARTS>
static int gram_ranks(long long rows_t, long long rows_v, int ka, int kg, const DeviceState* ds) {
  using Cfg = GramCfg<128, PARTS>;
  const long long tiles = static_cast<long long>(ceil_div(rows_t, Cfg::BM)) * ceil_div(rows_v, 128);
  return gram_cluster(tiles, ceil_div(ka, Cfg::BK) + ceil_div(kg, Cfg::BK), ds->sm_count, [&](int r) { return gram_resident<PARTS>(r, ds); });
}

template <int BN, int PARTS>
static int launch_gram(const GramOperands& o, int n_train, int n_val, long long T, int round_mode, float scale, float* M,
                       const DeviceState* ds, cudaStream_t stream) {
  using Cfg = GramCfg<BN, PARTS>;
  GramParams p;
  p.rows_t = static_cast<long long>(n_train) * T;
  p.rows_v = static_cast<long long>(n_val) * T;
  p.T = T;
  p.n_train = n_train;
  p.n_val = n_val;
  p.ka = o.ka;
  p.kg = o.kg;
  p.m_tiles = ceil_div(p.rows_t, Cfg::BM);
  p.n_tiles = ceil_div(p.rows_v, BN);
  p.round_mode = round_mode;
  p.scale = scale;
  p.M = M;
  p.err = ds->err_word;
  CUtensorMap t[4];
  int rc = gram_maps(t, o, p.rows_t, p.rows_v, Cfg::BM, BN);
  if (rc != GHOST_OK) return rc;
  const long long tiles = static_cast<long long>(p.m_tiles) * p.n_tiles;
  p.ranks = 1;
  if constexpr (BN == 128) {
    p.ranks = gram_ranks<PARTS>(p.rows_t, p.rows_v, p.ka, p.kg, ds);
    if (p.ranks > 1) {
      if ((rc = gram_smem_attr<BN, PARTS, true>(ds)) != GHOST_OK) return rc;
      GB_CUDA_OK(launch_next_cluster(dim3(p.ranks), ghost_gram_kernel<BN, PARTS, true>, dim3(static_cast<int>(tiles) * p.ranks), dim3(gram_threads(true)),
                                     Cfg::kSmemBytes, stream, t[0], t[1], t[2], t[3], p));
      count_launch();
      return post_launch("ghost_gram_kernel");
    }
  }
  if ((rc = gram_smem_attr<BN, PARTS, false>(ds)) != GHOST_OK) return rc;
  const int grid = static_cast<int>(tiles < ds->sm_count ? tiles : ds->sm_count);
  GB_CUDA_OK(launch_next(ghost_gram_kernel<BN, PARTS, false>, dim3(grid), dim3(gram_threads(false)), Cfg::kSmemBytes, stream, t[0], t[1], t[2], t[3], p));
  count_launch();
  return post_launch("ghost_gram_kernel");
}

// 0: single-CTA kernels only; 1: CTA-pair kernel for problems with at least 512 train tokens and 256
// to 8192 validation tokens (where it measured faster: 1474 against 1339 TFLOP/s with 32768 x 4096
// tokens, 985 against 1117 with 131072 x 16384); 2: CTA-pair kernel from 512 x 256 tokens up
static int g_gram_pair_mode = 1;
bool xty_pair_usable(const DeviceState* ds);     // a cluster of two ~198 KB CTAs fits on the device

// Validation columns of a tile of one CTA, 128 or 256, or 0: tiles of 256 x 256 on CTA pairs.
// Rounds of tiles over the GPU times the cycles of a K step of a tile (128 for 256 x 256 on a pair and 128 x 256 on one
// SM, 64 for 128 x 128, a tenth more for its operand traffic): 2048 x 1024 tokens are 32 tiles of 256 x 256 on 74
// pairs, and 128 of 128 x 128 on 148 SMs.
static int gram_tile(int parts, long long rows_t, long long rows_v, const DeviceState* ds) {
  auto tiles = [&](int bm, int bn) { return ((rows_t + bm - 1) / bm) * ((rows_v + bn - 1) / bn); };
  auto rounds = [](long long n, long long workers) { return static_cast<double>((n + workers - 1) / workers); };
  const double small_tiles = rounds(tiles(128, 128), ds->sm_count) * 70.;
  const bool pair_wanted = g_gram_pair_mode == 2 || (g_gram_pair_mode == 1 && rows_v <= 8192 &&
                                                     rounds(tiles(256, 256), ds->sm_count / 2) * 128. < small_tiles * 1.1);
  if (pair_wanted && rows_v >= 256 && rows_t >= 512 && xty_pair_usable(ds)) return 0;
  return parts == 2 || rows_v <= 128 || small_tiles * 1.1 < rounds(tiles(128, 256), ds->sm_count) * 128. ? 128 : 256;
}

int gram_dot(const GramOperands& o, int n_train, int n_val, long long T, int round_mode, float scale, float* M_out, bool cleared, void* stream) {
  const DeviceState* ds = device_state();
  if (!ds) return GHOST_ERR_DEVICE;
  GB_REQUIRE(o.a_t && o.a_v && o.g_t && o.g_v && M_out, "ghost_gram_dot_bf16: null pointer");
  GB_REQUIRE(n_train > 0, "No training samples to compute dot product, check batch sizes.");
  GB_REQUIRE(n_val > 0 && T > 0 && o.ka > 0 && o.kg > 0, "ghost_gram_dot_bf16: empty dimension");
  GB_REQUIRE(round_mode == 0 || round_mode == 1, "ghost_gram_dot_bf16: round_mode must be 0 or 1");
  GB_REQUIRE(static_cast<long long>(n_train) * T < (1ll << 31) - 256 &&
             static_cast<long long>(n_val) * T < (1ll << 31) - 256,
             "ghost_gram_dot_bf16: more than 2^31 tokens");
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  if (!cleared)
    if (int rc = clear_ahead(M_out, sizeof(float) * static_cast<size_t>(n_val) * n_train, st)) return rc;
  const int bn = gram_tile(o.parts, static_cast<long long>(n_train) * T, static_cast<long long>(n_val) * T, ds);
  if (bn == 0) return launch_gram_pair(o, n_train, n_val, T, round_mode, scale, M_out, ds, st);
  if (o.parts == 2) return launch_gram<128, 2>(o, n_train, n_val, T, round_mode, scale, M_out, ds, st);
  if (bn == 128) return launch_gram<128, 1>(o, n_train, n_val, T, round_mode, scale, M_out, ds, st);
  return launch_gram<256, 1>(o, n_train, n_val, T, round_mode, scale, M_out, ds, st);
}

}  // namespace gb

extern "C" int ghost_gram_cluster_size(int parts, int n_train, int n_val, long long T, int ka, int kg) {
  using namespace gb;
  const DeviceState* ds = device_state();
  if (!ds) return GHOST_ERR_DEVICE;
  GB_REQUIRE((parts == 1 || parts == 2) && n_train > 0 && n_val > 0 && T > 0 && ka > 0 && kg > 0, "ghost_gram_cluster_size: bad size");
  const long long rows_t = static_cast<long long>(n_train) * T, rows_v = static_cast<long long>(n_val) * T;
  if (gram_tile(parts, rows_t, rows_v, ds) != 128) return 1;
  return parts == 2 ? gram_ranks<2>(rows_t, rows_v, ka, kg, ds) : gram_ranks<1>(rows_t, rows_v, ka, kg, ds);
}

extern "C" int ghost_set_gram_pair_mode(int mode) {
  if (mode < 0 || mode > 2) return GHOST_ERR_INVALID;
  gb::g_gram_pair_mode = mode;
  return GHOST_OK;
}

extern "C" int ghost_gram_dot_bf16(const void* a_train, const void* a_val, const void* g_train,
                                   const void* g_val, int n_train, int n_val, long long T, int ka,
                                   int kg, long long ld_at, long long ld_av, long long ld_gt,
                                   long long ld_gv, int round_mode, float scale, float* M_out,
                                   void* stream) {
  const gb::GramOperands o = {a_train, a_val, g_train, g_val, ld_at, ld_av, ld_gt, ld_gv, ka, kg, 1, 0};
  return gb::gram_dot(o, n_train, n_val, T, round_mode, scale, M_out, false, stream);
}

extern "C" int ghost_gram_dot_parts(const void* A, const void* G, int parts, int n_train, int n_val, long long T, int d, int p,
                                    long long ld_a, long long ld_g, int round_mode, float scale, float* M_out, void* stream) {
  using namespace gb;
  GB_REQUIRE(A && G, "ghost_gram_dot_parts: null pointer");
  GB_REQUIRE(parts == 1 || parts == 2, "ghost_gram_dot_parts: one or two parts");
  GB_REQUIRE(n_train > 0, "No training samples to compute dot product, check batch sizes.");
  GB_REQUIRE(n_val > 0 && T > 0 && d > 0 && p > 0 && ld_a >= d && ld_g >= p, "ghost_gram_dot_parts: bad dimensions");
  return gram_dot(gram_operands(A, G, parts, n_train, n_val, T, d, p, ld_a, ld_g), n_train, n_val, T, round_mode, scale, M_out, false, stream);
}
