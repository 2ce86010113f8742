// gradproj_fused: per-sample Kronecker-projected weight gradients
//
//   out[b] = scale * (G_b P_r^T)^T (A_b P_c^T)            [k_r, k_c] fp32 per sample
//
// (ghostEngines/gradProjection/autograd_gradproj.py:120-165: for nn.Linear P_r = P_o, P_c = P_i and
// the result is [k_o, k_i]; for HF Conv1D the reference swaps the roles, P_r = P_i, P_c = P_o, and
// the result is [k_i, k_o].)  The activations and output gradients are streamed from HBM exactly
// once: per 128-token chunk the two skinny projections run on tcgen05 (TMA-fed, accumulators in
// TMEM), the projected [128, k] blocks are moved TMEM -> shared memory as fp32, and the small
// k_r x k_c contraction over the chunk's tokens is done in registers by the epilogue warps
// (< 1 % of the flops).  Results go straight into the caller's [B, total_proj_dim] row slices with
// fp32 atomics, so no [B, T, k] intermediate ever reaches HBM.  HBM-bound by design: arithmetic
// intensity is about k flop per byte.  What has to be kept small is the per-stage cost of the two
// single threads that drive the pipeline (a barrier wait, an expect-tx, the TMA and MMA issues --
// each on the order of 100 cycles), hence wide stages and one multi-lane TMA instruction per stage.
//
// The embedding form (kEmb) has token ids in place of A: the rows of P_c^T are gathered by id straight into
// the staged block, out[b] = scale * sum_t (P_r g_t)(P_c[:, id_t])^T, and only G is streamed.
//
// float32 rows, and bf16 rows that TMA cannot read, come through the registers of eight more warps (kSrc), which write
// the swizzled bf16 blocks -- of float32 data value and residual, three products -- so that such operands too are
// read once: copies in parts beforehand moved 16 bytes for every element of four (8 x 4096 tokens of 1024 + 1024
// float32, k = 32: 189 -> 97 us; token table of 1024 float32 features, 16 x 2048 tokens: 107 -> 56 with mma.sync before).
//
// Few (sample, 128-token) units: a unit is one CTA's chain over all columns of G and A, whatever the number of
// tokens in it, so a small batch leaves the GPU idle for the length of that chain.  There (kSome, kWhole) a cluster of
// up to eight CTAs shares a unit: each projects its part of the columns, the partial [128, k] blocks are added through
// distributed shared memory in rank order, and every CTA contracts its share of the tokens (10 tokens of 4407 + 452
// float32, k = 44: 77 -> 22 us; 6 x 54 tokens of 2944 + 6528 bf16, k = 13: 47 -> 15).
//
// Where one CTA or one cluster has all tokens of a sample (up to 128 of them, or gradproj_group) the result is stored, without
// zeroing it before and adding to it: calls of up to 128 tokens are 1.04 to 1.18 times as fast (12 x 1 token
// of 128 + 2112 bf16, k = 44: 18.1 -> 15.6 us with the host's part, 14 x 12 of 1088 + 256 float32 17.8 -> 15.3).
//
// CTA layout: warps 0-3 epilogue, warp 4 TMA producer, warp 5 MMA issuer, warps 6-13 loaders where kSrc asks for them.
#include <atomic>

#include "common.cuh"
#include "sm100_ptx.cuh"

namespace gb {

struct GpParams {
  int B;
  long long T;
  int n_r, n_c;            // contraction lengths: columns of G / of A (already padded & stacked)
  int k_r, k_c;            // projection ranks (rows of P_r / P_c)
  int kr_pad, kc_pad;      // MMA N extents (multiples of 16)
  int chunks_per_sample;
  long long units;         // B * chunks_per_sample
  int units_per_cta;       // base number of units per CTA
  int units_extra;         // the first `units_extra` CTAs take one more
  // register loaders: the operands themselves, and where the residual part of P_r / P_c starts (kSrcF32)
  const void *g, *a;
  long long ldg, lda;
  int lo_r, lo_c;
  int vec_g, vec_a;        // rows on 16-byte (float32) / 8-byte (bf16) boundaries
  int half_g, half_a;      // kSrcMixed: which operand is bf16
  float scale;
  float* out;              // sample b at out + b * out_stride, [k_r, k_c] row-major
  int accumulate;          // added to what is there, which the caller has zeroed or wants
  int direct;              // one CTA or one cluster has all of a sample's units: stored, neither zeroed before nor added to
  int group;               // > 1, with kNone: CTAs of the cluster that has a sample's units
  long long out_stride;
  int out_ld;              // pitch of an output row (k_c, or more inside a wider block)
  // embedding form: token ids [B, T] and the rows that stand for A P_c^T, [vocab, >= k_c] fp32
  const long long* ids;
  const float* rows;
  long long ld_rows;
  int vocab, rows_vec;
  int* err;
};

enum { kNone = 0, kSome = 1, kWhole = 2 };      // a cluster for each unit: no; with others of the sample; which is the sample
enum { kSrcTma = 0, kSrcF32 = 1, kSrcBf16 = 2, kSrcMixed = 3 };      // how the rows of G and A reach shared memory

template <int KMAX, int kSrc, int kCluster>   // KMAX: largest padded rank this instantiation handles (32, 64 or 128)
struct GpCfg {
  static constexpr int BM = 128, BK = 64;                  // BK: one 128-byte swizzle atom of bf16
  static constexpr int PARTS = kSrc == kSrcF32 || kSrc == kSrcMixed ? 2 : 1;    // bf16 parts of an element
  // Columns per pipeline stage = ATOMS * 64.  The single threads that drive the pipeline pay a few
  // hundred cycles per stage for the barrier round trip, so a stage carries two atoms when the
  // shared memory allows it.
  static constexpr int ATOMS = (KMAX == 128 || kSrc != kSrcTma) ? 1 : 2;
  static constexpr int kActAtomBytes = BM * BK * 2;
  static constexpr int kProjAtomBytes = KMAX * BK * 2;
  static constexpr int kStageBytes = ATOMS * PARTS * (kActAtomBytes + kProjAtomBytes);
  // The pipeline is bound by how many bytes are in flight per SM, so the fp32 staging of the
  // projected blocks is kept to half a tile (64 tokens at a time; a cluster's partial blocks are
  // staged whole) and the rest goes to stages: it fills the 227 KB of shared memory.
  static constexpr int kStageRows = kCluster != kNone ? 128 : 64;
  static constexpr int kProjBytes = 2 * kStageRows * KMAX * 4;
  static constexpr int kRoom = (232448 - 1280 - kProjBytes) / kStageBytes;
  static constexpr int kStages = kRoom < 8 ? kRoom : 8;
  static constexpr int kSmemBytes = kStages * kStageBytes + kProjBytes + 1024 + 256;
  static constexpr int kThreads = kSrc == kSrcTma ? 192 : 448;
  static constexpr int RT = KMAX / 16;   // output rows per thread (16 thread rows)
  static constexpr int CT = KMAX / 8;    // output cols per thread (8 thread cols)
};

// Staged fp32 rows are stored with their float4 chunks XOR-permuted by the row index, so that the
// 32 lanes of a warp (32 consecutive rows, same chunk) spread over all banks.
template <int KMAX>
__device__ __forceinline__ int gp_staged_index(int row, int elem) {
  return row * KMAX + ((((elem >> 2) ^ row) & (KMAX / 4 - 1)) << 2) + (elem & 3);
}

// A loader warp's share of a stage, 16 rows of 64 columns, held in registers between its load and its store; nothing looks
// at a loaded value before the store.  float32: lane l has columns 4 (l % 16) .. + 3 of rows l / 16 + 2 i, a vector where
// rows are on its boundaries.  bf16 rows the same way, but element by element where they are not: there a lane has
// columns l and l + 32 of all rows, so that a load of the warp covers neighbouring elements.
template <int kSrc> struct GpRows;
template <> struct GpRows<kSrcF32> {
  float4 v[8];
  // base + at: the warp's first row, column of the stage's first column; `left` columns and `rows` rows from there on
  __device__ __forceinline__ void load(const void* base, long long at, long long ld, int left, long long rows, bool vec, int lane) {
    const int r0 = lane >> 4, c = (lane & 15) * 4, cols = left - c;
    const float* p = static_cast<const float*>(base) + at + r0 * ld + c;
#pragma unroll
    for (int i = 0; i < 8; ++i, p += 2 * ld) {
      const bool in = r0 + 2 * i < rows;
      if (vec) {                           // widths are multiples of four here
        v[i] = in && cols > 0 ? *reinterpret_cast<const float4*>(p) : make_float4(0.f, 0.f, 0.f, 0.f);
      } else {
        v[i].x = in && cols > 0 ? *p : 0.f;
        v[i].y = in && cols > 1 ? p[1] : 0.f;
        v[i].z = in && cols > 2 ? p[2] : 0.f;
        v[i].w = in && cols > 3 ? p[3] : 0.f;
      }
    }
  }
  // into the stage's two [128 rows][64 columns] swizzled blocks; first: the warp's first row in them
  __device__ __forceinline__ void store(uint8_t* block, int lo_bytes, int first, int lane) const {
    const int c = (lane & 15) * 4;
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      const int row = first + (lane >> 4) + 2 * i;
      uint8_t* dst = block + row * 128 + (((c >> 3) ^ (row & 7)) << 4) + (c & 4) * 2;
      const __nv_bfloat162 h0 = __floats2bfloat162_rn(v[i].x, v[i].y), h1 = __floats2bfloat162_rn(v[i].z, v[i].w);
      const __nv_bfloat162 l0 = __floats2bfloat162_rn(v[i].x - __bfloat162float(h0.x), v[i].y - __bfloat162float(h0.y));
      const __nv_bfloat162 l1 = __floats2bfloat162_rn(v[i].z - __bfloat162float(h1.x), v[i].w - __bfloat162float(h1.y));
      *reinterpret_cast<uint2*>(dst) = make_uint2(*reinterpret_cast<const uint32_t*>(&h0), *reinterpret_cast<const uint32_t*>(&h1));
      *reinterpret_cast<uint2*>(dst + lo_bytes) = make_uint2(*reinterpret_cast<const uint32_t*>(&l0), *reinterpret_cast<const uint32_t*>(&l1));
    }
  }
};
// A float32 operand beside a bf16 one, whose elements stay as they are, without a residual.  A form of its own: with
// the type looked at in GpRows<kSrcF32> 10 x 3780 float32 tokens of 782 + 1024 took 149 us instead of 135.
template <> struct GpRows<kSrcMixed> : GpRows<kSrcF32> {
  int form;                // 0 float32; bf16: 1 vectors (bits of two elements each in x and y), 2 elements (one each in x to w)
  __device__ __forceinline__ void load(const void* base, long long at, long long ld, int left, long long rows, bool vec, bool half, int lane) {
    form = !half ? 0 : vec ? 1 : 2;
    if (!half) {
      GpRows<kSrcF32>::load(base, at, ld, left, rows, vec, lane);
      return;
    }
    const int r0 = lane >> 4, c = (lane & 15) * 4, cols = left - c;
    const unsigned short* p = static_cast<const unsigned short*>(base) + at + r0 * ld + c;
#pragma unroll
    for (int i = 0; i < 8; ++i, p += 2 * ld) {
      const bool in = r0 + 2 * i < rows;
      if (vec) {                           // widths are multiples of four here
        const uint2 w = in && cols > 0 ? *reinterpret_cast<const uint2*>(p) : make_uint2(0u, 0u);
        v[i].x = __uint_as_float(w.x);
        v[i].y = __uint_as_float(w.y);
      } else {
        v[i].x = __uint_as_float(in && cols > 0 ? p[0] : 0u);
        v[i].y = __uint_as_float(in && cols > 1 ? p[1] : 0u);
        v[i].z = __uint_as_float(in && cols > 2 ? p[2] : 0u);
        v[i].w = __uint_as_float(in && cols > 3 ? p[3] : 0u);
      }
    }
  }
  __device__ __forceinline__ void store(uint8_t* block, int lo_bytes, int first, int lane) const {
    if (form == 0) {
      GpRows<kSrcF32>::store(block, lo_bytes, first, lane);
      return;
    }
    const int c = (lane & 15) * 4;
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      const int row = first + (lane >> 4) + 2 * i;
      uint8_t* dst = block + row * 128 + (((c >> 3) ^ (row & 7)) << 4) + (c & 4) * 2;
      uint2 w = make_uint2(__float_as_uint(v[i].x), __float_as_uint(v[i].y));
      if (form == 2) w = make_uint2(w.x | w.y << 16, __float_as_uint(v[i].z) | __float_as_uint(v[i].w) << 16);
      *reinterpret_cast<uint2*>(dst) = w;
      *reinterpret_cast<uint2*>(dst + lo_bytes) = make_uint2(0u, 0u);
    }
  }
};
template <> struct GpRows<kSrcBf16> {
  uint32_t v[32];
  bool vec;
  __device__ __forceinline__ void load(const void* base, long long at, long long ld, int left, long long rows, bool by_vector, int lane) {
    const unsigned short* p = static_cast<const unsigned short*>(base) + at;
    vec = by_vector;
    if (vec) {
      const int r0 = lane >> 4, c = (lane & 15) * 4;
#pragma unroll
      for (int i = 0; i < 8; ++i) {
        const bool in = r0 + 2 * i < rows && c < left;         // widths are multiples of four here
        const uint2 w = in ? *reinterpret_cast<const uint2*>(p + (r0 + 2 * i) * ld + c) : make_uint2(0u, 0u);
        v[2 * i] = w.x; v[2 * i + 1] = w.y;
      }
    } else {
#pragma unroll
      for (int i = 0; i < 32; ++i) {
        const int r = i >> 1, c = (i & 1) * 32 + lane;
        v[i] = r < rows && c < left ? p[r * ld + c] : 0u;
      }
    }
  }
  __device__ __forceinline__ void store(uint8_t* block, int, int first, int lane) const {
#pragma unroll
    for (int i = 0; i < 32; ++i) {
      if (vec && i >= 8) break;
      const int row = vec ? first + (lane >> 4) + 2 * i : first + (i >> 1), c = vec ? (lane & 15) * 4 : (i & 1) * 32 + lane;
      uint8_t* dst = block + row * 128 + (((c >> 3) ^ (row & 7)) << 4) + (c & 7) * 2;
      if (vec) *reinterpret_cast<uint2*>(dst) = make_uint2(v[(2 * i) & 31], v[(2 * i + 1) & 31]);
      else *reinterpret_cast<unsigned short*>(dst) = static_cast<unsigned short>(v[i]);
    }
  }
};

__device__ __forceinline__ float4 gp_ld_cluster(uint32_t addr) {
  float4 v;
  asm volatile("ld.shared::cluster.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "r"(addr) : "memory");
  return v;
}

__device__ __forceinline__ float gp_ld_cluster1(uint32_t addr) {
  float v;
  asm volatile("ld.shared::cluster.f32 %0, [%1];" : "=f"(v) : "r"(addr) : "memory");
  return v;
}

template <int KMAX, int kSrc, bool kEmb, int kCluster>
__global__ void __launch_bounds__(kSrc == kSrcTma ? 192 : 448, 1)
gradproj_kernel(const __grid_constant__ CUtensorMap tm_g, const __grid_constant__ CUtensorMap tm_pr,
                const __grid_constant__ CUtensorMap tm_a, const __grid_constant__ CUtensorMap tm_pc,
                const GpParams p) {
  using Cfg = GpCfg<KMAX, kSrc, kCluster>;
  constexpr int BM = Cfg::BM, BK = Cfg::BK, kStages = Cfg::kStages, RT = Cfg::RT, CT = Cfg::CT;
  constexpr int ATOMS = Cfg::ATOMS, PARTS = Cfg::PARTS;

  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  float* s_r = reinterpret_cast<float*>(smem + kStages * Cfg::kStageBytes);   // [kStageRows][KMAX]
  float* s_c = s_r + Cfg::kStageRows * KMAX;                                  // [kStageRows][KMAX]
  uint64_t* bars = reinterpret_cast<uint64_t*>(smem + kStages * Cfg::kStageBytes + Cfg::kProjBytes);
  uint64_t* full_bar = bars;
  uint64_t* empty_bar = bars + kStages;
  uint64_t* acc_full = bars + 2 * kStages;    // [2]
  uint64_t* acc_empty = acc_full + 2;         // [2]
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(acc_empty + 2);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int kb_r = (p.n_r + ATOMS * BK - 1) / (ATOMS * BK);            // pipeline stages over G's columns
  const int kb_total = kEmb ? kb_r : kb_r + (p.n_c + ATOMS * BK - 1) / (ATOMS * BK);
  // units of this CTA and its stages [kb0, kb1) of each: all of them, or in a cluster (one unit) its rank's share
  long long u0, u1;
  int kb0 = 0, kb1 = kb_total;
  uint32_t rank = 0, ranks = 1;
  if constexpr (kCluster != kNone) {
    rank = cluster_ctarank();
    asm("mov.u32 %0, %%cluster_nctarank;" : "=r"(ranks));
    u0 = blockIdx.x / ranks;
    u1 = u0 + 1;
    kb0 = static_cast<int>(rank * kb_total / ranks);
    kb1 = static_cast<int>((rank + 1) * kb_total / ranks);
  } else if (p.group > 1) {
    rank = cluster_ctarank();
    ranks = p.group;
    const long long first = static_cast<long long>(blockIdx.x / ranks) * p.chunks_per_sample;
    u0 = first + static_cast<long long>(rank) * p.chunks_per_sample / ranks;
    u1 = first + static_cast<long long>(rank + 1) * p.chunks_per_sample / ranks;
  } else {
    const long long bx = blockIdx.x;
    u0 = bx * p.units_per_cta + (bx < p.units_extra ? bx : p.units_extra);
    u1 = u0 + p.units_per_cta + (bx < p.units_extra ? 1 : 0);
    if (u1 > p.units) u1 = p.units;
  }

  if (threadIdx.x == 0) {
    for (int s = 0; s < kStages; ++s) { mbar_init(&full_bar[s], kSrc == kSrcTma ? 1 : 9); mbar_init(&empty_bar[s], 1); }
    for (int a = 0; a < 2; ++a) { mbar_init(&acc_full[a], 1); mbar_init(&acc_empty[a], 4); }
    *abort_flag = 0;
    fence_barrier_init();
  }
  if (warp == 5) { tmem_alloc(tmem_slot, 512); tmem_relinquish(); }
  if (warp == 4 && lane == 0) {
    tma_prefetch_desc(&tm_pr);
    if (!kEmb) tma_prefetch_desc(&tm_pc);
    if (kSrc == kSrcTma) { tma_prefetch_desc(&tm_g); if (!kEmb) tma_prefetch_desc(&tm_a); }
  }
  tc_fence_before_sync();
  __syncthreads();
  tc_fence_after_sync();
  const uint32_t tmem_base = *tmem_slot;
  stream_order();

  if (warp == 4) {
    // Producer warp.  Lane 0 owns the barriers; each of the first lanes issues the TMA of one box -- activation
    // atoms (kSrcTma), then projection atoms or, of float32 operands, the two parts of the one atom -- in one
    // warp instruction per stage instead of one thread issuing the boxes back to back.
    constexpr int kActBoxes = kSrc == kSrcTma ? ATOMS : 0, kProjBoxes = ATOMS * PARTS;
    const bool is_p = lane >= kActBoxes;
    const int box = is_p ? lane - kActBoxes : lane;
    const uint32_t dst_off = is_p ? ATOMS * PARTS * Cfg::kActAtomBytes + box * Cfg::kProjAtomBytes
                                  : box * Cfg::kActAtomBytes;
    int stage = 0; uint32_t phase = 0; bool ok = true;
    for (long long u = u0; u < u1 && ok; ++u) {
      const int b = static_cast<int>(u / p.chunks_per_sample);
      const int row0 = static_cast<int>(u % p.chunks_per_sample) * BM;
      for (int kb = kb0; kb < kb1; ++kb) {
        int w = 1;
        if (lane == 0) w = mbar_wait(&empty_bar[stage], phase ^ 1, abort_flag, p.err, 421) ? 1 : 0;
        w = __shfl_sync(0xffffffffu, w, 0);
        if (!w) { ok = false; break; }
        const bool first = kb < kb_r;
        const int kpad = first ? p.kr_pad : p.kc_pad;
        if (lane == 0) mbar_arrive_expect_tx(&full_bar[stage], (kActBoxes * BM + kProjBoxes * kpad) * BK * 2);
        __syncwarp();
        if (lane < kActBoxes + kProjBoxes) {
          // an atom past the last column starts out of range and is zero-filled; what a residual box reads beyond
          // its part meets zeros of the operand
          int col = (first ? kb : kb - kb_r) * ATOMS * BK;
          if (PARTS == 2) col += box == 0 ? 0 : (first ? p.lo_r : p.lo_c);
          else col += box * BK;
          const CUtensorMap* m = first ? (is_p ? &tm_pr : &tm_g) : (is_p ? &tm_pc : &tm_a);
          tma_load_3d(smem + stage * Cfg::kStageBytes + dst_off, m, &full_bar[stage], col,
                      is_p ? 0 : row0, is_p ? 0 : b);
        }
        if (++stage == kStages) { stage = 0; phase ^= 1; }
      }
    }
  } else if (kSrc != kSrcTma && warp >= 6) {
    // Loader warps: 16 rows of a unit each.  The loads of the next stage are in flight while a stage is converted
    // and stored: two register sets.
    if constexpr (kSrc != kSrcTma) {
      const int lw = warp - 6;
      GpRows<kSrc> set[2];
      long long row = 0, rows_left = 0;                  // of the unit being fetched: this warp's first row, rows from there on
      auto fetch = [&](int kb, GpRows<kSrc>& q) {
        const bool first = kb < kb_r;
        const int col = (first ? kb : kb - kb_r) * BK;
        const long long ld = first ? p.ldg : p.lda;
        const void* src = first ? p.g : p.a;
        const int left = (first ? p.n_r : p.n_c) - col;
        const bool vec = first ? p.vec_g : p.vec_a;
        if constexpr (kSrc == kSrcMixed) q.load(src, row * ld + col, ld, left, rows_left, vec, first ? p.half_g : p.half_a, lane);
        else q.load(src, row * ld + col, ld, left, rows_left, vec, lane);
      };
      int stage = 0; uint32_t phase = 0;
      auto put = [&](const GpRows<kSrc>& q) -> bool {
        int w = 1;
        if (lane == 0) w = mbar_wait(&empty_bar[stage], phase ^ 1, abort_flag, p.err, 621) ? 1 : 0;
        w = __shfl_sync(0xffffffffu, w, 0);
        __syncwarp();
        if (!w) return false;
        q.store(smem + stage * Cfg::kStageBytes, Cfg::kActAtomBytes, lw * 16, lane);
        fence_proxy_async_smem();
        __syncwarp();
        if (lane == 0) mbar_arrive(&full_bar[stage]);
        if (++stage == kStages) { stage = 0; phase ^= 1; }
        return true;
      };
      const long long n = (u1 - u0) * (kb1 - kb0);       // this CTA's stages
      long long fu = u0;
      int fk = kb0;
      auto advance = [&](GpRows<kSrc>& q) {
        if (fu >= u1) return;
        if (fk == kb0) {
          const long long b = fu / p.chunks_per_sample, t0 = (fu - b * p.chunks_per_sample) * BM + lw * 16;
          row = b * p.T + t0;
          rows_left = p.T - t0;
        }
        fetch(fk, q);
        if (++fk == kb1) { fk = kb0; ++fu; }
      };
      if (n > 0) advance(set[0]);
      for (long long i = 0; i < n; i += 2) {
        advance(set[1]);
        if (!put(set[0])) break;
        if (i + 1 >= n) break;
        advance(set[0]);
        if (!put(set[1])) break;
      }
    }
  } else if (warp == 5) {
    if (lane == 0) {
      const uint32_t idesc_r = make_idesc_bf16(BM, p.kr_pad, 0, 0);
      const uint32_t idesc_c = make_idesc_bf16(BM, p.kc_pad, 0, 0);
      int stage = 0; uint32_t phase = 0; int acc = 0; uint32_t acc_phase = 0; bool ok = true;
      for (long long u = u0; u < u1 && ok; ++u) {
        if (!mbar_wait(&acc_empty[acc], acc_phase ^ 1, abort_flag, p.err, 522)) { ok = false; break; }
        tc_fence_after_sync();
        const uint32_t d_r = tmem_base + acc * 256;
        const uint32_t d_c = d_r + 128;
        for (int kb = kb0; kb < kb1; ++kb) {
          if (!mbar_wait(&full_bar[stage], phase, abort_flag, p.err, 523)) { ok = false; break; }
          tc_fence_after_sync();
          const uint32_t sa = smem_u32(smem + stage * Cfg::kStageBytes);
          const bool first = kb < kb_r;
          const bool fresh = (kb == kb0) || (kb == kb_r);
          const uint32_t d = first ? d_r : d_c;
          const uint32_t idesc = first ? idesc_r : idesc_c;
#pragma unroll
          for (int at = 0; at < ATOMS; ++at) {
            const uint64_t adesc = make_smem_desc_sw128(sa + at * Cfg::kActAtomBytes, 16, 1024);
            const uint64_t bdesc = make_smem_desc_sw128(sa + ATOMS * PARTS * Cfg::kActAtomBytes + at * Cfg::kProjAtomBytes, 16, 1024);
#pragma unroll
            for (int k = 0; k < BK / 16; ++k) {
              const uint32_t add = (fresh && at == 0 && k == 0) ? 0u : 1u;
              if constexpr (PARTS == 2) {      // residual parts lie behind the values
                umma_bf16(d, adesc + 2 * k + Cfg::kActAtomBytes / 16, bdesc + 2 * k, idesc, add);
                umma_bf16(d, adesc + 2 * k, bdesc + 2 * k + Cfg::kProjAtomBytes / 16, idesc, 1u);
                umma_bf16(d, adesc + 2 * k, bdesc + 2 * k, idesc, 1u);
              } else {
                umma_bf16(d, adesc + 2 * k, bdesc + 2 * k, idesc, add);
              }
            }
          }
          umma_commit(&empty_bar[stage]);
          if (++stage == kStages) { stage = 0; phase ^= 1; }
        }
        if (ok) umma_commit(&acc_full[acc]);
        if (++acc == 2) { acc = 0; acc_phase ^= 1; }
      }
    }
  } else {
    // ------------------------------------------------------------ epilogue: warps 0-3
    const int tid = threadIdx.x;              // 0..127 = token row inside the chunk
    const int ty = tid >> 3, tx = tid & 7;    // 16 x 8 thread grid over the [k_r, k_c] output
    float o[RT][CT];
#pragma unroll
    for (int i = 0; i < RT; ++i)
#pragma unroll
      for (int j = 0; j < CT; ++j) o[i][j] = 0.f;
    int acc = 0; uint32_t acc_phase = 0;
    const uint32_t lane_base = static_cast<uint32_t>(warp * 32) << 16;

    auto flush = [&](int b) {
      float* dst = p.out + static_cast<long long>(b) * p.out_stride;
#pragma unroll
      for (int i = 0; i < RT; ++i) {
        const int r = ty * RT + i;
#pragma unroll
        for (int j = 0; j < CT; ++j) {
          const int c = tx * CT + j;
          if (r < p.k_r && c < p.k_c && o[i][j] != 0.f)
            atomicAdd(dst + static_cast<long long>(r) * p.out_ld + c, o[i][j] * p.scale);
          o[i][j] = 0.f;
        }
      }
    };
    // This CTA, or the cluster, has all of sample b: its block goes through shared memory -- a cluster's through that of the
    // stages, which nothing is on its way to any more -- and each CTA adds up and stores its share, in rank order.
    auto store = [&](int b) {
      float* block = ranks > 1 ? reinterpret_cast<float*>(smem) : s_r;            // [KMAX][KMAX]
#pragma unroll
      for (int i = 0; i < RT; ++i)
#pragma unroll
        for (int j = 0; j < CT; j += 4) {
          *reinterpret_cast<float4*>(&block[(ty * RT + i) * KMAX + tx * CT + j]) = make_float4(o[i][j], o[i][j + 1], o[i][j + 2], o[i][j + 3]);
          o[i][j] = o[i][j + 1] = o[i][j + 2] = o[i][j + 3] = 0.f;
        }
      if (ranks > 1) cluster_sync_all();
      else named_bar_sync(1, 128);
      float* dst = p.out + static_cast<long long>(b) * p.out_stride;
#pragma unroll 1
      for (int e = static_cast<int>(rank) * 128 + tid; e < p.k_r * KMAX; e += static_cast<int>(ranks) * 128) {
        if (e % KMAX >= p.k_c) continue;
        float sum = block[e];
        if (ranks > 1) {
          sum = 0.f;
          for (uint32_t k = 0; k < ranks; ++k) sum += gp_ld_cluster1(map_to_cta(smem_u32(block + e), k));
        }
        dst[static_cast<long long>(e / KMAX) * p.out_ld + e % KMAX] = sum * p.scale;
      }
      if (ranks == 1) named_bar_sync(1, 128);
    };
    // TMEM -> shared (fp32): row `tid` of one projected block
    auto stage_block = [&](uint32_t taddr, int kpad, float* dst) {
#pragma unroll 1
      for (int c0 = 0; c0 < kpad; c0 += 32) {
        uint32_t r[32];
        tmem_ld32(taddr + c0, r);
        tmem_ld_wait();
#pragma unroll
        for (int j = 0; j < 32; j += 4)
          if (c0 + j < KMAX)
            *reinterpret_cast<float4*>(&dst[gp_staged_index<KMAX>(tid & (Cfg::kStageRows - 1), c0 + j)]) =
                make_float4(__uint_as_float(r[j]), __uint_as_float(r[j + 1]), __uint_as_float(r[j + 2]), __uint_as_float(r[j + 3]));
      }
    };

    // embedding form: row `tid` of the gathered block, fetched while the tensor core still works on the
    // unit; a token past the end or with an id outside the table contributes zeros
    constexpr int kRowQuads = kEmb ? KMAX / 4 : 1;
    float4 mine[kRowQuads];
    auto gather = [&](int b, long long t) {
      long long id = -1;
      if (t < p.T) {
        id = p.ids[static_cast<long long>(b) * p.T + t];
        if (id < 0 || id >= p.vocab) { id = -1; atomicExch(p.err, kErrBadIndex); }
      }
      const float* src = p.rows + (id < 0 ? 0 : id) * p.ld_rows;
#pragma unroll
      for (int q = 0; q < kRowQuads; ++q) {
        mine[q] = make_float4(0.f, 0.f, 0.f, 0.f);
        if (id < 0 || 4 * q >= p.k_c) continue;
        if (p.rows_vec) {
          mine[q] = *reinterpret_cast<const float4*>(src + 4 * q);
        } else {
          mine[q].x = src[4 * q];
          if (4 * q + 1 < p.k_c) mine[q].y = src[4 * q + 1];
          if (4 * q + 2 < p.k_c) mine[q].z = src[4 * q + 2];
          if (4 * q + 3 < p.k_c) mine[q].w = src[4 * q + 3];
        }
      }
    };

    // out[r, c] += sum over staged rows [t0, t1) of s_r[t][r] * s_c[t][c]
    auto contract = [&](int t0, int t1) {
#pragma unroll 4
      for (int t = t0; t < t1; ++t) {
        float rr[RT], cc[CT];
        if constexpr (RT >= 4) {
#pragma unroll
          for (int i = 0; i < RT; i += 4)
            *reinterpret_cast<float4*>(&rr[i]) = *reinterpret_cast<const float4*>(&s_r[gp_staged_index<KMAX>(t, ty * RT + i)]);
        } else {
          *reinterpret_cast<float2*>(&rr[0]) = *reinterpret_cast<const float2*>(&s_r[gp_staged_index<KMAX>(t, ty * RT)]);
        }
#pragma unroll
        for (int j = 0; j < CT; j += 4)
          *reinterpret_cast<float4*>(&cc[j]) = *reinterpret_cast<const float4*>(&s_c[gp_staged_index<KMAX>(t, tx * CT + j)]);
#pragma unroll
        for (int i = 0; i < RT; ++i)
#pragma unroll
          for (int j = 0; j < CT; ++j) o[i][j] = fmaf(rr[i], cc[j], o[i][j]);
      }
    };

    if constexpr (kCluster != kNone) {
      // One unit.  Row `tid` of this CTA's partial blocks is staged; rows [first, first + share) of all CTAs' blocks are
      // then added up here, in place: nobody else reads them from this CTA.
      const int most = (BM + static_cast<int>(ranks) - 1) / static_cast<int>(ranks), first = static_cast<int>(rank) * most;
      const int share = first + most < BM ? most : BM - first;
      const int b = static_cast<int>(u0 / p.chunks_per_sample);
      const long long t_first = u0 % p.chunks_per_sample * BM;
      const bool owned = tid >= first && tid < first + share;
      if constexpr (kEmb) { if (owned) gather(b, t_first + tid); }
      bool alive = true;
      if (kb1 > kb0) alive = named_bar_and(2, 128, mbar_wait(&acc_full[0], 0, abort_flag, p.err, 124));
      if (alive) {
        tc_fence_after_sync();
        const uint32_t t_r = tmem_base + lane_base;
        if (kb0 < kb_r && kb0 < kb1) stage_block(t_r, p.kr_pad, s_r);
        if (!kEmb && kb1 > kb_r) stage_block(t_r + 128, p.kc_pad, s_c);
        if constexpr (kEmb) {
          if (owned)
#pragma unroll
            for (int q = 0; q < kRowQuads; ++q) *reinterpret_cast<float4*>(&s_c[gp_staged_index<KMAX>(tid, 4 * q)]) = mine[q];
        }
      }
      cluster_sync_all();
      if (alive) {
        // ranks [0, last_r] hold columns of G, [first_c, ranks) columns of A
        auto begin = [&](int r) { return static_cast<int>(static_cast<unsigned>(r) * kb_total / ranks); };
        auto add_up = [&](float* block, int kpad, bool of_r) {
          const int quads = kpad / 4;
          for (int i = tid; i < share * quads; i += 128) {
            float* at = &block[gp_staged_index<KMAX>(first + i / quads, i % quads * 4)];
            float4 sum = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll 4
            for (int r = 0; r < static_cast<int>(ranks); ++r) {
              const int s0 = begin(r), s1 = begin(r + 1);
              if (s0 == s1 || (of_r ? s0 >= kb_r : s1 <= kb_r)) continue;
              const float4 v = gp_ld_cluster(map_to_cta(smem_u32(at), r));
              sum.x += v.x; sum.y += v.y; sum.z += v.z; sum.w += v.w;
            }
            *reinterpret_cast<float4*>(at) = sum;
          }
        };
        add_up(s_r, p.kr_pad, true);
        if (!kEmb) add_up(s_c, p.kc_pad, false);
        named_bar_sync(1, 128);
        contract(first, first + share);
        if constexpr (kCluster == kSome) flush(b);
      }
      if constexpr (kCluster == kWhole) store(b);
    }
    // (one place that stores or adds and no wide counters: with two places the embedding form of float32 and unaligned rows spilled
    // more registers, 237 us for 16 x 2048 tokens of 4000 float32, k = 64, and 200 as it is; 65 and 59 for 701)
    if constexpr (kCluster == kNone) {
      bool alive = true;
      int b = static_cast<int>(u0 / p.chunks_per_sample);
      int chunk = static_cast<int>(u0 % p.chunks_per_sample);
      // a cluster's CTA without a unit takes part in the storing too
#pragma unroll 1
      for (long long left = u1 - u0; left > 0 || p.group > 1; --left) {
        if (left > 0) {
          if constexpr (kEmb) gather(b, static_cast<long long>(chunk) * BM + tid);
          if (!named_bar_and(2, 128, mbar_wait(&acc_full[acc], acc_phase, abort_flag, p.err, 124))) { alive = false; break; }
          tc_fence_after_sync();
          const uint32_t t_r = tmem_base + lane_base + acc * 256;
          // two halves of 64 tokens: warps 0-1 own TMEM lanes 0-63, warps 2-3 lanes 64-127
#pragma unroll 1
          for (int half = 0; half < 2; ++half) {
            if ((warp >> 1) == half) {
              stage_block(t_r, p.kr_pad, s_r);
              if constexpr (kEmb) {
#pragma unroll
                for (int q = 0; q < kRowQuads; ++q)
                  *reinterpret_cast<float4*>(&s_c[gp_staged_index<KMAX>(tid & 63, 4 * q)]) = mine[q];
              } else {
                stage_block(t_r + 128, p.kc_pad, s_c);
              }
              tc_fence_before_sync();
              __syncwarp();
              if (lane == 0) mbar_arrive(&acc_empty[acc]);     // four arrivals per tile, one per warp
            }
            named_bar_sync(1, 128);                            // the four epilogue warps only
            contract(0, Cfg::kStageRows);
            named_bar_sync(1, 128);
          }
          if (++acc == 2) { acc = 0; acc_phase ^= 1; }
        }
        if (++chunk == p.chunks_per_sample || left <= 1) {     // done with the sample, or with this CTA's part of it
          if (p.direct) store(b);
          else flush(b);
          if (p.group > 1) break;
          chunk = 0;
          ++b;
        }
      }
      if (!alive && p.group > 1) cluster_sync_all();           // the one that the others wait at in store()
    }
  }

  if (kCluster != kNone || p.group > 1) {
    if (warp >= 4) {
      if constexpr (kCluster != kNone) cluster_sync_all();        // the epilogue's barrier before the partial blocks are added up
      if (kCluster != kSome) cluster_sync_all();                  // and the one before the results are
    }
    cluster_sync_all();                    // no CTA leaves while another reads its blocks
  }
  tc_fence_before_sync();
  __syncthreads();
  if (warp == 5) { tc_fence_after_sync(); tmem_dealloc(tmem_base, 512); }
}

template <int KMAX, int kSrc, bool kEmb, int kCluster>
static int launch_gradproj_t(const CUtensorMap& tg, const CUtensorMap& tpr, const CUtensorMap& ta, const CUtensorMap& tpc,
                             GpParams& p, int ranks, const DeviceState* ds, cudaStream_t st) {
  using Cfg = GpCfg<KMAX, kSrc, kCluster>;
  static bool attr_set[64] = {};
  if (!attr_set[ds->device]) {
    GB_CUDA_OK(cudaFuncSetAttribute(gradproj_kernel<KMAX, kSrc, kEmb, kCluster>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                    Cfg::kSmemBytes));
    attr_set[ds->device] = true;
  }
  cudaLaunchConfig_t cfg = {};
  cudaLaunchAttribute attr[2];
  cfg.attrs = attr;
  cfg.numAttrs = early_start(attr, st);
  cfg.blockDim = dim3(Cfg::kThreads, 1, 1);
  cfg.dynamicSmemBytes = Cfg::kSmemBytes;
  cfg.stream = st;
  if (kCluster != kNone || p.group > 1) {
    cudaLaunchAttribute& cluster = attr[cfg.numAttrs++];
    cluster.id = cudaLaunchAttributeClusterDimension;
    cluster.val.clusterDim.x = ranks;
    cluster.val.clusterDim.y = 1;
    cluster.val.clusterDim.z = 1;
    cfg.gridDim = dim3(static_cast<unsigned>((kCluster != kNone ? p.units : p.B) * ranks), 1, 1);
  } else {
    const int grid = static_cast<int>(p.units < ds->sm_count ? p.units : ds->sm_count);
    p.units_per_cta = static_cast<int>(p.units / grid);
    p.units_extra = static_cast<int>(p.units % grid);
    cfg.gridDim = dim3(grid, 1, 1);
  }
  GB_CUDA_OK(cudaLaunchKernelEx(&cfg, gradproj_kernel<KMAX, kSrc, kEmb, kCluster>, tg, tpr, ta, tpc, p));
  count_launch();
  return post_launch("gradproj_kernel");
}

// Clusters of `ranks` CTAs of this kernel that are resident at once, as the driver counts them: a cluster stays inside a GPC,
// whose SMs differ from device to device.  (On a 148-SM device 15 of eight, 22 of six, 33 of four, 45 of three; one more of them and
// the call takes two rounds: 17.5 us against 32.1 for 48 x 100 tokens of 640 + 640, k = 40, in threes.)
template <int KMAX, int kSrc, bool kEmb, int kCluster>
static int gradproj_resident(int ranks, const DeviceState* ds) {
  using Cfg = GpCfg<KMAX, kSrc, kCluster>;
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
    cfg.blockDim = dim3(Cfg::kThreads, 1, 1);
    cfg.dynamicSmemBytes = Cfg::kSmemBytes;
    cfg.attrs = &attr;
    cfg.numAttrs = 1;
    int count = 0;
    if (cudaFuncSetAttribute(gradproj_kernel<KMAX, kSrc, kEmb, kCluster>, cudaFuncAttributeMaxDynamicSharedMemorySize, Cfg::kSmemBytes) != cudaSuccess ||
        cudaOccupancyMaxActiveClusters(&count, gradproj_kernel<KMAX, kSrc, kEmb, kCluster>, &cfg) != cudaSuccess) {
      (void)cudaGetLastError();
      return 0;                              // no cluster for this call; the next one asks again
    }
    n = count + 1;
    slot.store(n, std::memory_order_relaxed);
  }
  return n - 1;
}

// CTAs that share a unit: as many as are resident with one unit per cluster.
// * Short chains of small ranks stay alone: the cluster's barriers and the exchange cost about 2 us, a stage is 0.5 us of a unit's
//   chain, the contraction, which the CTAs share too, 1 us at 32 x 32 and 3 at 64 x 64 (32 x 64 tokens of 256 + 256 columns, four
//   stages, k = 32: 10.3 us alone, 11.3 in pairs; 12 x 1 token of 128 + 2112, k = 44: 23.6 alone, 13.1 in eights).
// * Three or six share unevenly, which pays from so many stages on (17 x 60 of 640 + 640, ten stages: 13.9 us in fours, 14.8 in sixes;
//   20 x 100 of 9792 + 4160 bf16 21.0 and 16.9; 9 x 464 of the same float32 154 in pairs, 109 in threes).
// * Fives lost (24 units of 32 stages: 26.3 us, 24.7 in fours).
template <int KMAX, int kSrc, bool kEmb>
static int gradproj_ranks(long long units, int stages, const DeviceState* ds) {
  if ((stages < 8 && KMAX <= 32) || 2 * units > ds->sm_count) return 1;
  for (const int r : {8, 6, 4, 3, 2}) {
    if ((r == 6 && stages < 18) || (r == 3 && stages < 8)) continue;
    if (r * units <= ds->sm_count && units <= gradproj_resident<KMAX, kSrc, kEmb, kSome>(r, ds)) return r;
  }
  return 1;
}

// CTAs of a cluster that takes all units of a sample and stores its result, or 1: units dealt over the GPU, results added to zeros.
// A cluster saves the launch that zeroes and the additions (embedding form of bf16: 4 x 796 tokens of 192 11.6 -> 9.1 us; 12 x 900 of
// 256 + 512 11.0 -> 10.7).  It is taken where
// * each of its CTAs has a unit at most and all clusters are resident (16 x 2048 of 1024, embedding form, in eights: 36 us against 20);
// * a quarter of the SMs stays free: with the GPU full of units clusters come up later than CTAs do (64 x 256 of 768 + 768: 14.7
//   against 14.2; 64 x 300 of 512, embedding form, 15.2 and 14.8).
// The largest that fits: its CTAs share the storing (16 x 250 of 320 + 320, two units a sample: 10.8 in eights, 11.2 in pairs).
template <int KMAX, int kSrc, bool kEmb>
static int gradproj_group(int B, int chunks, const DeviceState* ds) {
  if (chunks == 1 || 4ll * B * chunks > 3ll * ds->sm_count) return 1;
  for (int c = 8; c > 1 && c >= chunks; c /= 2)
    if (c * B <= ds->sm_count && B <= gradproj_resident<KMAX, kSrc, kEmb, kNone>(c, ds)) return c;
  return 1;
}

// Operands of one projection as the entry points get them.
struct GpOperands {
  const void *G, *A;               // A null: the embedding form
  int is_f32;                      // 2: only G is, 3: only A
  long long ldg, lda;
  const void *P_r, *P_c;
  long long ldpr, ldpc;
  int pr_cols, pc_cols;            // columns of the P matrices that belong to the operand's (padded) columns
};

template <int KMAX, int kSrc, bool kEmb>
static int launch_gradproj_src(const GpOperands& o, GpParams& p, const DeviceState* ds, cudaStream_t st) {
  constexpr int kCols = GpCfg<KMAX, kSrc, kNone>::ATOMS * 64;
  const int stages = ceil_div(p.n_r, kCols) + (kEmb ? 0 : ceil_div(p.n_c, kCols));
  const int ranks = gradproj_ranks<KMAX, kSrc, kEmb>(p.units, stages, ds);
  p.group = ranks > 1 || p.accumulate ? 1 : gradproj_group<KMAX, kSrc, kEmb>(p.B, p.chunks_per_sample, ds);
  // a sample's tokens are one CTA's or one cluster's: the results are stored, else added to zeros (written before the host
  // is busy with the tensor maps)
  p.direct = !p.accumulate && (p.chunks_per_sample == 1 || p.group > 1);
  int rc;
  const size_t row = static_cast<size_t>(p.k_r) * p.k_c * sizeof(float);
  if (!p.accumulate && !p.direct) {
    if (p.out_stride * sizeof(float) != row) GB_CUDA_OK(cudaMemset2DAsync(p.out, p.out_stride * sizeof(float), 0, row, p.B, st));
    else if ((rc = clear_ahead(p.out, row * p.B, st)) != GHOST_OK) return rc;
  }
  CUtensorMap tg = {}, tpr, ta = {}, tpc = {};
  // the projection matrices as one-sample 3-D operands, so that one TMA instruction form serves all four
  if ((rc = make_tmap_bf16_3d(&tpr, o.P_r, 1, p.k_r, o.pr_cols, o.ldpr, p.kr_pad)) != GHOST_OK) return rc;
  if (!kEmb && (rc = make_tmap_bf16_3d(&tpc, o.P_c, 1, p.k_c, o.pc_cols, o.ldpc, p.kc_pad)) != GHOST_OK) return rc;
  if (kSrc == kSrcTma) {
    if ((rc = make_tmap_bf16_3d(&tg, o.G, p.B, p.T, p.n_r, o.ldg, 128)) != GHOST_OK) return rc;
    if (!kEmb && (rc = make_tmap_bf16_3d(&ta, o.A, p.B, p.T, p.n_c, o.lda, 128)) != GHOST_OK) return rc;
  }
  // (as one form with the test inside, those that add came out up to 4 % slower)
  if (ranks > 1 && p.direct) return launch_gradproj_t<KMAX, kSrc, kEmb, kWhole>(tg, tpr, ta, tpc, p, ranks, ds, st);
  if (ranks > 1) return launch_gradproj_t<KMAX, kSrc, kEmb, kSome>(tg, tpr, ta, tpc, p, ranks, ds, st);
  return launch_gradproj_t<KMAX, kSrc, kEmb, kNone>(tg, tpr, ta, tpc, p, p.group, ds, st);
}

template <int kSrc, bool kEmb>
static int launch_gradproj_k(const GpOperands& o, GpParams& p, const DeviceState* ds, cudaStream_t st) {
  const int kmax = p.kr_pad > p.kc_pad ? p.kr_pad : p.kc_pad;
  if (kmax <= 32) return launch_gradproj_src<32, kSrc, kEmb>(o, p, ds, st);
  if constexpr (!kEmb && kSrc == kSrcTma) { if (kmax > 64) return launch_gradproj_src<128, kSrc, kEmb>(o, p, ds, st); }
  return launch_gradproj_src<64, kSrc, kEmb>(o, p, ds, st);
}

// Chooses how the rows are read: bf16 through TMA where it can, else through registers
template <bool kEmb>
static int launch_gradproj(const GpOperands& o, GpParams& p, const DeviceState* ds, cudaStream_t st) {
  p.kr_pad = (p.k_r + 15) / 16 * 16;
  p.kc_pad = (p.k_c + 15) / 16 * 16;
  const long long chunks = (p.T + 127) / 128;
  GB_REQUIRE(chunks < (1ll << 31) && chunks * p.B < (1ll << 31) * 128, "gradproj: too many tokens");
  p.chunks_per_sample = static_cast<int>(chunks);
  p.units = chunks * p.B;
  p.g = o.G; p.a = o.A; p.ldg = o.ldg; p.lda = o.lda;
  p.err = ds->err_word;
  auto aligned = [](const void* x, long long ld, long long bytes, long long elem) {
    return (reinterpret_cast<uintptr_t>(x) % bytes) == 0 && ld * elem % bytes == 0;
  };
  if (o.is_f32) {
    p.half_g = o.is_f32 == 3;
    p.half_a = o.is_f32 == 2;
    p.vec_g = (p.half_g ? aligned(o.G, o.ldg, 8, 2) : aligned(o.G, o.ldg, 16, 4)) && p.n_r % 4 == 0;
    p.vec_a = (p.half_a ? aligned(o.A, o.lda, 8, 2) : aligned(o.A, o.lda, 16, 4)) && p.n_c % 4 == 0;
    if constexpr (!kEmb) {
      if (o.is_f32 != 1) return launch_gradproj_k<kSrcMixed, kEmb>(o, p, ds, st);
    }
    return launch_gradproj_k<kSrcF32, kEmb>(o, p, ds, st);
  }
  if (aligned(o.G, o.ldg, 16, 2) && (kEmb || aligned(o.A, o.lda, 16, 2)) && p.T < (1ll << 31) - 128)
    return launch_gradproj_k<kSrcTma, kEmb>(o, p, ds, st);
  p.vec_g = aligned(o.G, o.ldg, 8, 2) && p.n_r % 4 == 0;
  p.vec_a = aligned(o.A, o.lda, 8, 2) && p.n_c % 4 == 0;
  return launch_gradproj_k<kSrcBf16, kEmb>(o, p, ds, st);
}

}  // namespace gb

using namespace gb;

static int gradproj_dense(const GpOperands& o, GpParams& p, long long out_stride, void* stream) {
  const DeviceState* ds = device_state();
  if (!ds) return GHOST_ERR_DEVICE;
  GB_REQUIRE(o.G && o.A && o.P_r && o.P_c && p.out, "ghost_gradproj_dense_bf16: null pointer");
  GB_REQUIRE(p.B > 0 && p.T > 0 && p.n_r > 0 && p.n_c > 0 && p.k_r > 0 && p.k_c > 0, "ghost_gradproj_dense_bf16: empty dimension");
  GB_REQUIRE(p.k_r <= 128 && p.k_c <= 128, "ghost_gradproj_dense_bf16: projection ranks above 128 are not supported");
  GB_REQUIRE(out_stride >= static_cast<long long>(p.k_r) * p.k_c, "ghost_gradproj_dense_bf16: out_stride smaller than k_r * k_c");
  GB_REQUIRE(p.T < (1ll << 31) - 128, "ghost_gradproj_dense_bf16: T too large");
  GB_REQUIRE(o.ldg >= p.n_r && o.lda >= p.n_c, "ghost_gradproj_dense_bf16: pitch smaller than the row it holds");
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  p.out_stride = out_stride;
  p.out_ld = p.k_c;
  return launch_gradproj<false>(o, p, ds, st);
}

// G: [B, T, n_r] bf16 (pitch ldg), A: [B, T, n_c] bf16 (pitch lda), P_r: [k_r, n_r] bf16 (pitch ldpr),
// P_c: [k_c, n_c] bf16 (pitch ldpc).  out + b * out_stride receives [k_r, k_c] fp32 (overwritten).
extern "C" int ghost_gradproj_dense_bf16(const void* G, const void* A, int B, long long T, int n_r, int n_c,
                                         long long ldg, long long lda, const void* P_r, const void* P_c,
                                         int k_r, int k_c, long long ldpr, long long ldpc, float scale,
                                         float* out, long long out_stride, void* stream) {
  GB_REQUIRE(((reinterpret_cast<uintptr_t>(G) | reinterpret_cast<uintptr_t>(A)) & 15u) == 0 && ldg % 8 == 0 && lda % 8 == 0,
             "ghost_gradproj_dense_bf16: operands must be 16-byte aligned with pitches that are multiples of 8");
  GpParams p = {};
  p.B = B; p.T = T; p.n_r = n_r; p.n_c = n_c; p.k_r = k_r; p.k_c = k_c; p.scale = scale; p.out = out;
  const GpOperands o = {G, A, 0, ldg, lda, P_r, P_c, ldpr, ldpc, n_r, n_c};
  return gradproj_dense(o, p, out_stride, stream);
}

extern "C" int ghost_gradproj_dense(const void* G, const void* A, int is_f32, int B, long long T, int n_r, int n_c, long long ldg,
                                    long long lda, const void* P_r, const void* P_c, int k_r, int k_c, long long ldpr,
                                    long long ldpc, int lo_r, int lo_c, float scale, float* out, long long out_stride,
                                    void* stream) {
  GB_REQUIRE(is_f32 >= 0 && is_f32 <= 3, "ghost_gradproj_dense: is_f32 must be 0 to 3");
  GB_REQUIRE(n_r <= ldpr && n_c <= ldpc && ldpr % 8 == 0 && ldpc % 8 == 0, "ghost_gradproj_dense: bad layout of the projection matrices");
  GB_REQUIRE(!is_f32 || (lo_r % 8 == 0 && lo_c % 8 == 0 && lo_r >= n_r && lo_c >= n_c && lo_r + n_r <= ldpr && lo_c + n_c <= ldpc),
             "ghost_gradproj_dense: float32 operands need the residual parts of the projection matrices inside their rows");
  GpParams p = {};
  p.B = B; p.T = T; p.n_r = n_r; p.n_c = n_c; p.k_r = k_r; p.k_c = k_c; p.scale = scale; p.out = out;
  p.lo_r = lo_r; p.lo_c = lo_c;
  // The loaders' threads leave the epilogue 128 registers, which a block of 128 x 128 does not fit: 32 x 2048 tokens of
  // 1024 + 1024 float32 took 639 us against 462 for copies of the operands in three parts.
  GB_REQUIRE(k_r <= 64 && k_c <= 64, "ghost_gradproj_dense: projection ranks above 64 are left to ghost_gradproj_dense_bf16");
  const GpOperands o = {G, A, is_f32, ldg, lda, P_r, P_c, ldpr, ldpc, static_cast<int>(ldpr), static_cast<int>(ldpc)};
  return gradproj_dense(o, p, out_stride, stream);
}

extern "C" int ghost_gradproj_embedding(const long long* ids, const void* G, int g_is_f32, int B, long long T,
                                        int d, long long ldg, const void* P_o, long long ldp_o, int p_cols,
                                        int p_lo_offset, const float* P_i_t, long long ld_pit, int vocab, int k_o,
                                        int k_i, float scale, int accumulate, float* out, long long out_stride,
                                        int out_ld, void* stream) {
  const DeviceState* ds = device_state();
  if (!ds) return GHOST_ERR_DEVICE;
  GB_REQUIRE(ids && G && P_o && P_i_t && out, "ghost_gradproj_embedding: null pointer");
  GB_REQUIRE(B > 0 && T > 0 && d > 0 && vocab > 0, "ghost_gradproj_embedding: empty dimension");
  GB_REQUIRE(k_o >= 1 && k_o <= 64 && k_i >= 1 && k_i <= 64,
             "ghost_gradproj_embedding: k_o and k_i must be between 1 and 64 (got %d, %d)", k_o, k_i);
  GB_REQUIRE(ldg >= d && ld_pit >= k_i && out_ld >= k_i &&
                 out_stride >= static_cast<long long>(k_o - 1) * out_ld + k_i,
             "ghost_gradproj_embedding: pitch smaller than the row it holds");
  GB_REQUIRE(accumulate || out_ld == k_i,
             "ghost_gradproj_embedding: a block inside wider rows (out_ld > k_i) must be zeroed by the caller "
             "and passed with accumulate = 1");
  GB_REQUIRE(p_cols >= d && p_cols % 8 == 0 && ldp_o % 8 == 0 && ldp_o >= p_cols &&
                 (reinterpret_cast<uintptr_t>(P_o) & 15u) == 0,
             "ghost_gradproj_embedding: P_o must be 16-byte aligned bf16 with columns padded to a multiple of 8");
  GB_REQUIRE(!g_is_f32 || (p_lo_offset % 8 == 0 && p_lo_offset >= p_cols && p_lo_offset + p_cols <= ldp_o),
             "ghost_gradproj_embedding: float out-grads need the residual part of P_o inside its rows");
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  GpParams p = {};
  p.accumulate = accumulate ? 1 : 0;
  p.B = B; p.T = T; p.n_r = d; p.k_r = k_o; p.k_c = k_i; p.scale = scale;
  p.out = out; p.out_stride = out_stride; p.out_ld = out_ld;
  p.lo_r = p_lo_offset;
  p.ids = ids; p.rows = P_i_t; p.ld_rows = ld_pit; p.vocab = vocab;
  p.rows_vec = k_i % 4 == 0 && ld_pit % 4 == 0 && (reinterpret_cast<uintptr_t>(P_i_t) & 15u) == 0;
  const GpOperands o = {G, nullptr, g_is_f32, ldg, 0, P_o, nullptr, ldp_o, 0, g_is_f32 ? static_cast<int>(ldp_o) : p_cols, 0};
  return launch_gradproj<true>(o, p, ds, st);
}
