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
// float32 rows, and bf16 rows that TMA cannot read, come through shared memory as they are (kSrc): eight or sixteen more warps keep
// 16-byte copies of them on their way and write what has arrived as the swizzled bf16 blocks -- of float32 data value and residual,
// three products -- so that such operands too are read once, and several stages ahead (16 x 2048 tokens of 1024 + 1024 float32,
// k = 32: 99 us with eight warps that loaded into registers, two stages each, 63 so; 4 x 4096 of 2048 + 2049, k = 64: 109 and 94;
// 32 x 3000 of 1001 + 2003 bf16, k = 64, which were copied with padded rows before: 369 and 217; token table of 4000 float32 features,
// 16 x 2048 tokens, k = 64: 198 and 164).  Bound by the latency and the shared-memory traffic of the conversion.  (Those are times from
// cold caches.  With both operands in L2 the way through shared memory is the longer one for rows of a few stages: 16 x 207 of 779 + 256
// float32 13.6 and 14.5, 20 x 638 of 805 + 65, k = 64, 32 and 36, embedding form 7 x 923 of 76 9.8 and 10.7; from cold caches 19.5 and 19.5, 44
// and 42, 16.4 and 16.4.)
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
// CTA layout: warps 0-3 epilogue, warp 4 TMA producer, warp 5 MMA issuer, from warp 6 on 8 or 16 loaders where kSrc asks for them; all of
// them add up a cluster's blocks.
#include <atomic>
#include <type_traits>

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
  // loader warps: the operands themselves, and where the residual part of P_r / P_c starts (kSrcF32, kSrcMixed)
  const void *g, *a;
  long long ldg, lda;
  int lo_r, lo_c;
  int vec_g, vec_a;        // float32: rows on 16-byte boundaries whose width is a multiple of four
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

template <int KMAX, int kSrc, bool kEmb, int kCluster>   // KMAX: largest padded rank this instantiation handles (32, 64 or 128)
struct GpCfg {
  static constexpr int BM = 128, BK = 64;                  // BK: one 128-byte swizzle atom of bf16
  static constexpr bool kLoaders = kSrc != kSrcTma;
  static constexpr int PARTS = kSrc == kSrcF32 || kSrc == kSrcMixed ? 2 : 1;    // bf16 parts of an element
  // Columns per pipeline stage = ATOMS * 64.  The single threads that drive the pipeline pay a few
  // hundred cycles per stage for the barrier round trip, so a stage carries two atoms when the
  // shared memory allows it.
  static constexpr int ATOMS = (KMAX == 128 || kLoaders) ? 1 : 2;
  static constexpr int kActAtomBytes = BM * BK * 2;
  static constexpr int kProjAtomBytes = KMAX * BK * 2;
  static constexpr int kActBytes = ATOMS * PARTS * kActAtomBytes, kProjStageBytes = ATOMS * PARTS * kProjAtomBytes;
  // Activation and projection blocks of a stage lie side by side and arrive together, or, behind loaders, in rings of their
  // own: converted blocks wait for nothing but the tensor core, so two stages of them do, while projection blocks take
  // their time through L2 and the memory goes to rows on their way.
  static constexpr int kStageBytes = kActBytes + (kLoaders ? 0 : kProjStageBytes);
  // The pipeline is bound by how many bytes are in flight per SM, so the fp32 staging of the
  // projected blocks is kept to half a tile (64 tokens at a time; a cluster's partial blocks are
  // staged whole, behind loaders where the stages were) and the rest goes to stages: it fills the 227 KB of shared memory.
  static constexpr int kStageRows = kCluster != kNone ? 128 : 64;
  static constexpr int kProjBytes = kLoaders && kCluster != kNone ? 0 : 2 * kStageRows * KMAX * 4;
  static constexpr int kFree = 232448 - 1280 - kProjBytes;
  static constexpr int kStages = kLoaders ? (PARTS == 2 ? (KMAX == 32 ? 3 : 2) : 5) : kFree / kStageBytes < 8 ? kFree / kStageBytes : 8;
  static constexpr int kProjStages = kLoaders ? 3 : kStages;
  static constexpr int kRings = kStages * kStageBytes + (kLoaders ? kProjStages * kProjStageBytes : 0);
  // Sixteen loader warps, eight to a stage, or eight.  A warp's time for a stage is the latency of its instructions, so two groups take
  // turns (16 x 2048 tokens of 1024 + 1024 float32 77 us with eight, 64 with sixteen; 30 x 1000 of 77 + 1025, k = 64, 77.3 and 69.6), but
  // more threads come up later and leave each fewer registers.  Eight where that is the more, us with eight and with sixteen:
  // * embedding form, whose epilogue holds gathered rows (spills: k = 32 of units alone 10.9 and 13.5; bf16 in clusters, 2 x 142 tokens of 510
  //   7.5 and 8.0, 12 x 546 of 482 11.2 and 11.7), except float32 rows in clusters at k = 32 (8 x 372 of 1042 14.9 and 14.1);
  // * mixed operands at k = 64, units alone (14 x 1658 float32 tokens of 352 and bf16 of 128 38.6 and 39.2, the other way round 36.8 and 38.2).
  // Forms that spill a little with sixteen are the faster ones all the same (k = 64, bf16, units alone: 27 x 1543 of 3521 + 2048 208 and 175).
  static constexpr int kLoaderWarps = !kLoaders ? 0
                                      : kEmb    ? (kSrc == kSrcF32 && KMAX == 32 && kCluster != kNone ? 16 : 8)
                                                : (kSrc == kSrcMixed && KMAX == 64 && kCluster == kNone ? 8 : 16);
  // Rows on their way: a slot is 128 bytes of columns of a loader warp's 16 rows, from the 16-byte boundary before them
  static constexpr int kSlotPitch = 128 + 16, kSlotBytes = 16 * kSlotPitch;
  static constexpr int kSlotsBytes = kLoaderWarps * kSlotBytes;      // a slot of every warp
  static constexpr int kSlots = !kLoaders ? 0 : (kFree - kRings) / kSlotsBytes < 8 ? (kFree - kRings) / kSlotsBytes : 8;
  static constexpr int kSmemBytes = kRings + kSlots * kSlotsBytes + kProjBytes + 1024 + 256;
  static constexpr int kThreads = 192 + 32 * kLoaderWarps;
  static constexpr int RT = KMAX / 16;   // output rows per thread (16 thread rows)
  static constexpr int CT = KMAX / 8;    // output cols per thread (8 thread cols)
  static_assert(!kLoaders || kSlots >= 2, "rows on their way");
  static_assert(!kLoaders || kLoaderWarps / 8 <= kStages, "a stage for each group of loader warps");
  static_assert(!kLoaders || kCluster == kNone || KMAX * KMAX * 4 + 2 * kStageRows * KMAX * 4 <= kRings, "a cluster's blocks lie in the rings");
};

// Staged fp32 rows are stored with their float4 chunks XOR-permuted by the row index, so that the
// 32 lanes of a warp (32 consecutive rows, same chunk) spread over all banks.
template <int KMAX>
__device__ __forceinline__ int gp_staged_index(int row, int elem) {
  return row * KMAX + ((((elem >> 2) ^ row) & (KMAX / 4 - 1)) << 2) + (elem & 3);
}

// Rows of a unit that a loader warp brings: one of every eight, so that short units too are shared by all warps.  Row i lies 8 i rows
// below one of two rows, by the parity of i, which are four rows apart: what is written of two neighbours then lies in different
// banks.  Eight rows are a multiple of 16 bytes whatever their pitch, so that all of one parity begin as far behind a 16-byte boundary.
__device__ __forceinline__ int gp_loader_row(int warp, int i) { return 8 * i + ((warp + 4 * (i & 1)) & 7); }

// `bytes` from `src` (a multiple of 16) on, and zeros up to 16
__device__ __forceinline__ void gp_copy16(uint32_t dst, uintptr_t src, int bytes) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst), "l"(src), "r"(bytes) : "memory");
}

__device__ __forceinline__ void gp_copy16(uint32_t dst, uintptr_t src) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst), "l"(src) : "memory");
}

// One operand's part of a unit: the unit's rows, and of them the columns of the stages of this CTA that a group of loader warps
// fills, every kGroups-th, in slices of 128 bytes
struct GpSegment {
  uintptr_t at;            // first row, first column
  long long pitch;         // bytes from row to row
  long long bytes;         // of a row from there on
  int jump;                // bytes from a stage's last slice to the next one's first
  int rows, slices;        // (the second half of a last float32 stage may hold nothing)
  bool half, vec;          // bf16; float32 rows on 16-byte boundaries with widths that are multiples of four
};

// A lane's 16-byte pieces of a segment's slices: of rows row + 32 j the piece lane % 8, and of row `lane` the ninth, where rows begin behind
// a boundary.  A piece may begin before the row does, but not before the 16 bytes that hold the row's first element, and no byte
// behind the row's last one is read.
template <int kSlotPitch> struct GpAsk {
  uintptr_t c, c8;
  long long step;
  int jump, odd;           // 1 where a stage is two slices
  bool all;                // every row is there
  int n, end, end8, left;  // pieces of the first kind; bytes of the slice's rows from a piece's start on, were all of them whole; slices
  long long bytes;
  __device__ __forceinline__ void open(const GpSegment& x, int warp, int lane) {
    const int i = lane >> 3, row = gp_loader_row(warp, i), q = 16 * (lane & 7), row8 = gp_loader_row(warp, lane & 15);
    const uintptr_t a = x.at + row * x.pitch, a8 = x.at + row8 * x.pitch;
    c = (a & ~uintptr_t(15)) + q;
    c8 = (a8 & ~uintptr_t(15)) + 128;
    step = 32 * x.pitch;
    n = (x.rows - row + 31) >> 5;
    all = x.rows == 128;
    end = static_cast<int>(a & 15) - q;
    end8 = !x.vec && lane < 16 && row8 < x.rows ? static_cast<int>(a8 & 15) - 128 : -128;
    left = x.slices;
    bytes = x.bytes;
    jump = x.jump;
    odd = x.half ? 0 : 1;
  }
  __device__ __forceinline__ void request(uint32_t slot, int lane) {
    const int now = bytes >= 128 ? 128 : bytes > 0 ? static_cast<int>(bytes) : -16;       // nothing: no piece
    const int b8 = now + end8;
    const uint32_t dst = slot + (lane >> 3) * kSlotPitch + 16 * (lane & 7);
    if (all && bytes >= 128) {             // also of a row that begins behind a boundary the first eight pieces are whole
#pragma unroll
      for (int j = 0; j < 4; ++j) gp_copy16(dst + j * 4 * kSlotPitch, c + j * step);
    } else {
      const int b = now + end < 16 ? now + end : 16;
      if (b > 0) {
#pragma unroll
        for (int j = 0; j < 4; ++j)
          if (j < n) gp_copy16(dst + j * 4 * kSlotPitch, c + j * step, b);
      }
    }
    if (b8 > 0) gp_copy16(slot + lane * kSlotPitch + 128, c8, b8);
    const int go = (left & odd) == odd ? jump : 128;     // of two slices the second one has an odd number to go
    c += go;
    c8 += go;
    bytes -= go;
    --left;
  }
};

// Writes an arrived slice into the stage's swizzled [128 rows][64 columns] block, from its column `column` on, and of float32
// rows the residuals into the block `lo` bytes behind it.  `left` bytes of a row are there; columns that are not become
// zeros.  Rows that are not there keep what the block held: nobody reads what the tensor core makes of them.  off: how far behind a 16-byte boundary the lane's rows begin (all of one parity, gp_loader_row).
//
// bf16 rows go by sixteen bytes, shifted in registers; unaligned float32 ones by single elements, whose shifts would cost more than the
// loads they save (32 x 1000 tokens of 777 + 1025: 75.8 us so, 83.6 with shifts; bf16 32 x 3000 of 1001 + 2003: 223.5 by elements, 217).
template <int PARTS, int kSlotPitch, bool kHalf, bool kVec>
__device__ __forceinline__ void gp_convert(uint8_t* block, int lo, int column, const uint8_t* slot, int off, int rows,
                                           long long left, int warp, int lane) {
  // store(j) for all of a lane's rows, or for those that are there
  auto each = [&](auto count, int n, auto&& store) {
    constexpr int kCount = decltype(count)::value;
    if (rows == 128) {
#pragma unroll
      for (int j = 0; j < kCount; ++j) store(j);
    } else {
#pragma unroll
      for (int j = 0; j < kCount; ++j)
        if (j < n) store(j);
    }
  };
  if constexpr (kHalf) {                   // sixteen bytes a lane, four rows at a time, from the two aligned pieces that hold them
    const int i0 = lane >> 3, q = lane & 7, r = gp_loader_row(warp, i0);
    uint4 v[4], w[4];
#pragma unroll
    for (int j = 0; j < 4; ++j) v[j] = *reinterpret_cast<const uint4*>(slot + (i0 + 4 * j) * kSlotPitch + 16 * q);
#pragma unroll
    for (int j = 0; j < 4; ++j) w[j] = *reinterpret_cast<const uint4*>(slot + (i0 + 4 * j) * kSlotPitch + 16 * q + 16);
    const bool one = off & 4, two = off & 8;
    const uint32_t pick = off & 2 ? 0x5432 : 0x3210;
    uint32_t keep[4] = {0xffffffffu, 0xffffffffu, 0xffffffffu, 0xffffffffu};
    if (left < 128) {
      const int here = static_cast<int>(left) - 16 * q;
#pragma unroll
      for (int k = 0; k < 4; ++k) keep[k] = here >= 4 * k + 4 ? 0xffffffffu : here == 4 * k + 2 ? 0xffffu : 0u;
    }
    uint8_t* d = block + r * 128 + ((q ^ (r & 7)) << 4);
    each(std::integral_constant<int, 4>(), (rows - r + 31) >> 5, [&](int j) {
      uint32_t x[8] = {v[j].x, v[j].y, v[j].z, v[j].w, w[j].x, w[j].y, w[j].z, w[j].w};
#pragma unroll
      for (int k = 0; k < 7; ++k) x[k] = one ? x[k + 1] : x[k];
#pragma unroll
      for (int k = 0; k < 5; ++k) x[k] = two ? x[k + 2] : x[k];
#pragma unroll
      for (int k = 0; k < 4; ++k) x[k] = __byte_perm(x[k], x[k + 1], pick) & keep[k];
      *reinterpret_cast<uint4*>(d + j * 4096) = make_uint4(x[0], x[1], x[2], x[3]);
      if (PARTS == 2) *reinterpret_cast<uint4*>(d + j * 4096 + lo) = make_uint4(0u, 0u, 0u, 0u);
    });
  } else if constexpr (PARTS == 2) {
    auto split = [](float x0, float x1, uint32_t& h, uint32_t& l) {
      const __nv_bfloat162 hh = __floats2bfloat162_rn(x0, x1);
      const __nv_bfloat162 ll = __floats2bfloat162_rn(x0 - __bfloat162float(hh.x), x1 - __bfloat162float(hh.y));
      h = *reinterpret_cast<const uint32_t*>(&hh);
      l = *reinterpret_cast<const uint32_t*>(&ll);
    };
    if constexpr (kVec) {                  // four neighbouring elements a lane, four rows at a time
      const int i0 = lane >> 3, r = gp_loader_row(warp, i0), c = column + 4 * (lane & 7);
      float4 f[4];
#pragma unroll
      for (int j = 0; j < 4; ++j) f[j] = *reinterpret_cast<const float4*>(slot + (i0 + 4 * j) * kSlotPitch + 16 * (lane & 7));
      if (left < 128 && 16 * (lane & 7) >= left) {
#pragma unroll
        for (int j = 0; j < 4; ++j) f[j] = make_float4(0.f, 0.f, 0.f, 0.f);
      }
      uint8_t* d = block + r * 128 + (((c >> 3) ^ (r & 7)) << 4) + (c & 4) * 2;
      each(std::integral_constant<int, 4>(), (rows - r + 31) >> 5, [&](int j) {
        uint2 h, l;
        split(f[j].x, f[j].y, h.x, l.x);
        split(f[j].z, f[j].w, h.y, l.y);
        *reinterpret_cast<uint2*>(d + j * 4096) = h;
        *reinterpret_cast<uint2*>(d + j * 4096 + lo) = l;
      });
    } else {                               // two, two rows at a time
      const int i0 = lane >> 4, r = gp_loader_row(warp, i0), e = 2 * (lane & 15), c = column + e;
      const float* w = reinterpret_cast<const float*>(slot + i0 * kSlotPitch + off) + e;
      float f[16];
#pragma unroll
      for (int j = 0; j < 8; ++j) {
        f[2 * j] = w[j * (2 * kSlotPitch / 4)];
        f[2 * j + 1] = w[j * (2 * kSlotPitch / 4) + 1];
      }
      if (left < 128) {
        const int cols = static_cast<int>(left) / 4 - e;
#pragma unroll
        for (int j = 0; j < 8; ++j) {
          if (cols <= 0) f[2 * j] = 0.f;
          if (cols <= 1) f[2 * j + 1] = 0.f;
        }
      }
      uint8_t* d = block + r * 128 + (((c >> 3) ^ (r & 7)) << 4) + (c & 7) * 2;
      each(std::integral_constant<int, 8>(), (rows - r + 15) >> 4, [&](int j) {
        uint32_t h, l;
        split(f[2 * j], f[2 * j + 1], h, l);
        *reinterpret_cast<uint32_t*>(d + j * 2048) = h;
        *reinterpret_cast<uint32_t*>(d + j * 2048 + lo) = l;
      });
    }
  }
}

// Element-wise sum, in rank order, of four floats that lie at `at` in the shared memory of those CTAs of the cluster that have a bit
// in `mask`.  BATCH loads go out together, all eight where registers are free (in the loop over units one, as two cost it registers: 32 x 2000
// tokens of 128 float32, embedding form, k = 64: 63.5 -> 66.3 us): one after the other they took most of a small call (5 x 4 tokens of 368 + 448 float32, k = 42,
// cycles: partial blocks 5850, results 3850 of 24000).
template <int BATCH>
__device__ __forceinline__ float4 gp_cluster_sum(const float* at, uint32_t mask) {
  float4 sum = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
  for (int r0 = 0; r0 < 8; r0 += BATCH) {
    float4 v[BATCH];
#pragma unroll
    for (int r = 0; r < BATCH; ++r)
      if (mask >> (r0 + r) & 1) v[r] = ld_cluster_v4(map_to_cta(smem_u32(at), r0 + r));
#pragma unroll
    for (int r = 0; r < BATCH; ++r)
      if (mask >> (r0 + r) & 1) { sum.x += v[r].x; sum.y += v[r].y; sum.z += v[r].z; sum.w += v[r].w; }
  }
  return sum;
}

// o[r, c] += sum over staged rows [t0, t1) of s_r[t][r] * s_c[t][c], for the RT x CT block of thread (ty, tx)
template <int KMAX>
__device__ __forceinline__ void gp_contract(const float* s_r, const float* s_c, int t0, int t1, int ty, int tx, float (&o)[KMAX / 16][KMAX / 8]) {
  constexpr int RT = KMAX / 16, CT = KMAX / 8;
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
}

// The block of thread (ty, tx) in shared memory, [KMAX][KMAX], and zeros in its place
template <int KMAX>
__device__ __forceinline__ void gp_put_block(float* block, int ty, int tx, float (&o)[KMAX / 16][KMAX / 8]) {
  constexpr int RT = KMAX / 16, CT = KMAX / 8;
#pragma unroll
  for (int i = 0; i < RT; ++i)
#pragma unroll
    for (int j = 0; j < CT; j += 4) {
      *reinterpret_cast<float4*>(&block[(ty * RT + i) * KMAX + tx * CT + j]) = make_float4(o[i][j], o[i][j + 1], o[i][j + 2], o[i][j + 3]);
      o[i][j] = o[i][j + 1] = o[i][j + 2] = o[i][j + 3] = 0.f;
    }
}

// Adds the block of thread (ty, tx) to a sample's result, and zeros in its place
template <int KMAX>
__device__ __forceinline__ void gp_add_block(const GpParams& p, int b, int ty, int tx, float (&o)[KMAX / 16][KMAX / 8]) {
  constexpr int RT = KMAX / 16, CT = KMAX / 8;
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
}

// A sample's result from the blocks of `ranks` CTAs (rank order), of which this one stores its share with `threads` threads
template <int KMAX, int BATCH>
__device__ __forceinline__ void gp_store_block(const GpParams& p, int b, const float* block, uint32_t rank, uint32_t ranks, int tid, int threads) {
  float* dst = p.out + static_cast<long long>(b) * p.out_stride;
  const uint32_t mask = (1u << ranks) - 1;
#pragma unroll 1
  for (int e = 4 * (static_cast<int>(rank) * threads + tid); e < p.k_r * KMAX; e += 4 * static_cast<int>(ranks) * threads) {
    const int c = e % KMAX;
    if (c >= p.k_c) continue;
    const float4 v = ranks > 1 ? gp_cluster_sum<BATCH>(block + e, mask) : *reinterpret_cast<const float4*>(block + e);
    float* to = dst + static_cast<long long>(e / KMAX) * p.out_ld + c;
    to[0] = v.x * p.scale;
    if (c + 1 < p.k_c) to[1] = v.y * p.scale;
    if (c + 2 < p.k_c) to[2] = v.z * p.scale;
    if (c + 3 < p.k_c) to[3] = v.w * p.scale;
  }
}

template <int KMAX, int kSrc, bool kEmb, int kCluster>
__global__ void __launch_bounds__((GpCfg<KMAX, kSrc, kEmb, kCluster>::kThreads), 1)
gradproj_kernel(const __grid_constant__ CUtensorMap tm_g, const __grid_constant__ CUtensorMap tm_pr,
                const __grid_constant__ CUtensorMap tm_a, const __grid_constant__ CUtensorMap tm_pc,
                const GpParams p) {
  using Cfg = GpCfg<KMAX, kSrc, kEmb, kCluster>;
  constexpr int BM = Cfg::BM, BK = Cfg::BK, kStages = Cfg::kStages, RT = Cfg::RT, CT = Cfg::CT;
  constexpr int ATOMS = Cfg::ATOMS, PARTS = Cfg::PARTS, kProjStages = Cfg::kProjStages;
  constexpr bool kLoaders = Cfg::kLoaders;

  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  uint8_t* slots = smem + Cfg::kRings;                                         // [loader warps][kSlots]
  // Behind a cluster's loaders the staged blocks lie in the rings, whose last stage has been consumed by then, after the block that
  // store() puts at their start
  float* s_r = reinterpret_cast<float*>(kLoaders && kCluster != kNone ? smem + KMAX * KMAX * 4 : slots + Cfg::kSlots * Cfg::kSlotsBytes);   // [kStageRows][KMAX]
  float* s_c = s_r + Cfg::kStageRows * KMAX;                                  // [kStageRows][KMAX]
  uint64_t* bars = reinterpret_cast<uint64_t*>(slots + Cfg::kSlots * Cfg::kSlotsBytes + Cfg::kProjBytes);
  uint64_t* full_bar = bars;
  uint64_t* empty_bar = bars + kStages;
  uint64_t* proj_full = kLoaders ? bars + 2 * kStages : full_bar;             // the projection blocks' own ring
  uint64_t* proj_empty = kLoaders ? proj_full + kProjStages : empty_bar;
  uint64_t* acc_full = bars + 2 * kStages + (kLoaders ? 2 * kProjStages : 0);  // [2]
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
  // sample and 128-token chunk of the first unit; a division of 64 bits is the time of a pipeline stage
  const int chunks = p.chunks_per_sample;
  const int b0 = u0 >> 32 ? static_cast<int>(u0 / chunks) : static_cast<int>(static_cast<uint32_t>(u0) / static_cast<uint32_t>(chunks));
  const int chunk0 = static_cast<int>(u0 - static_cast<long long>(b0) * chunks);
  auto rows_of = [&](int chunk) -> int {     // tokens in a unit
    const long long left = p.T - static_cast<long long>(chunk) * BM;
    return left < BM ? static_cast<int>(left) : BM;
  };
  // a cluster's CTA adds up and contracts tokens [first, first + share) of its unit
  int first = 0, share = 0;
  if constexpr (kCluster != kNone) {
    const int rows = rows_of(chunk0), most = (rows + static_cast<int>(ranks) - 1) / static_cast<int>(ranks);
    first = min(static_cast<int>(rank) * most, rows);
    share = min(most, rows - first);
  }

  if (threadIdx.x == 0) {
    for (int s = 0; s < kStages; ++s) { mbar_init(&full_bar[s], kLoaders ? 8 : 1); mbar_init(&empty_bar[s], 1); }
    if (kLoaders)
      for (int s = 0; s < kProjStages; ++s) { mbar_init(&proj_full[s], 1); mbar_init(&proj_empty[s], 1); }
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
    uint8_t* const dst = kLoaders ? smem + kStages * Cfg::kStageBytes + box * Cfg::kProjAtomBytes
                                  : smem + (is_p ? Cfg::kActBytes + box * Cfg::kProjAtomBytes : box * Cfg::kActAtomBytes);
    constexpr int kPitch = kLoaders ? Cfg::kProjStageBytes : Cfg::kStageBytes;
    int stage = 0; uint32_t phase = 0; bool ok = true;
    int b = b0, chunk = chunk0;
    for (long long u = u0; u < u1 && ok; ++u) {
      const int row0 = chunk * BM;
      for (int kb = kb0; kb < kb1; ++kb) {
        int w = 1;
        if (lane == 0) w = mbar_wait(&proj_empty[stage], phase ^ 1, abort_flag, p.err, 421) ? 1 : 0;
        w = __shfl_sync(0xffffffffu, w, 0);
        if (!w) { ok = false; break; }
        const bool first = kb < kb_r;
        const int kpad = first ? p.kr_pad : p.kc_pad;
        if (lane == 0) mbar_arrive_expect_tx(&proj_full[stage], (kActBoxes * BM + kProjBoxes * kpad) * BK * 2);
        __syncwarp();
        if (lane < kActBoxes + kProjBoxes) {
          // an atom past the last column starts out of range and is zero-filled; what a residual box reads beyond
          // its part meets zeros of the operand
          int col = (first ? kb : kb - kb_r) * ATOMS * BK;
          if (PARTS == 2) col += box == 0 ? 0 : (first ? p.lo_r : p.lo_c);
          else col += box * BK;
          const CUtensorMap* m = first ? (is_p ? &tm_pr : &tm_g) : (is_p ? &tm_pc : &tm_a);
          tma_load_3d(dst + stage * kPitch, m, &proj_full[stage], col, is_p ? 0 : row0, is_p ? 0 : b);
        }
        if (++stage == kProjStages) { stage = 0; phase ^= 1; }
      }
      if (++chunk == chunks) { chunk = 0; ++b; }
    }
  } else if (kLoaders && warp >= 6) {
    // Loader warps: 16 rows of a stage each, requested kSlots - 1 slices ahead of the one that is converted
    if constexpr (kLoaders) {
      constexpr int kSlots = Cfg::kSlots, kGroups = Cfg::kLoaderWarps / 8;
      const int lw = (warp - 6) & 7, group = (warp - 6) >> 3;
      uint8_t* mine = slots + (warp - 6) * kSlots * Cfg::kSlotBytes;
      struct Place { long long left; int before, b, chunk; bool second; };     // units to come, stages behind, where
      const Place start = {u1 - u0, 0, b0, chunk0, false};
      auto advance = [&](Place& at) {
        at.second = !at.second;
        if (at.second) return;
        --at.left;
        at.before ^= kb1 - kb0;                          // their parity
        if (++at.chunk == chunks) { at.chunk = 0; ++at.b; }
      };
      auto segment = [&](const Place& at, GpSegment& x) -> bool {
        const bool second = at.second;
        int k0 = second && kb0 < kb_r ? kb_r : kb0;
        const int k1 = !second && kb1 > kb_r ? kb_r : kb1;
        if (kGroups == 2) k0 += (at.before + k0 - kb0 + group) & 1;      // the group's first stage
        if (k0 >= k1) return false;
        const long long t0 = static_cast<long long>(at.chunk) * BM;
        x.half = kSrc == kSrcBf16 || (kSrc == kSrcMixed && (second ? p.half_a : p.half_g));
        x.vec = second ? p.vec_a : p.vec_g;
        const int size = x.half ? 2 : 4;
        const long long from = static_cast<long long>(second ? k0 - kb_r : k0) * BK * size;
        x.pitch = (second ? p.lda : p.ldg) * size;
        x.at = reinterpret_cast<uintptr_t>(second ? p.a : p.g) + (at.b * p.T + t0) * x.pitch + from;
        x.bytes = static_cast<long long>(second ? p.n_c : p.n_r) * size - from;
        x.rows = rows_of(at.chunk);
        x.slices = (k1 - k0 + kGroups - 1) / kGroups * (x.half ? 1 : 2);
        x.jump = 128 + (kGroups - 1) * (x.half ? 128 : 256);
        return true;
      };
      int stage = group; uint32_t phase = 0;
      int to = 0, from = 0;                              // slots
      GpAsk<Cfg::kSlotPitch> ask;
      ask.left = 0;
      Place asked = start;                               // unit and operand to be requested next
      auto request = [&]() {
        while (ask.left == 0 && asked.left > 0) {
          GpSegment x;
          if (segment(asked, x)) ask.open(x, lw, lane);
          advance(asked);
        }
        if (ask.left > 0) ask.request(smem_u32(mine + to * Cfg::kSlotBytes), lane);
        asm volatile("cp.async.commit_group;" ::: "memory");
        if (++to == kSlots) to = 0;
      };
      for (int i = 0; i < kSlots - 1; ++i) request();
      auto convert = [&](const GpSegment& x, auto half, auto vec) -> bool {
        constexpr bool kHalf = decltype(half)::value, kVec = decltype(vec)::value;
        constexpr int kPerStage = kHalf ? 1 : 2;
        const int off = static_cast<int>((x.at + gp_loader_row(lw, kHalf ? lane >> 3 : lane >> 4) * x.pitch) & 15);
        long long bytes = x.bytes;
        for (int n = x.slices; n > 0; n -= kPerStage) {
          uint8_t* block = smem + stage * Cfg::kStageBytes;
#pragma unroll
          for (int part = 0; part < kPerStage; ++part) {
            request();
            asm volatile("cp.async.wait_group %0;" ::"n"(kSlots - 1) : "memory");
            if (part == 0 && !mbar_wait_warp(&empty_bar[stage], phase ^ 1, abort_flag, p.err, 621)) return false;
            __syncwarp();                                // all lanes' pieces have arrived
            gp_convert<PARTS, Cfg::kSlotPitch, kHalf, kVec>(block, Cfg::kActAtomBytes, part * 32, mine + from * Cfg::kSlotBytes, off, x.rows, bytes, lw, lane);
            bytes -= part == kPerStage - 1 ? x.jump : 128;
            if (++from == kSlots) from = 0;
            if (part == kPerStage - 1) fence_proxy_async_smem();
            __syncwarp();                                // all lanes are done with the slot, and with the stage
          }
          if (lane == 0) mbar_arrive(&full_bar[stage]);
          stage += kGroups;
          if (stage >= kStages) { stage -= kStages; phase ^= 1; }
        }
        return true;
      };
      bool ok = true;
      for (Place at = start; ok && at.left > 0; advance(at)) {
        GpSegment x;
        if (!segment(at, x)) continue;
        if constexpr (PARTS == 1) ok = convert(x, std::true_type(), std::false_type());
        else if (kSrc == kSrcMixed && x.half) ok = convert(x, std::true_type(), std::false_type());
        else if (x.vec) ok = convert(x, std::false_type(), std::true_type());
        else ok = convert(x, std::false_type(), std::false_type());
      }
      asm volatile("cp.async.wait_all;" ::: "memory");
    }
  } else if (warp == 5) {
    // The whole warp follows the loop, so that what the elected lane's instructions take is the same for all lanes and
    // lies in uniform registers: a product takes 60 cycles to issue, 100 from inside a branch of one lane (8 x 4096 tokens of
    // 4096 + 1024 bf16, k = 64: 70.6 -> 68.3 us).
    const uint32_t idesc_r = make_idesc_bf16(BM, p.kr_pad, 0, 0);
    const uint32_t idesc_c = make_idesc_bf16(BM, p.kc_pad, 0, 0);
    const uint64_t a0 = make_smem_desc_sw128(smem_u32(smem), 16, 1024);
    const uint64_t b0 = make_smem_desc_sw128(smem_u32(smem + (kLoaders ? kStages * Cfg::kStageBytes : Cfg::kActBytes)), 16, 1024);
    int stage = 0; uint32_t phase = 0; int acc = 0; uint32_t acc_phase = 0; bool ok = true;
    int ps = 0; uint32_t p_phase = 0;                    // of the projection blocks, where they have a ring of their own
    for (long long u = u0; u < u1 && ok; ++u) {
      int w = 1;                             // one lane polls: the epilogue is on the same schedulers
      if (lane == 0) w = mbar_wait(&acc_empty[acc], acc_phase ^ 1, abort_flag, p.err, 522) ? 1 : 0;
      if (!__shfl_sync(0xffffffffu, w, 0)) { ok = false; break; }
      tc_fence_after_sync();
      const uint32_t d_r = tmem_base + acc * 256;
      for (int kb = kb0; kb < kb1; ++kb) {
        if (kLoaders && !mbar_wait_warp(&proj_full[ps], p_phase, abort_flag, p.err, 524)) { ok = false; break; }
        if (!mbar_wait_warp(&full_bar[stage], phase, abort_flag, p.err, 523)) { ok = false; break; }
        tc_fence_after_sync();
        const bool first = kb < kb_r;
        const uint32_t d = first ? d_r : d_r + 128, idesc = first ? idesc_r : idesc_c;
        const uint32_t more = kb == kb0 || kb == kb_r ? 0u : 1u;
        const uint64_t adesc = a0 + stage * (Cfg::kStageBytes / 16);
        const uint64_t bdesc = b0 + (kLoaders ? ps * (Cfg::kProjStageBytes / 16) : stage * (Cfg::kStageBytes / 16));
        if (elect_one()) {
#pragma unroll
          for (int k = 0; k < ATOMS * BK / 16; ++k) {
            const uint64_t ak = adesc + (k / 4) * (Cfg::kActAtomBytes / 16) + 2 * (k % 4), bk = bdesc + (k / 4) * (Cfg::kProjAtomBytes / 16) + 2 * (k % 4);
            if constexpr (PARTS == 2) {      // residual parts lie behind the values
              umma_bf16(d, ak + Cfg::kActAtomBytes / 16, bk, idesc, k == 0 ? more : 1u);
              umma_bf16(d, ak, bk + Cfg::kProjAtomBytes / 16, idesc, 1u);
              umma_bf16(d, ak, bk, idesc, 1u);
            } else {
              umma_bf16(d, ak, bk, idesc, k == 0 ? more : 1u);
            }
          }
          umma_commit(&empty_bar[stage]);
          if (kLoaders) umma_commit(&proj_empty[ps]);
          if (kb == kb1 - 1) umma_commit(&acc_full[acc]);
        }
        __syncwarp();
        if (++stage == kStages) { stage = 0; phase ^= 1; }
        if (kLoaders && ++ps == kProjStages) { ps = 0; p_phase ^= 1; }
      }
      if (++acc == 2) { acc = 0; acc_phase ^= 1; }
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

    // This CTA, or the cluster, has all of sample b: its block goes through shared memory -- a cluster's through that of the
    // stages, which nothing is on its way to any more -- and each CTA adds up and stores its share.
    auto store = [&](int b) {
      float* block = ranks > 1 ? reinterpret_cast<float*>(smem) : s_r;            // [KMAX][KMAX]
      gp_put_block<KMAX>(block, ty, tx, o);
      if (ranks > 1) cluster_sync_all();
      else named_bar_sync(1, 128);
      gp_store_block<KMAX, 1>(p, b, block, rank, ranks, tid, 128);
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

    if constexpr (kCluster != kNone) {
      // One unit: row `tid` of this CTA's partial blocks is staged
      const long long t_first = static_cast<long long>(chunk0) * BM;
      const bool owned = tid >= first && tid < first + share;
      if constexpr (kEmb) { if (owned) gather(b0, t_first + tid); }
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
    }
    // (one place that stores or adds and no wide counters: with two places the embedding form of float32 and unaligned rows spilled
    // more registers, 237 us for 16 x 2048 tokens of 4000 float32, k = 64, and 200 as it is; 65 and 59 for 701)
    if constexpr (kCluster == kNone) {
      bool alive = true;
      int b = b0, chunk = chunk0;
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
            if constexpr (kLoaders) {          // of rows that are not there the block has none
              const int here = rows_of(chunk) - half * Cfg::kStageRows;
              gp_contract<KMAX>(s_r, s_c, 0, here < Cfg::kStageRows ? here : Cfg::kStageRows, ty, tx, o);
            } else {                           // TMA has written zeros
              gp_contract<KMAX>(s_r, s_c, 0, Cfg::kStageRows, ty, tx, o);
            }
            named_bar_sync(1, 128);
          }
          if (++acc == 2) { acc = 0; acc_phase ^= 1; }
        }
        if (++chunk == chunks || left <= 1) {     // done with the sample, or with this CTA's part of it
          if (p.direct) store(b);
          else gp_add_block<KMAX>(p, b, ty, tx, o);
          if (p.group > 1) break;
          chunk = 0;
          ++b;
        }
      }
      if (!alive && p.group > 1) cluster_sync_all();           // the one that the others wait at in store()
    }
  }

  if constexpr (kCluster != kNone) {
    // All warps: rows [first, first + share) of all CTAs' blocks are added up here, in place, as nobody else reads them from this CTA.
    // Ranks with columns of G have a bit in `of_r`, those with columns of A in `of_c`.
    const int s0 = static_cast<int>(static_cast<unsigned>(lane) * kb_total / ranks), s1 = static_cast<int>(static_cast<unsigned>(lane + 1) * kb_total / ranks);
    const bool some = lane < static_cast<int>(ranks) && s0 < s1;
    const uint32_t of_r = __ballot_sync(0xffffffffu, some && s0 < kb_r), of_c = __ballot_sync(0xffffffffu, some && s1 > kb_r);
    cluster_sync_all();
    const int quads_r = share * (p.kr_pad / 4), quads = quads_r + (kEmb ? 0 : share * (p.kc_pad / 4));
    for (int i = threadIdx.x; i < quads; i += Cfg::kThreads) {
      const bool r = i < quads_r;
      const int e = r ? i : i - quads_r, per = (r ? p.kr_pad : p.kc_pad) / 4;
      float* at = (r ? s_r : s_c) + gp_staged_index<KMAX>(first + e / per, e % per * 4);
      *reinterpret_cast<float4*>(at) = gp_cluster_sum<8>(at, r ? of_r : of_c);
    }
    __syncthreads();
    const int ty = threadIdx.x >> 3, tx = threadIdx.x & 7;         // of the first 128 threads
    if (warp < 4) {
      float o[RT][CT];
#pragma unroll
      for (int i = 0; i < RT; ++i)
#pragma unroll
        for (int j = 0; j < CT; ++j) o[i][j] = 0.f;
      if (!*abort_flag) gp_contract<KMAX>(s_r, s_c, first, first + share, ty, tx, o);
      if (kCluster == kSome) gp_add_block<KMAX>(p, b0, ty, tx, o);
      else gp_put_block<KMAX>(reinterpret_cast<float*>(smem), ty, tx, o);
    }
    if constexpr (kCluster == kWhole) {
      cluster_sync_all();
      gp_store_block<KMAX, 8>(p, b0, reinterpret_cast<const float*>(smem), rank, ranks, threadIdx.x, Cfg::kThreads);
    }
    cluster_sync_all();                    // no CTA leaves while another reads its blocks
  } else if (p.group > 1) {
    if (warp >= 4) cluster_sync_all();     // the epilogue's before the results are added up
    cluster_sync_all();
  }
  tc_fence_before_sync();
  __syncthreads();
  if (warp == 5) { tc_fence_after_sync(); tmem_dealloc(tmem_base, 512); }
}

template <int KMAX, int kSrc, bool kEmb, int kCluster>
static int launch_gradproj_t(const CUtensorMap& tg, const CUtensorMap& tpr, const CUtensorMap& ta, const CUtensorMap& tpc,
                             GpParams& p, int ranks, const DeviceState* ds, cudaStream_t st) {
  using Cfg = GpCfg<KMAX, kSrc, kEmb, kCluster>;
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
  using Cfg = GpCfg<KMAX, kSrc, kEmb, kCluster>;
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
// * Short chains of small ranks stay alone: the cluster's barriers and the exchange cost about 1.5 us, a stage 0.3 to 0.6 us of a unit's
//   chain, the contraction, which the CTAs share too, 1 us at 32 x 32 and 3 at 64 x 64.  (Four to seven stages, k <= 32, alone and in
//   clusters: 56 x 2 tokens of 321 float32, embedding form, 11.8 and 9.4 us; 2 x 165 of 107 + 166 float32 13.9 and 11.1; 14 x 80 of
//   134 + 192 bf16 10.1 and 8.8.  Fewer: 23 x 117 of 256 + 64 bf16 12.2 and 12.8.)  Rows that TMA reads in several units a sample, whose
//   results are then added and not stored, from eight stages on: 2 x 281 of 384 + 128 bf16 9.1 alone, 11.1 in clusters.
// * Three or six share unevenly, which pays from so many stages on (17 x 60 of 640 + 640, ten stages: 13.9 us in fours, 14.8 in sixes;
//   20 x 100 of 9792 + 4160 bf16 21.0 and 16.9; 9 x 464 of the same float32 154 in pairs, 109 in threes).
// * Fives lost (24 units of 32 stages: 26.3 us, 24.7 in fours).
template <int KMAX, int kSrc, bool kEmb>
static int gradproj_ranks(long long units, int chunks, int stages, const DeviceState* ds) {
  const int least = kSrc == kSrcTma && chunks > 1 ? 8 : 4;
  if ((stages < least && KMAX <= 32) || 2 * units > ds->sm_count) return 1;
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
  constexpr int kCols = GpCfg<KMAX, kSrc, kEmb, kNone>::ATOMS * 64;
  const int stages = ceil_div(p.n_r, kCols) + (kEmb ? 0 : ceil_div(p.n_c, kCols));
  const int ranks = gradproj_ranks<KMAX, kSrc, kEmb>(p.units, p.chunks_per_sample, stages, ds);
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

// Chooses how the rows are read: bf16 through TMA where it can, else by loader warps
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
    p.vec_g = !p.half_g && aligned(o.G, o.ldg, 16, 4) && p.n_r % 4 == 0;
    p.vec_a = !p.half_a && aligned(o.A, o.lda, 16, 4) && p.n_c % 4 == 0;
    if constexpr (!kEmb) {
      if (o.is_f32 != 1) return launch_gradproj_k<kSrcMixed, kEmb>(o, p, ds, st);
    }
    return launch_gradproj_k<kSrcF32, kEmb>(o, p, ds, st);
  }
  if (aligned(o.G, o.ldg, 16, 2) && (kEmb || aligned(o.A, o.lda, 16, 2)) && p.T < (1ll << 31) - 128)
    return launch_gradproj_k<kSrcTma, kEmb>(o, p, ds, st);
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
