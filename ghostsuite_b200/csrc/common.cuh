// Host-side plumbing shared by every translation unit of libghost_b200: status codes, the
// thread-local error message, the kernel-launch counter, the per-device error word that kernels
// write when a bounded wait gives up, and TMA tensor-map construction.
#pragma once
#include <cuda.h>
#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <stdint.h>
#include <stdio.h>

#include <utility>

#include "../../include/ghost_b200.h"

namespace gb {

// ---- error message (thread local) -------------------------------------------------------
void set_error(const char* fmt, ...);
int fail(int code, const char* fmt, ...);

// The status goes to the caller and not also to whoever asks the runtime for its last error next
#define GB_CUDA_OK(expr)                                                                   \
  do {                                                                                     \
    cudaError_t _e = (expr);                                                               \
    if (_e != cudaSuccess) {                                                               \
      (void)cudaGetLastError();                                                            \
      return ::gb::fail(GHOST_ERR_CUDA, "%s failed: %s (%s:%d)", #expr,                    \
                        cudaGetErrorString(_e), __FILE__, __LINE__);                       \
    }                                                                                      \
  } while (0)

#define GB_REQUIRE(cond, ...)                                                              \
  do {                                                                                     \
    if (!(cond)) return ::gb::fail(GHOST_ERR_INVALID, __VA_ARGS__);                        \
  } while (0)

// ---- launch accounting -------------------------------------------------------------------
void count_launch(int n = 1);
int post_launch(const char* what);  // cudaGetLastError -> status

// Launches a kernel that may start while the kernel ahead of it in the stream ends: blocks come up on the SMs that it leaves,
// set up what they have in shared and tensor memory, and wait in stream_order() for the rest of it.  A layer's
// hook is a chain of four to eight kernels of 2 to 40 us, with 1.5 to 3 us between one's end and the next one's first load.
// Graphs keep the plain order: replayed, such edges cost more than they gave (256 + 32 samples of 16 x (1024 -> 1024): 93 us
// against 79).
inline int early_start(cudaLaunchAttribute* attr, cudaStream_t st) {
  cudaStreamCaptureStatus capturing = cudaStreamCaptureStatusNone;
  if (cudaStreamIsCapturing(st, &capturing) != cudaSuccess) {
    (void)cudaGetLastError();            // the launch itself says what is wrong, if anything is
    return 0;
  }
  if (capturing != cudaStreamCaptureStatusNone) return 0;
  attr->id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr->val.programmaticStreamSerializationAllowed = 1;
  return 1;
}
// With blocks in clusters of a shape other than (1, 1, 1) that divides the grid.
template <typename... P, typename... A>
inline cudaError_t launch_next_cluster(dim3 cluster, void (*kernel)(P...), dim3 grid, dim3 block, size_t smem, cudaStream_t st, A&&... args) {
  cudaLaunchAttribute attr[2];
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = grid;
  cfg.blockDim = block;
  cfg.dynamicSmemBytes = smem;
  cfg.stream = st;
  cfg.attrs = attr;
  cfg.numAttrs = early_start(attr, st);
  if (cluster.x * cluster.y * cluster.z > 1) {
    cudaLaunchAttribute& c = attr[cfg.numAttrs++];
    c.id = cudaLaunchAttributeClusterDimension;
    c.val.clusterDim.x = cluster.x;
    c.val.clusterDim.y = cluster.y;
    c.val.clusterDim.z = cluster.z;
  }
  return cudaLaunchKernelEx(&cfg, kernel, std::forward<A>(args)...);
}
template <typename... P, typename... A>
inline cudaError_t launch_next(void (*kernel)(P...), dim3 grid, dim3 block, size_t smem, cudaStream_t st, A&&... args) {
  return launch_next_cluster(dim3(1, 1, 1), kernel, grid, block, smem, st, std::forward<A>(args)...);
}
// Zeros for the kernel behind it in the stream, that adds to them: a kernel in the same programmatic order.  A memset waits for
// the kernel ahead to end, and the kernel behind it for the memset, 1.5 to 3 us at either edge; this one is there by then and lets the
// next come up while it writes.  With a memset and with it, us: GradProj of 4 x 649 tokens of 640 + 8448 20.0 and 17.0; embedding
// hook of 16 x 1024 tokens of 768 54.3 and 52.2.  Alone it hides behind nothing, and on the host it is a launch instead of a memset, 0.9 us
// more: a user whose chain is one kernel weighs that (dispatch_similarity).  Words off sixteen bytes, large buffers, which a memset's
// bandwidth counts for, and captures, whose edges are plain ones, keep the memset.
static constexpr size_t kClearMost = 32u << 20;
int clear_ahead(void* dst, size_t bytes, cudaStream_t st);
// The other half of launch_next, in every kernel that is launched so, before its first access to global memory and in every
// block: waits until all work ahead in the stream has ended and can be read, then lets the next kernel come up.  (In
// that order: a kernel that ends has waited, so its end stands for everything before it.)
//
// Such a kernel exists while the one ahead still writes, so what it reads is not read-only for as long as it lives: no
// __ldg and no const __restrict__ pointers, whose loads may be served from a line that is older than the wait, or be moved
// ahead of it.  Ordinary loads stay behind the wait.
__device__ __forceinline__ void stream_order() {
  asm volatile("griddepcontrol.wait;" ::: "memory");
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
}

// Value kernels store in the device error word when they meet an embedding id outside [0, vocab):
// the id's contribution is skipped and ghost_poll_kernel_error reports GHOST_ERR_INDEX.
static constexpr int kErrBadIndex = 9001;

// ---- per-device state ----------------------------------------------------------------------
struct DeviceState {
  int device = -1;
  int sm_count = 0;
  int cc_major = 0, cc_minor = 0;
  int* err_word = nullptr;  // device address of the kernel error word
};
// Returns nullptr (and sets the error) if the current device is not sm_100.
const DeviceState* device_state();

// ---- TMA ---------------------------------------------------------------------------------------
// 2-D row-major bf16 tensor [rows, cols] with row pitch `ld` elements; box = [box_rows, 64 cols]
// (64 bf16 = 128 bytes) with the 128-byte swizzle.  Out-of-bounds elements read as zero.
int make_tmap_bf16_2d(CUtensorMap* out, const void* base, uint64_t rows, uint64_t cols, uint64_t ld,
                      uint32_t box_rows, uint32_t box_cols = 64);

// 3-D view [samples, rows, cols] of a row-major bf16 matrix (sample pitch = rows * ld); box =
// [1, box_rows, 64 cols].  Rows past the end of a sample read as zero, so a K-loop over one
// sample's tokens never sees its neighbour's.
int make_tmap_bf16_3d(CUtensorMap* out, const void* base, uint64_t samples, uint64_t rows,
                      uint64_t cols, uint64_t ld, uint32_t box_rows, uint32_t box_cols = 64);

// The same matrix seen as [samples, cols/64, rows, 64] (cols a multiple of 64): one box covers
// `box_blocks` adjacent 64-column blocks of `box_rows` rows, each block landing in shared memory
// as its own swizzled [box_rows][64] panel.  Coordinates: (0, row, block, sample).
int make_tmap_bf16_blocks(CUtensorMap* out, const void* base, uint64_t samples, uint64_t rows,
                          uint64_t cols, uint64_t ld, uint32_t box_rows, uint32_t box_blocks);

// Rows of a float32 matrix as two bf16 parts `part_rows` rows apart (columns zero-padded to the pitch), for K-major
// tiles: a box covers 64 columns of `box_rows` rows of both parts, the values first.  Coordinates: (column, row, 0).
int make_tmap_bf16_part_rows(CUtensorMap* out, const void* base, uint64_t part_rows, uint64_t rows, uint64_t ld, uint32_t box_rows);

// float32 operands as two bf16 parts (value and residual), [samples, 2, part_rows, cols] with cols a multiple of 64
// (zero-padded), of which the first `rows` of a part count: a box covers both parts of `box_blocks` adjacent 64-column blocks of `box_rows` rows, the
// value panels first.  Rows past the end of a sample read as zero.  Coordinates: (0, row, block, 0, sample).
int make_tmap_bf16_parts(CUtensorMap* out, const void* base, uint64_t samples, uint64_t part_rows, uint64_t rows,
                         uint64_t cols, uint32_t box_rows, uint32_t box_blocks);

// Validation tiles as an all-gather leaves them: [ranks][tiles][per_rank samples][32768] bf16, seen as
// [64, per_rank, ranks, 512 panels, tiles]; a box holds `box_rows` consecutive validation samples
// (global index = rank * per_rank + sample) of `box_blocks` panels, each panel a swizzled
// [box_rows][64] block -- the layout make_tmap_bf16_blocks gives for a tile-major buffer.  box_rows
// must divide per_rank or be a multiple of it.  Coordinates: (0, sample, rank, panel, tile).
int make_tmap_bf16_gathered_tiles(CUtensorMap* out, const void* base, uint64_t ranks, uint64_t tiles,
                                  uint64_t per_rank, uint32_t box_rows, uint32_t box_blocks);

// 2-D map of a dense row-major bf16 matrix for tiled STORES of [box_rows, 32 columns] boxes (64-byte
// rows) from shared memory written with the 64-byte swizzle: 16-byte chunk c of row r sits at
// r * 64 + ((c ^ ((r >> 1) & 3)) * 16).
int make_tmap_bf16_store_2d(CUtensorMap* out, const void* base, uint64_t rows, uint64_t cols, uint32_t box_rows);
// The same for fp32: boxes of [box_rows, 32 columns] (128-byte rows) written with the 128-byte swizzle, chunk c of row r at
// r * 128 + ((c ^ (r & 7)) * 16).
int make_tmap_f32_store_2d(CUtensorMap* out, const void* base, uint64_t rows, uint64_t cols, uint32_t box_rows);
// 2-D map of a row-major matrix of 2- or 4-byte elements for boxes of 128 bytes of columns and `box_rows` rows with the
// 128-byte swizzle.  Coordinates: (column, row).
int make_tmap_rows(CUtensorMap* out, const void* base, int elem_bytes, uint64_t rows, uint64_t cols, uint64_t ld, uint32_t box_rows);
// Per-sample fp32 tiles [tiles][samples][32768], of whose samples the `first` ones count (those behind read as zero), seen as
// [tiles, 1024 panels, first, 32]: a box holds eight panels (256 elements) of `box_rows` samples, each panel a
// swizzled [box_rows][32] block.  Coordinates: (0, sample, panel, tile).
int make_tmap_f32_tiles(CUtensorMap* out, const void* base, uint64_t tiles, uint64_t samples, uint64_t first, uint32_t box_rows);

inline int ceil_div(long long a, long long b) { return static_cast<int>((a + b - 1) / b); }

}  // namespace gb
