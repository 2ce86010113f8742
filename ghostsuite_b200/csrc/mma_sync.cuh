// Warp-level bf16 MMA (mma.sync m16n8k16, fp32 accumulate) with fragments loaded straight from
// global memory, for the small contractions around the projection path whose operands are streamed
// once and whose output is tiny (k x k, or batch x batch): the kernels are bound by the operand
// stream, not by the tensor pipe, so there is no shared-memory staging.
#pragma once
#include <cuda_bf16.h>
#include <stdint.h>

namespace gb {

__device__ __forceinline__ void mma_16816(float (&d)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3,
                                          uint32_t b0, uint32_t b1) {
  asm volatile(
      "mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, "
      "{%0, %1, %2, %3};"
      : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
      : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}

// The same product without a sum before it.
__device__ __forceinline__ void mma_16816_new(float (&d)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3,
                                              uint32_t b0, uint32_t b1) {
  asm volatile(
      "mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, "
      "{%10, %10, %10, %10};"
      : "=f"(d[0]), "=f"(d[1]), "=f"(d[2]), "=f"(d[3])
      : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1), "f"(0.f));
}

// d += a for the four entries of a fragment, two to an instruction
__device__ __forceinline__ void add_fragment(float (&d)[4], const float (&a)[4]) {
#pragma unroll
  for (int e = 0; e < 4; e += 2)
    asm("{\n\t.reg .b64 x, y;\n\tmov.b64 x, {%0, %1};\n\tmov.b64 y, {%2, %3};\n\tadd.rn.f32x2 x, x, y;\n\tmov.b64 {%0, %1}, x;\n\t}"
        : "+f"(d[e]), "+f"(d[e + 1]) : "f"(a[e]), "f"(a[e + 1]));
}

__device__ __forceinline__ uint32_t pack_bf16x2(__nv_bfloat16 x, __nv_bfloat16 y) {
  __nv_bfloat162 h(x, y);
  return *reinterpret_cast<uint32_t*>(&h);
}

}  // namespace gb
