// Whole words of small-float codes to fp16.
//
// The conversions take a byte (two e2m1 codes) or a half word (two e4m3 codes).  Handing them the parts of one unpacking move costs
// the conversions alone; shifting and masking each part out of the word first, as the headers' functions for single parts do, costs
// as much again: 13.8 against 25.4 cycles per word of eight e2m1 codes and scheduler, one product per pair included (sixteen warps).
#pragma once
#include <cuda_fp16.h>
#include <stdint.h>

namespace stk {

// Eight e2m1 codes, low nibble first -> four fp16 pairs
__device__ __forceinline__ void e2m1x8_to_half(uint32_t w, __half2 (&h)[4]) {
  uint32_t r[4];
  asm("{\n\t.reg .b8 a, b, c, d;\n\tmov.b32 {a, b, c, d}, %4;\n\t"
      "cvt.rn.f16x2.e2m1x2 %0, a;\n\tcvt.rn.f16x2.e2m1x2 %1, b;\n\tcvt.rn.f16x2.e2m1x2 %2, c;\n\tcvt.rn.f16x2.e2m1x2 %3, d;\n\t}"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(w));
#pragma unroll
  for (int i = 0; i < 4; ++i) h[i] = *reinterpret_cast<const __half2*>(&r[i]);
}

// Four e4m3 codes -> two fp16 pairs
__device__ __forceinline__ void e4m3x4_to_half(uint32_t w, __half2& lo, __half2& hi) {
  uint32_t a, b;
  asm("{\n\t.reg .b16 x, y;\n\tmov.b32 {x, y}, %2;\n\tcvt.rn.f16x2.e4m3x2 %0, x;\n\tcvt.rn.f16x2.e4m3x2 %1, y;\n\t}"
      : "=r"(a), "=r"(b) : "r"(w));
  lo = *reinterpret_cast<const __half2*>(&a);
  hi = *reinterpret_cast<const __half2*>(&b);
}

}  // namespace stk
