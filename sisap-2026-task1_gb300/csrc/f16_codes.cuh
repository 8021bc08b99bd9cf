// f16_codes.cuh -- int8 codes as f16 operands of the tensor cores.
//
// An int8 code is exact in f16, a product of two has magnitude <= 2^14, and
// every partial sum of a dot over d <= kMaxDim codes is an integer of magnitude
// <= d * 2^14 <= 2^24, which fp32 holds exactly: whatever the order of the
// additions, the fp32 result is the int32 dot.
#pragma once
#include "knng_internal.cuh"

namespace knng {

static_assert(int64_t(kMaxDim) * 128 * 128 <= int64_t(1) << 24, "a dot of kMaxDim codes is exact in fp32");

// Four int8 codes (one 32-bit word) widened to two f16 pairs, exactly and in
// integer/packed-half steps: u = code + 128 (xor 0x80 per byte) becomes the f16
// 1024 + u by placing 0x64 above each byte (0x6400 is 1024.0, whose unit in the
// last place is 1), and one packed add of -1152 leaves code = u - 128.
__device__ __forceinline__ void widen4(uint32_t w, uint32_t& lo, uint32_t& hi) {
  const uint32_t u = w ^ 0x80808080u;
  const uint32_t a = __byte_perm(u, 0x64646464u, 0x4140);  // codes 0, 1
  const uint32_t b = __byte_perm(u, 0x64646464u, 0x4342);  // codes 2, 3
  asm("add.f16x2 %0, %1, %2;" : "=r"(lo) : "r"(a), "r"(0xE480E480u));
  asm("add.f16x2 %0, %1, %2;" : "=r"(hi) : "r"(b), "r"(0xE480E480u));
}

// c += A B for one 16 x 8 tile over 16 codes, by a warp.
__device__ __forceinline__ void mma16816(float (&c)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0,
                                         uint32_t b1) {
  asm volatile(
      "mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
      : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
      : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}

}  // namespace knng
