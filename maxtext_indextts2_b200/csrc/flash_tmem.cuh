// tcgen05 pieces of the attention kernels: P as the TMEM operand, V as an MN-major operand, TMEM rows in and out of registers, values that are no
// finite numbers.
#pragma once

#include "common.cuh"

namespace mtx {

// B operand whose rows are k (keys) and whose 128-byte swizzled row pieces run along n: 64-element chunks of n are `lbo` bytes apart, groups of
// eight rows 1024
__device__ __forceinline__ uint64_t umma_desc_sw128_mn(uint32_t addr, uint32_t lbo) {
  uint64_t d = 0;
  d |= uint64_t((addr & 0x3FFFFu) >> 4);
  d |= uint64_t(lbo >> 4) << 16;
  d |= uint64_t(1024 >> 4) << 32;
  d |= uint64_t(1) << 46;
  d |= uint64_t(2) << 61;
  return d;
}
constexpr uint32_t kIdescBMajorMN = 1u << 16;

// D[tmem] (+)= A[tmem] * B[smem]
__device__ __forceinline__ void umma_bf16_ts(uint32_t tmem_d, uint32_t tmem_a, uint64_t desc_b, uint32_t idesc, uint32_t accumulate) {
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p;\n\t}"
      :
      : "r"(tmem_d), "r"(tmem_a), "l"(desc_b), "r"(idesc), "r"(accumulate)
      : "memory");
}

__device__ __forceinline__ void tmem_ld_x32(uint32_t taddr, uint32_t (&r)[32]) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x32.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, %16, %17, %18, %19, %20, %21, "
      "%22, %23, %24, %25, %26, %27, %28, %29, %30, %31}, [%32];"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]), "=r"(r[9]), "=r"(r[10]),
        "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15]), "=r"(r[16]), "=r"(r[17]), "=r"(r[18]), "=r"(r[19]), "=r"(r[20]),
        "=r"(r[21]), "=r"(r[22]), "=r"(r[23]), "=r"(r[24]), "=r"(r[25]), "=r"(r[26]), "=r"(r[27]), "=r"(r[28]), "=r"(r[29]), "=r"(r[30]),
        "=r"(r[31])
      : "r"(taddr)
      : "memory");
}
__device__ __forceinline__ void tmem_st_x32(uint32_t taddr, const uint32_t (&r)[32]) {
  asm volatile(
      "tcgen05.st.sync.aligned.32x32b.x32.b32 [%32], {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, %16, %17, %18, %19, %20, "
      "%21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31};"
      :
      : "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]), "r"(r[8]), "r"(r[9]), "r"(r[10]), "r"(r[11]),
        "r"(r[12]), "r"(r[13]), "r"(r[14]), "r"(r[15]), "r"(r[16]), "r"(r[17]), "r"(r[18]), "r"(r[19]), "r"(r[20]), "r"(r[21]), "r"(r[22]),
        "r"(r[23]), "r"(r[24]), "r"(r[25]), "r"(r[26]), "r"(r[27]), "r"(r[28]), "r"(r[29]), "r"(r[30]), "r"(r[31]), "r"(taddr)
      : "memory");
}
__device__ __forceinline__ void tmem_st_x16(uint32_t taddr, const uint32_t (&r)[16]) {
  asm volatile("tcgen05.st.sync.aligned.32x32b.x16.b32 [%16], {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15};"
               :
               : "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]), "r"(r[8]), "r"(r[9]), "r"(r[10]), "r"(r[11]),
                 "r"(r[12]), "r"(r[13]), "r"(r[14]), "r"(r[15]), "r"(taddr)
               : "memory");
}
__device__ __forceinline__ void tmem_wait_ld() { asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory"); }
__device__ __forceinline__ void tmem_wait_st() { asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory"); }

// ---- values that only some rows of a tile see ---------------------------------------------------------------------------------------
// A masked key has the probability 0, but 0 times an infinite or NaN value is NaN, and the MMA multiplies every row of P with every value of the tile.
// In the tiles that reach beyond the first position of a CTA, the warp that issues the MMAs puts 0 in the place of such values and notes
// their keys, one bit each; the rows that see a noted key add its values to the accumulator themselves.  The search is one load and four
// multiply-adds per 16 bytes, mostly under the softmax of the same tile: 4000 positions x 20 heads of 64 take 73.8 us with it, 72.8 without, the
// layered engine's 4096 rows x 16 heads of 128 140 us and 134.

// A V tile [CH][KT keys][128 B]; its key k is bit bit0 + k of `noted`.  The whole warp; the caller's MMAs come after a __syncwarp.
template <int KT, int CH>
__device__ __forceinline__ void flash_take_out_nonfinite(uint8_t* v, uint32_t* noted, int bit0, int lane) {
  uint32_t z[4] = {0, 0, 0, 0};  // 0 * value, added up: NaN in a half once a value is no finite number
  for (int c = 0; c < CH; ++c)
#pragma unroll 8
    for (int b = 0; b < KT * 128; b += 512) {
      const uint4 x = *reinterpret_cast<const uint4*>(v + c * KT * 128 + b + lane * 16);
      const uint32_t u[4] = {x.x, x.y, x.z, x.w};
#pragma unroll
      for (int i = 0; i < 4; ++i) asm("fma.rn.bf16x2 %0, %1, %2, %0;" : "+r"(z[i]) : "r"(u[i]), "r"(0u));
    }
  if (!__any_sync(0xffffffffu, ((z[0] | z[1] | z[2] | z[3]) & 0x7fff7fffu) != 0)) return;
  for (int c = 0; c < CH; ++c)
    for (int b = lane * 16; b < KT * 128; b += 512) {
      uint32_t* x = reinterpret_cast<uint32_t*>(v + c * KT * 128 + b);
      uint32_t out = 0;
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const uint32_t w = x[i], gone = ((w & 0x7f80u) == 0x7f80u ? 0xffffu : 0u) | ((w & 0x7f800000u) == 0x7f800000u ? 0xffff0000u : 0u);
        if (gone) x[i] = w & ~gone;
        out |= gone;
      }
      if (out) atomicOr(&noted[(bit0 + b / 128) >> 5], 1u << ((bit0 + b / 128) & 31));
    }
  fence_proxy_async();
}

// adds the noted keys' values that are no finite numbers, columns c .. c + 31, to the accumulator of a row at `pos`; bit 0 is the key `first`, value(key) a
// key's row.  (Whatever their probability: the sum is no finite number either way.)
template <int WORDS, class V>
__device__ __forceinline__ void flash_add_noted(uint32_t (&o)[32], const uint32_t* noted, int first, int pos, int c, V&& value) {
  for (int w = 0; w < WORDS; ++w)
    for (uint32_t left = noted[w]; left != 0; left &= left - 1) {
      const int key = first + 32 * w + __ffs(left) - 1;
      if (key > pos) return;
      const uint4* row = reinterpret_cast<const uint4*>(value(key) + c);
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const uint4 x = row[i];
        const uint32_t u[4] = {x.x, x.y, x.z, x.w};
#pragma unroll
        for (int e = 0; e < 8; ++e) {
          const float y = __uint_as_float(e & 1 ? u[e >> 1] & 0xffff0000u : u[e >> 1] << 16);
          if (!(fabsf(y) < INFINITY)) o[8 * i + e] = __float_as_uint(__uint_as_float(o[8 * i + e]) + y);
        }
      }
    }
}

}  // namespace mtx
