// Epilogues of the layered engine's projections on the pair GEMM (gemm_wide.cuh), where the 256-row GEMMs leave a bf16 copy that a kernel
// of its own then reads (63 us for 4096 x 4096 to fp32, 121 us for the gate of 4096 x 16384).  The accumulator is rounded to bf16 first,
// as that copy is: a row's result does not depend on how many rows its step has (a router further on turns a rounding into another
// choice of experts).  (ROUND = false: the experts' products, whose kernels keep the accumulator.)  bf16 outputs need 16-byte aligned rows (ldo a multiple of 8), fp32 outputs rows of whole float4s.
#pragma once

#include "gemm_wide.cuh"
#include "linear_any.cuh"

namespace mtx {

template <int EPI, bool ROUND = true>
struct WideLinEpi {
  static constexpr bool kFragments = true;
  const float* bias;
  float* out;
  bf16* act;
  long long ldo;
  float limit;
  int silu0, silu1;

  __device__ __forceinline__ int prepare(const WideTile&) const { return 0; }

  // 32 columns of a row
  __device__ __forceinline__ void fragment(const WideTile& w, int n, int, int c, float (&a)[16], float (&b)[16]) const {
    columns(w, n, c, a);
    columns(w, n, c + 16, b);
  }
  // 16 of them
  __device__ __forceinline__ void columns(const WideTile& w, int n, int c, float (&v)[16]) const {
    constexpr bool gated = EPI == LIN_GATED || EPI == LIN_GATED_CLAMP, narrow = gated || EPI == LIN_ACT || EPI == LIN_RELU2 || EPI == LIN_GELU;
#pragma unroll
    for (int j = 0; ROUND && j < 16; j += 2) {
      const uint32_t b = pack_bf16x2(v[j], v[j + 1]);
      v[j] = bf16_lo(b);
      v[j + 1] = bf16_hi(b);
    }
    const int col = w.n0 + c;
    if (gated) {  // (gate, up) of eight features
      float g[8];
#pragma unroll
      for (int j = 0; j < 8; ++j) {
        const float a = v[2 * j], u = v[2 * j + 1];
        g[j] = EPI == LIN_GATED ? gelu_tanh_f(a) * u : (limit > 0.0f ? clamped_gate_f(a, u, limit) : silu_gate_f(a, u));
      }
      *reinterpret_cast<uint4*>(act + (long long)w.row * ldo + (col >> 1)) =
          make_uint4(pack_bf16x2(g[0], g[1]), pack_bf16x2(g[2], g[3]), pack_bf16x2(g[4], g[5]), pack_bf16x2(g[6], g[7]));
    } else if (narrow) {
#pragma unroll
      for (int j = 0; j < 16; ++j) {
        if (EPI == LIN_GELU) v[j] = gelu_tanh_f(v[j]);
        if (EPI == LIN_RELU2) {
          v[j] = fmaxf(v[j], 0.0f);
          v[j] *= v[j];
        }
      }
      frag_store_bf16(act + (long long)w.row * ldo + col, v);
    } else {
      if (EPI == LIN_SILU_COLS && col + 16 > silu0 && col < silu1) {
#pragma unroll
        for (int j = 0; j < 16; ++j)
          if (col + j >= silu0 && col + j < silu1) v[j] = bf16r(silu_gate_f(v[j], 1.0f));
      }
      if (EPI == LIN_BIAS) {
#pragma unroll
        for (int j = 0; j < 16; j += 4) {
          const float4 b = __ldg(reinterpret_cast<const float4*>(bias + col + j));
          v[j] += b.x;
          v[j + 1] += b.y;
          v[j + 2] += b.z;
          v[j + 3] += b.w;
        }
      }
      float4* o = reinterpret_cast<float4*>(out + (long long)w.row * ldo + col);
#pragma unroll
      for (int j = 0; j < 4; ++j) o[j] = make_float4(v[4 * j], v[4 * j + 1], v[4 * j + 2], v[4 * j + 3]);
    }
  }

  template <class LD>
  __device__ __forceinline__ void operator()(const WideTile& w, int n, int, LD&& ld16) const {
    for (int c = w.c0; c < w.c1; c += 16) {
      float v[16];
      ld16(c, v);
      if (w.valid) columns(w, n, c, v);
    }
  }
};

}  // namespace mtx
