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

  static constexpr bool kGated = EPI == LIN_GATED || EPI == LIN_GATED_CLAMP, kNarrow = kGated || EPI == LIN_ACT || EPI == LIN_RELU2 || EPI == LIN_GELU;
  static constexpr int kChunks = kGated ? 2 : kNarrow ? 4 : 8;  // 16-byte chunks that 32 columns become
  static constexpr int kRowBytes = kNarrow ? 64 : 128;
  typedef WideStage<kRowBytes> Stage;

  __device__ __forceinline__ int prepare(const WideTile&, const Stage&) const { return 0; }

  // 32 columns of a row
  __device__ __forceinline__ void fragment(const WideTile& w, int, int c, float (&a)[16], float (&b)[16], const Stage& st) const {
    const int chunk = st.template chunk<kChunks>(w, c);
    if (w.valid) {  // (a row that is not there is zeros: 0 / x takes the quotient's slow way, alone in its warp)
      columns(w.n0 + c, a, chunk, st);
      columns(w.n0 + c + 16, b, chunk + kChunks / 2, st);
    }
    const long long row0 = (long long)(w.row - st.lane) * ldo;
    if constexpr (kNarrow) st.template done<kChunks>(w, c, act + row0 + ((w.n0 + w.c0) >> (kGated ? 1 : 0)), size_t(ldo) * 2);
    else st.template done<kChunks>(w, c, out + row0 + w.n0 + w.c0, size_t(ldo) * 4);
  }
  // 16 of them, from column col of the output on, into the chunks from `chunk` on
  __device__ __forceinline__ void columns(int col, float (&v)[16], int chunk, const Stage& st) const {
#pragma unroll
    for (int j = 0; ROUND && j < 16; j += 2) {
      const uint32_t b = pack_bf16x2(v[j], v[j + 1]);
      v[j] = bf16_lo(b);
      v[j + 1] = bf16_hi(b);
    }
    if constexpr (kGated) {  // (gate, up) of eight features
      float g[8];
#pragma unroll
      for (int j = 0; j < 8; ++j) {
        const float a = v[2 * j], u = v[2 * j + 1];
        g[j] = EPI == LIN_GATED ? gelu_tanh_f(a) * u : (limit > 0.0f ? clamped_gate_f(a, u, limit) : silu_gate_f(a, u));
      }
      st.put(chunk, wide_pack8(g));
    } else if constexpr (kNarrow) {
#pragma unroll
      for (int j = 0; j < 16; ++j) {
        if (EPI == LIN_GELU) v[j] = gelu_tanh_f(v[j]);
        if (EPI == LIN_RELU2) {
          v[j] = fmaxf(v[j], 0.0f);
          v[j] *= v[j];
        }
      }
      st.put(chunk, wide_pack8(v));
      st.put(chunk + 1, wide_pack8(v + 8));
    } else {
      if (EPI == LIN_SILU_COLS && col + 16 > silu0 && col < silu1) {
#pragma unroll
        for (int j = 0; j < 16; ++j) {
          const float g = bf16r(silu_gate_f(v[j], 1.0f));
          v[j] = col + j >= silu0 && col + j < silu1 ? g : v[j];
        }
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
#pragma unroll
      for (int j = 0; j < 4; ++j)
        st.put(chunk + j, make_uint4(__float_as_uint(v[4 * j]), __float_as_uint(v[4 * j + 1]), __float_as_uint(v[4 * j + 2]), __float_as_uint(v[4 * j + 3])));
    }
  }
};

}  // namespace mtx
