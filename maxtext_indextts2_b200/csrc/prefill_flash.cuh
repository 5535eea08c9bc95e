// Causal GQA attention of a long prompt's rows on tcgen05 (MaxEngine._prefill_jit, MaxText/maxengine.py:400-530; AttentionOp.apply_attention_dot
// with the causal + segment mask of attentions.py:606-643): the passes of more than 256 rows, whose keys and values sit in the prefill segment of
// one cache plane (rows of earlier passes, and this pass's own, written just before).
//
// CTA = (query head, NQ x 128 query positions).  Tiles of KT keys stream through a TMA ring; per tile and 128 positions
//   S = Q K^T      tcgen05.mma, M = 128, N = KT, fp32 in TMEM
//   P = exp2(..)   four softmax warps: a thread owns a position, reads its S row from TMEM, keeps maximum and sum in fp32 registers and writes
//                  P as bf16 over S
//   O += P V       tcgen05.mma with P as the TMEM operand and V as an MN-major operand (as the cache rows lie), fp32 in TMEM
// The accumulator is brought to a new maximum only when a position's maximum grew by more than 2^8 (its probabilities then reach 2^8 instead of 1;
// their relative rounding is the same), which after the first tiles is hardly ever: a rescale reads and writes D columns of TMEM.
//
//   D = 64:   NQ = 1, KT = 128, half of the TMEM: two CTAs per SM, each under the other's MMAs.  20 heads x 16 CTAs of 256 positions (NQ = 2, one CTA
//             per SM) left SMs idle behind the longest ones: 87 us for 4000 positions, 74 so
//   D = 128:  NQ = 2, KT = 128: the MMAs of one half of the positions run under the softmax of the other
//
// Bound: the special-function units at D = 64 (one exp2 per score: 16 per SM and clock), 4000 positions x 20 heads: 36 us at least.
// The mma.sync kernel (prefill_attention.cuh), 256 rows per launch, reads every tile for 16 positions at a time: 787 us for the same.  With the
// projections on the pair GEMM a prompt of 4000 tokens (24 layers) went from 37.1 to 6.4 ms.
#pragma once

#include "attention.cuh"
#include "flash_tmem.cuh"

namespace mtx {

constexpr float kPfLog2e = 1.4426950408889634f;

struct PrefillFlashParams {
  bf16* out;       // [rows, hq * D]
  const bf16* v;   // the cache rows of tm_v
  int rows;        // positions of the pass
  int start_pos;   // position of row 0
  int hq, hkv, T;
  int plane_row0;  // cache row of (layer, plane, kv head 0, position 0) in the K / V tensor maps; kv head h adds h * T
  float softcap;
};

template <int D>
struct FlashShape {
  static constexpr int NQ = D == 64 ? 1 : 2, KT = 128;
  static constexpr int kStages = 2;
  static constexpr int kThreads = 64 + NQ * 128, kCtas = D == 64 ? 2 : 1;  // CTAs per SM
  static constexpr int kQBytes = 128 * D * 2, kTileBytes = KT * D * 2;    // a Q tile; a K or a V tile
  static constexpr int kOCol = NQ * KT, kTmemCols = 512 / kCtas;           // first TMEM column of the accumulators; columns in all
  static constexpr int kNoteWords = (NQ * 128 + KT) / 32;                  // keys of the tiles that reach beyond the first position: at most so many bits
};

struct FlashTail {
  uint64_t q_full;
  uint64_t k_full[4], v_full[4], empty[4];
  uint64_t s_full[2], p_ready[2], o_done[2];
  uint64_t noted_all[2];  // the keys that a Q tile's rows see are searched
  uint32_t noted[12];     // see flash_take_out_nonfinite
  uint32_t tmem_base;
  uint32_t pad;
};

template <int D>
inline size_t prefill_flash_smem_bytes() {
  typedef FlashShape<D> F;
  return 1024 + size_t(F::NQ) * F::kQBytes + size_t(F::kStages) * 2 * F::kTileBytes + sizeof(FlashTail) + 16;
}

__device__ __forceinline__ float flash_ex2(float x) {
  float y;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}

// grid (query heads, ceil(rows / (NQ * 128))); blockIdx.y counts from the last positions, whose CTAs have the most keys
template <int D>
__global__ void __launch_bounds__(FlashShape<D>::kThreads, FlashShape<D>::kCtas)
prefill_flash_kernel(const __grid_constant__ CUtensorMap tm_q, const __grid_constant__ CUtensorMap tm_k, const __grid_constant__ CUtensorMap tm_v,
                     const PrefillFlashParams p) {
  typedef FlashShape<D> F;
  constexpr int NQ = F::NQ, KT = F::KT, CH = D / 64;  // CH: 64-channel chunks of a row
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = smem_raw + ((1024u - (smem_u32(smem_raw) & 1023u)) & 1023u);
  uint8_t* sq = smem;                              // [NQ][CH][128 rows][128 B]
  uint8_t* ring = sq + NQ * F::kQBytes;            // stage: K [CH][KT rows][128 B], then V
  FlashTail* tail = reinterpret_cast<FlashTail*>(ring + F::kStages * 2 * F::kTileBytes);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int head = blockIdx.x, h = head / (p.hq / p.hkv);
  const int q0 = (int(gridDim.y) - 1 - int(blockIdx.y)) * NQ * 128;
  const int plane_row = p.plane_row0 + h * p.T;
  // key tiles of the 128 positions from q0 + 128 t on: 0 .. last[t]; none when the pass has no such rows
  int last[NQ], hi = -1;
#pragma unroll
  for (int t = 0; t < NQ; ++t) {
    const int r0 = q0 + 128 * t, r1 = (r0 + 128 < p.rows ? r0 + 128 : p.rows) - 1;
    last[t] = r1 >= r0 ? (p.start_pos + r1) / KT : -1;
    hi = last[t] > hi ? last[t] : hi;
  }
  const int masked = (p.start_pos + q0 + 1) / KT;  // the first tile with keys beyond the CTA's first position

  griddep_launch_dependents();
  static_assert(F::kNoteWords <= 12, "FlashTail::noted");
  if (threadIdx.x < F::kNoteWords) tail->noted[threadIdx.x] = 0;
  if (warp == 0 && lane == 0) {
    tma_prefetch_desc(&tm_q);
    tma_prefetch_desc(&tm_k);
    tma_prefetch_desc(&tm_v);
    mbar_init(&tail->q_full, 1);
    for (int s = 0; s < F::kStages; ++s) {
      mbar_init(&tail->k_full[s], 1);
      mbar_init(&tail->v_full[s], 1);
      mbar_init(&tail->empty[s], 1);
    }
    for (int t = 0; t < 2; ++t) {
      mbar_init(&tail->s_full[t], 1);
      mbar_init(&tail->p_ready[t], 4);  // one arrival per softmax warp
      mbar_init(&tail->o_done[t], 1);
      mbar_init(&tail->noted_all[t], 1);
    }
    fence_barrier_init();
  }
  if (warp == 1) {
    tmem_alloc(&tail->tmem_base, F::kTmemCols);
    tmem_relinquish();
  }
  tcgen05_fence_before();
  __syncthreads();
  tcgen05_fence_after();
  const uint32_t tmem = tail->tmem_base;
  griddep_wait();  // q, and this pass's K / V rows, come from the kernel before

  if (warp == 0) {
    const bool issuer = elect_one();
    if (issuer) {
      mbar_expect_tx(&tail->q_full, uint32_t(NQ * F::kQBytes));
      for (int t = 0; t < NQ; ++t)
        for (int c = 0; c < CH; ++c) tma_load_2d(sq + t * F::kQBytes + c * 16384, &tm_q, head * D + c * 64, q0 + 128 * t, &tail->q_full, kEvictFirst);
    }
    int s = 0;
    uint32_t phase = 1;
    for (int j = 0; j <= hi; ++j) {
      mbar_wait(&tail->empty[s], phase);
      if (issuer) {
        uint8_t* st = ring + s * 2 * F::kTileBytes;
        for (int kv = 0; kv < 2; ++kv) {
          uint64_t* bar = kv == 0 ? &tail->k_full[s] : &tail->v_full[s];
          mbar_expect_tx(bar, uint32_t(F::kTileBytes));
          for (int c = 0; c < CH; ++c)
            for (int k = 0; k < KT; k += 64)  // (the cache's tensor maps have boxes of 64 rows)
              tma_load_2d(st + kv * F::kTileBytes + c * KT * 128 + k * 128, kv == 0 ? &tm_k : &tm_v, c * 64, plane_row + j * KT + k, bar, kEvictLast);
        }
      }
      if (++s == F::kStages) s = 0, phase ^= 1;
    }
  } else if (warp == 1) {
    const bool issuer = elect_one();
    const uint32_t idesc_s = umma_idesc_bf16(128, KT), idesc_o = umma_idesc_bf16(128, D) | kIdescBMajorMN;
    const uint64_t dq = umma_desc_sw128(sq), dk = umma_desc_sw128(ring);
    const uint32_t ring_addr = smem_u32(ring);
    // S of Q tile t from the K tile of `stage`
    auto issue_s = [&](int t, int stage) {
      if (!issuer) return;
#pragma unroll
      for (int c = 0; c < CH; ++c)
#pragma unroll
        for (int kk = 0; kk < 4; ++kk)
          umma_bf16(tmem + t * KT, dq + uint64_t((t * F::kQBytes + c * 16384 + kk * 32) >> 4), dk + uint64_t((stage * 2 * F::kTileBytes + c * KT * 128 + kk * 32) >> 4),
                    idesc_s, uint32_t((c | kk) != 0));
      umma_commit(&tail->s_full[t]);
    };
    // O of Q tile t += P (over its S) times the V tile of `stage`
    auto issue_o = [&](int t, int stage, bool start) {
      if (!issuer) return;
#pragma unroll
      for (int kk = 0; kk < KT / 16; ++kk)
        umma_bf16_ts(tmem + F::kOCol + t * D, tmem + t * KT + kk * 8, umma_desc_sw128_mn(ring_addr + stage * 2 * F::kTileBytes + F::kTileBytes + kk * 2048, KT * 128), idesc_o,
                     uint32_t(!start || kk != 0));
    };
    mbar_wait(&tail->q_full, 0);
    int s = 0;
    uint32_t par = 0;
    if (hi >= 0) {
      mbar_wait(&tail->k_full[0], 0);
      tcgen05_fence_after();
#pragma unroll
      for (int t = 0; t < NQ; ++t)
        if (last[t] >= 0) issue_s(t, 0);
    }
    for (int j = 0; j <= hi; ++j) {
      const int s1 = s + 1 == F::kStages ? 0 : s + 1;
      const uint32_t par1 = s1 == 0 ? par ^ 1 : par;
      if (j < hi) {
        mbar_wait(&tail->k_full[s1], par1);
        tcgen05_fence_after();
      }
      mbar_wait(&tail->v_full[s], par);
      const int beyond = p.start_pos + p.rows - j * KT;  // the tile's first key that the prompt does not have
      uint8_t* v = ring + s * 2 * F::kTileBytes + F::kTileBytes;
      if (beyond < KT) {                                 // rows of no key may hold anything, and 0 * NaN is not 0
        for (int c = 0; c < CH; ++c)
          for (int b = beyond * 128 + lane * 16; b < KT * 128; b += 512) *reinterpret_cast<uint4*>(v + c * KT * 128 + b) = make_uint4(0, 0, 0, 0);
        fence_proxy_async();
        __syncwarp();
      }
      if (j >= masked) {
        flash_take_out_nonfinite<KT, CH>(v, tail->noted, (j - masked) * KT, lane);
        __syncwarp();
#pragma unroll
        for (int t = 0; t < NQ; ++t)
          if (j == last[t] && lane == 0) mbar_arrive(&tail->noted_all[t]);
      }
#pragma unroll
      for (int t = 0; t < NQ; ++t) {
        if (j <= last[t]) {
          mbar_wait(&tail->p_ready[t], j & 1);
          tcgen05_fence_after();
          issue_o(t, s, j == 0);
          if (issuer && j == last[t]) umma_commit(&tail->o_done[t]);
        }
        if (j < last[t]) issue_s(t, s1);
      }
      if (issuer) umma_commit(&tail->empty[s]);
      s = s1;
      par = par1;
    }
    // the commits to the ring's barriers have to be in before the CTA may leave
    const int tail_n = hi + 1 < F::kStages ? hi + 1 : F::kStages;
    for (int i = 0; i < tail_n; ++i) {
      if (s == 0) s = F::kStages, par ^= 1;
      --s;
      mbar_wait(&tail->empty[s], par);
    }
  } else {
    const int t = (warp - 2) >> 2, quarter = warp & 3;
    const int row = q0 + 128 * t + quarter * 32 + lane, pos = p.start_pos + row;
    const int pos_lo = p.start_pos + q0 + 128 * t + quarter * 32;  // the warp's first position
    const uint32_t lanes = tmem + (uint32_t(quarter * 32) << 16), acc = lanes + F::kOCol + t * D;
    float m = -INFINITY, l = 0.0f;  // the maximum that the accumulator stands at (times log2 e), the sum
    int la = -1;
#pragma unroll
    for (int i = 0; i < NQ; ++i)
      if (i == t) la = last[i];
    for (int j = 0; j <= la; ++j) {
      mbar_wait(&tail->s_full[t], j & 1);
      tcgen05_fence_after();
      float x[KT];
      {
        uint32_t raw[KT / 32][32];
#pragma unroll
        for (int c = 0; c < KT / 32; ++c) tmem_ld_x32(lanes + t * KT + c * 32, raw[c]);
        tmem_wait_ld();
#pragma unroll
        for (int c = 0; c < KT; ++c) x[c] = __uint_as_float(raw[c / 32][c % 32]);
      }
      if (p.softcap != 0.0f) {
#pragma unroll
        for (int c = 0; c < KT; ++c) x[c] = tanhf(x[c] / p.softcap) * p.softcap;
      }
      const int key0 = j * KT;
      if (key0 + KT - 1 > pos_lo) {  // (uniform in the warp)
        const int over = pos - key0;
#pragma unroll
        for (int c = 0; c < KT; ++c)
          if (c > over) x[c] = -INFINITY;
      }
      float mx0 = x[0], mx1 = x[1], mx2 = x[2], mx3 = x[3];
#pragma unroll
      for (int c = 4; c < KT; c += 4) {
        mx0 = fmaxf(mx0, x[c]);
        mx1 = fmaxf(mx1, x[c + 1]);
        mx2 = fmaxf(mx2, x[c + 2]);
        mx3 = fmaxf(mx3, x[c + 3]);
      }
      const float m_new = fmaxf(m, fmaxf(fmaxf(mx0, mx1), fmaxf(mx2, mx3)) * kPfLog2e);
      if (__any_sync(0xffffffffu, m_new > m + 8.0f)) {  // (m = -inf: the first keys that the position sees)
        const float fix = m_new == -INFINITY ? 1.0f : flash_ex2(m - m_new);
        l *= fix;
        m = m_new;
        if (j > 0) {  // the accumulator holds the tiles before: they are complete (s_full came after them in order)
#pragma unroll 1
          for (int c = 0; c < D; c += 16) {
            float o[16];
            tmem_ld_x16(acc + c, o);
            uint32_t w[16];
#pragma unroll
            for (int e = 0; e < 16; ++e) w[e] = __float_as_uint(o[e] * fix);
            tmem_st_x16(acc + c, w);
          }
        }
      }
      const float ms = m == -INFINITY ? 0.0f : m;
      float l0 = 0.0f, l1 = 0.0f;
#pragma unroll
      for (int c = 0; c < KT; c += 32) {
        uint32_t pk[16];
#pragma unroll
        for (int e = 0; e < 16; ++e) {
          const float p0 = flash_ex2(fmaf(x[c + 2 * e], kPfLog2e, -ms)), p1 = flash_ex2(fmaf(x[c + 2 * e + 1], kPfLog2e, -ms));
          l0 += p0;
          l1 += p1;
          pk[e] = pack_bf16x2(p0, p1);
        }
        tmem_st_x16(lanes + t * KT + c / 2, pk);
      }
      l += l0 + l1;
      tmem_wait_st();
      tcgen05_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(&tail->p_ready[t]);
    }
    if (la >= 0) {
      mbar_wait(&tail->o_done[t], 0);
      tcgen05_fence_after();
      uint32_t noted = 0;
      if (la >= masked) {
        mbar_wait(&tail->noted_all[t], 0);
#pragma unroll
        for (int w = 0; w < F::kNoteWords; ++w) noted |= tail->noted[w];
      }
      const float inv = 1.0f / l;
      bf16* out = p.out + (long long)row * p.hq * D + (long long)head * D;
#pragma unroll 1
      for (int c = 0; c < D; c += 32) {
        uint32_t o[32];
        tmem_ld_x32(acc + c, o);
        tmem_wait_ld();
        if (row < p.rows) {
          if (noted != 0)
            flash_add_noted<F::kNoteWords>(o, tail->noted, masked * KT, pos, c, [&](int key) { return p.v + (long long)(plane_row + key) * D; });
#pragma unroll
          for (int e = 0; e < 32; e += 8) {
            uint32_t w[4];
#pragma unroll
            for (int i = 0; i < 4; ++i) w[i] = pack_bf16x2(__uint_as_float(o[e + 2 * i]) * inv, __uint_as_float(o[e + 2 * i + 1]) * inv);
            *reinterpret_cast<uint4*>(out + c + e) = make_uint4(w[0], w[1], w[2], w[3]);
          }
        }
      }
    }
  }
  tcgen05_fence_before();
  __syncthreads();
  tcgen05_fence_after();
  if (warp == 1) tmem_dealloc(tmem, F::kTmemCols);
}

}  // namespace mtx
