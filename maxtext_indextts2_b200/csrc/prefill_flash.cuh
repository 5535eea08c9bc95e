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
//   D = 64, 128:  NQ = 2, KT = 128: the MMAs of one half of the positions run under the softmax of the other
//   D = 256:      NQ = 1, KT = 64 (the accumulator takes 256 of the 512 TMEM columns, Q, K and V 192 KB): two S buffers, the next tile's S
//                 is issued before this tile's P V
//
// Bound: the special-function units at D = 64 (one exp2 per score: 16 per SM and clock), 4000 positions x 20 heads: 36 us at least.
// The mma.sync kernel (prefill_attention.cuh), 256 rows per launch, reads every tile for 16 positions at a time: 787 us for the same.  With the
// projections on the pair GEMM a prompt of 4000 tokens (24 layers) went from 37.1 to 6.8 ms, 3001 tokens through six gemma3 layers with heads of
// 256 from 17.5 to 3.7 ms.
#pragma once

#include "attention.cuh"
#include "flash_tmem.cuh"

namespace mtx {

constexpr float kPfLog2e = 1.4426950408889634f;

struct PrefillFlashParams {
  bf16* out;       // [rows, hq * D]
  int rows;        // positions of the pass
  int start_pos;   // position of row 0
  int hq, hkv, T;
  int plane_row0;  // cache row of (layer, plane, kv head 0, position 0) in the K / V tensor maps; kv head h adds h * T
  float softcap;
  int window;      // > 0: a query sees the keys (position - window, position]
};

template <int D>
struct FlashShape {
  static constexpr int NQ = D == 256 ? 1 : 2, KT = D == 256 ? 64 : 128;
  static constexpr int kStages = D == 64 ? 4 : 2;
  static constexpr int kThreads = 64 + NQ * 128;
  static constexpr int kQBytes = 128 * D * 2, kTileBytes = KT * D * 2;  // a Q tile; a K or a V tile
  static constexpr int kSBufs = 2;                                       // S of each Q tile (NQ = 2), or of alternate key tiles (NQ = 1)
  static constexpr int kOCol = kSBufs * KT;                              // first TMEM column of the accumulators
};

struct FlashTail {
  uint64_t q_full;
  uint64_t k_full[4], v_full[4], empty[4];
  uint64_t s_full[2], p_ready[2], o_done[2];
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
__global__ void __launch_bounds__(FlashShape<D>::kThreads, 1)
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
  // key tiles of the 128 positions from q0 + 128 t on: [first[t], last[t]]; none when the pass has no such rows
  int first[NQ], last[NQ], lo = 1 << 30, hi = -1;
#pragma unroll
  for (int t = 0; t < NQ; ++t) {
    const int r0 = q0 + 128 * t, r1 = (r0 + 128 < p.rows ? r0 + 128 : p.rows) - 1;
    const int k0 = p.window > 0 && p.start_pos + r0 - p.window + 1 > 0 ? p.start_pos + r0 - p.window + 1 : 0;
    first[t] = r1 >= r0 ? k0 / KT : 1 << 30;
    last[t] = r1 >= r0 ? (p.start_pos + r1) / KT : -1;
    lo = first[t] < lo ? first[t] : lo;
    hi = last[t] > hi ? last[t] : hi;
  }

  griddep_launch_dependents();
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
    }
    fence_barrier_init();
  }
  if (warp == 1) {
    tmem_alloc(&tail->tmem_base, 512);
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
    for (int j = lo; j <= hi; ++j) {
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
    // S of Q tile t from the K tile of `stage`, into the TMEM buffer `buf`
    auto issue_s = [&](int t, int stage, int buf) {
      if (!issuer) return;
#pragma unroll
      for (int c = 0; c < CH; ++c)
#pragma unroll
        for (int kk = 0; kk < 4; ++kk)
          umma_bf16(tmem + buf * KT, dq + uint64_t((t * F::kQBytes + c * 16384 + kk * 32) >> 4), dk + uint64_t((stage * 2 * F::kTileBytes + c * KT * 128 + kk * 32) >> 4),
                    idesc_s, uint32_t((c | kk) != 0));
      umma_commit(&tail->s_full[buf]);
    };
    // O of Q tile t += P (over S in buffer `buf`) times the V tile of `stage`
    auto issue_o = [&](int t, int stage, int buf, bool start) {
      if (!issuer) return;
#pragma unroll
      for (int kk = 0; kk < KT / 16; ++kk)
        umma_bf16_ts(tmem + F::kOCol + t * D, tmem + buf * KT + kk * 8, umma_desc_sw128_mn(ring_addr + stage * 2 * F::kTileBytes + F::kTileBytes + kk * 2048, KT * 128), idesc_o,
                     uint32_t(!start || kk != 0));
    };
    mbar_wait(&tail->q_full, 0);
    int s = 0;
    uint32_t par = 0, seen[2] = {0, 0};  // seen[b]: parity of the next P in buffer b
    if (lo <= hi) {
      mbar_wait(&tail->k_full[0], 0);
      tcgen05_fence_after();
#pragma unroll
      for (int t = 0; t < NQ; ++t)
        if (first[t] == lo) issue_s(t, 0, NQ == 2 ? t : 0);
    }
    for (int j = lo; j <= hi; ++j) {
      const int s1 = s + 1 == F::kStages ? 0 : s + 1;
      const uint32_t par1 = s1 == 0 ? par ^ 1 : par;
      if (j < hi) {
        mbar_wait(&tail->k_full[s1], par1);
        tcgen05_fence_after();
        if (NQ == 1) issue_s(0, s1, (j + 1 - lo) & 1);  // under this tile's softmax
      }
#pragma unroll
      for (int t = 0; t < NQ; ++t) {
        const int buf = NQ == 2 ? t : (j - lo) & 1;
        if (j >= first[t] && j <= last[t]) {
          mbar_wait(&tail->p_ready[buf], seen[buf]);
          seen[buf] ^= 1;
          mbar_wait(&tail->v_full[s], par);
          tcgen05_fence_after();
          issue_o(t, s, buf, j == first[t]);
          if (issuer && (NQ == 1 || j == last[t])) umma_commit(&tail->o_done[t]);
        }
        if (NQ == 2 && j < hi && j + 1 >= first[t] && j + 1 <= last[t]) issue_s(t, s1, t);
      }
      if (issuer) umma_commit(&tail->empty[s]);
      s = s1;
      par = par1;
    }
    // the commits to the ring's barriers have to be in before the CTA may leave
    const int n = hi - lo + 1, tail_n = n < F::kStages ? (n > 0 ? n : 0) : F::kStages;
    for (int i = 0; i < tail_n; ++i) {
      if (s == 0) s = F::kStages, par ^= 1;
      --s;
      mbar_wait(&tail->empty[s], par);
    }
  } else {
    const int t = NQ == 2 ? (warp - 2) >> 2 : 0, quarter = warp & 3;
    const int row = q0 + 128 * t + quarter * 32 + lane, pos = p.start_pos + row;
    const int pos_lo = p.start_pos + q0 + 128 * t + quarter * 32, pos_hi = pos_lo + 31;  // of the warp
    const uint32_t lanes = tmem + (uint32_t(quarter * 32) << 16), acc = lanes + F::kOCol + t * D;
    float m = -INFINITY, l = 0.0f;  // the maximum that the accumulator stands at (times log2 e), the sum
    int f = 0, la = -1;
#pragma unroll
    for (int i = 0; i < NQ; ++i)
      if (i == t) f = first[i], la = last[i];
    for (int j = f; j <= la; ++j) {
      const int i = j - f, buf = NQ == 2 ? t : i & 1;
      mbar_wait(&tail->s_full[buf], NQ == 2 ? (i & 1) : ((i >> 1) & 1));
      tcgen05_fence_after();
      float x[KT];
      {
        uint32_t raw[KT / 32][32];
#pragma unroll
        for (int c = 0; c < KT / 32; ++c) tmem_ld_x32(lanes + buf * KT + c * 32, raw[c]);
        tmem_wait_ld();
#pragma unroll
        for (int c = 0; c < KT; ++c) x[c] = __uint_as_float(raw[c / 32][c % 32]);
      }
      if (p.softcap != 0.0f) {
#pragma unroll
        for (int c = 0; c < KT; ++c) x[c] = tanhf(x[c] / p.softcap) * p.softcap;
      }
      const int key0 = j * KT;
      if (key0 + KT - 1 > pos_lo || (p.window > 0 && key0 <= pos_hi - p.window)) {  // (uniform in the warp)
        const int over = pos - key0, under = p.window > 0 ? pos - p.window - key0 : -1;  // keys key0 + c with under < c <= over are seen
#pragma unroll
        for (int c = 0; c < KT; ++c)
          if (c > over || c <= under) x[c] = -INFINITY;
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
        if (i > 0) {  // the accumulator holds the tiles before: they are complete (NQ = 2: s_full came after them in order)
          if (NQ == 1) {
            mbar_wait(&tail->o_done[0], (i - 1) & 1);
            tcgen05_fence_after();
          }
#pragma unroll 1
          for (int c = 0; c < D; c += 32) {
            uint32_t o[32];
            tmem_ld_x32(acc + c, o);
            tmem_wait_ld();
#pragma unroll
            for (int e = 0; e < 32; ++e) o[e] = __float_as_uint(__uint_as_float(o[e]) * fix);
            tmem_st_x32(acc + c, o);
          }
        }
      }
      const float ms = m == -INFINITY ? 0.0f : m;
      float l0 = 0.0f, l1 = 0.0f;
#pragma unroll
      for (int c = 0; c < KT; c += 64) {
        uint32_t pk[32];
#pragma unroll
        for (int e = 0; e < 32; ++e) {
          const float p0 = flash_ex2(fmaf(x[c + 2 * e], kPfLog2e, -ms)), p1 = flash_ex2(fmaf(x[c + 2 * e + 1], kPfLog2e, -ms));
          l0 += p0;
          l1 += p1;
          pk[e] = pack_bf16x2(p0, p1);
        }
        tmem_st_x32(lanes + buf * KT + c / 2, pk);
      }
      l += l0 + l1;
      tmem_wait_st();
      tcgen05_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(&tail->p_ready[buf]);
    }
    if (la >= f) {
      mbar_wait(&tail->o_done[t], NQ == 2 ? 0 : ((la - f) & 1));
      tcgen05_fence_after();
      const float inv = 1.0f / l;
      bf16* out = p.out + (long long)row * p.hq * D + (long long)head * D;
#pragma unroll 1
      for (int c = 0; c < D; c += 32) {
        uint32_t o[32];
        tmem_ld_x32(acc + c, o);
        tmem_wait_ld();
        if (row < p.rows) {
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
  if (warp == 1) tmem_dealloc(tmem, 512);
}

}  // namespace mtx
