// The layered engine's causal softmax attention (softmax_attention.cuh) of long runs on tcgen05, over the paged cache, for layers whose queries see
// every key before them (no window, chunks or pooled blocks); sinks, capped scores, distance penalties and gates as there.
//
// The bits are softmax_attention_mma_kernel's: the same key tiles (KT = 64, 32 for heads of 256), the running maximum of every tile (the
// accumulator follows it at once; a multiplication by 1 is left out, nothing else), a row's sum in the same four parts, probabilities rounded
// to bf16 against the same maximum, and products that add the same 16 terms at a time -- tcgen05.mma and mma.sync round alike.  Routers behind
// an attention layer then choose what they chose in steps of shorter runs.  Behind a window the mma.sync kernel's tiles begin at the
// window of each 16 rows; those layers stay there.
//
// CTA = (query head, NQ x 128 rows of one run); it finds its run by walking the runs' row ranges: gridDim.y covers rows / (NQ 128) + n_runs
// tiles, CTAs without one leave.  As in prefill_flash.cuh a thread of the softmax warps owns a row; S is free as soon as it is in registers.
//
// Bound: tcgen05 (43 us at the sizes below); what it spends is the softmax warps' time, half of it for the rescales.  4096 rows, 16 heads of 128
// over 4 key heads: 140 us.  softmax_attention_mma_kernel, where a warp reads all of a tile's K and V for 16 rows of one head, takes 700.
#pragma once

#include "flash_tmem.cuh"
#include "softmax_attention.cuh"

namespace mtx {

template <int D>
struct PagedFlashShape {
  static constexpr int NQ = D == 256 ? 1 : 2, KT = D == 256 ? 32 : 64;
  static constexpr int kStages = 4;
  static constexpr int kThreads = 64 + NQ * 128;
  static constexpr int kQBytes = 128 * D * 2, kTileBytes = KT * D * 2;
  static constexpr int kPCol = NQ * KT, kOCol = 256;  // TMEM columns: S, P, accumulators
  static constexpr int kNoteWords = (NQ * 128 + KT) / 32;  // keys of the tiles that reach beyond the first position: at most so many bits
};
struct PagedFlashTail {
  uint64_t q_full;
  uint64_t k_full[4], v_full[4], empty[4];
  uint64_t s_full[2], s_free[2], p_ready[2], o_done[2];
  uint64_t noted_all[2];  // the keys that a Q tile's rows see are searched
  uint32_t noted[10];     // see flash_take_out_nonfinite
  uint32_t tmem_base;
  uint32_t pad;
};

template <int D>
inline size_t paged_flash_smem_bytes() {
  typedef PagedFlashShape<D> F;
  return 1024 + size_t(F::NQ) * F::kQBytes + size_t(F::kStages) * 2 * F::kTileBytes + sizeof(PagedFlashTail) + 16;
}

struct PagedFlashArgs {
  SoftmaxAttnArgs<bf16> a;
  const int* run_row0;  // [n_runs + 1]
  int n_runs;
  int box;  // rows of a K / V copy: a page, or a part of one, at most KT
};

template <int D>
__global__ void __launch_bounds__(PagedFlashShape<D>::kThreads, 1)
paged_flash_kernel(const __grid_constant__ CUtensorMap tm_q, const __grid_constant__ CUtensorMap tm_k, const __grid_constant__ CUtensorMap tm_v, const PagedFlashArgs p) {
  typedef PagedFlashShape<D> F;
  constexpr int NQ = F::NQ, KT = F::KT, CH = D / 64;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = smem_raw + ((1024u - (smem_u32(smem_raw) & 1023u)) & 1023u);
  uint8_t* sq = smem;                    // [NQ][CH][128 rows][128 B]
  uint8_t* ring = sq + NQ * F::kQBytes;  // stage: K [CH][KT rows][128 B], then V
  PagedFlashTail* tail = reinterpret_cast<PagedFlashTail*>(ring + F::kStages * 2 * F::kTileBytes);
  const SoftmaxAttnArgs<bf16>& a = p.a;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  griddep_wait();
  // this CTA's rows: tile blockIdx.y of the runs' tiles, a run's last tile first (it has the most keys)
  int run = 0, left = int(blockIdx.y), r_begin = 0, r_end = 0;
  for (; run < p.n_runs; ++run) {
    r_begin = p.run_row0[run];
    r_end = p.run_row0[run + 1];
    const int nt = (r_end - r_begin + NQ * 128 - 1) / (NQ * 128);
    if (left < nt) {
      left = nt - 1 - left;
      break;
    }
    left -= nt;
  }
  if (run == p.n_runs) return;
  const int head = blockIdx.x, kvh = head / (a.heads / a.kv_heads);
  const int r0 = r_begin + left * NQ * 128;                       // first row
  const int p0 = a.pos[r_begin] + left * NQ * 128;                // its position
  const int p_end = a.pos[r_begin] + (r_end - r_begin) - 1;       // the run's last position
  const int* pages = a.page_map + size_t(a.group[r_begin]) * a.max_pages;
  const int tpp = a.tokens_per_page;
  int last[NQ], hi = -1;  // last key tile of the Q tiles (-1: the run has no such rows)
#pragma unroll
  for (int t = 0; t < NQ; ++t) {
    const int q_lo = p0 + 128 * t, q_hi = q_lo + 127 < p_end ? q_lo + 127 : p_end;
    last[t] = q_hi >= q_lo ? q_hi / KT : -1;
    hi = last[t] > hi ? last[t] : hi;
  }
  const int masked = (p0 + 1) / KT;  // the first tile with keys beyond the CTA's first position

  static_assert(F::kNoteWords <= 10, "PagedFlashTail::noted");
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
      mbar_init(&tail->s_free[t], 4);
      mbar_init(&tail->p_ready[t], 4);
      mbar_init(&tail->o_done[t], 1);
      mbar_init(&tail->noted_all[t], 1);
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
  griddep_launch_dependents();

  if (warp == 0) {
    const bool issuer = elect_one();
    if (issuer) {
      mbar_expect_tx(&tail->q_full, uint32_t(NQ * F::kQBytes));
      for (int t = 0; t < NQ; ++t)
        for (int c = 0; c < CH; ++c) tma_load_2d(sq + t * F::kQBytes + c * 16384, &tm_q, head * D + c * 64, r0 + 128 * t, &tail->q_full, kEvictFirst);
    }
    const int boxes = KT / p.box, head_row = kvh * a.num_pages * tpp;
    int s = 0;
    uint32_t phase = 1;
    for (int j = 0; j <= hi; ++j) {
      // lane i: the cache row where box i of the tile begins (boxes beyond the run's last key: any page of the sequence)
      const int key = j * KT + (lane < boxes ? lane : 0) * p.box, known = key < p_end ? key : p_end;
      const int row = head_row + pages[known / tpp] * tpp + key % tpp;
      mbar_wait(&tail->empty[s], phase);
      uint8_t* st = ring + s * 2 * F::kTileBytes;
      if (issuer) {
        mbar_expect_tx(&tail->k_full[s], uint32_t(F::kTileBytes));
        mbar_expect_tx(&tail->v_full[s], uint32_t(F::kTileBytes));
      }
      for (int kv = 0; kv < 2; ++kv)
        for (int b = 0; b < boxes; ++b) {
          const int from = __shfl_sync(0xffffffffu, row, b);
          if (issuer)
            for (int c = 0; c < CH; ++c)
              tma_load_2d(st + kv * F::kTileBytes + c * KT * 128 + b * p.box * 128, kv == 0 ? &tm_k : &tm_v, c * 64, from, kv == 0 ? &tail->k_full[s] : &tail->v_full[s], kEvictLast);
        }
      if (++s == F::kStages) s = 0, phase ^= 1;
    }
  } else if (warp == 1) {
    const bool issuer = elect_one();
    const uint32_t idesc_s = umma_idesc_bf16(128, KT), idesc_o = umma_idesc_bf16(128, D) | kIdescBMajorMN;
    const uint64_t dq = umma_desc_sw128(sq), dk = umma_desc_sw128(ring);
    const uint32_t ring_addr = smem_u32(ring);
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
    auto issue_o = [&](int t, int stage, bool start) {
      if (!issuer) return;
#pragma unroll
      for (int kk = 0; kk < KT / 16; ++kk)
        umma_bf16_ts(tmem + F::kOCol + t * D, tmem + F::kPCol + t * (KT / 2) + kk * 8,
                     umma_desc_sw128_mn(ring_addr + stage * 2 * F::kTileBytes + F::kTileBytes + kk * 2048, KT * 128), idesc_o, uint32_t(!start || kk != 0));
      umma_commit(&tail->o_done[t]);
    };
    mbar_wait(&tail->q_full, 0);
    int s = 0;
    uint32_t par = 0;
    for (int j = -1; j <= hi; ++j) {  // step j: the next tile's S, then this tile's P V
      const int s1 = j < 0 ? 0 : (s + 1 == F::kStages ? 0 : s + 1);
      const uint32_t par1 = j >= 0 && s1 == 0 ? par ^ 1 : par;
      if (j < hi) {
        mbar_wait(&tail->k_full[s1], par1);
#pragma unroll
        for (int t = 0; t < NQ; ++t)
          if (j + 1 <= last[t]) {
            if (j >= 0) mbar_wait(&tail->s_free[t], j & 1);  // the tile before is in registers
            tcgen05_fence_after();
            issue_s(t, s1);
          }
      }
      if (j < 0) continue;
      mbar_wait(&tail->v_full[s], par);
      const int beyond = p_end + 1 - j * KT;  // the tile's first key that the sequence does not have
      uint8_t* v = ring + s * 2 * F::kTileBytes + F::kTileBytes;
      if (beyond < KT) {                      // values of no key: 0 (their probabilities are 0, which a left-over NaN would not leave 0)
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
      for (int t = 0; t < NQ; ++t)
        if (j <= last[t]) {
          mbar_wait(&tail->p_ready[t], j & 1);
          tcgen05_fence_after();
          issue_o(t, s, j == 0);
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
    const int t = NQ == 2 ? (warp - 2) >> 2 : 0, quarter = warp & 3;
    const int row = r0 + 128 * t + quarter * 32 + lane, pos = p0 + 128 * t + quarter * 32 + lane;
    const int w_lo = p0 + 128 * t + quarter * 32;  // the warp's first position
    const uint32_t lanes = tmem + (uint32_t(quarter * 32) << 16), acc = lanes + F::kOCol + t * D, s_col = lanes + t * KT, p_col = lanes + F::kPCol + t * (KT / 2);
    const bool capped = a.softcap > 0.0f;
    const float cap_mul = capped ? a.scale * 2.8853900817779268f / a.softcap : 0.0f, slope = a.slopes ? a.slopes[head] : 0.0f;
    float m = a.sink ? a.sink[head] : -INFINITY;
    float l[4] = {a.sink ? 1.0f : 0.0f, 0.0f, 0.0f, 0.0f};  // the sums of the columns 8 n + 2 t and 8 n + 2 t + 1, t = 0 .. 3
    int la = -1;
#pragma unroll
    for (int i = 0; i < NQ; ++i)
      if (i == t) la = last[i];
    for (int j = 0; j <= la; ++j) {
      const int key0 = j * KT;
      mbar_wait(&tail->s_full[t], j & 1);
      tcgen05_fence_after();
      float x[KT];
      {
        uint32_t raw[KT / 32][32];
#pragma unroll
        for (int c = 0; c < KT / 32; ++c) tmem_ld_x32(s_col + c * 32, raw[c]);
        tmem_wait_ld();
        tcgen05_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(&tail->s_free[t]);
#pragma unroll
        for (int c = 0; c < KT; ++c) x[c] = __uint_as_float(raw[c / 32][c % 32]);
      }
      if (capped) {
#pragma unroll
        for (int c = 0; c < KT; ++c) x[c] = smax_softcap_scaled(x[c], cap_mul, a.softcap);
      } else {
#pragma unroll
        for (int c = 0; c < KT; ++c) x[c] = x[c] * a.scale;
      }
      if (a.slopes) {
#pragma unroll
        for (int c = 0; c < KT; ++c) x[c] -= slope * float(pos - (key0 + c));
      }
      if (key0 + KT - 1 > w_lo) {  // (uniform in the warp)
#pragma unroll
        for (int c = 0; c < KT; ++c)
          if (key0 + c > pos) x[c] = -INFINITY;
      }
      float mx0 = x[0], mx1 = x[1], mx2 = x[2], mx3 = x[3];
#pragma unroll
      for (int c = 4; c < KT; c += 4) {
        mx0 = fmaxf(mx0, x[c]);
        mx1 = fmaxf(mx1, x[c + 1]);
        mx2 = fmaxf(mx2, x[c + 2]);
        mx3 = fmaxf(mx3, x[c + 3]);
      }
      const float m_new = fmaxf(m, fmaxf(fmaxf(mx0, mx1), fmaxf(mx2, mx3)));
      const float base = m_new == -INFINITY ? 0.0f : m_new, fix = __expf(m - base);  // (exp(-inf) = 0 in the first tile)
      m = m_new;
      if (j > 0) {  // the tiles before are in the accumulator, and P's columns free
        mbar_wait(&tail->o_done[t], (j - 1) & 1);
        tcgen05_fence_after();
        if (__any_sync(0xffffffffu, fix != 1.0f)) {
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
      float sum[4] = {0.0f, 0.0f, 0.0f, 0.0f};
      uint32_t pk[KT / 2];
#pragma unroll
      for (int c = 0; c < KT; c += 2) {
        const float e0 = __expf(x[c] - base), e1 = __expf(x[c + 1] - base);
        sum[(c >> 1) & 3] += e0 + e1;
        pk[c / 2] = pack_bf16x2(e0, e1);
      }
#pragma unroll
      for (int q = 0; q < 4; ++q) l[q] = l[q] * fix + sum[q];
      if constexpr (KT == 64) {
        tmem_st_x32(p_col, pk);
      } else {
        tmem_st_x16(p_col, pk);
      }
      tmem_wait_st();
      tcgen05_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(&tail->p_ready[t]);
    }
    if (la >= 0) {
      mbar_wait(&tail->o_done[t], la & 1);
      tcgen05_fence_after();
      uint32_t noted = 0;
      if (la >= masked) {
        mbar_wait(&tail->noted_all[t], 0);
#pragma unroll
        for (int w = 0; w < F::kNoteWords; ++w) noted |= tail->noted[w];
      }
      const bool valid = row < r_end;
      const float total = (l[0] + l[1]) + (l[2] + l[3]), f = a.out_scale / total * (valid ? smax_gate(a, row, head) : 1.0f);
      bf16* out = a.out + size_t(valid ? row : r0) * a.ld_out + head * D;
#pragma unroll 1
      for (int c = 0; c < D; c += 32) {
        uint32_t o[32];
        tmem_ld_x32(acc + c, o);
        tmem_wait_ld();
        if (!valid) continue;
        if (noted != 0)
          flash_add_noted<F::kNoteWords>(o, tail->noted, masked * KT, pos, c,
                                         [&](int key) { return a.v_pages + (size_t(kvh) * a.num_pages * tpp + size_t(pages[key / tpp]) * tpp + key % tpp) * D; });
#pragma unroll
        for (int e = 0; e < 32; e += 2) {
          float v0 = __uint_as_float(o[e]), v1 = __uint_as_float(o[e + 1]);
          if (a.value_gate) {
            v0 *= smax_value_gate(a, row, head, c + e);
            v1 *= smax_value_gate(a, row, head, c + e + 1);
          }
          *reinterpret_cast<uint32_t*>(out + c + e) = smax_pack_bf16(v0 * f, v1 * f);
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
