// GQA decode attention for WIDE heads (head_dim 256: gemma3-1b/4b/12b), same contract, work list and cross-item merge as
// decode_attn_kernel (attention.cuh), different arithmetic layout.
//
// decode_attn_kernel keeps the group's query heads in the 16-row dimension of the MMA and D/2 accumulator registers per
// thread: 128 at D = 256, which does not fit beside the score and query fragments.  Here the products are TRANSPOSED, as in
// the persistent kernel (step_persistent.cuh): S^T = K Q^T and O^T = V^T P^T, so the 16-row dimension carries KV rows /
// head dims and the 8-column dimension the (up to 8) query heads of the group: D/4 accumulator registers, D/8 for the
// queries, no padding of the heads to 16.  A K or V tile of 64 rows is 32 KB at D = 256, so a CTA holds THREE warps' tiles
// (192 KB): kWideWarps.
#pragma once

#include "attention.cuh"

namespace mtx {

constexpr int kWideWarps = 3;
constexpr int kWideThreads = kWideWarps * 32;

__device__ __forceinline__ uint32_t aw_movmatrix_trans(uint32_t a) {
  uint32_t d;
  asm volatile("movmatrix.sync.aligned.m8n8.trans.b16 %0, %1;" : "=r"(d) : "r"(a));
  return d;
}
__device__ __forceinline__ void aw_bar_sync() { asm volatile("bar.sync 1, %0;" ::"n"(kWideThreads) : "memory"); }

__host__ inline size_t attn_wide_smem_bytes(int D) {
  return 1024 + size_t(kWideWarps) * 2 * (64 * D * 2) + size_t(kWideWarps) * 8 * D * 4 + 2 * kWideWarps * 8 + 2 * kWideWarps * 16 * 4 + 32;
}

template <int D>
__global__ void __launch_bounds__(kWideThreads)
decode_attn_wide_kernel(const __grid_constant__ CUtensorMap tm_k, const __grid_constant__ CUtensorMap tm_v, const AttnParams p) {
  constexpr int kSub = D / 64;
  constexpr int kTileBytes = 64 * D * 2;
  constexpr float kLog2e = 1.4426950408889634f;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = smem_raw + ((1024u - (smem_u32(smem_raw) & 1023u)) & 1023u);
  const int G = p.hq / p.hkv;  // <= 8 (checked by the host)
  float* sm_o_all = reinterpret_cast<float*>(smem + kWideWarps * 2 * kTileBytes);  // [warp][8][D]
  uint64_t* bars = reinterpret_cast<uint64_t*>(sm_o_all + kWideWarps * 8 * D);
  float* sm_m = reinterpret_cast<float*>(bars + 2 * kWideWarps);  // [warp][16]
  float* sm_l = sm_m + kWideWarps * 16;
  volatile int* s_last_p = reinterpret_cast<volatile int*>(sm_l + kWideWarps * 16);
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  griddep_launch_dependents();
  if (lane == 0) {
    mbar_init(bars + 2 * warp, 1);
    mbar_init(bars + 2 * warp + 1, 1);
    fence_barrier_init();
  }
  if (tid == 0) {
    tma_prefetch_desc(&tm_k);
    tma_prefetch_desc(&tm_v);
  }
  __syncthreads();
  griddep_wait();

  const int gid = lane >> 2, tid4 = lane & 3;
  const int a_row = (lane & 7) + 8 * ((lane >> 3) & 1), a_chunk = lane >> 4;  // ldmatrix addressing, K tile as A
  const int v_row = (lane & 7) + 8 * (lane >> 4), v_chunk = (lane >> 3) & 1;   // ldmatrix.trans addressing, V^T as A
  const int R = p.ring_size > 0 ? p.ring_size : p.T - p.P;
  const int TPI = p.tiles_per_item;
  uint8_t* k_tile = smem + warp * 2 * kTileBytes;
  uint8_t* v_tile = k_tile + kTileBytes;
  float* sm_o = sm_o_all + warp * 8 * D;
  uint64_t* bar_k = bars + 2 * warp;
  uint64_t* bar_v = bar_k + 1;
  const uint32_t kb = smem_u32(k_tile), vb = smem_u32(v_tile);
  uint32_t phase = 0;
  const int n_items = *p.work_count * p.hkv;

  for (int turn = 0; turn * int(gridDim.x) < n_items; ++turn) {
    const int item = attn_item(turn, blockIdx.x, gridDim.x);
    if (item >= n_items) continue;
    const int packed = p.work_items[item / p.hkv];
    const int h = item % p.hkv;
    const int r = packed >> 16, chunk = packed & 0xffff;
    const int len0 = p.len0[r], rf = p.ring_first[r], rl = p.ring_len[r];
    const int skip0 = p.skip0 + (p.skip0_rows != nullptr ? p.skip0_rows[r] : 0);
    const int nt = attn_num_tiles(len0, rf, rl, R);
    const int n_chunks = (nt + TPI - 1) / TPI;
    const int t_begin = chunk * TPI, t_end = min(nt, t_begin + TPI);
    const int plane_row = ((p.plane_base + p.plane[r]) * p.hkv + h) * p.T;

    int t = t_begin + warp;
    TileLoc loc = attn_tile(t < t_end ? t : nt, len0, rf, rl, p.P, R, skip0, p.ring_off);
    if (t < t_end && lane == 0) {
      mbar_expect_tx(bar_k, kTileBytes);
#pragma unroll
      for (int s = 0; s < kSub; ++s) tma_load_2d(k_tile + s * 8192, &tm_k, s * 64, plane_row + loc.p0, bar_k, kEvictFirst);
      mbar_expect_tx(bar_v, kTileBytes);
#pragma unroll
      for (int s = 0; s < kSub; ++s) tma_load_2d(v_tile + s * 8192, &tm_v, s * 64, plane_row + loc.p0, bar_v, kEvictFirst);
    }
    // Q^T fragments (B operand): thread (gid, tid4) holds head gid, dims 16 kk + 2 tid4 (+8)
    uint32_t qb[D / 16][2];
    {
      const bf16* qrow = p.q + (long long)r * p.hq * D + (long long)h * G * D + gid * D + tid4 * 2;
#pragma unroll
      for (int kk = 0; kk < D / 16; ++kk) {
        qb[kk][0] = gid < G ? *reinterpret_cast<const uint32_t*>(qrow + kk * 16) : 0u;
        qb[kk][1] = gid < G ? *reinterpret_cast<const uint32_t*>(qrow + kk * 16 + 8) : 0u;
      }
    }
    // thread (gid, tid4) owns heads h0 = 2 tid4, h1 = h0 + 1:
    //   s[mb][0..3] = S^T[kv = 16 mb + gid (+8 for 2,3)][h0, h1];  o[db][0..3] = O^T[d = 16 db + gid (+8 for 2,3)][h0, h1]
    float m0 = -INFINITY, m1 = -INFINITY, l0 = 0.0f, l1 = 0.0f;
    float o[D / 16][4];
#pragma unroll
    for (int db = 0; db < D / 16; ++db) o[db][0] = o[db][1] = o[db][2] = o[db][3] = 0.0f;

    for (; t < t_end; t += kWideWarps) {
      const int cnt = loc.cnt;
      const int tn = t + kWideWarps;
      const TileLoc nloc = attn_tile(tn < t_end ? tn : nt, len0, rf, rl, p.P, R, skip0, p.ring_off);
      float s[4][4];
#pragma unroll
      for (int mb = 0; mb < 4; ++mb) s[mb][0] = s[mb][1] = s[mb][2] = s[mb][3] = 0.0f;
      mbar_wait(bar_k, phase);
#pragma unroll
      for (int kk = 0; kk < D / 16; ++kk) {
#pragma unroll
        for (int mb = 0; mb < 4; ++mb) {
          const int row = 16 * mb + a_row;
          const int c = 2 * kk + a_chunk;
          const uint32_t addr = kb + (c >> 3) * 8192 + row * 128 + (((c & 7) ^ (row & 7)) << 4);
          uint32_t a[4];
          ldmatrix_x4(addr, a[0], a[1], a[2], a[3]);
          mma_m16n8k16_bf16(s[mb], a, qb[kk][0], qb[kk][1]);
        }
      }
      fence_proxy_async();
      __syncwarp();
      if (tn < t_end && lane == 0) {
        mbar_expect_tx(bar_k, kTileBytes);
#pragma unroll
        for (int ss = 0; ss < kSub; ++ss) tma_load_2d(k_tile + ss * 8192, &tm_k, ss * 64, plane_row + nloc.p0, bar_k, kEvictFirst);
      }
      // ---- mask + online softmax: a head's scores live in the 8 threads of equal tid4 ----
      float tm0 = -INFINITY, tm1 = -INFINITY;
#pragma unroll
      for (int mb = 0; mb < 4; ++mb) {
#pragma unroll
        for (int q = 0; q < 4; ++q) {
          float x = s[mb][q];
          if (p.softcap != 0.0f) x = tanhf(x / p.softcap) * p.softcap;
          s[mb][q] = 16 * mb + gid + (q >> 1) * 8 < cnt ? x : -INFINITY;
        }
        tm0 = fmaxf(tm0, fmaxf(s[mb][0], s[mb][2]));
        tm1 = fmaxf(tm1, fmaxf(s[mb][1], s[mb][3]));
      }
#pragma unroll
      for (int sh = 4; sh < 32; sh <<= 1) {
        tm0 = fmaxf(tm0, __shfl_xor_sync(0xffffffffu, tm0, sh));
        tm1 = fmaxf(tm1, __shfl_xor_sync(0xffffffffu, tm1, sh));
      }
      const float nm0 = fmaxf(m0, tm0), nm1 = fmaxf(m1, tm1);  // (a tile holds at least one valid row: finite)
      const float a0 = exp2f((m0 - nm0) * kLog2e), a1 = exp2f((m1 - nm1) * kLog2e);  // exp2(-inf) = 0 on the first tile
      m0 = nm0;
      m1 = nm1;
      l0 *= a0;
      l1 *= a1;
      uint32_t pb[4][2];  // P^T as the B operand of O^T += V^T P^T, one k-step per 16 KV rows
#pragma unroll
      for (int mb = 0; mb < 4; ++mb) {
        const float p0 = exp2f((s[mb][0] - m0) * kLog2e), p1 = exp2f((s[mb][1] - m1) * kLog2e);
        const float p2 = exp2f((s[mb][2] - m0) * kLog2e), p3 = exp2f((s[mb][3] - m1) * kLog2e);
        l0 += p0 + p2;
        l1 += p1 + p3;
        // probabilities are cast to the value dtype before the PV product (kernels/ragged_attention.py:156)
        pb[mb][0] = aw_movmatrix_trans(pack_bf16x2(p0, p1));
        pb[mb][1] = aw_movmatrix_trans(pack_bf16x2(p2, p3));
      }
#pragma unroll
      for (int db = 0; db < D / 16; ++db) {
        o[db][0] *= a0;
        o[db][1] *= a1;
        o[db][2] *= a0;
        o[db][3] *= a1;
      }
      mbar_wait(bar_v, phase);
      if (cnt < 64) {  // rows past the valid count may hold anything: zero them (0 * NaN != 0)
        const int nvec = (64 - cnt) * 8;
        for (int i = lane; i < nvec * kSub; i += 32) {
          const int sub = i / nvec, w = i % nvec;
          *reinterpret_cast<uint4*>(v_tile + sub * 8192 + (cnt + w / 8) * 128 + (w & 7) * 16) = make_uint4(0, 0, 0, 0);
        }
        __syncwarp();
      }
#pragma unroll
      for (int db = 0; db < D / 16; ++db) {
#pragma unroll
        for (int mb = 0; mb < 4; ++mb) {
          const int row = 16 * mb + v_row;
          const int c = 2 * db + v_chunk;
          const uint32_t addr = vb + (c >> 3) * 8192 + row * 128 + (((c & 7) ^ (row & 7)) << 4);
          uint32_t a[4];
          ldmatrix_x4_trans(addr, a[0], a[1], a[2], a[3]);
          mma_m16n8k16_bf16(o[db], a, pb[mb][0], pb[mb][1]);
        }
      }
      fence_proxy_async();
      __syncwarp();
      if (tn < t_end && lane == 0) {
        mbar_expect_tx(bar_v, kTileBytes);
#pragma unroll
        for (int ss = 0; ss < kSub; ++ss) tma_load_2d(v_tile + ss * 8192, &tm_v, ss * 64, plane_row + nloc.p0, bar_v, kEvictFirst);
      }
      phase ^= 1;
      loc = nloc;
    }
#pragma unroll
    for (int sh = 4; sh < 32; sh <<= 1) {
      l0 += __shfl_xor_sync(0xffffffffu, l0, sh);
      l1 += __shfl_xor_sync(0xffffffffu, l1, sh);
    }

    // ---- merge the warps of the item in shared memory: sm_o [head][D] ----
    const int h0 = tid4 * 2;
    if (m0 > -INFINITY) {
#pragma unroll
      for (int db = 0; db < D / 16; ++db) {
        const int d = 16 * db + gid;
        if (h0 < G) {
          sm_o[h0 * D + d] = o[db][0];
          sm_o[h0 * D + d + 8] = o[db][2];
        }
        if (h0 + 1 < G) {
          sm_o[(h0 + 1) * D + d] = o[db][1];
          sm_o[(h0 + 1) * D + d + 8] = o[db][3];
        }
      }
    }
    if (gid == 0) {
      sm_m[warp * 16 + h0] = m0;
      sm_m[warp * 16 + h0 + 1] = m1;
      sm_l[warp * 16 + h0] = l0;
      sm_l[warp * 16 + h0 + 1] = l1;
    }
    aw_bar_sync();

    const long long out_base = (long long)r * p.hq * D + (long long)h * G * D;
    const long long part_base = ((long long)(r * p.hkv + h) * p.max_chunks + chunk) * G;
    for (int e = tid; e < G * D; e += kWideThreads) {
      const int g = e / D, d = e - g * D;
      float M = -INFINITY;
#pragma unroll
      for (int w = 0; w < kWideWarps; ++w) M = fmaxf(M, sm_m[w * 16 + g]);
      float L = 0.0f, O = 0.0f;
#pragma unroll
      for (int w = 0; w < kWideWarps; ++w) {
        const float mw = sm_m[w * 16 + g];
        if (mw > -INFINITY) {
          const float sc = exp2f((mw - M) * kLog2e);
          L += sm_l[w * 16 + g] * sc;
          O += sm_o_all[(w * 8 + g) * D + d] * sc;
        }
      }
      if (n_chunks == 1) {
        p.out[out_base + e] = __float2bfloat16_rn(O / L);
      } else {
        __stcg(p.part_o + (part_base + g) * D + d, O);
        if (d == 0) {
          __stcg(p.part_ml + (part_base + g) * 2, M);
          __stcg(p.part_ml + (part_base + g) * 2 + 1, L);
        }
      }
    }
    if (n_chunks > 1) {
      __threadfence();
      aw_bar_sync();
      if (tid == 0) {
        const int old = atomicAdd(p.tickets + r * p.hkv + h, 1);
        const int last = old == n_chunks - 1;
        if (last) p.tickets[r * p.hkv + h] = 0;
        *s_last_p = last;
      }
      aw_bar_sync();
      if (*s_last_p) {
        __threadfence();
        const long long pbase = (long long)(r * p.hkv + h) * p.max_chunks * G;
        for (int e = tid; e < G * D; e += kWideThreads) {
          const int g = e / D, d = e - g * D;
          float M = -INFINITY;
          for (int c = 0; c < n_chunks; ++c) M = fmaxf(M, __ldcg(p.part_ml + (pbase + c * G + g) * 2));
          float L = 0.0f, O = 0.0f;
          for (int c = 0; c < n_chunks; ++c) {
            const float sc = exp2f((__ldcg(p.part_ml + (pbase + c * G + g) * 2) - M) * kLog2e);
            L += __ldcg(p.part_ml + (pbase + c * G + g) * 2 + 1) * sc;
            O += __ldcg(p.part_o + (pbase + c * G + g) * D + d) * sc;
          }
          p.out[out_base + e] = __float2bfloat16_rn(O / L);
        }
      }
    }
    aw_bar_sync();  // the merge buffer is rewritten by the next item
  }
}

// The same arithmetic for the positions of a prompt (one sequence, one plane; query i sees the keys up to itself, of the last `window` ones where
// there is a window), several positions per work item: the 8-column side of a warp's MMAs carries NP = 8 / G positions 64 apart, and kPromptGroups
// such warps read one key tile out of shared memory, so that an item is 64 kPromptGroups NP positions of one residue modulo 64, whose key tiles are the
// same rows -- tiles begin at the position's first key, and the windows of positions 64 apart begin 64 apart.  A tile that a column's
// position does not see leaves the column alone (probabilities 0, factor 1; a warp none of whose columns see it passes it by), and a column's partial
// sums over every third tile are merged in the order in which its own tiles went to them, so that a position gets the bits that
// decode_attn_wide_kernel gives it with one work item per (position, kv head).
// Positions before and behind the window's length begin their tiles at other offsets: an item that holds both is walked in two parts.  An item
// with a result that is no finite number is walked again position by position: 0 times an infinite or NaN value is NaN, and the value may be one that
// only another position of the item sees.
//
// Warp w = (class w / kPromptGroups, group w % kPromptGroups): class c takes the tiles c, c + 3, ..; its tile buffers are filled again by the last of
// its warps to be done with them.
//
// Bound: what an SM takes in from the L2 (64 KB per tile at about 64 B per ns), and the wait for it where the tiles are not yet used up.  3001 positions, 8 heads
// over 4 kv heads, the mean of five layers with a window of 1024 and a global one: 492 us with one group of columns per tile, 336 us with four (the last
// 185 positions a step of their own in both), 289 us with all of them in one launch (a windowed layer 280, the global one 351).
struct PromptWideParams {
  const bf16* q;   // [rows, hq * D]
  bf16* out;       // [rows, hq * D]
  int rows;        // positions
  int start_pos;   // position of row 0
  int hq, hkv, T;
  int plane_row0;  // cache row of (layer, plane, kv head 0, position 0); kv head h adds h * T
  float softcap;
  int window;      // 0: none
};

constexpr int kPromptGroups = 4;  // groups of eight columns that share a key tile
constexpr int kPromptWarps = kWideWarps * kPromptGroups;
constexpr int kPromptThreads = kPromptWarps * 32;

struct PromptWideTail {
  uint64_t full_k[kWideWarps], full_v[kWideWarps];
  int done_k[kWideWarps], done_v[kWideWarps];  // warps of the class that are done with its tile
  float m[kPromptWarps][8], l[kPromptWarps][8];
};
// (the partial sums, [warp][8][D] fp32, take the place of the tiles at an item's end)
__host__ __device__ inline size_t prompt_wide_smem_bytes(int D) { return 1024 + size_t(kWideWarps) * 2 * (64 * D * 2) + sizeof(PromptWideTail) + 16; }

template <int D>
__global__ void __launch_bounds__(kPromptThreads, 1)
prompt_attn_wide_kernel(const __grid_constant__ CUtensorMap tm_k, const __grid_constant__ CUtensorMap tm_v, const PromptWideParams p) {
  constexpr int kSub = D / 64;
  constexpr int kTileBytes = 64 * D * 2;
  constexpr float kLog2e = 1.4426950408889634f;
  static_assert(kPromptWarps * 8 * D * 4 <= kWideWarps * 2 * kTileBytes, "the partial sums fit in the tiles' place");
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = smem_raw + ((1024u - (smem_u32(smem_raw) & 1023u)) & 1023u);
  const int G = p.hq / p.hkv;  // <= 8 (checked by the host)
  const int NP = 8 / G;
  float* sm_o_all = reinterpret_cast<float*>(smem);  // [warp][8][D]
  PromptWideTail* tail = reinterpret_cast<PromptWideTail*>(smem + kWideWarps * 2 * kTileBytes);
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int cls = warp / kPromptGroups, grp = warp % kPromptGroups;
  griddep_launch_dependents();
  if (tid < kWideWarps) {
    mbar_init(&tail->full_k[tid], 1);
    mbar_init(&tail->full_v[tid], 1);
    tail->done_k[tid] = tail->done_v[tid] = 0;
    fence_barrier_init();
  }
  if (tid == 0) {
    tma_prefetch_desc(&tm_k);
    tma_prefetch_desc(&tm_v);
  }
  __syncthreads();
  griddep_wait();

  const int gid = lane >> 2, tid4 = lane & 3;
  const int a_row = (lane & 7) + 8 * ((lane >> 3) & 1), a_chunk = lane >> 4;  // ldmatrix addressing, K tile as A
  const int v_row = (lane & 7) + 8 * (lane >> 4), v_chunk = (lane >> 3) & 1;   // ldmatrix.trans addressing, V^T as A
  uint8_t* k_tile = smem + cls * 2 * kTileBytes;
  uint8_t* v_tile = k_tile + kTileBytes;
  float* sm_o = sm_o_all + warp * 8 * D;
  const uint32_t kb = smem_u32(k_tile), vb = smem_u32(v_tile);
  uint32_t phase = 0;
  const int n_blocks = (p.rows + 64 * kPromptGroups * NP - 1) / (64 * kPromptGroups * NP);
  const int n_items = n_blocks * 64 * p.hkv;
  auto first_key = [&](int row) { return p.window > 0 && p.start_pos + row + 1 > p.window ? p.start_pos + row + 1 - p.window : 0; };
  auto load_tile = [&](uint8_t* dst, const CUtensorMap* tm, uint64_t* bar, int row) {
    mbar_expect_tx(bar, kTileBytes);
#pragma unroll
    for (int s = 0; s < kSub; ++s) tma_load_2d(dst + s * 8192, tm, s * 64, row, bar, kEvictLast);
  };
  // this warp is done with its class's tile: true for one thread of the class's last warp, who may have it filled again
  auto last_done = [&](int* done) {
    fence_proxy_async();
    __syncwarp();
    if (lane != 0) return false;
    __threadfence_block();
    if (atomicAdd_block(done, 1) != kPromptGroups - 1) return false;
    __threadfence_block();
    *done = 0;  // (nobody counts before the next tile is there)
    return true;
  };

  for (int item = blockIdx.x; item < n_items; item += gridDim.x) {
    const int h = item % p.hkv, at = item / p.hkv;
    const int row0 = (n_blocks - 1 - at / 64) * 64 * kPromptGroups * NP + at % 64;  // (the last positions, with the most keys, first)
    if (row0 >= p.rows) continue;
    const int np = min(kPromptGroups * NP, (p.rows - row0 + 63) / 64);  // positions: rows row0 + 64 i
    const int plane_row = p.plane_row0 + h * p.T;
    int alone = 0;  // positions before this one are walked one by one
    for (int i_lo = 0; i_lo < np;) {
      int i_hi = i_lo + 1;
      if (i_lo >= alone)
        while (i_hi < np && ((first_key(row0 + 64 * i_hi) - first_key(row0 + 64 * i_lo)) & 63) == 0) ++i_hi;
      const int key0 = first_key(row0 + 64 * i_lo);                 // tile u holds the keys key0 + 64 u ..
      const int last_key = p.start_pos + row0 + 64 * (i_hi - 1);    // of the last position
      const int nt = (last_key - key0) / 64 + 1;
      // the positions of a group's columns (none: false), their first tile and last key
      auto column = [&](int g, int c, int* first, int* last) {
        const int i = g * NP + c / G;
        const bool in = c < NP * G && i >= i_lo && i < i_hi;
        *first = in ? (first_key(row0 + 64 * i) - key0) / 64 : 1 << 30;
        *last = in ? p.start_pos + row0 + 64 * i : -1;
        return in;
      };
      if (grp == 0 && cls < nt && lane == 0) {
        load_tile(k_tile, &tm_k, &tail->full_k[cls], plane_row + key0 + 64 * cls);
        load_tile(v_tile, &tm_v, &tail->full_v[cls], plane_row + key0 + 64 * cls);
      }
      // Q^T fragments (B operand): thread (gid, tid4) holds column gid, dims 16 kk + 2 tid4 (+8)
      uint32_t qb[D / 16][2];
      {
        int f, l;
        const bool in = column(grp, gid, &f, &l);
        const bf16* qrow = p.q + (long long)(in ? row0 + 64 * (grp * NP + gid / G) : row0) * p.hq * D + (long long)(h * G + gid % G) * D + tid4 * 2;
#pragma unroll
        for (int kk = 0; kk < D / 16; ++kk) {
          qb[kk][0] = in ? *reinterpret_cast<const uint32_t*>(qrow + kk * 16) : 0u;
          qb[kk][1] = in ? *reinterpret_cast<const uint32_t*>(qrow + kk * 16 + 8) : 0u;
        }
      }
      // thread (gid, tid4) owns columns c0 = 2 tid4, c1 = c0 + 1:
      //   s[mb][0..3] = S^T[kv = 16 mb + gid (+8 for 2,3)][c0, c1];  o[db][0..3] = O^T[d = 16 db + gid (+8 for 2,3)][c0, c1]
      int f0, f1, e0, e1;
      column(grp, 2 * tid4, &f0, &e0);
      column(grp, 2 * tid4 + 1, &f1, &e1);
      // the group's tiles: from its first position's first to its last position's last
      int t_first, t_last;
      {
        const int a = max(i_lo, grp * NP), b = min(i_hi, (grp + 1) * NP) - 1;
        t_first = a <= b ? (first_key(row0 + 64 * a) - key0) / 64 : 1 << 30;
        t_last = a <= b ? (p.start_pos + row0 + 64 * b - key0) / 64 : -1;
      }
      float m0 = -INFINITY, m1 = -INFINITY, l0 = 0.0f, l1 = 0.0f;
      float o[D / 16][4];
#pragma unroll
      for (int db = 0; db < D / 16; ++db) o[db][0] = o[db][1] = o[db][2] = o[db][3] = 0.0f;

      for (int t = cls; t < nt; t += kWideWarps) {
        const int tile_key = key0 + 64 * t, cnt = last_key + 1 - tile_key, tn = t + kWideWarps;
        const bool sees = t >= t_first && t <= t_last;
        uint32_t pb[4][2];  // P^T as the B operand of O^T += V^T P^T, one k-step per 16 KV rows
        float s[4][4];
        mbar_wait(&tail->full_k[cls], phase);
        if (sees) {
#pragma unroll
          for (int mb = 0; mb < 4; ++mb) s[mb][0] = s[mb][1] = s[mb][2] = s[mb][3] = 0.0f;
#pragma unroll
          for (int kk = 0; kk < D / 16; ++kk) {
#pragma unroll
            for (int mb = 0; mb < 4; ++mb) {
              const int row = 16 * mb + a_row;
              const int c = 2 * kk + a_chunk;
              const uint32_t addr = kb + (c >> 3) * 8192 + row * 128 + (((c & 7) ^ (row & 7)) << 4);
              uint32_t a[4];
              ldmatrix_x4(addr, a[0], a[1], a[2], a[3]);
              mma_m16n8k16_bf16(s[mb], a, qb[kk][0], qb[kk][1]);
            }
          }
        }
        if (last_done(&tail->done_k[cls]) && tn < nt) load_tile(k_tile, &tm_k, &tail->full_k[cls], plane_row + key0 + 64 * tn);
        if (sees) {
          // ---- mask + online softmax: a column's scores live in the 8 threads of equal tid4 ----
          const int seen0 = t >= f0 ? e0 + 1 - tile_key : 0, seen1 = t >= f1 ? e1 + 1 - tile_key : 0;  // keys of the tile that the column sees
          float tm0 = -INFINITY, tm1 = -INFINITY;
#pragma unroll
          for (int mb = 0; mb < 4; ++mb) {
#pragma unroll
            for (int q = 0; q < 4; ++q) {
              float x = s[mb][q];
              if (p.softcap != 0.0f) x = tanhf(x / p.softcap) * p.softcap;
              s[mb][q] = 16 * mb + gid + (q >> 1) * 8 < ((q & 1) ? seen1 : seen0) ? x : -INFINITY;
            }
            tm0 = fmaxf(tm0, fmaxf(s[mb][0], s[mb][2]));
            tm1 = fmaxf(tm1, fmaxf(s[mb][1], s[mb][3]));
          }
#pragma unroll
          for (int sh = 4; sh < 32; sh <<= 1) {
            tm0 = fmaxf(tm0, __shfl_xor_sync(0xffffffffu, tm0, sh));
            tm1 = fmaxf(tm1, __shfl_xor_sync(0xffffffffu, tm1, sh));
          }
          const float nm0 = fmaxf(m0, tm0), nm1 = fmaxf(m1, tm1);
          // (-inf: a column that has seen no key yet; its scores are all masked and the factor multiplies zeros)
          const float x0 = nm0 == -INFINITY ? 0.0f : nm0, x1 = nm1 == -INFINITY ? 0.0f : nm1;
          const float a0 = exp2f((m0 - x0) * kLog2e), a1 = exp2f((m1 - x1) * kLog2e);  // exp2(-inf) = 0 on the first tile
          m0 = nm0;
          m1 = nm1;
          l0 *= a0;
          l1 *= a1;
#pragma unroll
          for (int mb = 0; mb < 4; ++mb) {
            const float p0 = exp2f((s[mb][0] - x0) * kLog2e), p1 = exp2f((s[mb][1] - x1) * kLog2e);
            const float p2 = exp2f((s[mb][2] - x0) * kLog2e), p3 = exp2f((s[mb][3] - x1) * kLog2e);
            l0 += p0 + p2;
            l1 += p1 + p3;
            pb[mb][0] = aw_movmatrix_trans(pack_bf16x2(p0, p1));
            pb[mb][1] = aw_movmatrix_trans(pack_bf16x2(p2, p3));
          }
#pragma unroll
          for (int db = 0; db < D / 16; ++db) {
            o[db][0] *= a0;
            o[db][1] *= a1;
            o[db][2] *= a0;
            o[db][3] *= a1;
          }
        }
        mbar_wait(&tail->full_v[cls], phase);
        if (cnt < 64) {  // rows past the last position may hold anything: the class's warps zero them (0 * NaN != 0)
          const int nvec = (64 - cnt) * 8;
          for (int i = grp * 32 + lane; i < nvec * kSub; i += kPromptGroups * 32) {
            const int sub = i / nvec, w = i % nvec;
            *reinterpret_cast<uint4*>(v_tile + sub * 8192 + (cnt + w / 8) * 128 + (w & 7) * 16) = make_uint4(0, 0, 0, 0);
          }
          asm volatile("bar.sync %0, %1;" ::"r"(1 + cls), "n"(kPromptGroups * 32) : "memory");
        }
        if (sees) {
#pragma unroll
          for (int db = 0; db < D / 16; ++db) {
#pragma unroll
            for (int mb = 0; mb < 4; ++mb) {
              const int row = 16 * mb + v_row;
              const int c = 2 * db + v_chunk;
              const uint32_t addr = vb + (c >> 3) * 8192 + row * 128 + (((c & 7) ^ (row & 7)) << 4);
              uint32_t a[4];
              ldmatrix_x4_trans(addr, a[0], a[1], a[2], a[3]);
              mma_m16n8k16_bf16(o[db], a, pb[mb][0], pb[mb][1]);
            }
          }
        }
        if (last_done(&tail->done_v[cls]) && tn < nt) load_tile(v_tile, &tm_v, &tail->full_v[cls], plane_row + key0 + 64 * tn);
        phase ^= 1;
      }
#pragma unroll
      for (int sh = 4; sh < 32; sh <<= 1) {
        l0 += __shfl_xor_sync(0xffffffffu, l0, sh);
        l1 += __shfl_xor_sync(0xffffffffu, l1, sh);
      }

      // ---- merge the classes in shared memory: sm_o [column][D] in the place of the tiles ----
      __syncthreads();
      const int c0 = tid4 * 2;
#pragma unroll
      for (int db = 0; db < D / 16; ++db) {
        const int d = 16 * db + gid;
        if (m0 > -INFINITY) {
          sm_o[c0 * D + d] = o[db][0];
          sm_o[c0 * D + d + 8] = o[db][2];
        }
        if (m1 > -INFINITY) {
          sm_o[(c0 + 1) * D + d] = o[db][1];
          sm_o[(c0 + 1) * D + d + 8] = o[db][3];
        }
      }
      if (gid == 0) {
        tail->m[warp][c0] = m0;
        tail->m[warp][c0 + 1] = m1;
        tail->l[warp][c0] = l0;
        tail->l[warp][c0 + 1] = l1;
      }
      __syncthreads();
      bool finite = true;
      for (int e = tid; e < kPromptGroups * 8 * D; e += kPromptThreads) {
        const int g = e / (8 * D), c = e / D % 8, d = e % D;
        int first, last;
        if (!column(g, c, &first, &last)) continue;
        float M = -INFINITY;
#pragma unroll
        for (int w = 0; w < kWideWarps; ++w) M = fmaxf(M, tail->m[w * kPromptGroups + g][c]);
        float L = 0.0f, O = 0.0f;
#pragma unroll
        for (int n = 0; n < kWideWarps; ++n) {
          const int w = (n + first) % kWideWarps * kPromptGroups + g;  // the class of the position's n-th tile
          const float mw = tail->m[w][c];
          if (mw > -INFINITY) {
            const float sc = exp2f((mw - M) * kLog2e);
            L += tail->l[w][c] * sc;
            O += sm_o_all[(w * 8 + c) * D + d] * sc;
          }
        }
        const float y = O / L;
        finite &= fabsf(y) < INFINITY;
        p.out[(long long)(row0 + 64 * (g * NP + c / G)) * p.hq * D + (long long)(h * G + c % G) * D + d] = __float2bfloat16_rn(y);
      }
      fence_proxy_async();  // (the tiles' next contents come by TMA)
      const bool all_finite = __syncthreads_and(finite);
      if (i_hi - i_lo > 1 && !all_finite) alone = i_hi;
      else i_lo = i_hi;
    }
  }
}

}  // namespace mtx
