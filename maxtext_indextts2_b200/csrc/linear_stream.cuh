// linear_any.cuh's bf16 product for few rows (decode steps of small batches, experts with few tokens, a prompt's last row): the same argument block,
// modes and epilogues, and the same bits (every sum adds 16 products at a time in order of k), for k a multiple of 64 and 16-byte aligned rows.
//
// Bound: streaming the weights.  linear_mma_kernel holds one 64 x 64 tile of them in registers ahead of its use, 16 KB per SM in flight of the about 70
// that DRAM's latency asks for.  Here a CTA has 32 rows x BN columns and a ring of eight cp.async stages of 64 k (BN = 64: 56 KB of weights in
// flight per CTA and two CTAs per SM; BN = 32 for matrices that give fewer 64-column tiles than there are SMs).  Weights that do not depend
// on the kernel before are asked for before it has ended.
#pragma once

#include "linear_any.cuh"

namespace mtx {

constexpr int kLsThreads = 128, kLsBM = 32, kLsBK = 64, kLsPitch = kLsBK + 8, kLsStages = 8;
template <int BN>
constexpr size_t ls_smem_bytes() { return size_t(kLsStages) * (kLsBM + BN) * kLsPitch * sizeof(bf16); }

__device__ __forceinline__ void ls_cp_async_16(void* dst_smem, const void* src, bool valid) {
  const unsigned d = static_cast<unsigned>(__cvta_generic_to_shared(dst_smem));
  const int n = valid ? 16 : 0;  // (0: the 16 bytes are zero-filled, nothing is read)
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(d), "l"(src), "r"(n) : "memory");
}

template <int EPI, int BN>
__global__ void __launch_bounds__(kLsThreads) linear_stream_kernel(const LinArgs<bf16> p_in) {
  extern __shared__ __align__(16) unsigned char ls_raw[];
  bf16* const ring = reinterpret_cast<bf16*>(ls_raw);  // stage s: A [32][pitch], then W [BN][pitch]
  constexpr int STAGE = (kLsBM + BN) * kLsPitch, AC = kLsBM * 8 / kLsThreads, WC = BN * 8 / kLsThreads, NF = BN / 32;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, g = lane >> 2, t = lane & 3;
  griddep_launch_dependents();
  LinArgs<bf16> p = p_in;
  const bool grouped = p.group_off != nullptr;
  if (grouped) griddep_wait();  // the slot ranges come from the kernel before
  int row_tile;
  if (!lin_enter_group(p, kLsBM, row_tile)) return;
  const int row0 = row_tile * kLsBM, col0 = blockIdx.x * BN, k_tiles = p.k / kLsBK;
  auto load_w = [&](int kt) {
    bf16* sw = ring + size_t(kt % kLsStages) * STAGE + kLsBM * kLsPitch;
#pragma unroll
    for (int it = 0; it < WC; ++it) {
      const int chunk = tid + it * kLsThreads, r = chunk >> 3, c = (chunk & 7) * 8, col = col0 + r;
      ls_cp_async_16(sw + r * kLsPitch + c, p.w + size_t(col < p.n ? col : 0) * p.k + kt * kLsBK + c, col < p.n);
    }
  };
  const int pre = k_tiles < kLsStages - 1 ? k_tiles : kLsStages - 1;
  for (int kt = 0; kt < pre; ++kt) load_w(kt);
  if (!grouped) griddep_wait();
  const bf16* a_src[AC];
  bool a_ok[AC];
#pragma unroll
  for (int it = 0; it < AC; ++it) {
    const int chunk = tid + it * kLsThreads, r = row0 + (chunk >> 3);
    a_ok[it] = r < p.rows;
    a_src[it] = p.a + size_t(a_ok[it] ? (p.a_row ? p.a_row[r] : r) : 0) * p.lda + (chunk & 7) * 8;
  }
  auto load_a = [&](int kt) {
    bf16* sa = ring + size_t(kt % kLsStages) * STAGE;
#pragma unroll
    for (int it = 0; it < AC; ++it) {
      const int chunk = tid + it * kLsThreads;
      ls_cp_async_16(sa + (chunk >> 3) * kLsPitch + (chunk & 7) * 8, a_src[it] + kt * kLsBK, a_ok[it]);
    }
  };
#pragma unroll 1
  for (int kt = 0; kt < kLsStages - 1; ++kt) {
    if (kt < k_tiles) load_a(kt);
    asm volatile("cp.async.commit_group;" ::: "memory");  // (the first group holds all the weights asked for so far)
  }
  float acc[2][NF][4];
#pragma unroll
  for (int i = 0; i < 2; ++i)
#pragma unroll
    for (int j = 0; j < NF; ++j)
#pragma unroll
      for (int e = 0; e < 4; ++e) acc[i][j][e] = 0.0f;
  const bool second = p.rows - row0 > 16;  // (rows 16 .. 31 of the tile exist)
  const int wn = warp * 8 * NF;
  for (int kt = 0; kt < k_tiles; ++kt) {
    asm volatile("cp.async.wait_group %0;" ::"n"(kLsStages - 2) : "memory");  // k step kt has landed (this thread's part)
    __syncthreads();  // ... everybody's; and everybody is done with the stage of step kt - 1, which the next load overwrites
    if (kt + kLsStages - 1 < k_tiles) {
      load_w(kt + kLsStages - 1);
      load_a(kt + kLsStages - 1);
    }
    asm volatile("cp.async.commit_group;" ::: "memory");  // (an empty group keeps the count of groups per iteration uniform)
    const bf16* sa = ring + size_t(kt % kLsStages) * STAGE;
    const bf16* sw = sa + kLsBM * kLsPitch;
#pragma unroll
    for (int kk = 0; kk < kLsBK; kk += 16) {
      uint32_t bfr[NF][2];
#pragma unroll
      for (int j = 0; j < NF; ++j) {
        const bf16* base = sw + (wn + j * 8 + g) * kLsPitch + kk + 2 * t;
        bfr[j][0] = *reinterpret_cast<const uint32_t*>(base);
        bfr[j][1] = *reinterpret_cast<const uint32_t*>(base + 8);
      }
#pragma unroll
      for (int i = 0; i < 2; ++i) {
        if (i == 1 && !second) break;
        const bf16* base = sa + (i * 16 + g) * kLsPitch + kk + 2 * t;
        const uint32_t a0 = *reinterpret_cast<const uint32_t*>(base), a1 = *reinterpret_cast<const uint32_t*>(base + 8 * kLsPitch),
                       a2 = *reinterpret_cast<const uint32_t*>(base + 8), a3 = *reinterpret_cast<const uint32_t*>(base + 8 * kLsPitch + 8);
#pragma unroll
        for (int j = 0; j < NF; ++j)
          asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
                       : "+f"(acc[i][j][0]), "+f"(acc[i][j][1]), "+f"(acc[i][j][2]), "+f"(acc[i][j][3])
                       : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(bfr[j][0]), "r"(bfr[j][1]));
      }
    }
  }
  asm volatile("cp.async.wait_group 0;" ::: "memory");
#pragma unroll
  for (int i = 0; i < 2; ++i)
#pragma unroll
    for (int j = 0; j < NF; ++j) {
      const int r = row0 + i * 16 + g, c = col0 + wn + j * 8 + 2 * t;
      lin_store_pair<bf16, EPI>(p, r, c, acc[i][j][0], acc[i][j][1]);
      lin_store_pair<bf16, EPI>(p, r + 8, c, acc[i][j][2], acc[i][j][3]);
    }
}

}  // namespace mtx
