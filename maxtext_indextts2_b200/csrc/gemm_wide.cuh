// GEMM of steps with more than 256 rows (prompts and long portions of prompts): all rows of the step in one launch.
//
//   acc[r, n] = sum_k A[r, k] * W[n, k]        both operands K-major bf16, fp32 accumulation in TMEM
//
// gemm_rows.cuh takes at most 256 rows per launch, so a prompt of 4096 rows read every weight tile sixteen times and paid sixteen
// launches, pipeline fills and drains per projection: 20 % of the bf16 rate.  Here two CTAs of a cluster (a TPC's two SMs) work on one
// tile of 256 rows x BN columns with cta_group::2 MMAs (M = 256): CTA c of the pair holds rows 128 c .. of A and half of the
// weight tile's rows, so that an SM takes in 16 KB + BN * 64 B per k block of 64 for BN * 2^15 multiply-adds.  One pair per TPC walks the
// tiles (rows fastest, so that the pairs at work share weight tiles in L2), the 512 TMEM columns hold as many accumulators as fit (two of
// 256 columns, four of 128): the eight epilogue warps of each CTA drain a tile under the next tiles' MMAs.
//
// BN is chosen per shape (wide_tile_columns) so that the tiles fill whole waves of pairs.
//
// Bound: the tensor pipe at BN = 256 (0.32 us per k block of a tile with the grid full; 4096 x 2048 x 4096 in 47 us, 1.45 PFLOP/s, 0.91 of the 1.59 that
// cuBLAS reaches in a burst; gemm_rows.cuh in sixteen launches: 257 us), below that the round of barrier, four MMAs and commit
// (0.2 us per k block up to 128 columns).  That round took 0.29 us as long as the issuing threads were picked by `lane == 0`.
//
//   warp 0    TMA: its CTA's half of both operands into a ring of stages, both halves counted on the leader's barrier
//   warp 1    the leader's issues tcgen05.mma and commits (multicast to both CTAs' barriers)
//   warps 2-9 epilogue: a thread owns one row (TMEM lane) and half of the tile's columns
//
// The epilogue is a class with  prepare(tile)  (what a thread needs of its row, read while the tile's MMAs run) and
// operator()(tile, n, prepared, load)  where load(c, v) reads the accumulator's 16 columns c .. c + 15.
//
// Segments: gemm_rows.cuh cuts the k blocks of a narrow projection over a cluster and adds the parts in order.  With `segments` set to that
// number a tile's k range is accumulated in the same parts, which the epilogue threads add in registers, so that a row's result is bit
// for bit what the 256-row steps give it, however many rows its step has.  Such an epilogue works on one fragment of 16 columns at a
// time (kFragments; fragment(tile, n, column, values)).
// Grouped (GROUPED; the experts of a routed feed-forward): the rows are slots, group g's are [group_off[g], group_off[g + 1]) (known on the
// device only) and its weight the rows g * n .. of W.  The pairs walk the groups' row tiles one group after the other; a group's last tile
// reads the next group's rows and drops their results.
#pragma once

#include "gemm_rows.cuh"

namespace mtx {

constexpr int kPairThreads = 320;
constexpr int kPairRows = 256;    // rows of a pair's tile
constexpr int kPairMaxCols = 256;
constexpr int kPairMaxStages = 12;
constexpr int kPairMaxAcc = 8;    // accumulators in TMEM (tiles of 64 columns)
constexpr int kPairABytes = 128 * kBlockK * 2;  // a CTA's part of an A stage

struct WideParams {
  int rows, n, k;
  int bn;      // columns of a tile: a multiple of 32, at most 256
  int stages;  // depth of the ring
  int segments;  // parts that a tile's k blocks are accumulated in (1, or an epilogue with kFragments)
  const int* group_off;  // GROUPED: [groups + 1]
  int groups;
  int first;   // columns of a tile's first half (the epilogue warps 2-5; the warps 6-9 take the rest)
};

struct WideSmemTail {
  uint64_t full[kPairMaxStages];
  uint64_t empty[kPairMaxStages];
  uint64_t tmem_full[kPairMaxAcc];
  uint64_t tmem_empty[kPairMaxAcc];
  uint32_t tmem_base;
  uint32_t pad;
};

__host__ __device__ inline size_t wide_stage_bytes(int bn) { return size_t(kPairABytes) + size_t(bn / 2) * kBlockK * 2; }
__host__ __device__ inline size_t wide_smem_bytes(int bn, int stages) { return 1024 + stages * wide_stage_bytes(bn) + sizeof(WideSmemTail) + 16; }
// as many stages as an SM's shared memory holds: a stage comes round in one to two microseconds (TMA, the leader's barrier, the MMAs, the
// commit back to both CTAs) whatever its size, so narrow tiles want more of them
inline int wide_stages(int bn) {
  const int n = int((227 * 1024 - wide_smem_bytes(bn, 0)) / wide_stage_bytes(bn));
  return n < kPairMaxStages ? n : kPairMaxStages;
}

// what an epilogue thread works on: its row, and the columns [c0, c1) of the tile that starts at column n0 of the output
struct WideTile {
  int row;
  bool valid;
  int n0, c0, c1;
  int slice;  // index of this run of columns among all the runs of a row: 2 * tile + half
};

// ---- cta_group::2 forms ----------------------------------------------------------------------------------------------------

constexpr uint32_t kPairLeaderMask = 0xFEFFFFFFu;  // a shared::cluster address with the pair's low rank bit cleared: the leader's copy

// 2-D tiled load into this CTA's shared memory; the bytes count on the LEADER's barrier
__device__ __forceinline__ void tma_load_2d_pair(void* dst, const CUtensorMap* tm, int c0, int c1, uint64_t* bar, uint64_t hint) {
  asm volatile(
      "cp.async.bulk.tensor.2d.cta_group::2.shared::cluster.global.mbarrier::complete_tx::bytes.L2::cache_hint"
      " [%0], [%1, {%3, %4}], [%2], %5;"
      :
      : "r"(smem_u32(dst)), "l"(reinterpret_cast<uint64_t>(tm)), "r"(smem_u32(bar) & kPairLeaderMask), "r"(c0), "r"(c1), "l"(hint)
      : "memory");
}
__device__ __forceinline__ void tmem_alloc_pair(uint32_t* dst_smem, uint32_t ncols) {
  asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(dst_smem)), "r"(ncols) : "memory");
}
__device__ __forceinline__ void tmem_relinquish_pair() { asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory"); }
__device__ __forceinline__ void tmem_dealloc_pair(uint32_t taddr, uint32_t ncols) {
  asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(taddr), "r"(ncols) : "memory");
}
__device__ __forceinline__ void umma_bf16_pair(uint32_t tmem_d, uint64_t desc_a, uint64_t desc_b, uint32_t idesc, uint32_t accumulate) {
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::2.kind::f16 [%0], %1, %2, %3, p;\n\t}"
      :
      : "r"(tmem_d), "l"(desc_a), "l"(desc_b), "r"(idesc), "r"(accumulate)
      : "memory");
}
// arrives on the barrier at this offset in both CTAs of the pair once the MMAs issued so far are done
__device__ __forceinline__ void umma_commit_pair(uint64_t* bar) {
  asm volatile("tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], %1;" ::"r"(smem_u32(bar)), "h"(uint16_t(3))
               : "memory");
}
__device__ __forceinline__ void mbar_arrive_leader(uint64_t* bar) {
  asm volatile("mbarrier.arrive.release.cluster.shared::cluster.b64 _, [%0];" ::"r"(smem_u32(bar) & kPairLeaderMask) : "memory");
}

// ---- the kernel ----------------------------------------------------------------------------------------------------------------

template <class EPI, bool GROUPED>
__global__ void __launch_bounds__(kPairThreads, 1)
gemm_wide_kernel(const __grid_constant__ CUtensorMap tm_w, const __grid_constant__ CUtensorMap tm_a, const WideParams p, const EPI epi) {
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = smem_raw + ((1024u - (smem_u32(smem_raw) & 1023u)) & 1023u);
  const int stage_bytes = int(wide_stage_bytes(p.bn)), half_n = p.bn / 2;
  WideSmemTail* tail = reinterpret_cast<WideSmemTail*>(smem + size_t(p.stages) * stage_bytes);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int rank = int(blockIdx.x) & 1, pair = int(blockIdx.x) >> 1, pairs = int(gridDim.x) >> 1;  // (the cluster is two CTAs along x)
  const int nkb = p.k / kBlockK;
  const int n_acc = 512 / p.bn;

  griddep_launch_dependents();
  if (warp == 0 && lane == 0) {
    tma_prefetch_desc(&tm_w);
    tma_prefetch_desc(&tm_a);
    for (int s = 0; s < p.stages; ++s) {
      mbar_init(&tail->full[s], 1);
      mbar_init(&tail->empty[s], 1);
    }
    for (int b = 0; b < n_acc; ++b) {
      mbar_init(&tail->tmem_full[b], 1);
      mbar_init(&tail->tmem_empty[b], 16);  // the eight epilogue warps of both CTAs
    }
    fence_barrier_init();
  }
  if (warp == 1) {
    tmem_alloc_pair(&tail->tmem_base, 512);
    tmem_relinquish_pair();
  }
  tcgen05_fence_before();
  cluster_sync_all();
  tcgen05_fence_after();
  const uint32_t tmem_base = tail->tmem_base;

  int m_tiles = (p.rows + kPairRows - 1) / kPairRows;
  if (GROUPED) {
    griddep_wait();  // the slot ranges come from the kernel before
    m_tiles = 0;
    for (int g = 0; g < p.groups; ++g) m_tiles += (p.group_off[g + 1] - p.group_off[g] + kPairRows - 1) / kPairRows;
  }
  const int n_tiles = (p.n + p.bn - 1) / p.bn, tiles = m_tiles * n_tiles;
  const int my_tiles = pair < tiles ? (tiles - pair + pairs - 1) / pairs : 0;
  const int F = my_tiles * nkb;
  // row tile m: its first row, how many rows follow from there, the row of W where its weight begins
  struct Rows {
    int row0, left, w0;
  };
  auto rows_of = [&](int m) {
    Rows r = {m * kPairRows, p.rows - m * kPairRows, 0};
    if (GROUPED) {
      int off = p.group_off[0];
      for (int g = 0; g < p.groups; ++g) {
        const int end = p.group_off[g + 1], nt = (end - off + kPairRows - 1) / kPairRows;
        if (m < nt) {
          r.row0 = off + m * kPairRows;
          r.left = end - r.row0;
          r.w0 = g * p.n;
          break;
        }
        m -= nt;
        off = end;
      }
    }
    return r;
  };

  if (warp == 0) {
    // (the whole warp counts and waits, one elected lane issues: a branch on the lane number makes the compiler guard every issue against
    // divergence.  Stage, phase, k block and tile are counted, not divided out of a fill number.)
    const bool issuer = elect_one();
    const int m_div = m_tiles > 0 ? m_tiles : 1;  // (no slots at all: no tiles)
    int s = 0, kb = 0, m = pair % m_div, nt = pair / m_div;
    uint32_t phase = 1;
    const int m_step = pairs % m_div, n_step = pairs / m_div;
    Rows at = rows_of(m_tiles > 0 ? m : 0);
    auto w_load = [&](int stage, int k) {
      if (rank == 0) mbar_expect_tx(&tail->full[stage], uint32_t(2 * stage_bytes));
      tma_load_2d_pair(smem + stage * stage_bytes + kPairABytes, &tm_w, k * kBlockK, at.w0 + nt * p.bn + rank * half_n, &tail->full[stage], kEvictLast);
    };
    auto a_load = [&](int stage, int k) {
      tma_load_2d_pair(smem + stage * stage_bytes, &tm_a, k * kBlockK, at.row0 + rank * 128, &tail->full[stage], kEvictLast);
    };
    // the first tile's weights do not depend on the previous kernel
    const int pre = my_tiles == 0 ? 0 : (nkb < p.stages ? nkb : p.stages);
    if (issuer)
      for (int f = 0; f < pre; ++f) w_load(f, f);
    if (!GROUPED) griddep_wait();
    if (issuer)
      for (int f = 0; f < pre; ++f) a_load(f, f);
    for (int f = 0; f < F; ++f) {
      if (f >= pre) {
        mbar_wait(&tail->empty[s], phase);
        if (issuer) {
          w_load(s, kb);
          a_load(s, kb);
        }
      }
      if (++s == p.stages) s = 0, phase ^= 1;
      if (++kb == nkb) {
        kb = 0;
        nt += n_step;
        m += m_step;
        if (m >= m_tiles) m -= m_tiles, ++nt;
        if (f + 1 < F) at = rows_of(m);
      }
    }
    // the commits of the last stages arrive on this CTA's barriers too: they have to be there before it may leave
    const int last = F < p.stages ? F : p.stages;
    for (int f = 0; f < last; ++f) {
      if (s == 0) s = p.stages, phase ^= 1;
      --s;
      mbar_wait(&tail->empty[s], phase ^ 1);
    }
    __syncwarp();
  } else if (warp == 1) {
    if (rank == 0) {
      const bool issuer = elect_one();
      const uint32_t idesc = umma_idesc_bf16(kPairRows, p.bn);
      const uint64_t d0 = umma_desc_sw128(smem);
      const uint32_t step = uint32_t(stage_bytes) >> 4;  // descriptors count in 16-byte units
      int s = 0, buf = 0;
      uint32_t phase = 0, acc_phase = 1;
      for (int j = 0, seg = 0; j < my_tiles * p.segments; ++j) {  // (tile, segment)
        mbar_wait(&tail->tmem_empty[buf], acc_phase);
        tcgen05_fence_after();
        const uint32_t acc = tmem_base + uint32_t(buf * p.bn);
        const int n_seg = (seg + 1) * nkb / p.segments - seg * nkb / p.segments;
        if (++seg == p.segments) seg = 0;
        for (int i = 0; i < n_seg; ++i) {
          mbar_wait(&tail->full[s], phase);
          tcgen05_fence_after();
          if (issuer) {
            const uint64_t da = d0 + uint64_t(uint32_t(s) * step), dw = da + uint64_t(kPairABytes >> 4);
#pragma unroll
            for (int kk = 0; kk < kBlockK / kUmmaK; ++kk) umma_bf16_pair(acc, da + uint64_t(kk * 2), dw + uint64_t(kk * 2), idesc, uint32_t((i | kk) != 0));
            umma_commit_pair(&tail->empty[s]);
          }
          if (++s == p.stages) s = 0, phase ^= 1;
        }
        if (issuer) umma_commit_pair(&tail->tmem_full[buf]);
        if (++buf == n_acc) buf = 0, acc_phase ^= 1;
      }
    }
    __syncwarp();
  } else {
    const int half = (warp - 2) >> 2, quarter = warp & 3;
    const int c0 = half == 0 ? 0 : p.first, c1 = half == 0 ? p.first : p.bn;
    if (!GROUPED) griddep_wait();  // side inputs (residual rows, row statistics) come from earlier kernels
    int buf = 0;
    uint32_t acc_phase = 0;
    auto release = [&]() {  // this warp is done with the accumulator
      tcgen05_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive_leader(&tail->tmem_empty[buf]);
      if (++buf == n_acc) buf = 0, acc_phase ^= 1;
    };
    for (int j = 0; j < my_tiles; ++j) {
      const int t = pair + j * pairs;
      WideTile w;
      const Rows at = rows_of(t % m_tiles);
      const int local = rank * 128 + quarter * 32 + lane;
      w.row = at.row0 + local;
      w.valid = local < at.left;
      w.n0 = (t / m_tiles) * p.bn;
      w.c0 = c0;
      w.c1 = w.n0 + c1 < p.n ? c1 : (w.n0 + c0 < p.n ? p.n - w.n0 : c0);
      w.slice = 2 * (t / m_tiles) + half;
      const uint32_t lanes = tmem_base + (uint32_t(quarter * 32) << 16);
      if constexpr (EPI::kFragments) {
        if (p.segments > 1) {
          float acc[kPairMaxCols / 32][16];
          const auto pre = epi.prepare(w);
          for (int seg = 0; seg < p.segments; ++seg) {
            const uint32_t taddr = lanes + uint32_t(buf * p.bn + w.c0);
            mbar_wait(&tail->tmem_full[buf], acc_phase);
            tcgen05_fence_after();
#pragma unroll
            for (int i = 0; i < kPairMaxCols / 32; i += 2)  // (32 columns in flight: what the registers beside the sums hold)
              if (w.c0 + 16 * i < w.c1) {
                uint32_t v[2][16];
                tmem_ld_x16_issue(taddr + uint32_t(16 * i), v[0]);
                tmem_ld_x16_issue(taddr + uint32_t(16 * i + 16), v[1]);
                tmem_ld_wait();
#pragma unroll
                for (int x = 0; x < 32; ++x) {
                  const float y = __uint_as_float(v[x >> 4][x & 15]);
                  acc[i + (x >> 4)][x & 15] = seg == 0 ? y : acc[i + (x >> 4)][x & 15] + y;
                }
              }
            release();
          }
#pragma unroll
          for (int i = 0; i < kPairMaxCols / 32; i += 2)
            if (w.c0 + 16 * i < w.c1 && w.valid) epi.fragment(w, p.n, pre, w.c0 + 16 * i, acc[i], acc[i + 1]);
          continue;
        }
      }
      const uint32_t taddr = lanes + uint32_t(buf * p.bn);
      const auto pre = epi.prepare(w);
      mbar_wait(&tail->tmem_full[buf], acc_phase);
      tcgen05_fence_after();
      epi(w, p.n, pre, [&](int c, float (&v)[16]) { tmem_ld_x16(taddr + uint32_t(c), v); });
      release();
    }
  }
  tcgen05_fence_before();
  cluster_sync_all();  // the pair's shared memory and TMEM are in use until both CTAs are done
  tcgen05_fence_after();
  if (warp == 1) tmem_dealloc_pair(tmem_base, 512);
}

// ---- epilogues of the decoder engine --------------------------------------------------------------------------------------------
// What gemm_rows.cuh's fragments compute, with the arithmetic between the accumulator and the stored value in fp32 and one rounding
// at the end (those round every intermediate array to bf16; against float64 this side is the closer one); STEP: with their roundings.

// the row's 1 / rms from the partial sums of squares that a residual epilogue left
__device__ __forceinline__ float wide_rstd(const EpiArgs& e, int row) {
  float tot = 0.0f;
#pragma unroll 8
  for (int t = 0; t < e.ss_tiles; ++t) tot += __ldcg(e.ss_in + (long long)t * e.ss_pitch + row);
  return 1.0f / sqrtf(tot / float(e.ss_dim) + e.ss_eps);
}

// out = bf16(resid + acc); returns the sum of squares of the stored values
__device__ __forceinline__ float wide_residual(const EpiArgs& e, int r, int n0, const float (&v)[16]) {
  const long long o = (long long)r * e.ld_out + n0;
  const uint4 ra = *reinterpret_cast<const uint4*>(e.resid + o), rb = *reinterpret_cast<const uint4*>(e.resid + o + 8);
  const uint32_t w[8] = {ra.x, ra.y, ra.z, ra.w, rb.x, rb.y, rb.z, rb.w};
  uint32_t s[8];
  float sq = 0.0f;
#pragma unroll
  for (int j = 0; j < 8; ++j) {
    s[j] = pack_bf16x2(bf16_lo(w[j]) + v[2 * j], bf16_hi(w[j]) + v[2 * j + 1]);
    sq += bf16_lo(s[j]) * bf16_lo(s[j]) + bf16_hi(s[j]) * bf16_hi(s[j]);
  }
  *reinterpret_cast<uint4*>(e.out + o) = make_uint4(s[0], s[1], s[2], s[3]);
  *reinterpret_cast<uint4*>(e.out + o + 8) = make_uint4(s[4], s[5], s[6], s[7]);
  return sq;
}

// 16 gates and the 16 values that belong to them
__device__ __forceinline__ void wide_gate(const EpiArgs& e, int r, int n0, const float (&g)[16], const float (&u)[16]) {
  float o[16];
#pragma unroll
  for (int j = 0; j < 16; ++j) {
    o[j] = __fdividef(g[j], 1.0f + __expf(-g[j])) * u[j];
  }
  frag_store_bf16(e.out + (long long)r * e.ld_out + (n0 >> 1), o);
}

// dims d0 .. d0 + 15 of a head's first half and the same of its second half (d0 + D / 2): rotated queries, appended keys and values
__device__ __forceinline__ void wide_qkv(const EpiArgs& e, int r, int head, int d0, float (&a)[16], float (&b)[16]) {
  const int D = e.d, half = D >> 1;
  if (head < e.hq + e.hkv) {
    const float4* cs = reinterpret_cast<const float4*>(e.rope_cs + (long long)r * half + d0);
#pragma unroll
    for (int j = 0; j < 16; j += 2) {
      const float4 c = cs[j >> 1];
      const float a0 = a[j], b0 = b[j], a1 = a[j + 1], b1 = b[j + 1];
      a[j] = a0 * c.x - b0 * c.y;
      b[j] = b0 * c.x + a0 * c.y;
      a[j + 1] = a1 * c.z - b1 * c.w;
      b[j + 1] = b1 * c.z + a1 * c.w;
    }
  }
  bf16* dst;
  if (head < e.hq) {
    dst = e.q_out + (long long)r * (e.hq * D) + head * D + d0;
  } else {
    const int wr = e.write_row[r];
    if (wr < 0) return;
    const int kvh = (head - e.hq) % e.hkv;
    dst = (head < e.hq + e.hkv ? e.k_cache : e.v_cache) + (((long long)e.plane[r] * e.hkv + kvh) * e.t_alloc + wr) * D + d0;
  }
  frag_store_bf16(dst, a);
  frag_store_bf16(dst + half, b);
}

template <int KIND, bool STEP = false>
struct WideEpi {
  static constexpr bool kFragments = KIND == EPI_STORE_BF16 || (KIND == EPI_SWIGLU && STEP);
  EpiArgs e;

  __device__ __forceinline__ float prepare(const WideTile& w) const {
    if (KIND == EPI_RESIDUAL || e.ss_in == nullptr || !w.valid) return 1.0f;
    return STEP ? rows_rstd(e, w.row) : wide_rstd(e, w.row);
  }

  // 32 columns of a row
  __device__ __forceinline__ void fragment(const WideTile& w, int n, float rs, int c, float (&a)[16], float (&b)[16]) const {
    rows_scale16(a, rs);
    rows_scale16(b, rs);
    if (KIND == EPI_SWIGLU) {
      if (STEP) rows_epi_swiglu(e, n, w.row, w.n0 + c, a, b);
      else wide_gate(e, w.row, w.n0 + c, a, b);
    } else {
      rows_epi_store(e, n, w.row, w.n0 + c, a);
      rows_epi_store(e, n, w.row, w.n0 + c + 16, b);
    }
  }

  template <class LD>
  __device__ __forceinline__ void operator()(const WideTile& w, int n, float rs, LD&& ld16) const {
    if (KIND == EPI_STORE_BF16) {
      for (int c = w.c0; c < w.c1; c += 16) {
        float v[16];
        ld16(c, v);
        rows_scale16(v, rs);
        if (w.valid) rows_epi_store(e, n, w.row, w.n0 + c, v);
      }
    } else if (KIND == EPI_RESIDUAL) {
      float sq = 0.0f;
      for (int c = w.c0; c < w.c1; c += 16) {
        float v[16];
        ld16(c, v);
        if (w.valid) sq += wide_residual(e, w.row, w.n0 + c, v);
      }
      if (e.ss_out != nullptr && w.valid) e.ss_out[(long long)w.slice * e.ss_pitch + w.row] = sq;
    } else if (KIND == EPI_SWIGLU) {
      for (int c = w.c0; c < w.c1; c += 32) {
        float g[16], u[16];
        ld16(c, g);
        ld16(c + 16, u);
        if (w.valid) fragment(w, n, rs, c, g, u);
      }
    } else if (KIND == EPI_QKV_ROPE) {
      const int half = e.d >> 1;
      for (int h = w.c0; h < w.c1; h += e.d)
        for (int d = 0; d < half; d += 16) {
          float lo[16], hi[16];
          ld16(h + d, lo);
          ld16(h + d + half, hi);
          rows_scale16(lo, rs);
          rows_scale16(hi, rs);
          if (w.valid) wide_qkv(e, w.row, (w.n0 + h) / e.d, d, lo, hi);
        }
    }
  }
};

}  // namespace mtx
