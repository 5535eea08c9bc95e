// GEMM of steps with more than 256 rows (prompts and long portions of prompts), all rows of the step in one launch, and of some decode steps' gated up-projections
// (65 to 256 rows: takes_wide_up).
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
// (0.2 us per k block up to 128 columns, 0.13 with two k blocks per stage).  That round took 0.29 us as long as the issuing threads were picked by `lane == 0`.
//
//   warp 0    TMA: its CTA's half of both operands into a ring of stages, both halves counted on the leader's barrier
//   warp 1    the leader's issues tcgen05.mma and commits (multicast to both CTAs' barriers)
//   warps 2-9 epilogue: a thread owns one row (TMEM lane) and half of the tile's columns
//
// The epilogue is a class with  prepare(tile, stage)  (what a thread needs of its row, read while the tile's MMAs run) and either (kFragments)
// fragment(tile, prepared, c, a, b, stage)  for the accumulator's columns c .. c + 15 and c + 16 .. c + 31, or  operator()(tile, prepared, load, stage)
// where load(ca, a, cb, b) reads 16 columns from each of ca and cb on.  All lanes of a warp call them, rows that are not there included: `stage` (WideStage) takes
// a warp's outputs to whole lines.
//
// Segments: gemm_rows.cuh cuts the k blocks of a narrow projection over a cluster and adds the parts in order.  With `segments` set to that
// number a tile's k range is accumulated in the same parts, which the epilogue threads add in registers, so that a row's result is bit
// for bit what the 256-row steps give it, however many rows its step has (MODE kWideParts, epilogues with kFragments).
// Grouped (MODE kWideGrouped; the experts of a routed feed-forward): the rows are slots, group g's are [group_off[g], group_off[g + 1]) (known on the
// device only) and its weight the rows g * n .. of W.  The pairs walk the groups' row tiles one group after the other; a group's last tile
// reads the next group's rows and drops their results.
#pragma once

#include <type_traits>

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
  int group;   // k blocks of a stage: 1 or 2 (then every segment has an even number of them)
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

// (of one k block)
__host__ __device__ inline size_t wide_stage_bytes(int bn) { return size_t(kPairABytes) + size_t(bn / 2) * kBlockK * 2; }
__host__ __device__ inline size_t wide_smem_bytes(int bn, int stages, int group, int row) {
  return 1024 + size_t(stages) * group * wide_stage_bytes(bn) + 8 * 32 * row + sizeof(WideSmemTail) + 16;
}
// as many stages as an SM's shared memory holds: a stage comes round in one to two microseconds (TMA, the leader's barrier, the MMAs, the
// commit back to both CTAs) whatever its size, so narrow tiles want more of them
inline int wide_stages(int bn, int group, int row) {
  const int n = int((227 * 1024 - wide_smem_bytes(bn, 0, group, row)) / (group * wide_stage_bytes(bn)));
  return n < kPairMaxStages ? n : kPairMaxStages;
}

// what an epilogue thread works on: its row, and the columns [c0, c1) of the tile that starts at column n0 of the output
struct WideTile {
  int row;    // of this thread; row - lane is the warp's first
  int rows;   // rows of the warp that are there: its first so many lanes (32, or fewer in the last row tile)
  bool valid;
  int n0, c0, c1;
  int slice;  // index of this run of columns among all the runs of a row: 2 * tile + half
};

// A warp's 32 rows x 64 or 128 bytes between the arithmetic, where a thread owns a row, and global memory, where neighbouring lanes share a row's
// bytes.  Chunk j (16 bytes) of row r lies at j ^ (r & 7), at j ^ (r >> 1 & 3) in rows of 64 bytes: neither side has bank conflicts.  A thread that stored its own row wrote half sectors
// of 32 rows per instruction, and the next tile's operands waited behind them: 4000 x 1792 x 1280 (rotated q, k, v) took 12 us for
// the second of its tiles, 5 without an epilogue beside it.
template <int ROW>  // bytes of a row: 64 or 128
struct WideStage {
  static constexpr int kChunks = ROW / 16;
  uint8_t* buf;
  int lane;

  __device__ __forceinline__ uint4* at(int r, int j) const { return reinterpret_cast<uint4*>(buf + r * ROW + ((j ^ ((r >> (ROW == 64 ? 1 : 0)) & (kChunks - 1))) << 4)); }
  __device__ __forceinline__ void put(int j, const uint4& v) const { *at(lane, j) = v; }
  __device__ __forceinline__ uint4 get(int j) const { return *at(lane, j); }

  // f(i, r, j) for the chunks j < n of the rows r < rows: lane by lane in i = 0 .. kChunks - 1, rows of n chunks (rounded up to a power of two) side by side
  template <class F>
  __device__ __forceinline__ void each(int n, int rows, F&& f) const {
    const int sh = n > 4 ? 3 : n > 2 ? 2 : 1, j = lane & ((1 << sh) - 1);
#pragma unroll
    for (int i = 0; i < kChunks; ++i) {
      const int r = i * (32 >> sh) + (lane >> sh);
      if (i < (1 << sh) && j < n && r < rows) f(i, r, j);
    }
  }
  // chunks [0, n) of the first `rows` rows, row r at p + r * pitch: global -> registers -> the buffer (the caller syncs the warp after place)
  __device__ __forceinline__ void fetch(int n, const void* p, size_t pitch, int rows, uint4 (&v)[kChunks]) const {
    each(n, rows, [&](int i, int r, int j) { v[i] = *reinterpret_cast<const uint4*>(static_cast<const char*>(p) + r * pitch + j * 16); });
  }
  __device__ __forceinline__ void place(int n, const uint4 (&v)[kChunks]) const {
    each(n, 32, [&](int i, int r, int j) { *at(r, j) = v[i]; });
  }
  // the same without registers in between: on its way when this returns, there for the warp behind arrived()
  __device__ __forceinline__ void bring(int n, const void* p, size_t pitch, int rows) const {
    each(n, rows, [&](int, int r, int j) {
      asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(smem_u32(at(r, j))), "l"(static_cast<const char*>(p) + r * pitch + j * 16) : "memory");
    });
    asm volatile("cp.async.commit_group;" ::: "memory");
  }
  __device__ __forceinline__ void arrived() const {
    asm volatile("cp.async.wait_group 0;" ::: "memory");
    __syncwarp();
  }
  // the buffer's chunks [0, n) of the first `rows` rows to p + r * pitch
  __device__ __forceinline__ void flush(int n, void* p, size_t pitch, int rows) const {
    __syncwarp();
    each(n, rows, [&](int, int r, int j) { *reinterpret_cast<uint4*>(static_cast<char*>(p) + r * pitch + j * 16) = *at(r, j); });
    __syncwarp();
  }
  // four chunks of every row: two to the row's own `dst` (null: the row is not stored), two to dst + far
  __device__ __forceinline__ void flush_pairs(bf16* dst, int far) const {
    const int j = lane & 3;
    __syncwarp();
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const int r = i * 8 + (lane >> 2);
      bf16* p = reinterpret_cast<bf16*>(__shfl_sync(0xffffffffu, reinterpret_cast<unsigned long long>(dst), r));
      if (p != nullptr) *reinterpret_cast<uint4*>(p + (j >> 1) * far + (j & 1) * 8) = *at(r, j);
    }
    __syncwarp();
  }

  // 32 accumulator columns from c on become CH chunks of this thread's row: from which one on ...
  template <int CH>
  __device__ __forceinline__ int chunk(const WideTile& w, int c) const { return ((c - w.c0) / 32 & (kChunks / CH - 1)) * CH; }
  // ... and, once they are put, on to memory with the ones before them when the buffer's rows or the columns are full.  out: where the warp's first row has
  // what comes of column w.c0
  template <int CH>
  __device__ __forceinline__ void done(const WideTile& w, int c, void* out, size_t pitch) const {
    static_assert(CH <= kChunks, "32 columns have to fit a row of the buffer");
    const int f = (c - w.c0) / 32, s = f & (kChunks / CH - 1);
    if (s == kChunks / CH - 1 || c + 32 >= w.c1) flush((s + 1) * CH, static_cast<char*>(out) + size_t(f - s) * (CH * 16), pitch, w.rows);
  }
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
__device__ __forceinline__ uint64_t umma_desc_of(uint32_t lo, uint32_t hi) { return uint64_t(hi) << 32 | lo; }
// arrives on the barrier at this offset in both CTAs of the pair once the MMAs issued so far are done
__device__ __forceinline__ void umma_commit_pair(uint64_t* bar) {
  asm volatile("tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], %1;" ::"r"(smem_u32(bar)), "h"(uint16_t(3))
               : "memory");
}
__device__ __forceinline__ void mbar_arrive_leader(uint64_t* bar) {
  asm volatile("mbarrier.arrive.release.cluster.shared::cluster.b64 _, [%0];" ::"r"(smem_u32(bar) & kPairLeaderMask) : "memory");
}

// ---- the kernel ----------------------------------------------------------------------------------------------------------------

// rows of the step, a tile's k range as one sum; rows of the experts' slots; the sum in parts (a kernel of its own: the parts' registers)
enum WideMode { kWideRows = 0, kWideGrouped = 1, kWideParts = 2 };

template <class EPI, int MODE>
__global__ void __launch_bounds__(kPairThreads, 1)
gemm_wide_kernel(const __grid_constant__ CUtensorMap tm_w, const __grid_constant__ CUtensorMap tm_a, const WideParams p, const EPI epi) {
  constexpr bool GROUPED = MODE == kWideGrouped;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = smem_raw + ((1024u - (smem_u32(smem_raw) & 1023u)) & 1023u);
  const int block_bytes = int(wide_stage_bytes(p.bn)), stage_bytes = p.group * block_bytes, half_n = p.bn / 2;
  uint8_t* staged = smem + size_t(p.stages) * stage_bytes;
  WideSmemTail* tail = reinterpret_cast<WideSmemTail*>(staged + 8 * 32 * EPI::kRowBytes);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int rank = int(blockIdx.x) & 1, pair = int(blockIdx.x) >> 1, pairs = int(gridDim.x) >> 1;  // (the cluster is two CTAs along x)
  const int nkb = p.k / kBlockK / p.group;  // stages' worth of k blocks
  const int n_acc = 512 / p.bn, segments = MODE == kWideParts ? p.segments : 1;

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
    // Weights are read once per row tile: with one alone (a decode step's) nobody comes back for them, and what they would push out of L2 is what the step's next kernels
    // read.  Kept like several row tiles', they made a layer's kernels wait: 128 rows of a model of 2048 x 8192 108 us per layer, 103 so; 200 rows of 1280 x 5120 70 and 67.
    const uint64_t w_hint = !GROUPED && p.rows <= kPairRows ? kEvictFirst : kEvictLast;
    // the first tile's weights do not depend on the previous kernel
    const int pre = my_tiles == 0 ? 0 : (nkb < p.stages ? nkb : p.stages);
    auto fills = [&](auto group) {  // (as the MMAs below: in straight code, the issue of two loads takes as long as they do up to 128 columns)
      constexpr int G = decltype(group)::value;
      auto w_load = [&](int stage, int k) {
        if (rank == 0) mbar_expect_tx(&tail->full[stage], uint32_t(2 * stage_bytes));
#pragma unroll
        for (int g = 0; g < G; ++g)
          tma_load_2d_pair(smem + stage * stage_bytes + g * block_bytes + kPairABytes, &tm_w, (k * G + g) * kBlockK, at.w0 + nt * p.bn + rank * half_n, &tail->full[stage],
                           w_hint);
      };
      auto a_load = [&](int stage, int k) {
#pragma unroll
        for (int g = 0; g < G; ++g)
          tma_load_2d_pair(smem + stage * stage_bytes + g * block_bytes, &tm_a, (k * G + g) * kBlockK, at.row0 + rank * 128, &tail->full[stage], kEvictLast);
      };
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
    };
    if (p.group == 2) fills(std::integral_constant<int, 2>());
    else fills(std::integral_constant<int, 1>());
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
      // (the low words alone count on: an address in 16-byte units, 14 bits of it)
      const uint32_t desc_hi = uint32_t(d0 >> 32), desc_lo = uint32_t(d0), step = uint32_t(stage_bytes) >> 4;
      int s = 0, buf = 0;
      uint32_t phase = 0, acc_phase = 1;
      auto tiles_of = [&](auto group) {  // (the k blocks of a stage in straight code: the issue of four MMAs costs as much as they take up to 128 columns)
        constexpr int G = decltype(group)::value;
        const int whole = nkb / segments, over = nkb % segments;  // segment s ends at (s + 1) nkb / segments: counted, no division in the loop
        for (int j = 0, seg = 0, rest = 0; j < my_tiles * segments; ++j) {  // (tile, segment)
          mbar_wait(&tail->tmem_empty[buf], acc_phase);
          tcgen05_fence_after();
          const uint32_t acc = tmem_base + uint32_t(buf * p.bn);
          int n_seg = whole;
          if ((rest += over) >= segments) rest -= segments, ++n_seg;
          if (++seg == segments) seg = rest = 0;
          for (int i = 0; i < n_seg; ++i) {
            mbar_wait(&tail->full[s], phase);
            tcgen05_fence_after();
            if (issuer) {
              const uint32_t at = desc_lo + uint32_t(s) * step;
#pragma unroll
              for (int g = 0; g < G; ++g)
#pragma unroll
                for (int kk = 0; kk < kBlockK / kUmmaK; ++kk) {
                  const uint32_t da = at + uint32_t(g * (block_bytes >> 4) + kk * 2);
                  umma_bf16_pair(acc, umma_desc_of(da, desc_hi), umma_desc_of(da + uint32_t(kPairABytes >> 4), desc_hi), idesc, uint32_t((g | kk) != 0 || i != 0));
                }
              umma_commit_pair(&tail->empty[s]);
            }
            if (++s == p.stages) s = 0, phase ^= 1;
          }
          if (issuer) umma_commit_pair(&tail->tmem_full[buf]);
          if (++buf == n_acc) buf = 0, acc_phase ^= 1;
        }
      };
      if (p.group == 2) tiles_of(std::integral_constant<int, 2>());
      else tiles_of(std::integral_constant<int, 1>());
    }
    __syncwarp();
  } else {
    const int half = (warp - 2) >> 2, quarter = warp & 3;
    const int c0 = half == 0 ? 0 : p.first, c1 = half == 0 ? p.first : p.bn;
    if (!GROUPED) griddep_wait();  // side inputs (residual rows, row statistics) come from earlier kernels
    const typename EPI::Stage stage = {staged + (warp - 2) * 32 * EPI::kRowBytes, lane};
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
      w.rows = min(32, at.left - (local - lane));  // (none or less: the warp stores nothing)
      w.n0 = (t / m_tiles) * p.bn;
      w.c0 = c0;
      w.c1 = w.n0 + c1 < p.n ? c1 : (w.n0 + c0 < p.n ? p.n - w.n0 : c0);
      w.slice = 2 * (t / m_tiles) + half;
      const uint32_t lanes = tmem_base + (uint32_t(quarter * 32) << 16);
      auto pre = epi.prepare(w, stage);
      if constexpr (MODE == kWideParts) {
        float acc[kPairMaxCols / 32][16];
#pragma unroll
        for (int x = 0; x < kPairMaxCols / 2; ++x) acc[x >> 4][x & 15] = -0.0f;  // (-0 + y is y, its sign of zero too; a choice between y and the sum cost 3 us of 13 over eight parts)
        for (int seg = 0; seg < segments; ++seg) {
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
              for (int x = 0; x < 32; ++x) acc[i + (x >> 4)][x & 15] += __uint_as_float(v[x >> 4][x & 15]);
            }
          release();
        }
#pragma unroll
        for (int i = 0; i < kPairMaxCols / 32; i += 2)
          if (w.c0 + 16 * i < w.c1) epi.fragment(w, pre, w.c0 + 16 * i, acc[i], acc[i + 1], stage);
        continue;
      }
      mbar_wait(&tail->tmem_full[buf], acc_phase);
      tcgen05_fence_after();
      const uint32_t taddr = lanes + uint32_t(buf * p.bn);
      if constexpr (EPI::kFragments) {  // (the next columns are on their way to registers while these are worked on)
        uint32_t next[2][16];
        auto issue = [&](int c) {
          tmem_ld_x16_issue(taddr + uint32_t(c), next[0]);
          tmem_ld_x16_issue(taddr + uint32_t(c + 16), next[1]);
        };
        if (w.c0 < w.c1) issue(w.c0);
#pragma unroll 1
        for (int c = w.c0; c < w.c1; c += 32) {
          float a[16], b[16];
          tmem_ld_wait();
#pragma unroll
          for (int x = 0; x < 16; ++x) a[x] = __uint_as_float(next[0][x]), b[x] = __uint_as_float(next[1][x]);
          if (c + 32 < w.c1) issue(c + 32);
          epi.fragment(w, pre, c, a, b, stage);
        }
      } else {
        epi(w, pre,
            [&](int ca, float (&a)[16], int cb, float (&b)[16]) {
              uint32_t v[2][16];
              tmem_ld_x16_issue(taddr + uint32_t(ca), v[0]);
              tmem_ld_x16_issue(taddr + uint32_t(cb), v[1]);
              tmem_ld_wait();
#pragma unroll
              for (int x = 0; x < 16; ++x) a[x] = __uint_as_float(v[0][x]), b[x] = __uint_as_float(v[1][x]);
            },
            stage);
      }
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

// 16 columns of bf16(resid + acc), in two chunks (resid, then the sum); returns the sum of squares of the stored values
__device__ __forceinline__ float wide_residual(uint4& ra, uint4& rb, const float (&v)[16]) {
  const uint32_t w[8] = {ra.x, ra.y, ra.z, ra.w, rb.x, rb.y, rb.z, rb.w};
  uint32_t s[8];
  float sq = 0.0f;
#pragma unroll
  for (int j = 0; j < 8; ++j) {
    s[j] = pack_bf16x2(bf16_lo(w[j]) + v[2 * j], bf16_hi(w[j]) + v[2 * j + 1]);
    sq += bf16_lo(s[j]) * bf16_lo(s[j]) + bf16_hi(s[j]) * bf16_hi(s[j]);
  }
  ra = make_uint4(s[0], s[1], s[2], s[3]);
  rb = make_uint4(s[4], s[5], s[6], s[7]);
  return sq;
}

__device__ __forceinline__ uint4 wide_pack8(const float* v) {
  return make_uint4(pack_bf16x2(v[0], v[1]), pack_bf16x2(v[2], v[3]), pack_bf16x2(v[4], v[5]), pack_bf16x2(v[6], v[7]));
}

// Outputs: rows of a multiple of 8 bf16 (32 columns: n is a multiple of 32), 16-byte aligned.
template <int KIND, bool STEP = false>
struct WideEpi {
  static constexpr bool kFragments = KIND == EPI_STORE_BF16 || KIND == EPI_SWIGLU;
  static constexpr int kRowBytes = KIND == EPI_QKV_ROPE ? 192 : 64;  // (EPI_QKV_ROPE: 128 of angles, 64 of outputs)
  typedef WideStage<KIND == EPI_QKV_ROPE ? 128 : 64> Stage;
  static constexpr int kPiece = 32;  // bf16 columns of a staged row
  EpiArgs e;

  struct Pre {
    float rs;                                            // 1 / rms of the row
    int wr, plane;                                       // EPI_QKV_ROPE: its cache row and plane
    uint4 v[KIND == EPI_RESIDUAL ? Stage::kChunks : 1];  // the warp's next residuals
  };

  __device__ __forceinline__ const char* residuals(const WideTile& w, const Stage& st, int c) const {
    return reinterpret_cast<const char*>(e.resid + (long long)(w.row - st.lane) * e.ld_out + w.n0 + c);
  }
  __device__ __forceinline__ const char* angles(const WideTile& w, const Stage& st, int d) const {
    return reinterpret_cast<const char*>(e.rope_cs + (long long)(w.row - st.lane) * (e.d >> 1) + d);
  }

  __device__ __forceinline__ Pre prepare(const WideTile& w, const Stage& st) const {
    Pre p;
    p.rs = 1.0f;
    if constexpr (KIND == EPI_RESIDUAL) {
      st.fetch(min(kPiece, w.c1 - w.c0) / 8, residuals(w, st, w.c0), size_t(e.ld_out) * 2, w.rows, p.v);
    } else {
      if (e.ss_in != nullptr && w.valid) p.rs = STEP ? rows_rstd(e, w.row) : wide_rstd(e, w.row);
    }
    if constexpr (KIND == EPI_QKV_ROPE) {
      p.wr = w.valid ? e.write_row[w.row] : -1;
      p.plane = w.valid ? e.plane[w.row] : 0;
      st.bring(8, angles(w, st, 0), size_t(e.d) * 4, w.rows);
    }
    return p;
  }

  // 32 columns of a row
  __device__ __forceinline__ void fragment(const WideTile& w, const Pre& p, int c, float (&a)[16], float (&b)[16], const Stage& st) const {
    rows_scale16(a, p.rs);
    rows_scale16(b, p.rs);
    const long long row0 = (long long)(w.row - st.lane) * e.ld_out;
    if (KIND == EPI_SWIGLU) {
      float o[16];
      if (STEP) {
        rows_swiglu(e, a, b, o);
      } else {
#pragma unroll
        for (int j = 0; j < 16; ++j) o[j] = __fdividef(a[j], 1.0f + __expf(-a[j])) * b[j];
      }
      const int j = st.template chunk<2>(w, c);
      st.put(j, wide_pack8(o));
      st.put(j + 1, wide_pack8(o + 8));
      st.template done<2>(w, c, e.out + row0 + ((w.n0 + w.c0) >> 1), size_t(e.ld_out) * 2);
    } else {
      const int j = st.template chunk<4>(w, c);
      st.put(j, wide_pack8(a));
      st.put(j + 1, wide_pack8(a + 8));
      st.put(j + 2, wide_pack8(b));
      st.put(j + 3, wide_pack8(b + 8));
      st.template done<4>(w, c, e.out + row0 + w.n0 + w.c0, size_t(e.ld_out) * 2);
    }
  }

  template <class LD>
  __device__ __forceinline__ void operator()(const WideTile& w, Pre& p, LD&& load, const Stage& st) const {
    if constexpr (KIND == EPI_RESIDUAL) {
      const size_t pitch = size_t(e.ld_out) * 2;
      float sq = 0.0f;
      for (int c = w.c0; c < w.c1; c += kPiece) {  // the next ones' residuals are on their way meanwhile
        const int cols = min(kPiece, w.c1 - c);
        st.place(cols / 8, p.v);
        if (c + kPiece < w.c1) st.fetch(min(kPiece, w.c1 - c - kPiece) / 8, residuals(w, st, c + kPiece), pitch, w.rows, p.v);
        __syncwarp();
        for (int q = 0; q < cols; q += 32) {
          float a[16], b[16];
          load(c + q, a, c + q + 16, b);
          const int j = q / 8;
          uint4 x0 = st.get(j), x1 = st.get(j + 1), x2 = st.get(j + 2), x3 = st.get(j + 3);
          sq += wide_residual(x0, x1, a);
          sq += wide_residual(x2, x3, b);
          st.put(j, x0);
          st.put(j + 1, x1);
          st.put(j + 2, x2);
          st.put(j + 3, x3);
        }
        st.flush(cols / 8, e.out + (long long)(w.row - st.lane) * e.ld_out + w.n0 + c, pitch, w.rows);
      }
      if (e.ss_out != nullptr && w.valid) e.ss_out[(long long)w.slice * e.ss_pitch + w.row] = sq;
    } else if constexpr (KIND == EPI_QKV_ROPE) {
      // dims d .. d + 15 of a head's first half and the same of its second half (d + D / 2), of all the warp's heads: rotated queries, appended keys and values
      // (The next angles come by asynchronous copies.  In registers, beside these, 140 bytes of a thread's spilled, and a single wave of narrow tiles, whose epilogue nothing
      // hides, took longer than with angles loaded in place: 495 x 768 x 1472 10.3 us in place, 13.7 in registers, 10.3 so; 389 x 1792 x 1280 10.9, 11.5, 8.8;
      // 4000 rows of it 30.8, 23.5, 20.4.)
      const int D = e.d, half = D >> 1;
      const WideStage<64> outs = {st.buf + 32 * 128, st.lane};
#pragma unroll 1
      for (int d = 0; d < half; d += 16) {
        st.arrived();
        float cs[32];
#pragma unroll
        for (int j = 0; j < 8; ++j) {
          const uint4 x = st.get(j);
          cs[4 * j] = __uint_as_float(x.x), cs[4 * j + 1] = __uint_as_float(x.y), cs[4 * j + 2] = __uint_as_float(x.z), cs[4 * j + 3] = __uint_as_float(x.w);
        }
        __syncwarp();
        if (d + 16 < half) st.bring(8, angles(w, st, d + 16), size_t(D) * 4, w.rows);
#pragma unroll 1
        for (int h = w.c0; h < w.c1; h += D) {
          float a[16], b[16];
          load(h + d, a, h + d + half, b);
          rows_scale16(a, p.rs);
          rows_scale16(b, p.rs);
          const int head = (w.n0 + h) / D;
          if (head < e.hq + e.hkv) {
#pragma unroll
            for (int j = 0; j < 16; ++j) {
              const float x = a[j], y = b[j];
              a[j] = x * cs[2 * j] - y * cs[2 * j + 1];
              b[j] = y * cs[2 * j] + x * cs[2 * j + 1];
            }
          }
          bf16* dst = nullptr;
          if (head < e.hq) {
            if (w.valid) dst = e.q_out + (long long)w.row * (e.hq * D) + head * D + d;
          } else if (p.wr >= 0) {
            const int kvh = (head - e.hq) % e.hkv;
            dst = (head < e.hq + e.hkv ? e.k_cache : e.v_cache) + (((long long)p.plane * e.hkv + kvh) * e.t_alloc + p.wr) * D + d;
          }
          outs.put(0, wide_pack8(a));
          outs.put(1, wide_pack8(a + 8));
          outs.put(2, wide_pack8(b));
          outs.put(3, wide_pack8(b + 8));
          outs.flush_pairs(dst, half);
        }
      }
    }
  }
};

}  // namespace mtx
