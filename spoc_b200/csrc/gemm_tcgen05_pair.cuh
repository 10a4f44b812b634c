// gemm_tcgen05_pair.cuh — the GEMM kernel (tcgen05, cta_group::2 pairs or single blocks).
//
// A persistent, warp-specialised kernel.  With CTAS = 2 two thread blocks on neighbouring SMs form a cluster and compute one
// 256 x BN tile of D together: each block owns 128 rows (its own 128x32 A tile per k-block and its own fp32 accumulator in
// tensor memory) and loads only half of the B tile, the MMA unit reads the other half from the peer's shared memory.  With
// CTAS = 1 a block computes a 128 x BN tile alone, for products of few rows, where the second block of a pair would compute
// nothing.
//
// Roles per block: one lane of warp 0 loads this block's operand tiles with TMA into a ring of shared-memory stages
// (completion counted on the leader's `full` barrier); one lane of warp 1 of the leader block (cluster rank 0) issues the
// MMAs for both blocks and commits to the `empty` and `tmem_full` barriers of both; warps 2-5 run the epilogue on their own
// accumulator rows and hand the accumulator back by arriving on the leader's `tmem_empty` barrier, while the MMA warp
// already works on the next tile in the other accumulator.  On a block's last tile, behind which nothing is left to hide the epilogue,
// warps 6-9 (of pairs' tiles of 128 columns and more) take the right half of the columns, with staging tiles in the operand ring, which is
// idle then.  Passes repeated on the same operands: 2048^3 TF32 27.4 -> 26.3 us, with C, bias and clamp 30.1 -> 27.6, 3xF16 with them 60.3 -> 57.0,
// 1280^3 TF32 14.6 -> 14.2.
// Every TMA load is issued by the block that consumes it (plain per-block loads).
#pragma once
#include <type_traits>

#include "gemm_tcgen05.cuh"

namespace sb200 {

constexpr int PAIR_BM = 256;        // tile rows of a pair (128 per block)
constexpr int PAIR_GROUP_M = 8;     // rasterisation: bands of 8 row tiles
constexpr uint32_t PAIR_A_BYTES = 128 * GEMM_BK * 4;  // this block's A rows: 16 KiB

// Where a kernel's operand tiles come from.
//   SRC_PANELS  prepared K-major panels of the high (and low) parts, A [M x Kp] and B [N x Kp]
//   SRC_DIRECT  the caller's row-major A and B through TFLOAT32 tensor maps (TMA rounds to TF32 on the way in); B arrives as
//               [32 k][32 n] slabs (swizzle 128B with 32-byte atoms) and is consumed through an MN-major descriptor.  The low
//               parts of 3xTF32 come from prepared panels: A [M x Kp], B row-major [K x Np] read as slabs like B itself.
//   SRC_CONVERT, SRC_SPLIT  not this kernel: gemm_convert_kernel and gemm_split_kernel make the parts themselves (gemm_convert.cuh,
//               gemm_split.cuh).
enum { SRC_PANELS = 0, SRC_DIRECT = 1, SRC_CONVERT = 2, SRC_SPLIT = 3 };

template <int MODE, int SRC, int BN, int CTAS>
struct TileCfg {
  static_assert(BN == 256 || BN == 192 || BN == 128 || BN == 64, "tile columns");
  static_assert(CTAS == 2 || BN <= 128, "single blocks work on narrow tiles");
  static constexpr int kOperands = (MODE == 3 || MODE == 4 || MODE == 5) ? 2 : 1;  // high parts (+ low parts)
  static constexpr uint32_t kBBytes = (BN / CTAS) * GEMM_BK * 4;                   // this block's part of B (rows of 128 bytes)
  static constexpr uint32_t kStageBytes = kOperands * (PAIR_A_BYTES + kBBytes);
  static constexpr int kStagesFit = (192 * 1024) / kStageBytes;
  static constexpr int kStages = kStagesFit > 8 ? 8 : kStagesFit;  // pairs, 256/192/128/64 columns: 6/6/8/8, 3xTF32 3/3/4/4
  static constexpr uint32_t kSmemBytes = kStages * kStageBytes + GEMM_EPI_BUF_BYTES + GEMM_CTRL_BYTES + 1024;
  // Groups of four epilogue warps.  A half of 64 columns is not worth a second one, and blocks on their own nearly always divide their k-loop, whose
  // finish lost by the fewer registers a thread (64 x 4096 x 4096 TF32 13.1 and 13.4 us).
  static constexpr int kEpiGroups = BN >= 128 && CTAS == 2 ? 2 : 1;
  // Arrivals that hand an accumulator back: the epilogue warps of both blocks, the second group's among them.  That group has nothing to do with
  // a tile that is not the last, but waits for each accumulator in turn, and a wait on a barrier's parity takes the phase after the wanted one
  // for one still to come: no accumulator may be completed again before all warps have seen it complete.  (Nobody waits for these
  // arrivals where the k-loop is divided within a cluster, whose blocks have one tile and no second group.)
  static constexpr int kHandBacks = 4 * kEpiGroups * CTAS;
  static constexpr int kThreads = GEMM_THREADS + (kEpiGroups - 1) * 128;  // (GEMM_THREADS where the k-loop is divided within a cluster)
};

constexpr int REDUCE_THREADS = 64;     // gemm_reduce_kernel: small blocks, so that small results are spread over the SMs
constexpr int PAIR_EPOCH_RING = 64;    // epoch counters (a pair far ahead wraps onto an old counter: harmless, a hint)

// Count this pair into epoch e and wait, for wait_ns at most, until all `pairs` pairs of the launch have reached it.
__device__ __forceinline__ void pair_soft_epoch(unsigned int* ctr, unsigned int e, unsigned int pairs, uint64_t wait_ns) {
  unsigned int* slot = ctr + (e % PAIR_EPOCH_RING);
  const unsigned int target = pairs * (e / PAIR_EPOCH_RING + 1);
  atomicAdd(slot, 1u);
  const uint64_t t0 = global_timer_ns();
  while (*reinterpret_cast<volatile unsigned int*>(slot) < target && global_timer_ns() - t0 < wait_ns) {
  }
}

// Which part of a divided k-loop work item `item` is: item / num_tiles, without the division where it is 0.
__device__ __forceinline__ int item_split(int item, int num_tiles) {
  return item < num_tiles ? 0 : static_cast<int>(static_cast<unsigned int>(item) / static_cast<unsigned int>(num_tiles));
}
// The tile of work item `item`, in bands of group_m row tiles.  A division takes about 150 cycles, and every role of a block passes through
// here before its first load: a product of one band, or whose k-loop is undivided, does with one.
__device__ __forceinline__ void item_tile_coords(int item, const GemmParams& p, int num_tiles, int& tm, int& tn) {
  const unsigned int tile = item - item_split(item, num_tiles) * num_tiles, tiles_m = p.tiles_m, group_m = p.group_m;
  if (tiles_m <= group_m) {
    tn = tile / tiles_m;
    tm = tile - tn * tiles_m;
    return;
  }
  const unsigned int band_tiles = group_m * p.tiles_n;
  const unsigned int band = tile / band_tiles;
  const unsigned int within = tile - band * band_tiles;
  const unsigned int first_m = band * group_m;
  const unsigned int band_m = min(group_m, tiles_m - first_m);
  tn = within / band_m;
  tm = first_m + within - tn * band_m;
}

// Four columns of a row of D = act(alpha*sum + beta*C + bias): the operations of the other epilogues in the same order.  VEC: 128-bit
// accesses (p.vec_epilogue).  Columns from N on are left out.
struct QuadColumns {  // what the rows of a column quad share
  float bias[4], scale[4];
};
__device__ __forceinline__ QuadColumns quad_columns(const GemmParams& p, int col) {
  QuadColumns q;
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    const bool in = col + j < p.N;
    q.bias[j] = in && p.bias ? p.bias[col + j] : 0.0f;
    q.scale[j] = in && p.col_scale ? p.col_scale[col + j] : 1.0f;
  }
  return q;
}
template <bool VEC>
__device__ __forceinline__ float4 quad_of_c(const GemmParams& p, long long row, int col) {
  float4 c = make_float4(0.f, 0.f, 0.f, 0.f);
  if (!p.C || col >= p.N) return c;
  const float* src = p.C + row * p.ldc + col;
  if (VEC) return *reinterpret_cast<const float4*>(src);
  c.x = src[0];
  if (col + 1 < p.N) c.y = src[1];
  if (col + 2 < p.N) c.z = src[2];
  if (col + 3 < p.N) c.w = src[3];
  return c;
}
template <bool VEC>
__device__ __forceinline__ void finish_quad(const GemmParams& p, long long row, int col, const float4& sum, const float4& c4,
                                            const QuadColumns& q) {
  float x[4] = {sum.x, sum.y, sum.z, sum.w};
  const float c[4] = {c4.x, c4.y, c4.z, c4.w};
  if (p.row_scale) {
    const float rs = p.row_scale[row];
#pragma unroll
    for (int j = 0; j < 4; ++j) x[j] = (x[j] * rs) * q.scale[j];
  }
#pragma unroll
  for (int j = 0; j < 4; ++j) x[j] = __fmul_rn(p.alpha, x[j]);
  if (p.C) {
#pragma unroll
    for (int j = 0; j < 4; ++j) x[j] = fmaf(p.beta, c[j], x[j]);
  }
#pragma unroll
  for (int j = 0; j < 4; ++j) x[j] = __fadd_rn(x[j], q.bias[j]);
  if (p.act == 1) {
#pragma unroll
    for (int j = 0; j < 4; ++j) x[j] = (x[j] > 0.0f) ? x[j] : 0.0f;
  }
  const long long off = row * p.ldd + col;
  if (VEC) {
    *reinterpret_cast<float4*>(p.D + off) = make_float4(x[0], x[1], x[2], x[3]);
    for (int r = 0; r < p.n_replicas; ++r) *reinterpret_cast<float4*>(p.replicas[r] + off) = make_float4(x[0], x[1], x[2], x[3]);
  } else {
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      if (col + j >= p.N) break;
      p.D[off + j] = x[j];
      if (p.n_replicas) store_replicas(p, off + j, x[j]);
    }
  }
}
__device__ __forceinline__ void add_to(float4& s, const float4& v) {
  s.x += v.x;
  s.y += v.y;
  s.z += v.z;
  s.w += v.w;
}

// A k-loop divided among the blocks (pairs) of one cluster (p.cluster_splits > 1).  Each block leaves the partial sums of its 128 rows
// and BN columns in its operand ring, which is idle once the accumulator is complete, and sends every other block the rows that one
// finishes, with a bulk copy per block; what arrives is added up from the block's own shared memory, in order of k.  Block `share` of
// `splits` finishes rows [rows * share / splits, rows * (share + 1) / splits).  In order: cluster_arrive_relaxed once the ring is idle,
// cluster_part_store, and cluster_exchange: a barrier of the block, cluster_wait (all rings are idle), the copies, the wait for `recv`, and
// the share of this block.
// Bound by the way between the blocks, about 13 bytes a cycle and SM (32 KB 1600 to 2400 cycles), and by what runs once in a launch and
// so comes from a cold instruction cache.  It replaced 128-bit loads from the peers' shared memory behind a cluster barrier with a release:
// 512 x 512 x 2048 TF32 11.0 -> 9.2 us, 128 x 4096 x 4096 TF32 16.2 -> 15.8, 64 x 1024 x 1024 3xTF32 8.6 -> 8.3, 200 x 300 x 900 9.2 -> 8.6.
template <int BN>
struct ClusterPart {
  static constexpr uint32_t kRowBytes = BN * 4;  // quad q of row r lies at quad q ^ (r & 7): no bank conflicts with a lane a row
  // the partial sums, and (splits - 1) * ceil(rows / splits) rows that arrive: at most 114 with seven blocks, 96 with four pairs
  __host__ __device__ static constexpr uint32_t bytes(int ctas) { return (128 + (ctas == 2 ? 96 : 114)) * kRowBytes; }
};
// rows * share / splits, for at most 128 rows and eight splits: an integer division would take 150 cycles
__device__ __forceinline__ int share_row(int rows, int share, int splits) {
  return static_cast<int>(__fdividef(static_cast<float>(rows * share) + 0.5f, static_cast<float>(splits)));
}

// One warp's 32 rows (tensor-memory lanes from `row` of the block's 128) and `cols` columns from `col` on, for the copies to read.
template <int BN>
__device__ __forceinline__ void cluster_part_store(uint8_t* part, uint32_t taddr, int row, int col, int cols) {
#pragma unroll 1
  for (int c = 0; c < cols; c += 32) {
    uint32_t r[32];
    tmem_ld_32x32b_x32(taddr + c, r);
    tmem_ld_wait_x32(r);
    uint8_t* dst = part + row * ClusterPart<BN>::kRowBytes + (col + c) * 4;
#pragma unroll
    for (int j = 0; j < 8; ++j) *reinterpret_cast<uint4*>(dst + ((j ^ (row & 7)) << 4)) = make_uint4(r[4 * j], r[4 * j + 1], r[4 * j + 2], r[4 * j + 3]);
  }
  fence_async_shared();
}
// One warp, a lane a peer.  recv: the barrier of this block, at the same place in all, on which what arrives is counted.
template <int BN, int CTAS>
struct ClusterPush {
  uint32_t dst, src, bytes, bar, expected;
  // what is sent, and where to: before the others' rings are known to be idle
  __device__ __forceinline__ void prepare(const uint8_t* part, uint64_t* recv, int rows, int share, int rank, int splits, int lane) {
    constexpr uint32_t ROW = ClusterPart<BN>::kRowBytes;
    const int slot_rows = share_row(rows + splits - 1, 1, splits);
    const int to = share + 1 + lane < splits ? share + 1 + lane : share + 1 + lane - splits;  // of lane < splits - 1
    const int first = share_row(rows, to, splits), slot = share < to ? share : share - 1;
    bytes = lane < splits - 1 ? (share_row(rows, to + 1, splits) - first) * ROW : 0;
    expected = (splits - 1) * (share_row(rows, share + 1, splits) - share_row(rows, share, splits)) * ROW;
    src = smem_u32(part) + first * ROW;
    dst = map_to_cta(smem_u32(part) + (128 + slot * slot_rows) * ROW, (bytes ? to : share) * CTAS + rank);
    bar = map_to_cta(smem_u32(recv), (bytes ? to : share) * CTAS + rank);
  }
  __device__ __forceinline__ void send(uint64_t* recv, int lane) const {
    if (lane == 0) mbar_arrive_expect_tx(smem_u32(recv), expected);
    if (bytes) bulk_copy_to_cta(dst, src, bytes, bar);
    __syncwarp();
  }
};
// THREADS threads.  row0, n0: the first row and column of the block's part of the tile.  begin: what does not wait for the others.
// The rows of a batch go through every operation together, so that what a launch has or has not (C, scales, a clamp, replicas) is asked
// once a batch: asked for every quad it was 120 instructions a quad and 3100 of the 7500 cycles behind the k-loop (64 rows of 128 columns).
template <int BN, int THREADS, bool VEC>
struct ClusterFinish {
  static constexpr int QUADS = BN / 4, STEP = THREADS / QUADS;
  static constexpr int BATCH = STEP % 2 == 0 ? 4 : 8;  // rows a thread has in flight
  static_assert(THREADS % QUADS == 0, "a thread stays in its column quad");
  static_assert(BATCH * STEP % 8 == 0, "the swizzle of a thread's rows is the same in every batch");
  static constexpr uint32_t ROW = ClusterPart<BN>::kRowBytes;
  int first, row, left, col;  // left: rows of this thread
  uint32_t slot_bytes;
  QuadColumns columns;
  float4 c[BATCH];

  __device__ __forceinline__ void load_c(const GemmParams& p, int row0, int from, int have) {
#pragma unroll
    for (int u = 0; u < BATCH; ++u)
      if (u < have) c[u] = quad_of_c<VEC>(p, row0 + first + from + u * STEP, col);
  }
  __device__ __forceinline__ void begin(const GemmParams& p, int share, int rows, int row0, int n0, int tid) {
    const int splits = p.cluster_splits;
    row = tid / QUADS;
    col = n0 + tid % QUADS * 4;
    first = share_row(rows, share, splits);
    const int count = share_row(rows, share + 1, splits) - first;
    left = col < p.N && row < count ? (count - row + STEP - 1) / STEP : 0;
    slot_bytes = share_row(rows + splits - 1, 1, splits) * ROW;
    columns = quad_columns(p, col);
    if (p.C) load_c(p, row0, row, left);
  }
  __device__ __forceinline__ void run(const GemmParams& p, const uint8_t* part, int share, int row0, int tid) {
    uint32_t at[BATCH];  // of the batch's rows, from the first row of the share on
#pragma unroll
    for (int u = 0; u < BATCH; ++u) at[u] = (row + u * STEP) * ROW + ((tid % QUADS ^ ((first + row + u * STEP) & 7)) << 4);
    float* dp = p.D + static_cast<long long>(row0 + first + row) * p.ldd + col;
    for (; left > 0; left -= BATCH, row += BATCH * STEP) {
      float x[BATCH][4];
      const uint8_t* theirs = part + 128 * ROW;
      for (int k = 0; k < p.cluster_splits; ++k) {
        const uint8_t* from = k == share ? part + first * ROW : theirs;
        theirs += k == share ? 0 : slot_bytes;
#pragma unroll
        for (int u = 0; u < BATCH; ++u) {
          if (u >= left) break;
          const float4 v = *reinterpret_cast<const float4*>(from + at[u]);
          if (k == 0) {
            *reinterpret_cast<float4*>(x[u]) = v;
          } else {
            x[u][0] += v.x;
            x[u][1] += v.y;
            x[u][2] += v.z;
            x[u][3] += v.w;
          }
        }
      }
      if (p.row_scale) {
#pragma unroll
        for (int u = 0; u < BATCH; ++u) {
          const float rs = u < left ? p.row_scale[row0 + first + row + u * STEP] : 1.0f;
#pragma unroll
          for (int j = 0; j < 4; ++j) x[u][j] = (x[u][j] * rs) * columns.scale[j];
        }
      }
#pragma unroll
      for (int u = 0; u < BATCH; ++u)
#pragma unroll
        for (int j = 0; j < 4; ++j) x[u][j] = __fmul_rn(p.alpha, x[u][j]);
      if (p.C) {
#pragma unroll
        for (int u = 0; u < BATCH; ++u) {
          x[u][0] = fmaf(p.beta, c[u].x, x[u][0]);
          x[u][1] = fmaf(p.beta, c[u].y, x[u][1]);
          x[u][2] = fmaf(p.beta, c[u].z, x[u][2]);
          x[u][3] = fmaf(p.beta, c[u].w, x[u][3]);
        }
        load_c(p, row0, row + BATCH * STEP, left - BATCH);
      }
#pragma unroll
      for (int u = 0; u < BATCH; ++u)
#pragma unroll
        for (int j = 0; j < 4; ++j) x[u][j] = __fadd_rn(x[u][j], columns.bias[j]);
      if (p.act == 1) {
#pragma unroll
        for (int u = 0; u < BATCH; ++u)
#pragma unroll
          for (int j = 0; j < 4; ++j) x[u][j] = (x[u][j] > 0.0f) ? x[u][j] : 0.0f;
      }
#pragma unroll
      for (int u = 0; u < BATCH; ++u) {
        if (u >= left) break;
        if (VEC) {
          *reinterpret_cast<float4*>(dp + u * STEP * p.ldd) = *reinterpret_cast<const float4*>(x[u]);
        } else {
#pragma unroll
          for (int j = 0; j < 4; ++j)
            if (col + j < p.N) dp[u * STEP * p.ldd + j] = x[u][j];
        }
      }
      if (p.n_replicas) {
#pragma unroll
        for (int u = 0; u < BATCH; ++u) {
          if (u >= left) break;
#pragma unroll
          for (int j = 0; j < 4; ++j)
            if (col + j < p.N) store_replicas(p, dp + u * STEP * p.ldd + j - p.D, x[u][j]);
        }
      }
      dp += BATCH * STEP * p.ldd;
#pragma unroll
      for (int u = 0; u < BATCH; ++u) at[u] += BATCH * STEP * ROW;
    }
  }
};
// A block's part in the exchange behind cluster_part_store: all THREADS threads, `ok` whether all went well so far; false when the others'
// sums did not arrive in time.  SENDER: the warp that sends.
template <int BN, int CTAS, int THREADS, int SENDER, bool VEC, class Barrier>
__device__ __forceinline__ bool cluster_exchange(const GemmParams& p, const uint8_t* part, uint64_t* recv, int share, int rank, int row0, int n0, bool ok,
                                                 volatile int* abort_flag, Barrier&& barrier) {
  const int rows = max(0, min(128, p.M - row0)), lane = threadIdx.x & 31;
  ClusterPush<BN, CTAS> push;
  if (threadIdx.x / 32 == SENDER) push.prepare(part, recv, rows, share, rank, p.cluster_splits, lane);
  ok = barrier(ok);
  cluster_wait();
  if (!ok) return false;
  if (threadIdx.x / 32 == SENDER) push.send(recv, lane);
  ClusterFinish<BN, THREADS, VEC> finish;
  finish.begin(p, share, rows, row0, n0, threadIdx.x);
  if (!mbar_wait_bounded(smem_u32(recv), 0, abort_flag)) return false;
  finish.run(p, part, share, row0, threadIdx.x);
  return true;
}

// MODE 1: TF32, one MMA per k-step.  MODE 3: 3xTF32, lo*hi + hi*lo + hi*hi per k-step into one accumulator (the lo*lo term,
// 2^-22 relative, is dropped).  MODE 4: the same three-term split on fp16 panels (kind::f16): a 128-byte operand row holds 64
// halves instead of 32 floats, so a k-block spans 64 k and a k-step 16, in the same bytes, descriptors and cycles as the TF32
// forms.  MODE 2: fp16 panels, one MMA.
// map_a_x, map_b_x, but for the mixed mode: the high and low parts of A once more, for the last, partial 128 rows, with boxes of p.a_tail_rows.
// TMA takes 3 ns for a row past the end when a few blocks ask for such rows and 15 ns when all do, so that few rows went slower than 128.  Passes
// repeated on the same operands: TF32 10 x 6144 x 1024 30.0 -> 9.0 us, 64 x 4096 x 4096 with epilogue 17.0 -> 13.1 (16.4 with operands that come
// from HBM).  The accumulator's rows that nothing was loaded for come of whatever the ring held, and are not stored.
// MODE 5 (mixed; always SRC_DIRECT): map_a_hi / map_b_hi are TFLOAT32 maps over the caller's matrices, map_a_lo / map_b_lo lie
// over the fp16 panels of the high parts and map_a_x / map_b_x over those of the low parts (all K-major, [rows x Kp], Kp a
// multiple of 64).  A tile is computed in three runs of stages, every stage the same bytes: K/64 cross stages (the four fp16
// tiles of 64 k: lo*hi + hi*lo, eight fp16 MMAs), then the rescale stages (tiles from beyond the end of K, which TMA fills
// with zeros: one MMA each whose only effect is the scaling of the accumulator by 2^-15), then K/64 main stages (A and B of
// two consecutive k-blocks of 32 where the other modes keep high and low parts: eight TF32 MMAs, the first of which scales
// the accumulator by 2^-first_scale).
//
// p.splits > 1: the k-blocks of a tile are divided among `splits` work items, each of which stores its partial sums to rows
// [s * p.part_rows, ...) of a partial matrix (map_d); gemm_reduce_kernel adds them up in order and runs the epilogue.  With
// p.cluster_splits > 1 the items of a tile are the pairs of one cluster instead, one tile per cluster, and the sums stay on chip.
template <int MODE, int SRC, int BN, int CTAS>
__global__ void __launch_bounds__(TileCfg<MODE, SRC, BN, CTAS>::kThreads, 1)
gemm_pair_kernel(const __grid_constant__ CUtensorMap map_a_hi, const __grid_constant__ CUtensorMap map_b_hi,
                 const __grid_constant__ CUtensorMap map_a_lo, const __grid_constant__ CUtensorMap map_b_lo,
                 const __grid_constant__ CUtensorMap map_a_x, const __grid_constant__ CUtensorMap map_b_x,
                 const __grid_constant__ CUtensorMap map_d, const __grid_constant__ CUtensorMap map_c, const GemmParams p) {
  using Cfg = TileCfg<MODE, SRC, BN, CTAS>;
  constexpr bool MIXED = MODE == 5;
  constexpr bool THREE = MODE == 3 || MODE == 4;
  constexpr bool F16 = MODE == 4 || MODE == 2;
  constexpr bool DIRECT = SRC != SRC_PANELS;
  static_assert(!MIXED || SRC == SRC_DIRECT, "the mixed mode reads the main term's operands where they lie");
  static_assert(!(F16 && DIRECT), "fp16 panels are always prepared");
  constexpr int BK_ELEMS = F16 ? 2 * GEMM_BK : GEMM_BK;  // elements of K per k-block
  constexpr int STAGES = Cfg::kStages;
  constexpr uint32_t B_BYTES = Cfg::kBBytes;
  constexpr int PART_N = BN / CTAS;     // columns of B this block loads
  constexpr int SLABS = PART_N / 32;    // [32 k][32 n] slabs per stage in the direct layout
  constexpr int BM = 128 * CTAS;
  extern __shared__ uint8_t smem_raw[];
  // 1024-byte alignment is what the 128-byte swizzle pattern is anchored to
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  uint8_t* stage_base = smem;
  uint8_t* epi_base = smem + STAGES * Cfg::kStageBytes;
  uint8_t* ctrl = epi_base + GEMM_EPI_BUF_BYTES;
  uint64_t* bars = reinterpret_cast<uint64_t*>(ctrl);
  uint64_t* full_bar = bars;                         // used in the leader only
  uint64_t* empty_bar = bars + STAGES;               // one set per block
  uint64_t* tmem_full_bar = bars + 2 * STAGES;       // one set per block
  uint64_t* tmem_empty_bar = bars + 2 * STAGES + 2;  // used in the leader only
  uint64_t* recv = bars + 2 * STAGES + 4;            // in_cluster: the others' partial sums
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + 2 * STAGES + 5);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);
  static_assert((2 * STAGES + 6) * 8 <= GEMM_CTRL_CBAR, "the barriers fit the control area");

  const int warp = threadIdx.x >> 5;
  const int lane = threadIdx.x & 31;
  const bool in_cluster = MODE != 5 && p.cluster_splits > 1;
  const uint32_t cta = CTAS == 2 || in_cluster ? cluster_ctarank() : 0u;
  // Rank 0 is the leader of its pair.  From the block's index and not from its rank in the cluster, which is the same: so the compiler sees that
  // what depends on it is the same in all threads, and keeps descriptors in uniform registers behind branches on it.
  const uint32_t rank = blockIdx.x & (CTAS - 1u), leader = cta - rank;
  // in_cluster: item `split * num_tiles + tile` is this pair's only one
  const int split_rank = in_cluster ? static_cast<int>(cta) / CTAS : 0;
  const int pair_id = in_cluster ? static_cast<int>(blockIdx.x) / (CTAS * p.cluster_splits) + split_rank * p.tiles_m * p.tiles_n
                                 : static_cast<int>(blockIdx.x) / CTAS;
  const int num_pairs = in_cluster ? 1 << 30 : static_cast<int>(gridDim.x) / CTAS;

  if (warp == 0) {  // a lane a barrier: full and empty, tmem_full, tmem_empty, recv
    constexpr int BARS = 2 * STAGES + 5;
    static_assert(BARS <= 32, "a lane a barrier");
    if (lane < BARS) mbar_init(smem_u32(&bars[lane]), lane / 2 == STAGES + 1 ? Cfg::kHandBacks : 1);
    if (lane == 0) *abort_flag = 0;
    mbar_fence_init();
  }
  if (warp == 2) {  // the barriers of the tiles of C
    if (lane < 8 * Cfg::kEpiGroups) mbar_init(smem_u32(reinterpret_cast<uint64_t*>(ctrl + GEMM_CTRL_CBAR) + lane), 1);
    mbar_fence_init();
  }
  if (threadIdx.x == 96) {
    tma_prefetch_desc(&map_a_hi);
    tma_prefetch_desc(&map_b_hi);
    if (THREE || MIXED) {
      tma_prefetch_desc(&map_a_lo);
      tma_prefetch_desc(&map_b_lo);
    }
    tma_prefetch_desc(&map_a_x);
    if (THREE || MIXED) tma_prefetch_desc(&map_b_x);
    if (p.tma_epilogue) tma_prefetch_desc(&map_d);
  }
  if (warp == 1) {
    tmem_alloc_for<CTAS>(smem_u32(tmem_slot), GEMM_TMEM_COLS);
    tmem_relinquish_for<CTAS>();
    tc_fence_before_sync();
  }
  __syncthreads();
  if (CTAS == 2) {
    // the blocks' barriers exist before any signal crosses between them
    cluster_arrive_relaxed();
    cluster_wait();
  }
  tc_fence_after_sync();
  const uint32_t tmem_base = *tmem_slot;
  // Everything above touched no global memory, so it may overlap the tail of the kernel before this one in the stream; from
  // here on its results are needed.  The kernel behind this one may set itself up in the same way from now on.
  grid_launch_dependents();
  grid_dependency_wait();
  // a gated kernel whose gate is closed has no tiles: every role falls through to the common exit
  const bool gate_open = !p.gate || *p.gate == p.gate_value;
  const int num_tiles = gate_open ? p.tiles_m * p.tiles_n : 0;
  const int num_items = num_tiles * p.splits;
  int mix_rescale = 0, mix_first = 0;
  if (MIXED && gate_open) {
    const MixCtl* ctl = reinterpret_cast<const MixCtl*>(p.mix_ctl);
    mix_rescale = ctl->rescale_stages;
    mix_first = ctl->first_scale;
  }
  // stages of work item `item`: its k-blocks [k0, k0 + stages); in mixed mode (never divided) the cross stages, the rescale
  // stages, the main stages
  auto item_stages = [&](int item, int& k0) {
    k0 = item_split(item, num_tiles) * p.split_k_blocks;
    return MIXED ? 2 * p.num_k_blocks + mix_rescale : min(p.num_k_blocks - k0, p.split_k_blocks);
  };

  bool ok = true, arrived = false;
  if (warp == 0) {
    // ------------------------------------------------------ TMA producer
    if (elect_one()) {
      int stage = 0;
      uint32_t phase = 0;
      const uint64_t pol_a = l2_policy(p.l2_policy & 3), pol_b = l2_policy((p.l2_policy >> 2) & 3);
      const bool lockstep = p.epoch_ctr != nullptr && rank == 0;
      const int epoch_stages = p.epoch_stages > 0 ? p.epoch_stages : 64;
      int k_first;
      const int epochs_per_tile = lockstep && num_items > 0 ? (item_stages(0, k_first) + epoch_stages - 1) / epoch_stages : 0;
      int my_tiles = 0;
      for (int item = pair_id; item < num_items && ok; item += num_pairs, ++my_tiles) {
        int tm, tn, k0;
        item_tile_coords(item, p, num_tiles, tm, tn);
        const int stages = item_stages(item, k0);
        const int m0 = tm * BM + static_cast<int>(rank) * 128;     // this block's rows of A
        const int n0 = tn * BN + static_cast<int>(rank) * PART_N;  // this block's part of B's columns
        // the map of these rows is chosen here, so that the loads are the same straight line for every tile: behind branches on what lies
        // past the end each took 100 cycles more (8192^3 TF32 1370 -> 1600 us)
        auto rows_of_a = [&](int m) { return MIXED || m + 128 <= p.M ? 128 : p.a_tail_rows; };
        const CUtensorMap* const pa_hi = rows_of_a(m0) == 128 ? &map_a_hi : &map_a_x;
        const CUtensorMap* const pa_lo = rows_of_a(m0) == 128 ? &map_a_lo : &map_b_x;
        int stage_bytes = 0;  // of both blocks
        for (int r = 0; r < CTAS; ++r) stage_bytes += Cfg::kOperands * (rows_of_a(tm * BM + r * 128) * 128 + static_cast<int>(B_BYTES));
        for (int it = 0; it < stages; ++it) {
          const int kb = MIXED ? (it < p.num_k_blocks + mix_rescale ? it : it - p.num_k_blocks - mix_rescale) : k0 + it;
          if (lockstep && (it % epoch_stages) == 0)
            pair_soft_epoch(p.epoch_ctr, static_cast<unsigned int>(my_tiles * epochs_per_tile + it / epoch_stages),
                            static_cast<unsigned int>(num_pairs), static_cast<uint64_t>(p.epoch_wait_ns));
          if (!mbar_wait_bounded(smem_u32(&empty_bar[stage]), phase ^ 1u, abort_flag)) {
            atomicCAS(p.status, 0, 0x1100 | (rank << 4) | stage);
            ok = false;
            break;
          }
          // the leader arms its barrier with the bytes of both blocks
          if (rank == 0) mbar_arrive_expect_tx(smem_u32(&full_bar[stage]), stage_bytes);
          const uint32_t bar = CTAS == 2 ? map_to_cta(smem_u32(&full_bar[stage]), leader) : smem_u32(&full_bar[stage]);
          uint8_t* sp = stage_base + stage * Cfg::kStageBytes;
          auto load = [&](uint8_t* dst, const CUtensorMap& map, int x, int y, uint64_t pol) {
            tma_load_for<CTAS>(smem_u32(dst), &map, bar, x, y, pol);
          };
          if (MIXED) {
            if (it < p.num_k_blocks + mix_rescale) {
              // cross stage: 64 k of the four fp16 panels; a rescale stage asks for k-blocks past the end: zeros
              load(sp, map_a_lo, kb * 64, m0, pol_a);
              load(sp + PAIR_A_BYTES, map_b_lo, kb * 64, n0, pol_b);
              load(sp + PAIR_A_BYTES + B_BYTES, map_a_x, kb * 64, m0, pol_a);
              load(sp + 2 * PAIR_A_BYTES + B_BYTES, map_b_x, kb * 64, n0, pol_b);
            } else {
              // main stage: two consecutive k-blocks of 32 of the caller's A and B
#pragma unroll
              for (int h = 0; h < 2; ++h) {
                uint8_t* hp = sp + h * (PAIR_A_BYTES + B_BYTES);
                load(hp, map_a_hi, kb * 64 + 32 * h, m0, pol_a);
#pragma unroll
                for (int sl = 0; sl < SLABS; ++sl) load(hp + PAIR_A_BYTES + sl * 4096, map_b_hi, n0 + 32 * sl, kb * 64 + 32 * h, pol_b);
              }
            }
          } else {
            auto load_b = [&](uint8_t* dst, const CUtensorMap& map) {
              if (DIRECT) {
                // B is K x N row-major: x = column, y = k; slabs of 32 columns cover this block's part
#pragma unroll
                for (int sl = 0; sl < SLABS; ++sl) load(dst + sl * 4096, map, n0 + 32 * sl, kb * BK_ELEMS, pol_b);
              } else {
                load(dst, map, kb * BK_ELEMS, n0, pol_b);
              }
            };
            load(sp, *pa_hi, kb * BK_ELEMS, m0, pol_a);
            load_b(sp + PAIR_A_BYTES, map_b_hi);
            if (THREE) {
              load(sp + PAIR_A_BYTES + B_BYTES, *pa_lo, kb * BK_ELEMS, m0, pol_a);
              load_b(sp + 2 * PAIR_A_BYTES + B_BYTES, map_b_lo);
            }
          }
          if (++stage == STAGES) {
            stage = 0;
            phase ^= 1u;
          }
        }
      }
      if (lockstep) {
        // a pair with fewer tiles than the others counts itself into the epochs it will not reach
        const int most_tiles = (num_tiles + num_pairs - 1) / num_pairs;
        for (int e = my_tiles * epochs_per_tile; e < most_tiles * epochs_per_tile; ++e)
          atomicAdd(p.epoch_ctr + (e % PAIR_EPOCH_RING), 1u);
      }
      if (!ok) wait_for_copies();  // operand tiles: a load that was issued completes regardless of its consumer
    }
    __syncwarp();
  } else if (warp == 1) {
    // ------------------------------------------- MMA issuer (leader block)
    if (rank == 0 && elect_one()) {
      constexpr uint32_t idesc = F16 ? umma_idesc_f16(BM, BN) : umma_idesc_tf32(BM, BN, DIRECT);
      int stage = 0;
      uint32_t phase = 0;
      int local_tile = 0;
      for (int item = pair_id; item < num_items && ok; item += num_pairs, ++local_tile) {
        const int acc = local_tile & 1;
        const uint32_t acc_phase = (local_tile >> 1) & 1;
        int k0;
        const int stages = item_stages(item, k0);
        const uint32_t acc_free = smem_u32(&tmem_empty_bar[acc]);
        if (!(CTAS == 2 ? mbar_wait_cluster(acc_free, acc_phase ^ 1u, abort_flag) : mbar_wait_bounded(acc_free, acc_phase ^ 1u, abort_flag))) {
          atomicCAS(p.status, 0, 0x1200 | acc);
          ok = false;
          break;
        }
        tc_fence_after_sync();
        const uint32_t tmem_d = tmem_base + acc * 256;
        for (int kb = 0; kb < stages; ++kb) {
          if (!mbar_wait_bounded(smem_u32(&full_bar[stage]), phase, abort_flag)) {
            atomicCAS(p.status, 0, 0x1300 | stage);
            ok = false;
            break;
          }
          tc_fence_after_sync();
          const uint32_t sa_hi = smem_u32(stage_base + stage * Cfg::kStageBytes);
          const uint32_t sb_hi = sa_hi + PAIR_A_BYTES;
          const uint32_t sa_lo = sb_hi + B_BYTES;
          const uint32_t sb_lo = sa_lo + PAIR_A_BYTES;
          if constexpr (MIXED) {
            constexpr uint32_t idesc16 = umma_idesc_f16(BM, BN);
            if (kb < p.num_k_blocks) {
              // cross terms of 64 k: lo(a)*hi(b) + hi(a)*lo(b), four k-steps of 16
#pragma unroll
              for (int k = 0; k < 4; ++k) {
                const uint32_t koff = k * 32;
                umma_f16_pair(tmem_d, umma_desc_k_sw128(sa_lo + koff), umma_desc_k_sw128(sb_hi + koff), idesc16, (kb | k) ? 1u : 0u);
                umma_f16_pair(tmem_d, umma_desc_k_sw128(sa_hi + koff), umma_desc_k_sw128(sb_lo + koff), idesc16, 1u);
              }
            } else if (kb < p.num_k_blocks + mix_rescale) {
              // zero tiles: the product adds nothing, the accumulator is scaled by 2^-15
              umma_f16_pair_scaled(tmem_d, umma_desc_k_sw128(sa_hi), umma_desc_k_sw128(sb_hi), idesc16, 15);
            } else {
              const bool first = kb == p.num_k_blocks + mix_rescale;
#pragma unroll
              for (int h = 0; h < 2; ++h) {
                const uint32_t sa = h ? sa_lo : sa_hi, sb = h ? sb_lo : sb_hi;
#pragma unroll
                for (int k = 0; k < 4; ++k) {
                  const uint64_t da = umma_desc_k_sw128(sa + k * 32);
                  const uint64_t db = umma_desc_mn_sw128_32b(sb + k * 1024, 4096);
                  if (first && h == 0 && k == 0)
                    umma_tf32_pair_scaled(tmem_d, da, db, idesc, mix_first);
                  else
                    umma_for<false, CTAS>(tmem_d, da, db, idesc, 1u);
                }
              }
            }
          } else {
#pragma unroll
            for (int k = 0; k < GEMM_BK / GEMM_UMMA_K; ++k) {
              const uint32_t koff = k * GEMM_UMMA_K * 4;  // 32 bytes along K inside the swizzle row
              const uint64_t da_hi = umma_desc_k_sw128(sa_hi + koff);
              // MN-major B: k-step k is the k-th 8-row group (1024 bytes) of every slab
              const uint64_t db_hi = DIRECT ? umma_desc_mn_sw128_32b(sb_hi + k * 1024, 4096) : umma_desc_k_sw128(sb_hi + koff);
              const uint32_t accumulate = (kb | k) ? 1u : 0u;
              if (THREE) {
                const uint64_t da_lo = umma_desc_k_sw128(sa_lo + koff);
                const uint64_t db_lo = DIRECT ? umma_desc_mn_sw128_32b(sb_lo + k * 1024, 4096) : umma_desc_k_sw128(sb_lo + koff);
                umma_for<F16, CTAS>(tmem_d, da_lo, db_hi, idesc, accumulate);
                umma_for<F16, CTAS, A_KEEP>(tmem_d, da_hi, db_lo, idesc, 1u);
                umma_for<F16, CTAS, A_KEPT>(tmem_d, da_hi, db_hi, idesc, 1u);
              } else {
                umma_for<F16, CTAS>(tmem_d, da_hi, db_hi, idesc, accumulate);
              }
            }
          }
          umma_commit_for<CTAS>(smem_u32(&empty_bar[stage]), leader);  // the stage is free (in both blocks) once these MMAs retire
          if (++stage == STAGES) {
            stage = 0;
            phase ^= 1u;
          }
        }
        if (ok) umma_commit_for<CTAS>(smem_u32(&tmem_full_bar[acc]), leader);
      }
    }
    __syncwarp();
  } else {
    // --------------------------------------------------------- epilogue
    const int quarter = warp & 3;  // tensor-memory lanes [32*quarter, 32*quarter+32)
    constexpr int LAST_COLUMNS = BN / Cfg::kEpiGroups;  // of a group on the last tile
    const bool second = Cfg::kEpiGroups == 2 && warp >= 6;  // of the two groups
    EpiWarp epi = epi_warp(epi_base, ctrl, warp - 2);
    if (second) {
      epi.buf = reinterpret_cast<float*>(stage_base + (warp - 6) * GEMM_EPI_WARP_BYTES);
      epi.cols = reinterpret_cast<float*>(stage_base + 4 * GEMM_EPI_WARP_BYTES + (warp - 6) * 256);
    }
    int local_tile = 0;
    for (int item = pair_id; item < num_items && ok; item += num_pairs, ++local_tile) {
      const int acc = local_tile & 1;
      const uint32_t acc_phase = (local_tile >> 1) & 1;
      const bool last = item + num_pairs >= num_items;
      int tm, tn;
      item_tile_coords(item, p, num_tiles, tm, tn);
      const int row0 = tm * BM + static_cast<int>(rank) * 128 + quarter * 32;
      const int columns = last ? LAST_COLUMNS : BN, first_col = second ? LAST_COLUMNS : 0, n0 = tn * BN + first_col;
      if (p.tma_epilogue && !second) epilogue_tma_begin(p, &map_c, epi, lane, row0, n0);
      // every lane waits; the warp then agrees on the outcome so that the warp-collective tensor-memory loads below are
      // never partly skipped
      const bool landed = mbar_wait_bounded(smem_u32(&tmem_full_bar[acc]), acc_phase, abort_flag);
      if (!__all_sync(0xffffffffu, landed)) {
        if (lane == 0) atomicCAS(p.status, 0, 0x1400 | (rank << 4) | acc);
        ok = false;
        break;
      }
      auto hand_back = [&] {
        __syncwarp();
        if (lane == 0) {
          if (CTAS == 2)
            mbar_arrive_peer(map_to_cta(smem_u32(&tmem_empty_bar[acc]), leader));
          else
            mbar_arrive(smem_u32(&tmem_empty_bar[acc]));
        }
      };
      if (second && !last) {
        hand_back();  // (kHandBacks)
        continue;
      }
      tc_fence_after_sync();
      const uint32_t taddr = tmem_base + (static_cast<uint32_t>(quarter * 32) << 16) + acc * 256 + first_col;
      if (in_cluster) {
        static_assert(ClusterPart<BN>::bytes(CTAS) <= STAGES * Cfg::kStageBytes + GEMM_EPI_BUF_BYTES, "partial sums and what arrives fit the rings");
        cluster_arrive_relaxed();
        cluster_part_store<BN>(stage_base, taddr, quarter * 32 + lane, 0, BN);  // launched without the second group
        arrived = true;
        break;
      } else if (n0 >= p.N) {
      } else if (!p.tma_epilogue) {
        epilogue_rows(p, taddr, epi.buf, lane, row0, n0, columns);
      } else {
        if (second) epilogue_tma_begin(p, &map_c, epi, lane, row0, n0);
        if (!epilogue_tma(p, &map_d, &map_c, taddr, epi, lane, row0, n0, columns, item_split(item, num_tiles) * p.part_rows, abort_flag)) {
          if (lane == 0) atomicCAS(p.status, 0, 0x1500 | (rank << 4) | acc);
          ok = false;
          break;
        }
      }
      if (last) break;  // nobody waits for this accumulator
      tc_fence_before_sync();
      hand_back();
    }
    if (!ok && elect_one()) wait_for_copies();  // tiles of C
    __syncwarp();
  }

  if (in_cluster && gate_open) {  // a closed gate leaves no partial sums
    if (!arrived) cluster_arrive_relaxed();
    int tm, tn;
    item_tile_coords(pair_id - split_rank * num_tiles, p, num_tiles, tm, tn);
    const int row0 = tm * BM + static_cast<int>(rank) * 128;
    auto barrier = [](bool so_far) { return __syncthreads_and(so_far) != 0; };
    ok = p.vec_epilogue ? cluster_exchange<BN, CTAS, GEMM_THREADS, 0, true>(p, stage_base, recv, split_rank, rank, row0, tn * BN, ok, abort_flag, barrier)
                        : cluster_exchange<BN, CTAS, GEMM_THREADS, 0, false>(p, stage_base, recv, split_rank, rank, row0, tn * BN, ok, abort_flag, barrier);
    if (!ok) {
      if (threadIdx.x == 0) atomicCAS(p.status, 0, 0x1600 | rank);
      wait_for_copies();
    }
    __syncwarp();
  }

  // Neither block may retire, or free tensor memory, while its peer can still signal its barriers, read its shared memory or
  // write its accumulators.  The barrier orders no memory: what was read here is in registers.  A launch's end, in cycles: a release at cluster
  // scope behind the stores of D 1500, the wait until the last tile has been read up to 2000 where it stood in front of the barrier, on
  // the way to it; without either 256^3 TF32 6.9 -> 5.7 us, 8192 x 8192 x 128 146 -> 132 us.
  tc_fence_before_sync();
  __syncthreads();
  if (CTAS == 2 || in_cluster) {
    cluster_arrive_relaxed();
    cluster_wait();
  }
  if (warp == 1) {
    tc_fence_after_sync();
    tmem_dealloc_for<CTAS>(tmem_base, GEMM_TMEM_COLS);
  } else if (warp > 1 && elect_one()) {
    bulk_wait_read<0>();  // the epilogue's tiles outlive the stores that read them
  }
}

// The second half of a product whose k-loop was divided (p.splits > 1, p.cluster_splits == 1): the partial sums added in order
// of k, so that the result does not depend on which block finished first.  part: [splits][part_rows][ld]
// floats, ld a multiple of 4; one thread per four columns, which keeps eight partial sums in flight.  Bound by latency and L2 (the
// partials were just written): 32 partials of 128 x 96, 6.2 us with a row of dependent loads a thread, 4.4 so.
template <bool VEC>
__device__ __forceinline__ void reduce_quads(const float* part, long long ld, int part_rows, int splits, const GemmParams& p) {
  constexpr int AHEAD = 8;
  const long long quads = (p.N + 3) >> 2, total = quads * p.M;
  const long long step = static_cast<long long>(part_rows) * ld >> 2;
  for (long long i = blockIdx.x * static_cast<long long>(blockDim.x) + threadIdx.x; i < total;
       i += static_cast<long long>(gridDim.x) * blockDim.x) {
    const long long row = i / quads;
    const int col = static_cast<int>(i - row * quads) << 2;
    const float4* src = reinterpret_cast<const float4*>(part + row * ld + col);
    float4 s = make_float4(0.f, 0.f, 0.f, 0.f), c, v[AHEAD];
    QuadColumns columns;
    for (int k = 0; k < splits; k += AHEAD) {
#pragma unroll
      for (int u = 0; u < AHEAD; ++u) v[u] = src[min(k + u, splits - 1) * step];
      if (k == 0) {
        c = quad_of_c<VEC>(p, row, col);
        columns = quad_columns(p, col);
        s = v[0];
      }
#pragma unroll
      for (int u = 0; u < AHEAD; ++u)
        if (k + u > 0 && k + u < splits) add_to(s, v[u]);
    }
    finish_quad<VEC>(p, row, col, s, c, columns);
  }
}
__global__ void __launch_bounds__(REDUCE_THREADS) gemm_reduce_kernel(const float* part, long long ld, int part_rows, int splits, const GemmParams p) {
  grid_launch_dependents();
  grid_dependency_wait();
  if (p.vec_epilogue)
    reduce_quads<true>(part, ld, part_rows, splits, p);
  else
    reduce_quads<false>(part, ld, part_rows, splits, p);
}

}  // namespace sb200
