// gemm_split.cuh — 3xTF32 GEMM that splits its operands on chip.
//
// gemm_pair_kernel reads the high parts of A and B from the caller's matrices and the low parts from panels that a launch in
// front of it has written: every element crosses from L2 to the SM twice, at 64 bytes a cycle and SM at most, which is what bounds
// tiles of 64 and 128 columns (1024^3: 40 KB per k-block and SM in 340 ns).  Here the elements cross once and there is no launch in
// front.  TMA brings the raw float32 tiles of A and B into a ring; groups of four warps take the k-blocks in turn: hi(A) and lo(A)
// go to tensor memory, a lane a row, from where the MMAs read A; hi(B) and lo(B) go back to shared memory in the layout they came
// in.  One thread issues the MMAs, for a pair of blocks (CTAS = 2) or a block on its own.  When the k-loop is through the warps
// that split run the epilogue.  The parts and the order of their products are gemm_pair_kernel's, so the bits are the same.
//
// Rows of A from M on are not split: an accumulator row depends on its own row of A only, and those rows are not stored.
//
// Bound: the tensor pipe from 128 columns on (430, 645 and 850 ns per k-block of a pair with 128, 192 and 256 columns); with 64 columns, where the
// pipe would take 200 ns, the latency of the groups' way from shared memory through registers to tensor memory (363).  Blocks on their
// own: 540 and 375 ns.  Against the two launches, and for few rows gemm_convert_kernel, in turn on one B200: 64 x 4096 x 4096 40.6 -> 25.1 us,
// 128 x 4096 x 4096 65.1 -> 28.7, 512^3 13.6 -> 11.9, 1024^3 20.4 -> 17.1, 2048^3 79.8 -> 73.3, 4096^3 541 -> 503.
#pragma once
#include "gemm_tcgen05_pair.cuh"

namespace sb200 {

// ROWS: rows of A a block loads and splits per k-block, 128, or 64 for products of so few (the MMA has 128 all the same).
template <int BN, int CTAS, int ROWS>
struct SplitCfg {
  static_assert(BN == 256 || BN == 192 || BN == 128 || BN == 64, "tile columns");
  static_assert(ROWS == 128 || (ROWS == 64 && CTAS == 1), "rows");
  static constexpr int kPartN = BN / CTAS;                            // columns of B this block loads and splits
  // Groups of four warps that split.  A group needs 2000 cycles for a k-block, nearly all of it latency.  Tiles of 64 columns with two, three
  // and four groups: 1024^3 19.2, 17.1 and 19.2 us, 512^3 12.3, 11.3 and 12.9, 64 x 1024 x 1024 10.0, 9.2 and 9.3.
  static constexpr int kGroups = 3;
  // Tiles of 128 columns and more: registers of the last warpgroup go to the splitting ones, launched with 128 a thread.  48 x 16384 x 4096 90.6 ->
  // 83.6 us, 2304 x 2304 x 520 44.3 -> 43.2, 2048^3 69.6 -> 68.9, other sizes even; tiles of 64 columns need no more than 128.  How many: with
  // these no instance spills.  With 152 and 40 the divided ones of pairs did (300 bytes reloaded a thread; 1024^3 15.8 us and 15.2, 768^3 12.0 and
  // 11.4, 5113 x 148 x 2772 29.9 and 29.2), and blocks on their own did a little.
  static constexpr bool kMoveRegs = BN > 64;
  static constexpr int kRegsSplit = 144, kRegsRest = BN == 256 ? 64 : 56;
  static_assert(kGroups * kRegsSplit + kRegsRest <= (kGroups + 1) * 128, "the warpgroups share what the block was launched with");
  static constexpr int kThreads = kGroups * 128 + (kMoveRegs ? 128 : 64);
  static constexpr uint32_t kABytes = ROWS * GEMM_BK * 4;
  static constexpr uint32_t kBBytes = kPartN * GEMM_BK * 4;
  static constexpr uint32_t kRawBytes = kABytes + kBBytes;            // a raw k-block
  // K-blocks held in parts; the rest of shared memory holds raw ones, which a stream from HBM needs more of (64 x 4096 x 4096: four and three
  // 30.3 us, three and five 23.8).
  static constexpr int kParts = kPartN == 32 ? 6 : kPartN == 64 ? 4 : 3;
  static constexpr uint32_t kPartBytes = 2 * kBBytes;                 // hi(B), lo(B)
  static constexpr int kRawFit = (216 * 1024 - kParts * static_cast<int>(kPartBytes)) / static_cast<int>(kRawBytes);
  static constexpr int kRaw = kRawFit > 8 ? 8 : kRawFit;
  static constexpr int kEpiGroups = 2;                                // groups that run the epilogue, each on a half of the columns
  static constexpr uint32_t kCtrlBytes = 2560;  // barriers, and from GEMM_CTRL_COLS on 256 bytes for each epilogue warp
  static constexpr uint32_t kRingBytes = kRaw * kRawBytes + kParts * kPartBytes;
  // a k-loop divided within a cluster: the partial sums and what arrives lie where the rings were
  static constexpr uint32_t kClusterBytes = ClusterPart<BN>::bytes(CTAS);
  __host__ __device__ static constexpr uint32_t area(bool in_cluster) { return in_cluster && kClusterBytes > kRingBytes ? kClusterBytes : kRingBytes; }
  __host__ __device__ static constexpr uint32_t smem_bytes(bool in_cluster) { return area(in_cluster) + (in_cluster ? 1024 : kCtrlBytes) + 1024; }
  static_assert(smem_bytes(true) <= 227 * 1024, "shared memory of a block");
  static constexpr uint32_t kTmemA = BN;                              // first tensor-memory column of A's parts
  static_assert(kTmemA + kParts * 2 * GEMM_BK <= 512, "the accumulator and A's parts fit tensor memory");
  static_assert(kRaw * kRawBytes >= kEpiGroups * 4 * GEMM_EPI_WARP_BYTES, "epilogue tiles fit the raw ring");
  static_assert((2 * kRaw + 2 * kParts + 4) * 8 <= GEMM_CTRL_CBAR, "the barriers fit the control area");
  // split_waits: what a group knows when it comes to a k-block.
  static_assert(kGroups <= kParts && kParts <= kRaw, "the part ring is as long as a turn of the groups, the raw ring as long as the part ring");
};

// The waits of a group in front of k-block n, in this order: part_free(stage, parity) until its part stage has been multiplied,
// raw_landed(stage, parity) until its raw stage has landed.
// A wait on a barrier's parity also returns while the phase before the wanted one is still to complete, so in a ring of R stages the group
// has to know that what n - R waited for has happened.  Part stages become free in the order of the k-blocks, and the group has seen
// that of n - kGroups become free, behind all up to n - kGroups - kParts, among them n - 2 * kParts.  Raw stages may land in any order; but
// once the part stage of n is free, all k-blocks up to n - kParts have been multiplied and so have landed, among them n - kRaw.
// The other way round the wait for a raw stage took the stage's contents for those of a load still on its way where kRaw is neither a
// multiple of kGroups nor kGroups + kParts and more.  Loading a raw stage behind the wait for the part stage costs nothing: 1024^3 16.9 us
// either way, 64 x 4096 x 4096 25.3 and 25.2, 2304 x 2304 x 520 36.7 and 36.4.
template <class Cfg, class PartFree, class RawLanded>
__host__ __device__ __forceinline__ bool split_waits(unsigned int n, PartFree&& part_free, RawLanded&& raw_landed) {
  return part_free(n % Cfg::kParts, (n / Cfg::kParts & 1u) ^ 1u) && raw_landed(n % Cfg::kRaw, n / Cfg::kRaw & 1u);
}

// hi and lo of N values, the bits of tf32_round and tf32_lo.  Two conversions and a subtraction a value, and one multiply-add that
// finds the rare value without a finite low part: with the low part rounded in integer arithmetic and a selection a value this took
// twice the cycles (8.4 against 14.2 a value and scheduler in a loop of nothing else).
template <int N>
__device__ __forceinline__ void tf32_split(const float* x, uint32_t* hi, uint32_t* lo) {
  float check = 0.0f;
#pragma unroll
  for (int i = 0; i < N; ++i) {
    const float h = tf32_round(x[i]), l = tf32_round(x[i] - h);
    hi[i] = __float_as_uint(h);
    lo[i] = __float_as_uint(l);
    check = fmaf(l, 0.0f, check);
  }
  if (check != 0.0f) {  // a value is not finite, or rounds to infinity: it has no low part
#pragma unroll
    for (int i = 0; i < N; ++i)
      if (!(fabsf(__uint_as_float(hi[i])) <= 3.402823466e+38f)) lo[i] = 0u;
  }
}

// map_a, map_b: the caller's matrices without rounding, boxes of 32 x ROWS and of 32 x 32; map_a_tail: of 32 x p.a_tail_rows, for the last,
// partial ROWS rows.  Rows past the end, and slabs of B past the last column, are not loaded (gemm_pair_kernel says what they cost).
// IN_CLUSTER: a k-loop divided within a cluster, as in gemm_pair_kernel.
template <int BN, int CTAS, int ROWS, bool IN_CLUSTER>
__global__ void __launch_bounds__(SplitCfg<BN, CTAS, ROWS>::kThreads, 1)
gemm_split_kernel(const __grid_constant__ CUtensorMap map_a, const __grid_constant__ CUtensorMap map_b,
                  const __grid_constant__ CUtensorMap map_a_tail, const __grid_constant__ CUtensorMap map_d,
                  const __grid_constant__ CUtensorMap map_c, const GemmParams p) {
  using Cfg = SplitCfg<BN, CTAS, ROWS>;
  constexpr int RAW = Cfg::kRaw, PARTS = Cfg::kParts, GROUPS = Cfg::kGroups, PART_N = Cfg::kPartN;
  constexpr uint32_t B_BYTES = Cfg::kBBytes;
  constexpr int BM = 128 * CTAS, EPI_WARPS = Cfg::kEpiGroups * 4, EPI_N = BN / Cfg::kEpiGroups;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  uint8_t* parts = smem + RAW * Cfg::kRawBytes;
  uint8_t* ctrl = smem + Cfg::area(IN_CLUSTER);
  uint64_t* raw_full = reinterpret_cast<uint64_t*>(ctrl);
  uint64_t* raw_empty = raw_full + RAW;
  uint64_t* part_full = raw_empty + RAW;     // used in the leader only
  uint64_t* part_empty = part_full + PARTS;  // one set per block
  uint64_t* acc_full = part_empty + PARTS;   // per block
  uint64_t* acc_empty = acc_full + 1;        // per block: both blocks' epilogues are through
  uint64_t* recv = acc_empty + 1;            // IN_CLUSTER: the others' partial sums
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(recv + 1);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const uint32_t cta = CTAS == 2 || IN_CLUSTER ? cluster_ctarank() : 0u;
  const uint32_t rank = blockIdx.x & (CTAS - 1u), leader = cta - rank;  // uniform to the compiler, as in gemm_pair_kernel
  const int num_tiles = p.tiles_m * p.tiles_n, num_items = num_tiles * p.splits;
  // IN_CLUSTER: item `split * num_tiles + tile` is this pair's only one
  const int split_rank = IN_CLUSTER ? static_cast<int>(cta) / CTAS : 0;
  const int first_item = IN_CLUSTER ? static_cast<int>(blockIdx.x) / (CTAS * p.cluster_splits) + split_rank * num_tiles
                                    : static_cast<int>(blockIdx.x) / CTAS;
  const int item_step = IN_CLUSTER ? 1 << 30 : static_cast<int>(gridDim.x) / CTAS;

  if (warp == 0) {  // the lanes share the barriers: raw_full, raw_empty, part_full, part_empty, acc_full, acc_empty, recv
    constexpr int BARS = 2 * RAW + 2 * PARTS + 3;
    for (int i = lane; i < BARS; i += 32)
      mbar_init(smem_u32(raw_full + i), i < RAW ? 1 : i < 2 * RAW ? 4 : i < 2 * RAW + PARTS ? 4 * CTAS : i == BARS - 2 ? EPI_WARPS * CTAS : 1);
    if (lane == 0) *abort_flag = 0;
    mbar_fence_init();
  }
  if (warp == 1) {  // the barriers of the tiles of C
    if (lane < 2 * EPI_WARPS) mbar_init(smem_u32(reinterpret_cast<uint64_t*>(ctrl + GEMM_CTRL_CBAR) + lane), 1);
    mbar_fence_init();
  }
  if (threadIdx.x == 64) {
    tma_prefetch_desc(&map_a);
    tma_prefetch_desc(&map_b);
    tma_prefetch_desc(&map_a_tail);
    if (p.tma_epilogue) tma_prefetch_desc(&map_d);
  }
  if (warp == GROUPS * 4 + 1) {
    tmem_alloc_for<CTAS>(smem_u32(tmem_slot), GEMM_TMEM_COLS);
    tmem_relinquish_for<CTAS>();
    tc_fence_before_sync();
  }
  __syncthreads();
  // the blocks' barriers exist before any signal crosses between them; the producer's loads cross nothing
  if (CTAS == 2) {
    cluster_arrive_relaxed();
    if (warp != GROUPS * 4) cluster_wait();
  }
  tc_fence_after_sync();
  const uint32_t tmem_base = *tmem_slot;
  grid_launch_dependents();
  grid_dependency_wait();  // nothing above touched global memory

  auto item_blocks = [&](int item, int& kb0) {
    kb0 = item_split(item, num_tiles) * p.split_k_blocks;
    return min(p.num_k_blocks - kb0, p.split_k_blocks);
  };

  if (warp < GROUPS * 4) {
    // ----------------------------------------- split; then the epilogue
    if constexpr (Cfg::kMoveRegs) asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(Cfg::kRegsSplit));
    const int group = warp >> 2, quarter = warp & 3, tid = threadIdx.x & 127;
    const int row = quarter * 32 + lane;
    const uint32_t lanes = static_cast<uint32_t>(quarter * 32) << 16;
    EpiWarp epi = epi_warp(smem, ctrl, warp);
    unsigned int before = 0;  // k-blocks of the items before
    int local = 0;
    bool ok = true, arrived = false;
    for (int item = first_item; item < num_items && ok; item += item_step, ++local) {
      int tm, tn, kb0;
      item_tile_coords(item, p, num_tiles, tm, tn);
      const int blocks = item_blocks(item, kb0);
      const int m0 = tm * BM + static_cast<int>(rank) * 128, n0 = tn * BN;
      const bool rows_here = quarter * 32 < ROWS && m0 + quarter * 32 < p.M;
      // this group's k-blocks of the item: those whose running number is `group` modulo GROUPS
      for (unsigned int kb = (group + GROUPS - before % GROUPS) % GROUPS; kb < static_cast<unsigned int>(blocks); kb += GROUPS) {
        const unsigned int n = before + kb;
        const unsigned int rs = n % RAW, ps = n % PARTS;
        const bool landed = split_waits<Cfg>(
            n, [&](unsigned int stage, uint32_t parity) { return mbar_wait_bounded(smem_u32(&part_empty[stage]), parity, abort_flag); },
            [&](unsigned int stage, uint32_t parity) { return mbar_wait_bounded(smem_u32(&raw_full[stage]), parity, abort_flag); });
        // the whole k-block into registers first: one latency of shared memory
        const uint8_t* raw = smem + rs * Cfg::kRawBytes;
        float a[GEMM_BK], b[PART_N / 4];
#pragma unroll
        for (int j = 0; j < GEMM_BK / 4; ++j)
          *reinterpret_cast<float4*>(a + 4 * j) = *reinterpret_cast<const float4*>(raw + row % ROWS * 128 + ((j ^ (row & 7)) << 4));
#pragma unroll
        for (int j = 0; j < PART_N / 16; ++j)
          *reinterpret_cast<float4*>(b + 4 * j) = *reinterpret_cast<const float4*>(raw + Cfg::kABytes + (tid + 128 * j) * 16);
        if (!__all_sync(0xffffffffu, landed)) {
          if (lane == 0) atomicCAS(p.status, 0, 0x3100 | (rank << 4) | rs);
          ok = false;
          break;
        }
        tc_fence_after_sync();
        if (rows_here) {
          const uint32_t ta = tmem_base + lanes + Cfg::kTmemA + ps * (2 * GEMM_BK);
#pragma unroll
          for (int h = 0; h < 2; ++h) {
            uint32_t hi[16], lo[16];
            tf32_split<16>(a + 16 * h, hi, lo);
            tmem_st_32x32b_x16(ta + 16 * h, hi);
            tmem_st_32x32b_x16(ta + GEMM_BK + 16 * h, lo);
          }
        }
        // hi(B) and lo(B) keep the raw tile's layout: where an element lies does not matter here
        uint4* dst = reinterpret_cast<uint4*>(parts + ps * Cfg::kPartBytes) + tid;
        constexpr int QUADS = PART_N / 16, STEP = QUADS % 4 == 0 ? 4 : QUADS % 3 == 0 ? 3 : 1;
#pragma unroll
        for (int j = 0; j < QUADS; j += STEP) {
          uint32_t hi[4 * STEP], lo[4 * STEP];
          tf32_split<4 * STEP>(b + 4 * j, hi, lo);
#pragma unroll
          for (int i = 0; i < STEP; ++i) {
            dst[128 * (j + i)] = make_uint4(hi[4 * i], hi[4 * i + 1], hi[4 * i + 2], hi[4 * i + 3]);
            dst[128 * (j + i) + B_BYTES / 16] = make_uint4(lo[4 * i], lo[4 * i + 1], lo[4 * i + 2], lo[4 * i + 3]);
          }
        }
        tmem_st_wait();
        fence_async_shared();  // before the tensor core reads what was written here
        tc_fence_before_sync();
        __syncwarp();
        // Not before the values have been used: handed back right after the loads, the stage was written again while some of them, which the
        // compiler had moved behind the arrival of another lane, were still to come.
        if (lane == 0) {
          mbar_arrive(smem_u32(&raw_empty[rs]));
          if (CTAS == 2 && rank != 0)
            mbar_arrive_peer(map_to_cta(smem_u32(&part_full[ps]), leader));
          else
            mbar_arrive(smem_u32(&part_full[ps]));
        }
      }
      before += blocks;
      if (group >= Cfg::kEpiGroups || !ok) {
        if (IN_CLUSTER) break;  // its one item
        continue;
      }
      const int row0 = m0 + quarter * 32, c0 = n0 + group * EPI_N;
      const bool landed = mbar_wait_bounded(smem_u32(acc_full), local & 1, abort_flag);
      if (!__all_sync(0xffffffffu, landed)) {
        if (lane == 0) atomicCAS(p.status, 0, 0x3400 | (rank << 4));
        ok = false;
        break;
      }
      tc_fence_after_sync();
      // every tile of the item has been split and multiplied: the rings are idle until this epilogue hands them back
      const uint32_t taddr = tmem_base + lanes + group * EPI_N;
      if constexpr (IN_CLUSTER) {
        cluster_arrive_relaxed();
        cluster_part_store<BN>(smem, taddr, row, group * EPI_N, EPI_N);
        arrived = true;
      } else if (c0 < p.N) {
        if (!p.tma_epilogue) {
          epilogue_rows(p, taddr, epi.buf, lane, row0, c0, EPI_N);
          fence_async_shared();  // its ordinary stores to the tile before the loads of the next item, which land there
        } else {
          epilogue_tma_begin(p, &map_c, epi, lane, row0, c0);
          if (!epilogue_tma(p, &map_d, &map_c, taddr, epi, lane, row0, c0, EPI_N, item_split(item, num_tiles) * p.part_rows, abort_flag)) {
            if (lane == 0) atomicCAS(p.status, 0, 0x3500 | (rank << 4));
            ok = false;
          }
        }
      }
      if (IN_CLUSTER || item + item_step >= num_items) break;  // nothing follows that would wait for the accumulator or the rings
      if (elect_one()) bulk_wait_read<0>();  // the stores have read their tiles
      tc_fence_before_sync();
      __syncwarp();
      if (lane == 0) {
        mbar_arrive(smem_u32(acc_empty));
        if (CTAS == 2) mbar_arrive_peer(map_to_cta(smem_u32(acc_empty), cta ^ 1u));
      }
    }
    if (!ok && elect_one()) wait_for_copies();  // tiles of C
    __syncwarp();
    if constexpr (IN_CLUSTER) {
      if (!arrived) cluster_arrive_relaxed();
      int tm, tn;
      item_tile_coords(first_item - split_rank * num_tiles, p, num_tiles, tm, tn);
      const int row0 = tm * BM + static_cast<int>(rank) * 128;
      auto barrier = [](bool so_far) { return barrier_all(1, GROUPS * 128, so_far); };
      ok = p.vec_epilogue ? cluster_exchange<BN, CTAS, GROUPS * 128, GROUPS * 4 - 1, true>(p, smem, recv, split_rank, rank, row0, tn * BN, ok, abort_flag, barrier)
                          : cluster_exchange<BN, CTAS, GROUPS * 128, GROUPS * 4 - 1, false>(p, smem, recv, split_rank, rank, row0, tn * BN, ok, abort_flag, barrier);
      if (!ok) {
        if (threadIdx.x == 0) atomicCAS(p.status, 0, 0x3600 | rank);
        wait_for_copies();
      }
      __syncwarp();
    }
  } else {
    if constexpr (Cfg::kMoveRegs) asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(Cfg::kRegsRest));
    if (warp == GROUPS * 4) {
      // ------------------------------------------------------ TMA producer
      if (elect_one()) {
        const uint64_t pol_a = l2_policy(p.l2_policy & 3), pol_b = l2_policy((p.l2_policy >> 2) & 3);
        int stage = 0, local = 0;
        uint32_t phase = 0;
        bool ok = true;
        for (int item = first_item; item < num_items && ok; item += item_step, ++local) {
          int tm, tn, kb0;
          item_tile_coords(item, p, num_tiles, tm, tn);
          const int blocks = item_blocks(item, kb0);
          const int m0 = tm * BM + static_cast<int>(rank) * 128, n0 = tn * BN + static_cast<int>(rank) * PART_N;
          if (local > 0 && !(CTAS == 2 ? mbar_wait_cluster(smem_u32(acc_empty), (local - 1) & 1, abort_flag)
                                       : mbar_wait_bounded(smem_u32(acc_empty), (local - 1) & 1, abort_flag))) {
            atomicCAS(p.status, 0, 0x3200 | rank);
            ok = false;
            break;
          }
          const bool whole_rows = m0 + ROWS <= p.M;
          const int rows = whole_rows ? ROWS : m0 < p.M ? p.a_tail_rows : 0;
          const int slabs = max(0, min(PART_N / 32, (p.N - n0 + 31) >> 5));
          for (int kb = kb0; kb < kb0 + blocks; ++kb) {
            if (!mbar_wait_bounded(smem_u32(&raw_empty[stage]), phase ^ 1u, abort_flag)) {
              atomicCAS(p.status, 0, 0x3000 | (rank << 4) | stage);
              ok = false;
              break;
            }
            const uint32_t bar = smem_u32(&raw_full[stage]);
            uint8_t* dst = smem + stage * Cfg::kRawBytes;
            mbar_arrive_expect_tx(bar, rows * 128 + slabs * 4096);
            if (whole_rows)
              tma_load_2d_hint(smem_u32(dst), &map_a, bar, kb * GEMM_BK, m0, pol_a);
            else if (rows)
              tma_load_2d_hint(smem_u32(dst), &map_a_tail, bar, kb * GEMM_BK, m0, pol_a);
#pragma unroll
            for (int sl = 0; sl < PART_N / 32; ++sl)
              if (sl < slabs) tma_load_2d_hint(smem_u32(dst + Cfg::kABytes + sl * 4096), &map_b, bar, n0 + 32 * sl, kb * GEMM_BK, pol_b);
            if (++stage == RAW) {
              stage = 0;
              phase ^= 1u;
            }
          }
        }
        if (!ok) wait_for_copies();
      }
      __syncwarp();
      if (CTAS == 2) cluster_wait();  // of the barrier in front
    } else if (warp == GROUPS * 4 + 1 && rank == 0 && elect_one()) {
      // ------------------------------------------------------- MMA issuer (leader block)
      constexpr uint32_t idesc = umma_idesc_tf32(BM, BN, true);
      int stage = 0, local = 0;
      uint32_t phase = 0;
      bool ok = true;
      for (int item = first_item; item < num_items && ok; item += item_step, ++local) {
        int kb0;
        const int blocks = item_blocks(item, kb0);
        if (local > 0 && !(CTAS == 2 ? mbar_wait_cluster(smem_u32(acc_empty), (local - 1) & 1, abort_flag)
                                     : mbar_wait_bounded(smem_u32(acc_empty), (local - 1) & 1, abort_flag))) {
          atomicCAS(p.status, 0, 0x3210);
          break;
        }
        for (int kb = 0; kb < blocks; ++kb) {
          const uint32_t full = smem_u32(&part_full[stage]);
          if (!(CTAS == 2 ? mbar_wait_cluster(full, phase, abort_flag) : mbar_wait_bounded(full, phase, abort_flag))) {
            atomicCAS(p.status, 0, 0x3300 | stage);
            ok = false;
            break;
          }
          tc_fence_after_sync();
          const uint32_t ta = tmem_base + Cfg::kTmemA + stage * (2 * GEMM_BK);
          const uint32_t sb_hi = smem_u32(parts + stage * Cfg::kPartBytes), sb_lo = sb_hi + B_BYTES;
#pragma unroll
          for (int k = 0; k < GEMM_BK / GEMM_UMMA_K; ++k) {
            const uint64_t db_hi = umma_desc_mn_sw128_32b(sb_hi + k * 1024, 4096), db_lo = umma_desc_mn_sw128_32b(sb_lo + k * 1024, 4096);
            const uint32_t a_hi = ta + k * GEMM_UMMA_K, a_lo = a_hi + GEMM_BK;
            umma_tf32_tmem_a<CTAS>(tmem_base, a_lo, db_hi, idesc, (kb | k) ? 1u : 0u);
            umma_tf32_tmem_a<CTAS>(tmem_base, a_hi, db_lo, idesc, 1u);
            umma_tf32_tmem_a<CTAS>(tmem_base, a_hi, db_hi, idesc, 1u);
          }
          umma_commit_for<CTAS>(smem_u32(&part_empty[stage]), leader);
          if (++stage == PARTS) {
            stage = 0;
            phase ^= 1u;
          }
        }
        if (ok) umma_commit_for<CTAS>(smem_u32(acc_full), leader);
      }
    }
    __syncwarp();
    if constexpr (IN_CLUSTER) {
      cluster_arrive_relaxed();
      cluster_wait();
    }
  }
  // No block retires, or frees tensor memory, while its peers signal its barriers, read its memory or write its accumulator.  The barrier
  // orders no memory: what was read here is in registers.  Nor do the epilogue's last signals wait for anything: 1024^3 17.3 -> 16.1 us,
  // 256^3 8.5 -> 7.5.
  tc_fence_before_sync();
  __syncthreads();
  if (CTAS == 2 || IN_CLUSTER) {
    cluster_arrive_relaxed();
    cluster_wait();
  }
  if (warp == GROUPS * 4 + 1) {
    tc_fence_after_sync();
    tmem_dealloc_for<CTAS>(tmem_base, GEMM_TMEM_COLS);
  } else if (warp < EPI_WARPS && elect_one()) {
    bulk_wait_read<0>();  // the epilogue's tiles outlive the stores that read them
  }
}

}  // namespace sb200
