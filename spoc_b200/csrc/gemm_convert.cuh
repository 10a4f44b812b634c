// gemm_convert.cuh — GEMM whose operands are converted in registers on their way to shared memory.
//
// gemm_pair_kernel reads its operands with TMA, which needs 16-byte aligned rows, and takes the low parts of 3xTF32 from panels
// a launch before it has written.  For few rows against a large matrix (where the panels would triple the traffic), for small
// products of unaligned matrices and for tiny ones, this kernel does the whole operator in one launch: eight warps load A and
// B with ordinary loads, two k-blocks ahead in registers, round every element to its TF32 high part (and low part) and store
// both to the ring in the layouts gemm_pair_kernel's MMAs read; one more warp issues the MMAs (128 x BN per block,
// cta_group::1); when the k-loop is through, the eight warps run the epilogue, each on 32 rows and half of the columns.  Sums
// are formed in the same order from the same parts as there, so the bits are the same.
//
// Bound: the converting warps.  Per k-block, 128 and 64 columns: 3xTF32 1060 and 790 ns with aligned quads, 1430 and 1180 ns
// element by element; TF32 element by element 900 and 710 ns.  (The pair kernel behind prepared panels: 430 and 340 ns.)
// 64 x 4096 x 4096 in 3xTF32: 44 us against 85 through panels; 64^3 unaligned 7.5 against 14.5 us, 700^3 31 against 41 us.
#pragma once
#include "gemm_tcgen05_pair.cuh"

namespace sb200 {

constexpr int CONV_WARPS = 8;
constexpr int CONV_THREADS = CONV_WARPS * 32 + 128;  // two converting warpgroups and one that issues the MMAs
// Registers: launched with 168 a thread (384 x 168 = 64512); the converting warpgroups take 224, the third keeps 40
// (128 * (224 + 224 + 40) = 62464).
constexpr int CONV_REGS_CONVERT = 224, CONV_REGS_MMA = 40;
constexpr int CONV_AHEAD = 2;  // k-blocks loaded ahead of the one being converted
constexpr uint32_t CONV_CTRL_BYTES = 4096;

template <int MODE, int BN>
struct ConvCfg {
  static constexpr int kOperands = MODE == 3 ? 2 : 1;
  static constexpr uint32_t kBBytes = BN * GEMM_BK * 4;
  static constexpr uint32_t kStageBytes = kOperands * (PAIR_A_BYTES + kBBytes);
  static constexpr int kStagesFit = (192 * 1024) / kStageBytes;
  static constexpr int kStages = kStagesFit > 8 ? 8 : kStagesFit;
  // the epilogue's tiles reuse the ring, which is idle by then
  static_assert(kStages * kStageBytes >= CONV_WARPS * GEMM_EPI_WARP_BYTES, "epilogue tiles fit the ring");
  static constexpr uint32_t kSmemBytes = kStages * kStageBytes + CONV_CTRL_BYTES + 1024;
};

struct ConvOperands {
  const float* A;
  const float* B;
  long long lda, ldb;
  int K;
};

// Predicated loads, zero where the predicate is false.  volatile: they are issued where they stand, two k-blocks before their
// values are used; the compiler sank plain loads to their uses, and every k-block waited for memory.
__device__ __forceinline__ void ld4_if(float* x, const float* p, bool in) {
  asm volatile(
      "{\n"
      ".reg .pred q;\n"
      "setp.ne.b32 q, %5, 0;\n"
      "mov.b32 %0, 0;\n"
      "mov.b32 %1, 0;\n"
      "mov.b32 %2, 0;\n"
      "mov.b32 %3, 0;\n"
      "@q ld.global.v4.f32 {%0, %1, %2, %3}, [%4];\n"
      "}\n"
      : "=&f"(x[0]), "=&f"(x[1]), "=&f"(x[2]), "=&f"(x[3])
      : "l"(p), "r"(static_cast<int>(in)));
}
__device__ __forceinline__ void ld1_if(float* x, const float* p, bool in) {
  asm volatile(
      "{\n"
      ".reg .pred q;\n"
      "setp.ne.b32 q, %2, 0;\n"
      "mov.b32 %0, 0;\n"
      "@q ld.global.f32 %0, [%1];\n"
      "}\n"
      : "=&f"(x[0])
      : "l"(p), "r"(static_cast<int>(in)));
}

// One thread's elements of a k-block of A (128 x 32) and B (32 x BN) and where they go.  VEC: quads (rows 16-byte aligned, K and
// N multiples of 4); else single elements, a warp per row of A and per 32 columns of a row of B.
template <int BN, bool VEC>
struct ConvTile {
  static constexpr int NA = 16, NB = BN / 8;  // elements per thread
  float a[NA], b[NB];

  __device__ __forceinline__ void load(const ConvOperands& o, int M, int N, int m0, int n0, int k0, int tid) {
    if (VEC) {
      const int q = tid & 7, k = k0 + q * 4;
#pragma unroll
      for (int j = 0; j < NA / 4; ++j) {
        const int row = m0 + (tid >> 3) + 32 * j;
        ld4_if(a + 4 * j, o.A + static_cast<long long>(row) * o.lda + k, row < M && k < o.K);
      }
      constexpr int QN = BN / 4;  // quads per row of B
      const int n = n0 + (tid % QN) * 4;
#pragma unroll
      for (int j = 0; j < NB / 4; ++j) {
        const int kk = k0 + tid / QN + (256 / QN) * j;
        ld4_if(b + 4 * j, o.B + static_cast<long long>(kk) * o.ldb + n, kk < o.K && n < N);
      }
    } else {
      const int lane = tid & 31, w = tid >> 5;
      const bool k_in = k0 + lane < o.K;
      const float* ap = o.A + static_cast<long long>(m0 + w * 16) * o.lda + k0 + lane;
#pragma unroll
      for (int j = 0; j < NA; ++j) ld1_if(a + j, ap + j * o.lda, k_in && m0 + w * 16 + j < M);
      const float* bp = o.B + static_cast<long long>(k0 + w * 4) * o.ldb + n0 + lane;
#pragma unroll
      for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int c = 0; c < BN / 32; ++c)
          ld1_if(b + i * (BN / 32) + c, bp + i * o.ldb + 32 * c, k0 + w * 4 + i < o.K && n0 + lane + 32 * c < N);
    }
  }

  // High (and low) parts into a stage: A K-major in the 128-byte swizzle, B as [32 k][32 n] slabs in the 128-byte swizzle with
  // 32-byte atoms.  Every warp store covers whole 128-byte rows: no bank conflicts.
  template <int MODE>
  __device__ __forceinline__ void store(uint8_t* stage, int tid) const {
    constexpr uint32_t LO = PAIR_A_BYTES + BN * GEMM_BK * 4;
    if (VEC) {
      const int q = tid & 7;
#pragma unroll
      for (int j = 0; j < NA / 4; ++j) {
        const int row = (tid >> 3) + 32 * j;
        put4<MODE, LO>(stage + row * 128 + ((q ^ (row & 7)) << 4), a + 4 * j);
      }
      constexpr int QN = BN / 4;
      const int n = (tid % QN) * 4;
#pragma unroll
      for (int j = 0; j < NB / 4; ++j) {
        const int k = tid / QN + (256 / QN) * j;
        put4<MODE, LO>(stage + PAIR_A_BYTES + (n >> 5) * 4096 + k * 128 + ((((n & 31) >> 3) ^ (k & 3)) << 5) + (n & 7) * 4, b + 4 * j);
      }
    } else {
      const int lane = tid & 31, w = tid >> 5;
#pragma unroll
      for (int j = 0; j < NA; ++j) {
        const int row = w * 16 + j;
        put1<MODE, LO>(stage + row * 128 + (((lane >> 2) ^ (row & 7)) << 4) + (lane & 3) * 4, a[j]);
      }
#pragma unroll
      for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int c = 0; c < BN / 32; ++c) {
          const int k = w * 4 + i;
          put1<MODE, LO>(stage + PAIR_A_BYTES + c * 4096 + k * 128 + (((lane >> 3) ^ (k & 3)) << 5) + (lane & 7) * 4,
                         b[i * (BN / 32) + c]);
        }
    }
  }

  // hi and lo of x, the bits of tf32_round and tf32_lo.  The conversion instruction issues 16 lanes a cycle and SM (two per
  // element were half of this kernel's time), so the low part is rounded in integer arithmetic beside it.
  template <int MODE>
  __device__ __forceinline__ static void split(float x, float& hi, float& lo) {
    hi = tf32_round(x);
    if (MODE == 3) {
      const uint32_t d = __float_as_uint(x - hi);
      const float r = __uint_as_float((d + 0xfffu + ((d >> 13) & 1u)) & 0xffffe000u);
      lo = fabsf(hi) <= 3.402823466e+38f ? r : 0.0f;
    }
  }
  template <int MODE, uint32_t LO>
  __device__ __forceinline__ static void put4(uint8_t* dst, const float* x) {
    float4 h, l;
    split<MODE>(x[0], h.x, l.x);
    split<MODE>(x[1], h.y, l.y);
    split<MODE>(x[2], h.z, l.z);
    split<MODE>(x[3], h.w, l.w);
    *reinterpret_cast<float4*>(dst) = h;
    if (MODE == 3) *reinterpret_cast<float4*>(dst + LO) = l;
  }
  template <int MODE, uint32_t LO>
  __device__ __forceinline__ static void put1(uint8_t* dst, float x) {
    float h, l;
    split<MODE>(x, h, l);
    *reinterpret_cast<float*>(dst) = h;
    if (MODE == 3) *reinterpret_cast<float*>(dst + LO) = l;
  }
};

// The converting warps' barrier between two work items, and one decision for all of them: whether to go on to the next.  The MMA issuer
// is no part of the barrier and may give up at any time; if each warp read its flag behind the barrier, some could leave and the
// others wait for them at the next barrier without end.
__device__ __forceinline__ bool convert_go_on(bool ok, volatile int* abort_flag) {
  return barrier_all(1, CONV_WARPS * 32, ok && *abort_flag == 0);
}

// Exercises that decision: the converting warps of each block go from item to item in different time, warp CONV_WARPS gives up
// after block * step_ns, and every warp writes the number of its items (at most max_items).  All warps of a block write the same.
__global__ void go_on_probe_kernel(int* items, int max_items, unsigned int step_ns) {
  __shared__ int flag;
  volatile int* abort_flag = &flag;
  const int warp = threadIdx.x >> 5;
  if (threadIdx.x == 0) flag = 0;
  __syncthreads();
  if (warp == CONV_WARPS) {
    const uint64_t t0 = global_timer_ns();
    while (global_timer_ns() - t0 < static_cast<uint64_t>(blockIdx.x) * step_ns) {
    }
    if ((threadIdx.x & 31) == 0) *abort_flag = 1;
    return;
  }
  int n = 0;
  for (bool ok = true; ok && n < max_items; ++n) {
    for (int i = 0; i < ((warp * 5 + n) & 7); ++i) __nanosleep(20);
    __syncwarp();
    ok = convert_go_on(ok, abort_flag);
  }
  if ((threadIdx.x & 31) == 0) items[blockIdx.x * CONV_WARPS + warp] = n;
}

// IN_CLUSTER: a k-loop divided within a cluster; a form of its own, because what it adds cost the smallest products 0.3 to 0.6 us.
template <int MODE, int BN, bool VEC, bool IN_CLUSTER>
__global__ void __launch_bounds__(CONV_THREADS, 1)
gemm_convert_kernel(const ConvOperands o, const __grid_constant__ CUtensorMap map_d, const __grid_constant__ CUtensorMap map_c,
                    const GemmParams p) {
  using Cfg = ConvCfg<MODE, BN>;
  constexpr int STAGES = Cfg::kStages;
  constexpr uint32_t B_BYTES = Cfg::kBBytes;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  uint8_t* ctrl = smem + STAGES * Cfg::kStageBytes;
  uint64_t* full_bar = reinterpret_cast<uint64_t*>(ctrl);
  uint64_t* empty_bar = full_bar + STAGES;
  uint64_t* done_bar = full_bar + 2 * STAGES;
  uint64_t* recv = full_bar + 2 * STAGES + 1;  // in_cluster: the others' partial sums
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(full_bar + 2 * STAGES + 2);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  // in_cluster: item `split * num_tiles + tile` is this block's only one
  constexpr bool in_cluster = IN_CLUSTER;
  const int split_rank = in_cluster ? static_cast<int>(cluster_ctarank()) : 0;

  // Quads: a warp for the barriers, a lane each (64^3 5.7 -> 5.6 us).  Single elements: one thread, and below their own place of the wait for the
  // stores (with those of the quads up to 4 % longer: 7 x 5363 x 246 14.3 and 14.7 us, 4731 x 18 x 148 11.1 and 11.6; the difference is in
  // what the compiler makes of the kernel, whose registers are all taken, and not in the set-up's time).
  auto barrier_count = [](int i) { return i < STAGES ? CONV_WARPS : 1; };  // full, empty, done, recv
  constexpr int BARS = 2 * STAGES + 2;
  static_assert(BARS <= 32, "a lane a barrier");
  uint64_t* c_bars = reinterpret_cast<uint64_t*>(ctrl + GEMM_CTRL_CBAR);
  if constexpr (VEC) {
    if (warp == 0) {
      if (lane < BARS) mbar_init(smem_u32(&full_bar[lane]), barrier_count(lane));
      if (lane == 0) *abort_flag = 0;
      mbar_fence_init();
    } else if (warp == 1) {
      if (lane < 2 * CONV_WARPS) mbar_init(smem_u32(c_bars + lane), 1);
      mbar_fence_init();
    }
    if (threadIdx.x == 64 && p.tma_epilogue) tma_prefetch_desc(&map_d);
  } else if (threadIdx.x == 0) {
    for (int i = 0; i < BARS; ++i) mbar_init(smem_u32(&full_bar[i]), barrier_count(i));
    for (int i = 0; i < 2 * CONV_WARPS; ++i) mbar_init(smem_u32(c_bars + i), 1);
    *abort_flag = 0;
    mbar_fence_init();
    if (p.tma_epilogue) tma_prefetch_desc(&map_d);
  }
  if (warp == CONV_WARPS) {
    tmem_alloc(smem_u32(tmem_slot), BN);
    tmem_relinquish();
    tc_fence_before_sync();
  }
  __syncthreads();
  tc_fence_after_sync();
  const uint32_t tmem_base = *tmem_slot;
  grid_launch_dependents();
  grid_dependency_wait();  // nothing above touched global memory
  const int num_tiles = p.tiles_m * p.tiles_n, num_items = num_tiles * p.splits;
  const int first_item = in_cluster ? static_cast<int>(blockIdx.x) / p.cluster_splits + split_rank * num_tiles : static_cast<int>(blockIdx.x);
  const int item_step = in_cluster ? 1 << 30 : static_cast<int>(gridDim.x);

  if (warp < CONV_WARPS) {
    // ----------------------------------------- load, convert, store; then the epilogue
    asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(CONV_REGS_CONVERT));
    EpiWarp epi = epi_warp(smem, ctrl, warp);
    const int quarter = warp & 3, half = warp >> 2;
    int stage = 0, local = 0;
    uint32_t phase = 0;
    bool ok = true;
    for (int item = first_item; item < num_items && ok; item += item_step, ++local) {
      int tm, tn;
      item_tile_coords(item, p, num_tiles, tm, tn);
      const int m0 = tm * 128, n0 = tn * BN, split = item_split(item, num_tiles);
      const int kb0 = split * p.split_k_blocks, blocks = min(p.num_k_blocks - kb0, p.split_k_blocks);
      ConvTile<BN, VEC> t[CONV_AHEAD + 1];
#pragma unroll
      for (int u = 0; u < CONV_AHEAD; ++u)
        if (u < blocks) t[u].load(o, p.M, p.N, m0, n0, (kb0 + u) * GEMM_BK, threadIdx.x);
      for (int kb = 0; kb < blocks && ok; kb += CONV_AHEAD + 1) {
#pragma unroll
        for (int u = 0; u <= CONV_AHEAD; ++u) {  // t[] is indexed by constants: it stays in registers
          if (kb + u >= blocks) break;
          if (kb + u + CONV_AHEAD < blocks)
            t[(u + CONV_AHEAD) % (CONV_AHEAD + 1)].load(o, p.M, p.N, m0, n0, (kb0 + kb + u + CONV_AHEAD) * GEMM_BK, threadIdx.x);
          const bool free = mbar_wait_bounded(smem_u32(&empty_bar[stage]), phase ^ 1u, abort_flag);
          if (!__all_sync(0xffffffffu, free)) {
            if (lane == 0) atomicCAS(p.status, 0, 0x2100 | stage);
            ok = false;
            break;
          }
          t[u].template store<MODE>(smem + stage * Cfg::kStageBytes, threadIdx.x);
          fence_async_shared();  // before the tensor core reads what was written here
          __syncwarp();
          if (lane == 0) mbar_arrive(smem_u32(&full_bar[stage]));
          if (++stage == STAGES) {
            stage = 0;
            phase ^= 1u;
          }
        }
      }
      const bool landed = ok && mbar_wait_bounded(smem_u32(done_bar), local & 1, abort_flag);
      if (!__all_sync(0xffffffffu, landed)) {
        if (lane == 0) atomicCAS(p.status, 0, 0x2400);
        ok = false;
      }
      if (ok) {
        tc_fence_after_sync();
        if constexpr (in_cluster) {
          cluster_arrive_relaxed();  // the ring is idle
        }
        const int row0 = m0 + quarter * 32, c0 = n0 + half * (BN / 2);
        const uint32_t taddr = tmem_base + (static_cast<uint32_t>(quarter * 32) << 16) + half * (BN / 2);
        if (c0 < p.N) {
          if constexpr (in_cluster) {
            static_assert(ClusterPart<BN>::bytes(1) <= STAGES * Cfg::kStageBytes, "partial sums and what arrives fit the ring");
            cluster_part_store<BN>(smem, taddr, quarter * 32 + lane, half * (BN / 2), BN / 2);
          } else if (!p.tma_epilogue) {
            epilogue_rows(p, taddr, epi.buf, lane, row0, c0, BN / 2);
          } else {
            epilogue_tma_begin(p, &map_c, epi, lane, row0, c0);
            if (!epilogue_tma(p, &map_d, &map_c, taddr, epi, lane, row0, c0, BN / 2, split * p.part_rows, abort_flag)) {
              if (lane == 0) atomicCAS(p.status, 0, 0x2500);
              ok = false;
            }
          }
        }
        if (!VEC && elect_one()) bulk_wait_read<0>();  // (here for single elements: 2 % shorter than behind the closing barrier, as above)
        tc_fence_before_sync();
      }
      if (in_cluster || item + item_step >= num_items) break;  // the block's last item: nothing follows but the barrier all threads share
      if (VEC && ok && elect_one()) bulk_wait_read<0>();  // the ring takes operands again once the stores have read their tiles
      // every warp is through with the accumulator and the tiles before the next item's operands arrive
      __syncwarp();
      ok = convert_go_on(ok, abort_flag);
    }
    if (!ok && elect_one()) wait_for_copies();  // tiles of C
    __syncwarp();
    if constexpr (in_cluster) {
      if (!ok) cluster_arrive_relaxed();
      int tm, tn;
      item_tile_coords(first_item - split_rank * num_tiles, p, num_tiles, tm, tn);
      auto barrier = [](bool so_far) { return barrier_all(1, CONV_WARPS * 32, so_far); };
      ok = p.vec_epilogue ? cluster_exchange<BN, 1, CONV_WARPS * 32, 0, true>(p, smem, recv, split_rank, 0, tm * 128, tn * BN, ok, abort_flag, barrier)
                          : cluster_exchange<BN, 1, CONV_WARPS * 32, 0, false>(p, smem, recv, split_rank, 0, tm * 128, tn * BN, ok, abort_flag, barrier);
      if (!ok) {
        if (threadIdx.x == 0) atomicCAS(p.status, 0, 0x2600);
        wait_for_copies();
      }
      __syncwarp();
    }
  } else {
    // ------------------------------------------------------- MMA issuer
    asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(CONV_REGS_MMA));
    if (warp == CONV_WARPS && elect_one()) {
      constexpr uint32_t idesc = umma_idesc_tf32(128, BN, true);
      int stage = 0;
      uint32_t phase = 0;
      bool ok = true;
      for (int item = first_item; item < num_items && ok; item += item_step) {
        const int kb0 = item_split(item, num_tiles) * p.split_k_blocks, blocks = min(p.num_k_blocks - kb0, p.split_k_blocks);
        for (int kb = 0; kb < blocks; ++kb) {
          if (!mbar_wait_bounded(smem_u32(&full_bar[stage]), phase, abort_flag)) {
            atomicCAS(p.status, 0, 0x2300 | stage);
            ok = false;
            break;
          }
          tc_fence_after_sync();
          const uint32_t sa_hi = smem_u32(smem + stage * Cfg::kStageBytes), sb_hi = sa_hi + PAIR_A_BYTES;
          const uint32_t sa_lo = sb_hi + B_BYTES, sb_lo = sa_lo + PAIR_A_BYTES;
#pragma unroll
          for (int k = 0; k < GEMM_BK / GEMM_UMMA_K; ++k) {
            const uint64_t da_hi = umma_desc_k_sw128(sa_hi + k * 32), db_hi = umma_desc_mn_sw128_32b(sb_hi + k * 1024, 4096);
            const uint32_t accumulate = (kb | k) ? 1u : 0u;
            if (MODE == 3) {
              const uint64_t da_lo = umma_desc_k_sw128(sa_lo + k * 32), db_lo = umma_desc_mn_sw128_32b(sb_lo + k * 1024, 4096);
              umma_tf32(tmem_base, da_lo, db_hi, idesc, accumulate);
              umma_tf32<A_KEEP>(tmem_base, da_hi, db_lo, idesc, 1u);
              umma_tf32<A_KEPT>(tmem_base, da_hi, db_hi, idesc, 1u);
            } else {
              umma_tf32(tmem_base, da_hi, db_hi, idesc, accumulate);
            }
          }
          umma_commit(smem_u32(&empty_bar[stage]));
          if (++stage == STAGES) {
            stage = 0;
            phase ^= 1u;
          }
        }
        if (ok) umma_commit(smem_u32(done_bar));
      }
    }
    __syncwarp();
    if constexpr (in_cluster) {
      cluster_arrive_relaxed();
      cluster_wait();
    }
  }

  tc_fence_before_sync();
  __syncthreads();
  if constexpr (in_cluster) {  // no block retires while others read its partial sums
    cluster_arrive_relaxed();
    cluster_wait();
  }
  if (warp == CONV_WARPS) {
    tc_fence_after_sync();
    tmem_dealloc(tmem_base, BN);
  } else if (VEC && warp < CONV_WARPS && elect_one()) {
    bulk_wait_read<0>();  // the epilogue's tiles outlive the stores that read them
  }
}

}  // namespace sb200
