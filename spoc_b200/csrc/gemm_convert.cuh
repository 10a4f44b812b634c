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
