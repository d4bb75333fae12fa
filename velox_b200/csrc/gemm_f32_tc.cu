// float32 GEMM on the tensor cores, for large matrices: C[M,N] = A[M,K] * W[N,K]^T + bias with the accuracy of
// the FP32 pipes (gemm_f32.cu, which keeps the small ones).
//
// The numbers.  A float32 is the sum of three bfloat16 numbers, the value rounded, what that left rounded, and
// what both left (8 + 8 + 8 bits and their signs: nothing is lost unless the third is below 2^-133).  Of the nine
// products of two such sums the six of order 2^-16 and above are taken, each exact in the tensor core's
// float32 accumulator; what is left out is below 2^-24 of the product (two of up to 2^-25).  The accumulator does not
// round to nearest, so sums do not grow in it: a chunk of 32 of the inner dimension is made there, smallest
// products first, and added to the running sum in registers, which is an ordinary float32 addition.
// A sum that is not finite, or below 2^-96, is made again by FMAs from the operands (infinities have no such split, and the
// third terms of tiny operands are lost).
//
// Error against 64 bits (2-norm, normal operands): 9.5e-8 with K 512 (the FMA chains of gemm_f32.cu 2.9e-7), 1.4e-7 with 1,536
// (5.0e-7), 1.4e-7 with 8,960 in eight ranges (4.3e-7); operands of one sign 0.8e-7 - 1.2e-7 (0.9e-7 - 3.0e-7).  A sum that one or
// two products carry is up to 1.4e-7 off (6.0e-8): the accumulator cuts off where an FMA rounds.
//
// The order of a sum is a matter of N and K alone: K is cut into `ranks` ranges (f32_tc_ranks), the chunks of
// a range are added one after the other, and the ranges in their order.  A row's bits do not depend on M or
// on where the row sits in the batch.
//
// How the work is cut.  128 weight rows are the M side of the MMA, the rows of A (tokens) its N side, BN at a
// time.  A CTA makes whole tiles over its range of K; the CTAs of the ranges are a cluster, which adds up its
// tiles through distributed shared memory; without ranges a CTA goes on to its next tile, weights under way.
//   warp 0       TMA producer: weight tiles [128 x 32] float32 into a ring, 128-byte swizzle
//   warp 1       MMA issuer, owns tensor memory: twelve instructions a chunk
//   then two or four groups of four warps, a chunk each in turn: split the weights from shared memory into tensor memory
//                (the A operand: a thread has one row); up to 16 rows of A also those, from global memory, asked for a
//                turn ahead, into the three B tiles in shared memory (64-byte swizzle)
//   then eight or four warps: add the chunks up, a chunk in one of two accumulators while the next is made
//   last         more than 16 rows of A: they come split (f32_split_kernel, a launch of its own: every CTA would split
//                all of them again), three tensor-map copies a chunk
#include <map>
#include <mutex>
#include <tuple>

#include "gemm_f32.cuh"
#include "tensor_core.cuh"

namespace vx {

constexpr int FT_BK = 32;                // of the inner dimension in a chunk: one 128-byte row of float32
constexpr int FT_TERMS = 3;              // bfloat16 numbers to a float32
constexpr int FT_A_COLS = FT_TERMS * FT_BK / 2;  // columns of tensor memory of a chunk's weights, two bf16 to a column
constexpr uint32_t FT_W_BYTES = UMMA_M * FT_BK * 4;
constexpr int FT_MAX_RANKS = 8;
constexpr int FT_PITCH = UMMA_M + 4;     // of a token's row in the exchange
constexpr int FT_LAUNCH_ROWS = 8000;     // rows of A at a time: bounds the scratch, and the grid of clusters (at most 56 tiles of W)

template <int BN_>
struct F32Tensor {
  static constexpr int BN = BN_;
  static constexpr bool SPLIT = BN <= 16;  // the rows of A are split here
  // A few rows: the weights' way through the splitting warps bounds a chunk (two groups 0.41 us), and sums are few.
  static constexpr int GROUPS = SPLIT ? 4 : 2, SUM_WARPS = SPLIT ? 4 : 8;
  static constexpr int PART = BN / (SUM_WARPS / 4);  // columns of a summing warp
  static constexpr int FIRST_SUM = 2 + 4 * GROUPS, ROWS_WARP = FIRST_SUM + SUM_WARPS;
  static constexpr int THREADS = 32 * (SPLIT ? ROWS_WARP : ROWS_WARP + 1);
  static constexpr int STAGES = SPLIT ? 8 : 4;  // chunks of split operands
  static constexpr int W_STAGES = BN > 128 ? 6 : 8;
  static constexpr uint32_t TERM_BYTES = BN * FT_BK * 2, X_BYTES = FT_TERMS * TERM_BYTES;
  static constexpr uint32_t A_COL = 2 * BN;
  static constexpr uint32_t COLS = 2 * BN + STAGES * FT_A_COLS <= 256 ? 256 : 512;
  static constexpr size_t SMEM = (size_t)W_STAGES * FT_W_BYTES + STAGES * X_BYTES + 1024;
  static_assert(2 * BN + STAGES * FT_A_COLS <= 512, "tensor memory");
  static_assert((size_t)BN * FT_PITCH * 4 <= (size_t)W_STAGES * FT_W_BYTES + STAGES * X_BYTES, "the exchange");
};

struct F32TensorArgs {
  const float* A;
  const float* W;
  const float* bias;
  float* C;
  int* status;  // or null
  int M, N, K;
  int ranks, chunks_per_rank;
  int m_tiles, items;
};

__device__ __forceinline__ bool ft_wait(uint32_t bar, uint32_t parity, int* status) {
  if (mbar_try_wait(bar, parity)) return true;
  const unsigned long long start = clock64();
  while (!mbar_try_wait(bar, parity)) {
    if (clock64() - start > VX_WAIT_CYCLES) {
      if (status != nullptr) atomicOr(status, VX_STATUS_WAIT_TIMEOUT);
      return false;
    }
  }
  return true;
}

// K-major tile of 64-byte rows, 64-byte swizzle, groups of eight rows 512 bytes apart.
__device__ __forceinline__ uint64_t ft_b_desc(uint32_t smem_addr) {
  return (uint64_t)((smem_addr & 0x3FFFFu) >> 4) | (uint64_t)(512u >> 4) << 32 | (uint64_t)1 << 46 | (uint64_t)4 << 61;
}

__device__ __forceinline__ void ft_mma(uint32_t tmem_d, uint32_t tmem_a, uint64_t b_desc, uint32_t idesc, uint32_t accumulate) {
  asm volatile(
      "{\n"
      ".reg .pred p;\n"
      "setp.ne.b32 p, %4, 0;\n"
      "tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p;\n"
      "}\n"
      ::"r"(tmem_d), "r"(tmem_a), "l"(b_desc), "r"(idesc), "r"(accumulate)
      : "memory");
}

// Two numbers as three pairs of bfloat16, `a` in the lower halves.
__device__ __forceinline__ void ft_split(float a, float b, uint32_t (&out)[FT_TERMS]) {
#pragma unroll
  for (int t = 0; t < FT_TERMS; ++t) {
    asm("cvt.rn.bf16x2.f32 %0, %1, %2;" : "=r"(out[t]) : "f"(b), "f"(a));
    if (t + 1 < FT_TERMS) {
      asm("{\n"
          ".reg .b64 v, p;\n"
          "mov.b64 v, {%0, %1};\n"
          "mov.b64 p, {%2, %3};\n"
          "sub.rn.f32x2 v, v, p;\n"
          "mov.b64 {%0, %1}, v;\n"
          "}"
          : "+f"(a), "+f"(b)
          : "r"(out[t] << 16), "r"(out[t] & 0xffff0000u));
    }
  }
}

// a [rows, K] float32 as its three terms [3][rows][pitch] bfloat16, zeros from K to the pitch; a thread eight numbers.
__global__ void __launch_bounds__(256) f32_split_kernel(const float* __restrict__ a, __nv_bfloat16* __restrict__ out, int rows, int K, int pitch) {
  allow_dependents();
  const int per_row = pitch / 8;
  const long long item = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  grid_dependency_wait();
  if (item >= (long long)rows * per_row) return;
  const int m = (int)(item / per_row), k = (int)(item - (long long)m * per_row) * 8;
  const float4* from = reinterpret_cast<const float4*>(a + (size_t)m * K + k);
  const float4 lo = __ldcg(from), hi = k + 4 < K ? __ldcg(from + 1) : make_float4(0.f, 0.f, 0.f, 0.f);
  uint32_t pair[4][FT_TERMS];
  ft_split(lo.x, lo.y, pair[0]);
  ft_split(lo.z, lo.w, pair[1]);
  ft_split(hi.x, hi.y, pair[2]);
  ft_split(hi.z, hi.w, pair[3]);
#pragma unroll
  for (int t = 0; t < FT_TERMS; ++t)
    *reinterpret_cast<uint4*>(out + ((size_t)t * rows + m) * pitch + k) = make_uint4(pair[0][t], pair[1][t], pair[2][t], pair[3][t]);
}

__device__ __forceinline__ void ft_store16(uint32_t taddr, const uint32_t (&w)[16]) {
  asm volatile(
      "tcgen05.st.sync.aligned.32x32b.x16.b32 [%0], "
      "{%1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, %16};"
      ::"r"(taddr), "r"(w[0]), "r"(w[1]), "r"(w[2]), "r"(w[3]), "r"(w[4]), "r"(w[5]), "r"(w[6]), "r"(w[7]),
        "r"(w[8]), "r"(w[9]), "r"(w[10]), "r"(w[11]), "r"(w[12]), "r"(w[13]), "r"(w[14]), "r"(w[15])
      : "memory");
}

__device__ __forceinline__ void ft_load8(uint32_t taddr, uint32_t (&r)[8]) {
  asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7])
               : "r"(taddr)
               : "memory");
}

// sum += part, two at a time.
__device__ __forceinline__ void ft_add2(float& s0, float& s1, uint32_t p0, uint32_t p1) {
  asm("{\n"
      ".reg .b64 s, p;\n"
      "mov.b64 s, {%0, %1};\n"
      "mov.b64 p, {%2, %3};\n"
      "add.rn.f32x2 s, s, p;\n"
      "mov.b64 {%0, %1}, s;\n"
      "}"
      : "+f"(s0), "+f"(s1)
      : "r"(p0), "r"(p1));
}

// Sums that the split makes.  Not among them: those with infinities or NaN, and those so small that their operands' third
// terms are below bfloat16's smallest number (operands below 2^-109 beside others of up to 2^13 over sqrt(K)).
__device__ __forceinline__ bool ft_regular(float v) {
  const float size = fabsf(v);
  return size <= 3.402823466e38f && (size >= 0x1p-96f || size == 0.f);
}

// Whether a row has a NaN (the whole warp; K is a multiple of four, the row starts at 16 bytes).
__device__ __noinline__ bool ft_has_nan(const float* row, int K) {
  bool found = false;
#pragma unroll 4
  for (int k = (threadIdx.x & 31) * 4; k < K; k += 128) {
    const float4 v = __ldcg(reinterpret_cast<const float4*>(row + k));
    found = found || v.x != v.x || v.y != v.y || v.z != v.z || v.w != v.w;
  }
  return __any_sync(0xffffffffu, found);
}

// A row times a row by FMAs, an order that follows from K alone (the whole warp).
__device__ __noinline__ float ft_dot(const float* a, const float* w, int K) {
  float sum = 0.f;
#pragma unroll 4
  for (int k = (threadIdx.x & 31) * 4; k < K; k += 128) {
    const float4 x = __ldcg(reinterpret_cast<const float4*>(a + k)), y = __ldcg(reinterpret_cast<const float4*>(w + k));
    sum = fmaf(x.x, y.x, fmaf(x.y, y.y, fmaf(x.z, y.z, fmaf(x.w, y.w, sum))));
  }
#pragma unroll
  for (int step = 16; step > 0; step >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, step);
  return sum;
}

// Makes those of 32 elements (row `a` with weight rows `first` on, one a lane) again that `bad` names; the whole warp, every
// lane brings and gets its element.  A NaN in a row or a weight row is an answer without the products; `known` and
// `nans` remember what was found in the weight rows.  (One thread an element, one after the other, took 17.4 ms for 153 rows of
// NaN by 17,920 x 1,536, the FP32 pipes 0.19.)
__device__ __noinline__ float ft_again(const float* a, const float* W, int first, int K, uint32_t bad, uint32_t* known, uint32_t* nans,
                                       float element) {
  const int lane = threadIdx.x & 31;
  const float nan = __int_as_float(0x7fc00000);
  if (ft_has_nan(a, K)) return (bad >> lane & 1u) != 0 ? nan : element;
  for (uint32_t left = bad; left != 0; left &= left - 1) {
    const int at = __ffs((int)left) - 1;
    const float* const w = W + (size_t)(first + at) * K;
    if ((*known >> at & 1u) == 0) {
      *known |= 1u << at;
      if (ft_has_nan(w, K)) *nans |= 1u << at;
    }
    const float sum = (*nans >> at & 1u) != 0 ? nan : ft_dot(a, w, K);
    if (lane == at) element = sum;
  }
  return element;
}

template <typename S>
__global__ void __launch_bounds__(S::THREADS, 1)
gemm_f32_tc_kernel(const __grid_constant__ CUtensorMap map_w, const __grid_constant__ CUtensorMap map_a, F32TensorArgs g) {
  constexpr int BN = S::BN, STAGES = S::STAGES, W_STAGES = S::W_STAGES;
  extern __shared__ __align__(1024) unsigned char smem_raw[];
  __shared__ __align__(8) uint64_t w_full[W_STAGES], w_empty[W_STAGES];
  __shared__ __align__(8) uint64_t ready[STAGES], used[STAGES];  // split operands of a chunk: there, read
  __shared__ __align__(8) uint64_t a_full[STAGES];  // rows that come split
  __shared__ __align__(8) uint64_t acc_full[2], acc_empty[2];
  __shared__ uint32_t tmem_slot;
  allow_dependents();
  const uint32_t smem = (smem_u32(smem_raw) + 1023u) & ~1023u;
  unsigned char* const smem_p = smem_raw + (smem - smem_u32(smem_raw));
  const uint32_t x_base = smem + W_STAGES * FT_W_BYTES;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int rank = blockIdx.x;
  const int chunk0 = rank * g.chunks_per_rank;
  const int chunks = max(0, min(g.chunks_per_rank, (g.K + FT_BK - 1) / FT_BK - chunk0));  // of an item
  const int items = (g.items - (int)blockIdx.y + (int)gridDim.y - 1) / (int)gridDim.y;    // of this CTA
  const int total = items * chunks;
  const auto item_of = [&](int i, int& n0, int& m0) {
    const int item = blockIdx.y + i * gridDim.y;
    n0 = item / g.m_tiles * UMMA_M;
    m0 = item % g.m_tiles * BN;
  };

  if (threadIdx.x == 0) {
    for (int s = 0; s < W_STAGES; ++s) {
      mbar_init(smem_u32(&w_full[s]), 1);
      mbar_init(smem_u32(&w_empty[s]), 4);
    }
    for (int s = 0; s < STAGES; ++s) {
      mbar_init(smem_u32(&ready[s]), 4);
      mbar_init(smem_u32(&used[s]), 1);
      mbar_init(smem_u32(&a_full[s]), 1);
    }
    for (int s = 0; s < 2; ++s) {
      mbar_init(smem_u32(&acc_full[s]), 1);
      mbar_init(smem_u32(&acc_empty[s]), S::SUM_WARPS);
    }
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
  }
  if (warp == 1) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;"
                 ::"r"(smem_u32(&tmem_slot)), "r"(S::COLS)
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  const uint32_t tmem = tmem_slot;

  if (warp == 0) {
    // ---------------------------------------------------------------- weights
    if (lane == 0) {
      int at = 0, item = -1, n0 = 0, m0 = 0, left = 0;
      for (; at < total; ++at, --left) {
        if (left == 0) {
          item_of(++item, n0, m0);
          left = chunks;
        }
        const int s = at % W_STAGES;
        if (at >= W_STAGES && !ft_wait(smem_u32(&w_empty[s]), (uint32_t)(at / W_STAGES - 1) & 1u, g.status)) break;
        mbar_expect_tx(smem_u32(&w_full[s]), FT_W_BYTES);
        tma_load_2d(smem + s * FT_W_BYTES, &map_w, (chunk0 + chunks - left) * FT_BK, n0, smem_u32(&w_full[s]));
      }
      // (Nothing is under way any more when the CTA ends, also after a wait that gave up.)
      for (int i = max(0, at - W_STAGES); i < at; ++i)
        ft_wait(smem_u32(&w_full[i % W_STAGES]), (uint32_t)(i / W_STAGES) & 1u, g.status);
    }
  } else if (warp == 1) {
    // ---------------------------------------------------------------- products
    constexpr uint32_t idesc = umma_instr_desc(BN);
    const bool issues = elect_lane();
    for (int at = 0; at < total; ++at) {
      const int s = at % STAGES;
      bool ok = ft_wait(smem_u32(&ready[s]), (uint32_t)(at / STAGES) & 1u, g.status);
      if (!S::SPLIT && ok) ok = ft_wait(smem_u32(&a_full[s]), (uint32_t)(at / STAGES) & 1u, g.status);
      if (ok && at >= 2) ok = ft_wait(smem_u32(&acc_empty[at & 1]), (uint32_t)(at / 2 - 1) & 1u, g.status);
      if (!__all_sync(0xffffffffu, ok)) break;
      asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
      const uint32_t d = tmem + (uint32_t)(at & 1) * BN, a = tmem + S::A_COL + (uint32_t)s * FT_A_COLS;
      const uint64_t b = ft_b_desc(x_base + s * S::X_BYTES);
      if (issues) {
        // Term i of the weights with term j of the rows, those of order 2^-16 first, both steps of 16.
        const auto product = [&](int i, int j, int k, bool first) {
          ft_mma(d, a + (uint32_t)(i * (FT_BK / 2) + k * 8), b + (uint64_t)((j * S::TERM_BYTES + k * 32) >> 4), idesc, first ? 0u : 1u);
        };
#pragma unroll
        for (int order = FT_TERMS - 1; order >= 0; --order)
#pragma unroll
          for (int i = 0; i <= order; ++i)
#pragma unroll
            for (int k = 0; k < FT_BK / 16; ++k) product(i, order - i, k, order == FT_TERMS - 1 && i == 0 && k == 0);
        umma_commit(smem_u32(&used[s]));
        umma_commit(smem_u32(&acc_full[at & 1]));
      }
      __syncwarp();
    }
  } else if (warp < S::FIRST_SUM) {
    // ---------------------------------------------------------------- split operands
    constexpr int PIECES = (BN * 4 + 127) / 128;  // of eight numbers of a row, to a thread and chunk
    const int group = (warp - 2) >> 2, q = (int)threadIdx.x - 64 - group * 128, quarter = warp & 3;
    const int row = quarter * 32 + lane;
    int item = 0, chunk = group, n0 = 0, m0 = 0;  // of the chunk whose rows are asked for
    while (chunks > 0 && chunk >= chunks) chunk -= chunks, ++item;
    if (total > 0) item_of(item, n0, m0);
    float4 lo[PIECES], hi[PIECES];
    const auto ask = [&]() {
#pragma unroll
      for (int p = 0; p < PIECES; ++p) {
        const int r = (q >> 2) + 32 * p, k = (chunk0 + chunk) * FT_BK + (q & 3) * 8;
        const float* from = g.A + (size_t)(m0 + r) * g.K + k;
        const bool there = r < BN && m0 + r < g.M;
        lo[p] = there && k < g.K ? __ldcg(reinterpret_cast<const float4*>(from)) : make_float4(0.f, 0.f, 0.f, 0.f);
        hi[p] = there && k + 4 < g.K ? __ldcg(reinterpret_cast<const float4*>(from + 4)) : make_float4(0.f, 0.f, 0.f, 0.f);
      }
    };
    if (S::SPLIT) {
      grid_dependency_wait();
      if (group < total) ask();
    }
    for (int at = group; at < total; at += S::GROUPS) {
      const int s = at % STAGES, ws = at % W_STAGES;
      bool ok = at < STAGES || ft_wait(smem_u32(&used[s]), (uint32_t)(at / STAGES - 1) & 1u, g.status);
      if (ok) ok = ft_wait(smem_u32(&w_full[ws]), (uint32_t)(at / W_STAGES) & 1u, g.status);
      if (!__all_sync(0xffffffffu, ok)) break;
      if (S::SPLIT) {
        // The CTA's rows.
        unsigned char* const x_tile = smem_p + W_STAGES * FT_W_BYTES + s * S::X_BYTES;
#pragma unroll
        for (int p = 0; p < PIECES; ++p) {
          const int r = (q >> 2) + 32 * p;
          uint32_t pair[4][FT_TERMS];
          ft_split(lo[p].x, lo[p].y, pair[0]);
          ft_split(lo[p].z, lo[p].w, pair[1]);
          ft_split(hi[p].x, hi[p].y, pair[2]);
          ft_split(hi[p].z, hi[p].w, pair[3]);
          if (BN % 32 == 0 || r < BN) {
            unsigned char* const to = x_tile + r * (FT_BK * 2) + (((q & 3) ^ ((r >> 1) & 3)) << 4);
#pragma unroll
            for (int t = 0; t < FT_TERMS; ++t)
              *reinterpret_cast<uint4*>(to + t * S::TERM_BYTES) = make_uint4(pair[0][t], pair[1][t], pair[2][t], pair[3][t]);
          }
        }
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
        if (at + S::GROUPS < total) {
          chunk += S::GROUPS;
          if (chunk >= chunks) {
            while (chunk >= chunks) chunk -= chunks, ++item;
            item_of(item, n0, m0);
          }
          ask();
        }
      }
      // A weight row a thread.
      const unsigned char* const w_row = smem_p + ws * FT_W_BYTES + row * (FT_BK * 4);
      uint32_t terms[FT_TERMS][FT_BK / 2];
#pragma unroll
      for (int c = 0; c < FT_BK / 4; ++c) {
        const float4 v = *reinterpret_cast<const float4*>(w_row + ((c ^ (row & 7)) << 4));
        uint32_t pair[2][FT_TERMS];
        ft_split(v.x, v.y, pair[0]);
        ft_split(v.z, v.w, pair[1]);
#pragma unroll
        for (int t = 0; t < FT_TERMS; ++t) {
          terms[t][2 * c] = pair[0][t];
          terms[t][2 * c + 1] = pair[1][t];
        }
      }
      const uint32_t to = tmem + ((uint32_t)(quarter * 32) << 16) + S::A_COL + (uint32_t)s * FT_A_COLS;
#pragma unroll
      for (int t = 0; t < FT_TERMS; ++t) ft_store16(to + t * (FT_BK / 2), terms[t]);
      asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
      asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
      __syncwarp();
      if (lane == 0) {
        mbar_arrive(smem_u32(&w_empty[ws]));
        mbar_arrive(smem_u32(&ready[s]));
      }
    }
  } else if (warp == S::ROWS_WARP) {
    // ---------------------------------------------------------------- rows that come split
    if (lane == 0) {
      grid_dependency_wait();
      int at = 0, item = -1, n0 = 0, m0 = 0, left = 0;
      for (; at < total; ++at, --left) {
        if (left == 0) {
          item_of(++item, n0, m0);
          left = chunks;
        }
        const int s = at % STAGES;
        if (at >= STAGES && !ft_wait(smem_u32(&used[s]), (uint32_t)(at / STAGES - 1) & 1u, g.status)) break;
        const uint32_t bar = smem_u32(&a_full[s]), to = x_base + s * S::X_BYTES;
        mbar_expect_tx(bar, S::X_BYTES);
#pragma unroll
        for (int t = 0; t < FT_TERMS; ++t)
          tma_load_2d(to + t * S::TERM_BYTES, &map_a, (chunk0 + chunks - left) * FT_BK, t * g.M + m0, bar);
      }
      for (int i = max(0, at - STAGES); i < at; ++i)
        ft_wait(smem_u32(&a_full[i % STAGES]), (uint32_t)(i / STAGES) & 1u, g.status);
    }
  } else {
    // ---------------------------------------------------------------- sums
    const int quarter = warp & 3, half = (warp - S::FIRST_SUM) >> 2, row = quarter * 32 + lane;
    grid_dependency_wait();  // the rows written below may be what the kernel before still reads
    const uint32_t from = tmem + ((uint32_t)(quarter * 32) << 16) + (uint32_t)(half * S::PART);
    bool ok = true;
    int at = 0;
    for (int i = 0; i < items; ++i) {
      float sum[S::PART];
#pragma unroll
      for (int j = 0; j < S::PART; ++j) sum[j] = 0.f;
      for (int c = 0; c < chunks; ++c, ++at) {
        if (ok) ok = ft_wait(smem_u32(&acc_full[at & 1]), (uint32_t)(at / 2) & 1u, g.status);
        ok = __all_sync(0xffffffffu, ok);
        if (!ok) break;
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        // (As many columns asked for at a time as there are registers for.)
        constexpr int AT_ONCE = S::PART % 16 == 0 ? 16 : 8;
#pragma unroll
        for (int j0 = 0; j0 < S::PART; j0 += AT_ONCE) {
          uint32_t part[AT_ONCE / 8][8];
#pragma unroll
          for (int p = 0; p < AT_ONCE / 8; ++p) ft_load8(from + (uint32_t)((at & 1) * BN + j0 + p * 8), part[p]);
          asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
          for (int j = 0; j < AT_ONCE; j += 2)
            ft_add2(sum[j0 + j], sum[j0 + j + 1], part[j / 8][j % 8], part[j / 8][j % 8 + 1]);
        }
        asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
        __syncwarp();
        if (lane == 0) mbar_arrive(smem_u32(&acc_empty[at & 1]));
      }
      if (!ok) {
#pragma unroll
        for (int j = 0; j < S::PART; ++j) sum[j] = __int_as_float(0x7fc00000);
      }
      int n0, m0;
      item_of(i, n0, m0);
      if (g.ranks > 1) {
        // Every product has been made, so the rings are free: the tile for the cluster, token after token.
        float* const tile = reinterpret_cast<float*>(smem_p);
#pragma unroll
        for (int j = 0; j < S::PART; ++j) tile[(half * S::PART + j) * FT_PITCH + row] = sum[j];
        continue;
      }
      const int n = n0 + row;
      const bool there = n < g.N;
      const float add = g.bias != nullptr && there ? g.bias[n] : 0.f;
      // (What is to be made again is marked by a NaN.)
      bool regular = true;
#pragma unroll
      for (int j = 0; j < S::PART; ++j) {
        const int m = m0 + half * S::PART + j;
        if (m >= g.M || !there) continue;
        const bool good = ft_regular(sum[j]);
        regular = regular && good;
        g.C[(size_t)m * g.N + n] = good ? sum[j] + add : __int_as_float(0x7fc00000);
      }
      if (ok && __any_sync(0xffffffffu, !regular)) {
        uint32_t known = 0, nans = 0;
        for (int j = 0; j < S::PART && m0 + half * S::PART + j < g.M; ++j) {
          const int m = m0 + half * S::PART + j;
          float* const at = g.C + (size_t)m * g.N + n;
          const uint32_t bad = __ballot_sync(0xffffffffu, there && isnan(*at));
          if (bad == 0) continue;
          const float again = ft_again(g.A + (size_t)m * g.K, g.W, n0 + quarter * 32, g.K, bad, &known, &nans, 0.f);
          if ((bad >> lane & 1u) != 0) *at = again + add;
        }
      }
    }
  }
  if (g.ranks > 1) {
    // Each CTA adds up its share of the elements over the ranges.
    __syncwarp();
    cluster_meet();
    grid_dependency_wait();
    int n0, m0;
    item_of(0, n0, m0);
    uint32_t peers[FT_MAX_RANKS];
#pragma unroll
    for (int r = 0; r < FT_MAX_RANKS; ++r) peers[r] = r < g.ranks ? peer_address(smem_p, r) : 0u;
    for (int e = rank * S::THREADS + threadIdx.x; e < BN * UMMA_M; e += g.ranks * S::THREADS) {
      // (A warp has 32 weight rows of one m.)
      const int m = m0 + e / UMMA_M, n = n0 + e % UMMA_M;
      if (m >= g.M) break;
      float part[FT_MAX_RANKS];
#pragma unroll
      for (int r = 0; r < FT_MAX_RANKS; ++r)
        if (r < g.ranks)
          asm volatile("ld.shared::cluster.f32 %0, [%1];"
                       : "=f"(part[r])
                       : "r"(peers[r] + (uint32_t)(e / UMMA_M * FT_PITCH + e % UMMA_M) * 4u)
                       : "memory");
      float sum = part[0];
#pragma unroll
      for (int r = 1; r < FT_MAX_RANKS; ++r)
        if (r < g.ranks) sum += part[r];
      const uint32_t bad = __ballot_sync(0xffffffffu, n < g.N && !ft_regular(sum));
      if (bad != 0) {
        uint32_t known = 0, nans = 0;
        sum = ft_again(g.A + (size_t)m * g.K, g.W, n - lane, g.K, bad, &known, &nans, sum);
      }
      if (n < g.N) g.C[(size_t)m * g.N + n] = sum + (g.bias != nullptr ? g.bias[n] : 0.f);
    }
    cluster_meet();  // nobody leaves while a peer reads its tile
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  if (warp == 1) {
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(S::COLS) : "memory");
  }
}

// [rows, K] float32 in boxes of [128, 32], 128-byte swizzled, or (box_rows given) bfloat16 in boxes of [box_rows, 32],
// 64-byte swizzled.
static bool ft_tensor_map(CUtensorMap* map, const void* base, int rows, int K, int box_rows = 0) {
  static std::map<std::tuple<const void*, int, int, int>, CUtensorMap> cache;
  static std::mutex lock;
  std::lock_guard<std::mutex> guard(lock);
  const auto key = std::make_tuple(base, rows, K, box_rows);
  const auto it = cache.find(key);
  if (it != cache.end()) {
    *map = it->second;
    return true;
  }
  const EncodeTiledFn encode = encode_tiled_fn();
  if (encode == nullptr) return false;
  const bool terms = box_rows != 0;
  const cuuint64_t dims[2] = {(cuuint64_t)K, (cuuint64_t)rows};
  const cuuint64_t strides[1] = {(cuuint64_t)K * (terms ? 2 : 4)};
  const cuuint32_t box[2] = {FT_BK, (cuuint32_t)(terms ? box_rows : UMMA_M)}, elem[2] = {1, 1};
  if (encode(map, terms ? CU_TENSOR_MAP_DATA_TYPE_BFLOAT16 : CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 2, const_cast<void*>(base), dims,
             strides, box, elem, CU_TENSOR_MAP_INTERLEAVE_NONE, terms ? CU_TENSOR_MAP_SWIZZLE_64B : CU_TENSOR_MAP_SWIZZLE_128B,
             CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) != CUDA_SUCCESS)
    return false;
  if (cache.size() > 4096) cache.clear();
  cache[key] = *map;
  return true;
}

// Ranges of K: as many (a power of two) as 112 CTAs of 128 weight rows have, of four chunks and more: of clusters of
// eight a device of 148 SMs holds fourteen or so at a time (2,048 x 1,536 in sixteen of them takes two turns).  From N and
// K alone: the order of a sum must not depend on anything else.
static int f32_tc_ranks(int N, int K) {
  const int tiles = (N + UMMA_M - 1) / UMMA_M, chunks = (K + FT_BK - 1) / FT_BK;
  int ranks = 1;
  while (ranks < FT_MAX_RANKS && tiles * ranks * 2 <= 112 && chunks >= ranks * 8) ranks *= 2;
  return ranks;
}

// Numbers of a row of split rows: 16-byte multiples.
static int f32_tc_pitch(int K) { return (K + 7) / 8 * 8; }

template <int BN>
static int launch_gemm_f32_tc(const CUtensorMap& map, F32TensorArgs g, __nv_bfloat16* terms, cudaStream_t stream) {
  using S = F32Tensor<BN>;
  static const cudaError_t ready =
      cudaFuncSetAttribute(gemm_f32_tc_kernel<S>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)S::SMEM);
  if (ready != cudaSuccess) return (int)ready;
  CUtensorMap map_a = map;
  if (!S::SPLIT) {
    const int pitch = f32_tc_pitch(g.K);
    const long long items = (long long)g.M * (pitch / 8);
    if (terms == nullptr || !ft_tensor_map(&map_a, terms, FT_TERMS * g.M, pitch, BN)) return (int)cudaErrorInvalidValue;
    launch_pdl(f32_split_kernel, dim3((unsigned)((items + 255) / 256)), dim3(256), 0, stream, g.A, terms, g.M, g.K, pitch);
  }
  const int chunks = (g.K + FT_BK - 1) / FT_BK, n_tiles = (g.N + UMMA_M - 1) / UMMA_M;
  g.ranks = f32_tc_ranks(g.N, g.K);
  g.chunks_per_rank = (chunks + g.ranks - 1) / g.ranks;
  g.m_tiles = (g.M + BN - 1) / BN;
  g.items = n_tiles * g.m_tiles;
  if (g.ranks > 1) {
    launch_pdl_cluster(gemm_f32_tc_kernel<S>, dim3(g.ranks, g.items), dim3(S::THREADS), S::SMEM, g.ranks, stream, map, map_a, g);
  } else {
    // As many rounds as one CTA an SM takes, and no more CTAs than those rounds need.
    const int rounds = (g.items + 147) / 148;
    launch_pdl(gemm_f32_tc_kernel<S>, dim3(1, (g.items + rounds - 1) / rounds), dim3(S::THREADS), S::SMEM, stream, map, map_a, g);
  }
  return (int)cudaGetLastError();
}

// Matrices of 12 Mi elements and more, from what both kernels take (us, FP32 pipes -> here): 17,920 x 1,536 23.7 -> 21.8 at one
// row, 35.5 -> 22.1 at eight, 196 -> 48 at 153; 1,536 x 8,960 16.9 -> 16.9, 23.1 -> 17.4, 128 -> 37; 151,936 x 1,536 151 -> 158, 181 -> 159,
// 442 -> 233 at 40.  Smaller ones have too few CTAs of 128 rows for a few rows of A, and a row must have the same bits in every
// step: 9,728 x 896 8.7 -> 12.9 at one row (88 -> 29 at 153), 2,048 x 1,536 4.9 -> 7.4 (31 -> 17).
bool gemm_f32_tc_takes(const float* A, const float* W, int N, int K) {
  return K >= 512 && (long long)N * K >= 12 << 20 && K % 4 == 0 && (((uintptr_t)A | (uintptr_t)W) & 15) == 0;
}

long long gemm_f32_tc_scratch(int M, int K) {
  return M <= 16 ? 0 : (long long)FT_TERMS * (M < FT_LAUNCH_ROWS ? M : FT_LAUNCH_ROWS) * f32_tc_pitch(K) * 2;
}

// One launch: at most FT_LAUNCH_ROWS rows.
static int gemm_f32_tc_rows(const CUtensorMap& map, const F32TensorArgs& g, __nv_bfloat16* terms, cudaStream_t stream) {
  // Rows in as few tiles as take up to 160 each, and those as narrow as they can be.
  const int M = g.M, tiles = (M + 159) / 160, rows = (M + tiles - 1) / tiles;
  if (M <= 16) return launch_gemm_f32_tc<16>(map, g, terms, stream);
  if (rows <= 32) return launch_gemm_f32_tc<32>(map, g, terms, stream);
  if (rows <= 64) return launch_gemm_f32_tc<64>(map, g, terms, stream);
  if (rows <= 96) return launch_gemm_f32_tc<96>(map, g, terms, stream);
  if (rows <= 128) return launch_gemm_f32_tc<128>(map, g, terms, stream);
  return launch_gemm_f32_tc<160>(map, g, terms, stream);
}

int gemm_f32_tc(const float* A, const float* W, const float* bias, float* C, int M, int N, int K, void* scratch, int* status,
                cudaStream_t stream) {
  CUtensorMap map;
  if (!ft_tensor_map(&map, W, N, K)) return (int)cudaErrorInvalidValue;
  // (A launch's first kernel waits for the launch before it, whose split rows lie in the same scratch.)
  for (int m = 0;; m += FT_LAUNCH_ROWS) {
    const bool last = M - m <= FT_LAUNCH_ROWS;
    const F32TensorArgs g = {A + (size_t)m * K, W, bias, C + (size_t)m * N, status, last ? M - m : FT_LAUNCH_ROWS, N, K, 1, 0, 1, 0};
    const int code = gemm_f32_tc_rows(map, g, (__nv_bfloat16*)scratch, stream);
    if (code != 0 || last) return code;
  }
}

}  // namespace vx
