// float32 GEMM on the FP32 pipes (no TF32): C[M,N] = A[M,K] * W[N,K]^T + bias.  Large matrices go to the tensor cores
// (gemm_f32_tc.cu); what follows is for the others and for operands that its copies cannot take.
//
// The order of a sum.  K is cut into `ranks` ranges of as many 32-wide blocks each (the last ones may have
// fewer, or none), a number that follows from N and K alone (f32_ranks); in a range the products of even k
// and those of odd k are added up one after the other (the two halves of a packed fma.rn.f32x2), the two sums
// are added, and the ranges' sums are added in the order of the ranges.  That is the same for every tile shape
// below, so a row's result does not depend on M or on where the row sits in the batch; and as 2 * ranks
// shorter chains it is nearer the exact sum than one chain of K.
//
// How the work is cut.  A CTA makes BM x BN outputs over one range of K; the CTAs of the ranges are a
// thread-block cluster, which adds up its tiles through distributed shared memory, each CTA a slice of
// them.  A thread makes TM x TN outputs.  Both operands stay K-major in shared memory, as cp.async brings
// them, at a pitch of 36 floats: eight lanes that read 16 bytes of eight rows in a row hit all banks once.
// Pairs along k need no transposed tile and no duplicated operand.
//   TM 2 ... 10, TN 8 or 4 (9 rows and more): bound by the FP32 pipes and by what two CTAs an SM can hide of
//   the loads' latency.  TM + TN loads of 16 bytes for 2 TM TN packed FMAs; the weights of the next four k
//   are read under the products of these (232 -> 211 us for 153 x 17,920 x 1,536 launched alone).
//   One lane row of 4 or 8 rows (up to eight): bound by the weights' bytes; the rows of A are broadcasts.
// Weight tiles are asked for before the programmatic-dependency wait.
//
// Measured (us back to back in a graph; before: one 64 x 64 tile a CTA, 4 x 4 outputs a thread, K in one chain):
//   153 rows: 17,920 x 1,536 504 -> 197 (43 TFLOP/s), 1,536 x 8,960 657 -> 128, 2,048 x 1,536 120 -> 31;
//   4 rows: 702 -> 17.5 (1,536 x 8,960), 1,063 -> 159 (151,936 x 1,536, 5.9 TB/s);
//   2,048 rows: 17,920 x 1,536 4,390 -> 2,515, 1,152 x 896 207 -> 143.
// Error against 64 bits (2-norm, normal operands): 7.0e-7 -> 5.0e-7 with one range of 1,536, 1.9e-7 with
// eight; 1.7e-6 -> 4.3e-7 with 8,960 in eight.
#include "gemm_f32.cuh"

#include "common.cuh"

namespace vx {

constexpr int F32_BK = 32;
constexpr int F32_PITCH = F32_BK + 4;
constexpr int F32_MAX_RANKS = 8;

__device__ __forceinline__ void f32_copy16(uint32_t dst, const float* src, bool valid) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst), "l"(src), "r"(valid ? 16 : 0) : "memory");
}
__device__ __forceinline__ void f32_copy4(uint32_t dst, const float* src, bool valid) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;" ::"r"(dst), "l"(src), "r"(valid ? 4 : 0) : "memory");
}

// Rows [row0, row0 + ROWS) x columns [k0, k0 + 32) of a [rows, K] matrix into shared memory, zeros beyond it.
template <int ROWS, int THREADS, bool VEC>
__device__ __forceinline__ void f32_load_tile(uint32_t dst, const float* __restrict__ src, int row0, int rows, int k0, int K) {
  constexpr int PER_ROW = VEC ? F32_BK / 4 : F32_BK;
#pragma unroll
  for (int i = 0; i < (ROWS * PER_ROW + THREADS - 1) / THREADS; ++i) {
    const int item = i * THREADS + threadIdx.x;
    if ((ROWS * PER_ROW) % THREADS != 0 && item >= ROWS * PER_ROW) break;
    const int r = item / PER_ROW, c = (item % PER_ROW) * (VEC ? 4 : 1);
    const bool valid = row0 + r < rows && k0 + c < K;
    const float* from = valid ? src + (size_t)(row0 + r) * K + k0 + c : src;
    const uint32_t to = dst + (r * F32_PITCH + c) * 4;
    if (VEC)
      f32_copy16(to, from, valid);
    else
      f32_copy4(to, from, valid);
  }
}

__device__ __forceinline__ void f32_fma2(unsigned long long& acc, unsigned long long a, unsigned long long b) {
  asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(acc) : "l"(a), "l"(b));
}

// LM x (32 / LM) lanes of a warp, WM x WN warps, TM x TN outputs a thread.
template <int LM, int WM, int WN, int TM, int TN, int STAGES_, bool VEC_>
struct F32Tile {
  static constexpr int LN = 32 / LM, THREADS = 32 * WM * WN, STAGES = STAGES_;
  static constexpr int BM = LM * WM * TM, BN = LN * WN * TN;
  static constexpr int lanes_m = LM, warps_m = WM, warps_n = WN, thread_m = TM, thread_n = TN;
  static constexpr bool VEC = VEC_;
  static constexpr int STAGE_FLOATS = (BM + BN) * F32_PITCH;
  static constexpr int SUM_PITCH = BN + 4;
  static constexpr size_t SMEM = sizeof(float) * (STAGES * STAGE_FLOATS > BM * SUM_PITCH ? STAGES * STAGE_FLOATS : BM * SUM_PITCH);
};

// ROW: C's rows are that long rather than N (a launch that makes some of the columns).
template <typename S, bool ROW>
__global__ void __launch_bounds__(S::THREADS, 2)
gemm_f32_kernel(const float* __restrict__ A, const float* __restrict__ W, const float* __restrict__ bias,
                float* __restrict__ C, int M, int N, int K, int ranks, int blocks_per_rank, int row) {
  allow_dependents();
  extern __shared__ __align__(16) float f32_smem[];
  constexpr int TM = S::thread_m, TN = S::thread_n, STAGES = S::STAGES;
  constexpr int STEP_M = S::lanes_m * S::warps_m, STEP_N = S::LN * S::warps_n;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  // Neighbouring lanes read the same weights, and a quarter of a warp two rows of A: a 16-byte read of a
  // warp then takes two passes over the banks where lanes 0 ... 7 with eight rows took four.
  const int lane_m = S::lanes_m == 4 ? (lane & 1) | ((lane >> 4) << 1) : lane / S::LN;
  const int lane_n = S::lanes_m == 4 ? (lane >> 1) & 7 : lane % S::LN;
  const int row_m = (warp % S::warps_m) * S::lanes_m + lane_m;
  const int row_n = (warp / S::warps_m) * S::LN + lane_n;
  // x: the ranges of K, so that a cluster is one output tile; y: tiles of N; z: tiles of M.
  const int rank = blockIdx.x;
  const int n0 = blockIdx.y * S::BN, m0 = blockIdx.z * S::BM;
  const int block0 = rank * blocks_per_rank;
  const int blocks = max(0, min(blocks_per_rank, (K + F32_BK - 1) / F32_BK - block0));
  const uint32_t smem = smem_u32(f32_smem);

  const auto load_w = [&](int b) {
    f32_load_tile<S::BN, S::THREADS, S::VEC>(smem + ((b % STAGES) * S::STAGE_FLOATS + S::BM * F32_PITCH) * 4, W, n0, N,
                                             (block0 + b) * F32_BK, K);
  };
  const auto load_a = [&](int b) {
    f32_load_tile<S::BM, S::THREADS, S::VEC>(smem + (b % STAGES) * S::STAGE_FLOATS * 4, A, m0, M, (block0 + b) * F32_BK, K);
  };
#pragma unroll
  for (int b = 0; b < STAGES - 1; ++b)
    if (b < blocks) load_w(b);
  grid_dependency_wait();
  // (The first group holds all weight tiles asked for so far.)
#pragma unroll
  for (int b = 0; b < STAGES - 1; ++b) {
    if (b < blocks) load_a(b);
    asm volatile("cp.async.commit_group;" ::: "memory");
  }

  unsigned long long acc[TM][TN];
#pragma unroll
  for (int i = 0; i < TM; ++i)
#pragma unroll
    for (int j = 0; j < TN; ++j) acc[i][j] = 0ull;

  for (int b = 0; b < blocks; ++b) {
    asm volatile("cp.async.wait_group %0;" ::"n"(STAGES - 2) : "memory");
    __syncthreads();
    if (b + STAGES - 1 < blocks) {
      load_w(b + STAGES - 1);
      load_a(b + STAGES - 1);
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
    const float* as = f32_smem + (b % STAGES) * S::STAGE_FLOATS + row_m * F32_PITCH;
    const float* ws = f32_smem + (b % STAGES) * S::STAGE_FLOATS + (S::BM + row_n) * F32_PITCH;
    // The weights of the next four k are read under this step's products.
    ulonglong2 w[2][TN];
#pragma unroll
    for (int j = 0; j < TN; ++j) w[0][j] = *reinterpret_cast<const ulonglong2*>(ws + j * STEP_N * F32_PITCH);
#pragma unroll
    for (int step = 0; step < F32_BK / 4; ++step) {
      const int k = step * 4, now = step & 1;
      if (step + 1 < F32_BK / 4) {
#pragma unroll
        for (int j = 0; j < TN; ++j) w[now ^ 1][j] = *reinterpret_cast<const ulonglong2*>(ws + j * STEP_N * F32_PITCH + k + 4);
      }
#pragma unroll
      for (int i = 0; i < TM; ++i) {
        const ulonglong2 a = *reinterpret_cast<const ulonglong2*>(as + i * STEP_M * F32_PITCH + k);
#pragma unroll
        for (int j = 0; j < TN; ++j) f32_fma2(acc[i][j], a.x, w[now][j].x);
#pragma unroll
        for (int j = 0; j < TN; ++j) f32_fma2(acc[i][j], a.y, w[now][j].y);
      }
    }
  }
  const auto sum_of = [&](int i, int j) {
    return __uint_as_float((uint32_t)acc[i][j]) + __uint_as_float((uint32_t)(acc[i][j] >> 32));
  };

  if (ranks == 1) {
#pragma unroll
    for (int j = 0; j < TN; ++j) {
      const int n = n0 + row_n + j * STEP_N;
      if (n >= N) continue;
      const float add = bias ? bias[n] : 0.f;
#pragma unroll
      for (int i = 0; i < TM; ++i) {
        const int m = m0 + row_m + i * STEP_M;
        if (m < M) C[(size_t)m * (ROW ? row : N) + n] = sum_of(i, j) + add;
      }
    }
    return;
  }
  // Every CTA lays its tile down in its shared memory; then each adds up its share of the elements.
  asm volatile("cp.async.wait_all;" ::: "memory");
  __syncthreads();
#pragma unroll
  for (int i = 0; i < TM; ++i)
#pragma unroll
    for (int j = 0; j < TN; ++j) f32_smem[(row_m + i * STEP_M) * S::SUM_PITCH + row_n + j * STEP_N] = sum_of(i, j);
  cluster_meet();
  uint32_t peers[F32_MAX_RANKS];
#pragma unroll
  for (int r = 0; r < F32_MAX_RANKS; ++r) peers[r] = r < ranks ? peer_address(f32_smem, r) : 0u;
  for (int e = rank * S::THREADS + threadIdx.x; e < S::BM * S::BN; e += ranks * S::THREADS) {
    const int m = e / S::BN, n = e % S::BN;
    if (m0 + m >= M || n0 + n >= N) continue;
    float part[F32_MAX_RANKS];
#pragma unroll
    for (int r = 0; r < F32_MAX_RANKS; ++r)
      if (r < ranks)
        asm volatile("ld.shared::cluster.f32 %0, [%1];" : "=f"(part[r]) : "r"(peers[r] + (m * S::SUM_PITCH + n) * 4) : "memory");
    float total = part[0];
#pragma unroll
    for (int r = 1; r < F32_MAX_RANKS; ++r)
      if (r < ranks) total += part[r];
    C[(size_t)(m0 + m) * N + n0 + n] = total + (bias ? bias[n0 + n] : 0.f);
  }
  cluster_meet();  // nobody leaves while a peer reads its tile
}

// Ranges of K: enough CTAs of 64 weight rows for two on every SM of a 148-SM device, as long as that is two
// 32-wide blocks a range on average.  A range has as many whole blocks as the mean rounded up, so less is left for
// the last ones (28 blocks in eight ranges: seven of four and an empty one).  From N and K alone: the order of
// a sum must not depend on anything else.
inline int f32_ranks(int N, int K) {
  const int tiles = (N + 63) / 64, blocks = (K + F32_BK - 1) / F32_BK;
  int ranks = 1;
  while (ranks < F32_MAX_RANKS && tiles * ranks < 256 && blocks >= ranks * 4) ranks *= 2;
  return ranks;
}

template <typename S>
int launch_gemm_f32(const float* A, const float* W, const float* bias, float* C, int M, int N, int K, cudaStream_t stream) {
  static const cudaError_t ready =
      cudaFuncSetAttribute(gemm_f32_kernel<S, false>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)S::SMEM);
  if (ready != cudaSuccess) return (int)ready;
  const int ranks = f32_ranks(N, K);
  const int blocks = (K + F32_BK - 1) / F32_BK;
  const dim3 grid(ranks, (N + S::BN - 1) / S::BN, (M + S::BM - 1) / S::BM);
  if (ranks == 1)
    launch_pdl(gemm_f32_kernel<S, false>, grid, dim3(S::THREADS), S::SMEM, stream, A, W, bias, C, M, N, K, ranks, blocks, N);
  else
    launch_pdl_cluster(gemm_f32_kernel<S, false>, grid, dim3(S::THREADS), S::SMEM, ranks, stream, A, W, bias, C, M, N, K, ranks,
                       (blocks + ranks - 1) / ranks, N);
  return (int)cudaGetLastError();
}

// More weight rows than a grid has tiles in y, 65,535 of 64: one launch after the other.
template <typename S>
int launch_gemm_f32_parts(const float* A, const float* W, const float* bias, float* C, int M, int N, int K, cudaStream_t stream) {
  static const cudaError_t ready =
      cudaFuncSetAttribute(gemm_f32_kernel<S, true>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)S::SMEM);
  if (ready != cudaSuccess) return (int)ready;
  const int blocks = (K + F32_BK - 1) / F32_BK;
  constexpr int MOST = 65535 * S::BN;
  for (long long n = 0; n < N; n += MOST) {
    const int part = (int)(N - n < MOST ? N - n : MOST);
    launch_pdl(gemm_f32_kernel<S, true>, dim3(1, (part + S::BN - 1) / S::BN, (M + S::BM - 1) / S::BM), dim3(S::THREADS), S::SMEM,
               stream, A, W + (size_t)n * K, bias ? bias + n : nullptr, C + n, M, part, K, 1, blocks, N);
  }
  return (int)cudaGetLastError();
}

}  // namespace vx

using namespace vx;

// Tiles of 2 x 2 warps of 4 x 8 lanes: 8 TM rows x 16 TN weight rows.
template <int TM, int TN, bool VEC = true>
using F32Square = F32Tile<4, 2, 2, TM, TN, 3, VEC>;

template <int TM>
int launch_square(int tn, const float* A, const float* W, const float* bias, float* C, int M, int N, int K, cudaStream_t s) {
  return tn == 8 ? launch_gemm_f32<F32Square<TM, 8>>(A, W, bias, C, M, N, K, s)
                 : launch_gemm_f32<F32Square<TM, 4>>(A, W, bias, C, M, N, K, s);
}

VX_API long long vx_gemm_f32_scratch(const float* A, const float* W, int M, int N, int K, int tile) {
  return tile == 0 && M > 0 && N > 0 && gemm_f32_tc_takes(A, W, N, K) ? gemm_f32_tc_scratch(M, K) : 0;
}

// tile: 16 TM + TN of the tile to take (every one sums alike), 0: the one that takes least.
// scratch: vx_gemm_f32_scratch bytes, 16-byte aligned, or null where that says zero.  status: the device status word, or null.
VX_API int vx_gemm_f32(const float* A, const float* W, const float* bias, float* C, int M, int N, int K, int tile, void* scratch,
                       int* status, cudaStream_t stream) {
  if (M <= 0 || N <= 0) return 0;
  if (tile == 0 && gemm_f32_tc_takes(A, W, N, K)) return gemm_f32_tc(A, W, bias, C, M, N, K, scratch, status, stream);
  if (N > 65535 * 64) return launch_gemm_f32_parts<F32Square<4, 4, false>>(A, W, bias, C, M, N, K, stream);
  // Rows that 16-byte copies cannot take: odd inner sizes, operands that start between.
  if (K % 4 != 0 || ((uintptr_t)A | (uintptr_t)W) % 16 != 0) {
    // Tiles of 64 x 128 for many rows, where those of 32 x 64 are 1,024 CTAs and more (us with the small and the large
    // ones: 2,048 x 1,537 at 260 rows 106 and 92, at 1,024 364 and 276; 9,729 x 898 at 260 rows 217 and 212, at 153
    // 127 and 142; 200 x 301 at 2,048 rows, 1,024 CTAs, 28.3 and 21.2, at 1,024, 512 CTAs, 15.5 and 17.8).
    const bool many = M >= 256 && (long long)f32_ranks(N, K) * ((N + 63) / 64) * ((M + 31) / 32) >= 1024;
    if (tile == 0) tile = many ? 16 * 8 + 8 : 16 * 4 + 4;
    if (tile == 16 * 4 + 4) return launch_gemm_f32<F32Square<4, 4, false>>(A, W, bias, C, M, N, K, stream);
    if (tile == 16 * 8 + 8) return launch_gemm_f32<F32Square<8, 8, false>>(A, W, bias, C, M, N, K, stream);
    return (int)cudaErrorInvalidValue;
  }
  int best_tm = tile / 16, best_tn = tile % 16;
  if (tile == 0) {
    if (M <= 4) return launch_gemm_f32<F32Tile<1, 1, 2, 4, 1, 6, true>>(A, W, bias, C, M, N, K, stream);
    if (M <= 8) return launch_gemm_f32<F32Tile<1, 1, 2, 8, 1, 6, true>>(A, W, bias, C, M, N, K, stream);
    // The tile whose launch takes least.  A CTA's time goes with TN (TM + 2.3) (measured with 3 ... 10 rows a
    // thread and 4 and 8 weight rows, 17,920 x 1,536 at 153 and 260 rows; within 5 %), two share an SM, and one
    // that has it alone takes three quarters of what two take.  The device holds about 256 CTAs of clusters at
    // a time (whole clusters in a GPC).  Over the projections of the 0.5B and 1.5B sizes at 12 ... 2,048 rows the
    // choice takes as long as the best of the tiles within 10 % in 60 of 70 cases, 26 % longer at most (1,152 x 896 at 100 rows).
    const long long ranks = f32_ranks(N, K);
    double best = 1e300;
    for (int tm : {2, 3, 4, 5, 6, 7, 8, 10})
      for (int tn : {8, 4}) {
        const long long ctas = ranks * ((N + 16 * tn - 1) / (16 * tn)) * ((M + 8 * tm - 1) / (8 * tm));
        double turns = ctas <= 148 ? 1.5 : (double)((ctas + 147) / 148);
        if (ranks > 1) {
          const long long rest = ctas % 256;
          turns = 2.0 * (double)(ctas / 256) + (rest == 0 ? 0.0 : rest <= 148 ? 1.5 : 2.0);
        }
        const double cost = turns * tn * (tm + 2.3 + (tm == 10 ? 0.8 : 0.0));
        if (cost < best) best = cost, best_tm = tm, best_tn = tn;
      }
  }
  if (best_tn != 4 && best_tn != 8) return (int)cudaErrorInvalidValue;
  switch (best_tm) {
    case 2: return launch_square<2>(best_tn, A, W, bias, C, M, N, K, stream);
    case 3: return launch_square<3>(best_tn, A, W, bias, C, M, N, K, stream);
    case 4: return launch_square<4>(best_tn, A, W, bias, C, M, N, K, stream);
    case 5: return launch_square<5>(best_tn, A, W, bias, C, M, N, K, stream);
    case 6: return launch_square<6>(best_tn, A, W, bias, C, M, N, K, stream);
    case 7: return launch_square<7>(best_tn, A, W, bias, C, M, N, K, stream);
    case 8: return launch_square<8>(best_tn, A, W, bias, C, M, N, K, stream);
    case 10: return launch_square<10>(best_tn, A, W, bias, C, M, N, K, stream);
    default: return (int)cudaErrorInvalidValue;
  }
}
