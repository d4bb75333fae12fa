// bfloat16 projections of long steps (more than 256 tokens) on the 5th-generation tensor cores, with what follows a
// projection in its epilogue: Y[T, N] = X[T, K] * W[N, K]^T.
//
// A pair of CTAs (the two SMs of a cluster) makes tiles of 256 weight rows x BN tokens with
// tcgen05.mma.cta_group::2: each holds 128 weight rows and half of the tokens in shared memory, one thread of the
// first CTA issues for both, and each has the sums of its 128 rows for all BN tokens in its tensor memory.
// The pairs are persistent: a pair takes every `pairs`-th item, token tiles first, so that the pairs that run at a
// time share weight rows in the L2; two accumulators (columns 0 and 256), so that a tile is written out while the
// next one is made.
//   warp 0      TMA producer (both CTAs): W [128 x 64] and X [BN / 2 x 64] into a ring of 128-byte-swizzled stages; the
//               copies of both CTAs count on the first one's barrier
//   warp 1      MMA issuer (first CTA); owns the tensor memory
//   warps 2-9   epilogue: a thread has one weight row (output feature) and 16 tokens at a time, four warps every
//               other sixteen
// BN is a multiple of 16 up to 256, chosen so that the tiles come out even over the pairs (choose_tile).
//
// Epilogues:
//   2  out f32 [T, ldy] += acc + bias: a projection straight into the residual stream.  Up to 768 tokens, where the tiles do
//      not come out even over the pairs, K is cut into chunks, each a tile's item of its own that adds its share (the order of
//      those additions is not fixed; with one chunk an element has one addition)
//   3  out bf16 [T, ldy] = silu(gate) * up of W = N gate rows, then N up rows: the tensor map deals the rows in turn, so
//      that neighbouring lanes hold gate and up of a feature and hand each other one of two tokens
//   6  mode 3 with the options of the gated activation (GluArgs of gemm_bf16.cu: biases [2 N], clamps, the sigmoid's slope
//      and bend, a shift of up)
//   5  columns below a bound out bf16 [T, ldy] = acc + bias, the others through xIELU into a second dense buffer
//
// Every wait is bounded; a thread that gives up sets a status bit, and the CTAs still meet at the end and free
// their tensor memory.
// Which products come here is said by gw_pays.  A projection with nothing of this behind it stays with the library: the plain form took 15 us against 12 (2,048 tokens,
// 2048 x 1536), 20 against 15 (536, 4608 x 3584), 25 against 15 (2,048, 896 x 4864), equal at 7168 x 5120; with rotation
// and cache write in the epilogue 29, 40 and 134 us against the library's 12, 15 and 104 and the 4 - 14 us of a kernel behind
// it: a row of the accumulator is a feature, and the cache's and the output's lines are written two bytes a lane and token.
// The reference engine leaves these products to cuBLAS (nn.Linear; src/self_attention.py:32-33, src/mlp.py:9-15 of
// that project) and runs what follows as kernels of their own.
#include <map>
#include <mutex>
#include <tuple>

#include "tensor_core.cuh"

namespace vx {

constexpr int GW_BK = 64;
constexpr int GW_STAGES = 8;             // at most; as many as fit beside each other
constexpr int GW_EPILOGUE_WARPS = 8;
constexpr int GW_THREADS = 32 * (2 + GW_EPILOGUE_WARPS);
constexpr int GW_MAX_BN = 256;
constexpr uint32_t GW_W_BYTES = UMMA_M * GW_BK * 2;
constexpr uint32_t GW_RING_BYTES = 200 * 1024;

struct WideArgs {
  const float* bias;  // [N] or null (mode 3: none; mode 6: [2 N])
  void* out;
  int* status;
  long long ldy;
  int T, N, K;        // modes 3 and 6: N features, 2 N weight rows
  int bn, stages;
  int token_tiles, tiles;
  int chunks, blocks_per_chunk;  // of K (mode 2: every chunk of a tile is an item of its own and adds its share)
  // Mode 5: columns n >= act_from go to act_out [T, act_ld] at n - act_from.
  void* act_out;
  long long act_ld;
  int act_from;
  float a_pos, a_neg;
  // Mode 6.
  float glu_limit, glu_alpha, glu_shift, glu_cubic;
};

__device__ __forceinline__ uint32_t gw_rank() {
  uint32_t rank;
  asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(rank));
  return rank;
}

// The address of a barrier of the pair's first CTA.
__device__ __forceinline__ uint32_t gw_first(uint32_t bar) {
  uint32_t remote;
  asm volatile("mapa.shared::cluster.u32 %0, %1, 0;" : "=r"(remote) : "r"(bar));
  return remote;
}

// Copies into this CTA's shared memory that count on the first CTA's barrier.
__device__ __forceinline__ void gw_load_2d(uint32_t dst, const CUtensorMap* map, int x, int y, uint32_t bar) {
  asm volatile(
      "cp.async.bulk.tensor.2d.cta_group::2.shared::cluster.global.mbarrier::complete_tx::bytes "
      "[%0], [%1, {%2, %3}], [%4];"
      ::"r"(dst), "l"(reinterpret_cast<uint64_t>(map)), "r"(x), "r"(y), "r"(bar)
      : "memory");
}
__device__ __forceinline__ void gw_load_3d(uint32_t dst, const CUtensorMap* map, int x, int y, int z, uint32_t bar) {
  asm volatile(
      "cp.async.bulk.tensor.3d.cta_group::2.shared::cluster.global.mbarrier::complete_tx::bytes "
      "[%0], [%1, {%2, %3, %4}], [%5];"
      ::"r"(dst), "l"(reinterpret_cast<uint64_t>(map)), "r"(x), "r"(y), "r"(z), "r"(bar)
      : "memory");
}
__device__ __forceinline__ void gw_mma(uint32_t tmem_d, uint64_t a_desc, uint64_t b_desc, uint32_t idesc, uint32_t accumulate) {
  asm volatile(
      "{\n"
      ".reg .pred p;\n"
      "setp.ne.b32 p, %4, 0;\n"
      "tcgen05.mma.cta_group::2.kind::f16 [%0], %1, %2, %3, p;\n"
      "}\n"
      ::"r"(tmem_d), "l"(a_desc), "l"(b_desc), "r"(idesc), "r"(accumulate)
      : "memory");
}

// Arrives on the barrier at this offset in both CTAs when the products so far have finished.
__device__ __forceinline__ void gw_commit(uint32_t bar) {
  asm volatile(
      "tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], %1;"
      ::"r"(bar), "h"((uint16_t)3)
      : "memory");
}

__device__ __forceinline__ void gw_load16(uint32_t taddr, float (&v)[16]) {
  uint32_t r[16];
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x16.b32 "
      "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, [%16];"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]),
        "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
      : "r"(taddr)
      : "memory");
  asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
  for (int i = 0; i < 16; ++i) v[i] = __uint_as_float(r[i]);
}

template <int MODE>
__global__ void __launch_bounds__(GW_THREADS, 1)
gemm_bf16_wide_kernel(const __grid_constant__ CUtensorMap map_w, const __grid_constant__ CUtensorMap map_x, const WideArgs g) {
  extern __shared__ __align__(1024) unsigned char smem_raw[];
  __shared__ __align__(8) uint64_t full_bar[GW_STAGES], empty_bar[GW_STAGES];
  __shared__ __align__(8) uint64_t acc_full[2], acc_empty[2];
  __shared__ uint32_t tmem_slot;
  constexpr bool GATED = MODE == 3 || MODE == 6;
  VX_TRACE_SCOPE(40 + MODE);
  allow_dependents();
  const uint32_t smem = (smem_u32(smem_raw) + 1023u) & ~1023u;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const uint32_t rank = gw_rank();
  const int pair = blockIdx.x >> 1, pairs = gridDim.x >> 1;
  const int blocks = (g.K + GW_BK - 1) / GW_BK;
  const uint32_t stage_bytes = GW_W_BYTES + (uint32_t)g.bn * (GW_BK * 2 / 2);
  const int items = (g.tiles * g.chunks - pair + pairs - 1) / pairs;  // of this pair
  // Tile and first block of item i, and its number of blocks.  (All tiles of a chunk before the next chunk.)
  const auto item_of = [&](int i, int& tile, int& first) {
    const int item = pair + i * pairs, chunk = item / g.tiles;
    tile = item - chunk * g.tiles;
    first = chunk * g.blocks_per_chunk;
    return min(g.blocks_per_chunk, blocks - first);
  };

  if (threadIdx.x == 0) {
    for (int s = 0; s < GW_STAGES; ++s) {
      mbar_init(smem_u32(&full_bar[s]), 1);
      mbar_init(smem_u32(&empty_bar[s]), 1);
    }
    for (int b = 0; b < 2; ++b) {
      mbar_init(smem_u32(&acc_full[b]), 1);
      mbar_init(smem_u32(&acc_empty[b]), 2 * GW_EPILOGUE_WARPS);
    }
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
  }
  if (warp == 1) {
    asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&tmem_slot)), "r"(512)
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  cluster_meet();  // the other CTA's barriers are set up
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  const uint32_t tmem = tmem_slot;

  if (warp == 0) {
    // ---------------------------------------------------------------- TMA producer
    if (lane == 0) {
      // Where the walk over the items' blocks is.  (Counted up: a division a block would be on the chain of every stage.)
      struct Place {
        int i, kb, last, stage, phase, w_row, t_row;
      };
      const auto enter = [&](Place& p) {
        int tile;
        p.last = item_of(p.i, tile, p.kb);
        p.last += p.kb;
        const int wt = tile / g.token_tiles;
        p.t_row = (tile - wt * g.token_tiles) * g.bn + (int)rank * (g.bn / 2);
        p.w_row = GATED ? wt * UMMA_M + (int)rank * (UMMA_M / 2) : (wt * 2 + (int)rank) * UMMA_M;
      };
      const auto next = [&](Place& p) {
        if (++p.stage == g.stages) p.stage = 0, p.phase ^= 1;
        if (++p.kb == p.last && ++p.i < items) enter(p);
      };
      const uint32_t own_full = smem_u32(&full_bar[0]), first_full = gw_first(own_full);
      const auto load_w = [&](const Place& p) {
        const uint32_t bar = first_full + p.stage * 8, dst = smem + p.stage * stage_bytes;
        if (rank == 0) mbar_expect_tx(own_full + p.stage * 8, 2 * stage_bytes);
        if (GATED) {
          gw_load_3d(dst, &map_w, p.kb * GW_BK, 0, p.w_row, bar);
        } else {
          gw_load_2d(dst, &map_w, p.kb * GW_BK, p.w_row, bar);
        }
      };
      const auto load_x = [&](const Place& p) {
        gw_load_2d(smem + p.stage * stage_bytes + GW_W_BYTES, &map_x, p.kb * GW_BK, p.t_row, first_full + p.stage * 8);
      };
      // The weights of the first round of stages do not wait for the kernel before this one.
      Place p = {0, 0, 0, 0, 0, 0, 0};
      enter(p);
      Place q = p;
      int total = 0;
      for (int i = 0; i < items; ++i) {
        int tile, kb;
        total += item_of(i, tile, kb);
      }
      const int first = min(total, g.stages);
      for (int at = 0; at < first; ++at, next(p)) load_w(p);
      grid_dependency_wait();
      for (int at = 0; at < first; ++at, next(q)) load_x(q);
      int at = first;
      for (; at < total; ++at, next(p)) {
        if (!mbar_wait(smem_u32(&empty_bar[p.stage]), (uint32_t)p.phase ^ 1u, g.status)) break;
        load_w(p);
        load_x(p);
      }
      // (Nothing is under way any more when the pair ends, also after a wait that gave up.)
      if (rank == 0)
        for (int i = max(0, at - g.stages); i < at; ++i)
          mbar_wait(smem_u32(&full_bar[i % g.stages]), (uint32_t)(i / g.stages) & 1u, g.status);
    }
  } else if (warp == 1) {
    // ---------------------------------------------------------------- MMA issuer
    if (rank == 0) {
      // M = 256 over the pair.
      const uint32_t idesc = (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(g.bn >> 3) << 17) | ((uint32_t)(256 >> 4) << 24);
      const bool issues = elect_lane();
      bool ok = true;
      int s = 0;
      uint32_t phase = 0;
      for (int i = 0; i < items && ok; ++i) {
        const int b = i & 1;
        int tile, first;
        const int count = item_of(i, tile, first);
        if (i >= 2) ok = mbar_wait(smem_u32(&acc_empty[b]), (uint32_t)(i / 2 - 1) & 1u, g.status);
        for (int kb = 0; kb < count; ++kb) {
          if (ok) ok = mbar_wait(smem_u32(&full_bar[s]), phase, g.status);
          ok = __all_sync(0xffffffffu, ok);
          if (!ok) break;
          asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
          const uint64_t a = umma_smem_desc(smem + s * stage_bytes), x = umma_smem_desc(smem + s * stage_bytes + GW_W_BYTES);
          if (issues) {
#pragma unroll
            for (int k = 0; k < GW_BK / 16; ++k)
              gw_mma(tmem + (uint32_t)(b * GW_MAX_BN), a + k * 2, x + k * 2, idesc, kb > 0 || k > 0 ? 1u : 0u);
            gw_commit(smem_u32(&empty_bar[s]));
            if (kb == count - 1) gw_commit(smem_u32(&acc_full[b]));
          }
          __syncwarp();
          if (++s == g.stages) s = 0, phase ^= 1u;
        }
      }
    }
  } else {
    // ---------------------------------------------------------------- epilogue
    grid_dependency_wait();
    const int quarter = warp & 3, part = (warp - 2) >> 2, row = quarter * 32 + lane;
    const bool odd = (row & 1) != 0;
    const uint32_t lane_base = tmem + ((uint32_t)(quarter * 32) << 16);
    bool ok = true;  // (A warp that gave up goes on to the barriers that the others wait at.)
    for (int i = 0; i < items; ++i) {
      int tile, first;
      item_of(i, tile, first);
      const int wt = tile / g.token_tiles, t0 = (tile - wt * g.token_tiles) * g.bn;
      const int b = i & 1;
      const int row0 = (wt * 2 + (int)rank) * UMMA_M;  // of the CTA's rows
      // This thread's output feature.
      int n = row0 + row;
      if (GATED) n = (row0 + row) >> 1;
      const bool mine = n < g.N;
      const float bias = MODE != 3 && g.bias != nullptr && mine && first == 0 ? g.bias[n] : 0.f;  // (mode 6: gate's)
      const float bias_up = MODE == 6 && g.bias != nullptr && mine ? g.bias[g.N + n] : 0.f;
      if (ok) ok = mbar_wait(smem_u32(&acc_full[b]), (uint32_t)(i / 2) & 1u, g.status);
      ok = __all_sync(0xffffffffu, ok);
      if (!ok) continue;
      asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
      for (int c0 = part * 16; c0 < g.bn; c0 += 32) {
        float v[16];
        gw_load16(lane_base + (uint32_t)(b * GW_MAX_BN + c0), v);
        const int t1 = t0 + c0;
        if (t1 >= g.T) break;
        if (MODE == 5) {
          const bool plain = n < g.act_from;
          __nv_bfloat16* const out = plain ? (__nv_bfloat16*)g.out + (size_t)t1 * g.ldy + n
                                           : (__nv_bfloat16*)g.act_out + (size_t)t1 * g.act_ld + (n - g.act_from);
          const long long pitch = plain ? g.ldy : g.act_ld;
#pragma unroll
          for (int j = 0; j < 16; ++j) {
            const float z = v[j] + bias;
            const float bent = z > 0.f ? fmaf(g.a_pos * z, z, 0.5f * z) : fmaf(g.a_neg, (__expf(z) - 1.0f) - z, 0.5f * z);
            if (mine && t1 + j < g.T) out[(size_t)j * pitch] = __float2bfloat16_rn(plain ? z : bent);
          }
        } else if (GATED) {
          __nv_bfloat16* const out = (__nv_bfloat16*)g.out + (size_t)(t1 + (odd ? 1 : 0)) * g.ldy + n;
#pragma unroll
          for (int j = 0; j < 16; j += 2) {
            const float other = __shfl_xor_sync(0xffffffffu, odd ? v[j] : v[j + 1], 1);
            float gate = odd ? other : v[j], up = odd ? v[j + 1] : other;
            float result;
            if (MODE == 3) {
              result = __fdividef(gate, 1.0f + __expf(-gate)) * up;
            } else {
              gate += bias;
              up += bias_up;
              if (g.glu_limit > 0.f) {
                gate = fminf(gate, g.glu_limit);
                up = fminf(fmaxf(up, -g.glu_limit), g.glu_limit);
              }
              const float bent = fmaf(g.glu_cubic * gate, gate * gate, gate);
              result = gate / (1.0f + __expf(-g.glu_alpha * bent)) * (up + g.glu_shift);
            }
            if (mine && t1 + j + (odd ? 1 : 0) < g.T) out[(size_t)j * g.ldy] = __float2bfloat16_rn(result);
          }
        } else {
          float* const out = (float*)g.out + (size_t)t1 * g.ldy + n;
#pragma unroll
          for (int j = 0; j < 16; ++j)
            if (mine && t1 + j < g.T)
              asm volatile("red.global.add.f32 [%0], %1;" ::"l"(out + (size_t)j * g.ldy), "f"(v[j] + bias) : "memory");
        }
      }
      asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
      __syncwarp();
      if (lane == 0)
        asm volatile("mbarrier.arrive.release.cluster.shared::cluster.b64 _, [%0];" ::"r"(gw_first(smem_u32(&acc_empty[b])))
                     : "memory");
    }
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncwarp();
  cluster_meet();  // no products or arrivals of the other CTA are under way here any more
  if (warp == 1) {
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(512) : "memory");
  }
}

// ---------------------------------------------------------------------------------------------
// Host side.
// ---------------------------------------------------------------------------------------------
// A bf16 matrix as a map whose innermost dimension runs along K in boxes of 64: extents, pitches (in elements) and box
// extents of the one or two others.
struct WideMap {
  int dims;
  long long extent[2], pitch[2];
  int box[2];
};

static bool gw_tensor_map(CUtensorMap* map, const void* base, long long K, const WideMap& m) {
  using Key = std::tuple<const void*, long long, int, long long, long long, int, int>;
  static std::map<Key, CUtensorMap> cache;
  static std::mutex lock;
  const Key key{base, K, m.dims, m.extent[0], m.extent[1], m.box[0], m.box[1]};  // (the pitches follow from these)
  std::lock_guard<std::mutex> guard(lock);
  const auto it = cache.find(key);
  if (it != cache.end()) {
    *map = it->second;
    return true;
  }
  const EncodeTiledFn encode = encode_tiled_fn();
  if (encode == nullptr) return false;
  cuuint64_t extent[3] = {(cuuint64_t)K}, pitch[2];
  cuuint32_t box[3] = {GW_BK}, step[3] = {1, 1, 1};
  for (int i = 0; i < m.dims; ++i) {
    extent[i + 1] = (cuuint64_t)m.extent[i];
    pitch[i] = (cuuint64_t)m.pitch[i] * 2;
    box[i + 1] = (cuuint32_t)m.box[i];
  }
  if (encode(map, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, (cuuint32_t)m.dims + 1, const_cast<void*>(base), extent, pitch, box, step,
             CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
             CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) != CUDA_SUCCESS)
    return false;
  if (cache.size() > 4096) cache.clear();
  cache[key] = *map;
  return true;
}

// Pairs of CTAs that the device holds at a time (asked once).
static int gw_pairs() {
  static const int pairs = [] {
    cudaLaunchConfig_t config = {};
    cudaLaunchAttribute attribute[1];
    attribute[0].id = cudaLaunchAttributeClusterDimension;
    attribute[0].val.clusterDim = {2, 1, 1};
    config.gridDim = dim3(2);
    config.blockDim = dim3(GW_THREADS);
    config.dynamicSmemBytes = GW_RING_BYTES + 1024;
    config.attrs = attribute;
    config.numAttrs = 1;
    int found = 0;
    if (cudaFuncSetAttribute(gemm_bf16_wide_kernel<2>, cudaFuncAttributeMaxDynamicSharedMemorySize, GW_RING_BYTES + 1024) !=
            cudaSuccess ||
        cudaOccupancyMaxActiveClusters(&found, gemm_bf16_wide_kernel<2>, &config) != cudaSuccess || found < 1) {
      (void)cudaGetLastError();
      found = 64;
    }
    return found;
  }();
  return pairs;
}

// Tokens of a tile and chunks of K: rounds of items over the pairs times an item's time, in cycles, which is returned.  A block of
// K takes what its operands (16 KB + 64 bn bytes a CTA) take into shared memory, 43 bytes a cycle and SM as measured, which is longer
// than its products at every bn.  Sums into the stream by chunks are bound by the L2's additions where items are short (49 cycles a
// token and pair with all pairs at it); the last item's epilogue is not covered by another's products.  Within a few per cent of
// the best of 5 tiles x 6 numbers of chunks for the projections of the 0.5B to 14B sizes at 260 to 2,048 tokens.
static double choose_tile(int T, int weight_tiles, int blocks, int pairs, int most_chunks, int& bn_out, int& chunks_out) {
  double least = 1e300;
  const bool sums = most_chunks > 1;
  for (int chunks = 1; chunks <= most_chunks; ++chunks)
    for (int bn = GW_MAX_BN; bn >= 32; bn -= 16) {
      const int per = (blocks + chunks - 1) / chunks;
      if (chunks > 1 && per < 8) break;
      const long long items = (long long)weight_tiles * ((T + bn - 1) / bn) * chunks;
      const double busy = items < pairs ? (double)items / pairs : 1.0;
      const double main = per * (381.0 + 1.49 * bn) + 500.0, adds = sums ? 49.0 * bn * busy : 0.0;
      double cost = (double)((items + pairs - 1) / pairs) * (main > adds ? main : adds) + 14.0 * bn + 0.5 * adds;
      if (chunks > 1) cost *= 1.10;  // (one chunk has one order of additions, and the model flatters many)
      if (cost < least) least = cost, bn_out = bn, chunks_out = chunks;
    }
  return least;
}

// Sums of this many tokens at most may cut K: 1,024 tokens of the 14B output projection took 64 us in one chunk and 73 in several,
// 2,048 tokens 89 and 106, of the down projections 214 and 214, 198 and 203 (7B), 46 and 46 (1.5B).
constexpr int GW_CHUNKED_TOKENS = 768;

// Whether a product is better off here than as a library product with the kernel that follows it.  Measured (library -> here, us):
// both in graphs at 26 numbers of tokens between 257 and 6,000 of the 0.5B to 14B sizes, and whole steps, replayed and queued
// launch by launch.  Queued so, steps of the narrower models are bound by the host to about 1.5 Mi numbers of a stream (0.5B 1,755
// tokens, 1.5B 1,024, 3B 768), and a library product with its follower costs the host some 10 us more: there a few us of the
// device's time are given for it.
//   Sums, K the longer side (down), cut into chunks: 257 tokens 0.5B 11 -> 10, 1.5B 18 -> 14, 3B 21 -> 19, 7B 55 -> 44, 14B 63 -> 63; 536 tokens 12 ->
//     13, 21 -> 18, 34 -> 25, 63 -> 62, 73 -> 70.
//   Other sums (in one chunk beyond 768 tokens) pay where the tiles come out even, that is where the cost above leaves the tensor cores 49 % of
//     their time: 2,048 tokens 7B 54 -> 47 (output), 204 -> 198 (down), 14B 97 -> 89, 225 -> 214; from 0.92 to 1.13 times as fast; at 1,400
//     tokens 7B 35 -> 39, 138 -> 172 with 43 %.  Output projections come here where the host is the bound: 300 tokens
//     0.5B 5.8 -> 7.9, 1.5B 7.3 -> 8.6, 3B 8.9 -> 10.0; a step of them replayed takes up to 1 % more, queued 2,582 us where it took 2,830, 2,946
//     where 3,216, 3,695 where 4,053.
//   SwiGLU pays with 47 % (2,048 tokens 1.5B 90 -> 82, 3B 141 -> 122, 7B 379 -> 340; 300 tokens 7B 72 -> 75, 14B 73 -> 77) and K from 1,280 on (0.5B,
//     whose products are too short for the epilogue, at 2,048 tokens 37 -> 44), and where the host is the bound: 300 tokens 0.5B 12 -> 14, 1.5B
//     20 -> 21, 3B 32 -> 31; a 0.5B step of 300 tokens with all of these 3,120 -> 2,582 us queued, 1,181 -> 1,245 replayed.
//   Modes 5 and 6, whose epilogues take longer: 47 % and K from 3,072 on (0.96 to 1.17 times as fast).  K 896 to 2,048 takes 0.66 to
//     1.04: Peratar's 1.5B step of 505 tokens replayed 3,368 -> 3,831, queued 5,132 -> 4,749.
static bool gw_pays(int mode, int T, int N, int K, bool chunked) {
  const int width = mode == 2 ? N : K;
  const bool narrow = width < 3072 && (long long)T * width <= 3 << 19;
  if (mode == 2 && 2LL * K >= 5LL * N ? chunked && T <= GW_CHUNKED_TOKENS : (mode == 2 || mode == 3) && narrow) return true;
  if (K < (mode == 2 ? 2048 : mode == 3 ? 1280 : 3072)) return false;
  const long long rows = mode == 3 || mode == 6 ? 2LL * N : N;
  const int pairs = gw_pairs();
  int bn, chunks;
  const double cycles = choose_tile(T, (int)((rows + 2 * UMMA_M - 1) / (2 * UMMA_M)), (K + GW_BK - 1) / GW_BK, pairs, 1, bn, chunks);
  // (A pair makes 8,192 multiply-adds a cycle.)
  return (double)rows * T * K >= (mode == 2 ? 0.49 : 0.47) * 8192.0 * pairs * cycles;
}

template <int MODE>
static int launch_wide(const CUtensorMap& mw, const CUtensorMap& mx, const WideArgs& g, int pairs, cudaStream_t stream) {
  static const cudaError_t ready =
      cudaFuncSetAttribute(gemm_bf16_wide_kernel<MODE>, cudaFuncAttributeMaxDynamicSharedMemorySize, GW_RING_BYTES + 1024);
  if (ready != cudaSuccess) return (int)ready;
  const int items = g.tiles * g.chunks;
  launch_pdl_cluster(gemm_bf16_wide_kernel<MODE>, dim3(2 * (items < pairs ? items : pairs)), dim3(GW_THREADS),
                     GW_RING_BYTES + 1024, 2, stream, mw, mx, g);
  return (int)cudaGetLastError();
}

static int gemm_bf16_wide(const void* x, int x_rows, const void* w, int mode, WideArgs g, int tokens, int chunks,
                          cudaStream_t stream) {
  const int T = g.T, N = g.N, K = g.K;
  if (T <= 0 || N <= 0) return 0;
  if (K <= 0 || K % 8 != 0 || x_rows < T || (((uintptr_t)x | (uintptr_t)w) & 15) != 0) return -1;
  if (tokens != 0 && (tokens % 16 != 0 || tokens < 16 || tokens > GW_MAX_BN)) return -1;
  const bool gated = mode == 3 || mode == 6;
  const int rows = gated ? 2 * N : N;
  const int weight_tiles = (rows + 2 * UMMA_M - 1) / (2 * UMMA_M), pairs = gw_pairs();
  const int blocks = (K + GW_BK - 1) / GW_BK;
  if (chunks < 0 || (chunks > 1 && mode != 2)) return -1;
  choose_tile(T, weight_tiles, blocks, pairs, chunks == 0 && mode == 2 && T <= GW_CHUNKED_TOKENS ? 8 : 1, g.bn, g.chunks);
  if (tokens != 0) g.bn = tokens;
  if (chunks != 0) g.chunks = chunks < blocks ? chunks : blocks;
  g.blocks_per_chunk = (blocks + g.chunks - 1) / g.chunks;
  g.chunks = (blocks + g.blocks_per_chunk - 1) / g.blocks_per_chunk;  // no empty one
  g.stages = (int)(GW_RING_BYTES / (GW_W_BYTES + (uint32_t)g.bn * GW_BK));
  if (g.stages > GW_STAGES) g.stages = GW_STAGES;
  g.token_tiles = (T + g.bn - 1) / g.bn;
  if ((long long)weight_tiles * g.token_tiles * g.chunks > 1 << 30) return -1;
  g.tiles = weight_tiles * g.token_tiles;
  CUtensorMap mw, mx;
  WideMap wide = {1, {N, 1}, {K, 0}, {UMMA_M, 1}};
  if (gated) wide = {2, {2, N}, {(long long)N * K, K}, {2, UMMA_M / 2}};
  if (!gw_tensor_map(&mw, w, K, wide)) return -1;
  if (!gw_tensor_map(&mx, x, K, WideMap{1, {x_rows, 1}, {K, 0}, {g.bn / 2, 1}})) return -1;
  switch (mode) {
    case 2: return launch_wide<2>(mw, mx, g, pairs, stream);
    case 3: return launch_wide<3>(mw, mx, g, pairs, stream);
    case 5: return launch_wide<5>(mw, mx, g, pairs, stream);
    case 6: return launch_wide<6>(mw, mx, g, pairs, stream);
    default: return -1;
  }
}

}  // namespace vx

using namespace vx;

VX_TRACE_API(vx_wide)

// 1 where a product of a long step is better off here than with a library (mode 2: chunked says whether K may be cut).
VX_API int vx_gemm_bf16_wide_pays(int mode, int T, int N, int K, int chunked) {
  return T > 0 && N > 0 && K > 0 && gw_pays(mode, T, N, K, chunked != 0) ? 1 : 0;
}

// x [x_rows >= T, K] bf16, w [N, K] bf16 (modes 3 and 6: [2 N, K]); see the head of the file for the modes.  tokens: of a
// tile, chunks of K (mode 2): 0 for what takes least.  Return 0 on launch, a cudaError_t on failure, -1 for sizes and
// pointers that the kernel does not take.
VX_API int vx_gemm_bf16_wide(const void* x, int x_rows, const void* w, const float* bias, void* out, int mode, int T, int N, int K,
                             long long ldy, int tokens, int chunks, int* status, cudaStream_t stream) {
  if (mode != 2 && mode != 3) return -1;
  WideArgs g = {};
  g.bias = bias, g.out = out, g.status = status, g.ldy = ldy, g.T = T, g.N = N, g.K = K;
  return gemm_bf16_wide(x, x_rows, w, mode, g, tokens, chunks, stream);
}

// Mode 6.
VX_API int vx_gemm_bf16_wide_glu(const void* x, int x_rows, const void* w, const float* bias, void* out, int T, int N, int K,
                                 long long ldy, int tokens, float limit, float alpha, float shift, float cubic, int* status,
                                 cudaStream_t stream) {
  WideArgs g = {};
  g.bias = bias, g.out = out, g.status = status, g.ldy = ldy, g.T = T, g.N = N, g.K = K;
  g.glu_limit = limit, g.glu_alpha = alpha, g.glu_shift = shift, g.glu_cubic = cubic;
  return gemm_bf16_wide(x, x_rows, w, 6, g, tokens, 1, stream);
}

// Mode 5.
VX_API int vx_gemm_bf16_wide_xielu(const void* x, int x_rows, const void* w, const float* bias, void* out, void* act_out, int T,
                                   int N, int K, long long ldy, long long act_ld, int act_from, int tokens, float a_pos,
                                   float a_neg, int* status, cudaStream_t stream) {
  if (act_out == nullptr || act_from < 0 || act_from > N) return -1;
  WideArgs g = {};
  g.bias = bias, g.out = out, g.status = status, g.ldy = ldy, g.T = T, g.N = N, g.K = K;
  g.act_out = act_out, g.act_ld = act_ld, g.act_from = act_from, g.a_pos = a_pos, g.a_neg = a_neg;
  return gemm_bf16_wide(x, x_rows, w, 5, g, tokens, 1, stream);
}
