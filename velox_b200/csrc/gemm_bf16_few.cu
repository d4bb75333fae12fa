// bfloat16 projections of up to sixteen tokens whose matrix is a small one: Y[T, N] = X[T, K] * W[N, K]^T.
//
// What bounds such a launch is not bytes (the QKV and output matrices of the 0.5B to 1.5B sizes are read in a
// microsecond) but the chain behind the kernel before it.  So the chain is made short.  A CTA makes 16 rows of W; its
// warps share K in blocks of 32, interleaved, and every warp asks for all its weights at once, into registers, before
// the dependency wait.  Behind the wait there are left: one round of loads of X (a lane's values are the B fragments of
// its products as they lie in memory: the order of K inside a block is the same on both sides and of no consequence),
// some mma.sync of 16 x 8 x 16, one exchange through shared memory and the output.  No ring, no barriers of copies, no
// cluster, no trip through tensor memory.
//
// The input norm (resid given): X = bf16(resid * norm_w), sums of squares beside it, 1 / rms on the finished sum, as
// in gemm_bf16.cu.  The order of a sum is fixed.
//
// Modes (as in gemm_bf16.cu): 0 bf16 + bias, 1 float32 + bias, 2 float32 += (and a copy of the sums), 4 q | k | v of
// whole heads with rotation and cache write: a tile is eight pairs (d, d + half a head).  With the norm inside: 4 only.
#include "common.cuh"
#include "gemm_bf16_few.cuh"

namespace vx {

constexpr int FEW_ROWS = 16;
constexpr int FEW_BLOCK = 32;  // of K: 16 bytes of a row to a lane

__device__ __forceinline__ uint4 few_load_weights(const void* p) {
  uint4 v;
  asm volatile("ld.global.nc.L1::no_allocate.L2::256B.v4.u32 {%0, %1, %2, %3}, [%4];"
               : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w)
               : "l"(p));
  return v;
}

__device__ __forceinline__ uint32_t few_pack(float a, float b) {
  const __nv_bfloat162 p = __floats2bfloat162_rn(a, b);
  return *reinterpret_cast<const uint32_t*>(&p);
}

__device__ __forceinline__ void few_mma(float (&d)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0, uint32_t b1) {
  asm volatile(
      "mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, {%0, %1, %2, %3};"
      : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
      : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}

// WARPS share K, PER blocks each at most; TILES tiles of eight tokens; NORM: the input norm is made here.
template <int WARPS, int PER, int TILES, bool NORM>
__global__ void __launch_bounds__(WARPS * 32) gemm_bf16_few_kernel(const FewArgs g) {
  __shared__ float part[WARPS][TILES][4][32];
  __shared__ float squares[WARPS][TILES * 8];
  VX_TRACE_SCOPE(30 + g.mode);
  allow_dependents();
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int row = lane >> 2, c = lane & 3;
  // The tile's rows: `first` .. + 7, and as many again `apart` further on.
  int first = blockIdx.x * FEW_ROWS, apart = FEW_ROWS / 2;
  if (g.mode == 4) {
    const int half = g.head_dim / 2, tiles = half / 8;  // of a head
    const int head = blockIdx.x / tiles;
    first = head * g.head_dim + (blockIdx.x - head * tiles) * 8;
    apart = half;
  }
  const int low = first + row, high = low + apart;
  uint4 wl[PER], wh[PER];
#pragma unroll
  for (int i = 0; i < PER; ++i) {
    const int k = (i * WARPS + warp) * FEW_BLOCK + c * 8;
    const __nv_bfloat16* from = (const __nv_bfloat16*)g.w + k;
    wl[i] = k < g.K && low < g.N ? few_load_weights(from + (size_t)low * g.K) : make_uint4(0, 0, 0, 0);
    wh[i] = k < g.K && high < g.N ? few_load_weights(from + (size_t)high * g.K) : make_uint4(0, 0, 0, 0);
  }
  grid_dependency_wait();
  // What the output adds to is asked for with the input.
  constexpr int OUTPUTS = (FEW_ROWS * 8 * TILES + WARPS * 32 - 1) / (WARPS * 32);
  float old[OUTPUTS];
  if (g.mode == 2) {
#pragma unroll
    for (int u = 0; u < OUTPUTS; ++u) {
      const int e = threadIdx.x + u * WARPS * 32, t = e / FEW_ROWS, r = e % FEW_ROWS;
      old[u] = t < g.T && first + r < g.N ? __ldcg((const float*)g.out + (size_t)t * g.ldy + first + r) : 0.f;
    }
  }
  // Two chains of products a tile.
  float acc[TILES][4], more[TILES][4], sum_sq[TILES];
#pragma unroll
  for (int tile = 0; tile < TILES; ++tile) {
    sum_sq[tile] = 0.f;
#pragma unroll
    for (int j = 0; j < 4; ++j) acc[tile][j] = more[tile][j] = 0.f;
  }
#pragma unroll
  for (int tile = 0; tile < TILES; ++tile) {
    const int t = tile * 8 + row;  // this lane's token
    if (NORM) {
      float4 xa[PER], xb[PER];
#pragma unroll
      for (int i = 0; i < PER; ++i) {
        const int k = (i * WARPS + warp) * FEW_BLOCK + c * 8;
        const bool there = t < g.T && k < g.K;
        const float4* from = reinterpret_cast<const float4*>(g.resid + (size_t)t * g.resid_ld + k);
        xa[i] = there ? __ldcg(from) : make_float4(0.f, 0.f, 0.f, 0.f);
        xb[i] = there ? __ldcg(from + 1) : make_float4(0.f, 0.f, 0.f, 0.f);
      }
#pragma unroll
      for (int i = 0; i < PER; ++i) {
        const int k = (i * WARPS + warp) * FEW_BLOCK + c * 8;
        const float4* from = reinterpret_cast<const float4*>(g.norm_w + k);
        const float4 na = k < g.K ? __ldg(from) : make_float4(0.f, 0.f, 0.f, 0.f);
        const float4 nb = k < g.K ? __ldg(from + 1) : make_float4(0.f, 0.f, 0.f, 0.f);
        sum_sq[tile] += xa[i].x * xa[i].x + xa[i].y * xa[i].y + xa[i].z * xa[i].z + xa[i].w * xa[i].w + xb[i].x * xb[i].x +
                        xb[i].y * xb[i].y + xb[i].z * xb[i].z + xb[i].w * xb[i].w;
        few_mma(acc[tile], wl[i].x, wh[i].x, wl[i].y, wh[i].y, few_pack(xa[i].x * na.x, xa[i].y * na.y),
                few_pack(xa[i].z * na.z, xa[i].w * na.w));
        few_mma(more[tile], wl[i].z, wh[i].z, wl[i].w, wh[i].w, few_pack(xb[i].x * nb.x, xb[i].y * nb.y),
                few_pack(xb[i].z * nb.z, xb[i].w * nb.w));
      }
    } else {
      uint4 xv[PER];
#pragma unroll
      for (int i = 0; i < PER; ++i) {
        const int k = (i * WARPS + warp) * FEW_BLOCK + c * 8;
        xv[i] = t < g.T && k < g.K ? __ldcg(reinterpret_cast<const uint4*>((const __nv_bfloat16*)g.x + (size_t)t * g.K + k))
                                   : make_uint4(0, 0, 0, 0);
      }
#pragma unroll
      for (int i = 0; i < PER; ++i) {
        few_mma(acc[tile], wl[i].x, wh[i].x, wl[i].y, wh[i].y, xv[i].x, xv[i].y);
        few_mma(more[tile], wl[i].z, wh[i].z, wl[i].w, wh[i].w, xv[i].z, xv[i].w);
      }
    }
  }
#pragma unroll
  for (int tile = 0; tile < TILES; ++tile) {
#pragma unroll
    for (int j = 0; j < 4; ++j) part[warp][tile][j][lane] = acc[tile][j] + more[tile][j];
    if (NORM) {
      float s = sum_sq[tile];
      s += __shfl_xor_sync(0xffffffffu, s, 1);
      s += __shfl_xor_sync(0xffffffffu, s, 2);
      if (c == 0) squares[warp][tile * 8 + row] = s;
    }
  }
  __syncthreads();
  // Row r (of 16) of token t: the warps' parts in their order, the norm's factor, the bias.
  const auto finished = [&](int t, int r, int n) {
    float v = 0.f;
#pragma unroll
    for (int i = 0; i < WARPS; ++i) v += part[i][t >> 3][(r >> 3) * 2 + (t & 1)][(r & 7) * 4 + ((t & 7) >> 1)];
    if (NORM) {
      float s = 0.f;
#pragma unroll
      for (int i = 0; i < WARPS; ++i) s += squares[i][t];
      v *= rsqrtf(s / (float)g.K + g.eps);
    }
    return g.bias != nullptr ? v + g.bias[n] : v;
  };
  // (With the norm inside it is always this one.  Without the rest as dead code in them those instances come out with fewer loads of
  // X under way, 56 registers where they have 78, and a step of 8 tokens of the 1.5B sizes takes 1,276 us instead of 1,253.)
  if (g.mode == 4) {
    const int half = apart, head = first / g.head_dim;
    const bool is_q = head < g.heads, is_k = !is_q && head < g.heads + g.kv_heads;
    for (int e = threadIdx.x; e < 8 * g.T; e += WARPS * 32) {
      const int t = e >> 3, r = e & 7, n = first + r, d = n - head * g.head_dim;
      float lo = finished(t, r, n), hi = finished(t, r + 8, n + half);
      if (is_q || is_k) {
        int pos = g.positions[t];
        if (pos < 0 || pos >= g.max_pos) {
          atomicOr(g.status, VX_STATUS_BAD_POSITION);
          pos = 0;
        }
        const float cs = g.cos_t[(size_t)pos * half + d], sn = g.sin_t[(size_t)pos * half + d];
        const float turned = lo * cs - hi * sn;
        hi = lo * sn + hi * cs;
        lo = turned;
      }
      __nv_bfloat16* to;
      if (is_q) {
        to = (__nv_bfloat16*)g.out + (size_t)t * g.ldy + n;
      } else {
        if (g.k_cache == nullptr) continue;
        const int slot = g.slots[t];
        if (slot < 0) continue;
        if ((long long)slot >= g.num_slots) {
          atomicOr(g.status, VX_STATUS_BAD_SLOT);
          continue;
        }
        const int kv_head = head - g.heads - (is_k ? 0 : g.kv_heads);
        to = (__nv_bfloat16*)(is_k ? g.k_cache : g.v_cache) + ((size_t)slot * g.kv_heads + kv_head) * g.head_dim + d;
      }
      to[0] = __float2bfloat16_rn(lo);
      to[half] = __float2bfloat16_rn(hi);
    }
    return;
  }
#pragma unroll
  for (int u = 0; u < OUTPUTS; ++u) {
    const int e = threadIdx.x + u * WARPS * 32, t = e / FEW_ROWS, r = e % FEW_ROWS;
    const int n = first + r;
    if (t >= g.T || n >= g.N) continue;
    const float v = finished(t, r, n);
    const size_t at = (size_t)t * g.ldy + n;
    if (g.mode == 0) {
      ((__nv_bfloat16*)g.out)[at] = __float2bfloat16_rn(v);
    } else if (g.mode == 1) {
      ((float*)g.out)[at] = v;
    } else {
      ((float*)g.out)[at] = old[u] + v;
      if (g.out2 != nullptr) g.out2[(size_t)t * g.ld2 + n] = old[u] + v;
    }
  }
}

// Measured against the kernel with a ring (us back to back, QKV with norm, rotation and cache write | output projection with
// the second copy): 1 token of 256 5.5 | 4.6 -> 2.3 | 1.4, of 896 6.1 | 4.6 -> 4.3 | 2.5, of 1,536 6.4 | 4.3 -> 5.4 | 3.1; 8 tokens of 896
// 6.1 | 4.8 -> 4.3 | 2.6, of 1,536 6.4 | 4.4 -> 5.9 | 3.5, of 2,048 6.9 | 5.2 -> 7.4 | 4.8; 16 tokens of 896 6.8 | 5.2 -> 6.2 | 2.9,
// of 1,536 6.3 | 4.6 -> 7.8 | 4.9: a CTA reads all rows of X, float32 with the norm, so the line lies lower there.  From 3,584 on
// the weights no longer come at once (12.0 | 7.6 -> 13.4 | 8.8).
bool gemm_bf16_few_takes(int T, int N, int K, int mode, bool norm) {
  if (T > 16 || (mode != 0 && mode != 1 && mode != 2 && mode != 4) || (N + FEW_ROWS - 1) / FEW_ROWS > 2 * 148) return false;
  // (Plain outputs with the norm inside stay with the ring kernel, where they were before this one was there.  Here they would be
  // as near to 64 bits, 7e-8 to 1.2e-7 in the 2-norm beside the operands' rounding where the ring has 8e-8 to 7.6e-7, and sooner: one
  // token by 64 x 128 1.3 us against 4.8, 1,152 x 896 2.8 against 7.6, 2,048 x 1,536 4.8 against 9.2.  Open.)
  if (norm && mode != 4) return false;
  return K <= (T > 8 ? 1024 : norm ? 1536 : 2048);
}

template <int WARPS, int PER>
static int launch_few(const FewArgs& g, cudaStream_t stream) {
  const dim3 grid((g.N + FEW_ROWS - 1) / FEW_ROWS), block(WARPS * 32);
  const bool norm = g.x == nullptr;
  // (Only what gemm_bf16_few_takes lets through.)
  constexpr bool WIDE = WARPS * PER * FEW_BLOCK <= 1024, NORMED = WARPS * PER * FEW_BLOCK <= 1536;
  if (g.T <= 8) {
    if (!norm) launch_pdl(gemm_bf16_few_kernel<WARPS, PER, 1, false>, grid, block, 0, stream, g);
    else if constexpr (NORMED) launch_pdl(gemm_bf16_few_kernel<WARPS, PER, 1, true>, grid, block, 0, stream, g);
    else return (int)cudaErrorInvalidValue;
  } else if constexpr (WIDE) {
    if (norm) launch_pdl(gemm_bf16_few_kernel<WARPS, PER, 2, true>, grid, block, 0, stream, g);
    else launch_pdl(gemm_bf16_few_kernel<WARPS, PER, 2, false>, grid, block, 0, stream, g);
  } else {
    return (int)cudaErrorInvalidValue;
  }
  return (int)cudaGetLastError();
}

int gemm_bf16_few(const FewArgs& g, cudaStream_t stream) {
  const int blocks = (g.K + FEW_BLOCK - 1) / FEW_BLOCK;
  if (blocks <= 8) return launch_few<8, 1>(g, stream);
  if (blocks <= 32) return launch_few<8, 4>(g, stream);
  if (blocks <= 48) return launch_few<8, 6>(g, stream);
  if (blocks <= 64) return launch_few<8, 8>(g, stream);
  return (int)cudaErrorInvalidValue;
}

}  // namespace vx

VX_TRACE_API(vx_few)
