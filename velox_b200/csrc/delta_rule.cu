// The delta rule token after token: recurrent mixers whose state is a matrix per head that every token
// reads, corrects and writes.
//
//   delta_rule_scan_kernel        S <- diag(w) S - (a u)(u^T S) + k v^T,  o = S^T r  per head, with the
//                                 decay w, the removal rate a and the unit key u made on the way in
//   gated_delta_prepare_kernel    the gated delta rule's vectors: short convolutions, silu, unit q and k,
//                                 decay and write strength, packed for the scan
//   delta_rule_prepare_kernel     what the generalized rule's scan reads, made per token
//   delta_rule_fold_kernel        the starting states of a long portion's chunks
//
// What a recurrence reads and keeps is float32 whatever the storage type of the projections.
// A sequence is rows q_start[s] .. q_start[s] + q_len[s] - 1 of the step; its state lives in
// row seq_slots[s] of a slot-indexed array.
#include "common.cuh"
#include "delta_rule.cuh"
#include "recurrent.cuh"

namespace vx {

// ---------------------------------------------------------------------------------------------
// Generalized delta rule.  Per head, with key size Dk and value size Dv, the state S is Dk x Dv:
//     w_t = exp(-decay * sigmoid(wl_t + w0)),   a_t = sigmoid(al_t + a_bias),
//     u_t = k_t / sqrt(sum(k_t^2) + key_eps)
//     S_t = diag(w_t) S_(t-1) - (a_t * u_t) (u_t^T S_(t-1)) + k_t v_t^T,     o_t = S_t^T r_t
// Both middle terms read the old state.  Two kernels.
//
// delta_rule_prepare_kernel: a warp per (token, head) makes the token's vectors over the key
// channels in float32 (decay, removal rate times unit key, unit key, key, receptance) and copies
// the values, into packed rows [head][token]: [w | a u | u | k | r] of KD floats each (Dk padded
// with zeros to the lanes' rows) and then v (Dv padded to a multiple of four).  A head's rows of
// consecutive tokens are contiguous, so a tile of tokens is one bulk copy.
//
// delta_rule_scan_kernel: a column of S (one value channel) never meets another column, so a
// block takes CB columns of one head of one sequence; RL lanes share a column, each with KP rows
// of it in registers, and the two sums over the rows (u^T S and S^T r) meet by shuffles.  Every
// token waits for the token before it, and a warp alone on its scheduler issues an instruction
// every five to six cycles, so what counts is how few instructions a thread has per token: four
// rows a thread (sixteen lanes a column) for key sizes up to 128, sixteen rows beyond.  A block
// asks for more than half of an SM's shared memory, so that no two of the few blocks share an SM.  The
// tokens' packed rows come in tiles of TT tokens, one bulk copy a tile, into a ring of two stages,
// each with its mbarrier, so the next tile arrives while this one is worked through.  The state is
// stored [head][column][row]: a thread's rows are contiguous.  Every sum has a fixed order, so a
// token's result does not depend on how the sequence was cut into steps.
//
// The same scan runs the gated delta rule (see gated_delta_prepare_kernel): with the decay g, the unit
// key k and the write strength beta
//     S' = g S;   S_t = S' + beta k (v - S'^T k)^T;   o_t = S_t^T q
// is the rule above with w = g, u = g k, and beta k in the places of both a u and k, so its tokens
// are packed as [g | k | q] and beta (DR_CHANNEL: a decay per state row) or as [k | q], g and beta
// (DR_HEAD: one decay) and the products are made on the way.
//
// Long portions (a step of at least two chunks of DR_CHUNK tokens) run in three launches, chunks
// side by side.  A token's transition, diag(w) - (a u) u^T, is not diagonal, so a chunk's
// transition P is a dense Dk x Dk matrix: its columns are the images of the unit vectors, that is,
// Dk more columns of state that start as the identity and see no k v^T.  Pass A (mode 1) runs every
// chunk but a portion's last from zero over Dv + Dk columns and keeps the result Z | P; the fold
// kernel makes the chunks' starting states in order, S_0 the state, S_(c+1) = P_c S_c + Z_c; pass B (mode 2) runs
// every chunk again from its start and writes the outputs, its last chunk the state.  A portion of
// one chunk skips pass A and the fold.  In this form a token's result depends, within float32
// rounding, on where its chunk began.
constexpr int DR_KP_SMALL = 4, DR_KP_LARGE = 16, DR_SMALL_MAX_DK = 128;
constexpr size_t DR_MIN_SMEM = 116 * 1024;
constexpr int DR_CHUNK = 256;
// Where chunk `chunk` of sequence `seq` keeps its Z | P and its starting state: chunks of one
// sequence begin DR_CHUNK rows apart, and later sequences begin at later rows, so the number is
// taken by nobody else; it is below ceil(tokens / DR_CHUNK) + sequences.
__device__ __forceinline__ int dr_chunk_slot(int seq, int first_row) { return first_row / DR_CHUNK + seq; }

template <typename T>
__global__ void __launch_bounds__(256)
delta_rule_prepare_kernel(const T* __restrict__ r_in, const T* __restrict__ k_in, const T* __restrict__ v_in,
                          const T* __restrict__ a_in, long long in_stride, const T* __restrict__ w_in,
                          long long w_stride, const float* __restrict__ w0, const float* __restrict__ a_bias,
                          float decay, float key_eps, float* __restrict__ packed, long long head_stride,
                          int heads, int Dk, int Dv, int KD, int Dvp, int num_tokens) {
  allow_dependents();
  grid_dependency_wait();
  const int lane = threadIdx.x & 31;
  const long long unit = (long long)blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
  if (unit >= (long long)num_tokens * heads) return;
  const int t = (int)(unit / heads), h = (int)(unit - (long long)t * heads);
  const size_t hk = (size_t)h * Dk;
  const T* k_row = k_in + (size_t)t * in_stride + hk;
  float ss = 0.f;
  for (int ch = lane; ch < Dk; ch += 32) {
    const float kv = to_float(k_row[ch]);
    ss = fmaf(kv, kv, ss);
  }
  const float inv = 1.0f / sqrtf(warp_sum(ss) + key_eps);
  float* dst = packed + (size_t)h * head_stride + (size_t)t * (5 * KD + Dvp);
  for (int ch = lane; ch < KD; ch += 32) {
    float wv = 0.f, au = 0.f, u = 0.f, kv = 0.f, rv = 0.f;
    if (ch < Dk) {
      const size_t at = (size_t)t * in_stride + hk + ch;
      kv = to_float(k_row[ch]);
      rv = to_float(r_in[at]);
      u = kv * inv;
      au = sq_sigmoid(to_float(a_in[at]) + a_bias[hk + ch]) * u;
      wv = expf(-decay * sq_sigmoid(to_float(w_in[(size_t)t * w_stride + hk + ch]) + w0[hk + ch]));
    }
    dst[ch] = wv;
    dst[KD + ch] = au;
    dst[2 * KD + ch] = u;
    dst[3 * KD + ch] = kv;
    dst[4 * KD + ch] = rv;
  }
  for (int c = lane; c < Dvp; c += 32)
    dst[5 * KD + c] = c < Dv ? to_float(v_in[(size_t)t * in_stride + (size_t)h * Dv + c]) : 0.f;
}

template <int FORM, int DR_KP, int RL>
__global__ void delta_rule_scan_kernel(const float* __restrict__ packed, long long head_stride,
                                       float* __restrict__ state, long long state_stride, float* __restrict__ out,
                                       long long out_stride, int Dk, int Dv, int Dvp, int CB, int TT,
                                       const int* __restrict__ q_start, const int* __restrict__ q_len,
                                       const int* __restrict__ seq_slots, int mode, int max_chunks, int heads,
                                       float* __restrict__ chunk_results, float* __restrict__ chunk_starts,
                                       int* status, ConvRing conv) {
  extern __shared__ __align__(16) float dr_smem[];
  __shared__ __align__(8) unsigned long long dr_bars[2];
  // The successor is let in when the scan is over: its blocks would share the few busy SMs'
  // issue slots with a kernel whose every token waits for the token before it.
  const int seq = blockIdx.x / max_chunks, chunk = blockIdx.x - seq * max_chunks;
  const int h = blockIdx.y, tile = blockIdx.z;
  const int n_all = q_len[seq];
  const int chunks = mode == 0 ? 1 : (n_all + DR_CHUNK - 1) / DR_CHUNK;
  // Pass A has nothing to do for a portion's last chunk (nobody starts behind it).
  if (n_all <= 0 || chunk >= chunks || (mode == 1 && chunk == chunks - 1)) {
    allow_dependents();
    return;
  }
  const int t_first = q_start[seq] + (mode == 0 ? 0 : chunk * DR_CHUNK);
  const int n = mode == 0 ? n_all : min(DR_CHUNK, n_all - chunk * DR_CHUNK);
  constexpr int KD = RL * DR_KP;
  constexpr int vec = dr_vectors(FORM) * KD + dr_scalars(FORM);  // floats of a token's row before its values
  const int token_floats = vec + Dvp;
  const int p = threadIdx.x % RL, c = threadIdx.x / RL;
  const int col = tile * CB + c;
  const int num_cols = mode == 1 ? Dv + Dk : Dv;  // pass A: Dk more columns carry the chunk's transition
  const bool live = col < num_cols;
  const bool value_col = col < Dv;
  const size_t safe_col = live ? col : 0;
  // Where this thread's rows come from and go to.
  float* state_rows = state + (size_t)seq_slots[seq] * state_stride + ((size_t)h * Dv + (value_col ? col : 0)) * Dk;
  const int slot_here = dr_chunk_slot(seq, t_first);
  const float* from = state_rows;
  float* mine = state_rows;
  if (mode == 1) {
    from = nullptr;
    mine = chunk_results + (((size_t)slot_here * heads + h) * (size_t)(Dv + Dk) + safe_col) * Dk;
  } else if (mode == 2 && chunks > 1) {
    // Every chunk of a cut portion starts from the fold kernel's copy, the first one too: the block
    // of the last chunk writes the state row, and nothing says that it does so after the first
    // chunk's block has read it.
    from = chunk_starts + (((size_t)slot_here * heads + h) * (size_t)Dv + safe_col) * Dk;
    if (chunk < chunks - 1) mine = nullptr;  // only a portion's last chunk leaves the state behind
  }
  const uint32_t bar0 = smem_u32(&dr_bars[0]), bar1 = smem_u32(&dr_bars[1]);
  if (threadIdx.x == 0) {
    mbar_init(bar0, 1);
    mbar_init(bar1, 1);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
  }
  __syncthreads();
  const int num_tiles = (n + TT - 1) / TT;
  const float* src_base = packed + (size_t)h * head_stride + (size_t)t_first * token_floats;
  auto issue = [&](int index) {
    const int stage = index & 1;
    const int tt = min(TT, n - index * TT);
    const uint32_t bar = stage ? bar1 : bar0;
    const uint32_t bytes = (uint32_t)tt * (uint32_t)token_floats * 4u;
    mbar_expect_tx(bar, bytes);
    bulk_copy_g2s(smem_u32(dr_smem + (size_t)stage * TT * token_floats),
                  src_base + (size_t)index * TT * token_floats, bytes, bar);
  };
  grid_dependency_wait();
  if (threadIdx.x == 0) {
    issue(0);
    if (num_tiles > 1) issue(1);
  }
  if (FORM != DR_GENERAL && conv.x != nullptr && tile == 0 && (mode == 0 || (mode == 2 && chunk == chunks - 1))) {
    if (conv.dtype == VX_DTYPE_F32) ring_write_last<float>(conv, seq_slots[seq], q_start[seq], n_all, h);
    else ring_write_last<__nv_bfloat16>(conv, seq_slots[seq], q_start[seq], n_all, h);
  }
  float S[DR_KP];
#pragma unroll
  for (int q = 0; q < DR_KP; ++q) {
    const int row = p * DR_KP + q;
    if (from != nullptr) S[q] = (live && row < Dk) ? from[row] : 0.f;
    else S[q] = (live && !value_col && row == col - Dv) ? 1.f : 0.f;  // zero, or a column of the identity
  }
  // One pass over the rows per token makes both sums that read the state as it is before the
  // token's update: u_t^T S for this token and S^T r for the token before (whose update is the last
  // one S has seen).  Their shuffle trees run side by side.  `pending` says that a token's output is
  // still to be made; r_prev are its receptance values for this thread's rows.
  float r_prev[DR_KP];
#pragma unroll
  for (int q = 0; q < DR_KP; ++q) r_prev[q] = 0.f;
  bool pending = false;
  int pending_row = 0;
  for (int index = 0; index < num_tiles; ++index) {
    const int stage = index & 1;
    const int tt = min(TT, n - index * TT);
    mbar_wait(stage ? bar1 : bar0, (uint32_t)(index >> 1) & 1u, status);
    const float* buf = dr_smem + (size_t)stage * TT * token_floats;
    const float* tok = buf + p * DR_KP;
    int row_now = t_first + index * TT;
#pragma unroll 2
    for (int i = 0; i < tt; ++i, tok += token_floats, ++row_now) {
      constexpr int K_AT = FORM == DR_GENERAL ? 3 * KD : FORM == DR_CHANNEL ? KD : 0;
      const float4* w4 = reinterpret_cast<const float4*>(tok);
      const float4* a4 = reinterpret_cast<const float4*>(tok + KD);
      const float4* u4 = reinterpret_cast<const float4*>(tok + 2 * KD);
      const float4* k4 = reinterpret_cast<const float4*>(tok + K_AT);
      const float4* r4 = reinterpret_cast<const float4*>(tok + K_AT + KD);
      float us0 = 0.f, us1 = 0.f, us2 = 0.f, us3 = 0.f;
      float o0 = 0.f, o1 = 0.f, o2 = 0.f, o3 = 0.f;
#pragma unroll
      for (int q = 0; q < DR_KP / 4; ++q) {
        float4 u;
        if constexpr (FORM == DR_GENERAL) {
          u = u4[q];
        } else if constexpr (FORM == DR_HEAD) {
          u = k4[q];  // the decay multiplies the finished sum
        } else {
          const float4 w = w4[q], k = k4[q];
          u = make_float4(w.x * k.x, w.y * k.y, w.z * k.z, w.w * k.w);
        }
        us0 = fmaf(u.x, S[4 * q], us0);
        us1 = fmaf(u.y, S[4 * q + 1], us1);
        us2 = fmaf(u.z, S[4 * q + 2], us2);
        us3 = fmaf(u.w, S[4 * q + 3], us3);
        o0 = fmaf(S[4 * q], r_prev[4 * q], o0);
        o1 = fmaf(S[4 * q + 1], r_prev[4 * q + 1], o1);
        o2 = fmaf(S[4 * q + 2], r_prev[4 * q + 2], o2);
        o3 = fmaf(S[4 * q + 3], r_prev[4 * q + 3], o3);
      }
      float us = (us0 + us1) + (us2 + us3);
      float o = (o0 + o1) + (o2 + o3);
#pragma unroll
      for (int off = 16; off > 0; off >>= 1) {
        if (off < RL) {
          us += __shfl_xor_sync(0xffffffffu, us, off);
          o += __shfl_xor_sync(0xffffffffu, o, off);
        }
      }
      if (pending && mode != 1 && live && p == 0) out[(size_t)pending_row * out_stride + (size_t)h * Dv + col] = o;
      const float vj = value_col ? tok[vec - p * DR_KP + col] : 0.f;
      if constexpr (FORM == DR_GENERAL) {
#pragma unroll
        for (int q = 0; q < DR_KP / 4; ++q) {
          const float4 w = w4[q], a = a4[q], k = k4[q];
          S[4 * q] = fmaf(w.x, S[4 * q], fmaf(-a.x, us, k.x * vj));
          S[4 * q + 1] = fmaf(w.y, S[4 * q + 1], fmaf(-a.y, us, k.y * vj));
          S[4 * q + 2] = fmaf(w.z, S[4 * q + 2], fmaf(-a.z, us, k.z * vj));
          S[4 * q + 3] = fmaf(w.w, S[4 * q + 3], fmaf(-a.w, us, k.w * vj));
        }
      } else {
        const float2 gb = *reinterpret_cast<const float2*>(tok + vec - p * DR_KP - 2);  // g (DR_HEAD), beta
        const float change = FORM == DR_HEAD ? gb.y * fmaf(-gb.x, us, vj) : gb.y * (vj - us);
#pragma unroll
        for (int q = 0; q < DR_KP / 4; ++q) {
          const float4 k = k4[q];
          float4 w = make_float4(gb.x, gb.x, gb.x, gb.x);
          if constexpr (FORM == DR_CHANNEL) w = w4[q];
          S[4 * q] = fmaf(w.x, S[4 * q], k.x * change);
          S[4 * q + 1] = fmaf(w.y, S[4 * q + 1], k.y * change);
          S[4 * q + 2] = fmaf(w.z, S[4 * q + 2], k.z * change);
          S[4 * q + 3] = fmaf(w.w, S[4 * q + 3], k.w * change);
        }
      }
#pragma unroll
      for (int q = 0; q < DR_KP / 4; ++q) {
        const float4 r = r4[q];
        r_prev[4 * q] = r.x;
        r_prev[4 * q + 1] = r.y;
        r_prev[4 * q + 2] = r.z;
        r_prev[4 * q + 3] = r.w;
      }
      pending = true;
      pending_row = row_now;
    }
    __syncthreads();  // every thread is done with this stage before it is filled again
    if (threadIdx.x == 0 && index + 2 < num_tiles) issue(index + 2);
  }
  {
    // The last token's output, from the state as it is now.
    float o0 = 0.f, o1 = 0.f, o2 = 0.f, o3 = 0.f;
#pragma unroll
    for (int q = 0; q < DR_KP / 4; ++q) {
      o0 = fmaf(S[4 * q], r_prev[4 * q], o0);
      o1 = fmaf(S[4 * q + 1], r_prev[4 * q + 1], o1);
      o2 = fmaf(S[4 * q + 2], r_prev[4 * q + 2], o2);
      o3 = fmaf(S[4 * q + 3], r_prev[4 * q + 3], o3);
    }
    float o = (o0 + o1) + (o2 + o3);
#pragma unroll
    for (int off = 16; off > 0; off >>= 1)
      if (off < RL) o += __shfl_xor_sync(0xffffffffu, o, off);
    if (pending && mode != 1 && live && p == 0) out[(size_t)pending_row * out_stride + (size_t)h * Dv + col] = o;
  }
  allow_dependents();
  if (live && mine != nullptr) {
#pragma unroll
    for (int q = 0; q < DR_KP; ++q) {
      const int row = p * DR_KP + q;
      if (row < Dk) mine[row] = S[q];
    }
  }
}

// ---------------------------------------------------------------------------------------------
// The gated delta rule's vectors (delta_rule.cuh) packed for the scan, a warp per (token, head); NPL values a
// lane hold a head's key channels.
template <typename T, int FORM, int NPL>
__global__ void __launch_bounds__(256)
gated_delta_prepare_kernel(GatedDelta p, float* __restrict__ packed, long long head_stride, int KD, int Dvp,
                           const int* __restrict__ q_start, const int* __restrict__ q_len,
                           const int* __restrict__ seq_slots) {
  allow_dependents();
  grid_dependency_wait();
  const int lane = threadIdx.x & 31;
  const int seq = blockIdx.y;
  const int n = q_len[seq], start = q_start[seq];
  const int Dk = p.Dk, Dv = p.Dv, group = p.heads / p.kv_heads;
  const int keys = p.kv_heads * Dk, C = 2 * keys + p.heads * Dv;
  const float* ring = p.ring + (size_t)seq_slots[seq] * p.ring_stride;
  constexpr int VECS = dr_vectors(FORM);
  const int token_floats = VECS * KD + 4 + Dvp;
  const long long units = (long long)n * p.heads;
  for (long long unit = (long long)blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5); unit < units;
       unit += (long long)gridDim.x * (blockDim.x >> 5)) {
    const int i = (int)(unit / p.heads), h = (int)(unit - (long long)i * p.heads);
    const int row = start + i, pos = p.positions[row], kh = h / group;
    float qv[NPL], kv[NPL];
    float sq = 0.f, sk = 0.f;
#pragma unroll
    for (int j = 0; j < NPL; ++j) {
      const int ch = lane + 32 * j;
      qv[j] = kv[j] = 0.f;
      if (ch < Dk) {
        qv[j] = conv_at<T>(p, ring, C, kh * Dk + ch, row, i, pos);
        kv[j] = conv_at<T>(p, ring, C, keys + kh * Dk + ch, row, i, pos);
      }
      sq = fmaf(qv[j], qv[j], sq);
      sk = fmaf(kv[j], kv[j], sk);
    }
    const float iq = p.q_scale / sqrtf(warp_sum(sq) + p.unit_eps);
    const float ik = 1.0f / sqrtf(warp_sum(sk) + p.unit_eps);
    const float rate = -expf(p.a_log[h]);
    const float beta = sq_sigmoid(to_float(((const T*)p.b)[(size_t)row * p.b_stride + h]));
    const T* a_row = (const T*)p.a + (size_t)row * p.a_stride;
    float* dst = packed + (size_t)h * head_stride + (size_t)row * token_floats;
    float g = 0.f;
    if (FORM == DR_HEAD) g = expf(rate * sq_softplus(to_float(a_row[h]) + p.dt_bias[h]));
#pragma unroll
    for (int j = 0; j < NPL; ++j) {
      const int ch = lane + 32 * j;
      if (ch < KD) {
        if (FORM == DR_CHANNEL)
          dst[ch] = ch < Dk ? expf(rate * sq_softplus(to_float(a_row[h * Dk + ch]) + p.dt_bias[h * Dk + ch])) : 0.f;
        dst[(VECS - 2) * KD + ch] = kv[j] * ik;
        dst[(VECS - 1) * KD + ch] = qv[j] * iq;
      }
    }
    if (lane < 4) dst[VECS * KD + lane] = lane == 2 ? g : lane == 3 ? beta : 0.f;
    for (int c = lane; c < Dvp; c += 32)
      dst[VECS * KD + 4 + c] = c < Dv ? conv_at<T>(p, ring, C, 2 * keys + h * Dv + c, row, i, pos) : 0.f;
  }
}

// The chunks' starting states, in order: S_(c+1) = P_c S_c + Z_c with S_0 the sequence's state.  A
// block takes some value columns of one head of one sequence and keeps them in shared memory;
// thread (row k, column j) sums over the rows i of S in rising order, reading column i of P, which is
// stored as a run of Dk floats.
__global__ void delta_rule_fold_kernel(const float* __restrict__ state, long long state_stride,
                                       const float* __restrict__ chunk_results, float* __restrict__ chunk_starts,
                                       int Dk, int Dv, int CBF, int heads, const int* __restrict__ q_start,
                                       const int* __restrict__ q_len, const int* __restrict__ seq_slots,
                                       int stage_p) {
  extern __shared__ __align__(16) float fold_smem[];  // two buffers [CBF][Dk], then (stage_p) P [Dk][Dk]
  allow_dependents();
  const int seq = blockIdx.x, h = blockIdx.y, col0 = blockIdx.z * CBF;
  const int n_all = q_len[seq];
  const int chunks = (n_all + DR_CHUNK - 1) / DR_CHUNK;
  if (n_all <= 0 || chunks < 2) return;
  const int cols = min(CBF, Dv - col0);
  float* now = fold_smem;
  float* next = fold_smem + (size_t)CBF * Dk;
  grid_dependency_wait();
  const float* start = state + (size_t)seq_slots[seq] * state_stride + ((size_t)h * Dv + col0) * Dk;
  const int first_row = q_start[seq];
  float* first_start = chunk_starts + (((size_t)dr_chunk_slot(seq, first_row) * heads + h) * (size_t)Dv + col0) * Dk;
  for (int idx = threadIdx.x; idx < cols * Dk; idx += blockDim.x) {
    now[idx] = start[idx];
    first_start[idx] = start[idx];  // the first chunk's start is the state as the step found it
  }
  __syncthreads();
  for (int chunk = 0; chunk + 1 < chunks; ++chunk) {
    const size_t here = ((size_t)dr_chunk_slot(seq, first_row + chunk * DR_CHUNK) * heads + h) * (size_t)(Dv + Dk) * Dk;
    const float* Z = chunk_results + here + (size_t)col0 * Dk;   // [column j][row k]
    const float* P = chunk_results + here + (size_t)Dv * Dk;     // [column i][row k]; 16-byte aligned when Dk % 4 == 0
    float* dst = chunk_starts +
                 (((size_t)dr_chunk_slot(seq, first_row + (chunk + 1) * DR_CHUNK) * heads + h) * (size_t)Dv + col0) * Dk;
    if (stage_p) {
      // The chunk's transition into shared memory, every load under way at once.
      float* staged = fold_smem + 2 * (size_t)CBF * Dk;
      for (int idx = threadIdx.x * 4; idx < Dk * Dk; idx += blockDim.x * 4)
        *reinterpret_cast<float4*>(staged + idx) = *reinterpret_cast<const float4*>(P + idx);
      __syncthreads();
      P = staged;
    }
    // Four outputs a thread at a time, so that the loads of P (global memory, one per row i) of
    // several rows are under way together: a single output's sum would wait for each in turn.
    for (int base = threadIdx.x; base < cols * Dk; base += 4 * blockDim.x) {
      int j[4], k[4];
      float acc[4];
#pragma unroll
      for (int o = 0; o < 4; ++o) {
        const int idx = min(base + o * (int)blockDim.x, cols * Dk - 1);
        j[o] = idx / Dk;
        k[o] = idx - j[o] * Dk;
        acc[o] = Z[idx];
      }
#pragma unroll 8
      for (int i = 0; i < Dk; ++i) {
#pragma unroll
        for (int o = 0; o < 4; ++o) acc[o] = fmaf(P[(size_t)i * Dk + k[o]], now[j[o] * Dk + i], acc[o]);
      }
#pragma unroll
      for (int o = 0; o < 4; ++o) {
        const int idx = base + o * (int)blockDim.x;
        if (idx < cols * Dk) {
          next[idx] = acc[o];
          dst[idx] = acc[o];
        }
      }
    }
    __syncthreads();
    float* swap = now;
    now = next;
    next = swap;
  }
}

}  // namespace vx

using namespace vx;

static int dr_pow2_at_least(int v) {
  int p = 1;
  while (p < v) p <<= 1;
  return p;
}

// Floats of scratch the chunked form wants for a step of up to `num_tokens` tokens of `num_seqs` sequences.
VX_API long long vx_delta_rule_chunk_scratch(int num_tokens, int num_seqs, int heads, int Dk, int Dv) {
  const long long slots = (num_tokens + DR_CHUNK - 1) / DR_CHUNK + num_seqs;
  return slots * heads * ((long long)(Dv + Dk) * Dk + (long long)Dv * Dk);
}

static int dr_rows_per_lane(int Dk) { return Dk <= DR_SMALL_MAX_DK ? DR_KP_SMALL : DR_KP_LARGE; }

// Floats of one token's packed row (all heads), or -1 for a key size beyond the lanes of a warp.
static int dr_packed_width(int form, int heads, int Dk, int Dv) {
  const int KP = dr_rows_per_lane(Dk);
  const int RL = dr_pow2_at_least((Dk + KP - 1) / KP);
  if (RL > 32) return -1;
  return heads * (dr_vectors(form) * RL * KP + dr_scalars(form) + (Dv + 3) / 4 * 4);
}

VX_API int vx_delta_rule_packed_width(int heads, int Dk, int Dv) { return dr_packed_width(DR_GENERAL, heads, Dk, Dv); }

VX_API int vx_gated_delta_packed_width(int per_channel, int heads, int Dk, int Dv) {
  return dr_packed_width(per_channel ? DR_CHANNEL : DR_HEAD, heads, Dk, Dv);
}

static int dr_num_sms() {
  static int num_sms = 0;
  if (num_sms == 0) {
    int device = 0;
    cudaGetDevice(&device);
    cudaDeviceGetAttribute(&num_sms, cudaDevAttrMultiProcessorCount, device);
  }
  return num_sms;
}

// What a launch of the scan works on.
struct DeltaScan {
  const float* packed;
  long long head_stride;  // from one head's rows to the next head's
  float* state;
  long long state_stride;
  float* out;
  long long out_stride;
  int heads, Dk, Dv, Dvp;
  const int* q_start;
  const int* q_len;
  const int* seq_slots;
  int num_seqs, mode, max_chunks;
  float* chunk_results;
  float* chunk_starts;
  int* status;
  ConvRing conv;
};

template <int FORM, int KP, int RL>
static int dr_launch_scan(const DeltaScan& a, cudaStream_t stream) {
  constexpr int KD = RL * KP;
  // Columns a block: four warps' worth where the lanes allow, a whole number of warps at least.
  int CB = 128 / RL;
  if (CB > 32) CB = 32;
  if (CB < 1) CB = 1;
  const int TT = KD <= 64 ? 16 : (KD <= 128 ? 8 : 4);
  size_t smem = sizeof(float) * 2 * (size_t)TT * (dr_vectors(FORM) * KD + dr_scalars(FORM) + a.Dvp);
  const dim3 grid(a.num_seqs * a.max_chunks, a.heads, ((a.mode == 1 ? a.Dv + a.Dk : a.Dv) + CB - 1) / CB);
  // Few blocks (a prompt's portion): each gets an SM of its own.  Many blocks (single tokens of
  // many sequences) share the SMs as they fit.
  if ((long long)grid.x * grid.y * grid.z <= dr_num_sms() && smem < DR_MIN_SMEM) smem = DR_MIN_SMEM;
  // The kernel has a few bytes of static shared memory beside these: ask from a kilobyte below
  // the default limit on.
  static size_t limit = 0;  // one per instantiation
  if (smem + 1024 > 48 * 1024 && smem > limit) {
    cudaFuncSetAttribute(delta_rule_scan_kernel<FORM, KP, RL>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    limit = smem;
  }
  launch_pdl(delta_rule_scan_kernel<FORM, KP, RL>, grid, dim3(CB * RL), smem, stream, a.packed, a.head_stride, a.state,
             a.state_stride, a.out, a.out_stride, a.Dk, a.Dv, a.Dvp, CB, TT, a.q_start, a.q_len, a.seq_slots, a.mode,
             a.max_chunks, a.heads, a.chunk_results, a.chunk_starts, a.status, a.conv);
  return (int)cudaGetLastError();
}

template <int FORM>
static int dr_scan(const DeltaScan& a, cudaStream_t stream) {
  const int KP = dr_rows_per_lane(a.Dk);
  const int RL = dr_pow2_at_least((a.Dk + KP - 1) / KP);
#define VX_DR(KPV, RLV) \
  if (KP == KPV && RL == RLV) return dr_launch_scan<FORM, KPV, RLV>(a, stream)
  VX_DR(DR_KP_SMALL, 1);
  VX_DR(DR_KP_SMALL, 2);
  VX_DR(DR_KP_SMALL, 4);
  VX_DR(DR_KP_SMALL, 8);
  VX_DR(DR_KP_SMALL, 16);
  VX_DR(DR_KP_SMALL, 32);
  VX_DR(DR_KP_LARGE, 16);
  VX_DR(DR_KP_LARGE, 32);
#undef VX_DR
  return -1;
}

// The scan of a step over packed rows: in one launch, or, when the step is long and the caller has
// brought the scratch for it, in chunks (pass A, the fold, pass B).
template <int FORM>
static int dr_run(DeltaScan a, int num_tokens, float* chunk_scratch, long long chunk_scratch_floats,
                  cudaStream_t stream) {
  const bool chunked = num_tokens >= 2 * DR_CHUNK && chunk_scratch != nullptr &&
                       chunk_scratch_floats >= vx_delta_rule_chunk_scratch(num_tokens, a.num_seqs, a.heads, a.Dk, a.Dv);
  a.max_chunks = chunked ? (num_tokens + DR_CHUNK - 1) / DR_CHUNK : 1;
  a.mode = 0;
  a.chunk_results = a.chunk_starts = nullptr;
  if (!chunked) return dr_scan<FORM>(a, stream);
  const long long slots = (long long)a.max_chunks + a.num_seqs;
  a.chunk_results = chunk_scratch;
  a.chunk_starts = chunk_scratch + slots * a.heads * (long long)(a.Dv + a.Dk) * a.Dk;
  a.mode = 1;
  int code = dr_scan<FORM>(a, stream);
  if (code != 0) return code;
  const int CBF = a.Dk <= 128 ? 16 : 4;
  size_t fold_smem = sizeof(float) * 2 * (size_t)CBF * a.Dk;
  // The chunk's Dk x Dk transition beside them where it fits (and its rows are whole 16-byte packs).
  const int stage_p = a.Dk % 4 == 0 && fold_smem + sizeof(float) * (size_t)a.Dk * a.Dk <= 96 * 1024;
  if (stage_p) fold_smem += sizeof(float) * (size_t)a.Dk * a.Dk;
  static size_t fold_limit = 0;
  if (fold_smem > 47 * 1024 && fold_smem > fold_limit) {
    cudaFuncSetAttribute(delta_rule_fold_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)fold_smem);
    fold_limit = fold_smem;
  }
  launch_pdl(delta_rule_fold_kernel, dim3(a.num_seqs, a.heads, (a.Dv + CBF - 1) / CBF), dim3(256), fold_smem, stream,
             (const float*)a.state, a.state_stride, (const float*)a.chunk_results, a.chunk_starts, a.Dk, a.Dv, CBF,
             a.heads, a.q_start, a.q_len, a.seq_slots, stage_p);
  code = (int)cudaGetLastError();
  if (code != 0) return code;
  a.mode = 2;
  return dr_scan<FORM>(a, stream);
}

VX_API int vx_delta_rule_scan(const void* r, const void* k, const void* v, const void* a, int dtype, long long in_stride,
                              const void* w, long long w_stride, const float* w0, const float* a_bias, float decay,
                              float key_eps, float* packed, long long packed_rows, float* state, long long state_stride,
                              float* out,
                              long long out_stride, int heads, int Dk, int Dv, const int* q_start, const int* q_len,
                              const int* seq_slots, int num_seqs, int num_tokens, float* chunk_scratch,
                              long long chunk_scratch_floats, int* status, cudaStream_t stream) {
  if (num_seqs <= 0 || num_tokens <= 0) return 0;
  if (heads <= 0 || Dk <= 0 || Dv <= 0) return (int)cudaErrorInvalidValue;
  const int KP = dr_rows_per_lane(Dk);
  const int RL = dr_pow2_at_least((Dk + KP - 1) / KP);
  if (RL > 32) return -1;
  const int KD = RL * KP, Dvp = (Dv + 3) / 4 * 4;
  if (packed_rows < num_tokens) return (int)cudaErrorInvalidValue;
  const long long packed_stride = packed_rows * (5 * KD + Dvp);  // from one head's rows to the next head's
  const long long units = (long long)num_tokens * heads;
  VX_BY_DTYPE(dtype, launch_pdl(delta_rule_prepare_kernel<T>, dim3((unsigned)((units + 7) / 8)), dim3(256), 0, stream,
                                (const T*)r, (const T*)k, (const T*)v, (const T*)a, in_stride, (const T*)w, w_stride,
                                w0, a_bias, decay, key_eps, packed, packed_stride, heads, Dk, Dv, KD, Dvp, num_tokens));
  int code = (int)cudaGetLastError();
  if (code != 0) return code;
  DeltaScan scan = {packed, packed_stride, state, state_stride, out, out_stride, heads, Dk, Dv, Dvp, q_start, q_len,
                    seq_slots, num_seqs, 0, 1, nullptr, nullptr, status, {}};
  return dr_run<DR_GENERAL>(scan, num_tokens, chunk_scratch, chunk_scratch_floats, stream);
}

// The gated delta rule over each sequence's tokens, from and into the state and ring of its slot.
VX_API int vx_gated_delta_scan(const void* x, int dtype, long long x_stride, const void* b, long long b_stride,
                               const void* a, long long a_stride, int per_channel, const float* dt_bias,
                               const float* a_log, const float* conv_w, int taps, float* ring, long long ring_stride,
                               float* state, long long state_stride, const int* positions, float unit_eps,
                               float q_scale, int heads, int kv_heads, int Dk, int Dv, float* packed,
                               long long packed_rows, float* out, long long out_stride, const int* q_start,
                               const int* q_len, const int* seq_slots, int num_seqs, int num_tokens,
                               float* chunk_scratch, long long chunk_scratch_floats, int* status,
                               cudaStream_t stream) {
  if (num_seqs <= 0 || num_tokens <= 0) return 0;
  if (heads <= 0 || kv_heads <= 0 || heads % kv_heads != 0 || Dk <= 0 || Dv <= 0 || taps < 1) return (int)cudaErrorInvalidValue;
  const int KP = dr_rows_per_lane(Dk);
  const int RL = dr_pow2_at_least((Dk + KP - 1) / KP);
  if (RL > 32) return -1;
  const int KD = RL * KP, Dvp = (Dv + 3) / 4 * 4;
  if (packed_rows < num_tokens) return (int)cudaErrorInvalidValue;
  const int form = per_channel ? DR_CHANNEL : DR_HEAD;
  const long long head_stride = packed_rows * (dr_vectors(form) * KD + 4 + Dvp);
  const GatedDelta p = {x, x_stride, b, b_stride, a, a_stride, dt_bias, a_log, conv_w, ring, ring_stride, positions,
                        taps, heads, kv_heads, Dk, Dv, unit_eps, q_scale};
  long long blocks = ((long long)num_tokens * heads + 7) / 8;
  const long long most = (148 * 16 + num_seqs - 1) / num_seqs;
  if (blocks > most) blocks = most;
  const dim3 grid((unsigned)blocks, num_seqs);
#define VX_GD_PREPARE(FORM, NPL)                                                                                   \
  VX_BY_DTYPE(dtype, launch_pdl(gated_delta_prepare_kernel<T, FORM, NPL>, grid, dim3(256), 0, stream, p, packed,    \
                                head_stride, KD, Dvp, q_start, q_len, seq_slots))
#define VX_GD_PREPARE_FORM(NPL)                     \
  if (per_channel) { VX_GD_PREPARE(DR_CHANNEL, NPL) } \
  else { VX_GD_PREPARE(DR_HEAD, NPL) }
  if (KD <= 32) { VX_GD_PREPARE_FORM(1) }
  else if (KD <= 64) { VX_GD_PREPARE_FORM(2) }
  else if (KD <= 128) { VX_GD_PREPARE_FORM(4) }
  else if (KD <= 256) { VX_GD_PREPARE_FORM(8) }
  else { VX_GD_PREPARE_FORM(16) }
#undef VX_GD_PREPARE_FORM
#undef VX_GD_PREPARE
  const int code = (int)cudaGetLastError();
  if (code != 0) return code;
  DeltaScan scan = {packed, head_stride, state, state_stride, out, out_stride, heads, Dk, Dv, Dvp, q_start, q_len,
                    seq_slots, num_seqs, 0, 1, nullptr, nullptr, status,
                    {taps > 1 ? x : nullptr, x_stride, dtype, ring, ring_stride, positions, taps, kv_heads, Dk, Dv, heads}};
  if (per_channel) return dr_run<DR_CHANNEL>(scan, num_tokens, chunk_scratch, chunk_scratch_floats, stream);
  return dr_run<DR_HEAD>(scan, num_tokens, chunk_scratch, chunk_scratch_floats, stream);
}
