// On-device sampling over float32 logits [R, V]: greedy, temperature, top-k, top-p, and the
// repetition / presence / frequency penalties.
//
// What is sampled follows the reference's sampler (engine/sampler.py:131-258 in that project):
//   penalties   logit[v] -= frequency * count(v); then logit[v] = logit[v] > 0 ? logit[v] / rep
//               : logit[v] * rep; then logit[v] -= presence, for every token v in the request's
//               prompt and output so far (sampler.py:169-189);
//   greedy      argmax, first index on ties (sampler.py:155-156);
//   otherwise   scaled = logit / max(temperature, 1e-5); candidates are the k most probable
//               tokens and the smallest most-probable set whose mass reaches top_p
//               (sampler.py:216-228); the draw is the exponential race
//               argmax(p / noise), noise ~ Exp(1) clamped at 1e-10 (sampler.py:230-258).
// How it is done differs: the race runs over the whole vocabulary as argmax(scaled - log noise)
// (the same draw, since log is monotone and the normaliser is a constant), the candidate set is
// found as a value threshold, digit by digit of its bit pattern, instead of by a sort, and the noise comes from a
// counter-based generator (Philox4x32-10) keyed by the request's seed and counted by
// (index of the output token, vocabulary index), so a request's draws do not depend on what
// else is in the batch.  Bit-equality with torch's generator stream is not a goal.
#include "common.cuh"

#include <math_constants.h>

namespace vx {

// ---------------------------------------------------------------------------------------------
// Philox4x32-10 (Salmon et al., "Parallel random numbers: as easy as 1, 2, 3", SC'11).
// ---------------------------------------------------------------------------------------------
__device__ __forceinline__ uint4 philox4x32_10(uint4 ctr, uint2 key) {
  const uint32_t M0 = 0xD2511F53u, M1 = 0xCD9E8D57u, W0 = 0x9E3779B9u, W1 = 0xBB67AE85u;
#pragma unroll
  for (int round = 0; round < 10; ++round) {
    const uint32_t hi0 = __umulhi(M0, ctr.x), lo0 = M0 * ctr.x;
    const uint32_t hi1 = __umulhi(M1, ctr.z), lo1 = M1 * ctr.z;
    ctr = make_uint4(hi1 ^ ctr.y ^ key.x, lo1, hi0 ^ ctr.w ^ key.y, lo0);
    key.x += W0;
    key.y += W1;
  }
  return ctr;
}

// Uniform in (0, 1) from 32 random bits.
__device__ __forceinline__ float uniform_open(uint32_t bits) {
  return ((float)(bits >> 8) + 0.5f) * (1.0f / 16777216.0f);
}

// Order-preserving map float -> uint32 (larger float, larger key).
__device__ __forceinline__ uint32_t float_key(float v) {
  const uint32_t b = __float_as_uint(v);
  return (b & 0x80000000u) ? ~b : (b | 0x80000000u);
}
__device__ __forceinline__ float key_float(uint32_t k) {
  const uint32_t b = (k & 0x80000000u) ? (k & 0x7fffffffu) : ~k;
  return __uint_as_float(b);
}

struct Best {
  float score;
  int index;
};

__device__ __forceinline__ Best better(Best a, Best b) {
  // Larger score wins; on equal scores the lower index (torch.argmax returns the first maximum).
  if (b.index < 0) return a;
  if (a.index < 0) return b;
  if (b.score > a.score || (b.score == a.score && b.index < a.index)) return b;
  return a;
}

__device__ __forceinline__ Best block_best(Best v, Best* scratch /* 32 */) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int num_warps = (blockDim.x + 31) >> 5;
#pragma unroll
  for (int offset = 16; offset > 0; offset >>= 1) {
    Best o;
    o.score = __shfl_xor_sync(0xffffffffu, v.score, offset);
    o.index = __shfl_xor_sync(0xffffffffu, v.index, offset);
    v = better(v, o);
  }
  if (lane == 0) scratch[warp] = v;
  __syncthreads();
  if (warp == 0) {
    Best w;
    w.score = 0.f;
    w.index = -1;
    if (lane < num_warps) w = scratch[lane];
#pragma unroll
    for (int offset = 16; offset > 0; offset >>= 1) {
      Best o;
      o.score = __shfl_xor_sync(0xffffffffu, w.score, offset);
      o.index = __shfl_xor_sync(0xffffffffu, w.index, offset);
      w = better(w, o);
    }
    if (lane == 0) scratch[0] = w;
  }
  __syncthreads();
  const Best out = scratch[0];
  __syncthreads();
  return out;
}

// ---------------------------------------------------------------------------------------------
// One token per row.  temperature[r] == 0: argmax.  Otherwise the exponential race over the
// entries with logit / T >= threshold[r] (threshold may be null: no filter).
//
// A row is cut into gridDim.y segments (multiples of four entries, so that the generator's
// counter, the index of a group of four, means the same for every cut).  Every block leaves its
// best entry in `partial`; the block that arrives last at the row's counter takes the best of
// all of them (`better` is associative and commutative, ties included, so the result does not
// depend on the cut or on the order of arrival), writes the token and puts the counter back to
// zero for the next launch.
// ---------------------------------------------------------------------------------------------
constexpr int SAMPLE_THREADS = 256;
constexpr int SAMPLE_MAX_SEGMENTS = 64;

__global__ void __launch_bounds__(SAMPLE_THREADS)
sample_kernel(const float* __restrict__ logits, int vocab, long long row_stride,
              const float* __restrict__ temperature, const unsigned long long* __restrict__ seeds,
              const int* __restrict__ draw_index, const float* __restrict__ threshold,
              int* __restrict__ out, int* __restrict__ history, long long history_stride,
              const int* __restrict__ history_slots, const int* __restrict__ history_lengths,
              int segment_len, Best* __restrict__ partial, unsigned int* __restrict__ counters,
              const int* __restrict__ status_word) {
  __shared__ Best scratch[32];
  __shared__ bool is_last;
  allow_dependents();
  grid_dependency_wait();
  const int r = blockIdx.x;
  const int segments = (int)gridDim.y;
  const int begin = blockIdx.y * segment_len;
  const int end = min(vocab, begin + segment_len);
  const float* row = logits + (size_t)r * row_stride;
  const float temp = temperature ? temperature[r] : 0.f;
  // Groups of four entries by one 16-byte load where the row allows it.
  const bool vec = (row_stride & 3) == 0 && (reinterpret_cast<uintptr_t>(logits) & 15) == 0;
  Best best;
  best.score = 0.f;
  best.index = -1;

  if (temp == 0.f) {
    for (int base = begin + threadIdx.x * 4; base < end; base += SAMPLE_THREADS * 4) {
      float v[4];
      if (vec && base + 4 <= vocab) {
        const float4 q = *reinterpret_cast<const float4*>(row + base);
        v[0] = q.x, v[1] = q.y, v[2] = q.z, v[3] = q.w;
      } else {
#pragma unroll
        for (int j = 0; j < 4; ++j) v[j] = base + j < vocab ? row[base + j] : CUDART_NAN_F;
      }
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        Best c;
        c.score = v[j];
        c.index = base + j;
        if (c.score == c.score) best = better(best, c);
      }
    }
  } else {
    const float inv_t = 1.0f / fmaxf(temp, 1e-5f);
    const float cut = threshold ? threshold[r] : -CUDART_INF_F;
    const unsigned long long seed = seeds[r];
    const uint2 key = make_uint2((uint32_t)seed, (uint32_t)(seed >> 32));
    const uint32_t draw = (uint32_t)draw_index[r];
    for (int base = begin + threadIdx.x * 4; base < end; base += SAMPLE_THREADS * 4) {
      float v[4];
      if (vec && base + 4 <= vocab) {
        const float4 q = *reinterpret_cast<const float4*>(row + base);
        v[0] = q.x, v[1] = q.y, v[2] = q.z, v[3] = q.w;
      } else {
#pragma unroll
        for (int j = 0; j < 4; ++j) v[j] = base + j < vocab ? row[base + j] : CUDART_NAN_F;
      }
      // (Also what lies past the row's end, NaN, is no candidate.)  Behind a filter hardly a group has
      // one, and the generator's ten rounds are most of what an entry costs.
      if (!(v[0] * inv_t >= cut || v[1] * inv_t >= cut || v[2] * inv_t >= cut || v[3] * inv_t >= cut)) continue;
      const uint4 bits = philox4x32_10(make_uint4((uint32_t)(base >> 2), draw, 0u, 0u), key);
      const uint32_t b[4] = {bits.x, bits.y, bits.z, bits.w};
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const float scaled = v[j] * inv_t;
        if (!(scaled >= cut)) continue;
        const float noise = fmaxf(-logf(uniform_open(b[j])), 1e-10f);
        Best c;
        c.score = scaled - logf(noise);
        c.index = base + j;
        best = better(best, c);
      }
    }
  }
  best = block_best(best, scratch);
  if (segments > 1) {
    if (threadIdx.x == 0) {
      partial[(size_t)r * segments + blockIdx.y] = best;
      __threadfence();
      is_last = atomicAdd(&counters[r], 1u) == (unsigned int)segments - 1u;
    }
    __syncthreads();
    if (!is_last) return;
    __threadfence();
    best.score = 0.f;
    best.index = -1;
    if ((int)threadIdx.x < segments) {
      const volatile Best* p = partial + (size_t)r * segments + threadIdx.x;
      best.score = p->score;
      best.index = p->index;
    }
    best = block_best(best, scratch);
    if (threadIdx.x == 0) counters[r] = 0u;
  }
  if (threadIdx.x == 0) {
    const int token = best.index < 0 ? 0 : best.index;
    out[r] = token;
    // The device status word rides behind the tokens, so the host's one read-back of the step
    // also tells it whether a kernel of the step refused an access or gave up a wait.
    if (status_word != nullptr && r == 0) out[gridDim.x] = *reinterpret_cast<const volatile int*>(status_word);
    // Append to the request's token history (kept for the penalties) when there is one.
    if (history != nullptr) {
      const int n = history_lengths[r];
      if (n >= 0 && n < history_stride) history[(size_t)history_slots[r] * history_stride + n] = token;
    }
  }
}

// ---------------------------------------------------------------------------------------------
// Candidate threshold for top-k / top-p.  For a value x let count(x) be the number of entries
// with scaled > x and mass(x) their softmax probability.  An entry is a candidate iff
// count(scaled_i) < k (when k > 0) and mass(scaled_i) < top_p: it is among the k largest, and
// the entries before it do not already reach top_p.  Both are monotone in x, so the candidates
// are the entries >= a threshold: the smallest x with count(x) < k and mass(x) < top_p.
//
// The threshold is found digit by digit over the ordered bit patterns of float (11 + 11 + 10
// bits): a sweep over the row builds, in shared memory, the histogram of the next digit among
// the entries that share the digits found so far (how many, and their mass); the digit is the
// smallest one above which count and mass still pass.  Four sweeps over the row in all (maximum,
// three digits; the first digit's histogram also gives the normaliser) where a bisection over
// the patterns took up to 34.  Masses are summed as 2^-40 fixed-point
// integers, so the histogram, and with it the threshold, does not depend on the order in which
// threads add.
// ---------------------------------------------------------------------------------------------
constexpr int FILTER_THREADS = 1024;
constexpr int FILTER_BINS = 2048;
// Copies of the histogram for the first digit.  That digit is sign, exponent and two bits of
// the mantissa, so a row's entries share a few dozen of its values and their atomics queue up
// on those bins; with a copy per four warps the queues are an eighth as long.  The copies are
// added up before the digit is chosen (integer sums: the result does not depend on the copies).
constexpr int FILTER_COPIES = 8;
constexpr size_t FILTER_SMEM_BYTES = (size_t)FILTER_COPIES * FILTER_BINS * (sizeof(unsigned int) + sizeof(unsigned long long));
constexpr float FILTER_MASS_SCALE = 1099511627776.0f;  // 2^40

__device__ __forceinline__ unsigned long long fixed_mass(float e) {
  return (unsigned long long)(e * FILTER_MASS_SCALE);
}

// For this thread's values c and m: their sums over the block's threads with a larger index.
__device__ __forceinline__ void suffix_sums(unsigned int c, unsigned long long m, unsigned int* sc /* 32 */,
                                            unsigned long long* sm /* 32 */, unsigned int& c_above,
                                            unsigned long long& m_above) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  // inclusive suffix scan inside the warp
  unsigned int ci = c;
  unsigned long long mi = m;
#pragma unroll
  for (int offset = 1; offset < 32; offset <<= 1) {
    const unsigned int co = __shfl_down_sync(0xffffffffu, ci, offset);
    const unsigned long long mo = __shfl_down_sync(0xffffffffu, mi, offset);
    if (lane + offset < 32) {
      ci += co;
      mi += mo;
    }
  }
  if (lane == 0) {
    sc[warp] = ci;
    sm[warp] = mi;
  }
  __syncthreads();
  unsigned int cw = 0;
  unsigned long long mw = 0;
  const int warps = (int)(blockDim.x >> 5);
  for (int w = warp + 1; w < warps; ++w) {
    cw += sc[w];
    mw += sm[w];
  }
  c_above = cw + ci - c;
  m_above = mw + mi - m;
  __syncthreads();
}

// What the digit search carries from one digit to the next: how many entries, and how much
// mass, lie above the digits found so far, and the mass that top_p allows.
struct DigitSearch {
  unsigned int above_count;
  unsigned long long above_mass, mass_limit;
};

struct DigitChoice {
  unsigned int digit, count;
  unsigned long long mass, total;
};

// The next digit from the row's histogram of it, by a block of 1,024 threads: thread t brings
// the bins of digits 2t and 2t + 1.  A digit d passes if what lies above it (the larger digits,
// and everything above the digits found before) is fewer than k entries and less than top_p of
// the mass; passing is monotone in the digit, and the digit chosen is the smallest that passes.
// The first digit's histogram holds every entry of the row, so its masses add up to the
// normaliser: the sums that are compared are sums of the same integers.
__device__ __forceinline__ unsigned int choose_digit(unsigned int c0, unsigned int c1, unsigned long long m0,
                                                     unsigned long long m1, bool first, bool use_k, int k, bool use_p,
                                                     float p, DigitSearch& search, unsigned int* sc,
                                                     unsigned long long* sm, DigitChoice* choice) {
  unsigned int c_above;
  unsigned long long m_above;
  suffix_sums(c0 + c1, m0 + m1, sc, sm, c_above, m_above);
  if (first) {
    if (threadIdx.x == 0) choice->total = m_above + m0 + m1;
    __syncthreads();
    // (At least one: the largest entry, with nothing above it, is always a candidate.)
    search.mass_limit = max(1ull, (unsigned long long)((double)p * (double)choice->total));
  }
  const unsigned int c_hi = search.above_count + c_above, c_lo = c_hi + c1;  // above digit 2t + 1, above 2t
  const unsigned long long m_hi = search.above_mass + m_above, m_lo = m_hi + m1;
  const bool pass_hi = (!use_k || c_hi < (unsigned int)k) && (!use_p || m_hi < search.mass_limit);
  const bool pass_lo = (!use_k || c_lo < (unsigned int)k) && (!use_p || m_lo < search.mass_limit);
  // The smallest passing digit is the one whose lower neighbour fails (or digit 0).
  if (pass_hi && !pass_lo) {
    choice->digit = 2u * threadIdx.x + 1u;
    choice->count = c_hi;
    choice->mass = m_hi;
  }
  if (pass_lo) {
    // The digit below 2t is 2t - 1 (thread t - 1's); what lies above it is also digit 2t.
    bool below_fails = threadIdx.x == 0;
    if (!below_fails) {
      const unsigned int cb = c_lo + c0;
      const unsigned long long mb = m_lo + m0;
      below_fails = !((!use_k || cb < (unsigned int)k) && (!use_p || mb < search.mass_limit));
    }
    if (below_fails) {
      choice->digit = 2u * threadIdx.x;
      choice->count = c_lo;
      choice->mass = m_lo;
    }
  }
  __syncthreads();
  search.above_count = choice->count;
  search.above_mass = choice->mass;
  return choice->digit;
}

// Calls f(value) for every entry of a row, the block's threads side by side.  With a row that
// starts on a 16-byte boundary a thread asks for four vectors of four entries before it looks
// at the first: sixteen loads' worth under way per thread instead of one (a sweep with one was
// bound by the latency of its loads, about 15 GB/s a block).  The order in which entries are
// seen differs from a plain loop; every use below (maximum, integer sums, histograms) is
// independent of it.
template <typename F>
__device__ __forceinline__ void sweep_row(const float* __restrict__ row, int vocab, bool vectors, F&& f) {
  const int step = (int)blockDim.x;
  if (vectors) {
    const int n4 = vocab >> 2;
    const float4* row4 = reinterpret_cast<const float4*>(row);
    int i = (int)threadIdx.x;
    for (; i + 3 * step < n4; i += 4 * step) {
      const float4 a = row4[i], b = row4[i + step], c = row4[i + 2 * step], d = row4[i + 3 * step];
      f(a.x), f(a.y), f(a.z), f(a.w);
      f(b.x), f(b.y), f(b.z), f(b.w);
      f(c.x), f(c.y), f(c.z), f(c.w);
      f(d.x), f(d.y), f(d.z), f(d.w);
    }
    for (; i < n4; i += step) {
      const float4 a = row4[i];
      f(a.x), f(a.y), f(a.z), f(a.w);
    }
    for (int j = (n4 << 2) + (int)threadIdx.x; j < vocab; j += step) f(row[j]);
  } else {
    for (int i = (int)threadIdx.x; i < vocab; i += step) f(row[i]);
  }
}

__global__ void __launch_bounds__(FILTER_THREADS)
filter_threshold_kernel(const float* __restrict__ logits, int vocab, long long row_stride,
                        const float* __restrict__ temperature, const int* __restrict__ top_k,
                        const float* __restrict__ top_p, float* __restrict__ threshold) {
  __shared__ float scratch[32];
  __shared__ unsigned int sc[32];
  __shared__ unsigned long long sm[32];
  extern __shared__ __align__(16) unsigned char filter_smem[];
  unsigned long long* hist_mass = reinterpret_cast<unsigned long long*>(filter_smem);          // [COPIES][BINS]
  unsigned int* hist_count = reinterpret_cast<unsigned int*>(hist_mass + FILTER_COPIES * FILTER_BINS);  // [COPIES][BINS]
  __shared__ DigitChoice choice;
  allow_dependents();
  grid_dependency_wait();
  const int r = blockIdx.x;
  const float temp = temperature[r];
  const int k = top_k[r];
  const float p = top_p[r];
  const bool use_k = k > 0 && k < vocab;
  const bool use_p = p < 1.0f;
  if (temp == 0.f || (!use_k && !use_p)) {
    if (threadIdx.x == 0) threshold[r] = -CUDART_INF_F;
    return;
  }
  const float* row = logits + (size_t)r * row_stride;
  const float inv_t = 1.0f / fmaxf(temp, 1e-5f);

  const bool vectors = (reinterpret_cast<uintptr_t>(row) & 15) == 0;

  float m = -CUDART_INF_F;
  sweep_row(row, vocab, vectors, [&](float x) { m = fmaxf(m, __fmul_rn(x, inv_t)); });
  m = warp_max(m);
  if ((threadIdx.x & 31) == 0) scratch[threadIdx.x >> 5] = m;
  __syncthreads();
  if (threadIdx.x < 32) {
    float w = threadIdx.x < ((blockDim.x + 31) >> 5) ? scratch[threadIdx.x] : -CUDART_INF_F;
    w = warp_max(w);
    if (threadIdx.x == 0) scratch[0] = w;
  }
  __syncthreads();
  m = scratch[0];
  __syncthreads();

  // Digits of the threshold's pattern, most significant first.
  uint32_t prefix = 0u;
  DigitSearch search = {0u, 0ull, 0ull};
  const int shifts[3] = {21, 10, 0};
  const int bits[3] = {11, 11, 10};
  for (int level = 0; level < 3; ++level) {
    const int shift = shifts[level];
    const uint32_t digit_mask = (1u << bits[level]) - 1u;
    const int copies = level == 0 ? FILTER_COPIES : 1;
    for (int b = threadIdx.x; b < copies * FILTER_BINS; b += blockDim.x) {
      hist_count[b] = 0u;
      hist_mass[b] = 0ull;
    }
    __syncthreads();
    unsigned int* my_count = hist_count + (level == 0 ? ((threadIdx.x >> 7) % FILTER_COPIES) * FILTER_BINS : 0);
    unsigned long long* my_mass = hist_mass + (level == 0 ? ((threadIdx.x >> 7) % FILTER_COPIES) * FILTER_BINS : 0);
    const float top = m;
    const uint32_t above = prefix;
    const int level_bits = bits[level];
    sweep_row(row, vocab, vectors, [&](float x) {
      // The rounded product, never folded into the subtraction below: the scaled value is the
      // same number wherever it is looked at (here, in the cluster kernel, in the sampler).
      const float s = __fmul_rn(x, inv_t);
      if (!(s == s)) return;  // NaN is never a candidate
      const uint32_t key = float_key(s);
      if (level > 0 && (key >> (shift + level_bits)) != above) return;
      const uint32_t digit = (key >> shift) & digit_mask;
      // What the filter in force does not look at is not counted.
      if (use_k) atomicAdd(&my_count[digit], 1u);
      if (use_p) atomicAdd(&my_mass[digit], fixed_mass(expf(s - top)));
    });
    __syncthreads();
    unsigned int c[2] = {0u, 0u};
    unsigned long long w[2] = {0ull, 0ull};
    for (int copy = 0; copy < copies; ++copy)
#pragma unroll
      for (int i = 0; i < 2; ++i) {
        c[i] += hist_count[copy * FILTER_BINS + 2 * threadIdx.x + i];
        w[i] += hist_mass[copy * FILTER_BINS + 2 * threadIdx.x + i];
      }
    const unsigned int digit = choose_digit(c[0], c[1], w[0], w[1], level == 0, use_k, k, use_p, p, search, sc, sm, &choice);
    if (use_p && choice.total == 0ull) {  // no mass at all: a row whose maximum is not finite
      if (threadIdx.x == 0) threshold[r] = m;
      return;
    }
    prefix = (prefix << bits[level]) | digit;
    __syncthreads();
  }
  if (threadIdx.x == 0) threshold[r] = key_float(prefix);
}

// ---------------------------------------------------------------------------------------------
// The same threshold by a cluster of CTAs per row, for rows of up to 196,608 entries.  What bounds it is
// not the row's bytes (the head has just written them, they are in the L2) but the atomics of entries that
// share a bin, the cluster's meetings, and the waves of CTAs.
//
// One histogram finds the threshold's bin, and it takes only entries that can matter.  Each of n groups of
// threads has an entry that is no smaller than the smallest of the groups' maxima, so at least n entries lie at
// or above that bound: for groups of 32, 8 or 1 threads, the k-th largest entry is not below the bound of the
// largest groups of which there are k.  And vocab entries that lie w below the maximum have at most
// vocab * exp(-w) of its mass together: where that is less than the 1 - p of the normaliser that top_p leaves
// out, the threshold is not below.  The normaliser is at least the maximum's own mass; where that says little (no
// k, and a maximum that does not stand out) a pass that only sums up the mass comes first.  The bins are steps of
// equal width between the larger of the bounds and the maximum.  With top_p and a bound that is far down the
// histogram begins with the entries nearer by, and takes the others only if the threshold is not among those.
// The entries of the threshold's bin, a few hundred at most as a rule, are gathered in the cluster's first CTA,
// which looks for the smallest of them with fewer than k entries and less than top_p of the mass above it.  (A
// threshold is always the value of an entry, since nothing changes between two of them.)  A bin of more than
// FC_LIST entries is narrowed by the range of its patterns first.
//
// All sums are of the same integers as above and the histogram's bins are in the order of the values, so
// every form gives the same threshold bit for bit.
//
// Measured (us a launch, 151,936 normal logits of deviation 2, in the L2; in brackets a fixed window of eight
// units in 1/64 with rows read again for every pass and 18 rows in clusters of eight, and before that three
// digits of the pattern over a row in registers, always eight CTAs):
//                                  1 row              18 rows            64 rows
//   T 0.1, top_k 200               11.4 (36.4, 17.7)  17.1 (52.6, 34.9)  22.7 (72.2, 86.6)
//   T 0.7, top_k 200               11.4 (12.4, 17.8)  17.1 (25.1, 34.7)  22.7 (28.9, 86.6)
//   T 0.7, top_k 50, top_p 0.9     15.6 (15.7, 20.3)  20.2 (33.3, 40.7)  27.9 (43.0, 101)
//   T 0.7, top_p 0.99              21.7 (29.6, 23.1)  33.7 (57.1, 46.5)  52.5 (71.0, 115)
//   T 1.2, top_p 0.9               22.4 (27.2, 23.3)  34.7 (47.9, 46.1)  53.6 (79.7, 115)
//
// A 64-bit sum in shared memory is a compare-and-swap loop; the masses (41 bits at most) are
// therefore added as two 32-bit words, the low word's carry found from the value it held before.
// ---------------------------------------------------------------------------------------------
constexpr int FC_MAX_VOCAB = 196608;
constexpr int FC_SHARE = FC_MAX_VOCAB / 8;  // most entries of a CTA that keeps its share
constexpr int FC_COPIES = 2;
constexpr int FC_LIST = 1024;          // most entries of a bin that are gathered (an entry a thread)
constexpr int FC_PAIRS = 128;          // most entries that are compared with one another
// Bins of the first histogram.  Every one that is not empty is added to CTA 0's by every CTA (1,024: T 0.7 with
// top_k 1,000 and top_p 19.0 us for 18.4); in fewer, more entries share one (256: T 1.2, top_p 0.9 28.1 for 22.1).
constexpr int FC_STEPS = 512;
// A maximum stands out if one of 256 parts of the row (512 with four CTAs) has no entry within this distance:
// about a hundredth of the row is nearer then.
constexpr float FC_STANDS_OUT = 9.0f;
// Where the histogram begins with both filters, and with top_p alone which part of the way to the bound.  (A
// threshold further down costs a second round, 5 - 8 us; 0.6 for 0.75 had it at T 0.7, deviation 4, top_p 0.99.)
constexpr float FC_NEAR = 8.0f;
constexpr float FC_PART = 0.75f;
constexpr size_t FC_SMEM_BYTES = (size_t)FILTER_BINS * (sizeof(unsigned long long) + sizeof(unsigned int)) +
                                 (size_t)FC_LIST * (sizeof(unsigned long long) + sizeof(unsigned int)) +
                                 (size_t)FC_COPIES * FILTER_BINS * 3 * sizeof(unsigned int);

__device__ __forceinline__ void add_mass_words(unsigned int* lo, unsigned int* hi, uint32_t bin, unsigned long long w) {
  const unsigned int wl = (unsigned int)w;
  unsigned int wh = (unsigned int)(w >> 32);
  if (wl != 0u) {
    const unsigned int before = atomicAdd(&lo[bin], wl);
    if (before + wl < before) ++wh;  // the low word wrapped
  }
  if (wh != 0u) atomicAdd(&hi[bin], wh);
}

// The address, in this CTA's window onto the cluster's shared memory, of `local` in CTA `rank`.
template <typename T>
__device__ __forceinline__ T* cluster_peer(T* local, unsigned int rank) {
  uint64_t out;
  asm volatile("mapa.u64 %0, %1, %2;" : "=l"(out) : "l"(reinterpret_cast<uint64_t>(local)), "r"(rank));
  return reinterpret_cast<T*>(out);
}

// How far below the maximum an entry can be and still be the threshold of top_p, for a normaliser of `total`
// times the maximum's own mass.  (The margin covers the rounding here; the masses are rounded down.)
__device__ __forceinline__ float mass_reach(int vocab, float p, float total) {
  return logf(fmaxf((float)vocab / ((1.0f - p) * total), 1.0f)) + 0.02f;
}

// Patterns lo ... hi cut into at most FILTER_BINS ranges of 2^shift.
__device__ __forceinline__ int pattern_shift(uint32_t lo, uint32_t hi) { return max(0, 21 - __clz(hi - lo)); }

// HELD: a CTA keeps its share of the row in shared memory; else every pass reads it again.
template <int CLUSTER, bool HELD>
__global__ void __launch_bounds__(FILTER_THREADS, 1)
filter_threshold_cluster_kernel(const float* __restrict__ logits, int vocab, long long row_stride,
                                const float* __restrict__ temperature, const int* __restrict__ top_k,
                                const float* __restrict__ top_p, float* __restrict__ threshold) {
  __shared__ float warp_least[5][32], peer_least[CLUSTER][5];
  __shared__ unsigned int sc[32];
  __shared__ unsigned long long sm[32];
  __shared__ unsigned long long peer_total[CLUSTER];
  __shared__ uint2 peer_range[CLUSTER];
  __shared__ unsigned int chosen_digit, chosen_entries, chosen_all, listed;
  __shared__ DigitChoice choice;
  extern __shared__ __align__(16) unsigned char filter_smem[];
  unsigned long long* row_mass = reinterpret_cast<unsigned long long*>(filter_smem);   // [BINS], used in CTA 0
  unsigned long long* list_mass = row_mass + FILTER_BINS;                               // [LIST], used in CTA 0
  unsigned int* row_count = reinterpret_cast<unsigned int*>(list_mass + FC_LIST);       // [BINS], used in CTA 0
  unsigned int* list_key = row_count + FILTER_BINS;                                     // [LIST], used in CTA 0
  unsigned int* own_count = list_key + FC_LIST;                                         // [COPIES][BINS]
  unsigned int* own_lo = own_count + FC_COPIES * FILTER_BINS;
  unsigned int* own_hi = own_lo + FC_COPIES * FILTER_BINS;
  allow_dependents();
  grid_dependency_wait();
  unsigned int rank;
  asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(rank));
  const int r = blockIdx.x / CLUSTER;
  const int tid = (int)threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const float temp = temperature[r];
  const int k = top_k[r];
  const float p = top_p[r];
  const bool use_k = k > 0 && k < vocab;
  const bool use_p = p < 1.0f;
  // A property of the row: all CTAs of the cluster leave here or none does.
  if (temp == 0.f || (!use_k && !use_p)) {
    if (rank == 0u && tid == 0) threshold[r] = -CUDART_INF_F;
    return;
  }
  const float inv_t = 1.0f / fmaxf(temp, 1e-5f);
  // This CTA's share of the row, a multiple of four entries.
  const int share = ((vocab + CLUSTER - 1) / CLUSTER + 3) / 4 * 4;
  const int begin = min(vocab, (int)rank * share), entries = min(vocab, begin + share) - begin;
  const float* own_row = logits + (size_t)r * row_stride + begin;
  const bool vectors = (reinterpret_cast<uintptr_t>(own_row) & 15) == 0;

  // Calls f(scaled entry) for this thread's entries, the same ones every time (and for NaN past the row's end,
  // which nothing below counts).
  float4* held = reinterpret_cast<float4*>(own_hi + FC_COPIES * FILTER_BINS);
  const auto for_each = [&](auto&& f) {
    if constexpr (HELD) {
#pragma unroll 2
      for (int i = tid; i < (entries + 3) >> 2; i += FILTER_THREADS) {
        const float4 q = held[i];
        f(q.x), f(q.y), f(q.z), f(q.w);
      }
    } else {
      sweep_row(own_row, entries, vectors, [&](float x) { f(__fmul_rn(x, inv_t)); });
    }
  };
  if constexpr (HELD) {
#pragma unroll
    for (int j = 0; j < FC_SHARE / 4 / FILTER_THREADS; ++j) {
      const int i = j * FILTER_THREADS + tid;
      if (4 * i >= entries) break;
      float4 q;
      if (vectors && 4 * i + 4 <= entries) {
        q = reinterpret_cast<const float4*>(own_row)[i];
      } else {
        q.x = own_row[4 * i];
        q.y = 4 * i + 1 < entries ? own_row[4 * i + 1] : CUDART_NAN_F;
        q.z = 4 * i + 2 < entries ? own_row[4 * i + 2] : CUDART_NAN_F;
        q.w = 4 * i + 3 < entries ? own_row[4 * i + 3] : CUDART_NAN_F;
      }
      held[i] = make_float4(__fmul_rn(q.x, inv_t), __fmul_rn(q.y, inv_t), __fmul_rn(q.z, inv_t), __fmul_rn(q.w, inv_t));
    }
  }

  for (int b = tid; b < FILTER_BINS; b += FILTER_THREADS) {
    row_mass[b] = 0ull;
    row_count[b] = 0u;
  }
  for (int b = tid; b < FC_COPIES * FILTER_BINS; b += FILTER_THREADS) {
    own_count[b] = 0u;
    own_lo[b] = 0u;
    own_hi[b] = 0u;
  }
  if (tid == 0) {
    listed = 0u;
    choice.digit = FILTER_BINS - 1, choice.count = 0u, choice.mass = 0ull;
  }
  // The largest entry, the smallest maximum of 32, 8 and 1 threads, and the smallest entry above -inf: five minima.
  float most = -CUDART_INF_F, least = CUDART_INF_F;
  for_each([&](float s) {  // (passing over NaN)
    most = fmaxf(most, s);
    if (s > -CUDART_INF_F) least = fminf(least, s);
  });
  float of_8 = most;
#pragma unroll
  for (int offset = 1; offset < 8; offset <<= 1) of_8 = fmaxf(of_8, __shfl_xor_sync(0xffffffffu, of_8, offset));
  const float of_32 = warp_max(of_8);
  of_8 = -warp_max(-of_8), most = -warp_max(-most), least = -warp_max(-least);
  if (lane == 0) {
    warp_least[0][warp] = -of_32, warp_least[1][warp] = of_32;
    warp_least[2][warp] = of_8, warp_least[3][warp] = most, warp_least[4][warp] = least;
  }
  __syncthreads();
  if (warp < 5) {
    const float mine = -warp_max(-warp_least[warp][lane]);
    if (lane < CLUSTER) *cluster_peer(&peer_least[rank][warp], (unsigned int)lane) = mine;
  }
  // Everybody's minima are in every CTA, and CTA 0's row histogram is zero, before anyone adds.
  cluster_meet();
  const auto least_of = [&](int i) {
    float v = peer_least[0][i];
#pragma unroll
    for (int c = 1; c < CLUSTER; ++c) v = fminf(v, peer_least[c][i]);
    return v;
  };
  const float top = -least_of(0);
  least = least_of(4);
  if (use_p && !(fabsf(top) < CUDART_INF_F)) {
    if (rank == 0u && tid == 0) threshold[r] = top;
    return;
  }

  // No threshold lies below `lowest` (unless every entry passes).
  const float of_warps = least_of(1), of_eighths = least_of(2);
  float lowest = -CUDART_INF_F;
  if (use_k && k <= CLUSTER * 32)
    lowest = fmaxf(lowest, of_warps);
  else if (use_k && k <= CLUSTER * 128)
    lowest = fmaxf(lowest, of_eighths);
  else if (use_k && k <= CLUSTER * 1024)
    lowest = fmaxf(lowest, least_of(3));
  const auto mass_of = [&](float s) { return use_p ? fixed_mass(expf(s - top)) : 0ull; };
  DigitSearch search = {0u, 0ull, 0ull};
  unsigned long long total = 0ull;
  // The mass of the row from the threads' sums, in every CTA.
  const auto share_total = [&] {
#pragma unroll
    for (int offset = 16; offset > 0; offset >>= 1) total += __shfl_xor_sync(0xffffffffu, total, offset);
    if (lane == 0) sm[warp] = total;
    __syncthreads();
    if (tid < 32) {
      total = sm[tid];
#pragma unroll
      for (int offset = 16; offset > 0; offset >>= 1) total += __shfl_xor_sync(0xffffffffu, total, offset);
      if (tid < CLUSTER) *cluster_peer(&peer_total[rank], (unsigned int)tid) = total;
    }
    cluster_meet();
    total = 0ull;
#pragma unroll
    for (int c = 0; c < CLUSTER; ++c) total += peer_total[c];
    // (At least one: the largest entry, with nothing above it, is always a candidate.)
    search.mass_limit = max(1ull, (unsigned long long)((double)p * (double)total));
  };
  const bool stands_out = (CLUSTER == 8 ? of_warps : of_eighths) < top - FC_STANDS_OUT;
  const bool total_first = use_p && !(use_k && k <= CLUSTER * 1024) && !stands_out;
  if (total_first) {
    for_each([&](float s) {
      if (s == s) total += mass_of(s);  // NaN is never a candidate
    });
    share_total();
  }
  const auto reach = [&] { return top - mass_reach(vocab, p, (float)total / FILTER_MASS_SCALE); };
  if (use_p) lowest = fmaxf(lowest, total_first ? reach() : top - mass_reach(vocab, p, 1.0f));
  // Where the histogram begins.
  float near = fmaxf(lowest, least);
  if (use_p && !total_first) near = fmaxf(lowest, top - (use_k ? FC_NEAR : FC_PART * mass_reach(vocab, p, 1.0f)));
  const float window = top - fmaxf(lowest, least);
  const float steps = window > 0.f && window < CUDART_INF_F ? fminf((float)FC_STEPS / window, 1e30f) : (float)FC_STEPS / 32.f;
  // The bin of a value: the last one starts at the row's maximum.  Monotone in s, infinities included.
  const auto bin_of = [&](float s) {
    return FILTER_BINS - 1 - (s == top ? 0 : (int)fminf((top - s) * steps, (float)(FC_STEPS - 1)));
  };

  unsigned int* count0 = cluster_peer(row_count, 0u);
  unsigned long long* mass0 = cluster_peer(row_mass, 0u);
  const int copy = (warp % FC_COPIES) * FILTER_BINS;
  const auto count_entry = [&](int bin, unsigned long long w) {
    atomicAdd(&own_count[copy + bin], 1u);
    if (use_p) add_mass_words(own_lo + copy, own_hi + copy, (uint32_t)bin, w);
  };
  // The bins of all CTAs into the row's histogram, the digit that CTA 0 chooses into every CTA, with the
  // entries in it and whether even what lies below the first digit passes.  A CTA's own bins go back to zero;
  // with `keep`, in that last case, the row's histogram stays for what is added to it next.
  const auto choose_in_cluster = [&](bool keep) {
    __syncthreads();
    for (int b = tid; b < FILTER_BINS; b += FILTER_THREADS) {
      unsigned int c = 0u;
      unsigned long long w = 0ull;
#pragma unroll
      for (int i = 0; i < FC_COPIES; ++i) {
        const int at = i * FILTER_BINS + b;
        if (own_count[at] == 0u) continue;
        c += own_count[at];
        w += ((unsigned long long)own_hi[at] << 32) + own_lo[at];
        own_count[at] = 0u, own_lo[at] = 0u, own_hi[at] = 0u;
      }
      if (c != 0u) atomicAdd(&count0[b], c);
      if (w != 0ull) atomicAdd(&mass0[b], w);
    }
    cluster_meet();
    if (rank == 0u) {
      const unsigned int c0 = row_count[2 * tid], c1 = row_count[2 * tid + 1];
      const unsigned long long m0 = row_mass[2 * tid], m1 = row_mass[2 * tid + 1];
      const DigitSearch before = search;
      const unsigned int digit = choose_digit(c0, c1, m0, m1, false, use_k, k, use_p, p, search, sc, sm, &choice);
      bool all = false;
      if (digit == 0u) {
        if (tid == 0)
          chosen_all = (!use_k || search.above_count + c0 < (unsigned int)k) &&
                       (!use_p || search.above_mass + m0 < search.mass_limit);
        __syncthreads();
        all = chosen_all != 0u;
      }
      if (tid == (int)(digit >> 1))
        for (unsigned int c = 0; c < CLUSTER; ++c) {
          *cluster_peer(&chosen_digit, c) = digit;
          *cluster_peer(&chosen_entries, c) = (digit & 1u) ? c1 : c0;
          *cluster_peer(&chosen_all, c) = all;
        }
      if (keep && all)
        search = before;
      else
        row_count[2 * tid] = row_count[2 * tid + 1] = 0u, row_mass[2 * tid] = row_mass[2 * tid + 1] = 0ull;
    }
    cluster_meet();
    return chosen_digit;
  };

  if (use_p && !total_first) {
    for_each([&](float s) {
      if (!(s == s)) return;
      const unsigned long long w = mass_of(s);
      total += w;
      if (s >= near) count_entry(bin_of(s), w);
    });
    share_total();
  } else {
    for_each([&](float s) {
      if (s >= near) count_entry(bin_of(s), mass_of(s));
    });
  }
  unsigned int bin = choose_in_cluster(near > lowest);
  float next = use_p ? fmaxf(lowest, reach()) : lowest;
  while (chosen_all != 0u && near > lowest) {  // (The threshold is not among the entries so far.)
    const float until = near;
    near = next < until ? next : lowest;
    next = lowest;
    for_each([&](float s) {
      if (s >= near && s < until) count_entry(bin_of(s), mass_of(s));
    });
    bin = choose_in_cluster(near > lowest);
  }
  if (chosen_all != 0u) {  // No value is too small: a row with NaN that has fewer than k entries.
    if (rank == 0u && tid == 0) threshold[r] = key_float(0u);
    return;
  }

  // The patterns of the bin's entries: all of them, or, of more than FC_LIST, the range that holds the threshold.
  uint32_t lo = 0u, hi = 0xffffffffu;
  if (chosen_entries > (unsigned int)FC_LIST) {
    uint32_t least_key = 0xffffffffu, most_key = 0u;
    for_each([&](float s) {
      if (!(s >= near) || bin_of(s) != (int)bin) return;
      const uint32_t key = float_key(s);
      least_key = min(least_key, key), most_key = max(most_key, key);
    });
    least_key = __reduce_min_sync(0xffffffffu, least_key), most_key = __reduce_max_sync(0xffffffffu, most_key);
    if (lane == 0) sc[warp] = least_key, sm[warp] = most_key;
    __syncthreads();
    if (tid < 32) {
      const uint2 mine = make_uint2(__reduce_min_sync(0xffffffffu, sc[tid]), __reduce_max_sync(0xffffffffu, (uint32_t)sm[tid]));
      if (tid < CLUSTER) *cluster_peer(&peer_range[rank], (unsigned int)tid) = mine;
    }
    cluster_meet();
    lo = 0xffffffffu, hi = 0u;
#pragma unroll
    for (int c = 0; c < CLUSTER; ++c) lo = min(lo, peer_range[c].x), hi = max(hi, peer_range[c].y);
    while (lo < hi && chosen_entries > (unsigned int)FC_LIST) {
      const int shift = pattern_shift(lo, hi);
      for_each([&](float s) {
        if (!(s >= near) || bin_of(s) != (int)bin) return;
        const uint32_t key = float_key(s);
        if (key >= lo && key <= hi) count_entry((int)((key - lo) >> shift), mass_of(s));
      });
      lo += choose_in_cluster(false) << shift;
      hi = min(hi, lo + ((1u << shift) - 1u));
    }
    if (lo == hi) {
      if (rank == 0u && tid == 0) threshold[r] = key_float(lo);
      return;
    }
  }
  unsigned int* list0 = cluster_peer(list_key, 0u);
  unsigned int* listed0 = cluster_peer(&listed, 0u);
  for_each([&](float s) {
    if (!(s >= near) || bin_of(s) != (int)bin) return;
    const uint32_t key = float_key(s);
    if (key < lo || key > hi) return;
    const unsigned int together = __activemask();  // one request of the lanes that are here
    unsigned int at = 0u;
    if (lane == __ffs(together) - 1) at = atomicAdd(listed0, __popc(together));
    at = __shfl_sync(together, at, __ffs(together) - 1) + __popc(together & ((1u << lane) - 1u));
    if (at < (unsigned int)FC_LIST) list0[at] = key;
  });
  cluster_meet();
  if (rank != 0u) return;

  // CTA 0 alone: an entry a thread.  More than can be compared with one another are narrowed first.
  int n = (int)chosen_entries;
  bool mine = tid < n;
  const uint32_t key = mine ? list_key[tid] : 0u;
  const unsigned long long mass = mine ? mass_of(key_float(key)) : 0ull;
  if (n > FC_PAIRS) {
    while (true) {
      const uint32_t least_key = __reduce_min_sync(0xffffffffu, mine ? key : 0xffffffffu);
      const uint32_t most_key = __reduce_max_sync(0xffffffffu, mine ? key : 0u);
      if (lane == 0) sc[warp] = least_key, sm[warp] = most_key;
      __syncthreads();
      lo = __reduce_min_sync(0xffffffffu, sc[lane]), hi = __reduce_max_sync(0xffffffffu, (uint32_t)sm[lane]);
      if (n <= FC_PAIRS || lo == hi) break;
      const int shift = pattern_shift(lo, hi);
      if (mine) {
        atomicAdd(&own_count[(key - lo) >> shift], 1u);
        if (use_p) add_mass_words(own_lo, own_hi, (key - lo) >> shift, mass);
      }
      __syncthreads();
      const int at = 2 * tid;
      const unsigned int c0 = own_count[at], c1 = own_count[at + 1];
      const unsigned long long m0 = ((unsigned long long)own_hi[at] << 32) + own_lo[at];
      const unsigned long long m1 = ((unsigned long long)own_hi[at + 1] << 32) + own_lo[at + 1];
      own_count[at] = own_count[at + 1] = own_lo[at] = own_lo[at + 1] = own_hi[at] = own_hi[at + 1] = 0u;
      lo += choose_digit(c0, c1, m0, m1, false, use_k, k, use_p, p, search, sc, sm, &choice) << shift;
      hi = min(hi, lo + ((1u << shift) - 1u));
      mine = mine && key >= lo && key <= hi;
      n = __syncthreads_count(mine);
    }
    if (lo == hi) {
      if (tid == 0) threshold[r] = key_float(lo);
      return;
    }
    if (tid == 0) listed = 0u;
  }
  __syncthreads();
  if (n < (int)chosen_entries) {
    if (mine) {
      const unsigned int at = atomicAdd(&listed, 1u);
      list_key[at] = key, list_mass[at] = mass;
    }
  } else if (mine) {
    list_mass[tid] = mass;
  }
  __syncthreads();
  unsigned int above = search.above_count;
  unsigned long long above_mass = search.above_mass;
  if (mine) {
#pragma unroll 4
    for (int j = 0; j < n; ++j)
      if (list_key[j] > key) above += 1u, above_mass += list_mass[j];
  }
  const bool passes = mine && (!use_k || above < (unsigned int)k) && (!use_p || above_mass < search.mass_limit);
  const unsigned int smallest = __reduce_min_sync(0xffffffffu, passes ? key : 0xffffffffu);
  if (lane == 0) sc[warp] = smallest;
  __syncthreads();
  if (tid < 32) {
    const unsigned int found = __reduce_min_sync(0xffffffffu, sc[tid]);
    if (tid == 0) threshold[r] = key_float(found);
  }
}

// In a cluster of eight, a CTA's share of the longest row fits its shared memory.
template <int CLUSTER>
constexpr auto filter_cluster = filter_threshold_cluster_kernel<CLUSTER, CLUSTER == 8>;
template <int CLUSTER>
constexpr size_t filter_cluster_smem = FC_SMEM_BYTES + (CLUSTER == 8 ? FC_SHARE * sizeof(float) : 0);

template <int CLUSTER>
cudaError_t allow_filter_cluster() {
  static const cudaError_t ready = cudaFuncSetAttribute(filter_cluster<CLUSTER>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                                        (int)filter_cluster_smem<CLUSTER>);
  return ready;
}

// Rows that the device works on at once with this many CTAs a row.  (A CTA fills an SM, and whole clusters
// lie in a GPC: on 148 SMs there is room for 16 clusters of eight, not 18.)
template <int CLUSTER>
int filter_rows_at_once() {
  static const int rows = [] {
    if (allow_filter_cluster<CLUSTER>() != cudaSuccess) return 0;
    cudaLaunchConfig_t config = {};
    config.gridDim = dim3(CLUSTER * 64);
    config.blockDim = dim3(FILTER_THREADS);
    config.dynamicSmemBytes = filter_cluster_smem<CLUSTER>;
    cudaLaunchAttribute attribute[1];
    attribute[0].id = cudaLaunchAttributeClusterDimension;
    attribute[0].val.clusterDim.x = CLUSTER;
    attribute[0].val.clusterDim.y = attribute[0].val.clusterDim.z = 1;
    config.attrs = attribute;
    config.numAttrs = 1;
    int clusters = 0;
    if (cudaOccupancyMaxActiveClusters(&clusters, filter_cluster<CLUSTER>, &config) != cudaSuccess) {
      cudaGetLastError();
      return 0;
    }
    return clusters;
  }();
  return rows;
}

template <int CLUSTER>
cudaError_t launch_filter_cluster(const float* logits, int num_rows, int vocab, long long row_stride, const float* temperature,
                                  const int* top_k, const float* top_p, float* threshold, cudaStream_t stream) {
  const cudaError_t ready = allow_filter_cluster<CLUSTER>();
  if (ready != cudaSuccess) return ready;
  return launch_pdl_cluster(filter_cluster<CLUSTER>, dim3((unsigned)num_rows * CLUSTER), dim3(FILTER_THREADS),
                            filter_cluster_smem<CLUSTER>, CLUSTER, stream, logits, vocab, row_stride, temperature, top_k, top_p,
                            threshold);
}

// ---------------------------------------------------------------------------------------------
// Penalties.  `history` holds each request's prompt and output tokens, one row per state slot.
// counts is scratch [R, V] int32, zeroed by the first kernel.
// ---------------------------------------------------------------------------------------------
__global__ void penalty_count_kernel(const int* __restrict__ history, long long history_stride,
                                     const int* __restrict__ slots,
                                     const int* __restrict__ lengths, int* __restrict__ counts,
                                     int vocab) {
  allow_dependents();
  grid_dependency_wait();
  const int r = blockIdx.x;
  int* c = counts + (size_t)r * vocab;
  for (int i = threadIdx.x; i < vocab; i += blockDim.x) c[i] = 0;
  __syncthreads();
  const int* h = history + (size_t)slots[r] * history_stride;
  const int n = lengths[r];
  for (int i = threadIdx.x; i < n; i += blockDim.x) {
    const int v = h[i];
    if (v >= 0 && v < vocab) atomicAdd(&c[v], 1);
  }
}

__global__ void penalty_apply_kernel(float* __restrict__ logits, long long row_stride,
                                     const int* __restrict__ counts, int vocab,
                                     const float* __restrict__ repetition,
                                     const float* __restrict__ presence,
                                     const float* __restrict__ frequency) {
  allow_dependents();
  grid_dependency_wait();
  const int r = blockIdx.x;
  float* row = logits + (size_t)r * row_stride;
  const int* c = counts + (size_t)r * vocab;
  const float rep = repetition[r], pres = presence[r], freq = frequency[r];
  for (int i = threadIdx.x; i < vocab; i += blockDim.x) {
    const int n = c[i];
    if (n == 0) continue;
    float x = row[i] - freq * (float)n;
    x = x > 0.f ? x / rep : x * rep;
    row[i] = x - pres;
  }
}

}  // namespace vx

using namespace vx;

// How many segments vx_sample cuts a row into, and with that the size of its scratch:
// `partial` holds num_rows * segments pairs (float, int), `counters` num_rows zeroed uint32
// (the kernel leaves them zero).  Both may be null when the answer is 1.
VX_API int vx_sample_segments(int num_rows, int vocab) {
  if (num_rows <= 0 || vocab < 8192) return 1;
  // About two blocks per SM, and no segment below 2,048 entries.
  int segments = (2 * 148 + num_rows - 1) / num_rows;
  const int most = vocab / 2048;
  if (segments > most) segments = most;
  if (segments > SAMPLE_MAX_SEGMENTS) segments = SAMPLE_MAX_SEGMENTS;
  return segments < 1 ? 1 : segments;
}

VX_API int vx_sample(const float* logits, int num_rows, int vocab, long long row_stride,
                     const float* temperature, const unsigned long long* seeds,
                     const int* draw_index, const float* threshold, int* out, int* history,
                     long long history_stride, const int* history_slots,
                     const int* history_lengths, void* partial, unsigned int* counters,
                     const int* status_word, cudaStream_t stream) {
  if (num_rows <= 0) return 0;
  int segments = vx_sample_segments(num_rows, vocab);
  if (partial == nullptr || counters == nullptr) segments = 1;
  // Segments are multiples of four entries.
  const int segment_len = (((vocab + segments - 1) / segments) + 3) / 4 * 4;
  segments = (vocab + segment_len - 1) / segment_len;
  launch_pdl(sample_kernel, dim3(num_rows, segments), dim3(SAMPLE_THREADS), 0, stream, logits, vocab,
             row_stride, temperature, seeds, draw_index, threshold, out, history, history_stride,
             history_slots, history_lengths, segment_len, (Best*)partial, counters, status_word);
  return (int)cudaGetLastError();
}

// kind 0: the cluster kernel for rows of up to 196,608 entries, else one CTA a row; 1: one CTA a
// row; 2: the cluster kernel or an error.
VX_API int vx_filter_threshold(const float* logits, int num_rows, int vocab, long long row_stride,
                               const float* temperature, const int* top_k, const float* top_p,
                               float* threshold, int kind, cudaStream_t stream) {
  if (num_rows <= 0) return 0;
  static bool configured = false;
  if (!configured) {
    cudaError_t e = cudaFuncSetAttribute(filter_threshold_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                         (int)FILTER_SMEM_BYTES);
    if (e != cudaSuccess) return (int)e;
    configured = true;
  }
  if (kind == 2 && vocab > FC_MAX_VOCAB) return (int)cudaErrorInvalidValue;
  if (kind != 1 && vocab <= FC_MAX_VOCAB) {
    // The largest cluster with which all rows run at once.
    const auto launch = num_rows <= filter_rows_at_once<8>() ? launch_filter_cluster<8>
                        : num_rows <= filter_rows_at_once<4>() ? launch_filter_cluster<4> : launch_filter_cluster<2>;
    return (int)launch(logits, num_rows, vocab, row_stride, temperature, top_k, top_p, threshold, stream);
  }
  launch_pdl(filter_threshold_kernel, dim3(num_rows), dim3(FILTER_THREADS), FILTER_SMEM_BYTES, stream, logits, vocab, row_stride,
                                                            temperature, top_k, top_p, threshold);
  return (int)cudaGetLastError();
}

VX_API int vx_apply_penalties(float* logits, int num_rows, int vocab, long long row_stride,
                              const int* history, long long history_stride, const int* slots,
                              const int* lengths, int* counts, const float* repetition,
                              const float* presence, const float* frequency,
                              cudaStream_t stream) {
  if (num_rows <= 0) return 0;
  launch_pdl(penalty_count_kernel, dim3(num_rows), dim3(256), 0, stream, history, history_stride, slots, lengths,
                                                     counts, vocab);
  launch_pdl(penalty_apply_kernel, dim3(num_rows), dim3(256), 0, stream, logits, row_stride, counts, vocab,
                                                     repetition, presence, frequency);
  return (int)cudaGetLastError();
}
