// Acceptance sampler of the verify step: row argmax, greedy prefix acceptance with the
// device state update, token draws with explicit uniforms and rejection sampling with
// residual resampling.
//
// All of these are streaming reductions over [rows, vocab] logits (HBM-bound: rows * vocab *
// sizeof(T) bytes, a few flops per byte).  Argmax is exact and order independent (a packed
// (value, lowest index) key reduced with max).  The probabilistic kernels use the canonical
// arithmetic of include/rlt_canonical.h — an exp built from IEEE fused multiply-adds and
// 2^-40 fixed-point integer sums — so their results are identical to the CPU oracle's for
// any thread count or reduction shape.
#include "common.cuh"

#include "../../include/rlt_canonical.h"

namespace rlt {
namespace {

constexpr int kArgmaxThreads = 512;
constexpr int kSampleThreads = 1024;

// ---- packed argmax key ------------------------------------------------------------------
// Larger key = better candidate: NaN above every number, then by value (-0 == +0), then the
// LOWER index.  max() over keys therefore reproduces torch.argmax.
__device__ __forceinline__ unsigned long long argmax_key(float x, int index) {
  uint32_t bits;
  if (x != x) {
    bits = 0xffffffffu;
  } else {
    if (x == 0.0f) x = 0.0f;  // -0 -> +0
    bits = __float_as_uint(x);
    bits = (bits & 0x80000000u) ? ~bits : (bits | 0x80000000u);
  }
  return (static_cast<unsigned long long>(bits) << 32) | (0xffffffffu - static_cast<uint32_t>(index));
}
__device__ __forceinline__ int key_index(unsigned long long key) {
  return static_cast<int>(0xffffffffu - static_cast<uint32_t>(key & 0xffffffffu));
}

__device__ __forceinline__ unsigned long long warp_max(unsigned long long v) {
#pragma unroll
  for (int x = 16; x > 0; x >>= 1) {
    const unsigned long long o = __shfl_xor_sync(0xffffffffu, v, x);
    v = o > v ? o : v;
  }
  return v;
}
__device__ __forceinline__ unsigned long long warp_sum(unsigned long long v) {
#pragma unroll
  for (int x = 16; x > 0; x >>= 1) v += __shfl_xor_sync(0xffffffffu, v, x);
  return v;
}

// Block-wide reductions for kThreads threads; every thread receives the result.
template <int kThreads>
__device__ __forceinline__ unsigned long long block_max(unsigned long long v, unsigned long long* scratch) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  v = warp_max(v);
  __syncthreads();
  if (lane == 0) scratch[warp] = v;
  __syncthreads();
  v = lane < kThreads / 32 ? scratch[lane] : 0ull;
  return warp_max(v);
}
template <int kThreads>
__device__ __forceinline__ unsigned long long block_sum(unsigned long long v, unsigned long long* scratch) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  v = warp_sum(v);
  __syncthreads();
  if (lane == 0) scratch[warp] = v;
  __syncthreads();
  v = lane < kThreads / 32 ? scratch[lane] : 0ull;
  return warp_sum(v);
}

// Packed (value, lowest index) maximum of one row by the whole CTA.  16-byte loads when the row
// allows them, four in flight per thread (a row is only a few hundred KB: latency, not issue
// rate, decides how fast one CTA can stream it).
template <typename T, int kThreads>
__device__ __forceinline__ unsigned long long block_max_key(const T* __restrict__ row, int vocab,
                                                           unsigned long long* scratch) {
  constexpr int kVec = 16 / sizeof(T);
  constexpr int kDepth = 4;
  unsigned long long best = 0ull;
  if ((reinterpret_cast<uintptr_t>(row) & 15u) == 0 && vocab % kVec == 0) {
    const uint4* rv = reinterpret_cast<const uint4*>(row);
    const int nvec = vocab / kVec;
    for (int base = threadIdx.x; base < nvec; base += kThreads * kDepth) {
      uint4 raw[kDepth];
#pragma unroll
      for (int k = 0; k < kDepth; ++k) {
        const int i = base + k * kThreads;
        if (i < nvec) raw[k] = __ldcs(rv + i);
      }
#pragma unroll
      for (int k = 0; k < kDepth; ++k) {
        const int i = base + k * kThreads;
        if (i < nvec) {
          const T* e = reinterpret_cast<const T*>(&raw[k]);
#pragma unroll
          for (int j = 0; j < kVec; ++j) {
            const unsigned long long key = argmax_key(Elem<T>::to_float(e[j]), i * kVec + j);
            best = key > best ? key : best;
          }
        }
      }
    }
  } else {
    for (int i = threadIdx.x; i < vocab; i += kThreads) {
      const unsigned long long key = argmax_key(Elem<T>::to_float(row[i]), i);
      best = key > best ? key : best;
    }
  }
  return block_max<kThreads>(best, scratch);
}

template <typename T, int kThreads>
__device__ __forceinline__ int block_argmax(const T* __restrict__ row, int vocab, unsigned long long* scratch) {
  return key_index(block_max_key<T, kThreads>(row, vocab, scratch));
}

template <typename T>
__global__ void __launch_bounds__(kArgmaxThreads)
argmax_rows_kernel(const T* __restrict__ logits, int64_t row_stride, int vocab, int64_t* __restrict__ targets) {
  __shared__ unsigned long long scratch[32];
  const int index = block_argmax<T, kArgmaxThreads>(logits + static_cast<int64_t>(blockIdx.x) * row_stride, vocab, scratch);
  if (threadIdx.x == 0) targets[blockIdx.x] = index;
}

// Rows of request i: the span cu_rows[i] .. cu_rows[i+1]-1, of which only the first
// row_counts[i] are real when row_counts is given (a fixed-shape round pads every request to the
// same span).  Zero rows: the request is left alone (accepted 0, next position = its start, no
// slot update).
__device__ __forceinline__ int request_rows(const int32_t* __restrict__ cu_rows, const int32_t* __restrict__ row_counts,
                                            int i, int* first, int* span) {
  *first = cu_rows[i];
  *span = cu_rows[i + 1] - cu_rows[i];
  const int c = row_counts != nullptr ? min(row_counts[i], *span) : *span;
  return c > 0 ? c : 0;
}

// One thread per request: matching prefix, next token / position, slot update, wire buffer.
__global__ void greedy_finish_kernel(const int32_t* __restrict__ cu_rows, int n, int rows,
                                     const int32_t* __restrict__ row_counts,
                                     const int64_t* __restrict__ tokens, int tokens_width,
                                     const int64_t* __restrict__ starts, const int64_t* __restrict__ slots,
                                     int64_t* __restrict__ slot_values, int64_t* __restrict__ result) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  int a, span;
  const int c = request_rows(cu_rows, row_counts, i, &a, &span);
  for (int j = c; j < span; ++j) result[a + j] = -1;  // padding rows carry no target
  if (c == 0) {
    result[rows + i] = 0;
    result[rows + n + i] = starts[i];
    return;
  }
  const int64_t* tok = tokens + static_cast<int64_t>(i) * tokens_width;
  int accepted = 0;
  while (accepted < c - 1 && tok[accepted + 1] == result[a + accepted]) ++accepted;
  const int64_t next_token = result[a + accepted];
  const int64_t next_pos = starts[i] + accepted + 1;
  result[rows + i] = accepted;
  result[rows + n + i] = next_pos;
  if (slots != nullptr && slot_values != nullptr) {
    slot_values[2 * slots[i]] = next_token;
    slot_values[2 * slots[i] + 1] = next_pos;
  }
}

// ---- canonical distributions ----------------------------------------------------------
// Support of a row after top-k / top-p: the prefix of the ranking (scaled logit descending,
// token index ascending) that ends at (key, limit); see rlt_in_support.
struct Cut {
  uint32_t key;
  int limit;
};
__device__ __forceinline__ Cut whole_row() { return Cut{0u, 0x7fffffff}; }

struct RowNorm {
  float m;   // max of logits / T
  float z;   // normaliser over the support (from the fixed-point sum)
  int ok;    // 0: NaN / +inf / all -inf
  Cut cut;   // support of the distribution
};

template <typename T>
__device__ __forceinline__ float scaled_logit(const T* row, int v, float temperature) {
  return RLT_DIV(Elem<T>::to_float(row[v]), temperature);
}

// f(value, index) for every element of the row by the whole CTA, in no particular order: 16-byte loads, kDepth in flight per
// thread, and what lies in front of the first 16-byte boundary and behind the last one by itself, so that rows of any width and
// alignment are read alike (top-p of 148 rows of 50 257 fp32 logits: 94 us, 129 with such rows read element by element).  A row is a few hundred
// KB: the first pass over it reads HBM, the others L2.
template <typename T, int kThreads, int kDepth = 4, typename F>
__device__ __forceinline__ void for_row(const T* __restrict__ row, int vocab, F f) {
  constexpr int kVec = 16 / sizeof(T);
  const int head = min(static_cast<int>((-reinterpret_cast<uintptr_t>(row) & 15u) / sizeof(T)), vocab), nvec = (vocab - head) / kVec;
  const uint4* rv = reinterpret_cast<const uint4*>(row + head);
  const int alone = static_cast<int>(threadIdx.x) < head ? threadIdx.x : threadIdx.x + nvec * kVec;    // at most 14 of them
  float x = 0.0f;
  if (alone < vocab) x = Elem<T>::to_float(row[alone]);
  for (int base = threadIdx.x; base < nvec; base += kThreads * kDepth) {
    uint4 raw[kDepth];
#pragma unroll
    for (int k = 0; k < kDepth; ++k)
      if (base + k * kThreads < nvec) raw[k] = __ldg(rv + base + k * kThreads);
#pragma unroll
    for (int k = 0; k < kDepth; ++k) {
      const int i = base + k * kThreads;
      if (i < nvec) {
        const T* e = reinterpret_cast<const T*>(&raw[k]);
#pragma unroll
        for (int j = 0; j < kVec; ++j) f(Elem<T>::to_float(e[j]), head + i * kVec + j);
      }
    }
  }
  if (alone < vocab) f(x, alone);
}

// A raw value below which no logit can have a scaled value >= t (rounding of the division and of this product included):
// most tokens are outside a support and are dismissed by one comparison.
__device__ __forceinline__ float raw_floor(float t, float temperature) {
  const float x = t * temperature;
  const float floor = x - (fabsf(x) * 0x1p-20f + temperature * 0x1p-140f + 0x1p-120f);
  return floor == floor ? floor : -INFINITY;           // an infinite product says nothing
}
__device__ __forceinline__ float key_value(uint32_t key) {
  return __uint_as_float((key & 0x80000000u) ? (key & 0x7fffffffu) : ~key);
}
// The same for the tokens of a cut; -inf where everything belongs to it.
__device__ __forceinline__ float cut_floor(Cut cut, float temperature) {
  return cut.key == 0u ? -INFINITY : raw_floor(key_value(cut.key), temperature);
}

// Normaliser of softmax(row / temperature) over the whole row.
template <typename T, int kThreads>
__device__ __forceinline__ float block_full_sum(const T* __restrict__ row, int vocab, float temperature, float m,
                                                unsigned long long* scratch) {
  unsigned long long zfix = 0ull;
  for_row<T, kThreads, 2>(row, vocab, [&](float x, int) {
    zfix += rlt_fix_weight(rlt_expf(RLT_SUB(RLT_DIV(x, temperature), m)));
  });
  return rlt_fix_to_float(block_sum<kThreads>(zfix, scratch));
}

// Normaliser over the tokens inside `cut`.
template <typename T, int kThreads>
__device__ __forceinline__ float block_cut_sum(const T* __restrict__ row, int vocab, float temperature, float m,
                                               Cut cut, unsigned long long* scratch) {
  unsigned long long zfix = 0ull;
  const float floor = cut_floor(cut, temperature);
  for_row<T, kThreads>(row, vocab, [&](float x, int v) {
    if (x >= floor) {
      const float t = RLT_DIV(x, temperature);
      if (rlt_in_support(rlt_order_key(t), v, cut.key, cut.limit)) zfix += rlt_fix_weight(rlt_expf(RLT_SUB(t, m)));
    }
  });
  return rlt_fix_to_float(block_sum<kThreads>(zfix, scratch));
}

// ---- top-k / top-p: selection over the ranking ----------------------------------------------
// Both filters keep the ranks whose exclusive prefix WEIGHT is <= a limit: weight 1 per token
// and limit k - 1 for top-k, the fixed-point probability mass and rlt_top_p_limit for top-p.
// Integer weights make the cut independent of how it is found.  Three ways, all over the row where it lies (L2 after the first
// pass), several CTAs per SM:
//   candidates   top-k up to a token per thread: at least k tokens reach the k-th largest of the threads' own maxima, so the few
//                tokens at or above that value (70 for k = 50 of 49 152) hold the whole answer, and top-p inside it.
//   buckets      every other filter: a histogram of weight over the distance from the maximum finds the step in which the running
//                weight first exceeds the limit; its tokens are the candidates, or are divided once more where they do not fit.
//                Steps are as wide as the row is spread, so a flat row fills as many of them as a peaked one.
//   digits       what is left (values that a step cannot tell apart): a radix select over four 8-bit digits of the order key.
// 128 requests of 5 rows of 49 152 fp32 logits, half of them with top-k 50 and top-p 0.95: 107 us.  One row of 49 152, top-p 0.95 alone: 74 us of
// which 37 are the draw without a filter; 87 us where all logits lie within a hundredth of each other, 206 us where all are equal.  Top-k
// 50 of it: 23 us with one warp ranking the 70 candidates, 42 with the whole CTA, whose every bit of the key costs two barriers.
constexpr int kCandidates = 2048;
constexpr int kBuckets = 2048;
constexpr int kWarpCandidates = 128;        // up to this many are ranked by one warp, from registers

struct SelectScratch {
  union {
    struct {                                // candidates
      unsigned long long weight[kCandidates];
      uint32_t key[kCandidates];
      int index[kCandidates];
    };
    unsigned long long bucket[kBuckets];
  };
  unsigned long long mass[256];             // the digits' histogram
  unsigned int count[256];
  unsigned long long above;
  int digit;
  int found;
  int listed;
  uint32_t lowest, highest;                 // keys of the candidates
  Cut cut;
  int warp_counts[32];
};

// Sums of lanes' weights that are below 2^44 together per lane: two 22-bit halves, so that 32 of them fit a word.
__device__ __forceinline__ unsigned long long sum_weights(unsigned lanes, unsigned long long w) {
  const unsigned low = __reduce_add_sync(lanes, static_cast<unsigned>(w & 0x3fffffu));
  const unsigned high = __reduce_add_sync(lanes, static_cast<unsigned>(w >> 22));
  return (static_cast<unsigned long long>(high) << 22) + low;
}

// Adds a token to the candidates, one atomic for the lanes that are here together; those that do not fit are only counted.
__device__ __forceinline__ void list_token(SelectScratch& h, uint32_t key, int index, unsigned long long weight) {
  const unsigned here = __activemask();
  const int lane = threadIdx.x & 31, first = __ffs(here) - 1;
  int at = 0;
  if (lane == first) at = atomicAdd(&h.listed, __popc(here));
  at = __shfl_sync(here, at, first) + __popc(here & ((1u << lane) - 1u));
  if (at < kCandidates) { h.key[at] = key; h.index[at] = index; h.weight[at] = weight; }
}

// Adds to a bucket by atomics on its two words, the low one's carry going into the high one: 32-bit adds are done by the memory itself, a 64-bit
// one retries for as long as other lanes get in between (top-p of a row of 49 152 equal logits: 206 us, with 64-bit atomics 2144).
__device__ __forceinline__ void bucket_add(SelectScratch& h, int bucket, unsigned long long w) {
  unsigned* word = reinterpret_cast<unsigned*>(&h.bucket[bucket]);
  const unsigned low = static_cast<unsigned>(w), before = atomicAdd(word, low);
  const unsigned high = static_cast<unsigned>(w >> 32) + (before + low < low ? 1u : 0u);
  if (high != 0u) atomicAdd(word + 1, high);
}
// One shared-memory atomic per distinct digit in the warp: lanes with the same digit find each other with match.any and add their weights
// (below 2^41) first.  The leading byte of the key has only a few populated values.
template <bool kByMass>
__device__ __forceinline__ void digit_add(SelectScratch& h, int digit, unsigned long long w, bool valid) {
  const int lane = threadIdx.x & 31;
  const unsigned peers = __match_any_sync(0xffffffffu, valid ? digit : 0x7fff);
  const bool leader = valid && lane == __ffs(peers) - 1;
  if (kByMass) {
    const unsigned long long sum = sum_weights(peers, w);
    if (leader) atomicAdd(&h.mass[digit], sum);
  }
  if (leader) atomicAdd(&h.count[digit], static_cast<unsigned int>(__popc(peers)));
}

// The key at which the running weight of `count` items, ranked by key from the largest on and starting at `above`, first exceeds the limit:
// four passes over 8-bit digits, most significant first.  item(i, &key, &weight) says whether item i counts.  False where the limit is never
// exceeded.  `ties` items have the key and a weight of `each`; those before them add up to `before`.
struct Crossing { uint32_t key; unsigned int ties; unsigned long long each, before; };
template <int kThreads, bool kByMass, typename Item>
__device__ __forceinline__ bool digit_select(SelectScratch& h, int count, unsigned long long above, unsigned long long limit, Crossing* at, Item item) {
  uint32_t prefix = 0u;
  for (int pass = 0; pass < 4; ++pass) {
    const int shift = 24 - 8 * pass;
    __syncthreads();
    for (int i = threadIdx.x; i < 256; i += kThreads) { h.mass[i] = 0ull; h.count[i] = 0u; }
    __syncthreads();
    for (int base = 0; base < count; base += kThreads) {
      const int i = base + static_cast<int>(threadIdx.x);
      uint32_t key = 0u;
      unsigned long long w = 0ull;
      const bool valid = i < count && item(i, &key, pass, prefix >> (shift + 7) >> 1, &w);
      digit_add<kByMass>(h, static_cast<int>((key >> shift) & 255u), w, valid);
    }
    __syncthreads();
    if (threadIdx.x < 32) {
      // lane l scans digits 255 - 8l down to 248 - 8l
      const int lane = threadIdx.x, hi = 255 - 8 * lane;
      unsigned long long local = 0ull;
#pragma unroll
      for (int j = 0; j < 8; ++j) local += kByMass ? h.mass[hi - j] : static_cast<unsigned long long>(h.count[hi - j]);
      unsigned long long inc = local;
#pragma unroll
      for (int x = 1; x < 32; x <<= 1) {
        const unsigned long long o = __shfl_up_sync(0xffffffffu, inc, x);
        if (lane >= x) inc += o;
      }
      const unsigned crossing = __ballot_sync(0xffffffffu, above + inc > limit);
      if (crossing == 0u) {
        if (lane == 0) h.digit = -1;
      } else if (lane == __ffs(crossing) - 1) {
        unsigned long long acc = above + inc - local;
        int digit = hi;
        for (int j = 0; j < 8; ++j) {
          const unsigned long long wd = kByMass ? h.mass[hi - j] : static_cast<unsigned long long>(h.count[hi - j]);
          digit = hi - j;
          if (acc + wd > limit) break;
          acc += wd;
        }
        h.digit = digit;
        h.above = acc;
      }
    }
    __syncthreads();
    if (h.digit < 0) return false;
    prefix |= static_cast<uint32_t>(h.digit) << shift;
    above = h.above;
  }
  at->key = prefix;
  at->before = above;
  at->ties = h.count[prefix & 255u];
  at->each = kByMass ? h.mass[prefix & 255u] / at->ties : 1ull;
  return true;
}

// The cut among n listed candidates, `above` being the weight of the tokens ranked before all of them.  A candidate that no longer counts
// has weight 0 and key 0.  The running weight must exceed the limit inside the list.
template <int kThreads>
__device__ __noinline__ Cut list_select(SelectScratch& h, int n, unsigned long long above, unsigned long long limit, Cut outer) {
  if (n <= kWarpCandidates) {
    __syncthreads();
    if (threadIdx.x < 32) {
      constexpr int kOwn = kWarpCandidates / 32;
      const int lane = threadIdx.x;
      uint32_t own_key[kOwn];
      unsigned long long own[kOwn];
#pragma unroll
      for (int i = 0; i < kOwn; ++i) {
        own_key[i] = lane + 32 * i < n ? h.key[lane + 32 * i] : 0u;
        own[i] = lane + 32 * i < n ? h.weight[lane + 32 * i] : 0ull;
      }
      auto weight_from = [&](uint32_t from) {
        unsigned long long sum = 0ull;
#pragma unroll
        for (int i = 0; i < kOwn; ++i) sum += own_key[i] >= from ? own[i] : 0ull;
        return sum_weights(0xffffffffu, sum);
      };
      uint32_t key = 0u;                    // the largest key for which the weight of all tokens from it on exceeds the limit
      for (int bit = 31; bit >= 0; --bit)
        if (above + weight_from(key | (1u << bit)) > limit) key |= 1u << bit;
      const unsigned long long before = above + weight_from(key + 1u);
      int ties = 0;
      unsigned long long each = 0ull;
#pragma unroll
      for (int i = 0; i < kOwn; ++i) {
        const unsigned tied = __ballot_sync(0xffffffffu, own_key[i] == key);
        if (tied != 0u) each = __shfl_sync(0xffffffffu, own[i], __ffs(tied) - 1);
        ties += __popc(tied);
      }
      const unsigned long long keep = (limit - before) / each + 1ull;
      int index = key == outer.key ? outer.limit : 0x7fffffff;
      if (keep < static_cast<unsigned long long>(ties)) {
        index = 0;                          // the largest index with fewer than `keep` of the tied tokens before it
        for (int bit = 30; bit >= 0; --bit) {
          const int next = index | (1 << bit);
          int smaller = 0;
#pragma unroll
          for (int i = 0; i < kOwn; ++i)
            smaller += __popc(__ballot_sync(0xffffffffu, own_key[i] == key && h.index[lane + 32 * i] < next));
          if (smaller < static_cast<int>(keep)) index = next;
        }
      }
      if (lane == 0) h.cut = Cut{key, index};
    }
    __syncthreads();
    return h.cut;
  }
  Crossing at;
  digit_select<kThreads, true>(h, n, above, limit, &at, [&](int j, uint32_t* key, int pass, uint32_t chosen, unsigned long long* w) {
    *key = h.key[j];
    *w = h.weight[j];
    return *key >> (31 - 8 * pass) >> 1 == chosen;
  });
  const unsigned long long keep = (limit - at.before) / at.each + 1ull;
  if (keep >= at.ties) return Cut{at.key, at.key == outer.key ? outer.limit : 0x7fffffff};
  Crossing last;                            // the keep-th of the tied tokens, smallest index first
  digit_select<kThreads, false>(h, n, 0ull, keep - 1ull, &last, [&](int j, uint32_t* key, int pass, uint32_t chosen, unsigned long long* w) {
    *key = 0xffffffffu - static_cast<uint32_t>(h.index[j]);
    return h.key[j] == at.key && *key >> (31 - 8 * pass) >> 1 == chosen;
  });
  return Cut{at.key, static_cast<int>(0xffffffffu - last.key)};
}

// Index of the n-th (1-based) token in ascending index order with order key `key` inside `outer`.
template <typename T, int kThreads>
__device__ __forceinline__ int block_nth_index(const T* __restrict__ row, int vocab, float temperature,
                                               uint32_t key, Cut outer, unsigned int n, SelectScratch& h) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  if (threadIdx.x == 0) h.found = 0x7fffffff;
  unsigned int running = 0;
  for (int base = 0; base < vocab; base += kThreads) {
    const int v = base + static_cast<int>(threadIdx.x);
    bool flag = false;
    if (v < vocab) {
      const uint32_t k = rlt_order_key(scaled_logit(row, v, temperature));
      flag = k == key && rlt_in_support(k, v, outer.key, outer.limit);
    }
    const unsigned ballot = __ballot_sync(0xffffffffu, flag);
    __syncthreads();
    if (lane == 0) h.warp_counts[warp] = __popc(ballot);
    __syncthreads();
    unsigned int before = running, total = 0;
    for (int w = 0; w < kThreads / 32; ++w) {
      const unsigned int c = h.warp_counts[w];
      if (w < warp) before += c;
      total += c;
    }
    if (flag && before + __popc(ballot & ((1u << lane) - 1u)) + 1u == n) h.found = v;
    running += total;
    if (running >= n) break;  // uniform: every thread computes the same totals
  }
  __syncthreads();
  return h.found;
}

// The cut of the tokens in `outer`: by buckets; `inv` is 1 / z, `own` the thread's largest raw logit.
template <typename T, int kThreads, bool kByMass>
__device__ __forceinline__ Cut bucket_select(const T* __restrict__ row, int vocab, float temperature, float m, float inv, float own, Cut outer,
                                             unsigned long long limit, unsigned long long* scratch, SelectScratch& h) {
  constexpr int kOwn = kBuckets / kThreads;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const auto weight = [&](float t) { return kByMass ? rlt_fix_weight(rlt_draw_mass(rlt_expf(RLT_SUB(t, m)), inv)) : 1ull; };
  const auto cut_of_ties = [&](uint32_t key, unsigned long long ties, unsigned long long each, unsigned long long before) {
    const unsigned long long keep = (limit - before) / each + 1ull;
    if (keep >= ties) return Cut{key, key == outer.key ? outer.limit : 0x7fffffff};
    return Cut{key, block_nth_index<T, kThreads>(row, vocab, temperature, key, outer, static_cast<unsigned int>(keep), h)};
  };
  if (vocab <= kCandidates) {               // the whole row fits the list
    unsigned long long sum = 0ull;
    __syncthreads();
    for (int v = threadIdx.x; v < vocab; v += kThreads) {
      const float t = scaled_logit(row, v, temperature);
      const uint32_t key = rlt_order_key(t);
      const unsigned long long w = rlt_in_support(key, v, outer.key, outer.limit) ? weight(t) : 0ull;
      h.key[v] = w != 0ull ? key : 0u;
      h.index[v] = v;
      h.weight[v] = w;
      sum += w;
    }
    if (block_sum<kThreads>(sum, scratch) <= limit) return outer;
    return list_select<kThreads>(h, vocab, 0ull, limit, outer);
  }
  // Steps of the first histogram: four times the mean distance of the threads' own maxima, which the bulk of a row stays within however flat or
  // peaked it is; masses end 28 below the maximum.
  float distance = own == -INFINITY ? 0.0f : RLT_SUB(m, RLT_DIV(own, temperature)), holders = own == -INFINITY ? 0.0f : 1.0f;
#pragma unroll
  for (int x = 16; x > 0; x >>= 1) {
    distance += __shfl_xor_sync(0xffffffffu, distance, x);
    holders += __shfl_xor_sync(0xffffffffu, holders, x);
  }
  __syncthreads();
  if (lane == 0) scratch[warp] = static_cast<unsigned long long>(__float_as_uint(distance)) << 32 | __float_as_uint(holders);
  __syncthreads();
  distance = holders = 0.0f;
  for (int w = 0; w < kThreads / 32; ++w) {
    distance += __uint_as_float(static_cast<uint32_t>(scratch[w] >> 32));
    holders += __uint_as_float(static_cast<uint32_t>(scratch[w]));
  }
  float range = 4.0f * distance / holders;
  if (kByMass) range = fminf(range, 31.0f);
  float top = m;
  uint32_t low = 0u, high = 0xffffffffu;    // keys of the tokens that are being told apart
  unsigned long long above = 0ull;          // weight of those ranked before them
  for (int level = 0; level < 3; ++level) {
    const float floor = fmaxf(cut_floor(outer, temperature), level == 0 ? -INFINITY : raw_floor(key_value(low), temperature));
    const float scale = fminf((kBuckets - 2) / range, 0x1p120f);
    // a step, never a smaller one for a smaller t
    const auto bucket_of = [&](float t) { return static_cast<int>(fminf(fmaxf(RLT_SUB(top, t), 0.0f) * scale, kBuckets - 1.0f)); };
    const auto among = [&](uint32_t key, int v) { return key >= low && key <= high && rlt_in_support(key, v, outer.key, outer.limit); };
    __syncthreads();
    for (int i = threadIdx.x; i < kBuckets; i += kThreads) h.bucket[i] = 0ull;
    if (threadIdx.x == 0) { h.digit = -1; h.listed = 0; h.lowest = 0xffffffffu; h.highest = 0u; }
    __syncthreads();
    for_row<T, kThreads, 2>(row, vocab, [&](float x, int v) {
      if (x >= floor) {
        const float t = RLT_DIV(x, temperature);
        if (among(rlt_order_key(t), v)) {
          const unsigned long long w = weight(t);
          if (kByMass) {
            if (w != 0ull) bucket_add(h, bucket_of(t), w);
          } else {
            atomicAdd(reinterpret_cast<unsigned*>(&h.bucket[bucket_of(t)]), 1u);
          }
        }
      }
    });
    __syncthreads();
    // thread i scans buckets kOwn * i ..
    unsigned long long held[kOwn], local = 0ull;
#pragma unroll
    for (int j = 0; j < kOwn; ++j) { held[j] = h.bucket[kOwn * threadIdx.x + j]; local += held[j]; }
    unsigned long long before = local;
#pragma unroll
    for (int x = 1; x < 32; x <<= 1) {
      const unsigned long long o = __shfl_up_sync(0xffffffffu, before, x);
      if (lane >= x) before += o;
    }
    if (lane == 31) scratch[warp] = before;
    __syncthreads();
    before += above - local;
    for (int w = 0; w < warp; ++w) before += scratch[w];
    if (before <= limit && before + local > limit) {      // one thread at most
#pragma unroll
      for (int j = 0; j < kOwn; ++j) {
        if (h.digit < 0) {
          if (before + held[j] > limit) { h.digit = kOwn * threadIdx.x + j; h.above = before; }
          before += held[j];
        }
      }
    }
    __syncthreads();
    const int crossing = h.digit;
    above = h.above;
    if (crossing < 0) return outer;         // everything stays
    uint32_t lowest = 0xffffffffu, highest = 0u;
    for_row<T, kThreads>(row, vocab, [&](float x, int v) {
      if (x >= floor) {
        const float t = RLT_DIV(x, temperature);
        const uint32_t key = rlt_order_key(t);
        if (bucket_of(t) == crossing && among(key, v)) {
          const unsigned long long w = weight(t);
          if (w != 0ull) {
            lowest = min(lowest, key);
            highest = max(highest, key);
            list_token(h, key, v, w);
          }
        }
      }
    });
    lowest = __reduce_min_sync(0xffffffffu, lowest);
    highest = __reduce_max_sync(0xffffffffu, highest);
    if (lane == 0) { atomicMin(&h.lowest, lowest); atomicMax(&h.highest, highest); }
    __syncthreads();
    const int n = h.listed;
    if (n <= kCandidates) return list_select<kThreads>(h, n, above, limit, outer);
    low = h.lowest;
    high = h.highest;
    if (low == high) return cut_of_ties(low, n, weight(key_value(low)), above);
    top = key_value(high);
    range = RLT_SUB(top, key_value(low));
  }
  Crossing at;
  const float floor = raw_floor(key_value(low), temperature);
  digit_select<kThreads, kByMass>(h, vocab, above, limit, &at, [&](int v, uint32_t* key, int pass, uint32_t chosen, unsigned long long* w) {
    const float x = Elem<T>::to_float(row[v]);
    if (!(x >= floor)) return false;
    const float t = RLT_DIV(x, temperature);
    *key = rlt_order_key(t);
    if (*key < low || *key > high || !rlt_in_support(*key, v, outer.key, outer.limit) || *key >> (31 - 8 * pass) >> 1 != chosen) return false;
    *w = weight(t);
    return *w != 0ull;
  });
  return cut_of_ties(at.key, at.ties, at.each, at.before);
}

// max of row / temperature, and the thread's own largest raw logit.  Division by a positive temperature is monotonic, so
// max_v (x_v / T) == (max_v x_v) / T exactly: the pass is a plain maximum over the raw logits, one division at the end.
template <typename T, int kThreads>
__device__ __forceinline__ RowNorm block_row_max(const T* __restrict__ row, int vocab, float temperature, unsigned long long* scratch,
                                                 float* own) {
  float largest = -INFINITY;
  bool nan = false;
  for_row<T, kThreads>(row, vocab, [&](float x, int) {
    largest = fmaxf(largest, x);
    nan |= x != x;
  });
  *own = largest;
  const uint32_t top = __reduce_max_sync(0xffffffffu, nan ? 0xffffffffu : rlt_order_key(largest));
  RowNorm n;
  const uint32_t best = static_cast<uint32_t>(block_max<kThreads>(top, scratch));
  n.m = best == 0xffffffffu ? NAN : RLT_DIV(key_value(best), temperature);
  n.ok = n.m == n.m && n.m != INFINITY && n.m != -INFINITY;
  n.z = 0.0f;
  n.cut = whole_row();
  return n;
}

// max, support and normaliser of the distribution Sampler.probabilities builds for one row
// (vllm_rlt/worker/sampler.py:37-55): softmax(row / T) restricted to top-k, then to top-p.
// top_k <= 0 or >= vocab and top_p >= 1 switch the filters off.
template <typename T, int kThreads>
__device__ __forceinline__ RowNorm block_normalise(const T* __restrict__ row, int vocab, float temperature,
                                                   int top_k, float top_p, unsigned long long* scratch,
                                                   SelectScratch& h) {
  const bool use_k = top_k > 0 && top_k < vocab, use_p = top_p < 1.0f;
  float own;
  RowNorm n = block_row_max<T, kThreads>(row, vocab, temperature, scratch, &own);
  if (!n.ok) return n;
  const uint32_t own_key = rlt_order_key(own);
  const unsigned long long limit_p = rlt_top_p_limit(top_p);
  if (use_k) {
    int listed = kCandidates + 1;
    if (top_k <= kThreads) {
      uint32_t reached = 0u;                // at least top_k of the threads' maxima, in 18 bits
      for (int bit = 31; bit >= 14; --bit)
        if (__syncthreads_count(own_key >= (reached | (1u << bit))) >= top_k) reached |= 1u << bit;
      // (keys below that of the lowest finite value come from threads without one)
      const float floor = reached < 0x00800000u ? -INFINITY : raw_floor(RLT_DIV(key_value(reached), temperature), temperature);
      if (threadIdx.x == 0) h.listed = 0;
      __syncthreads();
      for_row<T, kThreads>(row, vocab, [&](float x, int v) {
        if (x >= floor) list_token(h, rlt_order_key(RLT_DIV(x, temperature)), v, 1ull);
      });
      __syncthreads();
      listed = h.listed;
    }
    if (listed <= kCandidates) {
      n.cut = list_select<kThreads>(h, listed, 0ull, static_cast<unsigned long long>(top_k - 1), whole_row());
      const auto sum_kept = [&]() {
        unsigned long long zfix = 0ull;
        for (int j = threadIdx.x; j < listed; j += kThreads)
          if (rlt_in_support(h.key[j], h.index[j], n.cut.key, n.cut.limit)) zfix += rlt_fix_weight(rlt_expf(RLT_SUB(key_value(h.key[j]), n.m)));
        return rlt_fix_to_float(block_sum<kThreads>(zfix, scratch));
      };
      n.z = sum_kept();
      if (use_p) {
        const Cut outer = n.cut;
        const float inv = RLT_DIV(1.0f, n.z);
        unsigned long long mass = 0ull;
        for (int j = threadIdx.x; j < listed; j += kThreads) {
          unsigned long long w = 0ull;
          if (rlt_in_support(h.key[j], h.index[j], outer.key, outer.limit)) w = rlt_fix_weight(rlt_draw_mass(rlt_expf(RLT_SUB(key_value(h.key[j]), n.m)), inv));
          else h.key[j] = 0u;
          h.weight[j] = w;
          mass += w;
        }
        if (block_sum<kThreads>(mass, scratch) > limit_p) {
          n.cut = list_select<kThreads>(h, listed, 0ull, limit_p, outer);
          n.z = sum_kept();
        }
      }
      return n;
    }
    n.cut = bucket_select<T, kThreads, false>(row, vocab, temperature, n.m, 0.0f, own, whole_row(),
                                              static_cast<unsigned long long>(top_k - 1), scratch, h);
    n.z = block_cut_sum<T, kThreads>(row, vocab, temperature, n.m, n.cut, scratch);
  } else {
    n.z = block_full_sum<T, kThreads>(row, vocab, temperature, n.m, scratch);
  }
  if (use_p) {
    const Cut outer = n.cut;
    n.cut = bucket_select<T, kThreads, true>(row, vocab, temperature, n.m, RLT_DIV(1.0f, n.z), own, outer, limit_p, scratch, h);
    if (n.cut.key != outer.key || n.cut.limit != outer.limit)
      n.z = block_cut_sum<T, kThreads>(row, vocab, temperature, n.m, n.cut, scratch);
  }
  return n;
}

// The same without filters, for kernels that keep their registers free of them.
template <typename T, int kThreads>
__device__ __forceinline__ RowNorm block_normalise_plain(const T* __restrict__ row, int vocab, float temperature, unsigned long long* scratch) {
  float own;
  RowNorm n = block_row_max<T, kThreads>(row, vocab, temperature, scratch, &own);
  if (n.ok) n.z = block_full_sum<T, kThreads>(row, vocab, temperature, n.m, scratch);
  return n;
}

// exp(t_v - max) for a token of the support, 0 outside it.
template <typename T>
__device__ __forceinline__ float exp_at(const T* row, int v, float temperature, const RowNorm& n) {
  const float t = scaled_logit(row, v, temperature);
  if (!rlt_in_support(rlt_order_key(t), v, n.cut.key, n.cut.limit)) return 0.0f;
  return rlt_expf(RLT_SUB(t, n.m));
}

template <typename T>
__device__ __forceinline__ float prob_at(const T* row, int v, float temperature, const RowNorm& n) {
  return RLT_DIV(exp_at(row, v, temperature, n), n.z);
}

// Inverse-CDF draw over fixed-point weights in ascending token index, p[v] (plain) or max(p[v] - q[v], 0) (residual) in the
// division-free form of rlt_canonical.h; -1 if the mass is zero.  A warp owns a run of tokens and reads it 128 tokens at a time, four
// per lane; the warp in whose run the threshold falls goes over its run once more.  Tokens outside p's support weigh nothing and are
// dismissed by one comparison, q is read where p has mass only.  128 requests that draw from the residual of two rows of 49 152, or from a
// bonus row: 55 us (74 us where a thread, not a warp, has a run of tokens, whose every load is a line of its own).
template <typename T, int kThreads>
__device__ __forceinline__ int block_draw(const T* __restrict__ prow, const RowNorm& pn,
                                          const T* __restrict__ qrow, const RowNorm& qn, bool residual,
                                          int vocab, float temperature, float u, unsigned long long* scratch,
                                          int* token_slot) {
  constexpr int kWarps = kThreads / 32, kLane = 4, kStep = 32 * kLane;
  struct __align__(kLane * sizeof(T)) Four { T e[kLane]; };
  const float inv = residual ? RLT_DIV(1.0f, RLT_MUL(pn.z, qn.z)) : RLT_DIV(1.0f, pn.z);
  const float floor = cut_floor(pn.cut, temperature);
  const int pad = static_cast<int>((reinterpret_cast<uintptr_t>(prow) & (sizeof(Four) - 1)) / sizeof(T));   // runs start on whole fours
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int run = (vocab + pad + kWarps * kStep - 1) / (kWarps * kStep) * kStep;
  const int begin = min(warp * run, vocab + pad) - pad, end = min(begin + run, vocab);
  const auto weigh = [&](int v, unsigned long long (&w)[kLane]) {      // tokens v .. v + 3
    float x[kLane];
    if (v >= 0 && v + kLane <= end) {
      const Four raw = *reinterpret_cast<const Four*>(prow + v);
#pragma unroll
      for (int j = 0; j < kLane; ++j) x[j] = Elem<T>::to_float(raw.e[j]);
    } else {
#pragma unroll
      for (int j = 0; j < kLane; ++j) x[j] = v + j >= 0 && v + j < end ? Elem<T>::to_float(prow[v + j]) : -INFINITY;
    }
    unsigned long long sum = 0ull;
#pragma unroll
    for (int j = 0; j < kLane; ++j) {
      w[j] = 0ull;
      if (v + j >= 0 && v + j < end && x[j] >= floor) {
        const float t = RLT_DIV(x[j], temperature);
        if (rlt_in_support(rlt_order_key(t), v + j, pn.cut.key, pn.cut.limit)) {
          const float e = rlt_expf(RLT_SUB(t, pn.m));
          w[j] = rlt_fix_weight(residual ? rlt_residual_mass(e, exp_at(qrow, v + j, temperature, qn), pn.z, qn.z, inv) : rlt_draw_mass(e, inv));
        }
      }
      sum += w[j];
    }
    return sum;
  };
  unsigned long long w[kLane] = {0ull, 0ull, 0ull, 0ull}, own = 0ull;
#pragma unroll 2
  for (int v = begin + lane * kLane; v < end; v += kStep) own += weigh(v, w);
  const unsigned long long local = warp_sum(own);
  __syncthreads();
  if (lane == 0) scratch[warp] = local;
  if (threadIdx.x == 0) *token_slot = -1;
  __syncthreads();
  unsigned long long before = 0ull, total = 0ull;
  for (int i = 0; i < kWarps; ++i) {
    const unsigned long long s = scratch[i];
    if (i < warp) before += s;
    total += s;
  }
  if (total != 0ull) {
    const unsigned long long threshold = rlt_draw_threshold(u, total);
    if (before <= threshold && threshold < before + local) {           // one warp
      for (int at = begin; at < end; at += kStep) {
        const unsigned long long sum = run == kStep ? own : weigh(at + lane * kLane, w);   // (a run of one step is still at hand)
        unsigned long long upto = sum;
#pragma unroll
        for (int x = 1; x < 32; x <<= 1) {
          const unsigned long long o = __shfl_up_sync(0xffffffffu, upto, x);
          if (lane >= x) upto += o;
        }
        unsigned long long prefix = before + upto - sum;
        if (prefix <= threshold && threshold < prefix + sum) {
#pragma unroll
          for (int j = 0; j < kLane; ++j) {
            if (prefix <= threshold && threshold < prefix + w[j]) *token_slot = at + lane * kLane + j;
            prefix += w[j];
          }
        }
        before += __shfl_sync(0xffffffffu, upto, 31);
        if (before > threshold) break;
      }
    }
  }
  __syncthreads();
  return *token_slot;
}

template <typename T>
__global__ void __launch_bounds__(kSampleThreads)
sample_rows_kernel(const T* __restrict__ logits, int64_t row_stride, int vocab,
                   const float* __restrict__ temperature, const int32_t* __restrict__ top_k,
                   const float* __restrict__ top_p, const float* __restrict__ uniforms,
                   int64_t* __restrict__ tokens, int32_t* __restrict__ status) {
  __shared__ unsigned long long scratch[32];
  __shared__ SelectScratch select;
  __shared__ int token_slot;
  const int r = blockIdx.x;
  const T* row = logits + static_cast<int64_t>(r) * row_stride;
  const float temp = temperature[r];
  int st = RLT_ROW_OK;
  int token = -1;
  if (temp == 0.0f) {
    token = block_argmax<T, kSampleThreads>(row, vocab, scratch);
  } else {
    const RowNorm n = block_normalise<T, kSampleThreads>(row, vocab, temp, top_k ? top_k[r] : -1,
                                                         top_p ? top_p[r] : 1.0f, scratch, select);
    if (!n.ok) {
      st = RLT_ROW_BAD_LOGITS;
    } else {
      token = block_draw<T, kSampleThreads>(row, n, row, n, false, vocab, temp, uniforms[r], scratch, &token_slot);
      if (token < 0) st = RLT_ROW_INVALID_RESIDUAL;
    }
  }
  if (threadIdx.x == 0) { tokens[r] = token; status[r] = st; }
}

// Sampler.probabilities for every row: fp32 [rows, vocab], zero outside the support.
template <typename T>
__global__ void __launch_bounds__(kSampleThreads)
probabilities_kernel(const T* __restrict__ logits, int64_t row_stride, int vocab,
                     const float* __restrict__ temperature, const int32_t* __restrict__ top_k,
                     const float* __restrict__ top_p, float* __restrict__ probs, int32_t* __restrict__ status) {
  __shared__ unsigned long long scratch[32];
  __shared__ SelectScratch select;
  const int r = blockIdx.x;
  const T* row = logits + static_cast<int64_t>(r) * row_stride;
  float* out = probs + static_cast<int64_t>(r) * vocab;
  const float temp = temperature[r];
  RowNorm n;
  n.ok = 0;
  if (temp > 0.0f)
    n = block_normalise<T, kSampleThreads>(row, vocab, temp, top_k ? top_k[r] : -1, top_p ? top_p[r] : 1.0f,
                                           scratch, select);
  for (int v = threadIdx.x; v < vocab; v += kSampleThreads) out[v] = n.ok ? prob_at(row, v, temp, n) : 0.0f;
  if (threadIdx.x == 0) status[r] = n.ok ? RLT_ROW_OK : RLT_ROW_BAD_LOGITS;
}

// ---- rejection sampling in two launches -------------------------------------------------
// 1. row_stats_kernel, one CTA per (verification row, target | draft): everything about a
//    row that does not depend on earlier accept decisions — max, normaliser and the
//    probability of the row's draft token (or the argmax for a greedy request) — so the
//    streaming over [rows, vocab] runs at full width instead of request by request.
// 2. decide_kernel, one CTA per request: the sequential accept walk over those few numbers,
//    then the single residual or bonus draw the request needs.
struct RowStats {
  float m;
  float z;
  float prob;  // probability of the row's draft token under this row's distribution
  int info;    // bit 0: distribution valid; greedy requests: argmax index << 1
  Cut cut;     // support after top-k / top-p
};

constexpr int kStatsThreads = 512;

__device__ __forceinline__ int request_of_row(const int32_t* cu_rows, int n, int row) {
  int lo = 0, hi = n - 1;  // last i with cu_rows[i] <= row
  while (lo < hi) {
    const int mid = (lo + hi + 1) >> 1;
    if (cu_rows[mid] <= row) lo = mid; else hi = mid - 1;
  }
  return lo;
}

template <typename T, int kThreads, bool kFilters>
__global__ void __launch_bounds__(kThreads, 3)
row_stats_kernel(const T* __restrict__ target_logits, const T* __restrict__ draft_logits, int64_t row_stride,
                 int vocab, const int32_t* __restrict__ cu_rows, int n, const int32_t* __restrict__ row_counts,
                 const int64_t* __restrict__ tokens, int tokens_width, const float* __restrict__ temperature,
                 const int32_t* __restrict__ top_k, const float* __restrict__ top_p, RowStats* __restrict__ stats) {
  __shared__ unsigned long long scratch[32];
  const int row = blockIdx.x, side = blockIdx.y;  // side 0: target, 1: draft
  const int i = request_of_row(cu_rows, n, row);
  int first, span;
  const int count = request_rows(cu_rows, row_counts, i, &first, &span);
  const int j = row - first;
  if (j >= count) return;  // a padding row: nothing reads its statistics
  const float temp = temperature[i];
  RowStats out = {0.0f, 0.0f, 0.0f, 0, whole_row()};
  if (temp == 0.0f) {
    if (side == 1) return;
    out.info = block_argmax<T, kThreads>(target_logits + static_cast<int64_t>(row) * row_stride, vocab, scratch) << 1;
  } else {
    if (side == 1 && j == count - 1) return;  // the bonus row has no draft distribution
    const T* logits = (side == 0 ? target_logits : draft_logits) + static_cast<int64_t>(row) * row_stride;
    RowNorm norm;
    if constexpr (kFilters) {
      __shared__ SelectScratch select;
      norm = block_normalise<T, kThreads>(logits, vocab, temp, top_k ? top_k[i] : -1, top_p ? top_p[i] : 1.0f, scratch, select);
    } else {
      norm = block_normalise_plain<T, kThreads>(logits, vocab, temp, scratch);
    }
    const int64_t d = j < count - 1 ? tokens[static_cast<int64_t>(i) * tokens_width + j + 1] : -1;
    out.m = norm.m;
    out.z = norm.z;
    out.info = norm.ok ? 1 : 0;
    out.cut = norm.cut;
    if (norm.ok && d >= 0 && d < vocab) out.prob = prob_at(logits, static_cast<int>(d), temp, norm);
  }
  if (threadIdx.x == 0) stats[2 * row + side] = out;
}

template <typename T>
__global__ void __launch_bounds__(kSampleThreads)
decide_kernel(const T* __restrict__ target_logits, const T* __restrict__ draft_logits, int64_t row_stride, int rows,
              int vocab, const int32_t* __restrict__ cu_rows, int n, const int32_t* __restrict__ row_counts,
              const int64_t* __restrict__ tokens, int tokens_width, const int64_t* __restrict__ starts,
              const float* __restrict__ temperature, const float* __restrict__ u_accept,
              const float* __restrict__ u_final, const int64_t* __restrict__ slots,
              int64_t* __restrict__ slot_values, const RowStats* __restrict__ stats,
              int64_t* __restrict__ result, int32_t* __restrict__ status) {
  __shared__ unsigned long long scratch[32];
  __shared__ int token_slot;
  const int i = blockIdx.x;
  int a, span;
  const int c = request_rows(cu_rows, row_counts, i, &a, &span);
  const int64_t* tok = tokens + static_cast<int64_t>(i) * tokens_width;
  const float temp = temperature[i];
  for (int j = threadIdx.x; j < span; j += kSampleThreads) result[a + j] = -1;
  if (c == 0) {  // no rows: the request is left alone
    if (threadIdx.x == 0) {
      result[rows + i] = 0;
      result[rows + n + i] = starts[i];
      status[i] = RLT_ROW_OK;
    }
    return;
  }
  __syncthreads();

  int accepted = 0, st = RLT_ROW_OK;
  int64_t final_token = -1;
  if (temp == 0.0f) {
    for (int j = 0; j < c; ++j) {
      const int target = stats[2 * (a + j)].info >> 1;
      if (threadIdx.x == 0) result[a + j] = target;
      final_token = target;
      if (j < c - 1 && tok[j + 1] == target) { ++accepted; continue; }
      break;
    }
  } else {
    int j = 0;
    for (; j < c - 1; ++j) {
      const RowStats ps = stats[2 * (a + j)], qs = stats[2 * (a + j) + 1];
      const int64_t d = tok[j + 1];
      if (!(ps.info & 1) || !(qs.info & 1) || d < 0 || d >= vocab) { st = RLT_ROW_BAD_LOGITS; break; }
      if (!(qs.prob > 0.0f)) { st = RLT_ROW_ZERO_PROPOSAL; break; }
      if (RLT_MUL(u_accept[a + j], qs.prob) < ps.prob) {
        if (threadIdx.x == 0) result[a + j] = d;
        ++accepted;
        continue;
      }
      const RowNorm pn = {ps.m, ps.z, 1, ps.cut}, qn = {qs.m, qs.z, 1, qs.cut};
      final_token = block_draw<T, kSampleThreads>(target_logits + static_cast<int64_t>(a + j) * row_stride, pn,
                                                  draft_logits + static_cast<int64_t>(a + j) * row_stride, qn, true,
                                                  vocab, temp, u_final[i], scratch, &token_slot);
      if (final_token < 0) st = RLT_ROW_INVALID_RESIDUAL;
      break;
    }
    if (st == RLT_ROW_OK && j == c - 1) {
      const RowStats ps = stats[2 * (a + c - 1)];
      if (!(ps.info & 1)) {
        st = RLT_ROW_BAD_LOGITS;
      } else {
        const RowNorm pn = {ps.m, ps.z, 1, ps.cut};
        const T* prow = target_logits + static_cast<int64_t>(a + c - 1) * row_stride;
        final_token = block_draw<T, kSampleThreads>(prow, pn, prow, pn, false, vocab, temp, u_final[i], scratch,
                                                    &token_slot);
        if (final_token < 0) st = RLT_ROW_INVALID_RESIDUAL;
      }
    }
  }
  if (threadIdx.x == 0) {
    if (temp != 0.0f && st == RLT_ROW_OK) result[a + accepted] = final_token;
    const int64_t next_pos = starts[i] + accepted + 1;
    result[rows + i] = accepted;
    result[rows + n + i] = next_pos;
    status[i] = st;
    // A failed request keeps its slot: the next round must not start from token -1.
    if (st == RLT_ROW_OK && slots != nullptr && slot_values != nullptr) {
      slot_values[2 * slots[i]] = final_token;
      slot_values[2 * slots[i] + 1] = next_pos;
    }
  }
}

int check_logits(const void* logits, int64_t row_stride, int rows, int vocab, int dtype) {
  RLT_REQUIRE(dtype_valid(dtype), "acceptance: logits must be float32, float16 or bfloat16");
  RLT_REQUIRE(rows >= 0 && vocab > 0 && row_stride >= vocab, "acceptance: invalid logits shape");
  RLT_REQUIRE(rows == 0 || logits != nullptr, "acceptance: null logits");
  return RLT_OK;
}

}  // namespace
}  // namespace rlt

extern "C" RLT_API int rlt_argmax_rows(const void* logits, int64_t row_stride, int rows, int vocab, int dtype,
                               int64_t* targets, rlt_stream_t stream) {
  using namespace rlt;
  int status = check_logits(logits, row_stride, rows, vocab, dtype);
  if (status != RLT_OK || rows == 0) return status;
  RLT_REQUIRE(targets != nullptr, "argmax_rows: null output");
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  RLT_DISPATCH_DTYPE(dtype, T, (argmax_rows_kernel<T><<<rows, kArgmaxThreads, 0, s>>>(
                                   static_cast<const T*>(logits), row_stride, vocab, targets)));
  return launch_status("argmax_rows_kernel");
}

extern "C" RLT_API int rlt_accept_greedy(const void* logits, int64_t row_stride, int rows, int vocab, int dtype,
                                 const int32_t* cu_rows, int n, const int32_t* row_counts, const int64_t* tokens,
                                 int tokens_width, const int64_t* starts, const int64_t* slots,
                                 int64_t* slot_values, int64_t* result, rlt_stream_t stream) {
  using namespace rlt;
  int status = check_logits(logits, row_stride, rows, vocab, dtype);
  if (status != RLT_OK) return status;
  RLT_REQUIRE(n >= 0 && tokens_width >= 1, "accept_greedy: invalid request count or token width");
  if (n == 0 && rows == 0) return RLT_OK;
  RLT_REQUIRE(cu_rows && tokens && starts && result, "accept_greedy: null pointer");
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  if (rows > 0) {
    RLT_DISPATCH_DTYPE(dtype, T, (argmax_rows_kernel<T><<<rows, kArgmaxThreads, 0, s>>>(
                                     static_cast<const T*>(logits), row_stride, vocab, result)));
    status = launch_status("argmax_rows_kernel");
    if (status != RLT_OK) return status;
  }
  if (n > 0) {
    greedy_finish_kernel<<<(n + 127) / 128, 128, 0, s>>>(cu_rows, n, rows, row_counts, tokens, tokens_width, starts,
                                                         slots, slot_values, result);
    status = launch_status("greedy_finish_kernel");
  }
  return status;
}

extern "C" RLT_API int rlt_sample_rows(const void* logits, int64_t row_stride, int rows, int vocab, int dtype,
                               const float* temperature, const int32_t* top_k, const float* top_p,
                               const float* uniforms, int64_t* tokens, int32_t* status_out, rlt_stream_t stream) {
  using namespace rlt;
  int status = check_logits(logits, row_stride, rows, vocab, dtype);
  if (status != RLT_OK || rows == 0) return status;
  RLT_REQUIRE(temperature && uniforms && tokens && status_out, "sample_rows: null pointer");
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  RLT_DISPATCH_DTYPE(dtype, T, (sample_rows_kernel<T><<<rows, kSampleThreads, 0, s>>>(
                                   static_cast<const T*>(logits), row_stride, vocab, temperature, top_k, top_p,
                                   uniforms, tokens, status_out)));
  return launch_status("sample_rows_kernel");
}

extern "C" RLT_API int rlt_probabilities(const void* logits, int64_t row_stride, int rows, int vocab, int dtype,
                                         const float* temperature, const int32_t* top_k, const float* top_p,
                                         float* probs, int32_t* status_out, rlt_stream_t stream) {
  using namespace rlt;
  int status = check_logits(logits, row_stride, rows, vocab, dtype);
  if (status != RLT_OK || rows == 0) return status;
  RLT_REQUIRE(temperature && probs && status_out, "probabilities: null pointer");
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  RLT_DISPATCH_DTYPE(dtype, T, (probabilities_kernel<T><<<rows, kSampleThreads, 0, s>>>(
                                   static_cast<const T*>(logits), row_stride, vocab, temperature, top_k, top_p,
                                   probs, status_out)));
  return launch_status("probabilities_kernel");
}

namespace rlt {
namespace {
__global__ void round_uniforms_kernel(const int64_t* __restrict__ seeds, const int64_t* __restrict__ rounds, int n,
                                      int width, float* __restrict__ u_draft, float* __restrict__ u_accept,
                                      float* __restrict__ u_final) {
  const int x = blockIdx.x * blockDim.x + threadIdx.x;
  if (x >= n * (2 * width + 1)) return;
  const int i = x / (2 * width + 1), j = x % (2 * width + 1);
  const uint64_t seed = static_cast<uint64_t>(seeds[i]), round = static_cast<uint64_t>(rounds[i]);
  if (j < width) u_draft[i * width + j] = rlt_uniform(seed, round, RLT_STREAM_DRAFT, j);
  else if (j < 2 * width) u_accept[i * width + j - width] = rlt_uniform(seed, round, RLT_STREAM_ACCEPT, j - width);
  else u_final[i] = rlt_uniform(seed, round, RLT_STREAM_FINAL, 0);
}
}  // namespace
}  // namespace rlt

extern "C" RLT_API int rlt_round_uniforms(const int64_t* seeds, const int64_t* rounds, int n, int width,
                                          float* u_draft, float* u_accept, float* u_final, rlt_stream_t stream) {
  using namespace rlt;
  RLT_REQUIRE(n >= 0 && width >= 1 && width <= 4096, "round_uniforms: invalid request count or width");
  if (n == 0) return RLT_OK;
  RLT_REQUIRE(seeds && rounds && u_draft && u_accept && u_final, "round_uniforms: null pointer");
  const int total = n * (2 * width + 1);
  round_uniforms_kernel<<<(total + 255) / 256, 256, 0, static_cast<cudaStream_t>(stream)>>>(
      seeds, rounds, n, width, u_draft, u_accept, u_final);
  return launch_status("round_uniforms_kernel");
}

extern "C" RLT_API size_t rlt_accept_rejection_workspace_bytes(int rows) {
  return rows > 0 ? static_cast<size_t>(rows) * 2 * sizeof(rlt::RowStats) : 32;
}

extern "C" RLT_API int rlt_accept_rejection(const void* target_logits, const void* draft_logits, int64_t row_stride,
                                            int rows, int vocab, int dtype, const int32_t* cu_rows, int n,
                                            const int32_t* row_counts, const int64_t* tokens, int tokens_width,
                                            const int64_t* starts,
                                            const float* temperature, const int32_t* top_k, const float* top_p,
                                            const float* u_accept, const float* u_final, const int64_t* slots,
                                            int64_t* slot_values, int64_t* result, int32_t* status_out,
                                            void* workspace, size_t workspace_bytes,
                                            rlt_stream_t stream) {
  using namespace rlt;
  int status = check_logits(target_logits, row_stride, rows, vocab, dtype);
  if (status != RLT_OK) return status;
  RLT_REQUIRE(n >= 0 && tokens_width >= 1, "accept_rejection: invalid request count or token width");
  if (n == 0) return RLT_OK;
  RLT_REQUIRE(draft_logits && cu_rows && tokens && starts && temperature && u_accept && u_final && result &&
                  status_out,
              "accept_rejection: null pointer");
  if (workspace == nullptr || workspace_bytes < rlt_accept_rejection_workspace_bytes(rows) ||
      (reinterpret_cast<uintptr_t>(workspace) & 15u) != 0) {
    set_last_error_text("accept_rejection: workspace missing, misaligned or too small");
    return RLT_ERR_WORKSPACE;
  }
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  RowStats* stats = static_cast<RowStats*>(workspace);
  const bool filters = top_k != nullptr || top_p != nullptr;
  RLT_DISPATCH_DTYPE(dtype, T, {
    auto kernel = filters ? row_stats_kernel<T, kStatsThreads, true> : row_stats_kernel<T, kStatsThreads, false>;
    kernel<<<dim3(rows, 2), kStatsThreads, 0, s>>>(static_cast<const T*>(target_logits), static_cast<const T*>(draft_logits), row_stride, vocab,
                                                   cu_rows, n, row_counts, tokens, tokens_width, temperature, top_k, top_p, stats);
  });
  status = launch_status("row_stats_kernel");
  if (status != RLT_OK) return status;
  RLT_DISPATCH_DTYPE(dtype, T, (decide_kernel<T><<<n, kSampleThreads, 0, s>>>(
                                   static_cast<const T*>(target_logits), static_cast<const T*>(draft_logits),
                                   row_stride, rows, vocab, cu_rows, n, row_counts, tokens, tokens_width, starts,
                                   temperature, u_accept, u_final, slots, slot_values, stats, result, status_out)));
  return launch_status("decide_kernel");
}
