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
// thread, where the row allows them.  A row is a few hundred KB: the first pass over it reads HBM, the others L2.
template <typename T, int kThreads, int kDepth = 4, typename F>
__device__ __forceinline__ void for_row(const T* __restrict__ row, int vocab, F f) {
  constexpr int kVec = 16 / sizeof(T);
  int done = 0;
  if ((reinterpret_cast<uintptr_t>(row) & 15u) == 0) {
    const uint4* rv = reinterpret_cast<const uint4*>(row);
    const int nvec = vocab / kVec;
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
          for (int j = 0; j < kVec; ++j) f(Elem<T>::to_float(e[j]), i * kVec + j);
        }
      }
    }
    done = nvec * kVec;
  }
  for (int v = done + static_cast<int>(threadIdx.x); v < vocab; v += kThreads) f(Elem<T>::to_float(row[v]), v);
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
//   buckets      every other filter: a histogram of weight over m - t in steps of 1/64 finds the step in which the running weight
//                first exceeds the limit; its tokens are the candidates.
//   digits       rows whose candidates do not fit (mass ties): a radix select over four 8-bit digits of the order key.
// 128 requests of 5 rows of 49 152 fp32 logits, half of them with top-k 50 and top-p 0.95: the digits alone, over a row copied
// to shared memory by one CTA per SM, took 595 us; this takes 141 us.
constexpr int kCandidates = 2048;
constexpr int kBuckets = 2048;

struct SelectScratch {
  union {
    struct {                                // candidates, and the digits' histogram
      unsigned long long weight[kCandidates];
      uint32_t key[kCandidates];
      int index[kCandidates];
    };
    unsigned long long bucket[kBuckets];
    struct {
      unsigned long long mass[256];
      unsigned int count[256];
    };
  };
  unsigned long long above;
  int digit;
  int found;
  int listed;
  int warp_counts[32];
};

__device__ __forceinline__ int bucket_of(float t, float m) {
  const float d = RLT_SUB(m, t);
  return d < 31.0f ? max(static_cast<int>(d * 64.0f), 0) : kBuckets - 1;
}

// Adds a token to the candidates; those that do not fit are only counted.
__device__ __forceinline__ void list_token(SelectScratch& h, uint32_t key, int index) {
  const int at = atomicAdd(&h.listed, 1);
  if (at < kCandidates) { h.key[at] = key; h.index[at] = index; }
}

// The cut among n listed candidates with their weights, `above` being the weight of the tokens ranked before all of them.
// A candidate whose weight no longer counts has weight 0 and key 0.  The running weight must exceed the limit inside the list.
template <int kThreads>
__device__ __forceinline__ Cut list_select(SelectScratch& h, int n, unsigned long long above, unsigned long long limit, Cut outer,
                                           unsigned long long* scratch) {
  auto weight_where = [&](auto&& counts) {
    unsigned long long sum = 0ull;
    for (int j = threadIdx.x; j < n; j += kThreads)
      if (counts(j)) sum += h.weight[j];
    return block_sum<kThreads>(sum, scratch);
  };
  uint32_t key = 0u;                        // the largest key for which the weight of all tokens from it on exceeds the limit
  for (int bit = 31; bit >= 0; --bit) {
    const uint32_t next = key | (1u << bit);
    if (above + weight_where([&](int j) { return h.key[j] >= next; }) > limit) key = next;
  }
  const unsigned long long before = above + weight_where([&](int j) { return h.key[j] > key; });
  int ties = 0;
  unsigned long long each = 0ull;
  for (int j = threadIdx.x; j < n; j += kThreads)
    if (h.key[j] == key) { ++ties; each = h.weight[j]; }
  ties = static_cast<int>(block_sum<kThreads>(static_cast<unsigned long long>(ties), scratch));
  each = block_max<kThreads>(each, scratch);
  const unsigned long long keep = (limit - before) / each + 1ull;
  if (keep >= static_cast<unsigned long long>(ties)) return Cut{key, key == outer.key ? outer.limit : 0x7fffffff};
  int index = 0;                            // the largest index with fewer than `keep` of the tied tokens before it
  for (int bit = 30; bit >= 0; --bit) {
    const int next = index | (1 << bit);
    unsigned long long count = 0ull;
    for (int j = threadIdx.x; j < n; j += kThreads) count += h.key[j] == key && h.index[j] < next;
    if (block_sum<kThreads>(count, scratch) < keep) index = next;
  }
  return Cut{key, index};
}

// One shared-memory atomic per distinct digit in the warp: lanes with the same digit find each
// other with match.any and add their weights with two integer warp reductions (a weight is below
// 2^41: 20 low and 21 high bits, so 32 of them cannot overflow a 32-bit partial sum).  The leading
// byte of the key has only a few populated values, so plain per-lane atomics would serialise.
template <bool kByMass>
__device__ __forceinline__ void hist_add(SelectScratch& h, int bucket, unsigned long long w, bool valid) {
  const int lane = threadIdx.x & 31;
  const unsigned peers = __match_any_sync(0xffffffffu, valid ? bucket : 0x7fff);
  const bool leader = valid && lane == __ffs(peers) - 1;
  if (kByMass) {
    const unsigned low = __reduce_add_sync(peers, static_cast<unsigned>(w & 0xfffffu));
    const unsigned high = __reduce_add_sync(peers, static_cast<unsigned>(w >> 20));
    if (leader) atomicAdd(&h.mass[bucket], (static_cast<unsigned long long>(high) << 20) + low);
  }
  if (leader) atomicAdd(&h.count[bucket], static_cast<unsigned int>(__popc(peers)));
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

template <typename T, int kThreads, bool kByMass>
__device__ __forceinline__ Cut block_select(const T* __restrict__ row, int vocab, float temperature, float m,
                                            float inv, Cut outer, unsigned long long limit, SelectScratch& h) {
  uint32_t prefix = 0u;
  unsigned long long above = 0ull;
  for (int pass = 0; pass < 4; ++pass) {
    const int shift = 24 - 8 * pass;
    __syncthreads();
    for (int i = threadIdx.x; i < 256; i += kThreads) { h.mass[i] = 0ull; h.count[i] = 0u; }
    __syncthreads();
    for (int base = 0; base < vocab; base += kThreads) {
      const int v = base + static_cast<int>(threadIdx.x);
      bool valid = false;
      int bucket = 0;
      unsigned long long w = 0ull;
      if (v < vocab) {
        const float t = scaled_logit(row, v, temperature);
        const uint32_t key = rlt_order_key(t);
        valid = rlt_in_support(key, v, outer.key, outer.limit) &&
                (pass == 0 || (key >> (shift + 8)) == (prefix >> (shift + 8)));
        bucket = static_cast<int>((key >> shift) & 255u);
        if (kByMass && valid) w = rlt_fix_weight(rlt_draw_mass(rlt_expf(RLT_SUB(t, m)), inv));
      }
      hist_add<kByMass>(h, bucket, w, valid);
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
    if (h.digit < 0) return outer;  // the whole of `outer` stays (its weight never exceeds the limit)
    prefix |= static_cast<uint32_t>(h.digit) << shift;
    above = h.above;
  }
  const unsigned int ties = h.count[prefix & 255u];
  const unsigned long long each = kByMass ? h.mass[prefix & 255u] / ties : 1ull;
  const unsigned long long keep = (limit - above) / each + 1ull;
  __syncthreads();
  if (keep >= ties) return Cut{prefix, prefix == outer.key ? outer.limit : 0x7fffffff};
  return Cut{prefix, block_nth_index<T, kThreads>(row, vocab, temperature, prefix, outer,
                                                  static_cast<unsigned int>(keep), h)};
}

// The cut by buckets (digits where the bucket's tokens do not fit the list); `inv` is 1 / z.
template <typename T, int kThreads, bool kByMass>
__device__ __forceinline__ Cut bucket_select(const T* __restrict__ row, int vocab, float temperature, float m, float inv, Cut outer,
                                             unsigned long long limit, unsigned long long* scratch, SelectScratch& h) {
  constexpr int kOwn = kBuckets / kThreads;
  const float floor = cut_floor(outer, temperature);
  const auto weight = [&](float t) { return kByMass ? rlt_fix_weight(rlt_draw_mass(rlt_expf(RLT_SUB(t, m)), inv)) : 1ull; };
  __syncthreads();
  for (int i = threadIdx.x; i < kBuckets; i += kThreads) h.bucket[i] = 0ull;
  if (threadIdx.x == 0) { h.digit = -1; h.listed = 0; }
  __syncthreads();
  for_row<T, kThreads, 2>(row, vocab, [&](float x, int v) {
    if (x >= floor) {
      const float t = RLT_DIV(x, temperature);
      if (rlt_in_support(rlt_order_key(t), v, outer.key, outer.limit)) {
        const unsigned long long w = weight(t);
        if (w != 0ull) atomicAdd(&h.bucket[bucket_of(t, m)], w);
      }
    }
  });
  __syncthreads();
  // thread i scans buckets kOwn * i ..
  unsigned long long own[kOwn], local = 0ull;
#pragma unroll
  for (int j = 0; j < kOwn; ++j) { own[j] = h.bucket[kOwn * threadIdx.x + j]; local += own[j]; }
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  unsigned long long before = local;
#pragma unroll
  for (int x = 1; x < 32; x <<= 1) {
    const unsigned long long o = __shfl_up_sync(0xffffffffu, before, x);
    if (lane >= x) before += o;
  }
  if (lane == 31) scratch[warp] = before;
  __syncthreads();
  before -= local;
  for (int w = 0; w < warp; ++w) before += scratch[w];
  if (before <= limit && before + local > limit) {      // one thread at most
#pragma unroll
    for (int j = 0; j < kOwn; ++j) {
      if (h.digit < 0) {
        if (before + own[j] > limit) { h.digit = kOwn * threadIdx.x + j; h.above = before; }
        before += own[j];
      }
    }
  }
  __syncthreads();
  const int crossing = h.digit;
  const unsigned long long above = h.above;
  if (crossing < 0) return outer;           // everything stays
  for_row<T, kThreads>(row, vocab, [&](float x, int v) {
    if (x >= floor) {
      const float t = RLT_DIV(x, temperature);
      const uint32_t key = rlt_order_key(t);
      if (bucket_of(t, m) == crossing && rlt_in_support(key, v, outer.key, outer.limit)) list_token(h, key, v);
    }
  });
  __syncthreads();
  const int n = h.listed;
  if (n > kCandidates) return block_select<T, kThreads, kByMass>(row, vocab, temperature, m, inv, outer, limit, h);
  for (int j = threadIdx.x; j < n; j += kThreads) h.weight[j] = weight(key_value(h.key[j]));
  return list_select<kThreads>(h, n, above, limit, outer, scratch);
}

// max, support and normaliser of the distribution Sampler.probabilities builds for one row
// (vllm_rlt/worker/sampler.py:37-55): softmax(row / T) restricted to top-k, then to top-p.
// top_k <= 0 or >= vocab and top_p >= 1 switch the filters off.
// Division by a positive temperature is monotonic, so max_v (x_v / T) == (max_v x_v) / T exactly: the first pass is a plain
// maximum over the raw logits, one division at the end.
template <typename T, int kThreads>
__device__ __forceinline__ RowNorm block_normalise(const T* __restrict__ row, int vocab, float temperature,
                                                   int top_k, float top_p, unsigned long long* scratch,
                                                   SelectScratch& h) {
  const bool use_k = top_k > 0 && top_k < vocab, use_p = top_p < 1.0f;
  float own = -INFINITY;
  bool nan = false;
  for_row<T, kThreads>(row, vocab, [&](float x, int) {
    own = fmaxf(own, x);
    nan |= x != x;
  });
  const uint32_t own_key = rlt_order_key(own);
  const uint32_t top = __reduce_max_sync(0xffffffffu, nan ? 0xffffffffu : own_key);
  RowNorm n;
  const uint32_t best = static_cast<uint32_t>(block_max<kThreads>(top, scratch));
  n.m = best == 0xffffffffu ? NAN : RLT_DIV(key_value(best), temperature);
  n.ok = n.m == n.m && n.m != INFINITY && n.m != -INFINITY;
  n.z = 0.0f;
  n.cut = whole_row();
  if (!n.ok) return n;
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
        if (x >= floor) list_token(h, rlt_order_key(RLT_DIV(x, temperature)), v);
      });
      __syncthreads();
      listed = h.listed;
    }
    if (listed <= kCandidates) {
      for (int j = threadIdx.x; j < listed; j += kThreads) h.weight[j] = 1ull;
      n.cut = list_select<kThreads>(h, listed, 0ull, static_cast<unsigned long long>(top_k - 1), whole_row(), scratch);
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
          n.cut = list_select<kThreads>(h, listed, 0ull, limit_p, outer, scratch);
          n.z = sum_kept();
        }
      }
      return n;
    }
    n.cut = bucket_select<T, kThreads, false>(row, vocab, temperature, n.m, 0.0f, whole_row(),
                                              static_cast<unsigned long long>(top_k - 1), scratch, h);
    n.z = block_cut_sum<T, kThreads>(row, vocab, temperature, n.m, n.cut, scratch);
  } else {
    n.z = block_full_sum<T, kThreads>(row, vocab, temperature, n.m, scratch);
  }
  if (use_p) {
    const Cut outer = n.cut;
    n.cut = bucket_select<T, kThreads, true>(row, vocab, temperature, n.m, RLT_DIV(1.0f, n.z), outer, limit_p, scratch, h);
    if (n.cut.key != outer.key || n.cut.limit != outer.limit)
      n.z = block_cut_sum<T, kThreads>(row, vocab, temperature, n.m, n.cut, scratch);
  }
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
// dismissed by one comparison, q is read where p has mass only.  (A run of tokens per THREAD, the earlier split, read a line per
// lane: a residual draw from two rows of 49 152 took 74 us, this 56.)
template <typename T, int kThreads>
__device__ __forceinline__ int block_draw(const T* __restrict__ prow, const RowNorm& pn,
                                          const T* __restrict__ qrow, const RowNorm& qn, bool residual,
                                          int vocab, float temperature, float u, unsigned long long* scratch,
                                          int* token_slot) {
  constexpr int kWarps = kThreads / 32, kLane = 4, kStep = 32 * kLane;
  struct __align__(kLane * sizeof(T)) Four { T e[kLane]; };
  const float inv = residual ? RLT_DIV(1.0f, RLT_MUL(pn.z, qn.z)) : RLT_DIV(1.0f, pn.z);
  const float floor = cut_floor(pn.cut, temperature);
  const bool vectors = (reinterpret_cast<uintptr_t>(prow) & (sizeof(Four) - 1)) == 0;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int run = (vocab + kWarps * kStep - 1) / (kWarps * kStep) * kStep;
  const int begin = min(warp * run, vocab), end = min(begin + run, vocab);
  const auto weigh = [&](int v, unsigned long long (&w)[kLane]) {      // tokens v .. v + 3
    float x[kLane];
    if (vectors && v + kLane <= end) {
      const Four raw = *reinterpret_cast<const Four*>(prow + v);
#pragma unroll
      for (int j = 0; j < kLane; ++j) x[j] = Elem<T>::to_float(raw.e[j]);
    } else {
#pragma unroll
      for (int j = 0; j < kLane; ++j) x[j] = v + j < end ? Elem<T>::to_float(prow[v + j]) : -INFINITY;
    }
    unsigned long long sum = 0ull;
#pragma unroll
    for (int j = 0; j < kLane; ++j) {
      w[j] = 0ull;
      if (v + j < end && x[j] >= floor) {
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
  unsigned long long w[kLane], local = 0ull;
#pragma unroll 2
  for (int v = begin + lane * kLane; v < end; v += kStep) local += weigh(v, w);
  local = warp_sum(local);
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
        const unsigned long long sum = weigh(at + lane * kLane, w);
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

template <typename T, int kThreads>
__global__ void __launch_bounds__(kThreads, 3)
row_stats_kernel(const T* __restrict__ target_logits, const T* __restrict__ draft_logits, int64_t row_stride,
                 int vocab, const int32_t* __restrict__ cu_rows, int n, const int32_t* __restrict__ row_counts,
                 const int64_t* __restrict__ tokens, int tokens_width, const float* __restrict__ temperature,
                 const int32_t* __restrict__ top_k, const float* __restrict__ top_p, RowStats* __restrict__ stats) {
  __shared__ unsigned long long scratch[32];
  __shared__ SelectScratch select;
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
    const RowNorm norm = block_normalise<T, kThreads>(logits, vocab, temp, top_k ? top_k[i] : -1, top_p ? top_p[i] : 1.0f, scratch,
                                                      select);
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
  RLT_DISPATCH_DTYPE(dtype, T, (row_stats_kernel<T, kStatsThreads><<<dim3(rows, 2), kStatsThreads, 0, s>>>(
                                   static_cast<const T*>(target_logits), static_cast<const T*>(draft_logits),
                                   row_stride, vocab, cu_rows, n, row_counts, tokens, tokens_width, temperature,
                                   top_k, top_p, stats)));
  status = launch_status("row_stats_kernel");
  if (status != RLT_OK) return status;
  RLT_DISPATCH_DTYPE(dtype, T, (decide_kernel<T><<<n, kSampleThreads, 0, s>>>(
                                   static_cast<const T*>(target_logits), static_cast<const T*>(draft_logits),
                                   row_stride, rows, vocab, cu_rows, n, row_counts, tokens, tokens_width, starts,
                                   temperature, u_accept, u_final, slots, slot_values, stats, result, status_out)));
  return launch_status("decide_kernel");
}
