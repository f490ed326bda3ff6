// Grouped expert product on the 5th-generation tensor cores: y = act(x W_e^T) over rows sorted by expert, bf16.
//
// The weights are the M operand and the tokens the N operand (D^T = W_e x^T): a tile is 128 outputs of one expert per CTA times up to
// kTokens of its rows, so a decoding step, whose experts have a handful of rows each, streams every weight once and pays for
// no more tensor work than its rows need.
//
// Prompts run on pairs of CTAs (cta_group::2): 256 outputs x 256 rows per pair, each CTA holding its own outputs of the weights, half of
// the rows, and its own outputs of the accumulator.  A CTA on its own took 48 KB per stage of 512 cycles out of L2, more than the 64 bytes
// per cycle an SM gets; half of a pair takes 32 KB.  Four warps then still left the accumulators late: with sixteen, 131072 rows of 64
// experts take 582 us for 2048 -> 2 x 704 gated and 330 us for 704 -> 2048 (789 and 547 us with single CTAs and four warps).
//
// One persistent CTA per SM:
//   warp 0      TMA: 64 columns of the weight tile and of the token tile per stage, several stages ahead
//   warp 1      tcgen05.mma into one of two accumulators in tensor memory (N = the tile's rows, rounded up to 16; to 32 in a pair, whose
//               first CTA issues for both)
//   warps 2..   the other accumulator: activation, and the transpose on the way out — lane = output, column = token, so
//               neighbouring lanes trade halves of two columns and store pairs of outputs, 64 bytes per token and warp; where a pair
//               of outputs is a gate and what it multiplies, a lane stores their one result of its token
// Tiles are dealt round-robin in the order expert, rows, outputs: CTAs that run together share token tiles and weights in L2.
#include "experts.cuh"
#include "sm100_primitives.cuh"

namespace rlt {
namespace {

constexpr int kOutputs = 128;      // outputs per tile: TMEM lanes
constexpr int kDepth = 64;         // input columns per stage: one 128-byte swizzled row
constexpr int kMaxExperts = 1024;
constexpr int kABytes = kOutputs * kDepth * 2;

template <int kTokens, int kCtas>
struct ExpertShared {
  static constexpr int kColumnWarps = kTokens <= 32 ? 1 : kTokens <= 128 ? 2 : 4;   // per quarter of the TMEM lanes: pieces of 32 columns in turn
  static constexpr int kThreads = 64 + 128 * kColumnWarps;
  static constexpr int kBBytes = kTokens / kCtas * kDepth * 2;
  static constexpr int kStages = 196 * 1024 / (kABytes + kBBytes) < 10 ? 196 * 1024 / (kABytes + kBBytes) : 10;
  unsigned char a[kStages][kABytes];
  unsigned char b[kStages][kBBytes];
  unsigned long long full[kStages], empty[kStages], done[2], taken[2];
  int first_row[kMaxExperts + 1], first_tile[kMaxExperts + 1];   // of every expert: its rows, its row tiles
  uint32_t tmem_base;
};

struct Tile { int expert, row, count, output; };   // first sorted row, rows of the tile, first output of this CTA

// ---- the forms a pair of CTAs needs (kCtas 1: the plain ones) ----
template <int kCtas>
__device__ __forceinline__ void alloc_tmem(uint32_t where, uint32_t columns) {
  if constexpr (kCtas == 1) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(where), "r"(columns) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  } else {
    asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(where), "r"(columns) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
  }
}
template <int kCtas>
__device__ __forceinline__ void free_tmem(uint32_t tmem, uint32_t columns) {
  if constexpr (kCtas == 1) asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(columns) : "memory");
  else asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(columns) : "memory");
}
// A box into this CTA's shared memory; its bytes count on the barrier `bar`, which may be the pair's first CTA's.
template <int kCtas>
__device__ __forceinline__ void load_box(uint32_t dst, const CUtensorMap* map, int x, int y, uint32_t bar) {
  if constexpr (kCtas == 1) tma_load_2d(dst, map, x, y, bar);
  else asm volatile("cp.async.bulk.tensor.2d.cta_group::2.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];"
                    ::"r"(dst), "l"(reinterpret_cast<uint64_t>(map)), "r"(x), "r"(y), "r"(bar) : "memory");
}
template <int kCtas>
__device__ __forceinline__ void issue_mma(uint32_t tmem_d, uint64_t a, uint64_t b, uint32_t idesc, uint32_t accumulate) {
  if constexpr (kCtas == 1) umma_issue(tmem_d, a, b, idesc, accumulate);
  else asm volatile("{\n.reg .pred p;\nsetp.ne.b32 p, %4, 0;\n"
                    "tcgen05.mma.cta_group::2.kind::f16 [%0], %1, %2, %3, p;\n}\n"
                    ::"r"(tmem_d), "l"(a), "l"(b), "r"(idesc), "r"(accumulate) : "memory");
}
// Arrives on the barrier of every CTA of the pair when the products issued so far are done.
template <int kCtas>
__device__ __forceinline__ void commit_mma(uint32_t bar) {
  if constexpr (kCtas == 1) umma_commit(bar);
  else asm volatile("tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], %1;"
                    ::"r"(bar), "h"(static_cast<uint16_t>(3)) : "memory");
}
__device__ __forceinline__ void cluster_sync() {
  asm volatile("barrier.cluster.arrive.release.aligned;\nbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}
// The shared::cluster address of `addr` in the cluster's first CTA.
__device__ __forceinline__ uint32_t in_first_cta(uint32_t addr) {
  uint32_t there;
  asm("mapa.shared::cluster.u32 %0, %1, 0;" : "=r"(there) : "r"(addr));
  return there;
}

template <int kTokens, int kCtas>
__global__ void __launch_bounds__(ExpertShared<kTokens, kCtas>::kThreads, 1)
expert_gemm_kernel(const __grid_constant__ CUtensorMap w_map, const __grid_constant__ CUtensorMap x_map, ExpertGemm g) {
  using Shared = ExpertShared<kTokens, kCtas>;
  constexpr int kStages = Shared::kStages, kColumnWarps = Shared::kColumnWarps;
  constexpr uint32_t kColumns = 2 * kTokens < 32 ? 32 : 2 * kTokens;
  extern __shared__ unsigned char smem_raw[];
  Shared& sm = *reinterpret_cast<Shared*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~static_cast<uintptr_t>(1023));
  const int lane = threadIdx.x & 31, warp = __shfl_sync(0xffffffffu, static_cast<int>(threadIdx.x >> 5), 0);
  const int rank = kCtas == 1 ? 0 : static_cast<int>(blockIdx.x) % kCtas;   // place in the pair: clusters are consecutive blocks
  if (blockIdx.x == 0 && threadIdx.x == 0) *g.error = 0;   // a wait gives up seconds later
  if (threadIdx.x == 0) {
    for (int s = 0; s < kStages; ++s) {
      mbar_init(smem_u32(&sm.full[s]), 1);
      mbar_init(smem_u32(&sm.empty[s]), 1);
    }
    for (int b = 0; b < 2; ++b) {
      mbar_init(smem_u32(&sm.done[b]), 1);
      mbar_init(smem_u32(&sm.taken[b]), 4 * kColumnWarps * kCtas);   // one arrival per epilogue warp
    }
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == 1) alloc_tmem<kCtas>(smem_u32(&sm.tmem_base), kColumns);
  if (warp == 0) {                                // prefix sums over the experts
    int rows = 0, tiles = 0;
    for (int base = 0; base < g.experts; base += 32) {
      const int n = base + lane < g.experts ? max(g.counts[base + lane], 0) : 0, t = (n + kTokens - 1) / kTokens;
      int in = n, it = t;
#pragma unroll
      for (int x = 1; x < 32; x <<= 1) {
        const int on = __shfl_up_sync(0xffffffffu, in, x), ot = __shfl_up_sync(0xffffffffu, it, x);
        if (lane >= x) { in += on; it += ot; }
      }
      if (base + lane < g.experts) {
        sm.first_row[base + lane] = rows + in - n;
        sm.first_tile[base + lane] = tiles + it - t;
      }
      rows += __shfl_sync(0xffffffffu, in, 31);
      tiles += __shfl_sync(0xffffffffu, it, 31);
    }
    if (lane == 0) { sm.first_row[g.experts] = rows; sm.first_tile[g.experts] = tiles; }
  }
  tcgen05_before_sync();
  __syncthreads();
  if constexpr (kCtas > 1) cluster_sync();         // the other CTA's barriers exist
  tcgen05_after_sync();
  const uint32_t tmem = sm.tmem_base;
  const int first = blockIdx.x / kCtas, stride = gridDim.x / kCtas;
  const int output_tiles = (g.out + kCtas * kOutputs - 1) / (kCtas * kOutputs), tiles = sm.first_tile[g.experts] * output_tiles;
  const int steps = (g.in + kDepth - 1) / kDepth;
  auto tile_at = [&](int t) {
    const int row_tile = t / output_tiles;
    int lo = 0, hi = g.experts - 1;               // last expert with first_tile <= row_tile (experts without rows share their successor's)
    while (lo < hi) {
      const int mid = (lo + hi + 1) >> 1;
      if (sm.first_tile[mid] <= row_tile) lo = mid; else hi = mid - 1;
    }
    const int within = (row_tile - sm.first_tile[lo]) * kTokens;
    const int row = sm.first_row[lo] + within;    // (counts that claim more rows than there are never lead outside)
    return Tile{lo, row, max(min(min(kTokens, sm.first_row[lo + 1] - row), g.rows - row), 0), ((t - row_tile * output_tiles) * kCtas + rank) * kOutputs};
  };
  auto columns_of = [](int count) { return max((count + 16 * kCtas - 1) / (16 * kCtas) * (16 * kCtas), 16 * kCtas); };   // N of a tile
  bool failed = false;

  if (warp == 0) {
    if (lane == 0) {
      int stage = 0;
      uint32_t parity = 1;                        // a fresh barrier lets the first round through
      for (int t = first; t < tiles && !failed; t += stride) {
        const Tile tile = tile_at(t);
        const int row = tile.row + rank * (columns_of(tile.count) / kCtas);
        for (int k = 0; k < steps; ++k) {
          if (!mbar_wait(smem_u32(&sm.empty[stage]), parity)) { failed = true; break; }
          uint32_t bar = smem_u32(&sm.full[stage]);
          if (rank == 0) mbar_expect_tx(bar, kCtas * (kABytes + Shared::kBBytes));
          if constexpr (kCtas > 1) bar = in_first_cta(bar);
          load_box<kCtas>(smem_u32(sm.a[stage]), &w_map, k * kDepth, tile.expert * g.out + tile.output, bar);
          load_box<kCtas>(smem_u32(sm.b[stage]), &x_map, k * kDepth, row, bar);
          if (++stage == kStages) { stage = 0; parity ^= 1u; }
        }
      }
      // The commits that give the last stages back arrive on their own time, a pair's in both CTAs: wait for them before the memory goes.
      for (int s = 0; s < kStages && !failed; ++s) {
        failed = !mbar_wait(smem_u32(&sm.empty[stage]), parity);
        if (++stage == kStages) { stage = 0; parity ^= 1u; }
      }
    }
    __syncwarp();
  } else if (warp == 1) {
    int stage = 0, buffer = 0;
    uint32_t parity = 0, buffer_parity = 1;
    for (int t = rank == 0 ? first : tiles; t < tiles && !failed; t += stride) {
      const Tile tile = tile_at(t);
      const uint32_t n = static_cast<uint32_t>(columns_of(tile.count));
      const uint32_t idesc = (1u << 4) | (1u << 7) | (1u << 10) | ((n >> 3) << 17) | (static_cast<uint32_t>(kCtas * kOutputs >> 4) << 24);
      if (!__all_sync(0xffffffffu, mbar_wait(smem_u32(&sm.taken[buffer]), buffer_parity))) { failed = true; break; }
      for (int k = 0; k < steps; ++k) {
        if (!__all_sync(0xffffffffu, mbar_wait(smem_u32(&sm.full[stage]), parity))) { failed = true; break; }
        tcgen05_after_sync();
        const uint64_t a = umma_desc(smem_u32(sm.a[stage]), 16, 1024), b = umma_desc(smem_u32(sm.b[stage]), 16, 1024);
        if (elect_one()) {
#pragma unroll
          for (int s = 0; s < kDepth / 16; ++s)
            issue_mma<kCtas>(tmem + buffer * kTokens, a + static_cast<uint64_t>(s * 2), b + static_cast<uint64_t>(s * 2), idesc, (k > 0 || s > 0) ? 1u : 0u);
          commit_mma<kCtas>(smem_u32(&sm.empty[stage]));
          if (k + 1 == steps) commit_mma<kCtas>(smem_u32(&sm.done[buffer]));
        }
        __syncwarp();
        if (++stage == kStages) { stage = 0; parity ^= 1u; }
      }
      buffer ^= 1;
      if (buffer == 0) buffer_parity ^= 1u;
    }
  } else {
    const int quarter = warp & 3, first_column = (warp - 2) / 4 * 32;   // the TMEM lanes this warp may read, its first columns
    const uint32_t rows = tmem + (static_cast<uint32_t>(quarter * 32) << 16);
    int buffer = 0;
    uint32_t parity = 0;
    for (int t = first; t < tiles; t += stride) {
      const Tile tile = tile_at(t);
      if (!__all_sync(0xffffffffu, mbar_wait(smem_u32(&sm.done[buffer]), parity))) { failed = true; break; }
      tcgen05_after_sync();
      const int pair = tile.output + quarter * 32 + (lane & ~1);   // this lane stores outputs pair, pair + 1 of every second token
      __nv_bfloat16* y = static_cast<__nv_bfloat16*>(g.y) + static_cast<int64_t>(tile.row) * g.y_stride + (g.paired ? pair / 2 : pair);
      for (int c = first_column; c < tile.count; c += kColumnWarps * 32) {
        uint32_t r[32];
        tmem_load32(rows + buffer * kTokens + c, r);
        tmem_load_wait();
        if (g.paired) {
#pragma unroll
          for (int i = 0; i < 32; i += 2) {
            const uint32_t give = (lane & 1) ? r[i] : r[i + 1], keep = (lane & 1) ? r[i + 1] : r[i];
            const float got = __uint_as_float(__shfl_xor_sync(0xffffffffu, give, 1)), mine = __uint_as_float(keep);
            const float gate = (lane & 1) ? got : mine, up = (lane & 1) ? mine : got;
            const int token = c + i + (lane & 1);
            if (token < tile.count && pair < g.out) y[token * g.y_stride] = __float2bfloat16_rn(activate<__nv_bfloat16>(gate, g.act) * up);
          }
          continue;
        }
        if (g.act == kActSquaredRelu) {
#pragma unroll
          for (int i = 0; i < 32; ++i) {
            const float v = fmaxf(__uint_as_float(r[i]), 0.0f);
            r[i] = __float_as_uint(v * v);
          }
        } else if (g.act != 0) {
#pragma unroll
          for (int i = 0; i < 32; ++i) r[i] = __float_as_uint(activate<__nv_bfloat16>(__uint_as_float(r[i]), g.act));
        }
#pragma unroll
        for (int i = 0; i < 32; i += 2) {
          const uint32_t give = (lane & 1) ? r[i] : r[i + 1], keep = (lane & 1) ? r[i + 1] : r[i];
          const uint32_t got = __shfl_xor_sync(0xffffffffu, give, 1);
          const uint32_t both = (lane & 1) ? pack2<true>(__uint_as_float(got), __uint_as_float(keep)) : pack2<true>(__uint_as_float(keep), __uint_as_float(got));
          const int token = c + i + (lane & 1);
          if (token < tile.count && pair < g.out) *reinterpret_cast<uint32_t*>(y + token * g.y_stride) = both;
        }
      }
      tcgen05_before_sync();
      __syncwarp();
      if (lane == 0) {
        if constexpr (kCtas == 1) mbar_arrive(smem_u32(&sm.taken[buffer]));
        else asm volatile("mbarrier.arrive.release.cluster.shared::cluster.b64 _, [%0];" ::"r"(in_first_cta(smem_u32(&sm.taken[buffer]))) : "memory");
      }
      buffer ^= 1;
      if (buffer == 0) parity ^= 1u;
    }
  }
  if (failed && lane == 0) atomicOr(g.error, 1u);
  tcgen05_before_sync();
  __syncthreads();
  if constexpr (kCtas > 1) cluster_sync();         // neither CTA leaves while the other's copies, products and arrivals may reach its memory
  if (warp == 1) free_tmem<kCtas>(tmem, kColumns);
}

int make_matrix_map(CUtensorMap* map, const void* base, int64_t rows, int64_t columns, int64_t stride, int box_rows) {
  return make_box_map<2>(map, base, {columns, rows}, {1, stride}, {kDepth, box_rows});
}

template <int kTokens, int kCtas>
int launch(const ExpertGemm& g, int sm_count, cudaStream_t stream) {
  CUtensorMap w_map, x_map;
  if (make_matrix_map(&w_map, g.w, static_cast<int64_t>(g.experts) * g.out, g.in, g.in, kOutputs) != RLT_OK ||
      make_matrix_map(&x_map, g.x, g.rows, g.in, g.x_stride, kTokens / kCtas) != RLT_OK) {
    set_last_error_text("expert_gemm: cuTensorMapEncodeTiled rejected the operands");
    return RLT_ERR_UNSUPPORTED;
  }
  auto kernel = expert_gemm_kernel<kTokens, kCtas>;
  const size_t smem = sizeof(ExpertShared<kTokens, kCtas>) + 1024;
  RLT_CUDA_TRY(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(smem)));
  const int64_t row_tiles = static_cast<int64_t>(g.rows) / kTokens + (g.rows < g.experts ? g.rows : g.experts);
  const int64_t most = row_tiles * ((g.out + kCtas * kOutputs - 1) / (kCtas * kOutputs)), groups = sm_count / kCtas;
  cudaLaunchConfig_t config = {};
  config.gridDim = dim3(static_cast<unsigned>((most < groups ? most : groups) * kCtas));
  config.blockDim = dim3(ExpertShared<kTokens, kCtas>::kThreads); config.dynamicSmemBytes = smem; config.stream = stream;
  cudaLaunchAttribute cluster;
  cluster.id = cudaLaunchAttributeClusterDimension;
  cluster.val.clusterDim.x = kCtas; cluster.val.clusterDim.y = 1; cluster.val.clusterDim.z = 1;
  config.attrs = &cluster; config.numAttrs = kCtas > 1 ? 1 : 0;
  RLT_CUDA_TRY(cudaLaunchKernelEx(&config, kernel, w_map, x_map, g));
  return launch_status("expert_gemm_kernel");
}

}  // namespace

bool expert_gemm_sm100_supported(const ExpertGemm& g) {
  return g.dtype == RLT_BF16 && g.in % 8 == 0 && g.out % 8 == 0 && g.x_stride % 8 == 0 && g.y_stride % 2 == 0 && g.experts <= kMaxExperts &&
         static_cast<int64_t>(g.experts) * g.out <= 0x7fffffff && aligned16(g.x) && aligned16(g.w) && aligned16(g.y) && g.error != nullptr;
}

int launch_expert_gemm_sm100(const ExpertGemm& g, cudaStream_t stream) {
  DeviceInfo info;
  const int status = current_device_info(&info);
  if (status != RLT_OK) return status;
  // Rows of 128 in single CTAs / of 256 in pairs, us: 64 experts of 704 -> 2048 with 64 rows each 37 / 40, 96: 40 / 42, 128: 42 / 44, 160: 58 / 48,
  // and of unequal numbers, which routing gives, 64: 38 / 40, 96: 42 / 42, 112: 46 / 44, 128: 49 / 47, 192: 61 / 53; 2048 -> 1408 unequal 96: 73 / 77,
  // 112: 79 / 77, 128: 87 / 81.  (8 experts of 4096 -> 2816 take pairs from 16 rows on, 47 / 46; at 96 50 / 47.)  Rows of 32 / of 128 at 24 rows: 63 / 64
  // and 70 / 64 unequal, at 48 88 / 66.  One block of outputs, 64 experts of 2048 -> 128: single CTAs 16 / pairs 16 for 128 rows, 35 / 37 for 512.
  const int64_t average = g.rows / g.experts;
  if (average <= 24) return launch<32, 1>(g, info.sm_count, stream);
  if (average <= 96 || g.out <= kOutputs) return launch<128, 1>(g, info.sm_count, stream);   // one block of outputs: nothing for a second CTA
  return launch<256, 2>(g, info.sm_count, stream);
}

}  // namespace rlt
