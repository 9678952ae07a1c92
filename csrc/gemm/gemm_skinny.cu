// K0s: "skinny" bf16 GEMM for decode, C[Mb, N] = X[Mb, K] . W[N, K]^T with Mb <= 32 rows.
//
// A decode step multiplies a handful of token rows by every weight matrix of the model: the work is the
// weight stream (HBM-bound), not the FLOPs.  The general kernel tiles C as 128 x BN with X as the 128-row A
// operand, which for Mb = 8 (a) launches only N/128 CTAs — 32 for a 4096-wide layer, so 116 of the 148 SMs
// pull nothing — and (b) spends half of every pipeline stage on a mostly zero-filled X tile.  Here the
// operands are swapped and K is split:
//   * UMMA M = 128 weight rows (A operand = W tile, 16 KB per 64-wide k block), UMMA N = MB = 16 or 32 token
//     rows (B operand = X tile, 2-4 KB): the stage is almost all weights, 10-11 stages = ~170 KB of weight
//     bytes in flight per SM;
//   * stream-K: the (128-row tile, 64-wide k block) space is flattened and cut into one equal range per SM, so
//     every SM streams the same number of weight bytes through ONE pipeline that never drains at a tile
//     boundary (persistent CTA, barriers / TMEM set up once).  A CTA accumulates each tile piece in TMEM
//     (128 lanes x MB fp32 columns, double buffered so the epilogue overlaps the next piece); tiles cut by a
//     range boundary go through an fp32 workspace and the last piece to arrive (atomic ticket) sums the
//     pieces in slot order — deterministic — and writes bf16 C.  The ticket counter is reset by that CTA, so
//     the workspace needs no clearing between calls.
// Measured alternative (B200, 8 x 4096 -> 12288): two 5-stage CTAs per SM with four ranges per SM (hardware hands the
// second wave to whichever SM drains first) — 38.5 us against 28.9 us for one 11-stage CTA per SM; kept as is.
// Warp roles as in gemm_tcgen05.cu: warp 0 TMA, warp 1 MMA, warps 2-5 epilogue (thread = weight row).
//
// Reference: decode in the reference is the HF model's cuBLAS GEMMs over the whole padded batch (reference
// llmctl/serve/server.py:199-204).  Baseline: cuBLAS (gemv-like kernels) at the same shapes.
#include "../common/ptx.cuh"
#include "../common/tma_host.h"
#include "../common/util.cuh"
#include "../common/dependent.cuh"

namespace llmctl {
using namespace ptx;

namespace skinny {
constexpr int kBM = 128;                 // weight rows per CTA (UMMA M)
constexpr int kBK = 64;                  // k elements per stage (128 bytes: one swizzle row)
constexpr int kWBytes = kBM * kBK * 2;   // 16 KB
constexpr int kThreads = 192;
template <int MB>
struct Cfg {
  static constexpr int kXBytes = MB * kBK * 2;                 // 2 KB (MB = 16) or 4 KB (MB = 32)
  static constexpr int kStageBytes = kWBytes + kXBytes;
  static constexpr int kStages = (MB == 16) ? 11 : 10;
  static constexpr int kSmem = kStages * kStageBytes + 1024;
};
}  // namespace skinny

template <int MB>
__global__ void __launch_bounds__(skinny::kThreads, 1)
gemm_skinny_kernel(const __grid_constant__ CUtensorMap tmW, const __grid_constant__ CUtensorMap tmX,
                   __nv_bfloat16* __restrict__ C, long long ldc, int Mb, int N, int num_kb, int n_tiles, int L,
                   int max_slots, float* __restrict__ workspace, unsigned int* __restrict__ counters) {
  using namespace skinny;
  using C_ = Cfg<MB>;
  extern __shared__ uint8_t smem_raw[];
  __shared__ uint64_t bar_full[C_::kStages], bar_empty[C_::kStages], bar_acc_full[2], bar_acc_empty[2];
  __shared__ uint32_t tmem_base_smem;
  __shared__ int s_last;
  const uint32_t smem_base = (smem_u32(smem_raw) + 1023u) & ~1023u;
  uint8_t* smem = smem_raw + (smem_base - smem_u32(smem_raw));
  const int warp = __shfl_sync(0xffffffffu, threadIdx.x >> 5, 0), lane = threadIdx.x & 31;
  // stream-K: the (tile, k block) space is flattened and cut into equal ranges, one per CTA
  const long long total = static_cast<long long>(n_tiles) * num_kb;
  const long long begin = static_cast<long long>(blockIdx.x) * L;
  const long long end = (begin + L < total) ? begin + L : total;

  if (threadIdx.x == 0) {
    for (int i = 0; i < C_::kStages; ++i) {
      mbar_init(&bar_full[i], 1);
      mbar_init(&bar_empty[i], 1);
    }
    for (int i = 0; i < 2; ++i) {
      mbar_init(&bar_acc_full[i], 1);
      mbar_init(&bar_acc_empty[i], 4);
    }
    fence_mbar_init();
  }
  if (warp == 0 && lane == 0) {
    prefetch_tmap(&tmW);
    prefetch_tmap(&tmX);
  }
  if (warp == 1) tmem_alloc<1>(&tmem_base_smem, 64);
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = tmem_base_smem;
  if (warp == 0 && lane == 0) {        // the first weights on their way to L2 beside the end of the kernel before
    int tile = static_cast<int>(begin / num_kb), kb = static_cast<int>(begin % num_kb);
    for (int i = 0; i < C_::kStages && begin + i < end; ++i) {
      tma_prefetch_2d(&tmW, kb * kBK, tile * kBM);
      if (++kb == num_kb) {
        kb = 0;
        ++tile;
      }
    }
  }
  wait_for_previous(C, workspace, counters);

  if (warp == 0) {
    if (lane == 0) {
      int stage = 0;
      uint32_t phase = 0;
      int tile = static_cast<int>(begin / num_kb), kb = static_cast<int>(begin % num_kb);
      for (long long pos = begin; pos < end; ++pos) {
        mbar_wait(&bar_empty[stage], phase ^ 1u);
        uint8_t* sW = smem + stage * C_::kStageBytes;
        uint8_t* sX = sW + kWBytes;
        mbar_expect_tx(&bar_full[stage], C_::kStageBytes);
        tma_load_2d(sW, &tmW, &bar_full[stage], kb * kBK, tile * kBM);   // rows past N read as zero
        tma_load_2d(sX, &tmX, &bar_full[stage], kb * kBK, 0);            // rows past Mb read as zero
        if (++stage == C_::kStages) {
          stage = 0;
          phase ^= 1u;
        }
        if (++kb == num_kb) {
          kb = 0;
          ++tile;
        }
      }
      release_dependents();
    }
  } else if (warp == 1) {
    // the whole warp walks the loop, one elected lane issues (descriptors stay in uniform registers, see gemm_tcgen05.cu)
    constexpr uint32_t idesc = make_idesc_bf16(kBM, MB, 0u, 0u);
    int stage = 0;
    uint32_t phase = 0;
    int seg = 0;
    for (long long pos = begin; pos < end; ++seg) {
      const int kb_s = static_cast<int>(pos % num_kb);
      const long long left = end - pos;
      const int seg_len = (num_kb - kb_s < left) ? num_kb - kb_s : static_cast<int>(left);
      const int buf = seg & 1;
      mbar_wait(&bar_acc_empty[buf], ((seg >> 1) & 1u) ^ 1u);
      __syncwarp();
      tc_fence_after();
      const uint32_t d_tmem = tmem_base + buf * 32;
      for (int i = 0; i < seg_len; ++i) {
        mbar_wait(&bar_full[stage], phase);
        __syncwarp();
        tc_fence_after();
        const uint32_t w_addr = smem_base + stage * C_::kStageBytes;
        const uint64_t dw = make_smem_desc(w_addr, 16, 1024, 2), dx = make_smem_desc(w_addr + kWBytes, 16, 1024, 2);
        if (elect_one()) {
#pragma unroll
          for (int k = 0; k < kBK / 16; ++k) umma_ss<1>(d_tmem, dw + k * 2, dx + k * 2, idesc, (i | k) != 0 ? 1u : 0u);
          umma_commit<1>(&bar_empty[stage]);
          if (i + 1 == seg_len) umma_commit<1>(&bar_acc_full[buf]);
        }
        if (++stage == C_::kStages) {
          stage = 0;
          phase ^= 1u;
        }
      }
      pos += seg_len;
    }
  } else {
    // ------------------------------ epilogue (4 warps, thread = weight row) ------------------------------
    const int q = warp & 3;
    const int row = q * 32 + lane;
    int seg = 0;
    for (long long pos = begin; pos < end; ++seg) {
      const int tile = static_cast<int>(pos / num_kb);
      const int kb_s = static_cast<int>(pos % num_kb);
      const long long left = end - pos;
      const int seg_len = (num_kb - kb_s < left) ? num_kb - kb_s : static_cast<int>(left);
      const int buf = seg & 1;
      const int n = tile * kBM + row;
      uint32_t r[MB];
      mbar_wait(&bar_acc_full[buf], (seg >> 1) & 1u);
      tc_fence_after();
      const uint32_t taddr = tmem_base + buf * 32 + (static_cast<uint32_t>(q * 32) << 16);
      if constexpr (MB == 16) {
        tmem_ld_x16(taddr, r);
      } else {
        tmem_ld_x32(taddr, r);
      }
      tmem_ld_wait();
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(&bar_acc_empty[buf]);       // the MMA warp may start the segment after next
      // CTAs that own a piece of this tile: ranges are L long, so it is pure arithmetic
      const long long t_begin = static_cast<long long>(tile) * num_kb;
      const int first = static_cast<int>(t_begin / L);
      const int last = static_cast<int>((t_begin + num_kb - 1) / L);
      const int count = last - first + 1;
      if (count == 1) {
        if (n < N) {
#pragma unroll
          for (int m = 0; m < MB; ++m)
            if (m < Mb) C[m * ldc + n] = __float2bfloat16(__uint_as_float(r[m]));
        }
      } else {
        float* wt = workspace + static_cast<size_t>(tile) * max_slots * MB * kBM;
        float* ws = wt + static_cast<size_t>(static_cast<int>(blockIdx.x) - first) * MB * kBM;
#pragma unroll
        for (int m = 0; m < MB; ++m)
          if (m < Mb) ws[m * kBM + row] = __uint_as_float(r[m]);
        __threadfence();
        named_bar_sync(1, 128);
        if (threadIdx.x == 64) {
          const unsigned int ticket = atomicAdd(&counters[tile], 1u);
          s_last = (ticket == static_cast<unsigned int>(count - 1)) ? 1 : 0;
        }
        named_bar_sync(1, 128);
        if (s_last) {                        // last piece to arrive: sum the pieces in slot order (deterministic)
          __threadfence();
          if (n < N) {
#pragma unroll 1
            for (int m0 = 0; m0 < Mb; m0 += 8) {
              // 8 rows x 4 pieces asked for together: one at a time, the L2 round trips of 32 rows x 4 pieces took 20 us
              float sum[8];
#pragma unroll
              for (int j = 0; j < 8; ++j) sum[j] = 0.f;
#pragma unroll 1
              for (int sp = 0; sp < count; sp += 4) {
                float v[4][8];
#pragma unroll
                for (int u = 0; u < 4; ++u)
#pragma unroll
                  for (int j = 0; j < 8; ++j)
                    v[u][j] = (sp + u < count && m0 + j < Mb) ? __ldcg(wt + (static_cast<size_t>(sp + u) * MB + m0 + j) * kBM + row) : 0.f;
#pragma unroll
                for (int u = 0; u < 4; ++u)
#pragma unroll
                  for (int j = 0; j < 8; ++j) sum[j] += v[u][j];
              }
#pragma unroll
              for (int j = 0; j < 8; ++j)
                if (m0 + j < Mb) C[(m0 + j) * ldc + n] = __float2bfloat16(sum[j]);
            }
          }
          if (threadIdx.x == 64) counters[tile] = 0u;     // ready for the next call on this stream
        }
      }
      pos += seg_len;
    }
  }

  tc_fence_before();
  __syncthreads();
  if (warp == 1) {
    tc_fence_after();
    tmem_dealloc<1>(tmem_base, 64);
  }
}

// A layer whose tiles of weight rows are few is no stream but a latency: launch, first bytes, and the way of the pieces through the workspace (store,
// fence, ticket, and their sum by one CTA), 6-10 us for any few MB of weights.  Here a cluster of S CTAs takes a tile's K, a share each, and every CTA sums and
// stores MB / S of the token rows, whose partial sums come through distributed shared memory (over the operand ring, idle by then) and are
// added in the order of the ranks: no workspace, no ticket.
template <int MB, int S>
__global__ void __launch_bounds__(skinny::kThreads, 1)
gemm_skinny_cluster_kernel(const __grid_constant__ CUtensorMap tmW, const __grid_constant__ CUtensorMap tmX, __nv_bfloat16* __restrict__ C, long long ldc, int Mb, int N,
                           int num_kb) {
  using namespace skinny;
  using C_ = Cfg<MB>;
  constexpr int kOwn = MB / S;               // token rows that a CTA sums and stores
  static_assert(kOwn >= 2 && (S * kBM * kOwn + 32) * 4 <= C_::kStages * C_::kStageBytes, "exchange");
  extern __shared__ uint8_t smem_raw[];
  __shared__ uint64_t bar_full[C_::kStages], bar_empty[C_::kStages], bar_done;
  __shared__ uint32_t tmem_base_smem;
  const uint32_t smem_base = (smem_u32(smem_raw) + 1023u) & ~1023u;
  uint8_t* smem = smem_raw + (smem_base - smem_u32(smem_raw));
  const int warp = __shfl_sync(0xffffffffu, threadIdx.x >> 5, 0), lane = threadIdx.x & 31;
  const int rank = static_cast<int>(cluster_ctarank()), tile = blockIdx.x / S;
  const int kb0 = num_kb * rank / S, kb1 = num_kb * (rank + 1) / S;

  if (threadIdx.x == 0) {
    for (int i = 0; i < C_::kStages; ++i) {
      mbar_init(&bar_full[i], 1);
      mbar_init(&bar_empty[i], 1);
    }
    mbar_init(&bar_done, 1);
    fence_mbar_init();
    prefetch_tmap(&tmW);
    prefetch_tmap(&tmX);
  }
  if (warp == 1) tmem_alloc<1>(&tmem_base_smem, 32);
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = tmem_base_smem;
  if (warp == 0 && lane == 0)          // the first weights on their way to L2 beside the end of the kernel before
    for (int kb = kb0; kb < kb1 && kb < kb0 + C_::kStages; ++kb) tma_prefetch_2d(&tmW, kb * kBK, tile * kBM);
  wait_for_previous(C);
  float acc[MB];
  if (warp == 0) {
    if (lane == 0) {
      for (int kb = kb0, i = 0; kb < kb1; ++kb, ++i) {
        const int stage = i % C_::kStages;
        mbar_wait(&bar_empty[stage], ((i / C_::kStages) & 1u) ^ 1u);
        uint8_t* sW = smem + stage * C_::kStageBytes;
        mbar_expect_tx(&bar_full[stage], C_::kStageBytes);
        tma_load_2d(sW, &tmW, &bar_full[stage], kb * kBK, tile * kBM);   // rows past N read as zero
        tma_load_2d(sW + kWBytes, &tmX, &bar_full[stage], kb * kBK, 0);  // rows past Mb read as zero
      }
      release_dependents();
    }
    __syncwarp();
  } else if (warp == 1) {
    constexpr uint32_t idesc = make_idesc_bf16(kBM, MB, 0u, 0u);
    for (int kb = kb0, i = 0; kb < kb1; ++kb, ++i) {
      const int stage = i % C_::kStages;
      mbar_wait(&bar_full[stage], (i / C_::kStages) & 1u);
      __syncwarp();
      tc_fence_after();
      const uint32_t w_addr = smem_base + stage * C_::kStageBytes;
      const uint64_t dw = make_smem_desc(w_addr, 16, 1024, 2), dx = make_smem_desc(w_addr + kWBytes, 16, 1024, 2);
      if (elect_one()) {
#pragma unroll
        for (int k = 0; k < kBK / 16; ++k) umma_ss<1>(tmem_base, dw + k * 2, dx + k * 2, idesc, (i | k) != 0 ? 1u : 0u);
        umma_commit<1>(&bar_empty[stage]);
        if (kb + 1 == kb1) umma_commit<1>(&bar_done);
      }
    }
    __syncwarp();
  } else {
    mbar_wait(&bar_done, 0u);
    __syncwarp();
    tc_fence_after();
    uint32_t r[MB];
    const uint32_t taddr = tmem_base + (static_cast<uint32_t>((warp & 3) * 32) << 16);
    if constexpr (MB == 16) tmem_ld_x16(taddr, r); else tmem_ld_x32(taddr, r);
    tmem_ld_wait();
#pragma unroll
    for (int m = 0; m < MB; ++m) acc[m] = __uint_as_float(r[m]);
  }
  const int row = (warp & 3) * 32 + lane;
  cluster_sync();                      // every CTA's loads have landed and been multiplied: the rings may be written over
  if (warp >= 2) {
#pragma unroll
    for (int to = 0; to < S; ++to) {
      const uint32_t at = mapa_u32(smem_base + (rank * kBM + row) * kOwn * 4, to);
#pragma unroll
      for (int m = 0; m < kOwn; m += (kOwn >= 4 ? 4 : 2)) {
        const float* v = acc + to * kOwn + m;
        if constexpr (kOwn >= 4) st_cluster_v4(at + m * 4, make_float4(v[0], v[1], v[2], v[3])); else st_cluster_v2(at + m * 4, make_float2(v[0], v[1]));
      }
    }
  }
  cluster_sync();
  const int n = tile * kBM + row;
  if (warp >= 2 && n < N) {
    const float* mine = reinterpret_cast<const float*>(smem) + row * kOwn;
    float sum[kOwn] = {};
#pragma unroll
    for (int src = 0; src < S; ++src)
#pragma unroll
      for (int m = 0; m < kOwn; ++m) sum[m] += mine[src * kBM * kOwn + m];
#pragma unroll
    for (int m = 0; m < kOwn; ++m)
      if (rank * kOwn + m < Mb) C[(rank * kOwn + m) * ldc + n] = __float2bfloat16(sum[m]);
  }
  tc_fence_before();
  __syncthreads();
  if (warp == 1) {
    tc_fence_after();
    tmem_dealloc<1>(tmem_base, 32);
  }
}

template <int MB, int S>
static int launch_skinny_cluster(const CUtensorMap& tw, const CUtensorMap& tx, __nv_bfloat16* C, long long ldc, int Mb, int N, int num_kb, int n_tiles, cudaStream_t s) {
  auto kern = gemm_skinny_cluster_kernel<MB, S>;
  LLMCTL_CHECK(allow_smem(kern, skinny::Cfg<MB>::kSmem));
  cudaLaunchAttribute at[2];
  at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at[0].val.programmaticStreamSerializationAllowed = 1;
  at[1].id = cudaLaunchAttributeClusterDimension;
  at[1].val.clusterDim = {S, 1, 1};
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = n_tiles * S;
  cfg.blockDim = skinny::kThreads;
  cfg.dynamicSmemBytes = skinny::Cfg<MB>::kSmem;
  cfg.stream = s;
  cfg.attrs = at;
  cfg.numAttrs = 2;
  LLMCTL_CHECK(cudaLaunchKernelEx(&cfg, kern, tw, tx, C, ldc, Mb, N, num_kb));
  LLMCTL_RETURN_LAST();
}

}  // namespace llmctl

using namespace llmctl;

namespace llmctl {
namespace skinny {
// CTAs of a cluster that share a tile's K, 0: the stream of all SMs (gemm_skinny_kernel).  As many as are resident together, one to an SM and whole
// clusters to a GPC: 96 CTAs in eights, 128 in fours (2048 x 2048: 16 tiles in eights 7.9 us, in fours 4.9).  us, stream / clusters, 32 rows (1 row),
// weights from HBM: 768 x 768 9.0 / 3.5 (6.5 / 3.1), 1344 x 2048 9.1 / 4.5 (6.2 / 4.0), 2048 x 5632 15.0 / 8.8 (9.7 / 7.8), 4096 x 4096 14.8 / 9.5
// (10.6 / 8.4), 4096 x 11008 23.7 / 18.0 (18.8 / 16.8), 6144 x 2048 13.0 / 8.4 (9.5 / 7.4), 8192 x 2048 13.5 / 9.4; beyond 64 tiles the stream fills the SMs better.
static int cluster_size(int n_tiles, int num_kb) {
  const int fit = n_tiles <= 12 ? 8 : n_tiles <= 32 ? 4 : n_tiles <= 64 ? 2 : 0;
  return fit <= num_kb ? fit : 0;
}
// k blocks per CTA and the floats of scratch that its pieces of tiles take
struct Plan {
  int MB, n_tiles, num_kb;
  long long total, L;
  Plan(int Mb, int N, int K, int splits) {
    MB = Mb <= 16 ? 16 : 32;
    n_tiles = (N + kBM - 1) / kBM;
    num_kb = (K + kBK - 1) / kBK;
    total = static_cast<long long>(n_tiles) * num_kb;
    // `splits` > 0 forces num_kb / splits (tests); otherwise an even share of all SMs, but never less than 8 blocks (128 KB of weights) so
    // small layers are not shredded
    if (splits > 0) {
      L = (num_kb + splits - 1) / splits;
    } else {
      L = (total + kNumSMs - 1) / kNumSMs;
      if (L < 8) L = 8;
    }
  }
  long long slots() const { return (num_kb + L - 1) / L + 1; }
  long long scratch() const { return n_tiles * slots() * MB * kBM; }
};
}  // namespace skinny
}  // namespace llmctl

// Floats of `workspace` with which llmctl_gemm_skinny_bf16 splits K as it would like to.
LLMCTL_API long long llmctl_gemm_skinny_scratch_elems(int Mb, int N, int K, int splits) {
  if (Mb < 1 || Mb > 32 || N < 1 || K < 1) return 0;
  return skinny::Plan(Mb, N, K, splits).scratch();
}

// The id of the capture that the stream is part of, 0 if it is not being captured.
LLMCTL_API unsigned long long llmctl_stream_capture_id(void* stream) {
  cudaStreamCaptureStatus status = cudaStreamCaptureStatusNone;
  unsigned long long id = 0;
  if (cudaStreamGetCaptureInfo((cudaStream_t)stream, &status, &id) != cudaSuccess || status != cudaStreamCaptureStatusActive) return 0;
  return id;
}

// C[Mb, N] (bf16, row stride ldc) = X[Mb, K] (row stride ldx) . W[N, K]^T (row stride ldw), 1 <= Mb <= 32.
// workspace: fp32 scratch for split-K partials (workspace_elems floats); counters: n_counters zero-initialised
// uint32 tickets (>= ceil(N/128)), left zero again on return.  One call at a time per (workspace, counters)
// pair: calls on the same stream are fine, concurrent streams need their own pair, and so does a graph that is replayed
// beside other work.  splits <= 0 picks it.
LLMCTL_API int llmctl_gemm_skinny_bf16(const void* X, const void* W, void* C, int Mb, int N, int K, long long ldx,
                                       long long ldw, long long ldc, float* workspace, long long workspace_elems,
                                       unsigned int* counters, int n_counters, int splits, void* stream) {
  LLMCTL_BEGIN();
  LLMCTL_REQUIRE(Mb >= 1 && Mb <= 32 && N >= 1 && K >= 8 && K % 8 == 0 && ldx % 8 == 0 && ldw % 8 == 0);
  skinny::Plan plan(Mb, N, K, splits);
  const int MB = plan.MB, n_tiles = plan.n_tiles, num_kb = plan.num_kb;
  const bool have_ws = workspace != nullptr && counters != nullptr && n_counters >= n_tiles;
  if (!have_ws || plan.scratch() > workspace_elems) {
    // no (or too little) scratch: whole tiles per CTA, no fix-up needed
    const long long tiles_per_cta = (n_tiles + kNumSMs - 1) / kNumSMs;
    plan.L = tiles_per_cta * num_kb;
  }
  const long long L = plan.L, total = plan.total;
  const int max_slots = static_cast<int>(plan.slots());
  const unsigned grid = static_cast<unsigned>((total + L - 1) / L);
  CUtensorMap tw, tx;
  int rc = get_tmap_2d_bf16(&tw, W, N, K, ldw, skinny::kBM, skinny::kBK, 1);
  if (rc) LLMCTL_FAIL(rc, "tensor map W");
  rc = get_tmap_2d_bf16(&tx, X, Mb, K, ldx, MB, skinny::kBK, 1);
  if (rc) LLMCTL_FAIL(rc, "tensor map X");
  cudaStream_t s = (cudaStream_t)stream;
  const int cluster = splits > 0 ? 0 : skinny::cluster_size(n_tiles, num_kb);
  if (cluster) {
    const auto launch = MB == 16 ? (cluster == 8 ? launch_skinny_cluster<16, 8> : cluster == 4 ? launch_skinny_cluster<16, 4> : launch_skinny_cluster<16, 2>)
                                 : (cluster == 8 ? launch_skinny_cluster<32, 8> : cluster == 4 ? launch_skinny_cluster<32, 4> : launch_skinny_cluster<32, 2>);
    return launch(tw, tx, (__nv_bfloat16*)C, ldc, Mb, N, num_kb, n_tiles, s);
  }
  if (MB == 16) {
    LLMCTL_CHECK(allow_smem(gemm_skinny_kernel<16>, skinny::Cfg<16>::kSmem));
    LLMCTL_CHECK(launch_dependent(gemm_skinny_kernel<16>, grid, skinny::kThreads, skinny::Cfg<16>::kSmem, s, tw, tx, (__nv_bfloat16*)C, ldc, Mb, N,
                                  num_kb, n_tiles, static_cast<int>(L), max_slots, workspace, counters));
  } else {
    LLMCTL_CHECK(allow_smem(gemm_skinny_kernel<32>, skinny::Cfg<32>::kSmem));
    LLMCTL_CHECK(launch_dependent(gemm_skinny_kernel<32>, grid, skinny::kThreads, skinny::Cfg<32>::kSmem, s, tw, tx, (__nv_bfloat16*)C, ldc, Mb, N,
                                  num_kb, n_tiles, static_cast<int>(L), max_slots, workspace, counters));
  }
  LLMCTL_RETURN_LAST();
}
