// K0: bf16 GEMM on the 5th-generation tensor cores.  D[M,N] (+)= op(A) * op(B), fp32 accumulation in
// tensor memory.
//
//   * operands staged by TMA (cp.async.bulk.tensor, 128-byte swizzle) into a multi-stage smem ring
//   * one elected thread issues tcgen05.mma (UMMA 128 x BN x 16, kind::f16) per k-slice
//   * accumulators double-buffered in TMEM (2 x BN columns) so the epilogue of tile i overlaps the
//     main loop of tile i+1
//   * persistent CTAs (one per SM) walk the tile list; warp roles: 0 = TMA producer, 1 = MMA issuer
//     (+ TMEM alloc), 2..5 = epilogue (tcgen05.ld -> convert -> global)
//
// Operand layouts (both operands independently):
//   K-major  : A is [M,K] row-major (K contiguous) / B is [N,K] row-major   (torch Linear weight)
//   MN-major : A is stored [K,M] row-major (M contiguous) / B is stored [K,N] row-major
// which covers forward (x Wt), dgrad (dy W) and wgrad (dyT x) without any transposes in HBM.
//
// Reference: none — every GEMM in the reference is a cuBLAS call made by HF modules behind
// `self.model(**batch)` (reference llmctl/runtime/engine.py:284) and `torch.matmul`
// (reference llmctl/cli/commands/hw.py:317-337, llmctl/plugins/autotuning.py:89-114).
// Baseline to beat: cuBLASLt bf16 (MEASURED_PEAKS.json).
#include "../comm/symm.cuh"
#include "../common/dependent.cuh"
#include "../common/tma_host.h"
#include "../common/util.cuh"

namespace llmctl {
using namespace ptx;

// K1 (sequence-parallel all-gather -> GEMM) runs on this kernel: the rows of A live in a symmetric buffer that the
// peers' producers fill over NVLink (csrc/fused/ag_push.cu); every `rows_per_flag` rows carry an epoch flag in the
// local signal pad.  The TMA producer waits for the flags of the rows a tile needs, so the MMAs of what has arrived
// overlap the transfer of what has not; tile rows are visited in arrival order (own chunk first, then the first
// slab of every peer, the second slab of every peer, ...).  flags == NULL: plain GEMM.
struct GemmGate {
  const uint32_t* flags;
  uint32_t epoch;
  int rows_per_flag;
  int own_lo, own_hi;        // rows that are local and never waited for
  int perm;                  // 1: arrival-order permutation of the tile-row blocks
  int rank, world;
  int bpc, bps;              // tile-row blocks per rank chunk / per flag slab
  // K8 (ZeRO-3 parameter gather consumed by the GEMM): the B operand lives in a symmetric buffer that the owners of
  // its shards fill over NVLink; flag f covers flat elements [f*b_slab, (f+1)*b_slab) of that buffer.
  const uint32_t* b_flags;
  uint32_t b_epoch;
  long long b_off;           // element offset of B inside the gathered buffer
  long long b_slab;          // elements per flag
  long long b_row_stride;    // K-major B: elements between consecutive N rows
  long long b_span;          // MN-major B: elements of the whole matrix (a tile touches every K row)
  // Grouped GEMM (mixture of experts): B is [experts * N, K] (K-major) and tile-row block i of A multiplies the matrix of
  // expert grp_tile_expert[i]; blocks at and beyond *grp_num_tiles (a device-side count) are skipped by every role.
  const int* grp_tile_expert;
  const int* grp_num_tiles;
  int grp_experts;
  __host__ __device__ bool waits() const { return flags != nullptr || b_flags != nullptr; }
};
// Row of B where the tile's N range starts, or -1 if this tile-row block holds no rows (grouped mode only).
__device__ __forceinline__ int grouped_b_row(const GemmGate& g, int m_blk, int n0, int N) {
  if (g.grp_tile_expert == nullptr) return n0;
  if (m_blk >= *g.grp_num_tiles) return -1;
  return g.grp_tile_expert[m_blk] * N + n0;
}
__device__ __forceinline__ int gate_perm(const GemmGate& g, int i) {
  if (!g.perm) return i;
  if (i < g.bpc) return g.rank * g.bpc + i;
  const int j = i - g.bpc, per_s = (g.world - 1) * g.bps;
  const int s = j / per_s, w = j - s * per_s, p = w / g.bps, b = w - p * g.bps;
  return ((g.rank + 1 + p) % g.world) * g.bpc + s * g.bps + b;
}
__device__ __forceinline__ void gate_wait(const GemmGate& g, int m0, int m_end) {
  if (g.flags == nullptr) return;
  const int R = g.rows_per_flag;
  for (int f = m0 / R; f <= (m_end - 1) / R; ++f) {
    const int fr = f * R;
    if (fr >= g.own_lo && fr < g.own_hi) continue;
    symm::signal_wait_ge(g.flags + f, g.epoch);
  }
  fence_proxy_async_all();      // generic-proxy flag reads -> async-proxy (TMA) reads of the rows
}
template <bool B_MN>
__device__ __forceinline__ void gate_wait_b(const GemmGate& g, int n0, int n_end) {
  if (g.b_flags == nullptr || n0 >= n_end) return;
  long long lo, hi;
  if (!B_MN) {
    lo = g.b_off + static_cast<long long>(n0) * g.b_row_stride;
    hi = g.b_off + static_cast<long long>(n_end) * g.b_row_stride;
  } else {
    lo = g.b_off;
    hi = g.b_off + g.b_span;
  }
  for (long long f = lo / g.b_slab; f <= (hi - 1) / g.b_slab; ++f) symm::signal_wait_ge(g.b_flags + f, g.b_epoch);
  fence_proxy_async_all();
}

constexpr int kBM = 128;
constexpr int kBK = 64;  // 64 bf16 = one 128-byte swizzle row
constexpr int kGemmThreads = 192;
// Output staging of the epilogue: boxes of 32 rows x 64 bf16 (128-byte swizzle) that TMA stores read.  Each of the four warps has one
// buffer, two with a gated activation.  A second one for the plain product gains nothing (its stores hide behind the next tile's main loop,
// and a CTA's last tile is staged in the operand ring, see OutStage) and takes the room that the kernels of the communication streams
// (fused/ag_push.cu, fused/rs_adam.cu) need beside a persistent GEMM, which holds its SM's shared memory to the end: with it one of their
// CTAs fitted, where their registers allow two; beside a gated activation's 196-209 registers they allow one.
constexpr int kOutBox = 32 * 128;
constexpr int kSmShared = 228 * 1024, kNeighbourShared = 1280;      // of an SM; of such a CTA (static, the reserved KB, rounded up)
enum class Gated { kNone, kForward, kBackward, kRotate };       // what the epilogue does besides storing
constexpr bool plain_output(Gated g) { return g == Gated::kNone || g == Gated::kRotate; }
constexpr int out_bufs(Gated g) { return plain_output(g) ? 1 : 2; }

template <int BN, Gated kGated = Gated::kNone>
struct GemmCfg {
  static constexpr int kStages = (BN == 256 || BN == 192) ? 4 : (BN == 128 ? 6 : 8);
  static constexpr int kABytes = kBM * kBK * 2;
  static constexpr int kBBytes = BN * kBK * 2;
  static constexpr int kStageBytes = kABytes + kBBytes;
  static constexpr int kOutAt = kStages * kStageBytes;
  static constexpr int kSmemBytes = kOutAt + 4 * out_bufs(kGated) * kOutBox + 1024;    // + alignment slack
  static constexpr int kTmemCols = (2 * BN <= 128) ? 128 : (2 * BN <= 256) ? 256 : 512;   // power of two >= 2 accumulators of BN columns
};

// Epilogue modes
enum : int { kEpiStore = 0, kEpiAccumulate = 1 };

// Grouped rasterisation: consecutive tile ids walk kGroupM row-blocks before moving to the next column block, so
// the tiles that are in flight at any moment share a small set of A and B panels (both stay L2-resident even
// when an operand is larger than L2; measured on the 7B wgrad shape: DRAM reads 1.06 GB -> ~0.2 GB).
constexpr int kGroupM = 8;
__device__ __forceinline__ void tile_to_mn(int tile, int num_m, int num_n, int& m_blk, int& n_blk) {
  const int per_group = kGroupM * num_n;
  const int group = tile / per_group;
  const int first_m = group * kGroupM;
  const int gsize = min(num_m - first_m, kGroupM);
  const int in_group = tile - group * per_group;
  m_blk = first_m + in_group % gsize;
  n_blk = in_group / gsize;
}

// Where a warp stages its boxes: kBufs buffers in turn, or, for the last tile of a CTA, a buffer per box in the operand ring, which is
// idle by then (the accumulator is finished, so every load has landed and been read).  Nobody waits for a store there: a problem of one
// wave is nothing but last tiles, and its epilogue is exposed (2048 x 2048 x 4096: 31.6 us with two buffers, 32.8 with one and no ring).
template <int kBufs>
struct OutStage {
  uint8_t* at;
  uint32_t n;              // boxes so far
  bool last;
  __device__ __forceinline__ void begin(uint8_t* bufs, uint8_t* ring, int q, int boxes, bool last_tile) {
    last = last_tile;
    at = last ? ring + q * boxes * kOutBox : bufs + q * kBufs * kOutBox;
    if (last) n = 0;
  }
};

// One 32-row x 64-column box: `pair(e)` gives columns 2e and 2e + 1 of this lane's row, packed to bf16.
template <int kBufs, typename Pair>
__device__ __forceinline__ void stage_box(OutStage<kBufs>& out, const CUtensorMap* tm, int col0, int row0, int lane, Pair pair) {
  uint8_t* buf = out.at + (out.last ? out.n : out.n % kBufs) * kOutBox;
  ++out.n;
  if (!out.last) {
    if (lane == 0) tma_store_wait_read<kBufs - 1>();          // the store that last read this buffer is through
    __syncwarp();
  }
#pragma unroll
  for (int j = 0; j < 8; ++j)
    *reinterpret_cast<uint4*>(buf + lane * 128 + ((j ^ (lane & 7)) << 4)) = make_uint4(pair(4 * j), pair(4 * j + 1), pair(4 * j + 2), pair(4 * j + 3));
  fence_proxy_async_smem();
  __syncwarp();
  if (lane == 0) {
    tma_store_2d(tm, buf, col0, row0);
    tma_store_commit();
  }
}

// Epilogue of one tile, one warp: BN accumulator columns of 32 rows (row0 = the warp's first) -> C.
// bf16 without accumulation goes through shared memory and TMA: 64 columns at a time, each lane packs its row into the swizzled
// buffer and one lane stores the box, while the next columns are read.  A row per lane straight to global memory touches 32 lines
// per instruction: an exposed epilogue (the problem is one tile per CTA) took longer than the main loop of K = 768.
template <int BN, typename OutT>
__device__ __forceinline__ void gemm_epilogue(uint32_t t_row, OutStage<1>& out, const CUtensorMap* tmC,
                                              OutT* __restrict__ C, long long ldc, int row0, int n0, int M, int N, int beta, int lane) {
  if constexpr (sizeof(OutT) == 2) {
    if (!beta) {
#pragma unroll 1
      for (int c = 0; c < BN / 64; ++c) {
        uint32_t r[64];
        tmem_ld_x32(t_row + c * 64, r);
        tmem_ld_x32(t_row + c * 64 + 32, r + 32);
        tmem_ld_wait();
        if (row0 >= M || n0 + c * 64 >= N) continue;      // uniform over the warp
        stage_box(out, tmC, n0 + c * 64, row0, lane,
                  [&](int e) { return pack_bf16x2(__uint_as_float(r[2 * e]), __uint_as_float(r[2 * e + 1])); });
      }
      return;
    }
  }
  const int row = row0 + lane;
  OutT* crow = C + static_cast<long long>(row) * ldc + n0;
#pragma unroll 1
  for (int c = 0; c < BN / 32; ++c) {
    uint32_t r[32];
    tmem_ld_x32(t_row + c * 32, r);
    tmem_ld_wait();
    if (row < M) {
      if constexpr (sizeof(OutT) == 2) {
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          const int col = n0 + c * 32 + j * 8;
          if (col < N) {
            float f[8], old[8];
            __nv_bfloat16* dst = reinterpret_cast<__nv_bfloat16*>(crow) + c * 32 + j * 8;
            unpack8(load8(dst), old);
#pragma unroll
            for (int e = 0; e < 8; ++e) f[e] = __uint_as_float(r[j * 8 + e]) + old[e];
            store8(dst, pack8(f));
          }
        }
      } else {
#pragma unroll
        for (int j = 0; j < 8; ++j) {
          const int col = n0 + c * 32 + j * 4;
          if (col < N) {
            float4 v = make_float4(__uint_as_float(r[j * 4]), __uint_as_float(r[j * 4 + 1]),
                                   __uint_as_float(r[j * 4 + 2]), __uint_as_float(r[j * 4 + 3]));
            float4* dst = reinterpret_cast<float4*>(reinterpret_cast<float*>(crow) + c * 32 + j * 4);
            if (beta) {
              const float4 o = *dst;
              v.x += o.x; v.y += o.y; v.z += o.z; v.w += o.w;
            }
            *dst = v;
          }
        }
      }
    }
  }
}

// Gated up-projection (llmctl_gemm_swiglu_bf16): the tile's first half of columns multiplies rows of the gate matrix, the second half the
// same rows of the up matrix, and the epilogue stores silu(gate) * up, and gate and up beside it when the backward will want them.
struct SwigluMaps {
  CUtensorMap w_up, gate, up, act;
  int keep;                  // gate and up are stored
  const __nv_bfloat16* gu;   // backward: gate | up as the forward left them; `gate` and `up` take their gradients
  long long ldgu;
  // rotation (kRotate): tables [positions][32], position of each row or null (row % seq), columns that are rotated
  const float *cos, *sin;
  const int* positions;
  int seq, rotated;
};

// Rotation of heads of 64 on their way out (llmctl_gemm_rope_bf16): a chunk of 64 columns is a head, and a lane holds its row of it, halves and all.
// The product is rounded to bf16 before it is rotated, as it would be between two kernels.  The row's angles are asked for before
// the accumulator is waited for.
struct Angles {
  float c[32], s[32];
  __device__ __forceinline__ void load(const SwigluMaps& sw, int row, int M) {
    if (row >= M) return;
    const long long at = static_cast<long long>(sw.positions != nullptr ? sw.positions[row] : row % sw.seq) * 32;
#pragma unroll
    for (int i = 0; i < 32; i += 4) {
      *reinterpret_cast<float4*>(c + i) = *reinterpret_cast<const float4*>(sw.cos + at + i);
      *reinterpret_cast<float4*>(s + i) = *reinterpret_cast<const float4*>(sw.sin + at + i);
    }
  }
};
template <int BN>
__device__ __forceinline__ void rotate_epilogue(uint32_t t_row, OutStage<1>& out, const CUtensorMap* tmC, const Angles& angles, int rotated, int row0, int n0,
                                                int M, int N, int lane) {
#pragma unroll 1
  for (int c = 0; c < BN / 64; ++c) {
    uint32_t r[64];
    tmem_ld_x32(t_row + c * 64, r);
    tmem_ld_x32(t_row + c * 64 + 32, r + 32);
    tmem_ld_wait();
    const int col = n0 + c * 64;
    if (row0 >= M || col >= N) continue;               // uniform over the warp
    if (col < rotated) {
#pragma unroll
      for (int i = 0; i < 32; ++i) {
        const float a = __bfloat162float(__float2bfloat16(__uint_as_float(r[i]))), b = __bfloat162float(__float2bfloat16(__uint_as_float(r[i + 32])));
        r[i] = __float_as_uint(__fmaf_rn(a, angles.c[i], -__fmul_rn(b, angles.s[i])));            // rounded as in rope.cu
        r[i + 32] = __float_as_uint(__fmaf_rn(b, angles.c[i], __fmul_rn(a, angles.s[i])));
      }
    }
    stage_box(out, tmC, col, row0, lane, [&](int e) { return pack_bf16x2(__uint_as_float(r[2 * e]), __uint_as_float(r[2 * e + 1])); });
  }
}
template <int BN>
__device__ __forceinline__ void swiglu_epilogue(uint32_t t_row, OutStage<2>& out, const SwigluMaps& maps, int row0, int f0,
                                                int M, int F, int lane) {
#pragma unroll 1
  for (int c = 0; c < BN / 128; ++c) {
    uint32_t g[64], u[64];
    tmem_ld_x32(t_row + c * 64, g);
    tmem_ld_x32(t_row + c * 64 + 32, g + 32);
    tmem_ld_x32(t_row + BN / 2 + c * 64, u);
    tmem_ld_x32(t_row + BN / 2 + c * 64 + 32, u + 32);
    tmem_ld_wait();
    const int col = f0 + c * 64;
    if (row0 >= M || col >= F) continue;               // uniform over the warp
    auto packed = [](const uint32_t* r, int e) { return pack_bf16x2(__uint_as_float(r[2 * e]), __uint_as_float(r[2 * e + 1])); };
    if (maps.keep) {
      stage_box(out, &maps.gate, col, row0, lane, [&](int e) { return packed(g, e); });
      stage_box(out, &maps.up, col, row0, lane, [&](int e) { return packed(u, e); });
    }
    auto act = [](uint32_t gv, uint32_t uv) {          // silu first, as in swiglu.cu: x * up may overflow where silu(x) * up does not
      const float x = __uint_as_float(gv);
      return x * __fdividef(1.f, 1.f + __expf(-x)) * __uint_as_float(uv);
    };
    stage_box(out, &maps.act, col, row0, lane, [&](int e) { return pack_bf16x2(act(g[2 * e], u[2 * e]), act(g[2 * e + 1], u[2 * e + 1])); });
  }
}

// Gradient of the gated activation (llmctl_gemm_swiglu_bwd_bf16): the tile is dL/d(silu(gate) * up).  Gate and up come in whole lines, eight
// lanes to a row, one box of 64 columns ahead of its use, and turn to a row per lane in the warp's staging buffers, where their gradients
// replace them.  All of it passes beside the main loop of the next tile, which it must not outlast: read a row per lane straight from
// global memory (32 lines per load) the 4096 x 5632 x 2048 problem took 94 us, with an IEEE reciprocal on top of that 146.
template <int BN>
__device__ __forceinline__ void swiglu_bwd_epilogue(uint32_t t_row, uint8_t* out_smem, const SwigluMaps& maps, int row0, int f0, int M, int F,
                                                    int lane) {
  uint4 g[8], u[8];
  const int sub = lane >> 3, part = lane & 7;
  auto fetch = [&](int c) {
    const int col = f0 + c * 64 + part * 8;
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      const int row = row0 + 4 * i + sub;
      g[i] = u[i] = make_uint4(0u, 0u, 0u, 0u);
      if (row < M && col < F) {
        const __nv_bfloat16* src = maps.gu + static_cast<long long>(row) * maps.ldgu + col;
        g[i] = *reinterpret_cast<const uint4*>(src);
        u[i] = *reinterpret_cast<const uint4*>(src + F);
      }
    }
  };
  uint8_t *gs = out_smem, *us = out_smem + kOutBox;
  fetch(0);
#pragma unroll 1
  for (int c = 0; c < BN / 64; ++c) {
    const int col = f0 + c * 64;
    if (row0 >= M || col >= F) break;                  // uniform over the warp
    if (lane == 0) tma_store_wait_read<0>();
    __syncwarp();
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      const int row = 4 * i + sub, at = row * 128 + ((part ^ (row & 7)) << 4);
      *reinterpret_cast<uint4*>(gs + at) = g[i];
      *reinterpret_cast<uint4*>(us + at) = u[i];
    }
    __syncwarp();
    if (c + 1 < BN / 64) fetch(c + 1);
    uint32_t r[64];
    tmem_ld_x32(t_row + c * 64, r);
    tmem_ld_x32(t_row + c * 64 + 32, r + 32);
    tmem_ld_wait();
#pragma unroll
    for (int j = 0; j < 8; ++j) {
      const int at = lane * 128 + ((j ^ (lane & 7)) << 4);
      float gv[8], uv[8];
      unpack8(*reinterpret_cast<const bf16x8*>(gs + at), gv);
      unpack8(*reinterpret_cast<const bf16x8*>(us + at), uv);
#pragma unroll
      for (int e = 0; e < 8; ++e) {
        const float d = __uint_as_float(r[8 * j + e]);
        const float sig = __fdividef(1.f, 1.f + __expf(-gv[e])), silu = gv[e] * sig;
        gv[e] = d * uv[e] * (sig + silu * (1.f - sig));
        uv[e] = d * silu;
      }
      *reinterpret_cast<bf16x8*>(gs + at) = pack8(gv);
      *reinterpret_cast<bf16x8*>(us + at) = pack8(uv);
    }
    fence_proxy_async_smem();
    __syncwarp();
    if (lane == 0) {
      tma_store_2d(&maps.gate, gs, col, row0);
      tma_store_2d(&maps.up, us, col, row0);
      tma_store_commit();
    }
  }
}

template <int BN, bool A_MN, bool B_MN, typename OutT, Gated kGated = Gated::kNone>
__global__ void __launch_bounds__(kGemmThreads, 1)
gemm_tcgen05_kernel(const __grid_constant__ CUtensorMap tmA, const __grid_constant__ CUtensorMap tmB,
                    const __grid_constant__ CUtensorMap tmC, OutT* __restrict__ C, long long ldc, int M, int N, int K, int beta, const GemmGate gate,
                    const __grid_constant__ SwigluMaps sw) {
  using Cfg = GemmCfg<BN, kGated>;
  static_assert(Cfg::kSmemBytes + 1280 + (plain_output(kGated) ? 2 : 1) * kNeighbourShared <= kSmShared, "no room for the kernels beside this one");
  extern __shared__ uint8_t smem_raw[];
  __shared__ uint64_t bar_full[Cfg::kStages];
  __shared__ uint64_t bar_empty[Cfg::kStages];
  __shared__ uint64_t bar_tfull[2];
  __shared__ uint64_t bar_tempty[2];
  __shared__ uint32_t tmem_base_smem;

  const uint32_t smem_base = (smem_u32(smem_raw) + 1023u) & ~1023u;
  uint8_t* smem = smem_raw + (smem_base - smem_u32(smem_raw));
  const int warp = __shfl_sync(0xffffffffu, threadIdx.x >> 5, 0);
  const int lane = threadIdx.x & 31;

  const int num_m = (M + kBM - 1) / kBM;
  constexpr bool kSwiglu = kGated == Gated::kForward;
  constexpr int kCols = kSwiglu ? BN / 2 : BN;         // output columns per tile; with the gate N counts those of one half
  const int num_n = (N + kCols - 1) / kCols;
  const int num_tiles = num_m * num_n;
  const int num_kb = (K + kBK - 1) / kBK;

  if (threadIdx.x == 0) {
    for (int i = 0; i < Cfg::kStages; ++i) {
      mbar_init(&bar_full[i], 1);
      mbar_init(&bar_empty[i], 1);
    }
    for (int i = 0; i < 2; ++i) {
      mbar_init(&bar_tfull[i], 1);
      mbar_init(&bar_tempty[i], 4);
    }
    fence_mbar_init();
  }
  if (warp == 0 && lane == 0) {
    prefetch_tmap(&tmA);
    prefetch_tmap(&tmB);
  }
  if (warp == 1) tmem_alloc<1>(&tmem_base_smem, Cfg::kTmemCols);
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = tmem_base_smem;
  wait_for_previous(C);

  if (warp == 0) {
    // ------------------------------ TMA producer ------------------------------
    if (lane == 0) {
      int stage = 0;
      uint32_t phase = 0;
      for (int tile = blockIdx.x; tile < num_tiles; tile += gridDim.x) {
        int mb_, nb_;
        tile_to_mn(tile, num_m, num_n, mb_, nb_);
        mb_ = gate_perm(gate, mb_);
        const int m0 = mb_ * kBM;
        const int n0 = nb_ * kCols;
        const int b_row = grouped_b_row(gate, mb_, n0, N);
        if (b_row < 0) continue;
        gate_wait(gate, m0, min(m0 + kBM, M));
        gate_wait_b<B_MN>(gate, n0, min(n0 + BN, N));
        for (int kb = 0; kb < num_kb; ++kb) {
          mbar_wait(&bar_empty[stage], phase ^ 1u);
          uint8_t* sA = smem + stage * Cfg::kStageBytes;
          uint8_t* sB = sA + Cfg::kABytes;
          mbar_expect_tx(&bar_full[stage], Cfg::kStageBytes);
          const int k0 = kb * kBK;
          if (!A_MN) {
            tma_load_2d(sA, &tmA, &bar_full[stage], k0, m0);
          } else {
#pragma unroll
            for (int g = 0; g < kBM / 64; ++g)
              tma_load_2d(sA + g * 8192, &tmA, &bar_full[stage], m0 + g * 64, k0);
          }
          if (kSwiglu) {
            tma_load_2d(sB, &tmB, &bar_full[stage], k0, n0);
            tma_load_2d(sB + Cfg::kBBytes / 2, &sw.w_up, &bar_full[stage], k0, n0);
          } else if (!B_MN) {
            tma_load_2d(sB, &tmB, &bar_full[stage], k0, b_row);
          } else {
#pragma unroll
            for (int g = 0; g < BN / 64; ++g)
              tma_load_2d(sB + g * 8192, &tmB, &bar_full[stage], n0 + g * 64, k0);
          }
          if (++stage == Cfg::kStages) {
            stage = 0;
            phase ^= 1u;
          }
        }
      }
      if (!gate.waits()) release_dependents();       // the last loads are on their way
    }
  } else if (warp == 1) {
    // ------------------------------ MMA issuer ------------------------------
    // The whole warp walks the loop, one elected lane issues: stage addresses and descriptors stay in uniform registers, which
    // the instruction reads.  From a single lane's branch a product took 85-107 clocks to issue, more than a 128-wide tile's 64.
    constexpr uint32_t idesc = make_idesc_bf16(kBM, BN, A_MN ? 1u : 0u, B_MN ? 1u : 0u);
    int stage = 0;
    uint32_t phase = 0;
    int acc = 0;
    uint32_t aphase = 0;
    for (int tile = blockIdx.x; tile < num_tiles; tile += gridDim.x) {
      if (gate.grp_tile_expert != nullptr) {
        int mb_, nb_;
        tile_to_mn(tile, num_m, num_n, mb_, nb_);
        if (grouped_b_row(gate, mb_, 0, N) < 0) continue;
      }
      mbar_wait(&bar_tempty[acc], aphase ^ 1u);
      __syncwarp();
      tc_fence_after();
      const uint32_t d_tmem = tmem_base + static_cast<uint32_t>(acc * BN);
      for (int kb = 0; kb < num_kb; ++kb) {
        mbar_wait(&bar_full[stage], phase);
        __syncwarp();
        tc_fence_after();
        const uint32_t a_addr = smem_base + stage * Cfg::kStageBytes;
        const uint64_t da = A_MN ? make_smem_desc(a_addr, 8192, 1024, 2) : make_smem_desc(a_addr, 16, 1024, 2);
        const uint64_t db = B_MN ? make_smem_desc(a_addr + Cfg::kABytes, 8192, 1024, 2) : make_smem_desc(a_addr + Cfg::kABytes, 16, 1024, 2);
        if (elect_one()) {
#pragma unroll
          for (int k = 0; k < kBK / 16; ++k)
            umma_ss<1>(d_tmem, da + ((A_MN ? k * 2048 : k * 32) >> 4), db + ((B_MN ? k * 2048 : k * 32) >> 4), idesc, (kb | k) != 0 ? 1u : 0u);
          umma_commit<1>(&bar_empty[stage]);  // frees the smem slot once these MMAs retire
          if (kb + 1 == num_kb) umma_commit<1>(&bar_tfull[acc]);  // accumulator complete -> epilogue
        }
        if (++stage == Cfg::kStages) {
          stage = 0;
          phase ^= 1u;
        }
      }
      acc ^= 1;
      if (acc == 0) aphase ^= 1u;
    }
  } else {
    // ------------------------------ epilogue (4 warps) ------------------------------
    const int q = warp & 3;  // TMEM lane quadrant this warp may access
    OutStage<out_bufs(kGated)> out{nullptr, 0u, false};
    int acc = 0;
    uint32_t aphase = 0;
    for (int tile = blockIdx.x; tile < num_tiles; tile += gridDim.x) {
      int mb_, nb_;
      tile_to_mn(tile, num_m, num_n, mb_, nb_);
      mb_ = gate_perm(gate, mb_);
      const int m0 = mb_ * kBM;
      const int n0 = nb_ * kCols;
      if (grouped_b_row(gate, mb_, n0, N) < 0) continue;
      [[maybe_unused]] Angles angles;
      if constexpr (kGated == Gated::kRotate) angles.load(sw, m0 + q * 32 + lane, M);
      mbar_wait(&bar_tfull[acc], aphase);
      tc_fence_after();
      const uint32_t t_row = tmem_base + (static_cast<uint32_t>(q * 32) << 16) + static_cast<uint32_t>(acc * BN);
      out.begin(smem + Cfg::kOutAt, smem, q, BN / 64, plain_output(kGated) && tile + static_cast<int>(gridDim.x) >= num_tiles);
      if constexpr (kSwiglu)
        swiglu_epilogue<BN>(t_row, out, sw, m0 + q * 32, n0, M, N, lane);
      else if constexpr (kGated == Gated::kBackward)
        swiglu_bwd_epilogue<BN>(t_row, out.at, sw, m0 + q * 32, n0, M, N, lane);
      else if constexpr (kGated == Gated::kRotate)
        rotate_epilogue<BN>(t_row, out, &tmC, angles, sw.rotated, m0 + q * 32, n0, M, N, lane);
      else
        gemm_epilogue<BN, OutT>(t_row, out, &tmC, C, ldc, m0 + q * 32, n0, M, N, beta, lane);
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(&bar_tempty[acc]);
      acc ^= 1;
      if (acc == 0) aphase ^= 1u;
    }
    if (lane == 0) tma_store_wait_read<0>();      // the staging buffers are read before the CTA gives them back
  }

  tc_fence_before();
  __syncthreads();
  if (warp == 1) {
    tc_fence_after();
    tmem_dealloc<1>(tmem_base, Cfg::kTmemCols);
  }
}


// ================================================================================================
// 2-CTA variant (cta_group::2): a CTA pair (cluster of 2, same TPC) computes one 256 x 256 tile.
// CTA r stages A rows [m0 + 128 r, +128) and B rows (N) [n0 + 128 r, +128); the leader CTA issues
// UMMA 256 x 256 x 16 which reads both CTAs' shared memory, so each SM moves only half of B through
// its own shared memory (smem traffic per SM: 64 KB/stage-pair instead of 96 KB) — this is what lets
// the tensor pipe stay fed.  Each CTA's TMEM holds its own 128 accumulator rows.
//   full[s]   (leader only): 1 arrive (leader producer expect_tx of BOTH CTAs' bytes) + tx bytes
//   empty[s]  (both CTAs)  : tcgen05.commit multicast from the leader
//   tfull[a]  (both CTAs)  : tcgen05.commit multicast from the leader
//   tempty[a] (leader only): 8 arrives = 4 epilogue warps x 2 CTAs (peer arrives remotely)
// ================================================================================================
// PBN = N of the pair tile: 256 (the throughput tile) or 128 (half the work per tile: fills the last wave of the
// 1-3 wave problems of a TP=8 shard, where a 256 x 256 tile is 26 us of tensor-core time).
template <int PBN, Gated kGated = Gated::kNone>
struct Gemm2Cfg {
  static constexpr int kBN = PBN;
  static constexpr int kStages = (PBN == 256) ? 6 : 8;
  static constexpr int kABytes = kBM * kBK * 2;          // 128 x 64 per CTA
  static constexpr int kBBytes = (kBN / 2) * kBK * 2;    // (PBN/2) x 64 per CTA
  static constexpr int kStageBytes = kABytes + kBBytes;  // 32 / 24 KB per CTA
  static constexpr int kOutAt = kStages * kStageBytes;
  static constexpr int kSmemBytes = kOutAt + 4 * out_bufs(kGated) * kOutBox + 1024;
  static constexpr int kTmemCols = 2 * PBN;              // 512 / 256
};

template <int PBN, bool A_MN, bool B_MN, typename OutT, Gated kGated = Gated::kNone>
__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(kGemmThreads, 1)
gemm2_tcgen05_kernel(const __grid_constant__ CUtensorMap tmA, const __grid_constant__ CUtensorMap tmB,
                     const __grid_constant__ CUtensorMap tmC, OutT* __restrict__ C, long long ldc, int M, int N, int K, int beta, const GemmGate gate,
                    const __grid_constant__ SwigluMaps sw) {
  using Cfg = Gemm2Cfg<PBN, kGated>;
  static_assert(Cfg::kSmemBytes + 1280 + (plain_output(kGated) ? 2 : 1) * kNeighbourShared <= kSmShared, "no room for the kernels beside this one");
  constexpr int BN = Cfg::kBN;
  extern __shared__ uint8_t smem_raw[];
  __shared__ uint64_t bar_full[Cfg::kStages];
  __shared__ uint64_t bar_empty[Cfg::kStages];
  __shared__ uint64_t bar_tfull[2];
  __shared__ uint64_t bar_tempty[2];
  __shared__ uint32_t tmem_base_smem;

  const uint32_t smem_base = (smem_u32(smem_raw) + 1023u) & ~1023u;
  uint8_t* smem = smem_raw + (smem_base - smem_u32(smem_raw));
  const int warp = __shfl_sync(0xffffffffu, threadIdx.x >> 5, 0);
  const int lane = threadIdx.x & 31;
  const uint32_t cta_rank = cluster_ctarank();   // 0 = leader
  const int pair = blockIdx.x >> 1;
  const int num_pairs = gridDim.x >> 1;

  const int num_m = (M + 2 * kBM - 1) / (2 * kBM);
  constexpr bool kSwiglu = kGated == Gated::kForward;
  constexpr int kCols = kSwiglu ? BN / 2 : BN;         // output columns per tile; with the gate N counts those of one half
  const int num_n = (N + kCols - 1) / kCols;
  const int num_tiles = num_m * num_n;
  const int num_kb = (K + kBK - 1) / kBK;

  if (threadIdx.x == 0) {
    for (int i = 0; i < Cfg::kStages; ++i) {
      mbar_init(&bar_full[i], 1);
      mbar_init(&bar_empty[i], 1);
    }
    for (int i = 0; i < 2; ++i) {
      mbar_init(&bar_tfull[i], 1);
      mbar_init(&bar_tempty[i], 8);
    }
    fence_mbar_init();
  }
  if (warp == 0 && lane == 0) {
    prefetch_tmap(&tmA);
    prefetch_tmap(&tmB);
  }
  cluster_sync();   // barrier inits visible to the peer before any remote arrive / multicast commit
  if (warp == 1) tmem_alloc<2>(&tmem_base_smem, Cfg::kTmemCols);
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = tmem_base_smem;
  wait_for_previous(C);

  if (warp == 0) {
    // ------------------------------ TMA producer (both CTAs) ------------------------------
    if (lane == 0) {
      int stage = 0;
      uint32_t phase = 0;
      for (int tile = pair; tile < num_tiles; tile += num_pairs) {
        int mb_, nb_;
        tile_to_mn(tile, num_m, num_n, mb_, nb_);
        mb_ = gate_perm(gate, mb_);
        const int m0 = mb_ * (2 * kBM) + static_cast<int>(cta_rank) * kBM;
        const int n0 = kSwiglu ? nb_ * kCols : nb_ * BN + static_cast<int>(cta_rank) * (BN / 2);
        if (m0 < M) gate_wait(gate, m0, min(m0 + kBM, M));
        gate_wait_b<B_MN>(gate, n0, min(n0 + BN / 2, N));
        for (int kb = 0; kb < num_kb; ++kb) {
          mbar_wait(&bar_empty[stage], phase ^ 1u);
          uint8_t* sA = smem + stage * Cfg::kStageBytes;
          uint8_t* sB = sA + Cfg::kABytes;
          // all bytes of the pair are accounted on the leader's barrier
          const uint32_t full_leader = mapa_u32(smem_u32(&bar_full[stage]), 0);
          if (cta_rank == 0) mbar_expect_tx(&bar_full[stage], 2 * Cfg::kStageBytes);
          const int k0 = kb * kBK;
          if (!A_MN) {
            tma_load_2d_cg2(sA, &tmA, full_leader, k0, m0);
          } else {
#pragma unroll
            for (int g = 0; g < kBM / 64; ++g)
              tma_load_2d_cg2(sA + g * 8192, &tmA, full_leader, m0 + g * 64, k0);
          }
          if (!B_MN) {
            tma_load_2d_cg2(sB, kSwiglu && cta_rank == 1 ? &sw.w_up : &tmB, full_leader, k0, n0);
          } else {
#pragma unroll
            for (int g = 0; g < (BN / 2) / 64; ++g)
              tma_load_2d_cg2(sB + g * 8192, &tmB, full_leader, n0 + g * 64, k0);
          }
          if (++stage == Cfg::kStages) {
            stage = 0;
            phase ^= 1u;
          }
        }
      }
      if (!gate.waits()) release_dependents();       // the last loads are on their way
    }
  } else if (warp == 1) {
    // ------------------------------ MMA issuer (leader CTA only) ------------------------------
    if (cta_rank == 0) {
      constexpr uint32_t idesc = make_idesc_bf16(2 * kBM, BN, A_MN ? 1u : 0u, B_MN ? 1u : 0u);
      int stage = 0;
      uint32_t phase = 0;
      int acc = 0;
      uint32_t aphase = 0;
      for (int tile = pair; tile < num_tiles; tile += num_pairs) {
        mbar_wait(&bar_tempty[acc], aphase ^ 1u);
        __syncwarp();
        tc_fence_after();
        const uint32_t d_tmem = tmem_base + static_cast<uint32_t>(acc * BN);
        for (int kb = 0; kb < num_kb; ++kb) {
          mbar_wait(&bar_full[stage], phase);
          __syncwarp();
          tc_fence_after();
          const uint32_t a_addr = smem_base + stage * Cfg::kStageBytes;
          const uint64_t da = A_MN ? make_smem_desc(a_addr, 8192, 1024, 2) : make_smem_desc(a_addr, 16, 1024, 2);
          const uint64_t db = B_MN ? make_smem_desc(a_addr + Cfg::kABytes, 8192, 1024, 2) : make_smem_desc(a_addr + Cfg::kABytes, 16, 1024, 2);
          if (elect_one()) {
#pragma unroll
            for (int k = 0; k < kBK / 16; ++k)
              umma_ss<2>(d_tmem, da + ((A_MN ? k * 2048 : k * 32) >> 4), db + ((B_MN ? k * 2048 : k * 32) >> 4), idesc, (kb | k) != 0 ? 1u : 0u);
            umma_commit_mc2(&bar_empty[stage], 0x3);   // both CTAs' slots are free once these retire
            if (kb + 1 == num_kb) umma_commit_mc2(&bar_tfull[acc], 0x3);
          }
          if (++stage == Cfg::kStages) {
            stage = 0;
            phase ^= 1u;
          }
        }
        acc ^= 1;
        if (acc == 0) aphase ^= 1u;
      }
    }
  } else {
    // ------------------------------ epilogue (4 warps, both CTAs) ------------------------------
    const int q = warp & 3;
    OutStage<out_bufs(kGated)> out{nullptr, 0u, false};
    int acc = 0;
    uint32_t aphase = 0;
    for (int tile = pair; tile < num_tiles; tile += num_pairs) {
      int mb_, nb_;
      tile_to_mn(tile, num_m, num_n, mb_, nb_);
      mb_ = gate_perm(gate, mb_);
      const int m0 = mb_ * (2 * kBM) + static_cast<int>(cta_rank) * kBM;
      const int n0 = nb_ * kCols;
      [[maybe_unused]] Angles angles;
      if constexpr (kGated == Gated::kRotate) angles.load(sw, m0 + q * 32 + lane, M);
      mbar_wait(&bar_tfull[acc], aphase);
      tc_fence_after();
      const uint32_t t_row = tmem_base + (static_cast<uint32_t>(q * 32) << 16) + static_cast<uint32_t>(acc * BN);
      out.begin(smem + Cfg::kOutAt, smem, q, BN / 64, plain_output(kGated) && tile + num_pairs >= num_tiles);
      if constexpr (kSwiglu)
        swiglu_epilogue<BN>(t_row, out, sw, m0 + q * 32, n0, M, N, lane);
      else if constexpr (kGated == Gated::kBackward)
        swiglu_bwd_epilogue<BN>(t_row, out.at, sw, m0 + q * 32, n0, M, N, lane);
      else if constexpr (kGated == Gated::kRotate)
        rotate_epilogue<BN>(t_row, out, &tmC, angles, sw.rotated, m0 + q * 32, n0, M, N, lane);
      else
        gemm_epilogue<BN, OutT>(t_row, out, &tmC, C, ldc, m0 + q * 32, n0, M, N, beta, lane);
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive_cluster(&bar_tempty[acc], 0);   // always the leader's barrier
      acc ^= 1;
      if (acc == 0) aphase ^= 1u;
    }
    if (lane == 0) tma_store_wait_read<0>();
  }

  tc_fence_before();
  cluster_sync();   // the leader's MMAs read the peer's smem: nobody leaves before everything retired
  if (warp == 1) {
    tc_fence_after();
    tmem_dealloc<2>(tmem_base, Cfg::kTmemCols);
  }
}

// ================================================================================================
// Split K: a cluster of `splits` CTAs computes one 128 x 64 tile, each over its share of the k-blocks, and each sums and stores its share of the
// columns: the others' partial sums come into its shared memory (distributed shared memory, over the operand ring, which is idle by
// then) and are added in the order of the ranks.  For problems with fewer tiles than SMs, which a CTA that walks all of K alone leaves waiting:
// the products of a few rows with a vocabulary's or an MLP's long side.
// ================================================================================================
constexpr int kSplitBN = 64, kMaxSplits = 8;
template <int kStages>
struct SplitCfg {
  static constexpr int kABytes = kBM * kBK * 2, kStageBytes = kABytes + kSplitBN * kBK * 2;
  static constexpr int kSmemBytes = kStages * kStageBytes + 1024;
};
// Columns go to the CTAs in units of 8.
__device__ __forceinline__ int first_unit(int rank, int splits) { return kSplitBN / 8 * rank / splits; }
__device__ __forceinline__ int unit_owner(int u, int splits) { return ((u + 1) * splits - 1) / (kSplitBN / 8); }

template <int kStages, bool A_MN, bool B_MN, typename OutT>
__global__ void __launch_bounds__(kGemmThreads, kStages <= 4 ? 2 : 1)
gemm_split_kernel(const __grid_constant__ CUtensorMap tmA, const __grid_constant__ CUtensorMap tmB, OutT* __restrict__ C, long long ldc, int M, int N, int K,
                  int beta, int splits) {
  using Cfg = SplitCfg<kStages>;
  extern __shared__ uint8_t smem_raw[];
  __shared__ uint64_t bar_full[kStages], bar_empty[kStages], bar_done;
  __shared__ uint32_t tmem_base_smem;
  const uint32_t smem_base = (smem_u32(smem_raw) + 1023u) & ~1023u;
  uint8_t* smem = smem_raw + (smem_base - smem_u32(smem_raw));
  const int warp = __shfl_sync(0xffffffffu, threadIdx.x >> 5, 0), lane = threadIdx.x & 31;
  const int rank = static_cast<int>(cluster_ctarank()), tile = blockIdx.x / splits;
  const int num_m = (M + kBM - 1) / kBM, num_n = (N + kSplitBN - 1) / kSplitBN, num_kb = (K + kBK - 1) / kBK;
  int m_blk, n_blk;
  tile_to_mn(tile, num_m, num_n, m_blk, n_blk);
  const int m0 = m_blk * kBM, n0 = n_blk * kSplitBN;
  const int kb0 = static_cast<int>(static_cast<long long>(num_kb) * rank / splits), kb1 = static_cast<int>(static_cast<long long>(num_kb) * (rank + 1) / splits);

  if (threadIdx.x == 0) {
    for (int i = 0; i < kStages; ++i) {
      mbar_init(&bar_full[i], 1);
      mbar_init(&bar_empty[i], 1);
    }
    mbar_init(&bar_done, 1);
    fence_mbar_init();
    prefetch_tmap(&tmA);
    prefetch_tmap(&tmB);
  }
  if (warp == 1) tmem_alloc<1>(&tmem_base_smem, kSplitBN);
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = tmem_base_smem;
  wait_for_previous(C);
  float acc[kSplitBN];
  if (warp == 0) {
    if (lane == 0) {
      for (int kb = kb0, i = 0; kb < kb1; ++kb, ++i) {
        const int stage = i % kStages;
        mbar_wait(&bar_empty[stage], ((i / kStages) & 1u) ^ 1u);
        uint8_t *sA = smem + stage * Cfg::kStageBytes, *sB = sA + Cfg::kABytes;
        mbar_expect_tx(&bar_full[stage], Cfg::kStageBytes);
        const int k0 = kb * kBK;
        if (!A_MN) {
          tma_load_2d(sA, &tmA, &bar_full[stage], k0, m0);
        } else {
          tma_load_2d(sA, &tmA, &bar_full[stage], m0, k0);
          tma_load_2d(sA + 8192, &tmA, &bar_full[stage], m0 + 64, k0);
        }
        if (!B_MN) tma_load_2d(sB, &tmB, &bar_full[stage], k0, n0); else tma_load_2d(sB, &tmB, &bar_full[stage], n0, k0);
      }
      release_dependents();
    }
    __syncwarp();
  } else if (warp == 1) {
    constexpr uint32_t idesc = make_idesc_bf16(kBM, kSplitBN, A_MN ? 1u : 0u, B_MN ? 1u : 0u);
    int stage = 0;
    uint32_t phase = 0;
    for (int kb = kb0; kb < kb1; ++kb) {
      mbar_wait(&bar_full[stage], phase);
      __syncwarp();
      tc_fence_after();
      const uint32_t a_addr = smem_base + stage * Cfg::kStageBytes;
      const uint64_t da = A_MN ? make_smem_desc(a_addr, 8192, 1024, 2) : make_smem_desc(a_addr, 16, 1024, 2);
      const uint64_t db = B_MN ? make_smem_desc(a_addr + Cfg::kABytes, 8192, 1024, 2) : make_smem_desc(a_addr + Cfg::kABytes, 16, 1024, 2);
      if (elect_one()) {
#pragma unroll
        for (int k = 0; k < kBK / 16; ++k)
          umma_ss<1>(tmem_base, da + ((A_MN ? k * 2048 : k * 32) >> 4), db + ((B_MN ? k * 2048 : k * 32) >> 4), idesc, (kb != kb0 || k != 0) ? 1u : 0u);
        umma_commit<1>(&bar_empty[stage]);
        if (kb + 1 == kb1) umma_commit<1>(&bar_done);
      }
      if (++stage == kStages) {
        stage = 0;
        phase ^= 1u;
      }
    }
    __syncwarp();
  } else {
    mbar_wait(&bar_done, 0u);
    __syncwarp();
    tc_fence_after();
    uint32_t r[kSplitBN];
    const uint32_t t_row = tmem_base + (static_cast<uint32_t>((warp & 3) * 32) << 16);
    tmem_ld_x32(t_row, r);
    tmem_ld_x32(t_row + 32, r + 32);
    tmem_ld_wait();
#pragma unroll
    for (int i = 0; i < kSplitBN; ++i) acc[i] = __uint_as_float(r[i]);
  }
  const int row = (warp & 3) * 32 + lane;
  cluster_sync();                      // every CTA's loads have landed and been multiplied: the rings may be written over
  if (warp >= 2) {
#pragma unroll
    for (int u = 0; u < kSplitBN / 8; ++u) {
      const int to = unit_owner(u, splits), first = first_unit(to, splits), width = (first_unit(to + 1, splits) - first) * 8;
      const uint32_t at = mapa_u32(smem_base + ((rank * kBM + row) * width + (u - first) * 8) * 4, to);
      st_cluster_v4(at, make_float4(acc[8 * u], acc[8 * u + 1], acc[8 * u + 2], acc[8 * u + 3]));
      st_cluster_v4(at + 16, make_float4(acc[8 * u + 4], acc[8 * u + 5], acc[8 * u + 6], acc[8 * u + 7]));
    }
  }
  cluster_sync();
  if (warp >= 2 && m0 + row < M) {
    const int first = first_unit(rank, splits), last = first_unit(rank + 1, splits), width = (last - first) * 8;
    const float* mine = reinterpret_cast<const float*>(smem) + row * width;
    for (int u = first; u < last; ++u) {
      const int col = n0 + u * 8;
      if (col >= N) break;
      float f[8] = {};
      for (int src = 0; src < splits; ++src) {
        const float4* p = reinterpret_cast<const float4*>(mine + src * kBM * width + (u - first) * 8);
        const float4 x = p[0], y = p[1];
        f[0] += x.x; f[1] += x.y; f[2] += x.z; f[3] += x.w;
        f[4] += y.x; f[5] += y.y; f[6] += y.z; f[7] += y.w;
      }
      OutT* dst = C + static_cast<long long>(m0 + row) * ldc + col;
      if constexpr (sizeof(OutT) == 2) {
        if (beta) {
          float old[8];
          unpack8(load8(dst), old);
#pragma unroll
          for (int e = 0; e < 8; ++e) f[e] += old[e];
        }
        store8(dst, pack8(f));
      } else {
        float4* to = reinterpret_cast<float4*>(dst);
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          float4 v = make_float4(f[4 * h], f[4 * h + 1], f[4 * h + 2], f[4 * h + 3]);
          if (beta) {
            const float4 o = to[h];
            v.x += o.x; v.y += o.y; v.z += o.z; v.w += o.w;
          }
          to[h] = v;
        }
      }
    }
  }
  tc_fence_before();
  __syncthreads();
  if (warp == 1) {
    tc_fence_after();
    tmem_dealloc<1>(tmem_base, kSplitBN);
  }
}

static int g_num_sms = 0;
static int num_sms() {
  if (g_num_sms == 0) {
    int dev = 0, n = 0;
    if (cudaGetDevice(&dev) == cudaSuccess &&
        cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev) == cudaSuccess && n > 0)
      g_num_sms = n;
    else
      g_num_sms = kNumSMs;
  }
  return g_num_sms;
}

// A GEMM that waits for flags of other streams' kernels is launched, and lets others be launched, the ordinary way (dependent.cuh, rule 3).
template <typename Kernel, typename OutT>
static cudaError_t launch_gemm_kernel(Kernel kern, int grid, int smem, cudaStream_t s, const CUtensorMap& tmA, const CUtensorMap& tmB, const CUtensorMap& tmC, OutT* C,
                                      long long ldc, int M, int N, int K, int beta, const GemmGate& gate, const SwigluMaps& sw) {
  if (!gate.waits()) return launch_dependent(kern, grid, kGemmThreads, smem, s, tmA, tmB, tmC, C, ldc, M, N, K, beta, gate, sw);
  kern<<<grid, kGemmThreads, smem, s>>>(tmA, tmB, tmC, C, ldc, M, N, K, beta, gate, sw);
  return cudaGetLastError();
}

template <int BN, bool A_MN, bool B_MN, typename OutT>
static int launch_gemm(const void* A, const void* B, void* C, int M, int N, int K, long long lda,
                       long long ldb, long long ldc, int beta, int max_ctas, cudaStream_t s, GemmGate gate) {
  if (gate.flags) {   // tile-row permutation needs whole tile blocks per chunk and per slab
    gate.bpc = (M / gate.world) / kBM;
    gate.bps = gate.rows_per_flag / kBM;
    gate.perm = (gate.perm && (M / gate.world) % kBM == 0 && gate.rows_per_flag % kBM == 0 && M % gate.world == 0) ? 1 : 0;
  }
  using Cfg = GemmCfg<BN>;
  CUtensorMap tmA, tmB;
  int rc;
  if (!A_MN) rc = get_tmap_2d_bf16(&tmA, A, M, K, lda, kBM, kBK, 1);
  else rc = get_tmap_2d_bf16(&tmA, A, K, M, lda, kBK, 64, 1);
  if (rc) LLMCTL_FAIL(rc, "tensor map A");
  if (!B_MN) rc = get_tmap_2d_bf16(&tmB, B, static_cast<uint64_t>(N) * (gate.grp_tile_expert ? gate.grp_experts : 1), K, ldb, BN, kBK, 1);
  else rc = get_tmap_2d_bf16(&tmB, B, K, N, ldb, kBK, 64, 1);
  if (rc) LLMCTL_FAIL(rc, "tensor map B");
  CUtensorMap tmC = tmA;                 // read only by the bf16 epilogue without accumulation
  if (sizeof(OutT) == 2 && !beta) rc = get_tmap_2d_bf16(&tmC, C, M, N, ldc, 32, 64, 1);
  if (rc) LLMCTL_FAIL(rc, "tensor map C");
  auto kern = gemm_tcgen05_kernel<BN, A_MN, B_MN, OutT>;
  LLMCTL_CHECK(allow_smem(kern, Cfg::kSmemBytes));
  const int tiles = ((M + kBM - 1) / kBM) * ((N + BN - 1) / BN);
  int grid = num_sms();
  if (max_ctas > 0 && max_ctas < grid) grid = max_ctas;
  if (tiles < grid) grid = tiles;
  LLMCTL_CHECK(launch_gemm_kernel(kern, grid, Cfg::kSmemBytes, s, tmA, tmB, tmC, (OutT*)C, ldc, M, N, K, beta, gate, SwigluMaps{}));
  LLMCTL_RETURN_LAST();
}

template <int BN, typename OutT>
static int dispatch_layout(int a_mn, int b_mn, const void* A, const void* B, void* C, int M, int N,
                           int K, long long lda, long long ldb, long long ldc, int beta,
                           int max_ctas, cudaStream_t s, const GemmGate& g) {
  if (!a_mn && !b_mn) return launch_gemm<BN, false, false, OutT>(A, B, C, M, N, K, lda, ldb, ldc, beta, max_ctas, s, g);
  if (!a_mn && b_mn) return launch_gemm<BN, false, true, OutT>(A, B, C, M, N, K, lda, ldb, ldc, beta, max_ctas, s, g);
  if (a_mn && !b_mn) return launch_gemm<BN, true, false, OutT>(A, B, C, M, N, K, lda, ldb, ldc, beta, max_ctas, s, g);
  return launch_gemm<BN, true, true, OutT>(A, B, C, M, N, K, lda, ldb, ldc, beta, max_ctas, s, g);
}


template <int kStages, bool A_MN, bool B_MN, typename OutT>
static int launch_split_stages(const CUtensorMap& tmA, const CUtensorMap& tmB, void* C, int M, int N, int K, long long ldc, int beta, int tiles, int splits,
                               cudaStream_t s) {
  auto kern = gemm_split_kernel<kStages, A_MN, B_MN, OutT>;
  LLMCTL_CHECK(allow_smem(kern, SplitCfg<kStages>::kSmemBytes));
  cudaLaunchAttribute at[2];
  at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at[0].val.programmaticStreamSerializationAllowed = 1;
  at[1].id = cudaLaunchAttributeClusterDimension;
  at[1].val.clusterDim = {static_cast<unsigned>(splits), 1, 1};
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = tiles * splits;
  cfg.blockDim = kGemmThreads;
  cfg.dynamicSmemBytes = SplitCfg<kStages>::kSmemBytes;
  cfg.stream = s;
  cfg.attrs = at;
  cfg.numAttrs = 2;
  LLMCTL_CHECK(cudaLaunchKernelEx(&cfg, kern, tmA, tmB, (OutT*)C, ldc, M, N, K, beta, splits));
  LLMCTL_RETURN_LAST();
}
template <bool A_MN, bool B_MN, typename OutT>
static int launch_split(const void* A, const void* B, void* C, int M, int N, int K, long long lda, long long ldb, long long ldc, int beta, int splits,
                        cudaStream_t s) {
  CUtensorMap tmA, tmB;
  int rc = A_MN ? get_tmap_2d_bf16(&tmA, A, K, M, lda, kBK, 64, 1) : get_tmap_2d_bf16(&tmA, A, M, K, lda, kBM, kBK, 1);
  if (!rc) rc = B_MN ? get_tmap_2d_bf16(&tmB, B, K, N, ldb, kBK, 64, 1) : get_tmap_2d_bf16(&tmB, B, N, K, ldb, kSplitBN, kBK, 1);
  if (rc) LLMCTL_FAIL(rc, "tensor maps");
  const int tiles = ((M + kBM - 1) / kBM) * ((N + kSplitBN - 1) / kSplitBN);
  // one CTA to an SM has all of its shared memory for loads in flight; beyond one wave two share it
  return tiles * splits <= num_sms() ? launch_split_stages<8, A_MN, B_MN, OutT>(tmA, tmB, C, M, N, K, ldc, beta, tiles, splits, s)
                                     : launch_split_stages<4, A_MN, B_MN, OutT>(tmA, tmB, C, M, N, K, ldc, beta, tiles, splits, s);
}
template <typename OutT>
static int dispatch_split(int a_mn, int b_mn, const void* A, const void* B, void* C, int M, int N, int K, long long lda, long long ldb, long long ldc, int beta,
                          int splits, cudaStream_t s) {
  if (!a_mn && !b_mn) return launch_split<false, false, OutT>(A, B, C, M, N, K, lda, ldb, ldc, beta, splits, s);
  if (!a_mn && b_mn) return launch_split<false, true, OutT>(A, B, C, M, N, K, lda, ldb, ldc, beta, splits, s);
  if (a_mn && !b_mn) return launch_split<true, false, OutT>(A, B, C, M, N, K, lda, ldb, ldc, beta, splits, s);
  return launch_split<true, true, OutT>(A, B, C, M, N, K, lda, ldb, ldc, beta, splits, s);
}

template <int PBN, bool A_MN, bool B_MN, typename OutT>
static int launch_gemm2(const void* A, const void* B, void* C, int M, int N, int K, long long lda,
                        long long ldb, long long ldc, int beta, int max_ctas, cudaStream_t s, GemmGate gate) {
  if (gate.flags) {
    gate.bpc = (M / gate.world) / (2 * kBM);
    gate.bps = gate.rows_per_flag / (2 * kBM);
    gate.perm = (gate.perm && (M / gate.world) % (2 * kBM) == 0 && gate.rows_per_flag % (2 * kBM) == 0 &&
                 M % gate.world == 0) ? 1 : 0;
  }
  using Cfg = Gemm2Cfg<PBN>;
  CUtensorMap tmA, tmB;
  int rc;
  if (!A_MN) rc = get_tmap_2d_bf16(&tmA, A, M, K, lda, kBM, kBK, 1);
  else rc = get_tmap_2d_bf16(&tmA, A, K, M, lda, kBK, 64, 1);
  if (rc) LLMCTL_FAIL(rc, "tensor map A");
  if (!B_MN) rc = get_tmap_2d_bf16(&tmB, B, N, K, ldb, Cfg::kBN / 2, kBK, 1);
  else rc = get_tmap_2d_bf16(&tmB, B, K, N, ldb, kBK, 64, 1);
  if (rc) LLMCTL_FAIL(rc, "tensor map B");
  CUtensorMap tmC = tmA;
  if (sizeof(OutT) == 2 && !beta) rc = get_tmap_2d_bf16(&tmC, C, M, N, ldc, 32, 64, 1);
  if (rc) LLMCTL_FAIL(rc, "tensor map C");
  auto kern = gemm2_tcgen05_kernel<PBN, A_MN, B_MN, OutT>;
  LLMCTL_CHECK(allow_smem(kern, Cfg::kSmemBytes));
  const int tiles = ((M + 2 * kBM - 1) / (2 * kBM)) * ((N + Cfg::kBN - 1) / Cfg::kBN);
  int pairs = num_sms() / 2;
  if (max_ctas > 0 && max_ctas / 2 < pairs) pairs = max_ctas / 2;
  if (pairs < 1) pairs = 1;
  if (tiles < pairs) pairs = tiles;
  LLMCTL_CHECK(launch_gemm_kernel(kern, 2 * pairs, Cfg::kSmemBytes, s, tmA, tmB, tmC, (OutT*)C, ldc, M, N, K, beta, gate, SwigluMaps{}));
  LLMCTL_RETURN_LAST();
}

template <int PBN, typename OutT>
static int dispatch_layout2(int a_mn, int b_mn, const void* A, const void* B, void* C, int M, int N,
                            int K, long long lda, long long ldb, long long ldc, int beta,
                            int max_ctas, cudaStream_t s, const GemmGate& g) {
  if (!a_mn && !b_mn) return launch_gemm2<PBN, false, false, OutT>(A, B, C, M, N, K, lda, ldb, ldc, beta, max_ctas, s, g);
  if (!a_mn && b_mn) return launch_gemm2<PBN, false, true, OutT>(A, B, C, M, N, K, lda, ldb, ldc, beta, max_ctas, s, g);
  if (a_mn && !b_mn) return launch_gemm2<PBN, true, false, OutT>(A, B, C, M, N, K, lda, ldb, ldc, beta, max_ctas, s, g);
  return launch_gemm2<PBN, true, true, OutT>(A, B, C, M, N, K, lda, ldb, ldc, beta, max_ctas, s, g);
}

template <bool kPair>
static int launch_swiglu(const void* X, const void* W, void* GU, void* ACT, int M, int F, int K, long long ldx, long long ldw, long long ldgu,
                         long long ldact, cudaStream_t s) {
  constexpr int kCols = kPair ? 128 : 64;            // gate rows (and up rows) per tile
  const __nv_bfloat16 *w = (const __nv_bfloat16*)W, *gu = (const __nv_bfloat16*)GU;
  CUtensorMap tmA, tmW;
  SwigluMaps sw;
  int rc = get_tmap_2d_bf16(&tmA, X, M, K, ldx, kBM, kBK, 1);
  if (!rc) rc = get_tmap_2d_bf16(&tmW, w, F, K, ldw, kCols, kBK, 1);
  if (!rc) rc = get_tmap_2d_bf16(&sw.w_up, w + static_cast<long long>(F) * ldw, F, K, ldw, kCols, kBK, 1);
  if (!rc) rc = get_tmap_2d_bf16(&sw.act, ACT, M, F, ldact, 32, 64, 1);
  sw.gate = sw.up = sw.act;
  sw.keep = GU != nullptr;
  if (!rc && GU != nullptr) rc = get_tmap_2d_bf16(&sw.gate, gu, M, F, ldgu, 32, 64, 1);
  if (!rc && GU != nullptr) rc = get_tmap_2d_bf16(&sw.up, gu + F, M, F, ldgu, 32, 64, 1);
  if (rc) LLMCTL_FAIL(rc, "tensor maps");
  const int tiles = ((M + (kPair ? 2 : 1) * kBM - 1) / ((kPair ? 2 : 1) * kBM)) * ((F + kCols - 1) / kCols);
  if constexpr (kPair) {
    auto kern = gemm2_tcgen05_kernel<256, false, false, __nv_bfloat16, Gated::kForward>;
    LLMCTL_CHECK(allow_smem(kern, Gemm2Cfg<256, Gated::kForward>::kSmemBytes));
    const int pairs = tiles < num_sms() / 2 ? tiles : num_sms() / 2;
    LLMCTL_CHECK(launch_gemm_kernel(kern, 2 * pairs, Gemm2Cfg<256, Gated::kForward>::kSmemBytes, s, tmA, tmW, tmA, (__nv_bfloat16*)ACT, ldact, M, F, K, 0, GemmGate{}, sw));
  } else {
    auto kern = gemm_tcgen05_kernel<128, false, false, __nv_bfloat16, Gated::kForward>;
    LLMCTL_CHECK(allow_smem(kern, GemmCfg<128, Gated::kForward>::kSmemBytes));
    LLMCTL_CHECK(launch_gemm_kernel(kern, tiles < num_sms() ? tiles : num_sms(), GemmCfg<128, Gated::kForward>::kSmemBytes, s, tmA, tmW, tmA, (__nv_bfloat16*)ACT, ldact,
                                    M, F, K, 0, GemmGate{}, sw));
  }
  LLMCTL_RETURN_LAST();
}

// kBN: 64 or 128 (one CTA), 256 (CTA pair).
template <int kBN>
static int launch_rotate(const void* X, const void* W, void* C, int M, int N, int K, long long ldx, long long ldw, long long ldc, const SwigluMaps& sw, cudaStream_t s) {
  constexpr bool kPair = kBN == 256;
  constexpr int kRows = (kPair ? 2 : 1) * kBM;
  CUtensorMap tmA, tmW, tmC;
  int rc = get_tmap_2d_bf16(&tmA, X, M, K, ldx, kBM, kBK, 1);
  if (!rc) rc = get_tmap_2d_bf16(&tmW, W, N, K, ldw, kPair ? kBN / 2 : kBN, kBK, 1);
  if (!rc) rc = get_tmap_2d_bf16(&tmC, C, M, N, ldc, 32, 64, 1);
  if (rc) LLMCTL_FAIL(rc, "tensor maps");
  const int tiles = ((M + kRows - 1) / kRows) * ((N + kBN - 1) / kBN), most = kPair ? num_sms() / 2 : num_sms();
  const int grid = tiles < most ? tiles : most;
  if constexpr (kPair) {
    auto kern = gemm2_tcgen05_kernel<256, false, false, __nv_bfloat16, Gated::kRotate>;
    LLMCTL_CHECK(allow_smem(kern, Gemm2Cfg<256, Gated::kRotate>::kSmemBytes));
    LLMCTL_CHECK(launch_gemm_kernel(kern, 2 * grid, Gemm2Cfg<256, Gated::kRotate>::kSmemBytes, s, tmA, tmW, tmC, (__nv_bfloat16*)C, ldc, M, N, K, 0, GemmGate{}, sw));
  } else {
    auto kern = gemm_tcgen05_kernel<kBN, false, false, __nv_bfloat16, Gated::kRotate>;
    LLMCTL_CHECK(allow_smem(kern, GemmCfg<kBN, Gated::kRotate>::kSmemBytes));
    LLMCTL_CHECK(launch_gemm_kernel(kern, grid, GemmCfg<kBN, Gated::kRotate>::kSmemBytes, s, tmA, tmW, tmC, (__nv_bfloat16*)C, ldc, M, N, K, 0, GemmGate{}, sw));
  }
  LLMCTL_RETURN_LAST();
}

// kBN: 64 or 128 (one CTA), 256 (CTA pair).
template <int kBN>
static int launch_swiglu_bwd(const void* DY, const void* W, const void* GU, void* DGU, int M, int F, int K, long long lddy, long long ldw,
                             long long ldgu, cudaStream_t s) {
  constexpr bool kPair = kBN == 256;
  constexpr int kRows = (kPair ? 2 : 1) * kBM;
  CUtensorMap tmA, tmW;
  SwigluMaps sw;
  int rc = get_tmap_2d_bf16(&tmA, DY, M, K, lddy, kBM, kBK, 1);
  if (!rc) rc = get_tmap_2d_bf16(&tmW, W, K, F, ldw, kBK, 64, 1);
  if (!rc) rc = get_tmap_2d_bf16(&sw.gate, DGU, M, F, ldgu, 32, 64, 1);
  if (!rc) rc = get_tmap_2d_bf16(&sw.up, (const __nv_bfloat16*)DGU + F, M, F, ldgu, 32, 64, 1);
  if (rc) LLMCTL_FAIL(rc, "tensor maps");
  sw.w_up = sw.act = sw.gate;
  sw.keep = 0;
  sw.gu = (const __nv_bfloat16*)GU;
  sw.ldgu = ldgu;
  const int tiles = ((M + kRows - 1) / kRows) * ((F + kBN - 1) / kBN), most = kPair ? num_sms() / 2 : num_sms();
  const int grid = tiles < most ? tiles : most;
  if constexpr (kPair) {
    auto kern = gemm2_tcgen05_kernel<256, false, true, __nv_bfloat16, Gated::kBackward>;
    LLMCTL_CHECK(allow_smem(kern, Gemm2Cfg<256, Gated::kBackward>::kSmemBytes));
    LLMCTL_CHECK(launch_gemm_kernel(kern, 2 * grid, Gemm2Cfg<256, Gated::kBackward>::kSmemBytes, s, tmA, tmW, tmA, (__nv_bfloat16*)DGU, ldgu, M, F, K, 0, GemmGate{}, sw));
  } else {
    auto kern = gemm_tcgen05_kernel<kBN, false, true, __nv_bfloat16, Gated::kBackward>;
    LLMCTL_CHECK(allow_smem(kern, GemmCfg<kBN, Gated::kBackward>::kSmemBytes));
    LLMCTL_CHECK(launch_gemm_kernel(kern, grid, GemmCfg<kBN, Gated::kBackward>::kSmemBytes, s, tmA, tmW, tmA, (__nv_bfloat16*)DGU, ldgu, M, F, K, 0, GemmGate{}, sw));
  }
  LLMCTL_RETURN_LAST();
}

}  // namespace llmctl

using namespace llmctl;

// The narrowest tile with which the problem is still one wave (see gemm_bf16_impl), 0 if there is none.
static int one_wave_tile(int M, int N) {
  const long long rows = (M + 127) / 128, sms = num_sms();
  if (rows * ((N + 63) / 64) <= sms) return 64;
  return rows * ((N + 127) / 128) <= sms ? 128 : 0;
}

// CTAs that share the K of each 128 x 64 tile (gemm_split_kernel), 1 where that does not pay: fewer tiles than SMs, and a K whose blocks, 0.2 us
// each for a CTA alone on its SM and 0.32 for two, outweigh the cluster's launch and exchange.  Clusters of 4 and 8 leave SMs of a GPC over: 128 CTAs
// of them are resident one to an SM.  us, one CTA a tile / split (operands from HBM): 64 x 768 x 32000 98 / 19 (8), 200 x 768 98 / 31 (4), 500 x 768
// 100 / 48 (4), 1000 x 768 104 / 83 (2), 500 x 2048 101 / 88 (2), 200 x 2048 x 11264 37 / 23, x 5632 20.1 / 15.3, 500 x 768 x 4096 15.8 / 12.9;
// left alone: 200 x 2048 x 2048 9.5 / 9.9, 300 x 768 x 2048 9.3 / 9.4, 777 x 768 x 2048 9.6 / 13.9, 500 x 2048 x 5632 20.5 / 22.9, and, though it would win,
// 768 x 768 x 3000 of M-major operands 14.0 / 12.4.  fp32 sums of another order: the bits of a product depend on its number of rows.
static int split_count(int M, int N, int K) {
  const long long tiles = static_cast<long long>((M + kBM - 1) / kBM) * ((N + kSplitBN - 1) / kSplitBN), sms = num_sms();
  if (tiles > sms) return 1;
  const double blocks = (K + kBK - 1) / kBK;
  double least = 0.87 * (2.7 + 0.2 * blocks);
  int best = 1;
  for (int splits = 2; splits <= kMaxSplits && 8 * splits <= blocks; splits *= 2) {
    const long long ctas = tiles * splits;
    if (ctas > 2 * sms) break;
    const bool alone = splits == 2 ? ctas <= sms : ctas <= sms * 128 / 148;
    const double us = (splits == 8 ? 2. : 0.) + (alone ? 6. + 0.2 * blocks / splits : 9.5 + 0.32 * blocks / splits);
    if (us < least) {
      least = us;
      best = splits;
    }
  }
  return best;
}

// D[M,N] = op(A) op(B) (+ D if beta).  a_mn / b_mn select the operand storage (see file header).
// out_fp32: D is fp32 (else bf16).  tile_n: 0 = auto, 64 / 128 / 192 / 256 (1-CTA tiles), 2 = 256x256 CTA-pair tile, 3 = 256x128 CTA-pair tile, -2 .. -8 = 128x64 tiles
// whose K that many CTAs share.  max_ctas: 0 = all SMs
// (a smaller value leaves SMs free for a concurrent communication kernel).
static int gemm_bf16_impl(const void* A, const void* B, void* C, int M, int N, int K,
                          long long lda, long long ldb, long long ldc, int a_mn, int b_mn,
                          int out_fp32, int beta, int tile_n, int max_ctas, void* stream, const GemmGate& g) {
  LLMCTL_BEGIN();
  LLMCTL_REQUIRE(M > 0 && N > 0 && K > 0);
  LLMCTL_REQUIRE(lda % 8 == 0 && ldb % 8 == 0 && N % 8 == 0);
  LLMCTL_REQUIRE((reinterpret_cast<uintptr_t>(A) & 15) == 0 && (reinterpret_cast<uintptr_t>(B) & 15) == 0 &&
                 (reinterpret_cast<uintptr_t>(C) & 15) == 0);
  LLMCTL_REQUIRE(out_fp32 ? (ldc % 4 == 0) : (ldc % 8 == 0));
  cudaStream_t s = (cudaStream_t)stream;
  // auto.  A problem of at most one wave of tiles is bound by what one CTA does (fill, K loop at the latency of L2, epilogue), not
  // by the chip: the narrowest tile that still fits one wave wins (M x N x K, us, pair 256 x 256 / 128 x 128 / 128 x 64:
  // 777 x 2304 x 768: 9.2 / 6.8 / 9.0, 777 x 768 x 2048: 14.6 / 10.6 / 10.1, 512 x 2048 x 5632: 30.7 / 23.4 / 21.4).
  // Beyond one wave operand traffic from L2 sets the pace and the 256 x 256 CTA-pair tile moves least of it (4096 x 2048 x 2048:
  // 26.7 / 33.1 / 49.0, 4096 x 11264 x 2048: 130 / 181 / 276); 128 x 192 and pair 256 x 128 never win by more than a few per cent
  // and stay selectable (tile_n = 192 / 3).  Gated operands arrive slab by slab and keep the pair tile.
  if (tile_n == 0 && !g.waits() && g.grp_tile_expert == nullptr && max_ctas == 0) {
    const int splits = split_count(M, N, K);
    if (splits > 1) tile_n = -splits;
  }
  if (tile_n == 0 && g.flags == nullptr && g.b_flags == nullptr && max_ctas == 0) tile_n = one_wave_tile(M, N);
  if (tile_n == 0 && M > 128 && N > 128) tile_n = 2;
  if (tile_n < 0) {
    LLMCTL_REQUIRE(tile_n >= -kMaxSplits && -tile_n <= (K + kBK - 1) / kBK && !g.waits() && g.grp_tile_expert == nullptr && max_ctas == 0);
    return (out_fp32 ? dispatch_split<float> : dispatch_split<__nv_bfloat16>)(a_mn, b_mn, A, B, C, M, N, K, lda, ldb, ldc, beta, -tile_n, s);
  }
  if (tile_n == 2) {   // 2-CTA pair tile 256 x 256 (cta_group::2)
    if (out_fp32) return dispatch_layout2<256, float>(a_mn, b_mn, A, B, C, M, N, K, lda, ldb, ldc, beta, max_ctas, s, g);
    return dispatch_layout2<256, __nv_bfloat16>(a_mn, b_mn, A, B, C, M, N, K, lda, ldb, ldc, beta, max_ctas, s, g);
  }
  if (tile_n == 3) {   // 2-CTA pair tile 256 x 128
    if (out_fp32) return dispatch_layout2<128, float>(a_mn, b_mn, A, B, C, M, N, K, lda, ldb, ldc, beta, max_ctas, s, g);
    return dispatch_layout2<128, __nv_bfloat16>(a_mn, b_mn, A, B, C, M, N, K, lda, ldb, ldc, beta, max_ctas, s, g);
  }
  int bn = tile_n;
  if (bn != 64 && bn != 128 && bn != 192 && bn != 256) {
    const int sms = num_sms();
    const long long t256 = static_cast<long long>((M + 127) / 128) * ((N + 255) / 256);
    const long long t128 = static_cast<long long>((M + 127) / 128) * ((N + 127) / 128);
    const double c256 = static_cast<double>((t256 + sms - 1) / sms) * 2.0;
    const double c128 = static_cast<double>((t128 + sms - 1) / sms) * 1.45;  // measured: a 128-wide tile runs at ~0.7x the rate
    bn = (c128 < c256) ? 128 : 256;
  }
  if (bn == 64) {
    if (out_fp32) return dispatch_layout<64, float>(a_mn, b_mn, A, B, C, M, N, K, lda, ldb, ldc, beta, max_ctas, s, g);
    return dispatch_layout<64, __nv_bfloat16>(a_mn, b_mn, A, B, C, M, N, K, lda, ldb, ldc, beta, max_ctas, s, g);
  }
  if (bn == 192) {
    if (out_fp32) return dispatch_layout<192, float>(a_mn, b_mn, A, B, C, M, N, K, lda, ldb, ldc, beta, max_ctas, s, g);
    return dispatch_layout<192, __nv_bfloat16>(a_mn, b_mn, A, B, C, M, N, K, lda, ldb, ldc, beta, max_ctas, s, g);
  }
  if (bn == 256) {
    if (out_fp32) return dispatch_layout<256, float>(a_mn, b_mn, A, B, C, M, N, K, lda, ldb, ldc, beta, max_ctas, s, g);
    return dispatch_layout<256, __nv_bfloat16>(a_mn, b_mn, A, B, C, M, N, K, lda, ldb, ldc, beta, max_ctas, s, g);
  }
  if (out_fp32) return dispatch_layout<128, float>(a_mn, b_mn, A, B, C, M, N, K, lda, ldb, ldc, beta, max_ctas, s, g);
  return dispatch_layout<128, __nv_bfloat16>(a_mn, b_mn, A, B, C, M, N, K, lda, ldb, ldc, beta, max_ctas, s, g);
}

LLMCTL_API int llmctl_gemm_bf16(const void* A, const void* B, void* C, int M, int N, int K,
                                long long lda, long long ldb, long long ldc, int a_mn, int b_mn,
                                int out_fp32, int beta, int tile_n, int max_ctas, void* stream) {
  return gemm_bf16_impl(A, B, C, M, N, K, lda, ldb, ldc, a_mn, b_mn, out_fp32, beta, tile_n, max_ctas, stream,
                        GemmGate{});
}

// ACT[M, F] = silu(X Wg^T) * (X Wu^T) for X [M, K] and the packed W [2F, K] = [Wg ; Wu]; GU [M, 2F] receives the two products (rounded
// to bf16) unless it is null.  The activation is taken from the fp32 accumulators.  One pass less over the 2F columns and one launch
// less than the product and llmctl_swiglu_fwd; tiles by the rule of llmctl_gemm_bf16 (128 of the 256 columns of a pair tile are gate
// columns, 64 of the 128 of a single one).
LLMCTL_API int llmctl_gemm_swiglu_bf16(const void* X, const void* W, void* GU, void* ACT, int M, int F, int K, long long ldx, long long ldw,
                                       long long ldgu, long long ldact, void* stream) {
  LLMCTL_BEGIN();
  LLMCTL_REQUIRE(M > 0 && F > 0 && K > 0 && F % 8 == 0 && ldx % 8 == 0 && ldw % 8 == 0 && ldact % 8 == 0 && (GU == nullptr || ldgu % 8 == 0));
  LLMCTL_REQUIRE(((reinterpret_cast<uintptr_t>(X) | reinterpret_cast<uintptr_t>(W) | reinterpret_cast<uintptr_t>(GU) |
                   reinterpret_cast<uintptr_t>(ACT)) & 15) == 0 && static_cast<long long>(ldact) >= F);
  const bool one_wave = static_cast<long long>((M + kBM - 1) / kBM) * ((F + 63) / 64) <= num_sms();
  return (one_wave || M <= 128 ? launch_swiglu<false> : launch_swiglu<true>)(X, W, GU, ACT, M, F, K, ldx, ldw, ldgu, ldact, (cudaStream_t)stream);
}

// DGU[M, 2F] = (d gate | d up) of a gated MLP from dy [M, K], the down-projection W [K, F] and the forward's GU [M, 2F] (row stride ldgu for
// both): the product dy W is never stored.  Against the product and llmctl_swiglu_bwd it saves writing and reading M x F and a launch, and
// the activation's arithmetic and traffic hide behind the products of the next tile (4096 x 5632 x 2048: 106 us
// in two, 86 us in one; 16384 rows: 380 / 297; 1000 x 2048 x 2048: 25.6 / 23.4).
LLMCTL_API int llmctl_gemm_swiglu_bwd_bf16(const void* DY, const void* W, const void* GU, void* DGU, int M, int F, int K, long long lddy,
                                           long long ldw, long long ldgu, void* stream) {
  LLMCTL_BEGIN();
  LLMCTL_REQUIRE(M > 0 && F > 0 && K > 0 && F % 8 == 0 && lddy % 8 == 0 && ldw % 8 == 0 && ldgu % 8 == 0 && ldgu >= 2LL * F);
  LLMCTL_REQUIRE(((reinterpret_cast<uintptr_t>(DY) | reinterpret_cast<uintptr_t>(W) | reinterpret_cast<uintptr_t>(GU) |
                   reinterpret_cast<uintptr_t>(DGU)) & 15) == 0);
  const int bn = one_wave_tile(M, F);
  auto launch = bn == 64 ? launch_swiglu_bwd<64> : bn == 128 || M <= 128 || F <= 128 ? launch_swiglu_bwd<128> : launch_swiglu_bwd<256>;
  return launch(DY, W, GU, DGU, M, F, K, lddy, ldw, ldgu, (cudaStream_t)stream);
}

// C[M, N] = X W^T with the first `rotated` columns, heads of 64, rotated as llmctl_rope_inplace does (sign 1; cos, sin: [positions, 32]): a packed
// projection and its rotation in one launch, without the pass over q and k between them.  Tiles by the one-wave and pair rule of
// llmctl_gemm_bf16; no K shared by a cluster, which that entry tries first and takes for no packed projection (N = 3 K has too many tiles).
// us of 12 layers of width 768 without gradients, two launches / one: 777 tokens 668 / 653, 2000 tokens 893 / 870, 100 tokens (host) 623 / 590.
LLMCTL_API int llmctl_gemm_rope_bf16(const void* X, const void* W, void* C, int M, int N, int K, long long ldx, long long ldw, long long ldc, const float* cos_t,
                                     const float* sin_t, const int* positions, int seq_len, int rotated, void* stream) {
  LLMCTL_BEGIN();
  LLMCTL_REQUIRE(M > 0 && N > 0 && K > 0 && N % 64 == 0 && rotated % 64 == 0 && rotated >= 0 && rotated <= N && ldx % 8 == 0 && ldw % 8 == 0 && ldc % 8 == 0 && ldc >= N &&
                 seq_len > 0 && cos_t != nullptr && sin_t != nullptr);
  LLMCTL_REQUIRE(aligned16(X, W, C, cos_t, sin_t));
  SwigluMaps sw{};
  sw.cos = cos_t;
  sw.sin = sin_t;
  sw.positions = positions;
  sw.seq = seq_len;
  sw.rotated = rotated;
  const int bn = one_wave_tile(M, N);
  const auto launch = bn == 64 ? launch_rotate<64> : bn == 128 || M <= 128 ? launch_rotate<128> : launch_rotate<256>;
  return launch(X, W, C, M, N, K, ldx, ldw, ldc, sw, (cudaStream_t)stream);
}

// Grouped GEMM for mixture-of-experts layers: C[r, :] = A[r, :] W[expert(r)]^T over `max_tiles` blocks of 128 rows of A
// ([max_tiles * 128, K], K-major); W: [experts, N, K] contiguous; tile_expert[i] names the expert of row block i and
// *num_tiles (on the device) says how many leading blocks hold rows — the others are skipped, their rows of C stay
// unwritten.  One persistent launch for all experts; no host synchronisation.
LLMCTL_API int llmctl_gemm_bf16_grouped(const void* A, const void* W, void* C, int max_tiles, int N, int K, long long lda,
                                        long long ldc, const int* tile_expert, const int* num_tiles, int experts,
                                        void* stream) {
  LLMCTL_REQUIRE(tile_expert != nullptr && num_tiles != nullptr && experts >= 1 && max_tiles >= 1 && K % 8 == 0 &&
                 static_cast<long long>(max_tiles) * kBM < (1LL << 31) && static_cast<long long>(experts) * N < (1LL << 31));
  GemmGate g{};
  g.grp_tile_expert = tile_expert;
  g.grp_num_tiles = num_tiles;
  g.grp_experts = experts;
  return gemm_bf16_impl(A, W, C, max_tiles * kBM, N, K, lda, K, ldc, 0, 0, 0, 0, N > 128 ? 256 : 128, 0, stream, g);
}

LLMCTL_SYMM_WATCHDOG_MODULE(gemm)

// K1 consumer: the same GEMM, but rows of A (K-major, [M, K] in a symmetric buffer) outside [own_lo, own_hi) are only
// read once their flag  flags[row / rows_per_flag]  (local signal pad, written by the peers' llmctl_ag_push) reached
// `epoch`.  M = world * rows_per_rank; tile rows are visited in arrival order when the shapes allow it.
LLMCTL_API int llmctl_gemm_bf16_gated(const void* A, const void* B, void* C, int M, int N, int K,
                                      long long lda, long long ldb, long long ldc, int b_mn, int out_fp32,
                                      int beta, int tile_n, int max_ctas, const unsigned int* flags,
                                      unsigned int epoch, int rows_per_flag, int rank, int world,
                                      void* stream) {
  LLMCTL_REQUIRE(flags != nullptr && world >= 1 && world <= symm::kMaxRanks && M % world == 0 && rows_per_flag > 0 &&
                 (M / world) % rows_per_flag == 0 && M / rows_per_flag <= 256);
  GemmGate g{};
  g.flags = flags;
  g.epoch = epoch;
  g.rows_per_flag = rows_per_flag;
  g.own_lo = rank * (M / world);
  g.own_hi = g.own_lo + M / world;
  g.perm = 1;
  g.rank = rank;
  g.world = world;
  return gemm_bf16_impl(A, B, C, M, N, K, lda, ldb, ldc, 0, b_mn, out_fp32, beta, tile_n, max_ctas, stream, g);
}

// K8 consumer: the same GEMM, with the B operand (a ZeRO-3 parameter matrix inside a gathered symmetric buffer) read
// tile by tile as its shards arrive: flag  b_flags[(b_off + element) / b_slab]  (local signal pad, raised by the shard
// owners' llmctl_ag_push) must have reached `epoch` before the tile's rows are loaded.  ldb must equal the row pitch of
// B inside the buffer.
LLMCTL_API int llmctl_gemm_bf16_bgated(const void* A, const void* B, void* C, int M, int N, int K,
                                       long long lda, long long ldb, long long ldc, int a_mn, int b_mn,
                                       int out_fp32, int beta, int tile_n, int max_ctas,
                                       const unsigned int* b_flags, unsigned int epoch, long long b_off,
                                       long long b_slab, void* stream) {
  LLMCTL_REQUIRE(b_flags != nullptr && b_slab > 0 && b_off >= 0);
  GemmGate g{};
  g.b_flags = b_flags;
  g.b_epoch = epoch;
  g.b_off = b_off;
  g.b_slab = b_slab;
  g.b_row_stride = ldb;
  g.b_span = static_cast<long long>(K) * ldb;
  return gemm_bf16_impl(A, B, C, M, N, K, lda, ldb, ldc, a_mn, b_mn, out_fp32, beta, tile_n, max_ctas, stream, g);
}
