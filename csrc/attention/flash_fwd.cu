// K6 (forward): causal flash attention on the 5th-generation tensor cores, bf16: head sizes 64 and 128, sequences of any
// length; and queries / keys of 192 (128 of each head's own + 64 of the key that all heads share) over values of 128, for batches
// of sequences of unlike lengths whose queries may begin behind earlier keys (prompts of latent attention with rebuilt keys and
// values, llmctl_latent_prompt_attention).
//
// Reference: HF modules choose SDPA/eager attention behind `self.model(**batch)` (reference
// llmctl/runtime/engine.py:284); the reference's tuner times a naive softmax(QK^T)V (reference
// llmctl/plugins/autotuning.py:149-188).  Baseline to beat: cuDNN / flash-attn SDPA.
#include <float.h>
#include <math.h>

#include "../common/ptx.cuh"
#include "../common/tma_host.h"
#include "../common/util.cuh"
#include "../common/dependent.cuh"
#include "../common/fast_div.h"
#include "../common/wait_status.h"
#include "flash_split.h"

namespace llmctl {
using namespace ptx;

// =====================================================================================================
// One work item = one (batch, head, 256-query block) handled as two 128-query tiles A and B that share every K/V tile (half
// the K/V smem traffic) and ping-pong on the tensor core: while the softmax warpgroup of tile A works on S_A, the MMA warp runs
// P_B V / Q_B K^T and vice versa.
//   warps 0-3   softmax warpgroup of tile A      warps 4-7  softmax warpgroup of tile B
//   warp 8      TMA producer (Q_A, Q_B once per item; rings of 128 keys)
//   warp 9      MMA issuer                       warps 10-11 idle (they complete the third warpgroup so that
//               setmaxnreg can move its registers to the softmax warpgroups: 200 per softmax thread, enough to
//               hold a whole 128-column S row plus the packed P chunk without spilling)
// TMEM (all 512 columns): S_A [0,128) S_B [128,256) O_A [256,384) O_B [384,512).  P never touches shared
// memory: the softmax thread overwrites the first 64 columns of its own S row with bf16x2 probabilities
// (tcgen05.st) and P V reads its A operand straight from TMEM.  The tensor pipe executes in issue order, so
// Q K^T of block j+1 (which overwrites S/P) is simply issued after P V of block j; tcgen05.commit covers every
// earlier MMA, so "S(j+1) ready" also means "P V(j) has retired" and the O rescale needs no extra barrier.
// A tile's chain (S ready -> softmax -> P V, Q K^T -> S ready) is longer than the two tiles' tensor work (3600 against 2048
// clocks per block when P was handed over whole), so P is handed over in two halves: the first 64 keys' P V runs while the
// second half is still being exponentiated.
// The running max is only advanced when it grows by more than 8 (log2 units): between rescales the reference stays put and
// P may reach 2^8, which fp32 accumulation and bf16 P hold exactly as well — this removes almost all TMEM read-modify-write
// passes over O.
// =====================================================================================================
namespace ffwd {
constexpr int kRows = 128;               // queries per tile, keys per tile
constexpr int kPanel = kRows * 128;      // bytes of one [128 rows x 64 bf16] swizzled panel
constexpr int kThreads = 384;
constexpr float kRescaleThreshold = 8.f;
// Stages of the K and V rings: what 227 KB hold beside the two query tiles (160 KB at D = 64, 192 KB at 128, 224 KB at 192 / 128).
template <int DQK, int DV>
struct Cfg {
  static constexpr int kQTile = DQK / 64 * kPanel, kVTile = DV / 64 * kPanel;
  static constexpr int kKStages = DQK == 64 ? 4 : 2;
  static constexpr int kVStages = DQK == 64 ? 4 : DQK == 128 ? 2 : 1;
  static constexpr int kKAt = 2 * kQTile, kVAt = kKAt + kKStages * kQTile;
  static constexpr int kSmem = kVAt + kVStages * kVTile + 1024;
};
__device__ unsigned int g_status = 0;    // != 0: a bounded wait of the kernel ran out

// One sequence of a batch of unlike lengths: its queries are rows [q_row, q_row + n) of Q and O at positions start + i, its keys
// (position 0 first) begin at row k_row of K and V.  Rows from its last key to the next multiple of 128 hold zeros.
struct Seq {
  int q_row, n, start, k_row;
};
// Items are numbered through (query block, batch, head).  Every role decodes every item: with divisions that was 700 clocks of the loading
// and of the issuing warp between two items (8 x 512 x 32 x 128 37.4 us, now 34.4; 8 x 512 x 12 x 64 13.9 / 13.2; 2 x 2048 x 40 x 128 90.5 / 88.5).
struct Order {
  int n_items, nqb;
  FastDiv per_qb, heads;
};
}  // namespace ffwd

// The mask is resolved per 32-column chunk, which is warp-uniform (warp q owns rows 32q .. 32q+31; row r sees the columns up to
// off + r): chunks that all its rows see take the plain path, chunks that none sees cost nothing (no compare, no exponential,
// P = 0), only the chunks in between compare their columns against the lane.
template <bool kMask, int DV>
__device__ __forceinline__ void softmax_block(uint32_t tS, uint32_t tO, int q, int lane, int off, bool first, float scale_log2,
                                              float& m_ref, float& l0, float& l1, uint64_t* bar_p0, uint64_t* bar_p1) {
  using namespace ffwd;
  const int w0 = off + q * 32;        // last column that the warp's first row sees
  const int mine = w0 + lane;         // ... and this row
  // The whole S row (128 fp32) is read from TMEM once and stays in registers for both passes: every
  // tcgen05.ld -> wait round trip removed here is latency the tensor pipe would otherwise sit idle for.
  uint32_t r[128];
  tmem_ld_x32(tS, r);
  tmem_ld_x32(tS + 32, r + 32);
  tmem_ld_x32(tS + 64, r + 64);
  tmem_ld_x32(tS + 96, r + 96);
  tmem_ld_wait();
  // pass 1: raw row maximum (the scale is positive, so it commutes with max)
  float m0 = -INFINITY, m1 = -INFINITY;
#pragma unroll
  for (int c = 0; c < 4; ++c) {
    if (kMask && c * 32 > w0 + 31) continue;             // fully masked chunk
    if (kMask && c * 32 + 31 > w0) {
#pragma unroll
      for (int e = c * 32; e < c * 32 + 32; ++e)
        if (e > mine) r[e] = 0xff800000u;                // -inf
    }
#pragma unroll
    for (int e = c * 32; e < c * 32 + 32; e += 4) {
      m0 = max3(m0, __uint_as_float(r[e]), __uint_as_float(r[e + 1]));
      m1 = max3(m1, __uint_as_float(r[e + 2]), __uint_as_float(r[e + 3]));
    }
  }
  const float bm = fmaxf(m0, m1) * scale_log2;
  // lazy reference update: only move the reference when the block maximum outgrows it by more than 2^8
  const bool need = bm > m_ref + kRescaleThreshold;
  float alpha = 1.f;
  if (need) {
    alpha = (m_ref == -INFINITY) ? 0.f : ex2_approx(m_ref - bm);
    m_ref = bm;
    l0 *= alpha;
    l1 *= alpha;
  }
  if (!first && __any_sync(0xffffffffu, need)) {
    // rare (reference moved by more than 2^8): scale the running O row
#pragma unroll 1
    for (int c = 0; c < DV / 32; ++c) {
      uint32_t o[32];
      tmem_ld_x32(tO + c * 32, o);
      tmem_ld_wait();
#pragma unroll
      for (int e = 0; e < 32; e += 2) {
        float x0, x1;
        mul2(x0, x1, __uint_as_float(o[e]), __uint_as_float(o[e + 1]), alpha);
        o[e] = __float_as_uint(x0);
        o[e + 1] = __float_as_uint(x1);
      }
      tmem_st_x16(tO + c * 32, o);
      tmem_st_x16(tO + c * 32 + 16, o + 16);
    }
  }
  // pass 2: p = 2^(s*scale - m_ref) -> bf16x2 -> back into the first 64 columns of this S row
  const float neg_m = -m_ref;
#pragma unroll
  for (int c = 0; c < 4; ++c) {
    uint32_t pk[16];
    if (kMask && c * 32 > w0 + 31) {                     // fully masked chunk: P = 0, nothing to compute
#pragma unroll
      for (int e = 0; e < 16; ++e) pk[e] = 0u;
    } else {
#pragma unroll
      for (int e = 0; e < 32; e += 2) {
        float a0, a1;
        fma2(a0, a1, __uint_as_float(r[c * 32 + e]), __uint_as_float(r[c * 32 + e + 1]), scale_log2, neg_m);
        const float p0 = ex2_approx(a0), p1 = ex2_approx(a1);
        add2(l0, l1, p0, p1);
        pk[e >> 1] = pack_bf16x2(p0, p1);
      }
    }
    tmem_st_x16(tS + c * 16, pk);
    if (c & 1) {                                         // half of P (and the rescaled O) is in place
      tmem_st_wait();
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(c == 1 ? bar_p0 : bar_p1);
    }
  }
}

// =====================================================================================================
// The kernel is PERSISTENT.  The timeline of a one-CTA-per-item launch (tools/trace_flash.py) showed ~5.5 k clocks
// between kernel start and the first usable S (barrier / TMEM set-up, tensor-map fetch, Q and K TMA latency,
// first Q K^T) and ~3 k for the epilogue, against ~3.5 k per 256x128 iteration: at the training shape
// (S = 512, 2-4 iterations per CTA) more than half of every CTA's life was set-up and drain, with nothing else
// resident on the SM (197 KB of shared memory) to hide it.  Here one CTA per SM walks a heavy-first list of
// (batch, head, 256-query block) items: TMEM, barriers and tensor maps are set up once, the K/V ring, the
// S/P ping-pong and all barrier phases run straight through item boundaries, the TMA warp prefetches the next
// item's Q tiles as soon as the last Q K^T of the current one has retired, and the MMA warp starts the next
// item's Q K^T while the softmax warpgroups are still normalising and storing O of the current one (O goes
// from registers straight to global memory, so no staging buffer blocks the Q prefetch).
//
// kSplit: an item is one tile of 128 queries whose keys the two softmax warpgroups share, A the first half of the key blocks, B the rest
// (with the diagonal); every K/V tile then serves one of them.  Both accumulators lie in the same lanes of TMEM, so each warpgroup puts half of the
// columns together.  For grids whose longest item decides: its chain of blocks is half as long (see split_keys).
template <int DQK, int DV, bool kSplit>
__global__ void __launch_bounds__(ffwd::kThreads, 1)
flash_fwd_kernel(const __grid_constant__ CUtensorMap tmQ, const __grid_constant__ CUtensorMap tmK,
                 const __grid_constant__ CUtensorMap tmKs, const __grid_constant__ CUtensorMap tmV, __nv_bfloat16* __restrict__ O,
                 long long o_tok_stride, int o_wide, float* __restrict__ lse, const ffwd::Seq* __restrict__ seqs, const ffwd::Order order, int max_q, int H,
                 int head_step, float scale_log2, int causal, unsigned char* wait_byte, long long* __restrict__ trace) {
  using namespace ffwd;
  using C = Cfg<DQK, DV>;
  constexpr int kOwn = DQK > 128 ? 2 : DQK / 64;         // panels of K that belong to the head; the last of three is shared by all
  extern __shared__ uint8_t smem_raw[];
  __shared__ uint64_t bar_q[2], bar_qfree[2], bar_kfull[C::kKStages], bar_vfull[C::kVStages], bar_kempty[C::kKStages], bar_vempty[C::kVStages];
  __shared__ uint64_t bar_s[2], bar_p0[2], bar_p1[2], bar_o[2], bar_ofree[2];
  __shared__ uint32_t tmem_base_smem;
  __shared__ int abort_flag;
  __shared__ float2 half_ml[kSplit ? 2 : 1][kRows];      // reference and sum of a row over each half of the keys
  __shared__ uint64_t bar_half[2];
  constexpr int kItemRows = kSplit ? kRows : 2 * kRows;

  const uint32_t smem_base = (smem_u32(smem_raw) + 1023u) & ~1023u;
  uint8_t* smem = smem_raw + (smem_base - smem_u32(smem_raw));      // layout: Q_A, Q_B, K ring, V ring
  const int warp = __shfl_sync(0xffffffffu, threadIdx.x >> 5, 0), lane = threadIdx.x & 31;

  if (threadIdx.x == 0) {
    for (int i = 0; i < 2; ++i) {
      mbar_init(&bar_q[i], 1);
      mbar_init(&bar_qfree[i], 1);
      mbar_init(&bar_s[i], 1);
      mbar_init(&bar_p0[i], 4);
      mbar_init(&bar_p1[i], 4);
      mbar_init(&bar_o[i], 1);
      mbar_init(&bar_half[i], 4);
      mbar_init(&bar_ofree[i], kSplit ? 8 : 4);
    }
    for (int i = 0; i < C::kKStages; ++i) {
      mbar_init(&bar_kfull[i], 1);
      mbar_init(&bar_kempty[i], 1);
    }
    for (int i = 0; i < C::kVStages; ++i) {
      mbar_init(&bar_vfull[i], 1);
      mbar_init(&bar_vempty[i], 1);
    }
    abort_flag = 0;
    fence_mbar_init();
  }
  if (warp == 8 && lane == 0) {
    prefetch_tmap(&tmQ);
    prefetch_tmap(&tmK);
    if (kOwn < DQK / 64) prefetch_tmap(&tmKs);
    prefetch_tmap(&tmV);
  }
  if (warp == 9) tmem_alloc<1>(&tmem_base_smem, 512);
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = tmem_base_smem;
  if constexpr (DQK > 128)
    wait_for_previous(seqs);
  else
    wait_for_previous();               // the outputs are stored to, not read
  volatile int* abort = &abort_flag;

  // optional event log of CTA 0 (LLMCTL_FLASH_TRACE): per role 127 x (code, clock) pairs after a count word.
  // roles: 0/1 softmax A/B (codes 1 = S ready, 2 = P written, 3 = O stored), 3 = TMA (40 = item start)
  const bool tracing = trace != nullptr && blockIdx.x == 0;
  const long long t_start = tracing ? clock64() : 0;
  int n_ev = 0;
  auto ev = [&](int role, int code) {
    if (tracing && n_ev < 127) {
      trace[role * 256 + 2 + 2 * n_ev] = code;
      trace[role * 256 + 3 + 2 * n_ev] = clock64() - t_start;
      ++n_ev;
      trace[role * 256] = n_ev;
    }
  };
  // The CTA's items: the list is sorted by length, and every other round runs over the CTAs backwards, so that nobody gets the
  // longest of every round (S = 2048, 40 heads x 2: 40 instead of 48 blocks on the busiest CTA, 39 on average).
  auto next_item = [&](int r, int& item) {
    item = r * gridDim.x + ((r & 1) ? gridDim.x - 1 - blockIdx.x : blockIdx.x);
    return item < order.n_items && !*abort;
  };
  // item -> (first query, head, batch, sequence); heavy (late) query blocks first so the tail is made of light items.
  // False: a shorter sequence of the batch has no such block.
  auto decode = [&](int item, int& q0, int& head, int& b, Seq& sq) {
    uint32_t rem, h;
    q0 = (order.nqb - 1 - static_cast<int>(order.per_qb.divide(item, rem))) * kItemRows;
    b = static_cast<int>(order.heads.divide(rem, h));
    head = static_cast<int>(h);
    if (seqs != nullptr)
      sq = seqs[b];
    else
      sq = Seq{0, max_q, 0, 0};
    return q0 < sq.n;
  };
  // key blocks of tile t of an item; a tile past the end of its sequence has none
  auto blocks = [&](const Seq& sq, int q0, int t) {
    if constexpr (kSplit) {
      const int all = static_cast<int>((sq.start + sq.n + kRows - 1u) / kRows);
      const int n = causal ? min(all, static_cast<int>((sq.start + q0 + kRows - 1u) / kRows) + 1) : all;
      return (n + 1 - t) >> 1;
    }
    const int qt = q0 + t * kRows;
    if (qt >= sq.n) return 0;
    const int all = static_cast<int>((sq.start + sq.n + kRows - 1u) / kRows);
    return causal ? min(all, static_cast<int>((sq.start + qt + kRows - 1u) / kRows) + 1) : all;
  };

  if (warp >= 8) {
   // register budget: the CTA owns 384 x 168; what warps 8-11 give back ((168-104) x 128) is exactly what the two
   // softmax warpgroups take ((200-168) x 256) — asking for more than was released blocks forever.
   setmaxnreg_dec<104>();
   if (warp == 8) {
    // ------------------------------------ TMA producer ------------------------------------
    if (lane == 0) {
      uint32_t g = 0;                 // K/V blocks so far (ring position and phase)
      uint32_t nA = 0, nB = 0;        // Q_A / Q_B loads so far
      uint32_t nk = 0, nv = 0;        // K / V loads so far
      bool ok = true;
      for (int item, r = 0; ok && next_item(r, item); ++r) {
        int q0, head, b;
        Seq sq;
        if (!decode(item, q0, head, b, sq)) continue;
        const int nblk_a = blocks(sq, q0, 0), nblk = kSplit ? nblk_a + blocks(sq, q0, 1) : max(nblk_a, blocks(sq, q0, 1));
        const int bc = seqs != nullptr ? 0 : b;          // batch coordinate of the maps
        const bool validB = !kSplit && q0 + kRows < sq.n;
        ev(3, 40);
        auto load_q = [&](int t, uint32_t done) {
          if (!mbar_wait_bounded(&bar_qfree[t], (done & 1u) ^ 1u, abort)) return false;      // the previous item's last Q K^T has retired
          mbar_expect_tx(&bar_q[t], C::kQTile);
#pragma unroll
          for (int p = 0; p < DQK / 64; ++p)
            tma_load_4d(smem + t * C::kQTile + p * kPanel, &tmQ, &bar_q[t], 64 * p, head, sq.q_row + q0 + t * kRows, bc);
          return true;
        };
        if (!(ok = load_q(0, nA))) break;
        ++nA;
        for (int j = 0; j < nblk; ++j, ++g) {
          const uint32_t ks = g % C::kKStages, vs = g % C::kVStages;
          const int row = sq.k_row + (kSplit ? (j & 1 ? nblk_a : 0) + (j >> 1) : j) * kRows;
          uint8_t* sK = smem + C::kKAt + ks * C::kQTile;
          uint8_t* sV = smem + C::kVAt + vs * C::kVTile;
          if (!(ok = mbar_wait_bounded(&bar_kempty[ks], ((g / C::kKStages) & 1u) ^ 1u, abort))) break;
          mbar_expect_tx(&bar_kfull[ks], C::kQTile);
          ++nk;
#pragma unroll
          for (int p = 0; p < kOwn; ++p) tma_load_4d(sK + p * kPanel, &tmK, &bar_kfull[ks], 64 * p, head + head_step, row, bc);
          if (kOwn < DQK / 64) tma_load_4d(sK + kOwn * kPanel, &tmKs, &bar_kfull[ks], 0, 0, row, bc);
          if (j == 0 && validB) {
            if (!(ok = load_q(1, nB))) break;
            ++nB;
          }
          if (!(ok = mbar_wait_bounded(&bar_vempty[vs], ((g / C::kVStages) & 1u) ^ 1u, abort))) break;
          mbar_expect_tx(&bar_vfull[vs], C::kVTile);
          ++nv;
#pragma unroll
          for (int p = 0; p < DV / 64; ++p) tma_load_4d(sV + p * kPanel, &tmV, &bar_vfull[vs], 64 * p, head + 2 * head_step, row, bc);
        }
      }
      release_dependents();
      // Copies still in flight when a wait ran out land before the CTA's shared memory is given back.
      if (*abort) {
        int none = 0;
        if (nA > 0) mbar_wait_bounded(&bar_q[0], (nA - 1) & 1u, &none);
        none = 0;
        if (nB > 0) mbar_wait_bounded(&bar_q[1], (nB - 1) & 1u, &none);
        none = 0;
        for (uint32_t j = nk > C::kKStages ? nk - C::kKStages : 0; j < nk; ++j, none = 0)
          mbar_wait_bounded(&bar_kfull[j % C::kKStages], (j / C::kKStages) & 1u, &none);
        for (uint32_t j = nv > C::kVStages ? nv - C::kVStages : 0; j < nv; ++j, none = 0)
          mbar_wait_bounded(&bar_vfull[j % C::kVStages], (j / C::kVStages) & 1u, &none);
      }
    }
   } else if (warp == 9) {
    // ------------------------------------ MMA issuer ------------------------------------
    // One warp issues for both tiles in strict A, B, A, B order: the issue order is what keeps the two tiles in
    // anti-phase (one in its softmax while the other owns the tensor pipe).  Measured alternatives (B1 S8192 H32):
    // two issuing warps, one per tile — the tiles drift into lock-step and the exponential unit and the tensor
    // core alternate instead of overlapping, 1010 -> 750 TFLOP/s; issuing the next item's first Q K^T early from
    // inside this loop — the extra live state spills into the issue sequences (or, with more registers here,
    // starves the softmax warps), 1010 -> 720-830 TFLOP/s.  This warp's issue latency is on the critical path:
    // the whole warp walks the loop and waits, only the products and commits are issued by one elected lane, so that
    // addresses and descriptors stay in uniform registers, which the instruction reads.
    constexpr uint32_t idesc_qk = make_idesc_bf16(kRows, kRows, 0u, 0u);   // A, B K-major
    constexpr uint32_t idesc_pv = make_idesc_bf16(kRows, DV, 0u, 1u);      // A from TMEM, B MN-major (V)
    auto wait = [&](uint64_t* bar, uint32_t parity) {
      mbar_wait_or_abort(bar, parity, abort);
      __syncwarp();
    };
    uint32_t g0 = 0;                 // K/V blocks consumed by earlier items
    uint32_t nQ0 = 0, nQ1 = 0;       // items done per tile (Q / O barrier phases)
    uint32_t nP0 = 0, nP1 = 0;       // P V products issued per tile (bar_p phases)
    for (int item, r = 0; next_item(r, item); ++r) {
      int q0, head, b;
      Seq sq;
      if (!decode(item, q0, head, b, sq)) continue;
      const int nblk_t0 = blocks(sq, q0, 0), nblk_t1 = blocks(sq, q0, 1);
      const int nblk = max(nblk_t0, nblk_t1);
      auto issue_qk = [&](int t, int j, bool release_k, bool last) {
        const uint32_t g = kSplit ? g0 + 2 * j + t : g0 + j, st = g % C::kKStages;
        wait(&bar_kfull[st], (g / C::kKStages) & 1u);
        tc_fence_after();
        const uint64_t qd = make_smem_desc(smem_base + (kSplit ? 0 : t * C::kQTile), 16, 1024, 2);
        const uint64_t kd = make_smem_desc(smem_base + C::kKAt + st * C::kQTile, 16, 1024, 2);
        if (elect_one()) {
#pragma unroll
          for (int ks = 0; ks < DQK / 16; ++ks) {
            const uint64_t off = ((ks >> 2) * kPanel + (ks & 3) * 32) >> 4;
            umma_ss<1>(tmem_base + t * 128, qd + off, kd + off, idesc_qk, ks != 0 ? 1u : 0u);
          }
          umma_commit<1>(&bar_s[t]);
          if (kSplit || release_k) umma_commit<1>(&bar_kempty[st]);
          if (kSplit ? t == (nblk_t1 > 0 && nblk_t1 == nblk_t0 ? 1 : 0) && j + 1 == nblk_t0 : last) umma_commit<1>(&bar_qfree[kSplit ? 0 : t]);      // last use of this item's Q_t
        }
      };
      // P V of tile t and block j, then Q K^T of its block j + 1
      auto step = [&](int t, int j, int mine, int other, uint32_t nQ, uint32_t nP) {
        const uint32_t g = kSplit ? g0 + 2 * j + t : g0 + j, vs = g % C::kVStages;
        wait(&bar_vfull[vs], (g / C::kVStages) & 1u);
        wait(&bar_p0[t], nP & 1u);                       // first half of P_t(j) is in TMEM, O_t rescaled if needed
        if (j == 0 && nQ > 0) wait(&bar_ofree[t], (nQ - 1) & 1u);                    // previous item's O_t was read out
        tc_fence_after();
        const uint64_t vd = make_smem_desc(smem_base + C::kVAt + vs * C::kVTile, kPanel, 1024, 2);
        const uint32_t tP = tmem_base + t * 128;
        const uint32_t tOt = tmem_base + 256 + t * 128;
        if (elect_one()) {
#pragma unroll
          for (int ks = 0; ks < kRows / 32; ++ks)
            umma_ts<1>(tOt, tP + ks * 8, vd + ks * (2048 >> 4), idesc_pv, (j | ks) != 0 ? 1u : 0u);
        }
        wait(&bar_p1[t], nP & 1u);
        tc_fence_after();
        if (elect_one()) {
#pragma unroll
          for (int ks = kRows / 32; ks < kRows / 16; ++ks)
            umma_ts<1>(tOt, tP + ks * 8, vd + ks * (2048 >> 4), idesc_pv, 1u);
          if (kSplit || t == 1 || j >= other) umma_commit<1>(&bar_vempty[vs]);    // last reader of V(j)
          if (j + 1 == mine) umma_commit<1>(&bar_o[t]);
        }
        if (j + 1 < mine) issue_qk(t, j + 1, t == 1 || j + 1 >= other, j + 2 == mine);
      };
      wait(&bar_q[0], nQ0 & 1u);
      issue_qk(0, 0, nblk_t1 == 0, nblk_t0 == 1);
      if (nblk_t1 > 0) {
        if (!kSplit) wait(&bar_q[1], nQ1 & 1u);
        issue_qk(1, 0, true, nblk_t1 == 1);
      }
      for (int j = 0; j < nblk; ++j) {
        if (j < nblk_t0) step(0, j, nblk_t0, nblk_t1, nQ0, nP0++);
        if (j < nblk_t1) step(1, j, nblk_t1, nblk_t0, nQ1, nP1++);
      }
      g0 += kSplit ? nblk_t0 + nblk_t1 : nblk;
      ++nQ0;
      if (nblk_t1 > 0) ++nQ1;
    }
   }
  } else {
    setmaxnreg_inc<200>();
    // ---------------------------- softmax warpgroups ----------------------------
    const int t = warp >> 2;
    const int q = warp & 3;                        // TMEM lane quadrant this warp may touch
    const int row = q * 32 + lane;
    const uint32_t lane_off = static_cast<uint32_t>(q * 32) << 16;
    const uint32_t tS = tmem_base + t * 128 + lane_off;
    const uint32_t tOt = tmem_base + 256 + t * 128 + lane_off;
    uint32_t nS = 0;                               // S tiles consumed so far (bar_s phase)
    uint32_t nO = 0, nOb = 0;                      // items finished by this tile (bar_o phase); split items with a second half
    for (int item, r = 0; next_item(r, item); ++r) {
      int q0, head, b;
      Seq sq;
      if (!decode(item, q0, head, b, sq)) continue;
      const int nb = blocks(sq, q0, t);
      if (!kSplit && nb == 0) continue;            // tile B past the end of the sequence: nobody touches its barriers
      const int qt0 = kSplit ? q0 : q0 + t * kRows, first_block = kSplit && t == 1 ? blocks(sq, q0, 0) : 0;
      // a half's reference starts finite: scores of -inf, all that a row may see of it, then weigh nothing instead of being no number
      float m_ref = kSplit ? -FLT_MAX : -INFINITY, l0 = 0.f, l1 = 0.f;
      for (int j = 0; j < nb; ++j, ++nS) {
        mbar_wait_or_abort(&bar_s[t], nS & 1u, abort);
        __syncwarp();
        tc_fence_after();
        if (q == 0 && lane == 0) ev(t, 1);
        const int off = sq.start + qt0 - (first_block + j) * kRows;      // the tile's first row sees the block's columns up to this one
        if (causal && off < kRows - 1)
          softmax_block<true, DV>(tS, tOt, q, lane, off, j == 0, scale_log2, m_ref, l0, l1, &bar_p0[t], &bar_p1[t]);
        else
          softmax_block<false, DV>(tS, tOt, q, lane, off, j == 0, scale_log2, m_ref, l0, l1, &bar_p0[t], &bar_p1[t]);
        if (q == 0 && lane == 0) ev(t, 2);
      }
      // ---- epilogue: O / l -> bf16 -> global (row per thread, whole 32-byte sectors), LSE ----
      float l = l0 + l1, by[2] = {1.f, 1.f};
      const bool both = kSplit && blocks(sq, q0, 1) > 0;
      if constexpr (kSplit) {
        // bar_ofree: the other warpgroup has read what stands there from the item before (and has passed its wait for this barrier's phase)
        if (nO > 0) mbar_wait_or_abort(&bar_ofree[0], (nO - 1) & 1u, abort);
        half_ml[t][row] = make_float2(m_ref, l);
        __syncwarp();
        if (lane == 0) mbar_arrive(&bar_half[t]);
        mbar_wait_or_abort(&bar_half[1 - t], nO & 1u, abort);
        const float2 other = half_ml[1 - t][row];
        const float m = fmaxf(m_ref, other.x);
        by[t] = ex2_approx(m_ref - m);
        by[1 - t] = ex2_approx(other.x - m);
        l = l * by[t] + other.y * by[1 - t];
        m_ref = m;
        if (both) mbar_wait_or_abort(&bar_o[1], nOb++ & 1u, abort);
      }
      mbar_wait_or_abort(&bar_o[kSplit ? 0 : t], nO & 1u, abort);
      __syncwarp();
      ++nO;
      tc_fence_after();
      const float inv_l = 1.f / l;
      constexpr int kChunks = kSplit ? DV / 64 : DV / 32;  // of 32 columns, that this warpgroup stores
      const int c0 = kSplit ? t * kChunks : 0;
      const uint32_t tOa = kSplit ? tmem_base + 256 + lane_off : tOt;
      const bool real = qt0 + row < sq.n;
      const long long tok = seqs != nullptr ? sq.q_row + qt0 + row : static_cast<long long>(b) * max_q + qt0 + row;
      __nv_bfloat16* orow = O + tok * o_tok_stride + head * DV + c0 * 32;
#pragma unroll
      for (int c = 0; c < kChunks; ++c) {
        uint32_t r[32];
        tmem_ld_x32(tOa + (c0 + c) * 32, r);
        if constexpr (kSplit) {
          uint32_t r1[32];
          if (both) tmem_ld_x32(tOa + 128 + (c0 + c) * 32, r1);
          tmem_ld_wait();
#pragma unroll
          for (int e = 0; e < 32; ++e) {
            float x = __uint_as_float(r[e]) * by[0];
            if (both) x += __uint_as_float(r1[e]) * by[1];
            r[e] = __float_as_uint(x);
          }
        } else {
          tmem_ld_wait();
        }
        if (c == kChunks - 1) {                    // O_t is in registers: the next item's P V may overwrite it
          tc_fence_before();
          __syncwarp();
          if (lane == 0) {
            mbar_arrive(&bar_ofree[kSplit ? 0 : t]);
            if (both) mbar_arrive(&bar_ofree[1]);
          }
        }
        if (!real) continue;
#pragma unroll
        for (int gq = 0; gq < 2; ++gq) {
          uint32_t w[8];
#pragma unroll
          for (int e = 0; e < 8; ++e)
            w[e] = pack_bf16x2(__uint_as_float(r[gq * 16 + 2 * e]) * inv_l, __uint_as_float(r[gq * 16 + 2 * e + 1]) * inv_l);
          __nv_bfloat16* dst = orow + c * 32 + gq * 16;
          if (o_wide) {
            st_v8(dst, w);
          } else {
            st_v4(dst, make_uint4(w[0], w[1], w[2], w[3]));
            st_v4(dst + 8, make_uint4(w[4], w[5], w[6], w[7]));
          }
        }
      }
      if (lse != nullptr && real && (!kSplit || t == 0))
        lse[(static_cast<long long>(b) * H + head) * max_q + qt0 + row] = (m_ref + log2f(l)) * 0.6931471805599453f;
      if (q == 0 && lane == 0) ev(t, 3);
    }
  }

  tc_fence_before();
  __syncthreads();
  if (threadIdx.x == 0 && abort_flag) {
    atomicCAS(&g_status, 0u, 1u);
    report_wait(wait_byte);
  }
  if (warp == 9) {
    tc_fence_after();
    tmem_dealloc<1>(tmem_base, 512);
  }
}

// Debug timeline buffer: allocated once when LLMCTL_FLASH_TRACE is set in the environment, NULL otherwise.
static long long* flash_trace_buffer() {
  static long long* buf = nullptr;
  static int init = 0;
  if (!init) {
    init = 1;
    if (getenv("LLMCTL_FLASH_TRACE") != nullptr && cudaMalloc(&buf, 2048 * sizeof(long long)) == cudaSuccess)
      cudaMemset(buf, 0, 2048 * sizeof(long long));
    else
      buf = nullptr;
  }
  return buf;
}

// Persistent launch: one CTA per SM over a heavy-first item list.
template <int DQK, int DV, bool kSplit = false>
static int flash_fwd_launch(const CUtensorMap& q, const CUtensorMap& k, const CUtensorMap& ks, const CUtensorMap& v, void* o,
                            long long o_tok_stride, float* lse, const ffwd::Seq* seqs, int B, int max_q, int H, int head_step, float scale, int causal,
                            cudaStream_t s) {
  using namespace ffwd;
  using C = Cfg<DQK, DV>;
  const cudaError_t e = allow_smem(flash_fwd_kernel<DQK, DV, kSplit>, C::kSmem);
  if (e != cudaSuccess) return static_cast<int>(e);
  constexpr int kItemRows = kSplit ? kRows : 2 * kRows;
  const long long nqb = (max_q + kItemRows - 1) / kItemRows, n_items = nqb * H * B;
  if (n_items >= (1ll << 31) - 2 * kNumSMs) return static_cast<int>(cudaErrorInvalidValue);
  const int grid = n_items < kNumSMs ? static_cast<int>(n_items) : kNumSMs;
  unsigned char* const wait_byte = wait_report(kWaitFlashForward);
  if (wait_byte == nullptr) return static_cast<int>(cudaErrorMemoryAllocation);
  const int wide = o_tok_stride % 16 == 0 && (reinterpret_cast<uintptr_t>(o) & 31) == 0;
  return static_cast<int>(launch_dependent(flash_fwd_kernel<DQK, DV, kSplit>, grid, kThreads, C::kSmem, s, q, k, ks, v, (__nv_bfloat16*)o, o_tok_stride, wide, lse, seqs,
                                           Order{static_cast<int>(n_items), static_cast<int>(nqb), FastDiv(H * B), FastDiv(H)}, max_q, H, head_step, scale * 1.4426950408889634f, causal, wait_byte, flash_trace_buffer()));
}

}  // namespace llmctl

using namespace llmctl;

// Copies the forward kernel's debug event log (2048 int64: per role a count, then (code, clock) pairs; see the
// kernel for roles and codes) to the host.
LLMCTL_API int llmctl_flash_trace_read(long long* host_out) {
  long long* b = flash_trace_buffer();
  if (b == nullptr) return static_cast<int>(cudaErrorNotReady);
  return static_cast<int>(cudaMemcpy(host_out, b, 2048 * sizeof(long long), cudaMemcpyDeviceToHost));
}

// 0 unless a bounded wait of the forward kernel ran out since the last clearing call (synchronises the device).
LLMCTL_API int llmctl_flash_fwd_status(int clear) {
  unsigned int v = 0;
  if (cudaMemcpyFromSymbol(&v, ffwd::g_status, sizeof(v)) != cudaSuccess) return -1;
  if (clear && v != 0) {
    const unsigned int zero = 0;
    (void)cudaMemcpyToSymbol(ffwd::g_status, &zero, sizeof(zero));
  }
  return static_cast<int>(v);
}

// q,k,v: [B, S, H, D] bf16 views, D = 64 or 128, with a common layout: element (b,s,h,d) at ((b*S+s)*tok_stride + h*D + d).
// o: same indexing with o_tok_stride.  lse: fp32 [B, H, S] (may be NULL).  Any S when causal, else a multiple of 128.
LLMCTL_API int llmctl_flash_attn_fwd(const void* q, const void* k, const void* v, void* o, float* lse, int B,
                                     int S, int H, int D, long long q_tok_stride, long long k_tok_stride,
                                     long long v_tok_stride, long long o_tok_stride, float scale, int causal,
                                     void* stream) {
  LLMCTL_BEGIN();
  LLMCTL_REQUIRE((D == 128 || D == 64) && (causal || S % 128 == 0) && B > 0 && S > 0 && H > 0);
  LLMCTL_REQUIRE(q_tok_stride % 8 == 0 && k_tok_stride % 8 == 0 && v_tok_stride % 8 == 0 && o_tok_stride % 8 == 0);
  LLMCTL_REQUIRE(scale > 0.f && (reinterpret_cast<uintptr_t>(o) & 15) == 0);      // q, k, v: the tensor maps check them
  CUtensorMap tq, tk, tv;
  int rc = 0;
  auto mkmap = [&](CUtensorMap* m, const void* base, long long tok, int heads) {
    if (!rc) rc = get_tmap_4d_bf16(m, base, D, heads, S, B, D, tok, static_cast<uint64_t>(S) * tok, 64, 1, ffwd::kRows, 1, 1);
  };
  // q | k | v side by side in a token, as one projection leaves them, are one tensor of 3 H heads: one map instead of three
  const long long step = 2ll * H * D;
  const bool packed = static_cast<const char*>(k) - static_cast<const char*>(q) == step && static_cast<const char*>(v) - static_cast<const char*>(k) == step &&
                      q_tok_stride == k_tok_stride && q_tok_stride == v_tok_stride;
  mkmap(&tq, q, q_tok_stride, packed ? 3 * H : H);
  if (packed) {
    tk = tv = tq;
  } else {
    mkmap(&tk, k, k_tok_stride, H);
    mkmap(&tv, v, v_tok_stride, H);
  }
  if (rc) LLMCTL_FAIL(rc, "tensor map Q / K / V");
  const bool split = split_keys(B * H, (S + ffwd::kRows - 1) / ffwd::kRows, D, causal, kNumSMs);
  rc = (D == 128 ? (split ? flash_fwd_launch<128, 128, true> : flash_fwd_launch<128, 128>) : split ? flash_fwd_launch<64, 64, true> : flash_fwd_launch<64, 64>)(tq, tk, tk, tv, o, o_tok_stride, lse, nullptr, B, S, H,
                                                                          packed ? H : 0, scale, causal, (cudaStream_t)stream);
  if (rc) LLMCTL_FAIL(rc, "flash forward");
  return 0;
}

// Causal attention of latent-attention prompts whose per-head keys and values have been rebuilt from the cache: q: [tokens, H * 192]
// (row stride ldq; the last 64 of a head already rotated), kn: [key_rows, H * 128], kr: [key_rows, 64] shared by all heads, v:
// [key_rows, H * 128], out: [tokens, H * 128].  seqs: int32 [B, 4] on the device = (first query row, queries, position of the first
// query, first key row; key rows in whole blocks of 128, zeros past the last key); max_q: the most queries of a sequence.
LLMCTL_API int llmctl_latent_prompt_attention(const void* q, long long ldq, long long tokens, const void* kn, const void* kr, const void* v,
                                              long long key_rows, const int* seqs, int B, int max_q, int H, void* out, float scale,
                                              void* stream) {
  LLMCTL_BEGIN();
  LLMCTL_REQUIRE(B > 0 && max_q > 0 && H > 0 && tokens > 0 && key_rows > 0 && key_rows % 128 == 0 && ldq % 8 == 0 && scale > 0.f && seqs != nullptr &&
                 (reinterpret_cast<uintptr_t>(out) & 15) == 0);
  CUtensorMap tq, tk, tks, tv;
  int rc = get_tmap_4d_bf16(&tq, q, 192, H, tokens, 1, 192, ldq, ldq * tokens, 64, 1, ffwd::kRows, 1, 1);
  const uint64_t ld = static_cast<uint64_t>(H) * 128;
  if (!rc) rc = get_tmap_4d_bf16(&tk, kn, 128, H, key_rows, 1, 128, ld, ld * key_rows, 64, 1, ffwd::kRows, 1, 1);
  if (!rc) rc = get_tmap_4d_bf16(&tks, kr, 64, 1, key_rows, 1, 64, 64, 64ull * key_rows, 64, 1, ffwd::kRows, 1, 1);
  if (!rc) rc = get_tmap_4d_bf16(&tv, v, 128, H, key_rows, 1, 128, ld, ld * key_rows, 64, 1, ffwd::kRows, 1, 1);
  if (rc) LLMCTL_FAIL(rc, "tensor map q / k / v");
  rc = flash_fwd_launch<192, 128>(tq, tk, tks, tv, out, static_cast<long long>(ld), nullptr, reinterpret_cast<const ffwd::Seq*>(seqs), B, max_q,
                                  H, 0, scale, 1, (cudaStream_t)stream);
  if (rc) LLMCTL_FAIL(rc, "latent prompt attention");
  return 0;
}
