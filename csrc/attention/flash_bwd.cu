// K6 (backward): one deterministic tcgen05 kernel over two kinds of items, head sizes 64 and 128, sequences of any length.
//
//   dKV items   — an item = (batch, head, 128-key block): K_j, V_j resident in shared memory, query blocks of 128 rows
//                 streamed.  It works on the TRANSPOSED scores,
//                     S^T = K_j Q_i^T      dP^T = V_j dO_i^T        (M = 128 keys in TMEM lanes, N = 128 queries)
//                 so that P^T and dS^T — written back by the softmax threads as bf16 over the very TMEM columns they
//                 were read from — are directly the A operands of
//                     dV += P^T dO_i       dK += dS^T Q_i
//   dQ items    — an item = (batch, head, 128-query block): Q_i, dO_i resident, key blocks of 128 streamed;
//                     S = Q_i K_j^T    dP = dO_i V_j^T    dS -> TMEM    dQ += dS K_j
// Recomputing S and dP for the second kind costs 7 products instead of 5, but needs no fp32 accumulator of dQ in memory and
// makes the gradient bit-reproducible.  The 1/sqrt(d) factor of dS is applied once in the dK / dQ epilogues.
//
// What bounds it: the tensor pipe (4 / 3 products of 128 x 128 x D per block pair, 2048 / 1536 clocks at D = 128) against
// 1024 clocks of exponentials and the hand-overs between them.  S and dP are single buffers of 128 columns, and the order of
// issue keeps the pipe busy instead: while the softmax warpgroups turn S(n) into P(n) the pipe runs dK(n-1) and dP(n), while
// they turn dP(n) into dS(n) it runs dV(n) and S(n+1).  (64-row blocks with double buffers, the earlier layout, read 192 bytes
// of operands per clock where shared memory gives 128, and started a CTA per item.)  The streamed tiles Q, dO, Q, dO, ... share
// one ring: with 5 slots beside the two resident tiles (all that 227 KB hold at D = 128) Q(n+1) is fetched as soon as dV(n-2)
// has retired, a block and a half ahead of its use; rings of two stages each left the pipe waiting 200-1000 clocks per block.
// P is handed over in two halves, as in the forward.  Persistent: one CTA per SM claims items, longest of a group first, the dKV
// items of a group of heads before its dQ items.  These read the same tiles again, from L2, and fill the SMs that the last dKV items
// leave idle (8 x 512 x 32 x 128: 94 us in two launches, 88 us in one).  TMEM, barriers and maps are set up once, an item's first
// tiles are fetched while the previous item is still in its softmax, and a warpgroup of its own reads the accumulators out and stores
// them meanwhile (a row per thread: 4900 clocks from the last product to the next item's first softmax when the softmax warps did it,
// against 2900 per block).
//
// A ragged sequence ends inside a block: rows past it are zero-filled by TMA, their statistics make P zero, and they are
// never stored (causal only: keys past the end are then hidden from every real query by the mask).
//
// Reference: autograd through HF attention (reference llmctl/runtime/engine.py:288-291).  Baseline: cuDNN SDPA bwd.
#include <type_traits>

#include "../common/ptx.cuh"
#include "../common/tma_host.h"
#include "../common/util.cuh"
#include "../common/wait_status.h"

namespace llmctl {
using namespace ptx;

namespace fbwd {
constexpr int kBlk = 128;                    // rows of a resident or streamed block
constexpr int kPanel = kBlk * 128;           // bytes of a [128 x 64 bf16] swizzled panel
constexpr int kThreads = 448;                // TMA, MMA issuer, 2 softmax warpgroups, epilogue warpgroup
constexpr int kStatBytes = 2 * kBlk * 4;     // -lse * log2e and -delta of 128 queries
// Items are claimed from a counter by the TMA warp and told to the others through a queue.  It runs at most two items ahead of
// the softmax warps (the resident tiles are single), so a slot is never overwritten before all have read it.
constexpr int kQueue = 4;
// Heads are worked through in groups whose q, k, v and dO stay in L2 (126 MB, with the outputs of the group before) while every
// block of the group streams them again; block by block over all heads, S = 2048 with 80 heads read them from HBM every time.
constexpr long long kGroupBytes = 32ll << 20;
template <int D>
struct Cfg {
  static constexpr int kPanels = D / 64;
  static constexpr int kTile = kPanels * kPanel;
  static constexpr int kSlots = D == 128 ? 5 : 9;                      // streamed tiles: element 2n = operand 0 of block n, 2n + 1 = operand 1
  // statistics of block n go with element 2n + 1, whose slot is free only when operand 0 of block n - (kSlots - 1) / 2 is: by
  // then the softmax is done with that block
  static constexpr int kStatSlots = (kSlots - 1) / 2;
  static constexpr int kStatAt = (2 + kSlots) * kTile;                 // behind all tiles: each starts at a multiple of 1024 bytes
  static constexpr int kBarsAt = kStatAt + kStatSlots * kStatBytes;
  static constexpr int kSmem = kBarsAt + 384;
  static_assert(kSmem <= 227 * 1024, "shared memory");
};
__device__ unsigned int g_status = 0;        // != 0: a bounded wait of the kernel ran out
using DKV = std::integral_constant<bool, false>;
using DQ = std::integral_constant<bool, true>;

struct Maps {
  CUtensorMap q, k, v, d_o;
};
}  // namespace fbwd

// nl2[bh, s] = -lse * log2(e) and ndl[bh, s] = -sum_d dO . O, rows padded to whole blocks with (-inf, 0): P = 0 there.
// D / 8 lanes per row with 16-byte loads, four rows per lane group in flight; bound by HBM (two reads of the activation):
// 4096 tokens x 32 heads x 128 take 13 us; 26 us with 8-byte loads and one row per warp.
template <int D>
__global__ void __launch_bounds__(256)
flash_bwd_prep_kernel(const __nv_bfloat16* __restrict__ O, const __nv_bfloat16* __restrict__ dO, long long tok_stride,
                      const float* __restrict__ lse, float* __restrict__ nl2, float* __restrict__ ndl, int S, int Sp, int H,
                      int chunks, int* __restrict__ counter) {
  if (blockIdx.x == 0 && threadIdx.x == 0) *counter = 0;       // the item counter of the kernel that follows
  constexpr int kLanes = D / 8, kGroups = 256 / kLanes, kRows = 4;
  const int g = threadIdx.x / kLanes, li = threadIdx.x % kLanes;
  const int bh = blockIdx.x / chunks, h = bh % H;
  const long long tok0 = static_cast<long long>(bh / H) * S;
  const int s0 = (blockIdx.x % chunks) * kGroups * kRows + g;
  bf16x8 o[kRows], d[kRows];
#pragma unroll
  for (int u = 0; u < kRows; ++u) {
    const int s = s0 + u * kGroups;
    if (s < S) {
      const long long at = (tok0 + s) * tok_stride + h * D + li * 8;
      o[u] = load8(O + at);
      d[u] = load8(dO + at);
    }
  }
#pragma unroll
  for (int u = 0; u < kRows; ++u) {
    const int s = s0 + u * kGroups;
    float sum = 0.f;
    if (s < S) {
      float a[8], b[8];
      unpack8(o[u], a);
      unpack8(d[u], b);
#pragma unroll
      for (int j = 0; j < 8; ++j) sum += a[j] * b[j];
    }
#pragma unroll
    for (int w = kLanes / 2; w > 0; w >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, w);
    if (li == 0 && s < Sp) {
      const long long i = static_cast<long long>(bh) * Sp + s;
      nl2[i] = s < S ? -lse[static_cast<long long>(bh) * S + s] * 1.4426950408889634f : -INFINITY;
      ndl[i] = -sum;
    }
  }
}

// 16 columns of an fp32 accumulator row -> 16 bf16 at dst (32 bytes)
__device__ __forceinline__ void fbwd_store16(__nv_bfloat16* dst, const uint32_t* r, float mul, bool wide) {
  uint32_t w[8];
#pragma unroll
  for (int e = 0; e < 8; ++e) w[e] = pack_bf16x2(__uint_as_float(r[2 * e]) * mul, __uint_as_float(r[2 * e + 1]) * mul);
  if (wide) {
    st_v8(dst, w);
  } else {
    st_v4(dst, make_uint4(w[0], w[1], w[2], w[3]));
    st_v4(dst + 8, make_uint4(w[4], w[5], w[6], w[7]));
  }
}

// dKV items: resident K, V; streamed Q, dO.  dQ items: resident Q, dO; streamed K, V.  Operand 0 of either pair (K / Q) makes the
// S-like product, operand 1 (V / dO) the dP-like one.
template <int D>
__global__ void __launch_bounds__(fbwd::kThreads, 1)
flash_bwd_kernel(const __grid_constant__ fbwd::Maps maps, const float* __restrict__ nl2, const float* __restrict__ ndl,
                 __nv_bfloat16* __restrict__ dq, __nv_bfloat16* __restrict__ dk, __nv_bfloat16* __restrict__ dv, long long out_tok,
                 int out_wide, int B, int S, int H, int group, int* __restrict__ counter, float scale_log2, float scale, int causal,
                 unsigned char* wait_byte) {
  using namespace fbwd;
  using C = Cfg<D>;
  extern __shared__ __align__(1024) uint8_t smem[];
  struct Bars {
    uint64_t full[C::kSlots], empty[C::kSlots], res, resfree, s, dp, p[2], ds, acc[2], accfree[2], item_full[kQueue];
    int item[kQueue];
    uint32_t tmem;
    int abort;
  };
  static_assert(sizeof(Bars) <= 384, "barriers");
  Bars& bar = *reinterpret_cast<Bars*>(smem + C::kBarsAt);
  const uint32_t smem_base = smem_u32(smem);
  if (smem_base & 1023u) {             // the swizzled tiles would not line up (uniform over the grid)
    if (threadIdx.x == 0) {
      atomicCAS(&g_status, 0u, 16u);
      report_wait(wait_byte);
    }
    return;
  }
  const int warp = __shfl_sync(0xffffffffu, threadIdx.x >> 5, 0), lane = threadIdx.x & 31;
  const int nblk = (S + kBlk - 1) / kBlk, Sp = nblk * kBlk;
  const int BH = B * H, n_items = 2 * nblk * BH;

  if (threadIdx.x == 0) {
    mbar_init(&bar.res, 1);
    mbar_init(&bar.resfree, 1);
    for (int i = 0; i < C::kSlots; ++i) {
      mbar_init(&bar.full[i], 1);
      mbar_init(&bar.empty[i], 1);
    }
    mbar_init(&bar.s, 1);
    mbar_init(&bar.dp, 1);
    mbar_init(&bar.ds, 8);
    for (int i = 0; i < 2; ++i) {
      mbar_init(&bar.p[i], 8);
      mbar_init(&bar.acc[i], 1);
      mbar_init(&bar.accfree[i], 4);
    }
    for (int i = 0; i < kQueue; ++i) mbar_init(&bar.item_full[i], 1);
    bar.abort = 0;
    fence_mbar_init();
  }
  if (warp == 0 && lane == 0) {
    prefetch_tmap(&maps.q);
    prefetch_tmap(&maps.k);
    prefetch_tmap(&maps.v);
    prefetch_tmap(&maps.d_o);
  }
  if (warp == 1) tmem_alloc<1>(&bar.tmem, 512);
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = bar.tmem;
  // A waiter of an mbarrier sees only the parity of its phase, so no barrier may complete its next phase before everyone has passed the
  // wait for this one.  acc[a] (product finished) is therefore committed only after accfree[a] (read out) of the use before has been
  // waited for.  acc[0] is used by every item, acc[1] by dKV items alone, each side counting them.
  // TMEM: S [0,128)  dP [128,256)  acc0 [256,256+D)  acc1 [384,384+D)
  const uint32_t tS = tmem_base, tdP = tmem_base + 128, tAcc0 = tmem_base + 256, tAcc1 = tmem_base + 384;
  volatile int* abort = &bar.abort;

  // item -> (kind, resident block, batch x head) and the streamed blocks [first, first + n); longest items of a group first
  auto decode = [&](int item, bool& is_dq, int& rb, int& bh, int& first, int& n) {
    const int base = item / (2 * group * nblk) * group, heads = min(group, BH - base);
    int rem = item - 2 * base * nblk;
    is_dq = rem >= heads * nblk;
    if (is_dq) rem -= heads * nblk;
    const int k = rem / heads;
    bh = base + rem % heads;
    rb = is_dq ? nblk - 1 - k : k;
    first = (!is_dq && causal) ? rb : 0;
    n = (causal ? (is_dq ? rb + 1 : nblk) : nblk) - first;
  };
  // the k-th item of this CTA, as the TMA warp published it; false when a wait ran out or there is none left
  auto next_item = [&](uint32_t k, int& item) {
    mbar_wait_or_abort(&bar.item_full[k % kQueue], (k / kQueue) & 1u, abort);
    __syncwarp();
    item = __shfl_sync(0xffffffffu, *reinterpret_cast<volatile int*>(&bar.item[k % kQueue]), 0);
    return item < n_items && !*abort;
  };

  if (warp == 0) {
    // ------------------------------------ TMA producer ------------------------------------
    if (lane == 0) {
      uint32_t e = 0, k = 0;           // streamed tiles / items so far
      uint32_t nr = 0;                 // resident pairs begun
      bool ok = true;
      // the next streamed tile: false when its slot does not become free
      auto stream = [&](const CUtensorMap* m, int h, int row, int b, const float* st0, const float* st1) {
        const uint32_t slot = e % C::kSlots;
        if (!mbar_wait_bounded(&bar.empty[slot], ((e / C::kSlots) & 1u) ^ 1u, abort)) return false;
        mbar_expect_tx(&bar.full[slot], C::kTile + (st0 != nullptr ? kStatBytes : 0));
        uint8_t* dst = smem + (2 + slot) * C::kTile;
#pragma unroll
        for (int p = 0; p < C::kPanels; ++p) tma_load_4d(dst + p * kPanel, m, &bar.full[slot], 64 * p, h, row, b);
        if (st0 != nullptr) {
          uint8_t* sStat = smem + C::kStatAt + ((e >> 1) % C::kStatSlots) * kStatBytes;
          bulk_load_1d(sStat, st0, kBlk * 4, &bar.full[slot]);
          bulk_load_1d(sStat + kBlk * 4, st1, kBlk * 4, &bar.full[slot]);
        }
        ++e;
        return true;
      };
      int item = blockIdx.x;
      for (;; ++k) {
        bar.item[k % kQueue] = item;
        mbar_arrive(&bar.item_full[k % kQueue]);
        if (item >= n_items) break;
        const int next = gridDim.x + atomicAdd(counter, 1);
        bool is_dq;
        int rb, bh, first, n;
        decode(item, is_dq, rb, bh, first, n);
        const int h = bh % H, b = bh / H;
        const CUtensorMap *res0 = is_dq ? &maps.q : &maps.k, *res1 = is_dq ? &maps.d_o : &maps.v;
        const CUtensorMap *sub0 = is_dq ? &maps.k : &maps.q, *sub1 = is_dq ? &maps.v : &maps.d_o;
        for (int i = 0; i < n; ++i) {
          const int row = (first + i) * kBlk;
          if (!(ok = stream(sub0, h, row, b, nullptr, nullptr))) break;
          if (i == 0) {                // the resident tiles: free once the previous item's last S and dP have retired
            if (!(ok = mbar_wait_bounded(&bar.resfree, (k & 1u) ^ 1u, abort))) break;
            mbar_expect_tx(&bar.res, 2 * C::kTile);
            ++nr;
#pragma unroll
            for (int p = 0; p < C::kPanels; ++p) {
              tma_load_4d(smem + p * kPanel, res0, &bar.res, 64 * p, h, rb * kBlk, b);
              tma_load_4d(smem + C::kTile + p * kPanel, res1, &bar.res, 64 * p, h, rb * kBlk, b);
            }
          }
          const long long at = static_cast<long long>(bh) * Sp + row;
          if (!(ok = stream(sub1, h, row, b, is_dq ? nullptr : nl2 + at, ndl + at))) break;
        }
        if (!ok) break;
        item = next;
      }
      // Copies still in flight when a wait ran out land before the CTA's shared memory is given back.
      if (!ok) {
        int none = 0;
        for (uint32_t j = e > C::kSlots ? e - C::kSlots : 0; j < e; ++j, none = 0)
          mbar_wait_bounded(&bar.full[j % C::kSlots], (j / C::kSlots) & 1u, &none);
        if (nr > 0) mbar_wait_bounded(&bar.res, (nr - 1) & 1u, &none);
      }
    }
  } else if (warp == 1) {
    // ------------------------------------ MMA issuer ------------------------------------
    // The whole warp walks the loop and waits; only the products and commits are issued by one elected lane.  Addresses and
    // descriptors then stay in uniform registers, which the instruction reads; computed in a single lane's branch they are
    // moved there one by one, and a product of 64 clocks took 85-107 to issue.
    constexpr uint32_t id_s = make_idesc_bf16(kBlk, kBlk, 0u, 0u);     // A, B K-major
    constexpr uint32_t id_acc = make_idesc_bf16(kBlk, D, 0u, 1u);      // A from TMEM, B MN-major
    const uint64_t kRes0 = make_smem_desc(smem_base, 16, 1024, 2), kRes1 = make_smem_desc(smem_base + C::kTile, 16, 1024, 2);
    auto tile_at = [&](uint32_t e) { return smem_base + (2 + e % C::kSlots) * C::kTile; };
    auto wait = [&](uint64_t* b, uint32_t parity) {
      mbar_wait_or_abort(b, parity, abort);
      __syncwarp();
    };
    auto arrived = [&](uint32_t e) { wait(&bar.full[e % C::kSlots], (e / C::kSlots) & 1u); };
    // scores: 16 of the D columns per instruction, a panel of 64 columns every fourth
    auto issue_scores = [&](uint32_t t, uint64_t res, uint32_t sub) {
      const uint64_t b0 = make_smem_desc(sub, 16, 1024, 2);
#pragma unroll
      for (int ks = 0; ks < D / 16; ++ks) {
        const uint64_t off = ((ks >> 2) * kPanel + (ks & 3) * 32) >> 4;
        umma_ss<1>(t, res + off, b0 + off, id_s, ks != 0 ? 1u : 0u);
      }
    };
    // accumulators: 16 of the 128 streamed rows per instruction; the second half of A lies 64 columns on (a softmax
    // warpgroup writes its half over the columns that it has read itself).  part 0 / 1: the rows that both warpgroups write
    // first / last, 2: all.
    auto issue_acc = [&](uint32_t t, uint32_t a, uint32_t sub, uint32_t fresh, int part) {
      const uint64_t b0 = make_smem_desc(sub, kPanel, 1024, 2);
#pragma unroll
      for (int ks = 0; ks < kBlk / 16; ++ks)
        if (part == 2 || ((ks >> 1) & 1) == part)
          umma_ts<1>(t, a + (ks >> 2) * 64 + (ks & 3) * 8, b0 + ((ks * 2048) >> 4), id_acc, ks == 0 ? 1u - fresh : 1u);
    };
    uint32_t g = 0, k = 0, kv = 0;     // blocks, items and dKV items so far
    auto run = [&](auto kind, int n) {
      constexpr bool kDQ = decltype(kind)::value;
      for (int i = 0; i < n; ++i, ++g) {
        const uint32_t e0 = 2 * g, e1 = e0 + 1;            // this block's streamed tiles; the next block's are e0 + 2, e1 + 2
        const uint32_t fresh = i == 0 ? 1u : 0u;
        if (i == 0) {
          arrived(e0);
          tc_fence_after();
          if (elect_one()) {
            issue_scores(tS, kRes0, tile_at(e0));
            umma_commit<1>(&bar.s);
          }
          arrived(e1);
          tc_fence_after();
          if (elect_one()) {
            issue_scores(tdP, kRes1, tile_at(e1));
            umma_commit<1>(&bar.dp);
            if (n == 1) umma_commit<1>(&bar.resfree);
            if (kDQ) umma_commit<1>(&bar.empty[e1 % C::kSlots]);
          }
        }
        if (!kDQ) {
          wait(&bar.p[0], g & 1u);      // half of P(g) is written
          if (i == 0 && k > 0) wait(&bar.accfree[0], (k - 1) & 1u);
          tc_fence_after();
          if (elect_one()) issue_acc(tAcc0, tS, tile_at(e1), fresh, 0);              // dV += P^T dO
        }
        wait(&bar.p[1], g & 1u);        // P(g) written (dKV) / S(g) read (dQ)
        tc_fence_after();
        if (!kDQ && elect_one()) {
          issue_acc(tAcc0, tS, tile_at(e1), 0, 1);
          umma_commit<1>(&bar.empty[e1 % C::kSlots]);
          if (i + 1 == n) umma_commit<1>(&bar.acc[0]);
        }
        if (i + 1 < n) {
          arrived(e0 + 2);
          tc_fence_after();
          if (elect_one()) {
            issue_scores(tS, kRes0, tile_at(e0 + 2));
            umma_commit<1>(&bar.s);
          }
        }
        wait(&bar.ds, g & 1u);
        if (i == 0 && (kDQ ? k : kv) > 0) wait(&bar.accfree[kDQ ? 0 : 1], ((kDQ ? k : kv) - 1) & 1u);
        tc_fence_after();
        if (elect_one()) {
          issue_acc(kDQ ? tAcc0 : tAcc1, tdP, tile_at(e0), fresh, 2);    // dK += dS^T Q  /  dQ += dS K
          umma_commit<1>(&bar.empty[e0 % C::kSlots]);
          if (i + 1 == n) umma_commit<1>(&bar.acc[kDQ ? 0 : 1]);
        }
        if (i + 1 < n) {
          arrived(e1 + 2);
          tc_fence_after();
          if (elect_one()) {
            issue_scores(tdP, kRes1, tile_at(e1 + 2));
            umma_commit<1>(&bar.dp);
            if (i + 2 == n) umma_commit<1>(&bar.resfree);
            if (kDQ) umma_commit<1>(&bar.empty[(e1 + 2) % C::kSlots]);
          }
        }
      }
    };
    for (int item; next_item(k, item); ++k) {
      bool is_dq;
      int rb, bh, first, n;
      decode(item, is_dq, rb, bh, first, n);
      wait(&bar.res, k & 1u);
      if (is_dq) {
        run(DQ{}, n);
      } else {
        run(DKV{}, n);
        ++kv;
      }
    }
  } else if (warp < 10) {
    // ------------------- softmax / dS warpgroups: half wg of the streamed columns, all 128 resident rows -------------------
    const int wg = (warp - 2) >> 2;
    const int q4 = warp & 3;
    const int row = q4 * 32 + lane;                       // resident row == TMEM lane
    const uint32_t lane_off = static_cast<uint32_t>(q4 * 32) << 16;
    const uint32_t tSb = tS + wg * 64 + lane_off, tPb = tdP + wg * 64 + lane_off;
    uint32_t g = 0, k = 0;
    auto run = [&](auto kind, int rb, int bh, int first, int n) {
      constexpr bool kDQ = decltype(kind)::value;
      float row_nl = 0.f, row_nd = 0.f;                   // dQ items: this query row's statistics
      if (kDQ) {
        row_nl = nl2[static_cast<long long>(bh) * Sp + rb * kBlk + row];
        row_nd = ndl[static_cast<long long>(bh) * Sp + rb * kBlk + row];
      }
      for (int i = 0; i < n; ++i, ++g) {
        const float* stat = reinterpret_cast<const float*>(smem + C::kStatAt + (g % C::kStatSlots) * kStatBytes) + wg * 64;
        const uint32_t e1 = 2 * g + 1;                    // the statistics came with this streamed tile
        const bool diag = causal && first + i == rb;
        // columns a row may see on the diagonal block: dKV key `row` <= query, dQ key <= query `row`
        const int edge = row - wg * 64;
        if (!kDQ) mbar_wait_or_abort(&bar.full[e1 % C::kSlots], (e1 / C::kSlots) & 1u, abort);
        mbar_wait_or_abort(&bar.s, g & 1u, abort);
        __syncwarp();
        tc_fence_after();
        uint32_t rs[64];
        tmem_ld_x32(tSb, rs);
        tmem_ld_x32(tSb + 32, rs + 32);
        tmem_ld_wait();
        if (kDQ) {                                        // S is in registers: the next scores may overwrite it
          tc_fence_before();
          __syncwarp();
          if (lane == 0) {
            mbar_arrive(&bar.p[0]);                       // every block completes both halves: phases follow the blocks
            mbar_arrive(&bar.p[1]);
          }
        }
#pragma unroll
        for (int c = 0; c < 4; ++c) {
          uint32_t pk[8];
#pragma unroll
          for (int e = c * 16; e < c * 16 + 16; e += 4) {
            float a0, a1, a2, a3;
            if (kDQ) {
              fma2(a0, a1, __uint_as_float(rs[e]), __uint_as_float(rs[e + 1]), scale_log2, row_nl);
              fma2(a2, a3, __uint_as_float(rs[e + 2]), __uint_as_float(rs[e + 3]), scale_log2, row_nl);
            } else {
              const float4 nl = *reinterpret_cast<const float4*>(stat + e);          // warp-uniform
              fma2v(a0, a1, __uint_as_float(rs[e]), __uint_as_float(rs[e + 1]), scale_log2, nl.x, nl.y);
              fma2v(a2, a3, __uint_as_float(rs[e + 2]), __uint_as_float(rs[e + 3]), scale_log2, nl.z, nl.w);
            }
            float p0 = ex2_approx(a0), p1 = ex2_approx(a1), p2 = ex2_approx(a2), p3 = ex2_approx(a3);
            if (diag) {
              if (kDQ ? (e > edge) : (e < edge)) p0 = 0.f;
              if (kDQ ? (e + 1 > edge) : (e + 1 < edge)) p1 = 0.f;
              if (kDQ ? (e + 2 > edge) : (e + 2 < edge)) p2 = 0.f;
              if (kDQ ? (e + 3 > edge) : (e + 3 < edge)) p3 = 0.f;
            }
            if (!kDQ) {
              pk[((e & 15) >> 1)] = pack_bf16x2(p0, p1);
              pk[((e & 15) >> 1) + 1] = pack_bf16x2(p2, p3);
            }
            rs[e] = __float_as_uint(p0);
            rs[e + 1] = __float_as_uint(p1);
            rs[e + 2] = __float_as_uint(p2);
            rs[e + 3] = __float_as_uint(p3);
          }
          if (!kDQ) {
            tmem_st_x8(tSb + c * 8, pk);
            if (c & 1) {
              tmem_st_wait();
              tc_fence_before();
              __syncwarp();
              if (lane == 0) mbar_arrive(&bar.p[c >> 1]);
            }
          }
        }
        mbar_wait_or_abort(&bar.dp, g & 1u, abort);
        __syncwarp();
        tc_fence_after();
#pragma unroll
        for (int half = 0; half < 2; ++half) {
          uint32_t rp[32], dk[16];
          tmem_ld_x32(tPb + half * 32, rp);
          tmem_ld_wait();
#pragma unroll
          for (int e = 0; e < 32; e += 4) {
            const int col = half * 32 + e;
            float t0, t1, t2, t3, d0, d1, d2, d3;
            if (kDQ) {
              add2v(t0, t1, __uint_as_float(rp[e]), __uint_as_float(rp[e + 1]), row_nd, row_nd);
              add2v(t2, t3, __uint_as_float(rp[e + 2]), __uint_as_float(rp[e + 3]), row_nd, row_nd);
            } else {
              const float4 nd = *reinterpret_cast<const float4*>(stat + kBlk + col);
              add2v(t0, t1, __uint_as_float(rp[e]), __uint_as_float(rp[e + 1]), nd.x, nd.y);
              add2v(t2, t3, __uint_as_float(rp[e + 2]), __uint_as_float(rp[e + 3]), nd.z, nd.w);
            }
            mul2v(d0, d1, __uint_as_float(rs[col]), __uint_as_float(rs[col + 1]), t0, t1);
            mul2v(d2, d3, __uint_as_float(rs[col + 2]), __uint_as_float(rs[col + 3]), t2, t3);
            dk[e >> 1] = pack_bf16x2(d0, d1);
            dk[(e >> 1) + 1] = pack_bf16x2(d2, d3);
          }
          tmem_st_x16(tPb + half * 16, dk);
        }
        tmem_st_wait();
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(&bar.ds);
      }
    };
    for (int item; next_item(k, item); ++k) {
      bool is_dq;
      int rb, bh, first, n;
      decode(item, is_dq, rb, bh, first, n);
      if (is_dq) run(DQ{}, rb, bh, first, n); else run(DKV{}, rb, bh, first, n);
    }
  } else {
    // ------------- epilogue warpgroup: accumulators -> registers -> bf16 -> global, a row per thread -------------
    const int q4 = warp & 3;
    const int row = q4 * 32 + lane;
    const uint32_t lane_off = static_cast<uint32_t>(q4 * 32) << 16;
    uint32_t k = 0, kv = 0;            // items and dKV items so far
    for (int item; next_item(k, item); ++k) {
      bool is_dq;
      int rb, bh, first, n;
      decode(item, is_dq, rb, bh, first, n);
      const bool real = rb * kBlk + row < S;
      const long long at = (static_cast<long long>(bh / H) * S + rb * kBlk + row) * out_tok + (bh % H) * D;
#pragma unroll 1
      for (int a = 0; a < (is_dq ? 1 : 2); ++a) {         // dKV: dV from acc0, then scale * dK from acc1.  dQ: scale * dQ from acc0.
        mbar_wait_or_abort(&bar.acc[a], (a == 0 ? k : kv) & 1u, abort);
        __syncwarp();
        tc_fence_after();
        const uint32_t tA = (a == 0 ? tAcc0 : tAcc1) + lane_off;
        const float mul = (is_dq || a == 1) ? scale : 1.f;
        __nv_bfloat16* dst = (is_dq ? dq : a == 0 ? dv : dk) + at;
#pragma unroll
        for (int c0 = 0; c0 < D; c0 += 64) {
          uint32_t r[64];
          tmem_ld_x32(tA + c0, r);
          tmem_ld_x32(tA + c0 + 32, r + 32);
          tmem_ld_wait();
          if (c0 + 64 == D) {                             // in registers: the next item may overwrite it
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(&bar.accfree[a]);
          }
          if (real) {
#pragma unroll
            for (int c = 0; c < 64; c += 16) fbwd_store16(dst + c0 + c, r + c, mul, out_wide);
          }
        }
      }
      if (!is_dq) ++kv;
    }
  }

  tc_fence_before();
  __syncthreads();
  if (threadIdx.x == 0 && bar.abort) {
    atomicCAS(&g_status, 0u, 1u);
    report_wait(wait_byte);
  }
  if (warp == 1) {
    tc_fence_after();
    tmem_dealloc<1>(tmem_base, 512);
  }
}

template <int D>
static int flash_bwd_launch(const void* q, const void* k, const void* v, const void* o, const void* d_o, const float* lse, void* dq,
                            void* dk, void* dv, float* scratch, int B, int S, int H, long long q_tok, long long k_tok, long long v_tok,
                            long long o_tok, long long dqkv_tok, float scale, int causal, cudaStream_t s) {
  using namespace fbwd;
  using C = Cfg<D>;
  const int nblk = (S + kBlk - 1) / kBlk, Sp = nblk * kBlk;
  float *nl2 = scratch, *ndl = scratch + static_cast<long long>(B) * H * Sp;
  int* counter = reinterpret_cast<int*>(ndl + static_cast<long long>(B) * H * Sp);
  const long long head_bytes = 4ll * Sp * D * 2, fit = kGroupBytes / head_bytes;
  const int group = static_cast<int>(fit < 1 ? 1 : fit < B * H ? fit : B * H);
  constexpr int kPrepRows = 256 / (D / 8) * 4;
  const int chunks = (Sp + kPrepRows - 1) / kPrepRows;
  flash_bwd_prep_kernel<D><<<chunks * B * H, 256, 0, s>>>((const __nv_bfloat16*)o, (const __nv_bfloat16*)d_o, o_tok, lse, nl2, ndl, S, Sp,
                                                          H, chunks, counter);
  CUtensorMap mq, mk, mv, mdo;
  int rc = 0;
  auto mkmap = [&](CUtensorMap* m, const void* base, long long tok) {
    if (!rc) rc = get_tmap_4d_bf16(m, base, D, H, S, B, D, tok, static_cast<uint64_t>(S) * tok, 64, 1, kBlk, 1, 1);
  };
  mkmap(&mq, q, q_tok);
  mkmap(&mk, k, k_tok);
  mkmap(&mv, v, v_tok);
  mkmap(&mdo, d_o, o_tok);
  if (rc) return rc;
  unsigned char* const wait_byte = wait_report(kWaitFlashBackward);
  if (wait_byte == nullptr) return static_cast<int>(cudaErrorMemoryAllocation);
  const cudaError_t e = allow_smem(flash_bwd_kernel<D>, C::kSmem);
  if (e != cudaSuccess) return static_cast<int>(e);
  const int n_items = 2 * nblk * B * H, grid = n_items < kNumSMs ? n_items : kNumSMs;
  const int wide = dqkv_tok % 16 == 0 && ((reinterpret_cast<uintptr_t>(dq) | reinterpret_cast<uintptr_t>(dk) | reinterpret_cast<uintptr_t>(dv)) & 31) == 0;
  flash_bwd_kernel<D><<<grid, kThreads, C::kSmem, s>>>(Maps{mq, mk, mv, mdo}, nl2, ndl, (__nv_bfloat16*)dq, (__nv_bfloat16*)dk, (__nv_bfloat16*)dv,
                                                       dqkv_tok, wide, B, S, H, group, counter, scale * 1.4426950408889634f, scale, causal, wait_byte);
  return static_cast<int>(cudaGetLastError());
}

}  // namespace llmctl

using namespace llmctl;

// q,k,v,o,do: [B,S,H,D] bf16 views, D = 64 or 128 (token strides given in elements, a batch S tokens on; do and o share
// o_tok_stride); dq,dk,dv: outputs with token stride dqkv_tok_stride; lse: fp32 [B,H,S] from the forward;
// scratch: fp32 [2 * B * H * (S rounded up to 128) + 2]: per-row log-sum-exp and delta, item counter.
// Any S when causal, else a multiple of 128.
LLMCTL_API int llmctl_flash_attn_bwd(const void* q, const void* k, const void* v, const void* o, const void* d_o,
                                     const float* lse, void* dq, void* dk, void* dv, float* scratch, int B, int S,
                                     int H, int D, long long q_tok_stride, long long k_tok_stride,
                                     long long v_tok_stride, long long o_tok_stride, long long dqkv_tok_stride,
                                     float scale, int causal, void* stream) {
  LLMCTL_BEGIN();
  LLMCTL_REQUIRE((D == 128 || D == 64) && (causal || S % 128 == 0) && B > 0 && S > 0 && H > 0);
  LLMCTL_REQUIRE(static_cast<long long>(B) * H * ((S + 31) / 32) < (1ll << 31));
  LLMCTL_REQUIRE(q_tok_stride % 8 == 0 && k_tok_stride % 8 == 0 && v_tok_stride % 8 == 0 && o_tok_stride % 8 == 0 &&
                 dqkv_tok_stride % 8 == 0);
  LLMCTL_REQUIRE(((reinterpret_cast<uintptr_t>(q) | reinterpret_cast<uintptr_t>(k) | reinterpret_cast<uintptr_t>(v) | reinterpret_cast<uintptr_t>(o) |
                   reinterpret_cast<uintptr_t>(d_o) | reinterpret_cast<uintptr_t>(dq) | reinterpret_cast<uintptr_t>(dk) |
                   reinterpret_cast<uintptr_t>(dv) | reinterpret_cast<uintptr_t>(scratch)) & 15) == 0);
  const int rc = (D == 128 ? flash_bwd_launch<128> : flash_bwd_launch<64>)(
      q, k, v, o, d_o, lse, dq, dk, dv, scratch, B, S, H, q_tok_stride, k_tok_stride, v_tok_stride, o_tok_stride, dqkv_tok_stride, scale,
      causal, (cudaStream_t)stream);
  if (rc) LLMCTL_FAIL(rc, "flash backward");
  return 0;
}

// 0 unless a bounded wait of the backward kernels ran out since the last clearing call (synchronises the device).
LLMCTL_API int llmctl_flash_bwd_status(int clear) {
  unsigned int v = 0;
  if (cudaMemcpyFromSymbol(&v, fbwd::g_status, sizeof(v)) != cudaSuccess) return -1;
  if (clear && v != 0) {
    const unsigned int zero = 0;
    (void)cudaMemcpyToSymbol(fbwd::g_status, &zero, sizeof(zero));
  }
  return static_cast<int>(v);
}
