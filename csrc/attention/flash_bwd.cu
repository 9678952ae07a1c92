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
// What bounds it: the softmax warps, 1600 clocks from S to P and 550 from dP to dS for a 128 x 128 block (1024 of exponentials alone), beside
// 2048 / 1536 clocks of tensor pipe (4 / 3 products of 128 x 128 x D at D = 128): 2740 clocks per dKV block, 2400 per dQ block.  S and dP
// are single buffers of 128 columns (with the accumulators all of TMEM), and the order of issue keeps the pipe busy instead: while the
// softmax warpgroups turn S(n) into P(n) the pipe runs dK(n-1) and dP(n), while they turn dP(n) into dS(n) it runs dV(n) and S(n+1).
// (64-row blocks with double buffers, an earlier layout, read 192 bytes of operands per clock where shared memory gives 128.)  P is handed
// over in two halves, as in the forward.
// The blocks of all items make one stream: an item's resident and streamed tiles share six slots that are handed on in the order of
// their last use, so the next item's first tiles are there and its first scores are made while this one's last block is in its softmax.
// (With two slots for the resident tiles alone these could only be fetched when the item before had let go of them: 4500 clocks between
// items, as long as one and a half blocks.)  Two warps issue the products: one could not wait, work out addresses and issue 32 products in
// the time that they take.  A warpgroup of its own reads the accumulators out, through a seventh slot and TMA stores (a row per
// thread straight to memory slowed the softmax warps' own loads twofold meanwhile).
// Persistent: one CTA per SM claims items, longest of a group first, the dKV items of a group of heads before its dQ items.  These
// read the same tiles again, from L2, and fill the SMs that the last dKV items leave idle.
// Before / after (one stream of blocks, two issuers, TMA stores): 8 x 512 x 32 x 128 105.6 / 96.3 us with the statistics pass, 2 x 2048 x 40 x 128
// 282 / 269, 1 x 4096 x 32 x 128 397 / 377, 8 x 512 x 12 x 64 32.7 / 28.1, 1 x 2048 x 33 x 64 110 / 104.
// Tried: dS^T kept in memory for the dQ items instead of the scores made again (5 products for 7): 399 us for 282, the dQ items wait for
// the last dKV items of their head.
//
// A ragged sequence ends inside a block: rows past it are zero-filled by TMA, their statistics make P zero, and they are
// never stored (causal only: keys past the end are then hidden from every real query by the mask).
//
// Reference: autograd through HF attention (reference llmctl/runtime/engine.py:288-291).  Baseline: cuDNN SDPA bwd.
#include <type_traits>

#include "../common/ptx.cuh"
#include "../common/tma_host.h"
#include "../common/util.cuh"
#include "../common/dependent.cuh"
#include "../common/fast_div.h"
#include "../common/wait_status.h"
#include "flash_bwd_slots.cuh"

namespace llmctl {
using namespace ptx;

namespace fbwd {
constexpr int kBlk = 128;                    // rows of a resident or streamed block
constexpr int kPanel = kBlk * 128;           // bytes of a [128 x 64 bf16] swizzled panel
constexpr int kThreads = 480;                // TMA, issuer A, 2 softmax warpgroups, epilogue warpgroup, issuer B
constexpr int kStatBytes = 2 * kBlk * 4;     // -lse * log2e and -delta of 128 queries
// Items are claimed from a counter by the TMA warp and told to the others through a queue.  When item m is published all tiles of item
// m - 1 are on their way, so item m - 3 has handed all of its back and item m - 4 has been read out: everyone has read the slot of item m - 8.
constexpr int kQueue = 8;
constexpr int kRing = 16;                    // barriers for loads and for hand-backs
// Heads are worked through in groups whose q, k, v and dO stay in L2 (126 MB, with the outputs of the group before) while every
// block of the group streams them again; block by block over all heads, S = 2048 with 80 heads read them from HBM every time.
constexpr long long kGroupBytes = 32ll << 20;
template <int D>
struct Cfg {
  static constexpr int kPanels = D / 64;
  static constexpr int kTile = kPanels * kPanel;
  static constexpr int kOutAt = kTiles * kTile;                       // a tile of gradients on its way out
  static constexpr int kStatSlots = D == 128 ? 2 : 4;
  static constexpr int kStatAt = kOutAt + kTile;                       // behind all tiles: each starts at a multiple of 1024 bytes
  static constexpr int kBarsAt = kStatAt + kStatSlots * kStatBytes;
  static constexpr int kSmem = kBarsAt + 640;
  static_assert(kSmem <= 227 * 1024, "shared memory");
};
__device__ unsigned int g_status = 0;        // != 0: a bounded wait of the kernel ran out
using DKV = std::integral_constant<bool, false>;
using DQ = std::integral_constant<bool, true>;

struct Maps {
  CUtensorMap q, k, v, d_o, dq, dk, dv;
};
// Items are numbered through (group of heads, dKV then dQ, block, head of the group).  With divisions the decoding held an item's first loads back by
// 700 clocks (with the statistics pass: 8 x 512 x 32 x 128 99.0 us, now 96.0; 8 x 512 x 12 x 64 27.9 / 26.9; 2 x 300 x 12 x 64 12.7 / 11.6).
struct Order {
  int n_items, group, heads;                 // heads: batch x head
  FastDiv items_of_group, of_group, of_last, H;
  Order(int nblk, int group_, int heads_, int H_)
      : n_items(2 * nblk * heads_), group(group_), heads(heads_), items_of_group(2 * group_ * nblk), of_group(group_), of_last((heads_ - 1) % group_ + 1), H(H_) {}
};
struct Item {
  bool dq;
  int rb, bh, first, n;      // resident block, batch x head, streamed blocks [first, first + n)
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
  wait_for_previous(O, dO, lse, nl2, ndl, counter);
  release_dependents();
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

// dKV items: resident K, V; streamed Q, dO.  dQ items: resident Q, dO; streamed K, V.  Operand 0 of either pair (K / Q) makes the
// S-like product, operand 1 (V / dO) the dP-like one.
template <int D>
__global__ void __launch_bounds__(fbwd::kThreads, 1)
flash_bwd_kernel(const __grid_constant__ fbwd::Maps maps, const float* __restrict__ nl2, const float* __restrict__ ndl,
                 int in_step, int out_step, int S, const fbwd::Order order, int* __restrict__ counter, float scale_log2, float scale, int causal,
                 unsigned char* wait_byte) {
  using namespace fbwd;
  using C = Cfg<D>;
  extern __shared__ __align__(1024) uint8_t smem[];
  struct Bars {
    uint64_t full[kRing], given[kRing], stat_full[C::kStatSlots], stat_free[C::kStatSlots], s, dp, p[2], ds, acc[2], accfree[2], item_full[kQueue];
    int4 item[kQueue];                 // Item as the TMA warp decoded it; no blocks: the end
    uint32_t tmem;
    int abort;
  };
  static_assert(sizeof(Bars) <= 640, "barriers");
  Bars& bar = *reinterpret_cast<Bars*>(smem + C::kBarsAt);
  const uint32_t smem_base = smem_u32(smem);
  if (smem_base & 1023u) {             // the swizzled tiles would not line up (uniform over the grid)
    wait_for_previous();
    if (threadIdx.x == 0) {
      atomicCAS(&g_status, 0u, 16u);
      report_wait(wait_byte);
    }
    return;
  }
  const int warp = __shfl_sync(0xffffffffu, threadIdx.x >> 5, 0), lane = threadIdx.x & 31;
  const int nblk = (S + kBlk - 1) / kBlk, Sp = nblk * kBlk;

  if (threadIdx.x == 0) {
    for (int i = 0; i < kRing; ++i) {
      mbar_init(&bar.full[i], 1);
      mbar_init(&bar.given[i], 2);     // e1 is read by both issuers
    }
    for (int i = 0; i < C::kStatSlots; ++i) {
      mbar_init(&bar.stat_full[i], 1);
      mbar_init(&bar.stat_free[i], 1);
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
    prefetch_tmap(&maps.dq);
    prefetch_tmap(&maps.dk);
    prefetch_tmap(&maps.dv);
  }
  if (warp == 1) tmem_alloc<1>(&bar.tmem, 512);
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = bar.tmem;
  wait_for_previous();                 // what is read comes by bulk copies and an atomic
  // A waiter of an mbarrier sees only the parity of its phase, so no barrier may complete its next phase before everyone has passed the
  // wait for this one.  acc[a] (product finished) is therefore committed only after accfree[a] (read out) of the use before has been
  // waited for.  acc[0] is used by dKV items alone, acc[1] by every item, each side counting them.
  // TMEM: S [0,128)  dP [128,256)  acc0 [256,256+D)  acc1 [384,384+D)
  const uint32_t tS = tmem_base, tdP = tmem_base + 128, tAcc0 = tmem_base + 256, tAcc1 = tmem_base + 384;
  volatile int* abort = &bar.abort;

  // longest items of a group first
  auto decode = [&](int item) {
    Item it{};
    if (item >= order.n_items) return it;
    uint32_t rem, head;
    const int base = static_cast<int>(order.items_of_group.divide(item, rem)) * order.group, heads = min(order.group, order.heads - base);
    it.dq = rem >= heads * nblk;
    if (it.dq) rem -= heads * nblk;
    const int k = static_cast<int>((heads == order.group ? order.of_group : order.of_last).divide(rem, head));
    it.bh = base + static_cast<int>(head);
    it.rb = it.dq ? nblk - 1 - k : k;
    it.first = (!it.dq && causal) ? it.rb : 0;
    it.n = (causal ? (it.dq ? it.rb + 1 : nblk) : nblk) - it.first;
    return it;
  };
  // the k-th item of this CTA, as the TMA warp published it; false when a wait ran out or
  // there is none left
  auto next_item = [&](uint32_t k, Item& it) {
    mbar_wait_or_abort(&bar.item_full[k % kQueue], (k / kQueue) & 1u, abort);
    const int4 w = bar.item[k % kQueue];
    __syncwarp();
    it.dq = __shfl_sync(0xffffffffu, w.x & 1, 0) != 0;
    it.rb = __shfl_sync(0xffffffffu, w.x >> 1, 0);
    it.bh = __shfl_sync(0xffffffffu, w.y, 0);
    it.first = __shfl_sync(0xffffffffu, w.z, 0);
    it.n = __shfl_sync(0xffffffffu, *abort ? 0 : w.w, 0);
    return it.n > 0;
  };

  if (warp == 0) {
    // ------------------------------------ TMA producer ------------------------------------
    if (lane == 0) {
      uint32_t l = 0, k = 0, gs = 0;   // loads, items and blocks with statistics so far
      bool ok = true;
      Slots sl;
      // the next tile: false when its slot is not handed back
      auto load = [&](uint32_t slot, const CUtensorMap* m, int h, int row, int b) {
        const uint32_t j = l - kTiles;
        if (l >= kTiles && !mbar_wait_bounded(&bar.given[j % kRing], (j / kRing) & 1u, abort)) return false;
        uint64_t* full = &bar.full[l % kRing];
        mbar_expect_tx(full, C::kTile);
        uint8_t* dst = smem + slot * C::kTile;
#pragma unroll
        for (int p = 0; p < C::kPanels; ++p) tma_load_4d(dst + p * kPanel, m, full, 64 * p, h, row, b);
        ++l;
        return true;
      };
      auto load_stats = [&](long long at) {
        const uint32_t slot = gs % C::kStatSlots;
        if (!mbar_wait_bounded(&bar.stat_free[slot], ((gs / C::kStatSlots) & 1u) ^ 1u, abort)) return false;
        mbar_expect_tx(&bar.stat_full[slot], kStatBytes);
        uint8_t* dst = smem + C::kStatAt + slot * kStatBytes;
        bulk_load_1d(dst, nl2 + at, kBlk * 4, &bar.stat_full[slot]);
        bulk_load_1d(dst + kBlk * 4, ndl + at, kBlk * 4, &bar.stat_full[slot]);
        ++gs;
        return true;
      };
      for (int item = blockIdx.x, next = 0;; ++k, item = next) {
        const Item it = decode(item);
        bar.item[k % kQueue] = make_int4(it.rb * 2 + (it.dq ? 1 : 0), it.bh, it.first, it.n);
        mbar_arrive(&bar.item_full[k % kQueue]);
        if (it.n == 0) break;
        uint32_t head;
        const int b = static_cast<int>(order.H.divide(it.bh, head)), h = static_cast<int>(head);
        const CUtensorMap *res0 = it.dq ? &maps.q : &maps.k, *res1 = it.dq ? &maps.d_o : &maps.v;
        const CUtensorMap *sub0 = it.dq ? &maps.k : &maps.q, *sub1 = it.dq ? &maps.v : &maps.d_o;
        const int hr0 = it.dq ? h : h + in_step, hr1 = it.dq ? h : h + 2 * in_step, hs0 = it.dq ? h + in_step : h, hs1 = it.dq ? h + 2 * in_step : h;
        const long long stat = static_cast<long long>(it.bh) * Sp;
        for (int i = 0; ok && i < it.n; ++i) {
          const int row = (it.first + i) * kBlk;
          // claimed as late as its latency can be hidden: what a CTA holds nobody else can begin
          if (i == max(0, it.n - 2)) next = gridDim.x + atomicAdd(counter, 1);
          ok = (i > 0 || load(sl.res(0), res0, hr0, it.rb * kBlk, b)) && load(sl.streamed(0, i), sub0, hs0, row, b) &&
               (i > 0 || load(sl.res(1), res1, hr1, it.rb * kBlk, b)) && load(sl.streamed(1, i), sub1, hs1, row, b) && (it.dq ? i > 0 || load_stats(stat + it.rb * kBlk) : load_stats(stat + row));
        }
        if (!ok) break;
        sl.next(it.n);
      }
      release_dependents();
      // Copies still in flight when a wait ran out land before the CTA's shared memory is given back.
      if (!ok) {
        int none = 0;
        for (uint32_t j = l > kTiles ? l - kTiles : 0; j < l; ++j, none = 0) mbar_wait_bounded(&bar.full[j % kRing], (j / kRing) & 1u, &none);
        for (uint32_t j = gs > C::kStatSlots ? gs - C::kStatSlots : 0; j < gs; ++j, none = 0)
          mbar_wait_bounded(&bar.stat_full[j % C::kStatSlots], (j / C::kStatSlots) & 1u, &none);
      }
    }
  } else if (warp == 1 || warp == 14) {
    // ------------------------------------ MMA issuers ------------------------------------
    // Two warps: A issues S and dV, B dP and dK / dQ.  They share no accumulator and no order: a product waits in its warp for the one
    // whose operand it writes over.  The tensor pipe takes few products ahead, so what one warp spends on waits, addresses and descriptors
    // between its products (300-500 clocks) left the pipe idle; now the other warp's products run meanwhile.
    // A whole warp walks the loop and waits; only the products and commits are issued by one elected lane.
    const bool is_a = warp == 1;
    constexpr uint32_t id_s = make_idesc_bf16(kBlk, kBlk, 0u, 0u);     // A, B K-major
    constexpr uint32_t id_acc = make_idesc_bf16(kBlk, D, 0u, 1u);      // A from TMEM, B MN-major
    const uint32_t tScore = is_a ? tS : tdP, tAcc = is_a ? tAcc0 : tAcc1;
    const int mine = is_a ? 0 : 1;     // the operand of this warp's scores; its gradients read the other
    auto tile_at = [&](uint32_t slot) { return smem_base + slot * C::kTile; };
    auto wait = [&](uint64_t* b, uint32_t parity) {
      mbar_wait_or_abort(b, parity, abort);
      __syncwarp();
    };
    auto arrived = [&](uint32_t l) { wait(&bar.full[l % kRing], (l / kRing) & 1u); };
    auto given = [&](uint32_t j) { return &bar.given[j % kRing]; };
    // scores: 16 of the D columns per instruction, a panel of 64 columns every fourth
    auto issue_scores = [&](uint32_t res_at, uint32_t sub) {
      const uint64_t a0 = make_smem_desc(res_at, 16, 1024, 2), b0 = make_smem_desc(sub, 16, 1024, 2);
#pragma unroll
      for (int ks = 0; ks < D / 16; ++ks) {
        const uint64_t off = ((ks >> 2) * kPanel + (ks & 3) * 32) >> 4;
        umma_ss<1>(tScore, a0 + off, b0 + off, id_s, ks != 0 ? 1u : 0u);
      }
    };
    // accumulators: 16 of the 128 streamed rows per instruction; the second half of A lies 64 columns on (a softmax
    // warpgroup writes its half over the columns that it has read itself).  part 0 / 1: the rows that both warpgroups write
    // first / last, 2: all.
    auto issue_acc = [&](uint32_t sub, uint32_t fresh, int part) {
      const uint64_t b0 = make_smem_desc(sub, kPanel, 1024, 2);
#pragma unroll
      for (int ks = 0; ks < kBlk / 16; ++ks)
        if (part == 2 || ((ks >> 1) & 1) == part)
          umma_ts<1>(tAcc, tScore + (ks >> 2) * 64 + (ks & 3) * 8, b0 + ((ks * 2048) >> 4), id_acc, ks == 0 ? 1u - fresh : 1u);
    };
    // The block whose scores are issued next runs ahead of the one whose gradients are, across the ends of items.
    Item it{};                         // its item, block in it, slots
    int i = 0;
    Slots sl;
    uint32_t k = 0;
    auto advance = [&]() {
      if (++i < it.n) return true;
      if (it.n > 0) sl.next(it.n);
      i = 0;
      return next_item(k++, it);
    };
    uint32_t at_res = 0, at_sub = 0;
    auto scores_ready = [&]() {
      if (i == 0) arrived(sl.load_res(mine));
      arrived(sl.load_streamed(mine, i));
      at_res = tile_at(sl.res(mine));
      at_sub = tile_at(sl.streamed(mine, i));
    };
    auto scores = [&]() {              // one lane
      issue_scores(at_res, at_sub);
      umma_commit<1>(is_a ? &bar.s : &bar.dp);
      if (!is_a) {
        uint64_t* b = given(sl.given_streamed(1, i, it.n));
        if (it.dq) mbar_arrive(b);     // A has no use for it
        umma_commit<1>(b);
      }
      if (i + 1 == it.n) {
        uint64_t* b = given(sl.given_res(mine, it.n));
        mbar_arrive(b);
        umma_commit<1>(b);
      }
    };
    bool more = advance();
    if (more) {
      scores_ready();
      tc_fence_after();
      if (elect_one()) scores();
    }
    uint32_t uses = 0;                 // of this warp's accumulator
    for (uint32_t g = 0, gs = 0; more; ++g) {
      const bool kdq = it.dq, last = i + 1 == it.n;
      const uint32_t fresh = i == 0 ? 1u : 0u, l1 = sl.load_streamed(1, i), at = tile_at(sl.streamed(1 - mine, i));
      uint64_t* const back = given(sl.given_streamed(1 - mine, i, it.n));
      more = advance();
      if (more) scores_ready();
      if (is_a) {
        if (!kdq) {
          arrived(l1);
          if (fresh) wait(&bar.accfree[0], (uses & 1u) ^ 1u);
          wait(&bar.p[0], g & 1u);      // half of P(g) is written
          tc_fence_after();
          if (elect_one()) issue_acc(at, fresh, 0);                    // dV += P^T dO
        }
        wait(&bar.p[1], g & 1u);        // P(g) written (dKV) / S(g) read (dQ)
        tc_fence_after();
        if (elect_one()) {
          if (!kdq) {
            issue_acc(at, 0, 1);
            umma_commit<1>(back);
            if (last) umma_commit<1>(&bar.acc[0]);
          }
          if (more) scores();
        }
        if (!kdq && last) ++uses;
      } else {
        if (fresh) wait(&bar.accfree[1], (uses & 1u) ^ 1u);
        wait(&bar.ds, g & 1u);
        tc_fence_after();
        if (elect_one()) {
          issue_acc(at, fresh, 2);                                     // dK += dS^T Q  /  dQ += dS K
          mbar_arrive(back);
          umma_commit<1>(back);
          if (last) umma_commit<1>(&bar.acc[1]);
          if (more) scores();
          if (!kdq || last) mbar_arrive(&bar.stat_free[gs % C::kStatSlots]);     // dS(g) is written: its statistics have been read
        }
        if (!kdq || last) ++gs;
        if (last) ++uses;
      }
    }
  } else if (warp < 10) {
    // ------------------- softmax / dS warpgroups: half wg of the streamed columns, all 128 resident rows -------------------
    const int wg = (warp - 2) >> 2;
    const int q4 = warp & 3;
    const int row = q4 * 32 + lane;                       // resident row == TMEM lane
    const uint32_t lane_off = static_cast<uint32_t>(q4 * 32) << 16;
    const uint32_t tSb = tS + wg * 64 + lane_off, tPb = tdP + wg * 64 + lane_off;
    uint32_t g = 0, gs = 0, k = 0;     // blocks, blocks with statistics and items so far
    auto run = [&](auto kind, int rb, int first, int n) {
      constexpr bool kDQ = decltype(kind)::value;
      float row_nl = 0.f, row_nd = 0.f;                   // dQ items: this query row's statistics
      if (kDQ) {
        const float* stat = reinterpret_cast<const float*>(smem + C::kStatAt + (gs % C::kStatSlots) * kStatBytes);
        mbar_wait_or_abort(&bar.stat_full[gs % C::kStatSlots], (gs / C::kStatSlots) & 1u, abort);
        ++gs;
        row_nl = stat[row];
        row_nd = stat[kBlk + row];
      }
      for (int i = 0; i < n; ++i, ++g) {
        const float* stat = reinterpret_cast<const float*>(smem + C::kStatAt + (gs % C::kStatSlots) * kStatBytes) + wg * 64;
        const bool diag = causal && first + i == rb;
        // columns a row may see on the diagonal block: dKV key `row` <= query, dQ key <= query `row`
        const int edge = row - wg * 64;
        if (!kDQ) {
          mbar_wait_or_abort(&bar.stat_full[gs % C::kStatSlots], (gs / C::kStatSlots) & 1u, abort);
          ++gs;
        }
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
    for (Item it; next_item(k, it); ++k) {
      if (it.dq) run(DQ{}, it.rb, it.first, it.n); else run(DKV{}, it.rb, it.first, it.n);
    }
  } else if (warp < 14) {
    // ------------- epilogue warpgroup: accumulators -> registers -> bf16 in shared memory -> TMA, a row per thread -------------
    const int q4 = warp & 3;
    const int row = q4 * 32 + lane;
    const uint32_t lane_off = static_cast<uint32_t>(q4 * 32) << 16;
    uint8_t* out = smem + C::kOutAt;
    const bool issuer = warp == 10 && lane == 0;
    uint32_t k = 0, kv = 0;            // items and dKV items so far
    for (Item it; next_item(k, it); ++k) {
      uint32_t h;
      const int b = static_cast<int>(order.H.divide(it.bh, h));
#pragma unroll 1
      for (int a = it.dq ? 1 : 0; a < 2; ++a) {           // dKV: dV from acc0, then scale * dK from acc1.  dQ: scale * dQ from acc1.
        mbar_wait_or_abort(&bar.acc[a], (a == 0 ? kv : k) & 1u, abort);
        __syncwarp();
        tc_fence_after();
        const uint32_t tA = (a == 0 ? tAcc0 : tAcc1) + lane_off;
        const float mul = a == 1 ? scale : 1.f;
        if (issuer) tma_store_wait_read<0>();             // the tile before is on its way
        named_bar_sync(1, 128);
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
#pragma unroll
          for (int c = 0; c < 8; ++c) {
            uint4 w;
            w.x = pack_bf16x2(__uint_as_float(r[8 * c]) * mul, __uint_as_float(r[8 * c + 1]) * mul);
            w.y = pack_bf16x2(__uint_as_float(r[8 * c + 2]) * mul, __uint_as_float(r[8 * c + 3]) * mul);
            w.z = pack_bf16x2(__uint_as_float(r[8 * c + 4]) * mul, __uint_as_float(r[8 * c + 5]) * mul);
            w.w = pack_bf16x2(__uint_as_float(r[8 * c + 6]) * mul, __uint_as_float(r[8 * c + 7]) * mul);
            *reinterpret_cast<uint4*>(out + c0 / 64 * kPanel + row * 128 + ((c ^ (row & 7)) * 16)) = w;
          }
        }
        fence_proxy_async_smem();
        named_bar_sync(1, 128);
        if (issuer) {
          const CUtensorMap* m = it.dq ? &maps.dq : a == 0 ? &maps.dv : &maps.dk;
#pragma unroll
          for (int p = 0; p < C::kPanels; ++p)
            tma_store_4d(m, out + p * kPanel, 64 * p, static_cast<int>(h) + (it.dq ? 0 : a == 0 ? 2 * out_step : out_step), it.rb * kBlk, b);
          tma_store_commit();
        }
      }
      if (!it.dq) ++kv;
    }
    if (issuer) tma_store_wait_read<0>();
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
  cudaError_t e = launch_dependent(flash_bwd_prep_kernel<D>, chunks * B * H, 256, 0, s, (const __nv_bfloat16*)o, (const __nv_bfloat16*)d_o, o_tok, lse, nl2,
                                   ndl, S, Sp, H, chunks, counter);
  if (e != cudaSuccess) return static_cast<int>(e);
  int rc = 0;
  auto mkmap = [&](CUtensorMap* m, const void* base, long long tok, int heads) {
    if (!rc) rc = get_tmap_4d_bf16(m, base, D, heads, S, B, D, tok, static_cast<uint64_t>(S) * tok, 64, 1, kBlk, 1, 1);
  };
  // q | k | v side by side in a token, as one projection leaves them, are one tensor of 3 H heads: one map instead of three (about 1 us of
  // host time each where the address is a new one)
  auto three = [&](CUtensorMap* m, const void* a, const void* b, const void* c, long long ta, long long tb, long long tc) {
    const long long step = 2ll * H * D;
    const bool packed = static_cast<const char*>(b) - static_cast<const char*>(a) == step && static_cast<const char*>(c) - static_cast<const char*>(b) == step && ta == tb && ta == tc;
    mkmap(m, a, ta, packed ? 3 * H : H);
    if (packed) {
      m[1] = m[2] = m[0];
    } else {
      mkmap(m + 1, b, tb, H);
      mkmap(m + 2, c, tc, H);
    }
    return packed ? H : 0;
  };
  Maps maps;
  const int in_step = three(&maps.q, q, k, v, q_tok, k_tok, v_tok), out_step = three(&maps.dq, dq, dk, dv, dqkv_tok, dqkv_tok, dqkv_tok);
  mkmap(&maps.d_o, d_o, o_tok, H);
  if (rc) return rc;
  unsigned char* const wait_byte = wait_report(kWaitFlashBackward);
  if (wait_byte == nullptr) return static_cast<int>(cudaErrorMemoryAllocation);
  e = allow_smem(flash_bwd_kernel<D>, C::kSmem);
  if (e != cudaSuccess) return static_cast<int>(e);
  const Order order(nblk, group, B * H, H);
  const int grid = order.n_items < kNumSMs ? order.n_items : kNumSMs;
  return static_cast<int>(launch_dependent(flash_bwd_kernel<D>, grid, kThreads, C::kSmem, s, maps, nl2, ndl, in_step, out_step, S, order, counter,
                                           scale * 1.4426950408889634f, scale, causal, wait_byte));
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
