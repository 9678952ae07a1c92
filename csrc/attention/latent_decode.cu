// Latent attention of single decoded tokens on the 5th-generation tensor cores: one token's heads against its sequence's paged cache rows.
//
//   out[t, h, :] = softmax_j( scale * q[t, h, :] . k[j, :] ) c[j, :]      k[j] = [c[j] | kr[j]]  (one cache row, D = R + dr)
//
// with the sinks, window and gates of llmctl_latent_attention (latent_attention.cu, whose merge kernel puts split contexts together).
//
// A token has only its heads to offer as rows, 16 or 32 of the 128 of a tcgen05 product, so the CACHE ROWS are the M side of both products and
// the heads their N:
//     S^T = K Q^T         64 keys x N heads, over D             (A: the key tile as it was loaded, K-major)
//     O^T += C^T P^T      128 latent dimensions x N heads, over 64 keys      (A: the same tile, M-major)
// A tile of 64 cache rows is read from memory once and serves both; nothing of it passes through registers.
//
//   warp 0      TMA producer: key tiles through the block table, two stages at D = 576 (74 KB each)
//   warp 1      MMA issuer
//   warps 2-5   assemble Q (absorbed part | rotated part) in shared memory, then turn S^T into P^T: a key per thread, all its heads; a running
//               reference per head that moves only when a score outgrows it by 2^8 (one vote per tile instead of maxima over keys,
//               which lie in different threads), probabilities in bf16, their sums in fp32 over what was rounded: a key that decides alone
//               then weighs 1, wherever the reference stands
// TMEM: S^T two buffers of N columns (64 rows: lanes 32q + 0 .. 15 of quadrant q), O^T R / 128 blocks of N columns.
//
// Bound by a CTA's chain from tile to tile (copy, scores, softmax, values, the stage handed back) with no more than two stages to hide it: about 3 TB/s,
// 35-38% of DRAM's peak; a tile's products alone are 36 of 27 and 16 of 46 clocks.  With the merge of split contexts, us, mma.sync kernel of latent_attention.cu / this one: 32 contexts of 2000-4000, 16 heads 65 / 39, 32 heads 92 / 42
// (112 MB: 17 at the rate of a copy); 32 of 500-1000, 16 heads 31 / 19; 8 of 1000-2000 28 / 14; one of 300 18.4 / 9.9, 32 heads 21 / 12.  Splits for one
// CTA to an SM (two: 39 -> 43).
// Every wait is bounded, as in latent_attention_t5.cu.
// Reference: none (the reference has no model code).
#include <float.h>

#include "../common/dependent.cuh"
#include "../common/dtype.cuh"
#include "../common/mma_sync.cuh"
#include "../common/ptx.cuh"
#include "../common/tma_host.h"
#include "../common/util.cuh"
#include "../common/wait_status.h"

namespace llmctl {
using namespace ptx;

int launch_latent_attention_merge_bf16(const float* partial, void* out, int R, int splits, int rows, int H, const void* head_gate,
                                       long long gate_ld, cudaStream_t s);

namespace ldec {
constexpr int kKeys = 64;                    // keys per tile (M of the score product)
constexpr int kPanel = kKeys * 128;          // bytes of 64 keys x 64 columns
constexpr int kThreads = 192;
constexpr int kMaxStages = 4, kMaxPanels = 9, kMaxRank = 512, kMaxParts = 3;
constexpr int kWindowAlign = 32;             // a window's first key tile starts at a multiple of this
constexpr float kLog2e = 1.4426950408889634f, kLn2 = 0.6931471805599453f;
constexpr float kRescaleThreshold = 8.f;
constexpr int fixed_smem(int panels, int N) { return panels * N * 128 + 2 * N * 128 + 1024; }      // Q, P, alignment
constexpr int smem_most(int ctas) { return (ctas == 1 ? 225 : 110) * 1024; }      // dynamic, of a CTA, where an SM has to hold that many
constexpr int stages_in(int bytes, int panels, int N) { return (bytes - fixed_smem(panels, N)) / (panels * kPanel); }

// A stage of nine panels (four 128-wide blocks of the latent, the rotated part) is handed back in three parts, as the value products of its blocks end, and
// loaded again part by part; other tiles in one.  A layer, 32 tokens behind 4000: 16 heads 70.1 -> 69.1 us, 32 heads 84.5 -> 83.7.  Scores that also
// start part by part, as the loads land, stand in front of the values of the tile before (72.9, 87.0).
template <int kPanels>
constexpr int kParts = kPanels ? kMaxParts : 1;
template <int kPanels>
__device__ constexpr int first_panel(int part, int panels) {
  static_assert(kPanels == 0 || kPanels == 9, "parts");
  return part == 0 ? 0 : kPanels == 0 || part == kMaxParts ? panels : part == 1 ? 4 : 6;
}

__device__ __forceinline__ bool any_of_softmax_warps(bool x) {
  uint32_t r;
  asm volatile(
      "{\n\t.reg .pred p, q;\n\t"
      "setp.ne.u32 p, %1, 0;\n\t"
      "barrier.cta.red.or.pred q, 1, 128, p;\n\t"
      "selp.u32 %0, 1, 0, q;\n\t}"
      : "=r"(r)
      : "r"(static_cast<uint32_t>(x))
      : "memory");
  return r != 0;
}
// Over the warp's lanes, heads as they become fewer spread over them: v[h] of every lane -> head (lane % N), N - 1 exchanges instead of 5 N.
// (Straight-line code for every head costs its instruction fetches as well: maxima, sums and read-out of 32 heads took 35000 clocks.)
template <int N, typename Op>
__device__ __forceinline__ float reduce_heads(float (&v)[N], int lane, Op op) {
#pragma unroll
  for (int w = N / 2; w >= 1; w /= 2) {
    const bool upper = lane & w;
#pragma unroll
    for (int i = 0; i < w; ++i) {
      const float keep = upper ? v[i + w] : v[i], send = upper ? v[i] : v[i + w];
      v[i] = op(keep, __shfl_xor_sync(0xffffffffu, send, w));
    }
  }
  if (N == 16) v[0] = op(v[0], __shfl_xor_sync(0xffffffffu, v[0], 16));
  return v[0];
}
template <int N>
__device__ __forceinline__ void tmem_ld(uint32_t at, uint32_t* r) {
  if constexpr (N == 16) tmem_ld_x16(at, r); else tmem_ld_x32(at, r);
}
}  // namespace ldec

// Grid: (tokens, groups of heads_per_tile heads, splits).  kPanels: 64-column panels of a cache row, 9 for latents of 512 with 64 rotated
// dimensions, or 0 for what R and dr say.  With 9 the products unroll and their descriptors are constants away from one register (32 contexts of
// 2000-4000 from stages that are not loaded: 34.6 us in loops, 28.5 unrolled).  kCtas: CTAs that an SM has to hold; the registers of 32 heads are as
// many as one may have, and a few have to be spilled for two.
template <int N, int kPanels, int kCtas>
__global__ void __launch_bounds__(ldec::kThreads, kCtas)
latent_decode_kernel(const __grid_constant__ CUtensorMap tmK, const __nv_bfloat16* __restrict__ ql, long long ql_st, long long ql_sh,
                     const __nv_bfloat16* __restrict__ q, long long ldq, int dn, const int* __restrict__ block_tables, int max_blocks, int block_size,
                     const int* __restrict__ tiles, const int* __restrict__ positions, const float* __restrict__ freq, float mult, float scale,
                     int H, int R_, int dr_, int heads_per_tile, int keys_per_split, int stages_, int box_rows, __nv_bfloat16* __restrict__ out,
                     float* __restrict__ partial, const float* __restrict__ sinks, int window, const __nv_bfloat16* __restrict__ head_gate,
                     long long gate_ld, unsigned char* wait_byte) {
  using namespace ldec;
  extern __shared__ uint8_t smem_raw[];
  __shared__ uint64_t bar_q, bar_kfull[kMaxStages], bar_kempty[kMaxStages][kMaxParts], bar_s[2], bar_p[2], bar_pv[2];
  __shared__ uint32_t tmem_base_smem;
  __shared__ int abort_flag;
  __shared__ float warp_row[4][N];                                     // per softmax warp and head: maxima, later sums
  __shared__ __align__(16) float new_ref[4][N], new_alpha[4][N];       // per softmax warp, so that no barrier is needed

  const uint32_t smem_base = (smem_u32(smem_raw) + 1023u) & ~1023u;
  uint8_t* smem = smem_raw + (smem_base - smem_u32(smem_raw));
  const int warp = __shfl_sync(0xffffffffu, threadIdx.x >> 5, 0), lane = threadIdx.x & 31;
  const int R = kPanels ? (kPanels - 1) * 64 : R_, dr = kPanels ? 64 : dr_, stages = kPanels ? 2 : stages_;
  const int panels = kPanels ? kPanels : (R + dr) >> 6, stage_bytes = panels * kPanel;
  const int q_at = stages * stage_bytes, p_at = q_at + panels * N * 128;

  if (threadIdx.x == 0) {
    mbar_init(&bar_q, 4);
    for (int i = 0; i < stages; ++i) {
      mbar_init(&bar_kfull[i], 1);
      for (int part = 0; part < kParts<kPanels>; ++part) mbar_init(&bar_kempty[i][part], 1);
    }
    for (int i = 0; i < 2; ++i) {
      mbar_init(&bar_s[i], 1);
      mbar_init(&bar_p[i], 4);
      mbar_init(&bar_pv[i], 1);
    }
    abort_flag = 0;
    fence_mbar_init();
    prefetch_tmap(&tmK);
  }
  if (warp == 1) tmem_alloc<1>(&tmem_base_smem, 256);
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = tmem_base_smem, tO = tmem_base + 2 * N;
  wait_for_previous(ql, q, block_tables, tiles, positions, freq, out, partial, sinks, head_gate);
  release_dependents();
  volatile int* abort = &abort_flag;

  const int tok = tiles[4 * blockIdx.x], seq = tiles[4 * blockIdx.x + 2];
  const int h0 = blockIdx.y * heads_per_tile, nh = min(heads_per_tile, H - h0);
  const int split = blockIdx.z, nsplit = gridDim.z;
  const int pos = positions[tok];
  const int* bt = block_tables + static_cast<long long>(seq) * max_blocks;
  const int k_begin = (window > 0 ? max(pos - window + 1, 0) / kWindowAlign * kWindowAlign : 0) + split * keys_per_split;
  const int k_end = min(pos + 1, k_begin + keys_per_split);
  const int nt = k_end > k_begin ? (k_end - k_begin + kKeys - 1) / kKeys : 0;
  const long long row0 = static_cast<long long>(tok) * H + h0;

  if (warp == 0) {
    // ------------------------------------ TMA producer ------------------------------------
    if (lane == 0) {
      const int boxes = kKeys / box_rows;
      auto cache_row = [&](int j) { return j < k_end ? bt[j / block_size] * block_size + j % block_size : -1; };
      int row[2] = {cache_row(k_begin), boxes == 2 ? cache_row(k_begin + box_rows) : -1};
      bool given = true;
      int loaded = 0;                                     // tiles, a last one in part if a wait ran out
      for (int n = 0; n < nt && given; ++n) {
        const int st = n % stages;
        const int next[2] = {cache_row(k_begin + (n + 1) * kKeys), boxes == 2 ? cache_row(k_begin + (n + 1) * kKeys + box_rows) : -1};
        for (int part = 0; part < kParts<kPanels>; ++part) {
          given = n < stages || mbar_wait_bounded(&bar_kempty[st][part], ((n / stages) & 1u) ^ 1u, abort);
          if (!given) break;
          const int first = first_panel<kPanels>(part, panels), last = first_panel<kPanels>(part + 1, panels);
          if (part == 0) {
            mbar_expect_tx(&bar_kfull[st], (row[1] >= 0 ? 2 : 1) * box_rows * 128 * panels);
            ++loaded;
          }
          for (int b = 0; b < boxes; ++b) {
            if (row[b] < 0) continue;                     // past the sequence: zeroed by the softmax warps
            for (int p = first; p < last; ++p)
              tma_load_2d(smem + st * stage_bytes + p * kPanel + b * box_rows * 128, &tmK, &bar_kfull[st], 64 * p, row[b]);
          }
        }
        row[0] = next[0];
        row[1] = next[1];
      }
      // Copies still in flight when a wait ran out land before the CTA's shared memory is given back.
      if (*abort)
        for (int i = loaded > stages ? loaded - stages : 0; i < loaded; ++i) {
          int none = 0;
          mbar_wait_bounded(&bar_kfull[i % stages], (i / stages) & 1u, &none);
        }
    }
  } else if (warp == 1) {
    // ------------------------------------ MMA issuer ------------------------------------
    // The whole warp walks the loop, one elected lane issues: whichever is there first, the next tile (its scores then run beside the softmax
    // of this one) or the probabilities of this one (whose products free the stage that the tile after next is loaded into).  In a fixed order
    // the products of one tile waited for the load of the next, and no load ran beside them (46.8 us, now 38.7).
    constexpr uint32_t id_s = make_idesc_bf16(kKeys, N, 0u, 0u);       // A, B K-major
    constexpr uint32_t id_o = make_idesc_bf16(128, N, 1u, 1u);         // A, B MN-major
    if (nt > 0) mbar_wait_or_abort(&bar_q, 0u, abort);
    const long long t0 = clock64();
    for (int ns = 0, np = 0; np < nt;) {
      const int st = ns % stages, sp = np % stages;
      const bool tile = ns < nt && ns <= np + 1 && __any_sync(0xffffffffu, mbar_test(&bar_kfull[st], (ns / stages) & 1u));
      const bool probs = !tile && np < ns && __any_sync(0xffffffffu, mbar_test(&bar_p[np & 1], (np >> 1) & 1u));
      if (tile) {
        mbar_wait_or_abort(&bar_kfull[st], (ns / stages) & 1u, abort);
        __syncwarp();
        tc_fence_after();
        const uint64_t a = make_smem_desc(smem_base + st * stage_bytes, 16, 1024, 2), b = make_smem_desc(smem_base + q_at, 16, 1024, 2);
        if (elect_one()) {
#pragma unroll(kPanels ? kPanels : 1)
          for (int p = 0; p < panels; ++p)
#pragma unroll
            for (int k = 0; k < 4; ++k)
              umma_ss<1>(tmem_base + (ns & 1) * N, a + ((p * kPanel + k * 32) >> 4), b + ((p * N * 128 + k * 32) >> 4), id_s, (p | k) != 0 ? 1u : 0u);
          umma_commit<1>(&bar_s[ns & 1]);
        }
        ++ns;
      } else if (probs) {
        mbar_wait_or_abort(&bar_p[np & 1], (np >> 1) & 1u, abort);
        __syncwarp();
        tc_fence_after();
        const uint64_t a = make_smem_desc(smem_base + sp * stage_bytes, kPanel, 1024, 2);
        const uint64_t b = make_smem_desc(smem_base + p_at + (np & 1) * N * 128, 128, 1024, 0);
        if (elect_one()) {
#pragma unroll
          for (int i = 0; i < kParts<kPanels>; ++i) {
#pragma unroll(kPanels ? kPanels / 2 : 1)
            for (int d = first_panel<kPanels>(i, panels) / 2; d < min(first_panel<kPanels>(i + 1, panels), R / 64) / 2; ++d)
#pragma unroll
              for (int k = 0; k < kKeys / 16; ++k)
                umma_ss<1>(tO + d * N, a + ((d * 2 * kPanel + k * 2048) >> 4), b + ((k * 256) >> 4), id_o, (np | k) != 0 ? 1u : 0u);
            umma_commit<1>(&bar_kempty[sp][i]);
          }
          umma_commit<1>(&bar_pv[np & 1]);
        }
        ++np;
      } else {
        const bool late = clock64() - t0 > kBoundedWaitCycles;
        if (late) *abort = 1;
        if (__any_sync(0xffffffffu, late || *abort)) break;
      }
    }
  } else {
    // ------------------------------------ softmax warps ------------------------------------
    const int w = warp - 2, t = threadIdx.x - 64, quad = warp & 3;
    const uint32_t lane_off = static_cast<uint32_t>(quad * 32) << 16;
    if (nt == 0) {               // a split past this token's context: an empty partial (uniform over the CTA)
      if (nsplit > 1)
        for (int h = 0; h < nh; ++h) {
          float* dst = partial + ((row0 + h) * nsplit + split) * (R + 2);
          for (int c = t; c < R; c += 128) dst[c] = 0.f;
          if (t == 0) {
            dst[R] = -INFINITY;
            dst[R + 1] = 0.f;
          }
        }
    } else {
      // Q: rows of heads, K-major panels of 64 columns.  A warp per row and nothing that waits for a load before the last is asked for.
      uint8_t* qs = smem + q_at;
      auto unit = [&](int r, int u) { return qs + (u >> 3) * N * 128 + r * 128 + (((u & 7) ^ (r & 7)) << 4); };
#pragma unroll
      for (int i = 0; i < N / 4; ++i) {
        const int r = w + 4 * i;
        for (int u = lane; u < R >> 3; u += 32) {
          if (r < nh) cp_async_16(unit(r, u), ql + tok * ql_st + (h0 + r) * ql_sh + u * 8);
          else *reinterpret_cast<uint4*>(unit(r, u)) = make_uint4(0u, 0u, 0u, 0u);
        }
      }
      cp_async_commit();
      for (int i = lane; i < dr >> 1; i += 32) {          // a rotated pair of all the warp's rows
        __nv_bfloat16 x[N / 4], y[N / 4];
#pragma unroll
        for (int k = 0; k < N / 4; ++k)
          if (w + 4 * k < nh) {
            const __nv_bfloat16* at = q + tok * ldq + static_cast<long long>(h0 + w + 4 * k) * (dn + dr) + dn + 2 * i;
            x[k] = at[0];
            y[k] = at[1];
          }
        float sn, cs;
        sincosf(static_cast<float>(pos) * freq[i], &sn, &cs);
        sn *= mult;
        cs *= mult;
        const int c = R + 2 * i;
#pragma unroll
        for (int k = 0; k < N / 4; ++k) {
          const float u = w + 4 * k < nh ? to_f32(x[k]) : 0.f, v = w + 4 * k < nh ? to_f32(y[k]) : 0.f;
          *reinterpret_cast<__nv_bfloat162*>(unit(w + 4 * k, c >> 3) + (c & 7) * 2) = __floats2bfloat162_rn(u * cs - v * sn, v * cs + u * sn);
        }
      }
      cp_async_wait_all();
      fence_proxy_async_smem();
      __syncwarp();
      if (lane == 0) mbar_arrive(&bar_q);

      const float scale_log2 = scale * kLog2e;
      const int key = quad * 16 + lane;                   // of the tile; lanes 16 .. 31 have none
      // a sink is a key without a value: it is the head's first reference, and its term of the sum.  References start finite, so that scores of -inf,
      // where a head has seen no other, weigh nothing instead of being no number.
      const bool sink = sinks != nullptr && split == 0;
      float __align__(16) ref[N];
      float sum[N], my_ref = sink && lane % N < nh ? fmaxf(sinks[h0 + lane % N] * kLog2e, -FLT_MAX) : -FLT_MAX;       // of the lane's own head
#pragma unroll
      for (int h = 0; h < N; ++h) {
        ref[h] = __shfl_sync(0xffffffffu, my_ref, h);
        sum[h] = sink && t == 0 && h < nh ? 1.f : 0.f;
      }
      for (int n = 0; n < nt; ++n) {
        const int j0 = k_begin + n * kKeys, j = j0 + key;
        const bool seen = lane < 16 && j < k_end && (window <= 0 || pos - j < window);
        mbar_wait_or_abort(&bar_s[n & 1], (n >> 1) & 1u, abort);
        __syncwarp();
        tc_fence_after();
        uint32_t s[N];
        tmem_ld<N>(tmem_base + (n & 1) * N + lane_off, s);
        tmem_ld_wait();
        bool grown = false;
#pragma unroll
        for (int h = 0; h < N; ++h) {
          const float v = seen ? __uint_as_float(s[h]) * scale_log2 : -INFINITY;
          s[h] = __float_as_uint(v);
          grown |= v > ref[h] + kRescaleThreshold;
        }
        if (any_of_softmax_warps(grown)) {                // rare after the first tile
          float v[N];
#pragma unroll
          for (int h = 0; h < N; ++h) v[h] = __uint_as_float(s[h]);
          const float mine = reduce_heads<N>(v, lane, [](float a, float b) { return fmaxf(a, b); });
          const int head = lane % N;
          if (lane < N) warp_row[w][head] = mine;
          named_bar_sync(1, 128);
          const float m = fmaxf(my_ref, fmaxf(fmaxf(warp_row[0][head], warp_row[1][head]), fmaxf(warp_row[2][head], warp_row[3][head])));
          if (lane < N) {
            new_ref[w][head] = m;
            new_alpha[w][head] = ex2_approx(my_ref - m);
          }
          my_ref = m;
          if (n > 0) mbar_wait_or_abort(&bar_pv[(n - 1) & 1], ((n - 1) >> 1) & 1u, abort);
          __syncwarp();
          tc_fence_after();
          float __align__(16) alpha[N];
#pragma unroll
          for (int h = 0; h < N; h += 4) {
            *reinterpret_cast<float4*>(ref + h) = *reinterpret_cast<const float4*>(&new_ref[w][h]);
            *reinterpret_cast<float4*>(alpha + h) = *reinterpret_cast<const float4*>(&new_alpha[w][h]);
          }
#pragma unroll
          for (int h = 0; h < N; ++h) sum[h] *= alpha[h];
          if (n > 0)
            for (int d = 0; d < R / 128; ++d) {
              uint32_t o[N];
              tmem_ld<N>(tO + d * N + lane_off, o);
              tmem_ld_wait();
#pragma unroll
              for (int h = 0; h < N; ++h) o[h] = __float_as_uint(__uint_as_float(o[h]) * alpha[h]);
              tmem_st_x16(tO + d * N + lane_off, o);
              if constexpr (N == 32) tmem_st_x16(tO + d * N + 16 + lane_off, o + 16);
            }
          tmem_st_wait();
          named_bar_sync(1, 128);                         // warp_row is read before the next tile's maxima
        }
        if (n >= 2) mbar_wait_or_abort(&bar_pv[n & 1], ((n - 2) >> 1) & 1u, abort);          // P(n - 2) has been read
        if (lane < 16) {
          uint8_t* dst = smem + p_at + (n & 1) * N * 128 + key * 16;
#pragma unroll
          for (int g = 0; g < N / 8; ++g) {
            float f[8];
#pragma unroll
            for (int e = 0; e < 8; ++e) {
              const int h = g * 8 + e;
              f[e] = seen ? ex2_approx(__uint_as_float(s[h]) - ref[h]) : 0.f;
            }
            const bf16x8 p = pack8(f);
            *reinterpret_cast<bf16x8*>(dst + g * 1024) = p;
            unpack8(p, f);
#pragma unroll
            for (int e = 0; e < 8; ++e) sum[g * 8 + e] += f[e];
          }
        }
        // Rows past the last key: nothing that the cache holds there may meet a probability of zero.
        if (j0 + kKeys > k_end) {
          const int first = k_end - j0, per = R >> 3;
          uint8_t* at = smem + (n % stages) * stage_bytes;
          for (int i = t; i < (kKeys - first) * per; i += 128) {
            const int r = i / per, u = i - r * per;
            *reinterpret_cast<uint4*>(at + (u >> 3) * kPanel + (first + r) * 128 + (u & 7) * 16) = make_uint4(0u, 0u, 0u, 0u);
          }
        }
        fence_proxy_async_smem();
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(&bar_p[n & 1]);
      }
      // ---- read-out: a latent dimension per thread -> rows of heads in the stages, which are idle now -> memory ----
      const float l = reduce_heads<N>(sum, lane, [](float a, float b) { return a + b; });
      if (lane < N) warp_row[w][lane] = l;
      mbar_wait_or_abort(&bar_pv[(nt - 1) & 1], ((nt - 1) >> 1) & 1u, abort);
      __syncwarp();
      tc_fence_after();
      float* rows = reinterpret_cast<float*>(smem);
      for (int d = 0; d < R / 128; ++d) {
        uint32_t o[N];
        tmem_ld<N>(tO + d * N + lane_off, o);
        tmem_ld_wait();
#pragma unroll
        for (int h = 0; h < N; ++h) rows[h * R + d * 128 + quad * 32 + lane] = __uint_as_float(o[h]);
      }
      named_bar_sync(1, 128);
      for (int h = w; h < nh; h += 4) {
        const float2* src = reinterpret_cast<const float2*>(rows + h * R);
        const float total = (warp_row[0][h] + warp_row[1][h]) + (warp_row[2][h] + warp_row[3][h]);
        if (nsplit > 1) {
          float* dst = partial + ((row0 + h) * nsplit + split) * (R + 2);
          for (int c = lane; c < R / 2; c += 32) reinterpret_cast<float2*>(dst)[c] = src[c];
          if (lane == h % 32) {
            dst[R] = my_ref * kLn2;
            dst[R + 1] = total;
          }
        } else {
          const float gate = head_gate ? 1.f / (1.f + expf(-to_f32(head_gate[tok * gate_ld + h0 + h]))) : 1.f;
          const float inv = (total > 0.f ? 1.f / total : 0.f) * gate;
          __nv_bfloat162* dst = reinterpret_cast<__nv_bfloat162*>(out + (row0 + h) * R);
          for (int c = lane; c < R / 2; c += 32) dst[c] = __floats2bfloat162_rn(src[c].x * inv, src[c].y * inv);
        }
      }
    }
  }

  tc_fence_before();
  __syncthreads();
  if (threadIdx.x == 0 && abort_flag) report_wait(wait_byte);
  if (warp == 1) {
    tc_fence_after();
    tmem_dealloc<1>(tmem_base, 256);
  }
}

template <int N, int kPanels, int kCtas = 1>
static int launch_latent_decode(const CUtensorMap& tmK, const void* ql, long long ql_st, long long ql_sh, const void* q, long long ldq, int dn,
                                const int* block_tables, int max_blocks, int block_size, const int* tiles, int ntiles, const int* positions,
                                const float* freq, float mult, float scale, int H, int R, int dr, int heads_per_tile, int splits, int keys_per_split,
                                int box_rows, void* out, float* partial, const float* sinks, int window, const void* head_gate, long long gate_ld,
                                cudaStream_t s) {
  using namespace ldec;
  const int panels = (R + dr) >> 6, room = stages_in(smem_most(kCtas), panels, N);
  const int stages = room < kMaxStages ? room : kMaxStages, smem = fixed_smem(panels, N) + stages * panels * kPanel;
  unsigned char* const wait_byte = wait_report(kWaitLatentAttention);
  if (wait_byte == nullptr) return static_cast<int>(cudaErrorMemoryAllocation);
  auto kern = latent_decode_kernel<N, kPanels, kCtas>;
  const cudaError_t e = allow_smem(kern, smem);
  if (e != cudaSuccess) return static_cast<int>(e);
  const dim3 grid(ntiles, (H + heads_per_tile - 1) / heads_per_tile, splits);
  return static_cast<int>(launch_dependent(kern, grid, kThreads, smem, s, tmK, (const __nv_bfloat16*)ql, ql_st, ql_sh, (const __nv_bfloat16*)q, ldq, dn, block_tables,
                                           max_blocks, block_size, tiles, positions, freq, mult, scale, H, R, dr, heads_per_tile, keys_per_split, stages, box_rows,
                                           (__nv_bfloat16*)out, splits > 1 ? partial : nullptr, sinks, window, (const __nv_bfloat16*)head_gate, gate_ld, wait_byte));
}

}  // namespace llmctl

using namespace llmctl;

// Whether llmctl_latent_decode has a kernel for these sizes: whole blocks of 128 latent dimensions, whole panels of 64 columns, pages of
// whole boxes of 32 rows.
LLMCTL_API int llmctl_latent_decode_ok(int R, int dr, int block_size) {
  return R > 0 && R % 128 == 0 && R <= ldec::kMaxRank && dr >= 0 && (R + dr) % 64 == 0 && (R + dr) / 64 <= ldec::kMaxPanels && block_size % 32 == 0;
}

// llmctl_latent_attention for tiles of one token (tiles[i][1] == 1) with up to 32 heads, bf16 absorbed queries whose rows (ql + token * ql_st +
// head * ql_sh) and cache begin at 16-byte boundaries.  cache_rows: rows of the cache tensor (blocks x block_size).
LLMCTL_API int llmctl_latent_decode(const void* ql, long long ql_st, long long ql_sh, const void* q, long long ldq, int dn, const void* cache,
                                    long long cache_rows, const int* block_tables, int max_blocks, int block_size, const int* tiles, int ntiles, int tokens,
                                    const int* positions, const float* freq, float mult, float scale, int H, int R, int dr, int heads_per_tile, int splits,
                                    int keys_per_split, void* out, float* partial, const float* sinks, int window, const void* head_gate, long long gate_ld,
                                    void* stream) {
  LLMCTL_BEGIN();
  LLMCTL_REQUIRE(llmctl_latent_decode_ok(R, dr, block_size) && H > 0 && heads_per_tile >= 1 && heads_per_tile <= 32 && splits >= 1 && keys_per_split > 0 &&
                 keys_per_split % ldec::kKeys == 0 && (splits == 1 || partial != nullptr) && cache_rows >= block_size && cache_rows < (1LL << 31) && window >= 0);
  LLMCTL_REQUIRE(ql_st % 8 == 0 && ql_sh % 8 == 0 && aligned16(ql, cache));
  if (ntiles == 0 || tokens == 0) return 0;
  const int box_rows = block_size % 64 == 0 && window == 0 ? 64 : 32;        // a box never straddles a page
  CUtensorMap tmK;
  int rc = get_tmap_2d_bf16(&tmK, cache, cache_rows, R + dr, R + dr, box_rows, 64, 1);
  if (rc) LLMCTL_FAIL(rc, "tensor map of the cache");
  const bool usual = R == 512 && dr == 64;
  // More CTAs than SMs (many tokens, or one long context beside short ones, whose splits are mostly empty): two to an SM where both have stages
  // enough.  A layer, us, mma.sync kernel / one / two: 32 heads of 128 + 64 columns, 200 contexts of 100 43.1 / 46.3 / 38.7, one of 8000 beside 30 of 50
  // 93.6 / 119 / 81; 16 heads of 256 + 64, the same 40.6 / 40.0 / 33.2 and 171 / 90.7 / 66.4.  Up to 148 CTAs one each is as fast, and spills nothing.
  const long long ctas = static_cast<long long>(ntiles) * ((H + heads_per_tile - 1) / heads_per_tile) * splits;
  auto two = [&](int N, int stages) { return ctas > kNumSMs && ldec::stages_in(ldec::smem_most(2), (R + dr) / 64, N) >= stages; };
  rc = (heads_per_tile <= 16 ? (usual ? launch_latent_decode<16, 9> : two(16, 2) ? launch_latent_decode<16, 0, 2> : launch_latent_decode<16, 0>)
                             : (usual ? launch_latent_decode<32, 9> : two(32, 3) ? launch_latent_decode<32, 0, 2> : launch_latent_decode<32, 0>))(tmK, ql, ql_st, ql_sh, q, ldq, dn, block_tables, max_blocks, block_size, tiles,
                                                                                  ntiles, positions, freq, mult, scale, H, R, dr, heads_per_tile, splits,
                                                                                  keys_per_split, box_rows, out, partial, sinks, window, head_gate, gate_ld,
                                                                                  (cudaStream_t)stream);
  if (rc) LLMCTL_FAIL(rc, "latent decode");
  if (splits > 1) {
    rc = launch_latent_attention_merge_bf16(partial, out, R, splits, tokens * H, H, head_gate, gate_ld, (cudaStream_t)stream);
    if (rc) LLMCTL_FAIL(rc, "merge");
  }
  LLMCTL_RETURN_LAST();
}
