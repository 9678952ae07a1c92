// Prompts of latent attention with rebuilt keys and values.
//
// Absorbed queries make every head attend to the latent rows themselves: 2 R + dr products per (query, key) and head (1088 at
// R = 512, dr = 64) on a kernel whose output alone fills tensor memory (latent_attention_t5.cu).  Where many queries of a
// sequence are in the batch it is cheaper to rebuild each head's keys and values from the cached latents once (k = Uk c, v = Uv c:
// two plain GEMMs over the sequence's rows) and run ordinary causal attention over them: dn + dr + dv = 320 products per pair, on
// the flash kernel (flash_fwd.cu).  This file holds the step before the GEMMs, one launch:
//   * the rope part of every query head is rotated in place (once per token: the angles are shared by the heads);
//   * the latent and the shared rotated key part of every sequence are gathered from the pages into contiguous rows, each
//     sequence's rows filled up with zeros to a multiple of 128 (the GEMMs turn them into zero keys and values).
// Bound by memory: 4096 tokens, 16 heads, 4096 key rows move 19 MB; a warp per row or token, 16 bytes per lane.
// Reference: none (the reference has no model code).
#include "../common/dtype.cuh"
#include "../common/util.cuh"
#include "../common/dependent.cuh"
#include "../rope/rope_interleaved.cuh"

namespace llmctl {

constexpr int kPrepWarps = 4;

__global__ void __launch_bounds__(32 * kPrepWarps)
latent_prompt_prepare_kernel(__nv_bfloat16* __restrict__ q, long long ldq, int tokens, int H, int dn, int dr,
                             const int* __restrict__ positions, const float* __restrict__ freq, float mult,
                             const __nv_bfloat16* __restrict__ cache, int R, const int* __restrict__ block_tables, int max_blocks,
                             int block_size, const int4* __restrict__ seqs, int B, int key_rows, __nv_bfloat16* __restrict__ c_out,
                             __nv_bfloat16* __restrict__ kr_out) {
  wait_for_previous(q, positions, freq, cache, block_tables, seqs, c_out, kr_out);
  release_dependents();
  const int lane = threadIdx.x & 31;
  const int w = blockIdx.x * kPrepWarps + (threadIdx.x >> 5);
  if (w < tokens) {
    // ---- rotate: lane = coordinate pair; all heads of the token, kAhead of them asked for before the first is stored (a head is stored where
    // the next might be read, so the loads do not move up by themselves and the heads of a token were a chain).  A layer over two prompts of 2048
    // tokens, 16 heads: 141.4 -> 140.6 us, three runs of each within 0.4 ----
    constexpr int kAhead = 16;
    __nv_bfloat16* row = q + w * ldq + dn;
    for (int i = lane; i < dr / 2; i += 32) {
      float s = 0.f, c = 0.f;
      for (int h0 = 0; h0 < H; h0 += kAhead) {
        __nv_bfloat162 x[kAhead];
#pragma unroll
        for (int u = 0; u < kAhead; ++u)
          if (h0 + u < H) x[u] = *reinterpret_cast<const __nv_bfloat162*>(row + (h0 + u) * (dn + dr) + 2 * i);
        if (h0 == 0) {
          sincosf(static_cast<float>(positions[w]) * freq[i], &s, &c);
          s *= mult;
          c *= mult;
        }
#pragma unroll
        for (int u = 0; u < kAhead; ++u) {
          const float2 v = __bfloat1622float2(x[u]);
          if (h0 + u < H) *reinterpret_cast<__nv_bfloat162*>(row + (h0 + u) * (dn + dr) + 2 * i) = __floats2bfloat162_rn(v.x * c - v.y * s, v.y * c + v.x * s);
        }
      }
    }
    return;
  }
  const int g = w - tokens;
  if (g >= key_rows) return;
  // ---- gather: the sequence whose key rows hold row g (their first rows grow with the index) ----
  int lo = 0, hi = B - 1;
  while (lo < hi) {
    const int mid = (lo + hi + 1) >> 1;
    if (seqs[mid].w <= g) lo = mid; else hi = mid - 1;
  }
  const int4 sq = seqs[lo];
  const int j = g - sq.w, D = R + dr;
  const uint4 zero = make_uint4(0u, 0u, 0u, 0u);
  const uint4* src = nullptr;
  if (j < sq.y + sq.z) {
    const int page = block_tables[static_cast<long long>(lo) * max_blocks + j / block_size];
    src = reinterpret_cast<const uint4*>(cache + (static_cast<long long>(page) * block_size + j % block_size) * D);
  }
  uint4* dc = reinterpret_cast<uint4*>(c_out + static_cast<long long>(g) * R);
  uint4* dk = reinterpret_cast<uint4*>(kr_out + static_cast<long long>(g) * dr);
#pragma unroll 4
  for (int i = lane; i < D / 8; i += 32) {
    const uint4 v = src != nullptr ? src[i] : zero;
    if (i < R / 8) dc[i] = v; else dk[i - R / 8] = v;
  }
}

}  // namespace llmctl

using namespace llmctl;

// q: [tokens, H * (dn + dr)] bf16 (row stride ldq), the last dr of every head are rotated in place.  seqs: int32 [B, 4] = (first query
// row, queries, position of the first query, first key row), key rows growing with the index, row b using block_tables[b].
// cache: [pages, block_size, R + dr] bf16.  c_out: [key_rows, R], kr_out: [key_rows, dr].
LLMCTL_API int llmctl_latent_prompt_prepare(void* q, long long ldq, int tokens, int H, int dn, int dr, const int* positions,
                                            const float* freq, float mult, const void* cache, int R, const int* block_tables,
                                            int max_blocks, int block_size, const int* seqs, int B, int key_rows, void* c_out, void* kr_out,
                                            void* stream) {
  LLMCTL_BEGIN();
  LLMCTL_REQUIRE(tokens >= 0 && key_rows >= 0 && H > 0 && dn % 2 == 0 && dr % 8 == 0 && R % 8 == 0 && ldq % 2 == 0 && B > 0 && block_size > 0);
  LLMCTL_REQUIRE(((reinterpret_cast<uintptr_t>(cache) | reinterpret_cast<uintptr_t>(c_out) | reinterpret_cast<uintptr_t>(kr_out) |
                   reinterpret_cast<uintptr_t>(seqs)) & 15) == 0 && (reinterpret_cast<uintptr_t>(q) & 3) == 0);
  const long long warps = static_cast<long long>(tokens) + key_rows;
  if (warps == 0) return 0;
  LLMCTL_REQUIRE(warps < (1ll << 31));
  LLMCTL_CHECK(launch_dependent(latent_prompt_prepare_kernel, static_cast<unsigned>((warps + kPrepWarps - 1) / kPrepWarps), 32 * kPrepWarps, 0, (cudaStream_t)stream,
                                (__nv_bfloat16*)q, ldq, tokens, H, dn, dr, positions, freq, mult, (const __nv_bfloat16*)cache, R, block_tables, max_blocks, block_size,
                                reinterpret_cast<const int4*>(seqs), B, key_rows, (__nv_bfloat16*)c_out, (__nv_bfloat16*)kr_out));
  LLMCTL_RETURN_LAST();
}
