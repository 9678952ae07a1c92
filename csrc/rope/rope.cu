// K4: rotary position embedding (rotate-half / NeoX pairing, as used by LLaMA-style models),
// applied in place to the q and k heads of a packed [tokens, (q|k|v)] activation.  `sign = -1`
// applies the inverse rotation, which is exactly the backward pass.
//
// Reference: none — the reference reaches HF rotary through `self.model(**batch)`
// (reference llmctl/runtime/engine.py:284); config keys rope.base / rope.scaling come from
// reference configs/models/llama-7b.json:11-14.  The cos/sin table is built by the caller so
// "linear"/"su" scaling only changes the table, not the kernel.
#include "../common/dependent.cuh"
#include "../common/fast_div.h"
#include "../common/util.cuh"

namespace llmctl {

// One thread rotates 8 pairs: elements [d0, d0+8) of the first half with the matching second half.  Bound by the two passes over the rows; with three
// 64-bit divisions for each thread's place it took 2.8 us for 777 x 24 heads of 64, now 2.5 (1500 x 32 of 128 6.0 / 5.5, 4096 x 32 of 128 12.3 / 12.0).
__global__ void __launch_bounds__(256)
rope_kernel(__nv_bfloat16* __restrict__ x, long long row_stride, uint32_t total, FastDiv per_token, FastDiv per_head, FastDiv seq,
            int head_dim, const float* __restrict__ cos_t, const float* __restrict__ sin_t,
            const int* __restrict__ positions, int tok0, float sign) {
  wait_for_previous(x, cos_t, sin_t, positions);
  release_dependents();
  const int half = head_dim >> 1;
  for (uint32_t idx = blockIdx.x * blockDim.x + threadIdx.x; idx < total; idx += gridDim.x * blockDim.x) {
    uint32_t unit, vh, at;
    const int tok = tok0 + static_cast<int>(per_token.divide(idx, unit)), head = static_cast<int>(per_head.divide(unit, vh));
    seq.divide(tok, at);
    const int pos = positions ? positions[tok] : static_cast<int>(at);
    __nv_bfloat16* p = x + tok * row_stride + static_cast<long long>(head) * head_dim + vh * 8;
    float a[8], b[8], c[8], s[8], oa[8], ob[8];
    unpack8(load8(p), a);
    unpack8(load8(p + half), b);
    const float* cp = cos_t + static_cast<long long>(pos) * half + vh * 8;
    const float* sp = sin_t + static_cast<long long>(pos) * half + vh * 8;
    *reinterpret_cast<float4*>(c) = *reinterpret_cast<const float4*>(cp);
    *reinterpret_cast<float4*>(c + 4) = *reinterpret_cast<const float4*>(cp + 4);
    *reinterpret_cast<float4*>(s) = *reinterpret_cast<const float4*>(sp);
    *reinterpret_cast<float4*>(s + 4) = *reinterpret_cast<const float4*>(sp + 4);
#pragma unroll
    for (int j = 0; j < 8; ++j) {
      const float sj = s[j] * sign;
      oa[j] = __fmaf_rn(a[j], c[j], -__fmul_rn(b[j], sj));      // spelt out: the projection's epilogue rounds alike
      ob[j] = __fmaf_rn(b[j], c[j], __fmul_rn(a[j], sj));
    }
    store8(p, pack8(oa));
    store8(p + half, pack8(ob));
  }
}

}  // namespace llmctl

using namespace llmctl;

LLMCTL_API int llmctl_rope_inplace(void* x, long long row_stride, int n_tokens, int n_heads,
                                   int head_dim, const float* cos_t, const float* sin_t,
                                   const int* positions, int seq_len, float sign, void* stream) {
  LLMCTL_BEGIN();
  LLMCTL_REQUIRE(head_dim % 16 == 0 && row_stride % 8 == 0 && seq_len > 0);
  LLMCTL_REQUIRE(((reinterpret_cast<uintptr_t>(x) | reinterpret_cast<uintptr_t>(cos_t) | reinterpret_cast<uintptr_t>(sin_t)) & 15) == 0);
  const long long per_token = static_cast<long long>(n_heads) * (head_dim / 16);
  if (per_token == 0 || n_tokens == 0) return 0;
  LLMCTL_REQUIRE(n_heads > 0 && head_dim > 0 && n_tokens > 0 && per_token < (1 << 30));
  const long long most = (1 << 30) / per_token;              // tokens of a launch: its units are counted in 31 bits
  for (long long tok0 = 0; tok0 < n_tokens; tok0 += most) {
    const long long tokens = n_tokens - tok0 < most ? n_tokens - tok0 : most, total = tokens * per_token;
    long long blocks = (total + 255) / 256;
    if (blocks > kNumSMs * 16) blocks = kNumSMs * 16;
    LLMCTL_CHECK(launch_dependent(rope_kernel, static_cast<int>(blocks), 256, 0, (cudaStream_t)stream, (__nv_bfloat16*)x, row_stride,
                                  static_cast<uint32_t>(total), FastDiv(static_cast<uint32_t>(per_token)), FastDiv(head_dim / 16), FastDiv(seq_len),
                                  head_dim, cos_t, sin_t, positions, static_cast<int>(tok0), sign));
  }
  LLMCTL_RETURN_LAST();
}
