// K12 + K13: paged KV cache writes and single-query (decode) attention over block tables.
//
// Cache layout per layer: k_cache / v_cache = [num_blocks, block_size, heads, head_dim] bf16.
// A sequence's tokens live in the blocks listed by its block table (host side: csrc/host/
// kv_block_manager.cpp); token t sits in slot block_table[t / block_size] * block_size + t % block_size.
//
// Decode attention is HBM-bound (every K and V byte of the context is read once), so the kernel is built
// for bytes in flight and few instructions per byte: the context is split over CTAs (split-K) so B x H x splits covers the
// 148 SMs even at batch 1, each warp streams groups of 16 tokens through the tensor cores and keeps an online-softmax
// state in registers.  Where all CTAs fit one wave the (max, sum, acc) triples of up to 8 splits are merged inside a cluster
// through distributed shared memory, in one launch; otherwise they go through scratch and a second kernel.
//
// Reference: the reference has no paged attention — it re-runs the HF model over the whole right-padded
// sequence every step and throws the cache away (reference llmctl/serve/server.py:199-204; README.md:12,67
// only claims the feature).
#include "../common/mma_sync.cuh"
#include "../common/ptx.cuh"
#include "../common/util.cuh"
#include "../common/dependent.cuh"

namespace llmctl {

// ---------------------------------------------------------------------------------------------
// K13: scatter new K/V rows (post-RoPE) from the packed [tokens, 3*H*D] activation into the cache.
// ---------------------------------------------------------------------------------------------
__global__ void __launch_bounds__(128)
kv_append_kernel(const __nv_bfloat16* __restrict__ qkv, long long row_stride, int k_off, int v_off,
                 __nv_bfloat16* __restrict__ k_cache, __nv_bfloat16* __restrict__ v_cache,
                 const long long* __restrict__ slot_mapping, int row_elems) {
  wait_for_previous(qkv, k_cache, v_cache, slot_mapping);
  release_dependents();
  const int tok = blockIdx.x;
  const long long slot = slot_mapping[tok];
  if (slot < 0) return;  // padded token
  const __nv_bfloat16* ksrc = qkv + tok * row_stride + k_off;
  const __nv_bfloat16* vsrc = qkv + tok * row_stride + v_off;
  __nv_bfloat16* kdst = k_cache + slot * row_elems;
  __nv_bfloat16* vdst = v_cache + slot * row_elems;
  for (int i = threadIdx.x * 8; i < row_elems; i += blockDim.x * 8) {
    *reinterpret_cast<uint4*>(kdst + i) = *reinterpret_cast<const uint4*>(ksrc + i);
    *reinterpret_cast<uint4*>(vdst + i) = *reinterpret_cast<const uint4*>(vsrc + i);
  }
}

__device__ __forceinline__ float ld_cluster_f32(uint32_t addr) {
  float v;
  asm volatile("ld.shared::cluster.f32 %0, [%1];" : "=f"(v) : "r"(addr) : "memory");
  return v;
}

// ---------------------------------------------------------------------------------------------
// K12: decode attention.  grid = (heads, splits, batch), block = 128 threads.
// A warp takes every fourth group of 16 tokens, whose K and V rows come through a ring of its own in shared memory (16-byte
// asynchronous copies, no block barrier).  Both products run on the tensor cores (mma.sync m16n8k16) with the tokens, then the head's
// dimensions, as the 16 rows: the one query fills a column of eight, and the probabilities, which stay fp32, take three of them as the bf16
// pieces of their 24 bits (high + middle + low, each the rest truncated: exact).  Bound by HBM.  With fp32 FMAs, a token to a
// half-warp (360 instructions per 16 tokens and head for 190 here), 63% of the issue slots were taken and DRAM was active 66% of the
// time.  us, FMAs / now: 16 contexts of up to 4096, 32 heads of 128 (697 MB) 125.2 / 110.2 (6.3 TB/s), 32 of them 220.9 / 199.2, 8 of up to 2304
// 47.5 / 39.6, 4 of up to 700 15.5 / 11.7; 16 of up to 4096, 12 heads of 64 36.3 / 30.7, 64 of 500 17.6 / 13.5, one of 300 3.9 / 3.8.
// partial layout: [batch, heads, splits, head_dim + 2] fp32 = {acc[head_dim], max, sum}.
// kCluster: the splits of a (head, sequence) are one cluster and its first CTA writes the output itself.
// ---------------------------------------------------------------------------------------------
constexpr int kMaxClusterSplits = 8;         // portable cluster size
constexpr int kDecodeStages = 2;             // of 16 tokens: deeper rings leave fewer CTAs on an SM (3 stages 120 us, 4 199 us)
constexpr int decode_smem(int head_dim) { return 4 * kDecodeStages * 2 * 16 * head_dim * 2; }

__device__ __forceinline__ void cp_async_16_or_zero(uint32_t dst, const void* src, bool valid) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst), "l"(src), "r"(valid ? 16 : 0) : "memory");
}
__device__ __forceinline__ void ldmatrix_x4(uint32_t (&a)[4], uint32_t addr) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0,%1,%2,%3}, [%4];" : "=r"(a[0]), "=r"(a[1]), "=r"(a[2]), "=r"(a[3]) : "r"(addr) : "memory");
}
__device__ __forceinline__ void ldmatrix_x4_trans(uint32_t (&a)[4], uint32_t addr) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0,%1,%2,%3}, [%4];" : "=r"(a[0]), "=r"(a[1]), "=r"(a[2]), "=r"(a[3]) : "r"(addr) : "memory");
}

template <int kHeadDim, bool kCluster>
__global__ void __launch_bounds__(128)
paged_attn_decode_kernel(const __nv_bfloat16* __restrict__ q, long long q_stride,
                         const __nv_bfloat16* __restrict__ k_cache,
                         const __nv_bfloat16* __restrict__ v_cache,
                         const int* __restrict__ block_tables, int max_blocks_per_seq,
                         const int* __restrict__ context_lens, float* __restrict__ partial,
                         int heads, int block_size, int block_shift, int tokens_per_split, float scale_log2,
                         __nv_bfloat16* __restrict__ out, long long out_stride) {
  constexpr int kUnits = kHeadDim / 8;                // 16-byte units of a row
  constexpr int kRowsPerCopy = 32 / kUnits;           // rows that a warp copies at a time
  constexpr int kTile = 16 * kHeadDim * 2;            // bytes of 16 rows
  constexpr int kSteps = kHeadDim / 16;
  extern __shared__ __align__(128) uint8_t ring[];
  __shared__ float s_out[kHeadDim + 2];
  __shared__ float s_acc[4][kHeadDim], s_m[4], s_l[4];
  wait_for_previous(q, k_cache, v_cache, block_tables, context_lens, partial, out);
  release_dependents();
  // heads vary fastest in launch order: the CTAs of all heads of one (sequence, split) are co-resident and walk
  // the same token rows together, so each [heads x head_dim] cache row is fetched from DRAM as one burst
  const int head = blockIdx.x, split = blockIdx.y, b = blockIdx.z;
  const int nsplit = gridDim.y;
  const int ctx = context_lens[b];
  const int t0 = split * tokens_per_split;
  const int t1 = min(ctx, t0 + tokens_per_split);
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int g = lane >> 2, t = lane & 3;              // fragment coordinates
  const int* bt = block_tables + static_cast<long long>(b) * max_blocks_per_seq;
  const long long row_elems = static_cast<long long>(heads) * kHeadDim;
  const int unit = lane % kUnits, sub = lane / kUnits;
  const __nv_bfloat16* kc = k_cache + head * kHeadDim + unit * 8;
  const __nv_bfloat16* vc = v_cache + head * kHeadDim + unit * 8;

  // the query as the first column of B
  uint32_t bq[kSteps][2];
#pragma unroll
  for (int ks = 0; ks < kSteps; ++ks) {
    bq[ks][0] = bq[ks][1] = 0u;
    if (g == 0) {
      const uint32_t* src = reinterpret_cast<const uint32_t*>(q + b * q_stride + head * kHeadDim + ks * 16) + t;
      bq[ks][0] = src[0];
      bq[ks][1] = src[4];
    }
  }
  float m = -INFINITY, l = 0.f, acc[kSteps][4];
#pragma unroll
  for (int i = 0; i < kSteps; ++i)
#pragma unroll
    for (int e = 0; e < 4; ++e) acc[i][e] = 0.f;

  // group n of this warp: tokens t0 + (4 n + warp) * 16 ..; rows are stored with their 16-byte units swizzled by row % 8
  const int groups = t1 > t0 ? (t1 - t0 + 63) / 64 : 0;      // uniform over the CTA
  const uint32_t mine = ptx::smem_u32(ring) + warp * (kDecodeStages * 2 * kTile);
  auto first_of = [&](int n) { return t0 + (4 * n + warp) * 16; };
  int slot = 0;                                       // cache row of token lane % 16 of the next group to be fetched, looked up a group ahead
  auto look_up = [&](int n) {
    const int tok = first_of(n) + (lane & 15);
    slot = 0;
    if (n < groups && tok < t1) {
      const int page = bt[block_shift >= 0 ? tok >> block_shift : tok / block_size];
      slot = page * block_size + (block_shift >= 0 ? tok & (block_size - 1) : tok % block_size);
    }
  };
  auto fetch = [&](int n) {
    if (n < groups) {
      const int valid = t1 - first_of(n);
      const uint32_t at = mine + (n % kDecodeStages) * (2 * kTile);
#pragma unroll
      for (int i = 0; i < 16 / kRowsPerCopy; ++i) {
        const int row = i * kRowsPerCopy + sub;
        const long long off = __shfl_sync(0xffffffffu, slot, row) * row_elems;
        const uint32_t dst = at + row * (kHeadDim * 2) + ((unit ^ (row & 7)) << 4);
        cp_async_16_or_zero(dst, kc + off, row < valid);
        cp_async_16_or_zero(dst + kTile, vc + off, row < valid);
      }
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
  };
  look_up(0);
#pragma unroll
  for (int n = 0; n < kDecodeStages - 1; ++n) {
    fetch(n);
    look_up(n + 1);
  }
  const int krow = lane & 15, kswz = krow & 7;        // K as A: lanes 0-15 address the first eight columns of 16 rows, 16-31 the next
  const int vrow = (lane & 7) + ((lane >> 4) << 3);   // V transposed as A: columns (dimensions) by lane / 8 % 2, rows (tokens) by lane / 16
  const uint32_t k_at = mine + krow * (kHeadDim * 2), v_at = mine + kTile + vrow * (kHeadDim * 2);
  for (int n = 0; n < groups; ++n) {
    __syncwarp();                                     // the stage that is filled now was read by all lanes a turn ago
    fetch(n + kDecodeStages - 1);
    look_up(n + kDecodeStages);
    asm volatile("cp.async.wait_group %0;" ::"n"(kDecodeStages - 1) : "memory");
    __syncwarp();
    const uint32_t stage = (n % kDecodeStages) * (2 * kTile);
    float sc[2][4] = {};
#pragma unroll
    for (int ks = 0; ks < kSteps; ++ks) {
      uint32_t a[4];
      ldmatrix_x4(a, k_at + stage + (((2 * ks + (lane >> 4)) ^ kswz) << 4));
      mma_bf16_16816(sc[ks & 1], a, bq[ks]);
    }
    // lanes 4 g hold the scores of tokens g and g + 8
    const int left = t1 - first_of(n);
    float x0 = g < left ? (sc[0][0] + sc[1][0]) * scale_log2 : -INFINITY, x1 = g + 8 < left ? (sc[0][2] + sc[1][2]) * scale_log2 : -INFINITY;
    x0 = __shfl_sync(0xffffffffu, x0, lane & 28);
    x1 = __shfl_sync(0xffffffffu, x1, lane & 28);
    float m_new = fmaxf(x0, x1);
#pragma unroll
    for (int o = 4; o < 32; o <<= 1) m_new = fmaxf(m_new, __shfl_xor_sync(0xffffffffu, m_new, o));
    m_new = fmaxf(m, m_new);
    const float ref = m_new == -INFINITY ? 0.f : m_new;      // nothing seen yet: every weight below is 0
    if (m_new != m) {                                 // uniform over the warp
      const float corr = exp2f(m - ref);
      l *= corr;
#pragma unroll
      for (int i = 0; i < kSteps; ++i)
#pragma unroll
        for (int e = 0; e < 4; ++e) acc[i][e] *= corr;
      m = m_new;
    }
    const float p0 = exp2f(x0 - ref), p1 = exp2f(x1 - ref);
    l += p0 + p1;
    // column c of B is the c-th piece of the probabilities
    uint32_t bp[2];
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      float w[2] = {__shfl_sync(0xffffffffu, h ? p1 : p0, 8 * t), __shfl_sync(0xffffffffu, h ? p1 : p0, 8 * t + 4)};
#pragma unroll
      for (int e = 0; e < 2; ++e) {
        const float high = __uint_as_float(__float_as_uint(w[e]) & 0xffff0000u), rest = w[e] - high;
        const float middle = __uint_as_float(__float_as_uint(rest) & 0xffff0000u);
        w[e] = g == 0 ? high : g == 1 ? middle : g == 2 ? rest - middle : 0.f;
      }
      bp[h] = __byte_perm(__float_as_uint(w[0]), __float_as_uint(w[1]), 0x7632);
    }
#pragma unroll
    for (int i = 0; i < kSteps; ++i) {
      uint32_t a[4];
      ldmatrix_x4_trans(a, v_at + stage + (((2 * i + ((lane >> 3) & 1)) ^ (vrow & 7)) << 4));
      mma_bf16_16816(acc[i], a, bp);
    }
  }
  asm volatile("cp.async.wait_all;" ::: "memory");

  // The pieces of a dimension: columns 0 and 1 in lanes with t = 0, column 2 in those with t = 1.  A sum that is not finite in its first
  // piece (an infinity or NaN among the values) is that piece alone: the others multiplied it by zeros.
#pragma unroll
  for (int i = 0; i < kSteps; ++i)
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      const float low = __shfl_sync(0xffffffffu, acc[i][2 * h], lane | 1);
      const float high = acc[i][2 * h];
      if (t == 0) s_acc[warp][i * 16 + h * 8 + g] = isfinite(high) ? high + (acc[i][2 * h + 1] + low) : high;
    }
#pragma unroll
  for (int o = 4; o < 32; o <<= 1) l += __shfl_xor_sync(0xffffffffu, l, o);
  if (lane == 0) {
    s_m[warp] = m;
    s_l[warp] = l;
  }
  __syncthreads();
  if (threadIdx.x < kHeadDim) {
    float gm = -INFINITY;
#pragma unroll
    for (int i = 0; i < 4; ++i) gm = fmaxf(gm, s_m[i]);
    float gl = 0.f, ga = 0.f;
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const float w = (s_m[i] == -INFINITY) ? 0.f : exp2f(s_m[i] - gm);
      gl += s_l[i] * w;
      ga += s_acc[i][threadIdx.x] * w;
    }
    float* dst = kCluster ? s_out : partial + ((static_cast<long long>(b) * heads + head) * nsplit + split) * (kHeadDim + 2);
    dst[threadIdx.x] = ga;
    if (threadIdx.x == 0) {
      dst[kHeadDim] = gm;
      dst[kHeadDim + 1] = gl;
    }
  }
  if (kCluster) {
    ptx::cluster_sync();                              // every split's triple is in its CTA's shared memory
    if (split == 0 && threadIdx.x < kHeadDim) {       // split == rank: the cluster spans the grid's y axis
      float v[kMaxClusterSplits], ms[kMaxClusterSplits], ls[kMaxClusterSplits], gm = -INFINITY;
#pragma unroll
      for (int s = 0; s < kMaxClusterSplits; ++s) {
        ms[s] = -INFINITY;
        ls[s] = v[s] = 0.f;
        if (s < nsplit) {
          const uint32_t at = ptx::mapa_u32(ptx::smem_u32(s_out), s);
          v[s] = ld_cluster_f32(at + threadIdx.x * 4);
          ms[s] = ld_cluster_f32(at + kHeadDim * 4);
          ls[s] = ld_cluster_f32(at + kHeadDim * 4 + 4);
        }
        gm = fmaxf(gm, ms[s]);
      }
      float gl = 0.f, ga = 0.f;
#pragma unroll
      for (int s = 0; s < kMaxClusterSplits; ++s) {
        const float w = (ms[s] == -INFINITY) ? 0.f : exp2f(ms[s] - gm);
        gl += ls[s] * w;
        ga += v[s] * w;
      }
      out[b * out_stride + head * kHeadDim + threadIdx.x] = __float2bfloat16(gl > 0.f ? ga / gl : 0.f);
    }
    ptx::cluster_sync();                              // nobody's shared memory goes before it was read
  }
}

template <int kHeadDim>
__global__ void __launch_bounds__(kHeadDim)
paged_attn_merge_kernel(const float* __restrict__ partial, __nv_bfloat16* __restrict__ out,
                        long long out_stride, int heads, int nsplit) {
  wait_for_previous(partial, out);
  release_dependents();
  const int head = blockIdx.x, b = blockIdx.y;
  const float* p = partial + (static_cast<long long>(b) * heads + head) * nsplit * (kHeadDim + 2);
  float gm = -INFINITY;
  for (int s = 0; s < nsplit; ++s) gm = fmaxf(gm, p[s * (kHeadDim + 2) + kHeadDim]);
  float gl = 0.f, ga = 0.f;
  for (int s = 0; s < nsplit; ++s) {
    const float ms = p[s * (kHeadDim + 2) + kHeadDim];
    const float w = (ms == -INFINITY) ? 0.f : exp2f(ms - gm);
    gl += p[s * (kHeadDim + 2) + kHeadDim + 1] * w;
    ga += p[s * (kHeadDim + 2) + threadIdx.x] * w;
  }
  out[b * out_stride + head * kHeadDim + threadIdx.x] = __float2bfloat16(gl > 0.f ? ga / gl : 0.f);
}

}  // namespace llmctl

using namespace llmctl;

LLMCTL_API int llmctl_kv_append(const void* qkv, long long row_stride, int k_off, int v_off,
                                void* k_cache, void* v_cache, const long long* slot_mapping,
                                int num_tokens, int heads, int head_dim, void* stream) {
  LLMCTL_BEGIN();
  LLMCTL_REQUIRE((heads * head_dim) % 8 == 0 && row_stride % 8 == 0 && k_off % 8 == 0 && v_off % 8 == 0);
  if (num_tokens == 0) return 0;
  LLMCTL_REQUIRE(aligned16(qkv, k_cache, v_cache));
  LLMCTL_CHECK(launch_dependent(kv_append_kernel, num_tokens, 128, 0, (cudaStream_t)stream, (const __nv_bfloat16*)qkv, row_stride, k_off, v_off,
                                (__nv_bfloat16*)k_cache, (__nv_bfloat16*)v_cache, slot_mapping, heads * head_dim));
  LLMCTL_RETURN_LAST();
}

// One launch, merged inside clusters: one split, or up to 8 while all CTAs are resident together.  A CTA that ends early waits for
// its cluster and keeps its place on the SM meanwhile, so beyond one wave of unlike contexts clusters lose (16 contexts of 1200-4096,
// 32 heads, 8 splits, with the loads in registers: 252 us in clusters, 195 us with a merge kernel; with the ring 127 us with one); below,
// the second launch is a third of the time (300 keys, 12 heads of 64: 6.0 us in two launches, 4.1 us in one).
static bool decode_in_clusters(long long batch, int heads, int num_splits) {
  return num_splits == 1 || (num_splits <= kMaxClusterSplits && batch * heads * num_splits <= 3 * kNumSMs);
}

// Number of fp32 scratch elements llmctl_paged_attn_decode needs for a given launch.
LLMCTL_API long long llmctl_paged_attn_scratch_elems(int batch, int heads, int head_dim, int num_splits) {
  return decode_in_clusters(batch, heads, num_splits) ? 0 : static_cast<long long>(batch) * heads * num_splits * (head_dim + 2);
}

// out[b, h, :] = softmax(q[b, h, :] . K[b]^T * scale) V[b] over the paged cache.
// scratch: fp32 [llmctl_paged_attn_scratch_elems(...)] (may be null when that is 0).  num_splits >= 1.
LLMCTL_API int llmctl_paged_attn_decode(const void* q, long long q_stride, const void* k_cache,
                                        const void* v_cache, const int* block_tables,
                                        int max_blocks_per_seq, const int* context_lens, void* out,
                                        long long out_stride, float* scratch, int batch, int heads,
                                        int head_dim, int block_size, int max_context, int num_splits,
                                        float scale, void* stream) {
  LLMCTL_BEGIN();
  LLMCTL_REQUIRE(head_dim == 128 || head_dim == 64);
  const bool cluster = decode_in_clusters(batch, heads, num_splits);
  LLMCTL_REQUIRE(num_splits >= 1 && block_size >= 1 && q_stride % 8 == 0 && (cluster || scratch != nullptr));
  if (batch == 0) return 0;
  LLMCTL_REQUIRE(aligned16(k_cache, v_cache) && (reinterpret_cast<uintptr_t>(q) & 3) == 0);       // queries are read in pairs
  cudaStream_t s = (cudaStream_t)stream;
  int per = (max_context + num_splits - 1) / num_splits;
  per = ((per + block_size - 1) / block_size) * block_size;  // whole blocks per split
  if (per < block_size) per = block_size;
  const float scale_log2 = scale * 1.4426950408889634f;
  int shift = -1;
  if ((block_size & (block_size - 1)) == 0)
    for (shift = 0; (1 << shift) < block_size; ++shift) {
    }
  auto launch = [&](auto kern) -> cudaError_t {
    const int smem = decode_smem(head_dim);
    const cudaError_t e = allow_smem(kern, smem);
    if (e != cudaSuccess) return e;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(heads, num_splits, batch);
    cfg.blockDim = dim3(128, 1, 1);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = s;
    cudaLaunchAttribute at[2];
    at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at[0].val.programmaticStreamSerializationAllowed = 1;
    at[1].id = cudaLaunchAttributeClusterDimension;
    at[1].val.clusterDim.x = 1;
    at[1].val.clusterDim.y = static_cast<unsigned>(num_splits);
    at[1].val.clusterDim.z = 1;
    cfg.attrs = at;
    cfg.numAttrs = cluster ? 2 : 1;
    return cudaLaunchKernelEx(&cfg, kern, (const __nv_bfloat16*)q, q_stride, (const __nv_bfloat16*)k_cache, (const __nv_bfloat16*)v_cache,
                              block_tables, max_blocks_per_seq, context_lens, scratch, heads, block_size, shift, per, scale_log2,
                              (__nv_bfloat16*)out, out_stride);
  };
  if (head_dim == 128) LLMCTL_CHECK(cluster ? launch(paged_attn_decode_kernel<128, true>) : launch(paged_attn_decode_kernel<128, false>));
  else LLMCTL_CHECK(cluster ? launch(paged_attn_decode_kernel<64, true>) : launch(paged_attn_decode_kernel<64, false>));
  if (!cluster) {
    if (head_dim == 128)
      LLMCTL_CHECK(launch_dependent(paged_attn_merge_kernel<128>, dim3(heads, batch), 128, 0, s, scratch, (__nv_bfloat16*)out, out_stride, heads, num_splits));
    else
      LLMCTL_CHECK(launch_dependent(paged_attn_merge_kernel<64>, dim3(heads, batch), 64, 0, s, scratch, (__nv_bfloat16*)out, out_stride, heads, num_splits));
  }
  LLMCTL_RETURN_LAST();
}
