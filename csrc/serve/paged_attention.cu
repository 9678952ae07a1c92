// K12 + K13: paged KV cache writes and single-query (decode) attention over block tables.
//
// Cache layout per layer: k_cache / v_cache = [num_blocks, block_size, heads, head_dim] bf16.
// A sequence's tokens live in the blocks listed by its block table (host side: csrc/host/
// kv_block_manager.cpp); token t sits in slot block_table[t / block_size] * block_size + t % block_size.
//
// Decode attention is HBM-bound (every K and V byte of the context is read once), so the kernel is built
// for bytes in flight, not FLOPs: the context is split over CTAs (split-K) so B x H x splits covers the
// 148 SMs even at batch 1, each half-warp streams one token (16-byte loads) and keeps an online-softmax
// state in registers.  Where all CTAs fit one wave the (max, sum, acc) triples of up to 8 splits are merged inside a cluster
// through distributed shared memory, in one launch; otherwise they go through scratch and a second kernel.
//
// Reference: the reference has no paged attention — it re-runs the HF model over the whole right-padded
// sequence every step and throws the cache away (reference llmctl/serve/server.py:199-204; README.md:12,67
// only claims the feature).
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
// head_dim = 128: a half-warp (16 lanes x 8 elements) covers one K/V row.  A warp takes every fourth group of 4 rows per lane group;
// the rows come through a ring in shared memory that every lane fills and reads for itself (16-byte asynchronous copies, four
// groups deep, no barrier): 64 KB in flight per CTA, three CTAs per SM.  Loads into registers that were all waited for before the
// arithmetic left HBM idle in between: 16 contexts of up to 4096 (697 MB) took 195 us, now 123 us (5.7 TB/s).
// partial layout: [batch, heads, splits, head_dim + 2] fp32 = {acc[head_dim], max, sum}.
// kCluster: the splits of a (head, sequence) are one cluster and its first CTA writes the output itself.
// ---------------------------------------------------------------------------------------------
constexpr int kMaxClusterSplits = 8;         // portable cluster size
constexpr int kDecodeStages = 4, kDecodeRows = 4;
constexpr int kDecodeSmem = 128 * kDecodeStages * kDecodeRows * 32;      // a lane's ring: stages x rows x (16 bytes of K + 16 of V)

__device__ __forceinline__ void cp_async_16_or_zero(uint32_t dst, const void* src, bool valid) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst), "l"(src), "r"(valid ? 16 : 0) : "memory");
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
  constexpr int kLanesPerRow = kHeadDim / 8;          // 16 for D=128, 8 for D=64
  constexpr int kRowsPerWarp = 32 / kLanesPerRow;
  extern __shared__ __align__(16) uint8_t ring[];
  __shared__ float s_out[kHeadDim + 2];
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
  const int sub = lane / kLanesPerRow;                // which row of the warp's group
  const int li = lane % kLanesPerRow;                 // 8-element slice of the row
  const int* bt = block_tables + static_cast<long long>(b) * max_blocks_per_seq;
  const long long row_elems = static_cast<long long>(heads) * kHeadDim;
  const __nv_bfloat16* kc = k_cache + head * kHeadDim + li * 8;
  const __nv_bfloat16* vc = v_cache + head * kHeadDim + li * 8;

  float qf[8];
  unpack8(load8(q + b * q_stride + head * kHeadDim + li * 8), qf);
#pragma unroll
  for (int j = 0; j < 8; ++j) qf[j] *= scale_log2;

  float m = -INFINITY, l = 0.f, acc[8];
#pragma unroll
  for (int j = 0; j < 8; ++j) acc[j] = 0.f;

  // group g of this warp: rows t0 + ((g * 4 + warp) * kDecodeRows + u) * kRowsPerWarp + sub, u < kDecodeRows
  constexpr int kGroupTokens = kDecodeRows * kRowsPerWarp;
  const int first = t0 + warp * kGroupTokens + sub;
  const int groups = t1 > t0 ? (t1 - t0 + 4 * kGroupTokens - 1) / (4 * kGroupTokens) : 0;      // uniform over the CTA
  const uint32_t mine = ptx::smem_u32(ring) + threadIdx.x * 16;
  constexpr uint32_t kRow = 128 * 16;                 // bytes between a lane's consecutive 16-byte pieces
  auto token = [&](int g, int u) { return first + g * 4 * kGroupTokens + u * kRowsPerWarp; };
  auto page_of = [&](int t) { return bt[block_shift >= 0 ? t >> block_shift : t / block_size]; };
  auto rest_of = [&](int t) { return block_shift >= 0 ? t & (block_size - 1) : t % block_size; };
  int page[kDecodeRows];                              // pages of the next group to be fetched, looked up a group ahead
  auto look_up = [&](int g) {
#pragma unroll
    for (int u = 0; u < kDecodeRows; ++u) {
      const int t = token(g, u);
      page[u] = g < groups && t < t1 ? page_of(t) : 0;
    }
  };
  auto fetch = [&](int g) {
    if (g < groups) {
      const uint32_t at = mine + (g % kDecodeStages) * (2 * kDecodeRows * kRow);
#pragma unroll
      for (int u = 0; u < kDecodeRows; ++u) {
        const int t = token(g, u);
        const bool valid = t < t1;
        const long long off = valid ? (static_cast<long long>(page[u]) * block_size + rest_of(t)) * row_elems : 0;
        cp_async_16_or_zero(at + (2 * u) * kRow, kc + off, valid);
        cp_async_16_or_zero(at + (2 * u + 1) * kRow, vc + off, valid);
      }
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
  };
  look_up(0);
#pragma unroll
  for (int g = 0; g < kDecodeStages - 1; ++g) {
    fetch(g);
    look_up(g + 1);
  }
  // The trip count is uniform across the warp: the shuffles below use the full mask, so a lane whose token
  // is out of range still executes them (with a masked score) instead of leaving the loop early.
  for (int g = 0; g < groups; ++g) {
    fetch(g + kDecodeStages - 1);
    look_up(g + kDecodeStages);
    asm volatile("cp.async.wait_group %0;" ::"n"(kDecodeStages - 1) : "memory");
    const uint8_t* at = ring + threadIdx.x * 16 + (g % kDecodeStages) * (2 * kDecodeRows * kRow);
    float sc[kDecodeRows];
#pragma unroll
    for (int u = 0; u < kDecodeRows; ++u) {
      float kf[8];
      unpack8(*reinterpret_cast<const bf16x8*>(at + (2 * u) * kRow), kf);
      float s = 0.f;
#pragma unroll
      for (int j = 0; j < 8; ++j) s += qf[j] * kf[j];
      sc[u] = s;
    }
#pragma unroll
    for (int o = kLanesPerRow / 2; o > 0; o >>= 1)
#pragma unroll
      for (int u = 0; u < kDecodeRows; ++u) sc[u] += __shfl_xor_sync(0xffffffffu, sc[u], o);
    float m_new = m;
#pragma unroll
    for (int u = 0; u < kDecodeRows; ++u) {
      if (token(g, u) >= t1) sc[u] = -INFINITY;
      m_new = fmaxf(m_new, sc[u]);
    }
    const float ref = m_new == -INFINITY ? 0.f : m_new;      // nothing seen yet: every weight below is 0
    const float corr = exp2f(m - ref);
    l *= corr;
#pragma unroll
    for (int j = 0; j < 8; ++j) acc[j] *= corr;
#pragma unroll
    for (int u = 0; u < kDecodeRows; ++u) {
      float vf[8];
      unpack8(*reinterpret_cast<const bf16x8*>(at + (2 * u + 1) * kRow), vf);
      const float pr = exp2f(sc[u] - ref);
      l += pr;
#pragma unroll
      for (int j = 0; j < 8; ++j) acc[j] += pr * vf[j];
    }
    m = m_new;
  }
  asm volatile("cp.async.wait_all;" ::: "memory");
  __syncthreads();                                    // the ring is idle: it takes the groups' partial states

  // merge the (4 warps x kRowsPerWarp) partial states through shared memory
  constexpr int ngroups = 4 * kRowsPerWarp;
  float* s_acc = reinterpret_cast<float*>(ring);      // [ngroups][kHeadDim], then max and sum per group
  float *s_m = s_acc + ngroups * kHeadDim, *s_l = s_m + ngroups;
  const int gi = warp * kRowsPerWarp + sub;           // group id
  if (li == 0) {
    s_m[gi] = m;
    s_l[gi] = l;
  }
#pragma unroll
  for (int j = 0; j < 8; ++j) s_acc[gi * kHeadDim + li * 8 + j] = acc[j];
  __syncthreads();
  if (threadIdx.x < kHeadDim) {
    float gm = -INFINITY;
    for (int i = 0; i < ngroups; ++i) gm = fmaxf(gm, s_m[i]);
    float gl = 0.f, ga = 0.f;
    for (int i = 0; i < ngroups; ++i) {
      const float w = (s_m[i] == -INFINITY) ? 0.f : exp2f(s_m[i] - gm);
      gl += s_l[i] * w;
      ga += s_acc[i * kHeadDim + threadIdx.x] * w;
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
    const cudaError_t e = allow_smem(kern, kDecodeSmem);
    if (e != cudaSuccess) return e;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(heads, num_splits, batch);
    cfg.blockDim = dim3(128, 1, 1);
    cfg.dynamicSmemBytes = kDecodeSmem;
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
