// K15 (single-rank part): fused softmax cross-entropy forward + backward over bf16 logits.
// One pass over HBM: the row is held in registers, the per-row loss (fp32) is written out and the
// logits buffer is overwritten in place with d(loss)/d(logits) = (softmax - onehot) * grad_scale.
//
// Reference: HF `CrossEntropyLoss` on fp32-upcast logits inside `self.model(**batch)`
// (reference llmctl/runtime/engine.py:284-285).  Baseline to beat: ATen log_softmax + nll_loss
// (+ their backward), which materialises [M, V] fp32 twice.
//
// The vocab-parallel variant (logits sharded over TP ranks) splits this into "partial max/sumexp",
// an all-reduce, and "finalize"; both halves are exposed below.
#include "../common/dependent.cuh"
#include "../common/ptx.cuh"
#include "../common/util.cuh"
#include "../common/wait_status.h"

namespace llmctl {

constexpr int kCEThreads = 512;

// kVec: 16-byte groups cached in registers per thread (V <= kVec * 512 * 8).
template <int kVec>
__global__ void __launch_bounds__(kCEThreads)
ce_fwd_bwd_kernel(__nv_bfloat16* __restrict__ logits, long long ld, const long long* __restrict__ targets,
                  float* __restrict__ loss_out, float* __restrict__ lse_out, int V,
                  long long ignore_index, float host_scale, const float* __restrict__ scale_dev,
                  int write_grad) {
  __shared__ float red[32];
  const int row = blockIdx.x;
  __nv_bfloat16* p = logits + static_cast<long long>(row) * ld;
  const int nvec = V >> 3;
  const long long tgt = targets[row];
  bf16x8 data[kVec];
  float mx = -INFINITY;
#pragma unroll
  for (int i = 0; i < kVec; ++i) {
    const int v = i * kCEThreads + threadIdx.x;
    if (v < nvec) {
      data[i] = load8(p + v * 8);
      float a[8];
      unpack8(data[i], a);
#pragma unroll
      for (int j = 0; j < 8; ++j) mx = fmaxf(mx, a[j]);
    }
  }
  mx = block_max(mx, red);
  float se = 0.f;
#pragma unroll
  for (int i = 0; i < kVec; ++i) {
    const int v = i * kCEThreads + threadIdx.x;
    if (v < nvec) {
      float a[8];
      unpack8(data[i], a);
#pragma unroll
      for (int j = 0; j < 8; ++j) se += __expf(a[j] - mx);
    }
  }
  se = block_sum(se, red);
  const float lse = mx + __logf(se);
  const bool ignored = (tgt == ignore_index) || tgt < 0 || tgt >= V;
  if (threadIdx.x == 0) {
    if (lse_out) lse_out[row] = lse;
    float tl = 0.f;
    if (!ignored) tl = lse - __bfloat162float(p[tgt]);
    loss_out[row] = tl;
  }
  if (!write_grad) return;
  float scale = host_scale;
  if (scale_dev != nullptr) scale *= *scale_dev;
  if (ignored) scale = 0.f;
  __syncthreads();  // thread 0 has read p[tgt] before anyone overwrites the row
  const float inv_se = 1.f / se;
#pragma unroll
  for (int i = 0; i < kVec; ++i) {
    const int v = i * kCEThreads + threadIdx.x;
    if (v < nvec) {
      float a[8], g[8];
      unpack8(data[i], a);
#pragma unroll
      for (int j = 0; j < 8; ++j) {
        float sm = __expf(a[j] - mx) * inv_se;
        if (v * 8 + j == tgt) sm -= 1.f;
        g[j] = sm * scale;
      }
      store8(p + v * 8, pack8(g));
    }
  }
}

// Rows of 8 K (8200) to 55 K logits (kCERingBytes / 4 = 56320): persistent CTAs with a ring of two or three whole rows in shared memory.  Bound by HBM (the row is read and
// written once): while a row is reduced and differentiated the next is copied in and the one before is copied out by bulk copies,
// which a CTA that loads, reduces and stores one row after the other cannot do (4096 x 32000: 204 us, two of them
// per SM; here 118 us = 4.4 TB/s).  Maximum
// and sum of exponentials come from one pass per thread and one block reduction of (maximum, sum) pairs, and up to 32 K logits the
// exponentials are kept for the gradient.
constexpr int kCERingBytes = 220 * 1024;
__device__ unsigned int g_ce_status = 0;       // != 0: a bounded wait ran out

template <int kVec>
__global__ void __launch_bounds__(kCEThreads, 1)
ce_rows_kernel(__nv_bfloat16* __restrict__ logits, long long ld, const long long* __restrict__ targets, float* __restrict__ loss_out,
               float* __restrict__ lse_out, int rows, int V, int stages, long long ignore_index, float host_scale,
               const float* __restrict__ scale_dev, int write_grad, unsigned char* wait_byte) {
  using namespace ptx;
  extern __shared__ __align__(128) uint8_t ring[];
  __shared__ uint64_t full[3];
  __shared__ float red_m[2][kCEThreads / 32], red_s[2][kCEThreads / 32];
  __shared__ int abort_flag;
  constexpr float kLog2e = 1.4426950408889634f;
  constexpr bool kKeep = kVec <= 8;      // the exponentials fit the registers: the gradient needs no second ones
  const int nvec = V >> 3, lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const uint32_t row_bytes = static_cast<uint32_t>(V) * 2;
  if (threadIdx.x == 0) {
    for (int i = 0; i < 3; ++i) mbar_init(&full[i], 1);
    abort_flag = 0;
    fence_mbar_init();
  }
  __syncthreads();
  auto begin_load = [&](int row, int st) {
    mbar_expect_tx(&full[st], row_bytes);
    bulk_load_1d(ring + st * row_bytes, logits + static_cast<long long>(row) * ld, row_bytes, &full[st]);
  };
  const int first = blockIdx.x, step = gridDim.x;
  if (threadIdx.x == 0)
    for (int i = 0; i < stages - 1 && first + i * step < rows; ++i) begin_load(first + i * step, i);
  float scale0 = host_scale;
  if (scale_dev != nullptr) scale0 *= *scale_dev;
  int i = 0;
  for (int row = first; row < rows; row += step, ++i) {
    const int st = i % stages;
    const long long tgt = targets[row];
    const bool ignored = (tgt == ignore_index) || tgt < 0 || tgt >= V;
    const bool ok = mbar_wait_bounded(&full[st], (i / stages) & 1, &abort_flag);
    if (!__syncthreads_and(ok)) break;
    __nv_bfloat16* p = reinterpret_cast<__nv_bfloat16*>(ring + st * row_bytes);
    bf16x8 data[kVec];
    float m = -INFINITY, se = 0.f;
#pragma unroll
    for (int v = 0; v < kVec; ++v) {
      const int at = v * kCEThreads + threadIdx.x;
      if (at < nvec) {
        data[v] = load8(p + at * 8);
        float a[8];
        unpack8(data[v], a);
        m = max3(m, a[0], a[1]);
        m = max3(m, a[2], a[3]);
        m = max3(m, a[4], a[5]);
        m = max3(m, a[6], a[7]);
      }
    }
    const float neg_m = m == -INFINITY ? 0.f : -m;
    float se1 = 0.f;
    float ex[kKeep ? kVec * 8 : 1];      // exponentials relative to this thread's maximum
#pragma unroll
    for (int v = 0; v < kVec; ++v) {
      if (v * kCEThreads + threadIdx.x < nvec) {
        float a[8];
        unpack8(data[v], a);
#pragma unroll
        for (int j = 0; j < 8; j += 2) {
          float x0, x1;
          add2v(x0, x1, a[j], a[j + 1], neg_m, neg_m);
          mul2(x0, x1, x0, x1, kLog2e);
          const float e0 = ex2_approx(x0), e1 = ex2_approx(x1);
          add2(se, se1, e0, e1);
          if (kKeep) {
            ex[v * 8 + j] = e0;
            ex[v * 8 + j + 1] = e1;
          }
        }
      }
    }
    se += se1;
    // (maximum, sum) of the warp, then of the block; the rows alternate between two sets of slots
    const float wm = warp_max(m);
    se = warp_sum(m == -INFINITY && se == 0.f ? 0.f : se * __expf(m - wm));
    if (lane == 0) {
      red_m[i & 1][warp] = wm;
      red_s[i & 1][warp] = se;
    }
    float target_logit = 0.f;
    if (threadIdx.x == 0 && !ignored) target_logit = __bfloat162float(p[tgt]);
    __syncthreads();
    const float pm = lane < kCEThreads / 32 ? red_m[i & 1][lane] : -INFINITY;
    const float ps = lane < kCEThreads / 32 ? red_s[i & 1][lane] : 0.f;
    const float mx = warp_max(pm);
    float sum = warp_sum(pm == -INFINITY && ps == 0.f ? 0.f : ps * __expf(pm - mx));
    if (mx == -INFINITY) sum = NAN;      // a row without a finite logit has no distribution: NaN in its loss and gradient, as everywhere else
    if (threadIdx.x == 0) {
      const float lse = mx + __logf(sum);
      if (lse_out) lse_out[row] = lse;
      loss_out[row] = ignored ? 0.f : lse - target_logit;
    }
    if (write_grad) {
      const float scale = ignored ? 0.f : scale0, by = scale / sum;
      const float mine = __expf(m - mx) * by;
#pragma unroll
      for (int v = 0; v < kVec; ++v) {
        const int at = v * kCEThreads + threadIdx.x;
        if (at < nvec) {
          float a[8];
          if (kKeep) {
#pragma unroll
            for (int j = 0; j < 8; j += 2) mul2(a[j], a[j + 1], ex[v * 8 + j], ex[v * 8 + j + 1], mine);
          } else {
            unpack8(data[v], a);
#pragma unroll
            for (int j = 0; j < 8; j += 2) {
              float x0, x1;
              add2v(x0, x1, a[j], a[j + 1], -mx, -mx);
              mul2(x0, x1, x0, x1, kLog2e);
              mul2(a[j], a[j + 1], ex2_approx(x0), ex2_approx(x1), by);
            }
          }
          if (!ignored && tgt >> 3 == at) {
#pragma unroll
            for (int j = 0; j < 8; ++j)
              if ((tgt & 7) == j) a[j] -= scale;
          }
          store8(p + at * 8, pack8(a));
        }
      }
      fence_proxy_async_smem();
    }
    __syncthreads();                     // the row is done with (and, with gradients, whole in shared memory)
    if (threadIdx.x == 0) {
      if (write_grad) {
        bulk_store_1d(logits + static_cast<long long>(row) * ld, p, row_bytes);
        tma_store_commit();
      }
      const int next = row + (stages - 1) * step;
      if (next < rows) {                 // into the stage of the row before, whose copy out has been read by then
        tma_store_wait_read<1>();
        begin_load(next, (i + stages - 1) % stages);
      }
    }
  }
  if (threadIdx.x == 0) {
    if (abort_flag) {
      // let the copies in flight land before the shared memory is given back
      int none = 0;
      for (int k = i; k < i + stages - 1 && first + k * step < rows; ++k, none = 0)
        mbar_wait_bounded(&full[k % stages], (k / stages) & 1, &none);
      atomicCAS(&g_ce_status, 0u, 1u);
      report_wait(wait_byte);
    }
    tma_store_wait_read<0>();
  }
}

// Large-vocab fallback: three sweeps over the row (the 2nd and 3rd hit L2).
__global__ void __launch_bounds__(kCEThreads)
ce_fwd_bwd_stream_kernel(__nv_bfloat16* __restrict__ logits, long long ld,
                         const long long* __restrict__ targets, float* __restrict__ loss_out,
                         float* __restrict__ lse_out, int V, long long ignore_index,
                         float host_scale, const float* __restrict__ scale_dev, int write_grad) {
  __shared__ float red[32];
  const int row = blockIdx.x;
  __nv_bfloat16* p = logits + static_cast<long long>(row) * ld;
  const int nvec = V >> 3;
  const long long tgt = targets[row];
  float mx = -INFINITY;
  for (int v = threadIdx.x; v < nvec; v += kCEThreads) {
    float a[8];
    unpack8(load8(p + v * 8), a);
#pragma unroll
    for (int j = 0; j < 8; ++j) mx = fmaxf(mx, a[j]);
  }
  mx = block_max(mx, red);
  float se = 0.f;
  for (int v = threadIdx.x; v < nvec; v += kCEThreads) {
    float a[8];
    unpack8(load8(p + v * 8), a);
#pragma unroll
    for (int j = 0; j < 8; ++j) se += __expf(a[j] - mx);
  }
  se = block_sum(se, red);
  const float lse = mx + __logf(se);
  const bool ignored = (tgt == ignore_index) || tgt < 0 || tgt >= V;
  if (threadIdx.x == 0) {
    if (lse_out) lse_out[row] = lse;
    loss_out[row] = ignored ? 0.f : lse - __bfloat162float(p[tgt]);
  }
  if (!write_grad) return;
  float scale = host_scale;
  if (scale_dev != nullptr) scale *= *scale_dev;
  if (ignored) scale = 0.f;
  __syncthreads();
  const float inv_se = 1.f / se;
  for (int v = threadIdx.x; v < nvec; v += kCEThreads) {
    float a[8], g[8];
    unpack8(load8(p + v * 8), a);
#pragma unroll
    for (int j = 0; j < 8; ++j) {
      float sm = __expf(a[j] - mx) * inv_se;
      if (v * 8 + j == tgt) sm -= 1.f;
      g[j] = sm * scale;
    }
    store8(p + v * 8, pack8(g));
  }
}

// Vocab-parallel pieces.  Stage A: per-row local max and sum(exp(x - local_max)) plus the target
// logit if this shard owns it (else 0).  stats[row] = {max, sumexp, target_logit}.
__global__ void __launch_bounds__(kCEThreads)
ce_partial_kernel(const __nv_bfloat16* __restrict__ logits, long long ld,
                  const long long* __restrict__ targets, float* __restrict__ stats, int V_local,
                  long long vocab_start) {
  __shared__ float red[32];
  const int row = blockIdx.x;
  const __nv_bfloat16* p = logits + static_cast<long long>(row) * ld;
  const int nvec = V_local >> 3;
  float mx = -INFINITY;
  for (int v = threadIdx.x; v < nvec; v += kCEThreads) {
    float a[8];
    unpack8(load8(p + v * 8), a);
#pragma unroll
    for (int j = 0; j < 8; ++j) mx = fmaxf(mx, a[j]);
  }
  mx = block_max(mx, red);
  float se = 0.f;
  for (int v = threadIdx.x; v < nvec; v += kCEThreads) {
    float a[8];
    unpack8(load8(p + v * 8), a);
#pragma unroll
    for (int j = 0; j < 8; ++j) se += __expf(a[j] - mx);
  }
  se = block_sum(se, red);
  if (threadIdx.x == 0) {
    const long long t = targets[row] - vocab_start;
    stats[row * 3 + 0] = mx;
    stats[row * 3 + 1] = se;
    stats[row * 3 + 2] = (t >= 0 && t < V_local) ? __bfloat162float(p[t]) : 0.f;
  }
}
// Stage B: given the global log-sum-exp per row, overwrite the local shard with the gradient.
__global__ void __launch_bounds__(kCEThreads)
ce_finalize_kernel(__nv_bfloat16* __restrict__ logits, long long ld,
                   const long long* __restrict__ targets, const float* __restrict__ lse, int V_local,
                   long long vocab_start, long long ignore_index, float host_scale,
                   const float* __restrict__ scale_dev) {
  const int row = blockIdx.x;
  __nv_bfloat16* p = logits + static_cast<long long>(row) * ld;
  const int nvec = V_local >> 3;
  const long long tg = targets[row];
  const long long t = tg - vocab_start;
  float scale = host_scale;
  if (scale_dev != nullptr) scale *= *scale_dev;
  if (tg == ignore_index || tg < 0) scale = 0.f;
  const float l = lse[row];
  for (int v = threadIdx.x; v < nvec; v += kCEThreads) {
    float a[8], g[8];
    unpack8(load8(p + v * 8), a);
#pragma unroll
    for (int j = 0; j < 8; ++j) {
      float sm = __expf(a[j] - l);
      if (v * 8 + j == t) sm -= 1.f;
      g[j] = sm * scale;
    }
    store8(p + v * 8, pack8(g));
  }
}

// 1 / max(1, number of targets that are not ignore_index)
__global__ void __launch_bounds__(1024)
ce_count_kernel(const long long* __restrict__ targets, int rows, long long ignore_index, float* __restrict__ inv_count) {
  wait_for_previous(targets, inv_count);
  int n = 0;
#pragma unroll 8
  for (int i = threadIdx.x; i < rows; i += 1024) n += targets[i] != ignore_index ? 1 : 0;
  __shared__ int warp_count[32];
  n = __reduce_add_sync(0xffffffffu, n);
  if ((threadIdx.x & 31) == 0) warp_count[threadIdx.x >> 5] = n;
  __syncthreads();
  if (threadIdx.x < 32) {
    n = __reduce_add_sync(0xffffffffu, warp_count[threadIdx.x]);
    if (threadIdx.x == 0) *inv_count = 1.f / static_cast<float>(n < 1 ? 1 : n);
  }
}

// loss = scale * inv_count * sum of the rows' losses, summed in a fixed order; inv_count lies behind them
__global__ void __launch_bounds__(1024)
ce_mean_kernel(const float* __restrict__ row_losses, int rows, float scale, float* __restrict__ loss) {
  __shared__ float red[32];
  wait_for_previous(row_losses, loss);
  float sum = 0.f;
#pragma unroll 8
  for (int i = threadIdx.x; i < rows; i += 1024) sum += row_losses[i];
  sum = block_sum(sum, red);
  if (threadIdx.x == 0) *loss = sum * row_losses[rows] * scale;
}

}  // namespace llmctl

using namespace llmctl;

LLMCTL_API int llmctl_cross_entropy_fwd_bwd(void* logits, long long ld, const long long* targets,
                                            float* loss_per_row, float* lse_per_row, int rows,
                                            int V, long long ignore_index, float host_scale,
                                            const float* scale_dev, int write_grad, void* stream) {
  LLMCTL_BEGIN();
  LLMCTL_REQUIRE(V % 8 == 0 && ld % 8 == 0 && ld >= V && (reinterpret_cast<uintptr_t>(logits) & 15) == 0);
  if (rows == 0) return 0;
  cudaStream_t s = (cudaStream_t)stream;
  const int nvec = V / 8;
  const int kv = (nvec + kCEThreads - 1) / kCEThreads;
#define LAUNCH(KV)                                                                             \
  ce_fwd_bwd_kernel<KV><<<rows, kCEThreads, 0, s>>>((__nv_bfloat16*)logits, ld, targets,        \
                                                    loss_per_row, lse_per_row, V, ignore_index, \
                                                    host_scale, scale_dev, write_grad)
  const size_t row_bytes = static_cast<size_t>(V) * 2;
  const int stages = row_bytes * 3 <= kCERingBytes ? 3 : 2;
  auto rows_launch = [&](auto kern) -> cudaError_t {
    unsigned char* const wait_byte = wait_report(kWaitCrossEntropy);
    if (wait_byte == nullptr) return cudaErrorMemoryAllocation;
    const cudaError_t e = allow_smem(kern, kCERingBytes);
    if (e != cudaSuccess) return e;
    kern<<<rows < kNumSMs ? rows : kNumSMs, kCEThreads, stages * row_bytes, s>>>((__nv_bfloat16*)logits, ld, targets, loss_per_row, lse_per_row, rows,
                                                                                 V, stages, ignore_index, host_scale, scale_dev, write_grad, wait_byte);
    return cudaSuccess;
  };
  // short rows: several CTAs per SM overlap each other; rows that do not fit the ring twice stream through L2
  if (kv <= 2) LAUNCH(2);
  else if (row_bytes * 2 > kCERingBytes)
    ce_fwd_bwd_stream_kernel<<<rows, kCEThreads, 0, s>>>((__nv_bfloat16*)logits, ld, targets,
                                                         loss_per_row, lse_per_row, V, ignore_index,
                                                         host_scale, scale_dev, write_grad);
  else if (kv <= 4) LLMCTL_CHECK(rows_launch(ce_rows_kernel<4>));
  else if (kv <= 8) LLMCTL_CHECK(rows_launch(ce_rows_kernel<8>));
  else LLMCTL_CHECK(rows_launch(ce_rows_kernel<14>));
#undef LAUNCH
  LLMCTL_RETURN_LAST();
}

// The mean over the rows whose target is not ignore_index, times grad_scale, with the gradient's 1 / count.  Bound by launches: three
// here, where the count, its reciprocal and the mean took ten of the library's around the rows' kernel.  us per call before / after:
// 64 x 4096 76 / 26, 300 x 32000 72 / 26, 1024 x 32000 75 / 40, 4096 x 32000 148 / 116 (the rows' kernel alone 112).  One block each: 4096
// targets are four loads in flight per thread, 8192 and more eight, and the sum has a fixed order.
// work: fp32 [rows + 1], loss: fp32 [1].
LLMCTL_API int llmctl_cross_entropy_mean(void* logits, long long ld, const long long* targets, float* work, int rows, int V, long long ignore_index,
                                         float grad_scale, int write_grad, float* loss, void* stream) {
  LLMCTL_BEGIN();
  LLMCTL_REQUIRE(V % 8 == 0 && ld % 8 == 0 && ld >= V && (reinterpret_cast<uintptr_t>(logits) & 15) == 0);
  cudaStream_t s = (cudaStream_t)stream;
  LLMCTL_CHECK(launch_dependent(ce_count_kernel, 1, 1024, 0, s, targets, rows, ignore_index, work + rows));
  const int rc = llmctl_cross_entropy_fwd_bwd(logits, ld, targets, work, nullptr, rows, V, ignore_index, grad_scale, work + rows, write_grad, stream);
  if (rc) return rc;
  LLMCTL_CHECK(launch_dependent(ce_mean_kernel, 1, 1024, 0, s, work, rows, grad_scale, loss));
  return 0;
}

LLMCTL_API int llmctl_cross_entropy_partial(const void* logits, long long ld,
                                            const long long* targets, float* stats, int rows,
                                            int V_local, long long vocab_start, void* stream) {
  LLMCTL_BEGIN();
  LLMCTL_REQUIRE(V_local % 8 == 0 && ld % 8 == 0 && (reinterpret_cast<uintptr_t>(logits) & 15) == 0);
  if (rows == 0) return 0;
  ce_partial_kernel<<<rows, kCEThreads, 0, (cudaStream_t)stream>>>(
      (const __nv_bfloat16*)logits, ld, targets, stats, V_local, vocab_start);
  LLMCTL_RETURN_LAST();
}

LLMCTL_API int llmctl_cross_entropy_finalize(void* logits, long long ld, const long long* targets,
                                             const float* lse, int rows, int V_local,
                                             long long vocab_start, long long ignore_index,
                                             float host_scale, const float* scale_dev,
                                             void* stream) {
  LLMCTL_BEGIN();
  LLMCTL_REQUIRE(V_local % 8 == 0 && ld % 8 == 0 && (reinterpret_cast<uintptr_t>(logits) & 15) == 0);
  if (rows == 0) return 0;
  ce_finalize_kernel<<<rows, kCEThreads, 0, (cudaStream_t)stream>>>(
      (__nv_bfloat16*)logits, ld, targets, lse, V_local, vocab_start, ignore_index, host_scale,
      scale_dev);
  LLMCTL_RETURN_LAST();
}

// 0 unless a bounded wait of the loss kernel ran out since the last clearing call (synchronises the device).
LLMCTL_API int llmctl_cross_entropy_status(int clear) {
  unsigned int v = 0;
  if (cudaMemcpyFromSymbol(&v, g_ce_status, sizeof(v)) != cudaSuccess) return -1;
  if (clear && v != 0) {
    const unsigned int zero = 0;
    (void)cudaMemcpyToSymbol(g_ce_status, &zero, sizeof(zero));
  }
  return static_cast<int>(v);
}
