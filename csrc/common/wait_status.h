// Bounded waits that ran out, told to the host without a copy or a synchronisation of their own.
//
// A kernel whose wait runs out leaves its outputs wrong or unwritten and still ends in order.  Beside its device-side status word it sets
// its byte of one word in mapped host memory; the host reads the word wherever it waits for results anyway, and before each launch.
#pragma once

namespace llmctl {

enum WaitReport { kWaitFlashForward = 0, kWaitFlashBackward = 1, kWaitCrossEntropy = 2, kWaitLatentAttention = 3 };

// The byte for this kernel, valid on the host and on every device; null if pinned memory cannot be had.
unsigned char* wait_report(WaitReport which);

#ifdef __CUDACC__
__device__ __forceinline__ void report_wait(unsigned char* byte) {
  *reinterpret_cast<volatile unsigned char*>(byte) = 1;
  __threadfence_system();
}
#endif

}  // namespace llmctl
