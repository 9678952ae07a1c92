// The host word of wait_status.h.
//
// Reference: none.
#include "wait_status.h"

#include "util.cuh"

namespace llmctl {

// Pinned on first use and kept: kernels in captured graphs hold the address.
static unsigned char* wait_word() {
  static unsigned char* const word = [] {
    void* p = nullptr;
    cudaStreamCaptureMode mode = cudaStreamCaptureModeRelaxed;      // the first launch may be inside a capture
    (void)cudaThreadExchangeStreamCaptureMode(&mode);
    if (cudaHostAlloc(&p, 64, cudaHostAllocPortable | cudaHostAllocMapped) != cudaSuccess) {
      (void)cudaGetLastError();
      p = nullptr;
    }
    (void)cudaThreadExchangeStreamCaptureMode(&mode);
    if (p != nullptr)
      for (int i = 0; i < 64; ++i) static_cast<unsigned char*>(p)[i] = 0;
    return static_cast<unsigned char*>(p);
  }();
  return word;
}

unsigned char* wait_report(WaitReport which) {
  unsigned char* const w = wait_word();
  return w == nullptr ? nullptr : w + which;
}

__global__ void wait_report_kernel(unsigned char* byte) { report_wait(byte); }

}  // namespace llmctl

using namespace llmctl;

// The host word (one byte per kernel in the order of WaitReport), or null.
LLMCTL_API void* llmctl_wait_status_word() { return wait_word(); }

// Sets a kernel's byte from the device, as its waits do when they run out.
LLMCTL_API int llmctl_wait_status_report(int which, void* stream) {
  LLMCTL_BEGIN();
  LLMCTL_REQUIRE(which >= 0 && which < 4);
  unsigned char* const byte = wait_report(static_cast<WaitReport>(which));
  LLMCTL_REQUIRE(byte != nullptr);
  wait_report_kernel<<<1, 1, 0, (cudaStream_t)stream>>>(byte);
  LLMCTL_RETURN_LAST();
}
