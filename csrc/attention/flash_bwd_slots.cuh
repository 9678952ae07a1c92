// Slots of shared memory of the flash attention backward (flash_bwd.cu): which one a tile is loaded into, and when it is free again.
#pragma once
#include <stdint.h>

namespace llmctl {
namespace fbwd {
constexpr int kTiles = 6;

// The tiles of an item are loaded in the order res0, e0(0), res1, e1(0), e0(1), e1(1), ... (resident and streamed operands 0 and 1) and
// handed back in the order e1(0), e0(0), ..., e1(n - 2), res0, e0(n - 2), res1, e1(n - 1), e0(n - 1), that of the last products that
// read them, and a load takes the slot that was handed back first.  So the tiles of the next item's first scores are fetched while this
// one's last block is still in its softmax.  Loads and hand-backs are numbered; load l waits for hand-back l - kTiles.
struct Slots {
  uint32_t at = 0x543210u, base = 0; // the slots in the order in which this item's loads take them, four bits each; number of its first load
  __device__ __forceinline__ uint32_t slot(int j) const { return at >> (4 * j) & 15u; }
  __device__ __forceinline__ uint32_t res(int which) const { return slot(2 * which); }
  __device__ __forceinline__ uint32_t streamed(int which, int i) const {
    return ((i & 2) == 0 ? which : 1 - which) == 0 ? slot(i & 1 ? 4 : 1) : slot(i & 1 ? 5 : 3);
  }
  __device__ __forceinline__ uint32_t load_res(int which) const { return base + 2 * which; }
  __device__ __forceinline__ uint32_t load_streamed(int which, int i) const { return base + 2 + 2 * i + which - (i + which == 0 ? 1 : 0); }
  __device__ __forceinline__ uint32_t given_res(int which, int n) const { return base + (which ? 2 * n - 1 : n > 1 ? 2 * n - 3 : 0); }
  __device__ __forceinline__ uint32_t given_streamed(int which, int i, int n) const {
    return base + 2 * i + (i + 1 == n ? 3 - which : which ? 0 : i + 2 == n ? 2 : 1);
  }
  __device__ __forceinline__ void next(int n) {
    if (n == 1) {
      at = slot(4) | slot(5) << 4 | slot(0) << 8 | slot(2) << 12 | slot(3) << 16 | slot(1) << 20;
    } else {
      at = streamed(1, n - 2) | slot(0) << 4 | streamed(0, n - 2) << 8 | slot(2) << 12 | streamed(1, n - 1) << 16 | streamed(0, n - 1) << 20;
    }
    base += 2 * n + 2;
  }
};
}  // namespace fbwd
}  // namespace llmctl
