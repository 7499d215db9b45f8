// Most device bytes that the kernels' scratch and a thread's staging take, shared
// by the code that allocates them and the server's admission estimate.
#pragma once
#include <stddef.h>

namespace lakgb {

constexpr size_t kBitplaneScratchBytes = size_t(64) << 20;  // terms of the bit-plane product (bitplane_tc.cu)
constexpr size_t kAnZtSnScratch = size_t(32) << 20;         // counts of An_ZtSn (bitplane.cu)
constexpr size_t kSplitMaxBytes = size_t(256) << 20;        // counts of a split Gram (gram.cu)
constexpr size_t kArenaBytes = size_t(4) << 20;             // one staging arena (lakgb_runtime.cu)
constexpr int kArenas = 8;
constexpr size_t kUpChunk = size_t(4) << 20;                // an ordinary chunk of scope uploads (loopsum.cu)
constexpr int kIdleUpChunks = 4;

}  // namespace lakgb
