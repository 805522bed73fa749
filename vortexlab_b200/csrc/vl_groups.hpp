// When the channel moves of the warm-start network (vl_nn.cu) go in 16-byte groups.
#pragma once

#include <cstdint>

namespace vl {

constexpr long long kMoveThreads = 148LL * 32 * 256;   // of the largest grid: the step of a thread's loop
// The kernels count groups in 32 bits, and a thread's counter runs one step past the last group before its loop
// ends: from 2^32 less a step on it would wrap round and never end.
constexpr long long kMoveMost = 0x7fffffffLL;
static_assert(kMoveMost + kMoveThreads <= 0xffffffffLL, "a thread's counter must not wrap");

// Whether moves of `values` values between [.., C] and channels [coff, coff + C) of [.., ctot] go in groups of v.
inline bool move_grouped(uintptr_t a, uintptr_t b, long long values, int C, int ctot, int coff, int v) {
  return C % v == 0 && ctot % v == 0 && coff % v == 0 && !((a | b) & 15) && values / v <= kMoveMost;
}

}  // namespace vl
