// climb_message.h -- what a node written by k_emit_climb carries in the padding of its two corners while its
// parent is missing (see emit.cuh).  Plain C++ as well, so that it can be checked without a GPU.
#pragma once
#include <cstdint>

#ifdef __CUDACC__
#define BVHGB_HD __host__ __device__ __forceinline__
#else
#define BVHGB_HD inline
#endif

namespace bvhgb {

// The corners are two independent 16-byte stores and arrive in any order, so each says for itself that it is
// there: the lower one by the build's epoch (a nonzero multiple of 64), the upper one by a mark that is
// made from it and never 0.  Before the climb both words of every node that it writes are 0, or what a build
// that gave up left there, with another epoch (see Workspace::nodes).
BVHGB_HD uint32_t climb_mark(uint32_t epoch) { return (epoch >> 6) % 0xffffu + 1u; }
// The upper corner's word: the mark, the delta byte past the node's far end and its height.
BVHGB_HD uint32_t climb_hi_word(uint32_t mark, uint32_t delta, uint32_t height) {
  return mark << 16 | (delta & 0xffu) << 8 | (height < 255u ? height : 255u);
}
BVHGB_HD bool climb_whole(uint32_t lo_word, uint32_t hi_word, uint32_t epoch, uint32_t mark) {
  return lo_word == epoch && hi_word >> 16 == mark;
}
BVHGB_HD uint32_t climb_delta(uint32_t hi_word) { return (hi_word >> 8) & 0xffu; }
BVHGB_HD uint32_t climb_height(uint32_t hi_word) { return hi_word & 0xffu; }

}  // namespace bvhgb
