// What the attention kernel's producer warp tells the softmax warps about one 64-key block of a step: its index, and in the
// top bit that its keys need masks. (No other header: the host compiler can read this one alone.)
#pragma once
#if defined(__CUDACC__)
#define SPARGE_HOST_DEVICE __host__ __device__ __forceinline__
#else
#define SPARGE_HOST_DEVICE inline
#endif

namespace sparge {

constexpr int kStepMasked = -2147483647 - 1;

SPARGE_HOST_DEVICE int step_word(int block, bool masked) { return masked ? block | kStepMasked : block; }
SPARGE_HOST_DEVICE bool step_masked(int word) { return word < 0; }
SPARGE_HOST_DEVICE int step_index(int word) { return word & ~kStepMasked; }
// The index for a load from global memory. A wait that ran out leaves the softmax warps running on a word that was perhaps
// never written: any word gives one of the nk blocks. (Masks take step_index: they only compare it, and the clamp in their
// place cost 1-2 % of the kernel, a register that the loop does not have.)
SPARGE_HOST_DEVICE int step_block(int word, int nk) {
  const int j = step_index(word);
  return j < nk ? j : nk - 1;
}

}  // namespace sparge
