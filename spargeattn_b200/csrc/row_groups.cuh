// The heads whose rows are ordered together by length: all heads of a call in `groups` even groups of consecutive ones. The
// group that is started last decides how the call ends: a remainder of one or two heads there starts its longest rows when
// the others are nearly done. (No other header but step_word.cuh: the host compiler can read this one alone.)
#pragma once
#include "step_word.cuh"

namespace sparge {

struct HeadGroup {
  int first, heads;
};

// Group g; groups differ by one head at most. 1 <= groups <= heads <= 65 535: the products fit 32 bits.
SPARGE_HOST_DEVICE HeadGroup head_group(int g, int heads, int groups) {
  const unsigned first = (unsigned)g * (unsigned)heads / (unsigned)groups, end = (unsigned)(g + 1) * (unsigned)heads / (unsigned)groups;
  return HeadGroup{(int)first, (int)(end - first)};
}
SPARGE_HOST_DEVICE int group_of_head(int head, int heads, int groups) {
  return (int)(((unsigned)(head + 1) * (unsigned)groups - 1u) / (unsigned)heads);
}

}  // namespace sparge
