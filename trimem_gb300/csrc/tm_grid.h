// Sizes of grids whose blocks must all be on the GPU at once (host code).
#pragma once

namespace tmg {

// Launches with up to `blocks` blocks: an eighth fewer for as long as
// launch(blocks) answers `too_many`.  How many fit depends on the SMs that the
// process has, on a smaller device or in a partition of one; the runtime
// decides that at the launch and refuses it without further effect.  Returns
// the last answer and leaves in `blocks` the number it was given for.
template <class Answer, class Launch>
Answer launch_as_fits(int& blocks, Answer too_many, Launch&& launch) {
  Answer a = launch(blocks);
  while (a == too_many && blocks > 1) {
    blocks -= blocks >= 16 ? blocks / 8 : 1;
    a = launch(blocks);
  }
  return a;
}

// Elements of n that a thread of `threads` holds in registers: 1, 2, 4 or 8,
// or 0 where that is not enough
inline int elements_held(long long n, long long threads) {
  for (int e = 1; e <= 8; e *= 2)
    if (e * threads >= n) return e;
  return 0;
}

}  // namespace tmg
