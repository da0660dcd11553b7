// The grid of a kernel whose blocks wait for one another. Plain C++ (no CUDA header).
#pragma once

namespace dlp {

enum class Launch { ok, too_large, refused, failed };  // of a cooperative launch; refused: not at any size

// A cooperative launch of a kernel that takes any number of blocks: where the device (a part of it, under a
// partition) does not hold `grid` blocks at once, half as many are tried, down to one; where it refuses
// cooperative launches, `one_block()` launches a single block, whose barriers are its own.
template <class Cooperative, class OneBlock>
inline Launch launch_resident(int grid, Cooperative cooperative, OneBlock one_block) {
  Launch r = cooperative(grid);
  while (r == Launch::too_large && grid > 1) r = cooperative(grid /= 2);
  if (r == Launch::too_large || r == Launch::refused) r = one_block();
  return r;
}

}  // namespace dlp
