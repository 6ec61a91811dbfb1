// Launch shape of the Hermite 2D limiter (kh_limit).  Host code, no CUDA.
#pragma once

#include <algorithm>

namespace hteno {

struct LimitShape {
  bool wide;       // 32 lines a block (else 16)
  int lines;       // lines per block
  int segx, segy;  // segments of an x line, of a y line
};

// Segments of a line of n cells: 8 from 112 cells on, then fewer, an even number (16 lines by an odd one
// are not whole warps) of 12 cells or more, about what a repeated sweep takes to agree; 2 below 48 cells.
// One step in float, us, with the number that the shorter side of the grid gave both directions and now:
// 40 x 1000 1022 -> 572, 2000 x 40 1822 -> 779, 45 x 180 392 -> 304; 50 x 60 (four steps), 2 segments a line
// and now 4: 815 -> 736.  In double 40 x 1000 11.36 -> 7.78 ms.
inline int limit_segments(int n) { return std::max(2, std::min(8, (n + 16) / 32 * 2)); }

// 32 lines a block (coalesced) while that gives the chip's 608 sub-partitions two warps each or more; else 16:
// a small grid is bound by the length of a chain, and twice the blocks, of one warp per sub-partition, put
// its warps on more of the chip.  Measured at 2048^2 in float 0.55 -> 0.27 ms a launch (one warp per line
// group before, its block's three other warps staging the lines), at 300 x 211 in double 2.42 -> 0.43 ms.
inline LimitShape limit_shape(int nx, int ny) {
  auto blocks = [](int nl, int lines) { return 4 * ((nl + lines - 1) / lines); };
  LimitShape s;
  s.wide = (blocks(nx, 32) + blocks(ny, 32)) * 8 >= 2 * 608;
  s.lines = s.wide ? 32 : 16;
  s.segx = limit_segments(nx);
  s.segy = limit_segments(ny);
  return s;
}

}  // namespace hteno
