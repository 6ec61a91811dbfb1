// Launch of the kernels that find the largest wave speed of a new state (k_max_speed, k_inst_max_speed,
// kh_prim_f).  Host code, no CUDA.
#pragma once

#include <algorithm>
#include <cstddef>

namespace hteno {

struct SpeedLaunch {
  bool filter;      // skip cells that a float bound shows to be slower than the largest speed found
  unsigned blocks;  // of 256 threads
};

// A thread's first cell is evaluated whatever the bound says, so the filter pays where threads take several
// cells or later blocks profit from earlier ones.  set_state, us, every cell evaluated / filtered:
//   FV 2D (speed alone): 128^2 28.9 / 29.3, 400^2 44.6 / 44.9, 512^2 57.1 / 52.2, 1024^2 131 / 76;
//   Hermite 2D (prims: the float primitives too, computed twice in a filtered thread's evaluated cells):
//   128^2 30.2 / 32.5, 400^2 51.0 / 56.3, 558^2 80.0 / 85.2, 700^2 104 / 100, 1024^2 168 / 125.
// Filtered, up to 8 blocks an SM.
inline SpeedLaunch speed_launch(size_t cells, bool prims) {
  SpeedLaunch l;
  l.filter = cells > (prims ? size_t(7) << 16 : size_t(3) << 16);
  const size_t each = (cells + 255) / 256;
  l.blocks = unsigned(l.filter ? std::min<size_t>(8 * 152, each) : each);
  return l;
}

}  // namespace hteno
