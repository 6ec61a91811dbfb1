// Which tile shapes of the mixed FV 2D stage are timed for a grid.  Host code, no CUDA.
#pragma once

namespace hteno {

// Writes the indices (into kVariants, fv2d_fused.cu) of the candidates for `tiles` tiles of 32 x 16 cells
// on `sms` SMs, the likeliest first, and returns their number.  Timing a shape costs a new solver four
// stages, so only shapes that can win are tried.  Measured, us per pass of six steps (index: time):
//   70 to 96 tiles (224 x 160 to 256 x 192): 8, 9 or 2 win (8: 419-661, 9: 480-582, 2: 569-585), shapes for
//     three blocks an SM 690-905, 10 wins only below (96 x 80: 10: 321, 2: 468, 6: 714);
//   112 to 150 tiles: 2 wins (583-590), 1 620, 5 694-706, the small shapes 624-998, the others 848-1015;
//   160 to 252 tiles: 5, 2 or 4 win (711, 893, 919), by less and less; the small shapes 772-1634;
//   325 tiles and more: 11 or 6 win (400^2 1105, 1191; 1024^2 4417, 4506), the small shapes 1309-12387.
inline int tile_candidates(long tiles, int sms, int* out) {
  static const int few[] = {9, 8, 10, 2, 5}, wave[] = {2, 1, 5, 0}, some[] = {5, 2, 4, 0, 3, 1, 11, 6, 7},
                   many[] = {11, 6, 7, 5, 2, 4, 3, 0, 1};
  const int* list = many;
  int n = 9;
  if (3 * tiles <= 2l * sms) list = few, n = 5;
  else if (tiles <= sms) list = wave, n = 4;
  else if (tiles <= 2l * sms) list = some;
  for (int k = 0; k < n; ++k) out[k] = list[k];
  return n;
}

// Above one tile an SM a stage takes long enough for its first, cold launch to tell: a shape that is this
// much slower there than the best so far is not timed further.
inline bool tile_dropped(long tiles, int sms, float first_ms, float best_ms) {
  return tiles > sms && first_ms > 1.25f * best_ms;
}

}  // namespace hteno
