// Split of a march along z among blocks (host arithmetic, no CUDA).
#pragma once

#include <cstdint>

namespace simp {

// Node layers a block marches of `layers` layers with `columns` block columns
// in x and y on a GPU that holds `slots` blocks at a time: the fewest block
// steps, waves x (layers + 2), since a block's march costs its layers and about
// two more to fill and drain (97x49x49: one wave of 5 layers 12.8 us, 4 layers
// in 1.2 waves 14.9, 8 layers in 0.6 waves 14.9); of equals the least.  For
// each number of waves the least layers that fit it: about layers / slots tries,
// where trying every count of layers took 0.2 ms of host time a launch at 60,001
// layers (1x1x60000 cells: 148 against 141 ms a design pass without the kernel).
inline int64_t march_layers(int64_t columns, int64_t layers, int64_t slots) {
  int64_t best = layers, steps = INT64_MAX;
  for (int64_t waves = (columns + slots - 1) / slots; 3 * waves <= steps; ++waves) {
    int64_t chunks = waves * slots / columns;
    if (chunks > layers) chunks = layers;
    const int64_t l = (layers + chunks - 1) / chunks;
    const int64_t s = (columns * ((layers + l - 1) / l) + slots - 1) / slots * (l + 2);
    if (s <= steps) {
      steps = s;
      best = l;
    }
    if (l == 1) break;
  }
  return best;
}

}  // namespace simp
