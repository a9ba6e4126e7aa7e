// How many columns a block takes in the kernels that keep whole columns in shared memory.
#pragma once

#include <algorithm>

// Columns of a block in the kernels that keep whole columns in shared memory (`items`: the
// levels or faces of one that the block's 256 threads share out): whole passes of the threads
// over a block's items, so that no pass is nearly empty (33 levels, 10242 columns: acoustic
// stage 276 us with 14 columns, 303 with 11, whose last pass fills 46 of 256 threads), and no
// more than `most`.  The serial sweeps take one lane a column, and a warp takes the float64
// pipe for as long with 9 lanes as with 32, so the factorisation, whose sweep is the longer
// one, takes up to 31 columns in 6 passes (40962 x 55: 27 columns, step 24.75 ms against 24.90
// with 9, mixed form 16.46 against 16.76); the acoustic columns up to 18 in 2, where shared
// memory would otherwise hold too few blocks an SM (stage 1440 us with 9, 1466 with 15).
// A small mesh takes fewer, one pass, down to 4: float64 work is bound to its SM and the
// sweeps of a block wait for all its levels (162 columns of 12 levels: step 666 us with 4, 674
// with 16, 724 with 32; 642 of 55: 1013, 1159, 1319).
inline int columns_per_block(int nCells, int items, int cells_per_column, int most, int passes) {
  const int least = std::max(2, std::min(4, kBlock / items));
  return std::max(least, std::min({most, passes * kBlock / items, nCells / cells_per_column}));
}
