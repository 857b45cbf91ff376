// Which tiles of a grouped launch a CTA pair runs, and in which order.  Plain C++, so that the walk can be
// model-checked on the host.
#pragma once

#ifdef __CUDACC__
#define SD3_TILES_FN __host__ __device__ __forceinline__
#else
#define SD3_TILES_FN inline
#endif

namespace sd3 {

// The tiles of up to three problems are numbered one problem after the other: the first problem's up to end0,
// the second's up to end1, the third's up to end2.  Pair p starts with tile p; next() gives the tile that a pair runs
// after `tile`, end2 after its last.  With `sum` the third problem adds to what the first one adds to, element by
// element and after it: the pair that runs a tile of the first then runs the third's tile of the same rows
// and columns, so no pair ever waits for another one, which may not have started (pairs are not launched
// together: other work may hold SMs).  A pair's tiles are then at most those that two launches
// would give it, one of the third problem alone.
struct PairTiles {
  int end0, end1, end2;
  int sum;

  SD3_TILES_FN int next(int tile, int num_pairs) const {
    if (sum && tile < end0) return tile + end1;
    if (sum && tile >= end1) tile -= end1;
    tile += num_pairs;
    return tile < starts() ? tile : end2;
  }
  // tiles that a pair reaches by steps of num_pairs
  SD3_TILES_FN int starts() const { return sum ? end1 : end2; }
};

}  // namespace sd3
