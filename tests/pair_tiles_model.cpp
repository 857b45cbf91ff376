// Walks the tiles of a grouped GEMM launch (pair_tiles.h) with any number of the launch's pairs running at a time: every
// tile has to run once, a tile that adds after another one right behind it on the same pair, and no pair may ever have
// to wait for one that has not started.  Exit status 0: holds for all sizes below, and the walk by fixed steps is found wrong.
#include <stdio.h>

#include <algorithm>
#include <vector>

#include "pair_tiles.h"

// every pair takes every num_pairs-th tile, whatever adds to what
struct FixedSteps : sd3::PairTiles {
  int next(int tile, int num_pairs) const { return tile + num_pairs < end2 ? tile + num_pairs : end2; }
  int starts() const { return end2; }
};

template <typename Walk>
static const char* check(const Walk& w, int max_pairs) {
  const int pairs = std::min(w.starts(), max_pairs);
  std::vector<int> runs(w.end2, 0);
  for (int p = 0; p < pairs; ++p) {
    int before = -1, count = 0;
    for (int t = p; t < w.end2; before = t, t = w.next(t, pairs), ++count) {
      if (t < 0 || t == before) return "a pair does not advance";
      ++runs[t];
      if (w.sum && t >= w.end1 && before != t - w.end1) return "a tile adds after one of another pair, or of an earlier turn";
    }
    // no more than a launch of the first two problems and one of the third would give the pair
    auto waves = [&](int tiles) { return (tiles + pairs - 1) / pairs; };
    if (w.sum && count > waves(w.end1) + waves(w.end2 - w.end1)) return "a pair runs more tiles than in two launches";
    if (!w.sum && count > waves(w.end2)) return "a pair runs more tiles than its share";
  }
  for (int t = 0; t < w.end2; ++t)
    if (runs[t] != 1) return "a tile does not run once";
  return nullptr;
}

int main() {
  const char* fixed = nullptr;
  for (int max_pairs : {1, 2, 3, 9, 74})
    for (int first = 1; first <= 200; first += 1 + first / 16)
      for (int second = 0; second <= 90; second += 1 + second / 8) {
        for (int third : {0, 1, first, 2 * first + 1}) {
          const sd3::PairTiles w{first, first + second, first + second + third, 0};
          if (const char* e = check(w, max_pairs)) return printf("%d %d %d of %d pairs: %s\n", first, second, third, max_pairs, e), 1;
        }
        const sd3::PairTiles w{first, first + second, 2 * first + second, 1};
        if (const char* e = check(w, max_pairs)) return printf("%d %d sum, %d pairs: %s\n", first, second, max_pairs, e), 1;
        FixedSteps f;
        static_cast<sd3::PairTiles&>(f) = w;
        if (const char* e = check(f, max_pairs)) fixed = e;
      }
  if (!fixed) return printf("the walk by fixed steps was not found wrong\n"), 1;
  printf("holds; by fixed steps: %s\n", fixed);
  return 0;
}
