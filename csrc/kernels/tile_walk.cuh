// How a product's tiles are walked and divided: index arithmetic without anything of the device in it, so that
// tests/test_tile_walk.py runs it on the host.
#pragma once
#include <stdint.h>

namespace ft {
namespace gemm {

constexpr int GROUP_M = 16;

// Tile t of the walk: groups of `group_m` row blocks, inside a group column by column, so that
// the tiles in flight at one time share few A and few B blocks (L2 reuse).  Past the end the last tile: a
// producer looks a tile ahead, and the arithmetic would divide by the rows of a group that is not there.
__device__ __forceinline__ void tile_coords(int t, int mt, int nt, int& mb, int& nb, int group_m = GROUP_M) {
  t = t < mt * nt ? t : mt * nt - 1;
  const int group_size = group_m * nt;
  const int group = t / group_size;
  const int first_m = group * group_m;
  const int gm = mt - first_m < group_m ? mt - first_m : group_m;
  const int in_group = t - group * group_size;
  mb = first_m + in_group % gm;
  nb = in_group / gm;
}

// Division of a product's work over the pairs.  Whole tiles alone leave the last round over the pairs partly
// empty: 16 x 16 tiles on 74 pairs take four rounds for 3.46 rounds of work, 12 x 7 two for 1.14, and 12 tiles of a
// long reduction use 12 pairs.  So the tiles that do not fill a round (split_tiles of them, the last of the walk)
// are cut along the reduction into split_pairs equal runs of k-blocks, one per pair, which each pair works through
// BEFORE its whole tiles.  A run holds the first part of one tile, after the last part of the tile before it, or a middle part;
// cuts that would leave fewer than SPLIT_MIN k-blocks move to the tile's edge.  The pair with a tile's last part
// owns it: the others leave their fp32 accumulators in the workspace and raise a flag per warp, and the owner's
// epilogue warps add them in the order of the reduction (the same bits every time) and store the tile, under the products of the
// pair's whole tiles where it has any.  A pair takes its first part of a tile before its last part of another, and an owner
// waits only for pairs with lower numbers, which wait for nothing that it does: any number of resident pairs make progress
// if they start in the order of their numbers.  That is how the hardware starts a grid, though nothing promises it; the
// wait is bounded like every other.
// The flags hold a token of the launch, cleared when it has been read, so that the workspace needs no preparation.
constexpr int SPLIT_MIN = 4;

struct SplitWork {
  int kt, pairs, total;                              // k-blocks of a tile, pairs that share, k-blocks shared
  __device__ __forceinline__ int begin(int p) const {
    const int b = (int)((int64_t)p * total / pairs), r = b % kt;
    return r < SPLIT_MIN ? b - r : kt - r < SPLIT_MIN ? b + kt - r : b;
  }
};

// Part `i` of a pair's work: k-blocks [kb0, kb1) of a tile; false when there is no more.
struct WorkPart { int tile, kb0, kb1; };

struct PairWork {
  SplitWork split;
  int pair, step, whole, first_split, lo, hi, mid;   // the pair's shared k-blocks [lo, hi), cut at tile edge `mid`
  __device__ __forceinline__ PairWork(int pair_, int num_pairs, int num_tiles, int kt, int split_tiles, int split_pairs)
      : split{kt, split_pairs, split_tiles * kt}, pair(pair_), step(num_pairs), whole(num_tiles - split_tiles),
        first_split(num_tiles - split_tiles), lo(0), hi(0), mid(0) {
    if (pair < split_pairs) {
      lo = split.begin(pair);
      hi = split.begin(pair + 1);
      mid = hi / kt * kt;
      if (mid < lo) mid = lo;
    }
  }
  __device__ __forceinline__ int shared() const { return (hi > mid) + (mid > lo); }
  __device__ __forceinline__ bool part(int i, WorkPart& w) const {
    const int kt = split.kt;
    if (i >= shared()) w = {pair + (i - shared()) * step, 0, kt};
    else if (i == 0 && hi > mid) w = {first_split + mid / kt, mid % kt, hi - mid / kt * kt};
    else return w = {first_split + lo / kt, lo % kt, kt}, true;
    return i < shared() || w.tile < whole;
  }
};

}  // namespace gemm
}  // namespace ft
