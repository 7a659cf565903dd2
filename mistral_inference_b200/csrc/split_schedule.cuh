// Which thread block does which part of a sum that several blocks share.  Plain arithmetic, for the kernels and for a host compiler (the tests
// build it by itself).
//
// Some blocks wait for others of their launch: the owner of a tile adds the sums that the other parts of the tile's k range leave for it.  Blocks
// are started in the order of their index, so a block may only wait for LOWER ones: whatever share of the chip a launch gets -- another stream's
// kernels beside it, a limited set of SMs -- the lowest unfinished block never waits.
#pragma once
#ifdef __CUDACC__
#define MB_HD __host__ __device__ __forceinline__
#else
#define MB_HD inline
#endif

namespace mb200 {

// Tiles of pairs of CTAs (gemm_pair.cuh: 256 features x up to 256 tokens) run in rounds of `units` clusters; when the last round is at most half full, its tiles are cut along k
// into as many parts as fit it (at most four, eight k-blocks each, max_parts partial sums): cut_pairs tiles in `cut` parts.  No cut: 0, 1.
struct CutPlan {
  int cut_pairs, cut;
};
MB_HD CutPlan cut_plan(long long pairs, int num_k, int units, int max_parts) {
  CutPlan c = {0, 1};
  const int rest = (int)(pairs % units);
  if (rest == 0) return c;
  int cut = units / rest;
  if (cut > 4) cut = 4;
  while (cut > 1 && ((cut - 1) * rest > max_parts || num_k < 8 * cut)) --cut;
  if (cut < 2) return c;
  c.cut_pairs = rest;
  c.cut = cut;
  return c;
}

// Item s of the last round: which part of which cut tile.  The last parts come first and the owners (part 0, which holds the first k-blocks) last;
// a round is one item a cluster, so item s runs on cluster s of the launch.
struct CutItem {
  int part, slot;
};
MB_HD CutItem cut_item(int s, int cut, int cut_pairs) {
  CutItem i;
  i.part = cut - 1 - s / cut_pairs;
  i.slot = s % cut_pairs;
  return i;
}

// gemm_streamk.cuh cuts its units into one contiguous range a block; the range that holds a tile's first k-block waits for the ranges behind it.  Block
// b takes the b-th range from the end.
MB_HD int streamk_range(int block, int grid) { return grid - 1 - block; }

}  // namespace mb200
