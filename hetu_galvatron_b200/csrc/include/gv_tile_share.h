// Which part of which tile a CTA pair of the GEMM multiplies. Plain C++: the kernel, its host side and the host-side check of the
// arithmetic (sim/tile_share_sim.cpp) share it.
#ifndef GV_TILE_SHARE_H
#define GV_TILE_SHARE_H

#ifdef __CUDACC__
#define GV_SHARE_FN __host__ __device__ __forceinline__
#else
#define GV_SHARE_FN inline
#endif

namespace gv {

// The first `tiles` tiles of a product have `each` CTA pairs apiece, pairs each * t .. for tile t, which multiply even parts of the
// tile's `kb` k-blocks. The tiles behind them go to all the pairs whole.
struct TileShare { int tiles, each, kb; };

constexpr int MAX_SHARE = 4;

// `left` tiles that do not fill a wave of `all` pairs; none where fewer than two pairs a tile are there.
GV_SHARE_FN TileShare share_of(int left, int all, int kb) {
  int each = left > 0 ? all / left : 0;
  if (each > MAX_SHARE) each = MAX_SHARE;
  if (each > kb) each = kb;                     // no part is empty
  return each < 2 ? TileShare{0, 1, kb} : TileShare{left, each, kb};
}
GV_SHARE_FN int share_cut(const TileShare& s, int part) { return static_cast<int>(static_cast<long long>(s.kb) * part / s.each); }

struct Segment { int tile, kb0, kb1; };

// The work of one pair, in order: its part of a shared tile first, so that joining the parts overlaps with the whole tiles.
struct SegmentWalk {
  TileShare s;
  int pair, tile, step, num_tiles;
  bool part;

  GV_SHARE_FN SegmentWalk(const TileShare& share, int pair_, int num_pairs, int tiles)
      : s(share), pair(pair_), tile(share.tiles + pair_), step(num_pairs), num_tiles(tiles), part(pair_ < share.tiles * share.each) {}
  GV_SHARE_FN bool next(Segment& g) {
    if (part) {
      part = false;
      g.tile = pair / s.each;
      g.kb0 = share_cut(s, pair % s.each);
      g.kb1 = share_cut(s, pair % s.each + 1);
      return true;
    }
    g.tile = tile; g.kb0 = 0; g.kb1 = s.kb;
    tile += step;
    return g.tile < num_tiles;
  }
};

}  // namespace gv
#endif
