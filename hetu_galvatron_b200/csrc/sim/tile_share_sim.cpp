// Host-side check of the shared tiles of the GEMM (include/gv_tile_share.h): for products of `--tiles` 256 x 256 tiles of `--kb` k-blocks on
// `--pairs` CTA pairs, every k-block of every tile is multiplied once, by as many pairs as a tile's joining warp counts and by those
// whose sums it reads.
//
//   g++ -std=c++17 -O1 tile_share_sim.cpp -o tile_share_sim && ./tile_share_sim --pairs 74 --tiles 300 --kb 40
#include <algorithm>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <set>
#include <vector>

#include "../include/gv_tile_share.h"

int main(int argc, char** argv) {
  int pairs = 74, most_tiles = 300, most_kb = 40;
  for (int i = 1; i + 1 < argc; i += 2) {
    if (!strcmp(argv[i], "--pairs")) pairs = atoi(argv[i + 1]);
    if (!strcmp(argv[i], "--tiles")) most_tiles = atoi(argv[i + 1]);
    if (!strcmp(argv[i], "--kb")) most_kb = atoi(argv[i + 1]);
  }
  long wrong = 0, products = 0;
  int most = 0;
  for (int tiles = 1; tiles <= most_tiles; ++tiles)
    for (int kb = 1; kb <= most_kb; ++kb) {
      const int left = tiles % pairs;
      const gv::TileShare s = gv::share_of(left, pairs, kb);
      if (s.tiles * s.each > pairs || (s.tiles != 0 && s.tiles != left)) ++wrong;
      std::vector<std::vector<int>> seen(tiles, std::vector<int>(kb, 0));
      std::vector<std::set<int>> who(tiles);
      for (int p = 0; p < pairs; ++p) {
        gv::SegmentWalk walk(s, p, pairs, tiles);
        for (gv::Segment g; walk.next(g);) {
          if (g.kb1 <= g.kb0 || g.tile < 0 || g.tile >= tiles || g.kb0 < 0 || g.kb1 > kb) { ++wrong; continue; }
          for (int k = g.kb0; k < g.kb1; ++k) ++seen[g.tile][k];
          who[g.tile].insert(p);
        }
      }
      for (auto& t : seen)
        for (int n : t) wrong += n != 1;
      for (int t = 0; t < s.tiles; ++t) {
        if (static_cast<int>(who[t].size()) != s.each || *who[t].begin() != t * s.each || *who[t].rbegin() != (t + 1) * s.each - 1) ++wrong;
        most = std::max(most, s.each);
      }
      ++products;
    }
  printf("{\"products\": %ld, \"wrong\": %ld, \"most_pairs_per_tile\": %d}\n", products, wrong, most);
  return wrong != 0;
}
