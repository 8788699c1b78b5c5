// Host-side check of the pair kernel's work-list split (bnb::work_split and
// bnb::work_level, the functions the list rebuild runs on the device): for
// every candidate count, tile count per item and tail length, the items of a
// block cover its candidates once and in order, level by level, with item
// sizes that never grow from one level to the next, and the items of either
// part of the list (full size, tail) take the places that the rebuild reserves,
// each once.  Prints "ok" or the first failing case.
#include <cstdio>
#include <initializer_list>

#include "work_split.h"

int main() {
  // a work item's word: every tile count beside the first and the last block
  for (int n = 1; n <= 32; n++)
    for (int b : {0, 1, bnb::kMaxListBlocks - 1})
      if (bnb::work_block(bnb::work_pack(b, n)) != b || bnb::work_tiles(bnb::work_pack(b, n)) != n) {
        std::printf("pack block=%d tiles=%d\n", b, n);
        return 1;
      }
  const int tails[] = {0, 1, 2, 4, 8};
  for (int T = 1; T <= 32; T++)
    for (int tail : tails)
      for (int nc = 0; nc <= 400; nc++) {
        int tiles[bnb::kWorkLevels], items[bnb::kWorkLevels];
        const int L = bnb::work_split(nc, T, tail * T, tiles, items);
        int sumTiles = 0;
        for (int l = 0; l < bnb::kWorkLevels; l++) sumTiles += tiles[l];
        const int K = nc < tail * T ? nc : tail * T;
        if (sumTiles != nc || tiles[0] != nc - K || L < 1 || L > bnb::kWorkLevels) {
          std::printf("split T=%d tail=%d nc=%d: tiles %d head %d L %d\n", T, tail, nc, sumTiles, tiles[0], L);
          return 1;
        }
        const int c0 = 1000;
        int next = c0, lastSize = 1 << 30, place[2] = {0, 0};  // places of the full-size and the tail items
        bool bad = false;
        for (int l = 0; l < L; l++) {
          const bnb::WorkLevel w = bnb::work_level(c0, T, l, tiles, items);
          int &at = place[l > 0];
          if (w.items != items[l] || w.size != bnb::work_item_size(T, l) || w.size > lastSize || w.before != at)
            bad = true;
          lastSize = w.size;
          for (int k = 0; k < w.items; k++) {
            int first, n;
            w.item(k, &first, &n);
            if (first != next || n < 1 || n > w.size) bad = true;
            next = first + n;
          }
          at += w.items;
        }
        int tail = 0;
        for (int l = 1; l < bnb::kWorkLevels; l++) tail += items[l];
        if (place[0] != items[0] || place[1] != tail) bad = true;
        if (bad || next != c0 + nc) {
          std::printf("items T=%d tail=%d nc=%d\n", T, tail, nc);
          return 1;
        }
      }
  std::printf("ok\n");
  return 0;
}
