// Split of the pair kernel's work list into levels (no CUDA dependencies, so
// the host-side check in tests/work_split compiles it with a plain C++
// compiler).
#pragma once

#ifdef __CUDACC__
#define BNB_HD __host__ __device__
#else
#define BNB_HD
#endif

namespace bnb {

constexpr int kWorkLevels = 8;  // levels of the work list: items of T, T/2, ..., 1 tiles (T <= 32)

// A work item holds its i block and tile count (1..32) in one word.  The rebuild
// refuses lists of kMaxListBlocks blocks and more.
constexpr int kWorkBlockBits = 22, kMaxListBlocks = 1 << kWorkBlockBits;
BNB_HD inline int work_pack(int iBlock, int tiles) { return iBlock | (tiles << kWorkBlockBits); }
BNB_HD inline int work_block(int packed) { return packed & (kMaxListBlocks - 1); }
BNB_HD inline int work_tiles(int packed) { return packed >> kWorkBlockBits; }

// Split of one i block's nc candidate tiles into work items.  Level 0 takes
// the first nc - K tiles (K = min(nc, tailTiles)) in items of T tiles; the
// last K tiles form the tail, which levels 1, 2, ... take from the front in
// two items each of max(1, T >> level) tiles, the level of 1-tile items
// taking the rest.  tiles[l] and items[l] are per level; returns the number
// of levels used.  The split depends on the block's own count only.
BNB_HD inline int work_split(int nc, int T, int tailTiles, int *tiles, int *items) {
  const int K = nc < tailTiles ? nc : tailTiles;
  tiles[0] = nc - K;
  items[0] = (tiles[0] + T - 1) / T;
  int rest = K, l = 1;
  for (; l < kWorkLevels; l++) {
    const int size = (T >> l) > 1 ? (T >> l) : 1;
    const int take = size == 1 || l == kWorkLevels - 1 ? rest : (rest < 2 * size ? rest : 2 * size);
    tiles[l] = take;
    items[l] = (take + size - 1) / size;
    rest -= take;
    if (size == 1) { l++; break; }
  }
  for (int k = l; k < kWorkLevels; k++) tiles[k] = items[k] = 0;
  return l;
}

// Tile size of the items of a level.
BNB_HD inline int work_item_size(int T, int level) {
  return level == 0 ? T : ((T >> level) > 1 ? (T >> level) : 1);
}

// Work items of one level of one i block: item k (0 <= k < items) holds
// candidates first + k size .. and has place before + k among the block's items
// of its part of the list (full-size items, or tail items).
struct WorkLevel {
  int first, tiles, size, items, before;
  BNB_HD void item(int k, int *firstTile, int *n) const {
    *firstTile = first + k * size;
    const int left = first + tiles - *firstTile;
    *n = left < size ? left : size;
  }
};

// Level `level` of the block whose candidates begin at c0; tiles and items from
// work_split.  The levels together cover the candidates once, in order.
BNB_HD inline WorkLevel work_level(int c0, int T, int level, const int *tiles, const int *items) {
  WorkLevel w{c0, tiles[level], work_item_size(T, level), items[level], 0};
  for (int l = 0; l < level; l++) {
    w.first += tiles[l];
    if (l > 0) w.before += items[l];  // level 0 is a part of its own
  }
  return w;
}

}  // namespace bnb
