// Elimination order of the dense bottom inverse.
//
// The bottom operator couples a node with its 26 neighbours only.  Its inverse
// is dense, but while the blocked Gauss-Jordan elimination runs most tiles are
// still zero if the unknowns are numbered well: a step touches only the tiles
// its pivot row reaches.  Nodes are numbered by nested dissection (a node plane
// across the longest extent separates two halves that do not see one another
// until the plane itself is eliminated, last) and plane by plane inside a part.
// Parts start on tile boundaries, so that no tile ties two of them together;
// the padding is identity rows.  Parts of up to LEAF_UNKNOWNS are not cut:
// below that the padding (half a tile a part on average, which every
// application of the inverse pays) costs more than the cut saves.
#pragma once
#include <algorithm>
#include <array>
#include <climits>
#include <unordered_map>
#include <vector>

namespace sgs {

struct BottomOrder {
  static constexpr int LEAF_UNKNOWNS = 4096;
  int tile = 128;
  std::vector<std::array<int, 3>> at;      // node coordinates
  std::vector<int> pos;                    // node -> its first unknown
  std::vector<int> pad;                    // identity rows
  long ld = 0;                             // unknowns and padding, a multiple of tile
  std::vector<int> list;                   // concatenated: the tiles step K touches, ascending, without K
  std::vector<int> first;                  // step K's are list[first[K]] .. list[first[K + 1]]
  std::vector<int> below;                  // how many of them are smaller than K
  // the application: for each phase the row tiles and, per tile, the column
  // ranges [c0, c1) of its nonzero tiles (range k of row i: at[first[i] + k])
  struct Phase {
    std::vector<int> tiles, first, ranges;
  };
  Phase phase[3];
  // no separators: phase 0 alone, with the full inverse.  (Not "one leaf": where
  // the plane at one end holds more nodes than the rest, a cut through it leaves
  // one leaf and that separator.)
  bool single = true;

  void build(int tile_size) {
    tile = tile_size;
    pos.assign(at.size(), 0);
    pad.clear();
    ld = 0;
    std::vector<int> all(at.size());
    for (size_t i = 0; i < all.size(); ++i) all[i] = int(i);
    leaf.clear();
    dissect(all);
    symbolic();
    single = phase[1].tiles.empty();
  }

 private:
  std::vector<char> leaf;                  // tile -> whether it is a leaf's (else a separator's)
  // the axis of the largest extent of `nodes` and its range
  int longest(const std::vector<int>& nodes, int* lo, int* hi) const {
    int best = 0;
    for (int a = 0; a < 3; ++a) {
      int l = INT_MAX, h = INT_MIN;
      for (int i : nodes) l = std::min(l, at[size_t(i)][size_t(a)]), h = std::max(h, at[size_t(i)][size_t(a)]);
      if (a == 0 || h - l > *hi - *lo) best = a, *lo = l, *hi = h;
    }
    return best;
  }
  void place(std::vector<int>& nodes, int axis, bool is_leaf) {
    const int b = (axis + 1) % 3, c = (axis + 2) % 3;
    std::sort(nodes.begin(), nodes.end(), [&](int i, int j) {
      const auto &p = at[size_t(i)], &q = at[size_t(j)];
      if (p[size_t(axis)] != q[size_t(axis)]) return p[size_t(axis)] < q[size_t(axis)];
      if (p[size_t(b)] != q[size_t(b)]) return p[size_t(b)] < q[size_t(b)];
      return p[size_t(c)] < q[size_t(c)];
    });
    for (int i : nodes) {
      pos[size_t(i)] = int(ld);
      ld += 3;
    }
    while (ld % tile) pad.push_back(int(ld++));
    leaf.resize(size_t(ld / tile), is_leaf);
  }
  void dissect(std::vector<int>& nodes) {
    if (nodes.empty()) return;
    int lo = 0, hi = 0;
    const int axis = longest(nodes, &lo, &hi);
    if (3 * long(nodes.size()) <= LEAF_UNKNOWNS || hi - lo < 2) return place(nodes, axis, true);
    // the plane that splits the nodes most evenly
    std::vector<long> count(size_t(hi - lo + 1), 0);
    for (int i : nodes) ++count[size_t(at[size_t(i)][size_t(axis)] - lo)];
    long left = 0, best = LONG_MAX;
    int cut = lo;
    for (int p = lo; p <= hi; ++p) {
      const long right = long(nodes.size()) - left - count[size_t(p - lo)];
      if (std::max(left, right) < best) best = std::max(left, right), cut = p;
      left += count[size_t(p - lo)];
    }
    std::vector<int> side[3];
    for (int i : nodes) {
      const int c = at[size_t(i)][size_t(axis)];
      side[c < cut ? 0 : (c > cut ? 1 : 2)].push_back(i);
    }
    dissect(side[0]);
    dissect(side[1]);
    int l2 = 0, h2 = 0;
    if (!side[2].empty()) place(side[2], longest(side[2], &l2, &h2), false);
  }
  // tiles that each Gauss-Jordan step touches: row K's nonzero tiles S (a
  // separator's: separators only); the step fills all tiles of S x S
  void symbolic() {
    const int nt = int(ld / tile);
    std::vector<std::vector<char>> on(size_t(nt), std::vector<char>(size_t(nt), 0));
    for (int K = 0; K < nt; ++K) on[size_t(K)][size_t(K)] = 1;
    if (!at.empty()) {
      int lo[3], dim[3];
      for (int a = 0; a < 3; ++a) {
        int l = INT_MAX, h = INT_MIN;
        for (const auto& p : at) l = std::min(l, p[size_t(a)]), h = std::max(h, p[size_t(a)]);
        lo[a] = l - 1;
        dim[a] = h - l + 3;
      }
      // node at a place: a dense grid, or a map where the nodes are few and far apart
      auto cell = [&](int x, int y, int z) { return (long(x - lo[0]) * dim[1] + (y - lo[1])) * dim[2] + (z - lo[2]); };
      const long volume = long(dim[0]) * dim[1] * dim[2];
      const bool dense = volume <= (1L << 24);
      std::vector<int> grid(dense ? size_t(volume) : 0, -1);
      std::unordered_map<long, int> sparse;
      for (size_t i = 0; i < at.size(); ++i) {
        const long c = cell(at[i][0], at[i][1], at[i][2]);
        if (dense) grid[size_t(c)] = int(i);
        else sparse.emplace(c, int(i));
      }
      auto node = [&](long c) {
        if (dense) return grid[size_t(c)];
        const auto it = sparse.find(c);
        return it == sparse.end() ? -1 : it->second;
      };
      for (size_t i = 0; i < at.size(); ++i)
        for (int q = 0; q < 27; ++q) {
          const int j = node(cell(at[i][0] + q / 9 - 1, at[i][1] + q / 3 % 3 - 1, at[i][2] + q % 3 - 1));
          if (j < 0) continue;
          for (int r : {pos[i] / tile, (pos[i] + 2) / tile})
            for (int c : {pos[size_t(j)] / tile, (pos[size_t(j)] + 2) / tile}) on[size_t(r)][size_t(c)] = 1;
        }
    }
    list.clear();
    first.assign(1, 0);
    below.clear();
    for (int K = 0; K < nt; ++K) {
      int low = 0;
      std::vector<int> S;
      for (int J = 0; J < nt; ++J)
        if (J != K && on[size_t(K)][size_t(J)] && (leaf[size_t(K)] || !leaf[size_t(J)])) {
          S.push_back(J);
          low += J < K;
        }
      for (int I : S)
        for (int J : S) on[size_t(I)][size_t(J)] = 1;
      list.insert(list.end(), S.begin(), S.end());
      first.push_back(int(list.size()));
      below.push_back(low);
    }
    for (int f = 0; f < 3; ++f) {
      Phase& p = phase[f];
      p = Phase();
      p.first.push_back(0);
      for (int I = 0; I < nt; ++I) {
        if ((f == 1 && leaf[size_t(I)]) || (f == 2 && !leaf[size_t(I)])) continue;
        p.tiles.push_back(I);
        for (int J = 0; J < nt; ++J) {
          if (!on[size_t(I)][size_t(J)] || bool(leaf[size_t(J)]) != (f == 0)) continue;
          if (int(p.ranges.size()) > 2 * p.first.back() && p.ranges.back() == J * tile) p.ranges.back() += tile;
          else p.ranges.insert(p.ranges.end(), {J * tile, (J + 1) * tile});
        }
        p.first.push_back(int(p.ranges.size() / 2));
      }
    }
  }
};

}  // namespace sgs
