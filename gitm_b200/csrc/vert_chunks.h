// vert_chunks.h -- how the columns of a plan are cut for an adjoint without
// saved states: the saving step and the adjoint kernel in turn over chunks of
// columns, each chunk whole tiles of both.  Host code.
#pragma once

#include <algorithm>
#include <cstddef>
#include <cstdint>
#include <vector>

#include "vert_common.cuh"

namespace gv {

struct AdjChunk {
  int save0, save1;  // its saving tiles
  int adj0, adj1;    // its adjoint tiles
  int64_t c0, n;     // its columns of the plan
};

// save, adj: the two tilings, member by member in column order, each of tiles
// of one size but for a member's last; n_cols: columns of every member.  A
// chunk has at most `columns` columns, or one boundary of both tilings where
// that is more; it does not cross members.
inline std::vector<AdjChunk> adjoint_cut(const std::vector<Tile>& save, const std::vector<Tile>& adj,
                                         const std::vector<int64_t>& n_cols, int64_t columns) {
  std::vector<AdjChunk> out;
  size_t s = 0, a = 0;
  int64_t off = 0;
  for (size_t m = 0; m < n_cols.size(); off += n_cols[m], ++m) {
    if (n_cols[m] <= 0) continue;
    const int64_t both = int64_t(save[s].nc) * adj[a].nc;
    const int64_t step = std::max<int64_t>(1, columns / both) * both;
    for (int64_t c0 = 0; c0 < n_cols[m]; c0 += step) {
      const int64_t c1 = std::min(n_cols[m], c0 + step);
      AdjChunk ch{int(s), 0, int(a), 0, off + c0, c1 - c0};
      while (s < save.size() && save[s].member == int(m) && save[s].c0 < c1) ++s;
      while (a < adj.size() && adj[a].member == int(m) && adj[a].c0 < c1) ++a;
      ch.save1 = int(s);
      ch.adj1 = int(a);
      out.push_back(ch);
    }
  }
  return out;
}

inline int64_t adjoint_cut_largest(const std::vector<AdjChunk>& chunks) {
  int64_t most = 0;
  for (const AdjChunk& c : chunks) most = std::max(most, c.n);
  return most;
}

}  // namespace gv
