"""The chunks of columns of an adjoint without saved states (adjoint_cut of
csrc/vert_chunks.h, compiled as plain C++): over random plans every tile of
both tilings is in one chunk, in order, and a chunk's columns are those of its
tiles."""
import ctypes
import os
import subprocess

import numpy as np
import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CUDA = os.environ.get("CUDA_HOME", "/usr/local/cuda")

SOURCE = """
#include "vert_chunks.h"
static std::vector<gv::Tile> cut(int n_members, const long long* n_cols, const int* nc) {
  std::vector<gv::Tile> t;
  for (int m = 0; m < n_members; ++m)
    for (long long c0 = 0; c0 < n_cols[m]; c0 += nc[m])
      t.push_back({m, int(std::min<long long>(nc[m], n_cols[m] - c0)), c0});
  return t;
}
// out: 6 numbers a chunk; tiles: member, nc, c0 of the saving tiles, then of the adjoint tiles
extern "C" int chunks(int n, const long long* n_cols, const int* nc_save, const int* nc_adj, long long columns,
                      long long* out, long long* tiles, int* n_tiles) {
  const auto s = cut(n, n_cols, nc_save), a = cut(n, n_cols, nc_adj);
  const auto c = gv::adjoint_cut(s, a, std::vector<int64_t>(n_cols, n_cols + n), columns);
  int k = 0;
  for (const auto& x : c)
    for (long long v : {(long long)x.save0, (long long)x.save1, (long long)x.adj0, (long long)x.adj1, (long long)x.c0, (long long)x.n}) out[k++] = v;
  k = 0;
  for (const auto* t : {&s, &a})
    for (const auto& x : *t)
      for (long long v : {(long long)x.member, (long long)x.nc, (long long)x.c0}) tiles[k++] = v;
  n_tiles[0] = int(s.size());
  n_tiles[1] = int(a.size());
  return int(c.size());
}
"""


@pytest.fixture(scope="module")
def chunks(tmp_path_factory):
    d = tmp_path_factory.mktemp("chunks")
    src, so = d / "c.cpp", d / "c.so"
    src.write_text(SOURCE)
    subprocess.run(["g++", "-O1", "-std=c++17", "-shared", "-fPIC", f"-I{CUDA}/include",
                    "-I" + os.path.join(ROOT, "gitm_b200", "csrc"), str(src), "-o", str(so)], check=True)
    return ctypes.CDLL(str(so)).chunks


@pytest.mark.parametrize("case", range(40))
def test_adjoint_cut(chunks, case):
    rng = np.random.default_rng(case)
    n = int(rng.integers(1, 5))
    n_cols = np.where(rng.random(n) < 0.2, 0, rng.integers(1, 4000, n)).astype(np.int64)
    nc_save, nc_adj = rng.integers(1, 65, n).astype(np.int32), rng.integers(1, 5, n).astype(np.int32)
    columns = int(rng.choice([1, 7, 100, 640, 2960, 10 ** 6]))
    out, tiles, nt = np.zeros((16384, 6), np.int64), np.zeros((65536, 3), np.int64), np.zeros(2, np.int32)
    p = lambda a: a.ctypes.data_as(ctypes.c_void_p)  # noqa: E731
    k = chunks(n, p(n_cols), p(nc_save), p(nc_adj), ctypes.c_longlong(columns), p(out), p(tiles), p(nt))
    out, save, adj = out[:k], tiles[:nt[0]], tiles[nt[0]:nt.sum()]
    first = np.concatenate([[0], np.cumsum(n_cols)])
    assert out[:, 5].sum() == first[-1]
    at, sa, ad = 0, 0, 0
    for s0, s1, a0, a1, c0, cols in out:
        assert (s0, a0, c0) == (sa, ad, at) and s1 > s0 and a1 > a0  # one after the other, none empty
        for t in (save[s0:s1], adj[a0:a1]):
            m = t[0, 0]
            assert (t[:, 0] == m).all()
            assert first[m] + t[0, 2] == c0 and t[:, 1].sum() == cols  # whole tiles, and only its columns
        both = int(save[s0, 1]) * int(adj[a0, 1])
        assert cols <= max(columns, both)
        sa, ad, at = s1, a1, c0 + cols
    assert (sa, ad, at) == (nt[0], nt[1], first[-1])
