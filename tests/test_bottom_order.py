"""The elimination order of the dense bottom (csrc/bottom_order.hpp), on the CPU:
the header is compiled with a small C interface, the blocked Gauss-Jordan steps
and the phases of the application are carried out with numpy exactly as they are
listed (no tile outside a list is touched), and the result has to solve the
system.  FP64 round-off: rows of up to 81 entries dominated by their diagonal
(condition below 21), the residual to 1e-12 of the right-hand side.
"""
import ctypes
import subprocess

import numpy as np
import pytest

from spgrid_topo_opt_b200 import build

TILE = 128

HARNESS = r"""
#include "bottom_order.hpp"
using sgs::BottomOrder;
extern "C" {
void* order_new(const int* xyz, int n) {
  auto* o = new BottomOrder;
  for (int i = 0; i < n; ++i) o->at.push_back({xyz[3 * i], xyz[3 * i + 1], xyz[3 * i + 2]});
  o->build(%d);
  return o;
}
void order_delete(void* p) { delete static_cast<BottomOrder*>(p); }
int order_single(void* p) { return static_cast<BottomOrder*>(p)->single; }
// which: 0 pos, 1 pad, 2 list, 3 first, 4 below, 5 + 3 f: phase f's tiles, first, ranges
int order_vector(void* p, int which, int* out) {
  auto& o = *static_cast<BottomOrder*>(p);
  const std::vector<int>* v[14] = {&o.pos, &o.pad, &o.list, &o.first, &o.below};
  for (int f = 0; f < 3; ++f) v[5 + 3 * f] = &o.phase[f].tiles, v[6 + 3 * f] = &o.phase[f].first, v[7 + 3 * f] = &o.phase[f].ranges;
  if (out) std::copy(v[which]->begin(), v[which]->end(), out);
  return int(v[which]->size());
}
}
""" % TILE


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    d = tmp_path_factory.mktemp("order")
    (d / "order.cpp").write_text(HARNESS)
    so = str(d / "order.so")
    subprocess.run([build.host_compiler(), "-std=c++17", "-O2", "-shared", "-fPIC", "-I", build.CSRC,
                    str(d / "order.cpp"), "-o", so], check=True)
    l = ctypes.CDLL(so)
    l.order_new.restype = ctypes.c_void_p
    for f in (l.order_delete, l.order_single, l.order_vector):
        f.argtypes = [ctypes.c_void_p] + ([ctypes.c_int, ctypes.c_void_p] if f is l.order_vector else [])
    return l


class Order:
    def __init__(self, lib, xyz):
        xyz = np.ascontiguousarray(xyz, np.int32)
        o = lib.order_new(xyz.ctypes.data_as(ctypes.c_void_p), len(xyz))
        v = []
        for w in range(14):
            a = np.zeros(lib.order_vector(o, w, None), np.int32)
            lib.order_vector(o, w, a.ctypes.data_as(ctypes.c_void_p))
            v.append(a)
        self.pos, self.pad, self.list, self.first, self.below = v[:5]
        self.phase = [v[5 + 3 * f:8 + 3 * f] for f in range(3)]
        self.single = bool(lib.order_single(o))
        lib.order_delete(o)
        self.ld = 3 * len(xyz) + len(self.pad)
        assert self.ld % TILE == 0


def _box(nx, ny, nz, at=(0, 0, 0)):
    g = np.stack(np.meshgrid(np.arange(nx), np.arange(ny), np.arange(nz), indexing="ij"), -1).reshape(-1, 3)
    return g + np.asarray(at)


def _nodes(name):
    if name == "one part":
        return _box(5, 7, 9)
    if name == "box":              # two halves and a plane
        return _box(10, 11, 15)
    if name == "four parts":
        return _box(4, 20, 37)
    if name == "plate and rod":    # most nodes lie in the plane at one end: one part and a separator
        return np.concatenate([_box(37, 37, 1), _box(4, 4, 44, (17, 17, 1))])
    if name == "rod and plate":
        return np.concatenate([_box(3, 3, 44, (17, 17, 0)), _box(37, 37, 1, (0, 0, 44))])
    if name == "apart":            # nodes that no path connects
        return np.concatenate([_box(8, 9, 10), _box(8, 9, 10, (60, 60, 60))])
    if name == "far apart":        # the same further off: looked up in a map
        return np.concatenate([_box(8, 9, 10), _box(8, 9, 10, (300, 300, 300))])
    rng = np.random.default_rng(11)  # "scattered": a ragged set with holes
    g = _box(13, 14, 15)
    return g[rng.random(len(g)) < 0.55]


def _matrix(o, xyz, rng):
    """Random symmetric matrix, diagonally dominant, coupling a node with its 26 neighbours."""
    M = np.zeros((o.ld, o.ld))
    key = {tuple(p): i for i, p in enumerate(xyz.tolist())}
    off = [(a, b, c) for a in (-1, 0, 1) for b in (-1, 0, 1) for c in (-1, 0, 1)]
    for i, p in enumerate(xyz.tolist()):
        for q in off:
            j = key.get((p[0] + q[0], p[1] + q[1], p[2] + q[2]))
            if j is None or j < i:
                continue
            B = rng.uniform(-1, 1, (3, 3))
            if i == j:
                B += B.T
            r, c = o.pos[i], o.pos[j]
            M[r:r + 3, c:c + 3] = B
            M[c:c + 3, r:r + 3] = B.T
    M[np.arange(o.ld), np.arange(o.ld)] = np.abs(M).sum(1) * 1.1 + 1
    return M


def _eliminate(o, M):
    rows = lambda tiles: (np.asarray(tiles, int)[:, None] * TILE + np.arange(TILE)).ravel()
    for K in range(o.ld // TILE):
        S = o.list[o.first[K]:o.first[K + 1]]
        assert o.below[K] == np.count_nonzero(S < K)
        k, s = rows([K]), rows(S)
        P = np.linalg.inv(M[np.ix_(k, k)])
        T, C = P @ M[np.ix_(k, s)], M[np.ix_(s, k)]
        M[np.ix_(s, s)] -= C @ T
        M[np.ix_(k, s)], M[np.ix_(s, k)] = T, -C @ P
        M[np.ix_(k, k)] = P
    return np.tril(M) + np.tril(M, -1).T  # the lower half is kept and mirrored


def _apply(o, M, b):
    def phase(f, v):
        tiles, first, ranges = o.phase[f]
        out = np.zeros(o.ld)
        for i, t in enumerate(tiles):
            r = slice(t * TILE, (t + 1) * TILE)
            for c0, c1 in ranges[2 * first[i]:2 * first[i + 1]].reshape(-1, 2):
                out[r] += M[r, c0:c1] @ v[c0:c1]
        return out
    if o.single:
        return phase(0, b)
    sep = np.zeros(o.ld, bool)
    for t in o.phase[1][0]:
        sep[t * TILE:(t + 1) * TILE] = True
    y = phase(0, b) + np.where(sep, b, 0)
    xs = phase(1, y)
    return np.where(sep, xs, y + phase(2, xs))


@pytest.mark.parametrize("name,single", [("one part", True), ("box", False), ("four parts", False),
                                         ("plate and rod", False), ("rod and plate", False), ("apart", False),
                                         ("far apart", False), ("scattered", False)])
def test_order_solves_the_system(lib, name, single):
    xyz = _nodes(name)
    o = Order(lib, xyz)
    rng = np.random.default_rng(3)
    M = _matrix(o, xyz, rng)
    b = rng.standard_normal(o.ld)
    b[o.pad] = 0
    x = _apply(o, _eliminate(o, M.copy()), b)
    x[o.pad] = 0
    assert np.abs(M @ x - b).max() <= 1e-12 * np.abs(b).max()
    assert o.single == single


def test_map_gives_the_tiles_of_the_grid(lib):
    a, b = Order(lib, _nodes("apart")), Order(lib, _nodes("far apart"))
    assert np.array_equal(a.list, b.list) and np.array_equal(a.pos, b.pos)
