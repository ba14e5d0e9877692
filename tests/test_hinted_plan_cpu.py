"""Plans with heavy-child hints (linked reservoirs): the walkers' lanes advance together, so a chain
must not share a chunk, whose chains may share a warp, with a longer chain that joins it earlier than
that chain ends. Such joins exist only with hints, where the heavy child need not be the highest one."""

import ctypes as C

import numpy as np
import pytest

from wflow_gb300 import abi, build


@pytest.fixture(scope="module")
def lib():
    build.build_all()
    return abi.load_library()


def _plan(lib, ds, hint, members):
    ds, hint = np.ascontiguousarray(ds, np.int32), np.ascontiguousarray(hint, np.int64)
    n = len(ds)
    counts, chain, ok, g = np.zeros(4, np.int64), np.zeros(n, np.int64), C.c_int32(), C.c_int32()
    st = lib.wf_plan_routing_hinted(n, ds.ctypes.data_as(C.POINTER(C.c_int32)), members,
                                    hint.ctypes.data_as(C.POINTER(C.c_int64)),
                                    counts.ctypes.data_as(C.POINTER(C.c_int64)),
                                    chain.ctypes.data_as(C.POINTER(C.c_int64)), C.byref(ok), C.byref(g))
    assert st == 0 and ok.value == 1, (st, ok.value)
    return chain, counts, g.value


def _chunks(chain, counts, G):
    """Chunk of each node: chunks of G chains first, then chunks of one."""
    solo = (G * counts[1] - counts[0]) // (G - 1)  # n_chains = G (n_chunks - solo) + solo
    packed = counts[0] - solo
    return np.where(chain < packed, chain // G, packed // G + chain - packed)


def _late_joins(ds, chain, counts, G):
    """Joins of a light child into a chain of its own chunk at a position not above its length."""
    n = len(ds)
    length = np.bincount(chain)
    chunk = _chunks(chain, counts, G)
    indeg = np.zeros(n, int)
    np.add.at(indeg, ds[ds >= 0], 1)
    pos = np.zeros(n, int)
    for v in np.nonzero(indeg == 0)[0]:
        k, u = 0, int(v)
        while True:
            pos[u] = k
            d = int(ds[u])
            if d < 0 or chain[d] != chain[u]:
                break
            u, k = d, k + 1
    return [(u, int(ds[u])) for u in range(n)
            if ds[u] >= 0 and chain[ds[u]] != chain[u] and chunk[ds[u]] == chunk[u]
            and length[chain[u]] > pos[ds[u]]]


def _path(ds, n):
    """Appends a river of n cells, from its head to its mouth; returns its first cell."""
    start = len(ds)
    ds += [start + i + 1 for i in range(n - 1)] + [-1]
    return start


@pytest.mark.parametrize("members", [1, 2, 8])
@pytest.mark.parametrize("rivers,short,branch,link", [(300, 0, 10, 2), (300, 6000, 10, 2), (400, 500, 40, 5)])
def test_joins_of_hinted_chains_leave_the_warp(lib, members, rivers, short, branch, link):
    # many rivers of equal length, which fill the group of chains with chunks of their own, and one
    # more: a branch that joins near the head of the hinted (linked) path
    ds = []
    for _ in range(rivers):
        _path(ds, 100)
    for _ in range(short):
        _path(ds, 3)
    low = _path(ds, link + 6)            # the linked path: low + 0 .. low + link, hinted
    b = _path(ds, branch)
    ds[b + branch - 1] = low + 1
    ds = np.array(ds, np.int32)
    hint = np.full(len(ds), -1, np.int64)
    hint[low + 1 : low + link + 1] = np.arange(low, low + link)
    chain, counts, G = _plan(lib, ds, hint, members)
    assert len(set(chain[low : low + link + 1].tolist())) == 1
    assert _late_joins(ds, chain, counts, G) == []


@pytest.mark.parametrize("members", [1, 4, 16])
def test_random_forests_with_hints(lib, members):
    rng = np.random.default_rng(11)
    for trial in range(12):
        n = int(rng.integers(2000, 6000))
        ds = np.full(n, -1, np.int32)
        for i in range(3, n):  # long and short branches
            ds[i] = i - 1 if rng.random() < 0.6 else rng.integers(0, i)
        hint = np.full(n, -1, np.int64)
        for u in rng.integers(0, n, 60):  # linked paths that share no cell
            path = [int(u)]
            while ds[path[-1]] >= 0 and len(path) < 8:
                path.append(int(ds[path[-1]]))
            if all(hint[v] < 0 for v in path) and not np.isin(hint, path).any():
                hint[path[1:]] = path[:-1]
        chain, counts, G = _plan(lib, ds, hint, members)
        assert _late_joins(ds, chain, counts, G) == [], trial
