"""Flattening a slot space close to 2^32 slots.  The slots are 4096 fragments
over the same 2^20 deleted ones, so the level's arrays stay small; the live
rows are the last ones, where 32-bit sums of slots would wrap."""
import numpy as np
import pytest

from llama_b200 import Store, _lib
from llama_b200._lib import VT_DTYPE

pytestmark = pytest.mark.gpu

DEAD = 1 << 20
FRESH = np.uint64(((1 << 26) - 1) << 38)


def _desc(V, rows, dead):
    """One level: vertex v has dead[v] slots of the deleted range, or the live
    row rows[v] (sorted ids); the in-CSR holds the live edges alone."""
    d = _lib.lg_level_desc()
    keep = []

    def csr(c, vt, slots, w=None):
        c.max_nodes, c.n_slots = V, len(slots)
        c.vt, c.slots = vt.ctypes.data, slots.ctypes.data
        c.weights = w.ctypes.data if w is not None else None
        keep.extend((vt, slots, w))
    vt = np.zeros(V + 1, VT_DTYPE)
    vt["adj_list_start"] = -1
    live = [np.zeros(0, np.uint64)]
    at = DEAD
    for v in range(V):
        n = len(rows[v])
        if dead[v]:
            vt[v] = (0, dead[v], 0)
        elif n:
            vt[v] = (at, n, n)
            live.append(np.asarray(rows[v], np.uint64))
            at += n
    live = np.concatenate(live)
    # deleted slots: visible in no snapshot
    csr(d.out, vt, np.concatenate([np.zeros(DEAD, np.uint64), live | FRESH]),
        np.ones(DEAD + len(live), np.uint32))
    src = np.concatenate([np.full(len(r), v, np.int64) for v, r in enumerate(rows)])
    dst = live.astype(np.int64)
    o = np.lexsort((src, dst))
    cnt = np.bincount(dst, minlength=V)
    ivt = np.zeros(V + 1, VT_DTYPE)
    ivt["adj_list_start"] = -1
    start = np.concatenate([[0], np.cumsum(cnt)])
    has = np.flatnonzero(cnt)
    ivt["adj_list_start"][has] = start[has]
    ivt["level_length"][has] = ivt["degree"][has] = cnt[has]
    csr(d.in_, ivt, src[o].astype(np.uint64) | FRESH)
    return d, keep, src, dst


@pytest.mark.parametrize("short_of", [0, 31, 200])
def test_slots_up_to_the_limit(short_of):
    rng = np.random.default_rng(short_of)
    V, tail = 4500, 2000
    dead = np.zeros(V, np.int64)
    dead[:4095] = DEAD
    dead[4095] = DEAD - tail
    rows = [[] for _ in range(V)]
    left, v = tail - 1 - short_of, 4096
    while left:                                  # rows of 1 to 40, gaps between them
        n = min(left, int(rng.integers(1, 41)))
        rows[v] = np.sort(rng.choice(np.arange(4096, V), n, replace=False))
        left -= n
        v += 1 + int(rng.random() < 0.2)
    d, keep, src, dst = _desc(V, rows, dead)
    assert dead.sum() + len(src) == 2 ** 32 - 1 - short_of
    with Store() as st:
        st.ingest_level(d)
        with st.snapshot() as sn:
            assert sn.num_edges == len(src)
            want = sn.bfs(4096)[0]
            sn.flatten(0).flatten(1)
            assert np.array_equal(sn.bfs(4096)[0], want)
            # the maps between the directions read every slot's edge position
            w = rng.uniform(0.01, 0.04, len(src))
            t = rng.uniform(0.5, 1.0, V)
            x, _, r = sn.pagerank_fwd(w, t, 0.85, keep_tape=False)
            y = t.copy()
            for _ in range(r.iterations):
                y = 0.15 * t + 0.85 * np.bincount(dst, w * y[src], V)
            # sums of at most 500 positive terms, contracting by 0.85 at most
            assert np.max(np.abs(x - y) / y) <= 1e-12


@pytest.mark.parametrize("hub", [33 * 512 - 1, 33 * 512, 33 * 512 + 1, 70_001])
def test_rows_over_many_tiles(hub):
    """Rows and fragments whose marks among the tiles they cover are shared by a
    warp: several in one warp, in one level and split over three, both ways."""
    V = hub + 40
    rng = np.random.default_rng(hub)
    src, dst = [], []
    for v, n in ((0, hub), (3, hub), (4, 5), (17, hub), (V - 1, hub), (40, 17_000 % V)):
        src.append(np.full(n, v))
        dst.append(rng.permutation(V)[:n])
    s, d = np.concatenate(src), np.concatenate(dst)
    k = np.unique(np.concatenate([s * V + d, d * V + s]))
    s, d = k // V, k % V
    lev = rng.integers(0, 3, len(s))
    lev[(s == 3) | (d == 3)] = 0
    deg = np.bincount(s, minlength=V).astype(np.float64)
    x = np.full(V, 1.0 / V)
    for _ in range(3):
        x = 0.15 / V + 0.85 * np.bincount(d, (x / np.maximum(deg, 1))[s], V)
    tol = 3 * 2 * V * 2.0 ** -53                  # three sums of at most V terms
    with Store() as st:
        for l in range(3):
            st.build_level(V, s[lev == l], d[lev == l])
        with st.snapshot() as sn:
            off, nbr = sn.adjacency(0)
            own = np.repeat(np.arange(V), np.diff(off.astype(np.int64)))
            bfs, labels = sn.bfs(0)[0], sn.scc()[0]
            w, v = rng.uniform(0.5, 1.0, len(s)), rng.uniform(0.5, 1.0, V)
            # one iteration: every edge's weight by its place among the out-edges
            y = 0.15 * v + 0.85 * np.bincount(nbr, w * v[own], V)
            for flat in (False, True):
                if flat:
                    sn.flatten(0).flatten(1)
                assert np.max(np.abs(sn.pagerank_pull(3) - x) / x) <= tol
                assert np.array_equal(sn.bfs(0)[0], bfs)
                assert np.array_equal(sn.scc()[0], labels)
                got = sn.pagerank_fwd(w, v, 0.85, tol=1e-300, max_iter=1, keep_tape=False)[0]
                assert np.max(np.abs(got - y) / y) <= tol
