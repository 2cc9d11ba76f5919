"""Device-built levels whose edge counts sit at the edges of the radix sort's
tiles, with weights (a payload) and without, against the host builder."""
import numpy as np
import pytest

from llama_b200 import HostGraph, Store

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("weighted", [False, True])
@pytest.mark.parametrize("n", [1, 2, 31, 33, 511, 513, 4095, 4096, 4097, 12289])
def test_level_of_n_edges(n, weighted):
    rng = np.random.default_rng(n)
    V = 70_000 if n > 500 else 300
    key = rng.choice(V * V, size=n, replace=False)
    # a few targets taken often: digits with long runs inside a tile
    s, d = (key // V).astype(np.uint32), (key % V).astype(np.uint32)
    if n > 4000:
        s[: n // 2] = rng.permutation(V)[: n // 2]
        d[: n // 2] = 17
        keep = np.unique(s.astype(np.int64) * V + d, return_index=True)[1]
        s, d = s[keep], d[keep]
        p = rng.permutation(len(s))
        s, d = s[p], d[p]
    w = rng.integers(1, 1 << 30, len(s)).astype(np.uint32) if weighted else None
    hg = HostGraph(V)
    hg.add_level(s, d, weights=w)
    with Store() as a, Store() as b:
        a.ingest(hg)
        b.build_level(V, s, d, w)
        for dr in (0, 1):
            va, ia = a.read_level(0, dr)
            vb, ib = b.read_level(0, dr)
            assert np.array_equal(va.view(np.uint8), vb.view(np.uint8))
            assert np.array_equal(ia, ib)
        if weighted:
            assert np.array_equal(a.read_level(0, 0, weights=True)[2],
                                  b.read_level(0, 0, weights=True)[2])
