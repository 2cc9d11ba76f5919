"""Personalised PageRank where its edge ranges, rows over many ranges, rows
without in-edges and repeated seeds meet, against a plain FP64 evaluation.
Bar: 1e-12 relative, as for every PageRank here."""
import numpy as np
import pytest

from llama_b200 import Store
from llama_b200.graph import ppr, tune_reset, tune_set
from tests._util import max_rel_err

pytestmark = pytest.mark.gpu


def _reference(V, s, d, seeds, iterations, damping):
    deg = np.bincount(s, minlength=V).astype(np.float64)[:, None]
    x = np.zeros((V, len(seeds)))
    x[seeds, np.arange(len(seeds))] = 1.0
    for _ in range(iterations):
        y = np.divide(x, deg, out=np.zeros_like(x), where=deg > 0)
        acc = np.zeros_like(x)
        np.add.at(acc, d, y[s])
        x = damping * acc
        x[seeds, np.arange(len(seeds))] += 1.0 - damping
    return x


def _edges(shape, V, n, seed):
    rng = np.random.default_rng(seed)
    key = rng.choice(V * V, size=n, replace=False)
    s, d = key // V, key % V
    if shape == "hub":                   # one target over many ranges, one source of many
        s = np.concatenate([s, np.arange(1, V), np.full(V - 2, V - 1)])
        d = np.concatenate([d, np.zeros(V - 1, np.int64), np.arange(1, V - 1)])
    elif shape == "lower":               # half of the vertices have no in-edges
        d = d // 2
    k = np.unique(s * V + d)
    return k // V, k % V


@pytest.mark.parametrize("K", [32, 64, 96, 160, 256])
@pytest.mark.parametrize("shape,V,n", [
    ("any", 40, 31), ("any", 40, 32), ("any", 40, 33), ("lower", 500, 4000), ("hub", 6001, 9000)])
def test_ppr(shape, V, n, K):
    s, d = _edges(shape, V, n, n + K)
    rng = np.random.default_rng(5)
    seeds = rng.integers(0, V, K)
    seeds[1] = seeds[0]
    seeds[2] = V - 1                     # without in-edges in "lower"
    with Store() as st:
        a = rng.random(len(s)) < 0.7
        st.build_level(V, s[a], d[a])
        st.build_level(V, s[~a], d[~a])
        with st.snapshot(0) as s0, st.snapshot(1) as s1:
            for it in (1, 2, 5):
                want = [_reference(V, s[m], d[m], seeds, it, 0.85) for m in (a, a | ~a)]
                got = ppr([s0, s1], seeds, iterations=it)
                assert max_rel_err(got[0], want[0]) <= 1e-12
                assert max_rel_err(got[1], want[1]) <= 1e-12
            s1.flatten(1)
            assert np.array_equal(ppr([s1], seeds, iterations=5)[0], got[1])
            tune_set(0, "ppr_ktile", 32)
            try:
                assert np.array_equal(ppr([s1], seeds, iterations=5)[0], got[1])
            finally:
                tune_reset(0)


def test_ppr_without_edges():
    seeds = np.arange(32) % 7
    with Store() as st:
        st.build_level(7, np.zeros(0, np.uint32), np.zeros(0, np.uint32))
        with st.snapshot() as sn:
            x = ppr([sn], seeds, iterations=3)[0]
            assert np.allclose(x, _reference(7, np.zeros(0, int), np.zeros(0, int), seeds, 3, 0.85),
                               rtol=1e-12, atol=0)
