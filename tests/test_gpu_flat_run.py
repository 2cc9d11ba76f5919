"""Iterations inside one launch (PageRank over small in-CSRs, the weighted fixed
point) at the edges of tiles, warp runs and CTAs, with rows over many of them,
against a plain FP64 evaluation."""
import numpy as np
import pytest

from llama_b200 import Store
from tests._util import max_rel_err

pytestmark = pytest.mark.gpu


def _edges(V, n, hub, seed):
    rng = np.random.default_rng(seed)
    k = rng.choice(V * V, n, replace=False) if n else np.zeros(0, np.int64)
    s, d = k // V, k % V
    if hub:                                      # rows of thousands, first, last and between
        for h, m in ((0, V), (V // 2, V // 3), (V - 1, V)):
            s, d = np.concatenate([s, np.arange(m)]), np.concatenate([d, np.full(m, h)])
    k = np.unique(s * V + d)
    return k // V, k % V


CASES = [(3, 0, False), (3, 1, False), (40, 255, False), (40, 256, False), (40, 257, False),
         (600, 8191, False), (600, 8193, False), (9000, 5000, True), (70000, 300000, True),
         (150000, 2500000, False)]


@pytest.mark.parametrize("V,n,hub", CASES)
def test_pagerank(V, n, hub):
    s, d = _edges(V, n, hub, n + V)
    deg = np.bincount(s, minlength=V).astype(np.float64)
    with Store() as st:
        st.build_level(V, s, d)
        with st.snapshot() as sn:
            for it in (1, 2, 3, 8):
                x = np.full(V, 1.0 / V)
                for _ in range(it):
                    y = np.divide(x, deg, out=np.zeros(V), where=deg > 0)
                    x = 0.15 / V + 0.85 * np.bincount(d, y[s], V)
                got = sn.pagerank_pull(it)
                assert max_rel_err(got, x) <= 1e-12
                assert np.array_equal(sn.pagerank_pull(it), got)


def test_pagerank_device_output_and_sync():
    import torch
    s, d = _edges(600, 8193, False, 1)
    with Store() as st:
        st.build_level(600, s, d)
        with st.snapshot() as sn:
            want = sn.pagerank_pull(7)
            out = torch.empty(600, dtype=torch.float64, device="cuda")
            for _ in range(3):
                sn.pagerank_pull(7, out=out)
                sn.pagerank_pull(7, out=out)
                st.sync()
                assert np.array_equal(out.cpu().numpy(), want)


@pytest.mark.parametrize("V,n,hub", CASES)
def test_fixed_point_and_gradient(V, n, hub):
    s, d = _edges(V, n, hub, n + V + 1)
    rng = np.random.default_rng(2)
    deg = np.bincount(s, minlength=V)
    w = rng.uniform(0.5, 1.0, len(s)) / np.maximum(deg[s], 1)      # edges in (s, d) order
    v, g = rng.random(V) / V, rng.standard_normal(V) / V
    with Store() as st:
        st.build_level(V, s, d)
        with st.snapshot() as sn:
            x, tape, r = sn.pagerank_fwd(w, v, tol=1e-13)
            dw, dv, rb = tape.backward(g)
            tape.close()
            # the fixed points' own equations, and the gradients' definition
            assert np.abs(0.15 * v + 0.85 * np.bincount(d, w * x[s], V) - x).sum() <= 1e-13
            lam = dv / 0.15
            assert np.abs(g + 0.85 * np.bincount(s, w * lam[d], V) - lam).sum() <= 2e-13
            assert np.allclose(dw, 0.85 * lam[d] * x[s], rtol=1e-12, atol=0)
            x3, _, r3 = sn.pagerank_fwd(w, v, tol=1e-300, max_iter=3, keep_tape=False)
            # (without a path of three edges the residual is 0 before)
            assert r3.iterations == 3 if n > 1 else r3.iterations <= 3


def test_fixed_point_repeats_bit_for_bit():
    """The residual, which ends the iterations, is added up in one order too."""
    V, n = 150000, 2500000
    s, d = _edges(V, n, False, 5)
    rng = np.random.default_rng(2)
    deg = np.bincount(s, minlength=V)
    w = rng.uniform(0.5, 1.0, len(s)) / np.maximum(deg[s], 1)
    v = rng.random(V) / V
    with Store() as st:
        st.build_level(V, s, d)
        with st.snapshot() as sn:
            x, _, r = sn.pagerank_fwd(w, v, tol=1e-300, max_iter=5, keep_tape=False)
            for _ in range(15):
                x2, _, r2 = sn.pagerank_fwd(w, v, tol=1e-300, max_iter=5, keep_tape=False)
                assert (r2.iterations, r2.residual) == (r.iterations, r.residual)
                assert np.array_equal(x2, x)


@pytest.mark.parametrize("longest", [1, 2, 3, 9])
def test_short_rows(longest):
    """From 25 to 256 rows begin in a tile: the counts at which a lane finishes
    one more, or four more."""
    rng = np.random.default_rng(longest)
    V = 30000
    n = rng.integers(1, longest + 1, V)
    n[::97] = 0
    d = np.repeat(np.arange(V), n)
    s = (d * 7919 + np.concatenate([np.arange(k) for k in n]) * 104729) % V
    k = np.unique(s * V + d)
    s, d = k // V, k % V
    deg = np.bincount(s, minlength=V).astype(np.float64)
    w = rng.uniform(0.5, 1.0, len(s)) / deg[s]
    v = rng.random(V) / V
    with Store() as st:
        st.build_level(V, s, d)
        with st.snapshot() as sn:
            x, y = np.full(V, 1.0 / V), v.copy()
            for it in (1, 2, 3):
                x = 0.15 / V + 0.85 * np.bincount(d, (x / np.maximum(deg, 1))[s], V)
                y = 0.15 * v + 0.85 * np.bincount(d, w * y[s], V)
                assert max_rel_err(sn.pagerank_pull(it), x) <= 1e-14
                got, _, r = sn.pagerank_fwd(w, v, tol=1e-300, max_iter=it, keep_tape=False)
                assert max_rel_err(got, y) <= 1e-14
