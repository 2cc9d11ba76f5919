"""PageRank push on both sides of the rule that transposes the out-edges: few
iterations over few edges push, more of them pull over the transpose.  Against
a plain FP64 evaluation, 1e-12 relative as for every PageRank here."""
import numpy as np
import pytest

from llama_b200 import Store
from tests._util import max_rel_err

pytestmark = pytest.mark.gpu


def _reference(V, s, d, iterations):
    deg = np.bincount(s, minlength=V).astype(np.float64)
    x = np.full(V, 1.0 / V)
    for _ in range(iterations):
        y = np.divide(x, deg, out=np.zeros(V), where=deg > 0)
        x = 0.15 / V + 0.85 * np.bincount(d, y[s], V)
    return x


@pytest.mark.parametrize("reverse", [False, True])
@pytest.mark.parametrize("V,n,hub", [(1 << 16, 900000, False), (70001, 1300000, True)])
def test_push_both_ways(V, n, hub, reverse):
    rng = np.random.default_rng(V)
    s, d = rng.integers(0, V, n), rng.integers(0, V // 2, n)       # half without in-edges
    if hub:
        s, d = np.concatenate([s, np.arange(V)]), np.concatenate([d, np.full(V, 7)])
    k = np.unique(s * V + d)
    s, d = k // V, k % V
    old = rng.random(len(k)) < 0.8
    gone = old & (rng.random(len(k)) < 0.1)
    live = ~gone
    with Store(reverse_edges=reverse) as st:
        st.build_level(V, s[old], d[old])
        st.build_level(V, s[~old], d[~old], None, s[gone], d[gone])
        with st.snapshot() as sn:
            for flat in (False, True):
                if flat:
                    sn.flatten(0)
                for it in (0, 1, 2, 4, 9):      # 5 M edge-iterations lie between
                    got = sn.pagerank_push(it)
                    assert max_rel_err(got, _reference(V, s[live], d[live], it)) <= 1e-12


def test_graphs_without_hubs_push_for_longer():
    """The rule's two lines.  A push takes a launch to begin and two per
    iteration, the transpose a dozen and some more."""
    rng = np.random.default_rng(5)
    V, n = 100_000, 1_000_000
    k = np.unique(rng.integers(0, V * V, n))
    hub = np.unique(np.concatenate([k, 3 * V + np.arange(0, V, 50), np.arange(0, V, 50) * V + 3]))
    for keys, last in ((k, 14), (hub, 5)):
        s, d = keys // V, keys % V
        for reverse in (False, True):
            with Store(reverse_edges=reverse) as st:
                st.build_level(V, s, d)
                with st.snapshot() as sn:
                    for it in (last, last + 1):
                        before = st.launch_count
                        got = sn.pagerank_push(it)
                        pushed = st.launch_count - before == 1 + 2 * it
                        assert pushed == (it == last)
                        assert max_rel_err(got, _reference(V, s, d, it)) <= 1e-12


def test_fewer_edges_than_vertices():
    """Transposed from the lower line on, hubs or not."""
    rng = np.random.default_rng(6)
    V = 1_500_000
    k = np.unique(rng.integers(0, V * V, 600_000))
    s, d = k // V, k % V
    with Store(reverse_edges=False) as st:
        st.build_level(V, s, d)
        with st.snapshot() as sn:
            for it, push in ((9, True), (10, False)):
                before = st.launch_count
                got = sn.pagerank_push(it)
                assert (st.launch_count - before == 1 + 2 * it) == push
                assert max_rel_err(got, _reference(V, s, d, it)) <= 1e-12
