"""Multi-source BFS and batched BC over vertices whose in-edges are cut into
pieces (2048 edges) in the bottom-up steps: each row equals a one-root BFS."""
import numpy as np
import pytest

from llama_b200 import Store

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("deg", [513, 2047, 2048, 2049, 6200])
def test_hub_rows(deg):
    V, rng = 12000, np.random.default_rng(deg)
    hubs = [0, 31, 32, V - 1]
    s = np.concatenate([rng.integers(0, V, 60000)] + [rng.choice(V, deg, replace=False)
                                                     for _ in hubs])
    d = np.concatenate([rng.integers(0, V, 60000)] + [np.full(deg, h) for h in hubs])
    k = np.unique(s * V + d)
    s, d = k // V, k % V
    roots = rng.choice(V, 70, replace=False)
    with Store() as st:
        st.build_level(V, s, d)
        with st.snapshot() as sn:
            plain = sn.bc(roots[:40], batched=False)
            sn.flatten(1)
            rows, res = sn.bfs_multi(roots)
            for r, row, x in zip(roots, rows, res):
                want, one = sn.bfs(int(r))
                assert np.array_equal(row, want)
                assert (x.reached, x.reach_edges, x.max_level) == (
                    one.reached, one.reach_edges, one.max_level)
            assert np.allclose(sn.bc(roots[:40]), plain, rtol=1e-9, atol=1e-9)
