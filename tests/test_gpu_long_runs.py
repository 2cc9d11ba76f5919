"""Traversals of very many steps: no launch takes them all, so that none holds
the GPU for as long as they take.  A launch ends after 50 ms; a step ends at a
barrier of the whole grid, or of one CTA after some dependent loads, which
takes a microsecond or (there) half of one at the least."""
import numpy as np
import pytest

from llama_b200 import Store

pytestmark = pytest.mark.gpu


def _path(st, V, weights=None):
    a = np.arange(V - 1)
    st.build_level(V, a, a + 1, weights)


def test_bfs_along_a_path():
    V = 200_000                                   # 0.2 s of barriers
    with Store() as st:
        _path(st, V)
        with st.snapshot() as sn:
            sn.flatten(0).flatten(1)
            before = st.launch_count
            lv, r = sn.bfs(0)
            assert np.array_equal(lv, np.arange(V))
            assert (r.reached, r.max_level) == (V, V - 1)
            assert r.top_down_steps + r.bottom_up_steps == V
            assert st.launch_count - before >= 4
