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


@pytest.mark.parametrize("delta", [1, 1000])
def test_sssp_along_a_path(delta):
    """Steps of one CTA alone; a bucket for every vertex, or for fifty."""
    V = 200_000
    w = np.random.default_rng(1).integers(1, 40, V - 1)
    with Store(reverse_edges=False) as st:
        _path(st, V, w)
        with st.snapshot() as sn:
            sn.flatten(0)
            before = st.launch_count
            got, r = sn.sssp(0, delta)
            assert np.array_equal(got, np.concatenate([[0], np.cumsum(w)]))
            assert (r.reached, r.reach_edges, r.max_dist) == (V, V - 1, w.sum())
            assert r.relaxations == V - 1 and r.rounds >= V
            assert st.launch_count - before >= 2         # 0.1 s of dependent loads


def test_sssp_long_runs_of_the_whole_grid():
    """A chain of 30000 groups of 66 vertices: queues too long for one CTA."""
    n, k = 30_000, 66
    V = n * k
    a = np.arange(n - 1)
    first = a * k
    src = np.repeat(first, k)                     # to all of the next group
    dst = np.repeat(first + k, k) + np.tile(np.arange(k), n - 1)
    w = np.full(len(src), 3)
    with Store(reverse_edges=False) as st:
        st.build_level(V, src, dst, w)
        with st.snapshot() as sn:
            sn.flatten(0)
            before = st.launch_count
            got, r = sn.sssp(0, 16)
            want = np.repeat(np.arange(n) * 3, k).astype(np.uint32)
            want[1:k] = 2147483646                # the first group's others
            assert np.array_equal(got, want)
            assert r.reached == (n - 1) * k + 1
            assert st.launch_count - before >= 2
