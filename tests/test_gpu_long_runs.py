"""Traversals of very many steps: no launch takes them all, so that none holds
the GPU for as long as they take.  A launch ends after 50 ms; a step ends at a
barrier of the whole grid, or of one CTA after some dependent loads, which
takes a microsecond or (there) half of one at the least."""
import numpy as np
import pytest

from llama_b200 import Store, _lib
from tests._util import max_rel_err

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


def _graph(V, n):
    rng = np.random.default_rng(V)
    k = np.unique(np.concatenate([rng.integers(0, V * V, n), np.arange(V) * V]))  # a hub
    return k // V, k % V


@pytest.mark.parametrize("V,n", [(50, 200), (3000, 40000)])
def test_pagerank_of_very_many_iterations(V, n):
    """A launch takes some 7000 iterations; damping close to 1, so that every
    one of them counts."""
    s, d = _graph(V, n)
    deg = np.bincount(s, minlength=V).astype(np.float64)
    x = np.full(V, 1.0 / V)
    damping = 0.9999
    with Store() as st:
        st.build_level(V, s, d)
        with st.snapshot() as sn:
            sn.flatten(1)
            done = 0
            for it in (7001, 14500):
                for _ in range(it - done):
                    y = np.divide(x, deg, out=np.zeros(V), where=deg > 0)
                    x = (1 - damping) / V + damping * np.bincount(d, y[s], V)
                done = it
                before = st.launch_count
                got = sn.pagerank_pull(it, damping)
                # an iteration adds V terms at the most, its error shrinks by the
                # damping at the least: V * 2^-53 / (1 - damping) on either side
                assert max_rel_err(got, x) <= 2 * V * 2.0 ** -53 * 1e4
                assert st.launch_count - before >= it // 7143


def test_fixed_point_of_very_many_iterations():
    V, n = 3000, 40000
    s, d = _graph(V, n)
    rng = np.random.default_rng(3)
    deg = np.bincount(s, minlength=V)
    w = rng.uniform(0.5, 1.0, len(s)) / np.maximum(deg[s], 1)
    v = rng.random(V) / V
    damping = 0.9999
    with Store() as st:
        st.build_level(V, s, d)
        with st.snapshot() as sn:
            sn.pagerank_fwd(w, v, damping, max_iter=1, keep_tape=False)
            x, done = v.copy(), 0
            for it in (7001, 14500):
                for _ in range(it - done):
                    x = (1 - damping) * v + damping * np.bincount(d, w * x[s], V)
                done = it
                got, _, r = sn.pagerank_fwd(w, v, damping, tol=1e-300, max_iter=it,
                                            keep_tape=False)
                # (the residual is 0 from where the rounding stands still)
                assert r.iterations == it or r.residual == 0
                assert max_rel_err(got, x) <= 2 * V * 2.0 ** -53 * 1e4
            before = st.launch_count
            nan, _, r = sn.pagerank_fwd(w * np.nan, v, damping, max_iter=20000, keep_tape=False)
            assert r.iterations == 20000 and np.isnan(r.residual)
            assert st.launch_count - before >= 5      # 3 with one launch of the iterations


@pytest.fixture
def one_step():
    f = _lib.lib.lg_test_one_step
    f.argtypes, f.restype = [_lib.C.c_int], None
    yield f
    f(0)


@pytest.mark.parametrize("V,n,hub", [(2000, 9000, False), (60000, 500000, True),
                                     (300000, 3000000, False)])
def test_a_launch_for_every_step(one_step, V, n, hub):
    """State handed from launch to launch at every step there is: top-down and
    bottom-up levels, buckets, light and heavy phases, colouring, iterations."""
    rng = np.random.default_rng(V)
    k = rng.integers(0, V * V, n)
    if hub:
        k = np.concatenate([k, np.arange(V), np.arange(V) * V])
    k = np.unique(k)
    s, d = k // V, k % V
    w = rng.uniform(0.5, 1.0, len(s)) / np.bincount(s, minlength=V)[s]
    v = rng.random(V) / V
    with Store() as st:
        st.build_level(V, s, d, rng.integers(1, 200, len(s)))
        with st.snapshot() as sn:
            sn.flatten(0).flatten(1)

            def results():
                out = [x for root in (0, 7) for x in (sn.bfs(root), sn.sssp(root, 40))]
                out.append(sn.scc())
                x, tape, r = sn.pagerank_fwd(w, v, max_iter=9)
                dw, dv, rb = tape.backward(v)
                tape.close()
                return out, (x, dw, dv, sn.pagerank_pull(9)), (r, rb)

            def fields(r):
                # (what a step finds of the improvements of the same step, and so
                # these, depends on the order of the warps)
                vary = ("reserved", "rounds", "relaxations", "steps")
                return [getattr(r, f) for f, _ in type(r)._fields_ if f not in vary]
            one_step(0)
            before = st.launch_count
            out, real, fix = results()
            few = st.launch_count - before
            one_step(1)
            before = st.launch_count
            out1, real1, fix1 = results()
            assert st.launch_count - before > few + 40
            one_step(0)
            for (a, r), (b, r1) in zip(out, out1):
                assert np.array_equal(a, b) and fields(r) == fields(r1)
            for a, b in zip(real, real1):
                assert np.array_equal(a, b)
            for r, r1 in zip(fix, fix1):
                assert fields(r) == fields(r1)
