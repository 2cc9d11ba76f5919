"""Device allocations that fail, one after the other: a call returns LG_ENOMEM or,
where it has a form that needs less, the right result; and runs again after."""
import numpy as np
import pytest

from llama_b200 import LgError, Store, _lib
from llama_b200.graph import ppr, tune_reset, tune_set
from tests._util import max_rel_err

pytestmark = pytest.mark.gpu

C = _lib.C


@pytest.fixture
def fail_at():
    f = _lib.lib.lg_test_limits
    f.argtypes, f.restype = [C.c_int64, C.c_int64], C.c_int64
    yield lambda k: f(k, -1)
    f(-1, -1)


def _graph(V, n, seed):
    rng = np.random.default_rng(seed)
    k = np.unique(rng.integers(0, V * V, n))
    return k // V, k % V


def _each_failure(fail_at, build, call):
    """call(snapshot) on a new store with its first, second ... allocation
    failing, until none does; yields (result or None for LG_ENOMEM)."""
    for k in range(100):
        with build() as st, st.snapshot() as sn:
            fail_at(k)
            try:
                got = call(sn)
            except LgError as e:
                assert e.status == _lib.LG_ENOMEM, e
                got = None
            left = fail_at(-1)
            again = call(sn)
            if got is None:
                got = (None, again)
            else:
                got = (got, again)
            yield got
            if left >= 0:
                return
    raise AssertionError("allocations without end")


def test_push_runs_without_the_transpose(fail_at):
    V = 20000
    s, d = _graph(V, 800_000, 1)
    k = np.unique(np.concatenate([s * V + d, np.arange(V)]))     # vertex 0 to all: a hub
    s, d = k // V, k % V

    def build():
        st = Store(reverse_edges=False)
        st.build_level(V, s, d)
        return st
    results = list(_each_failure(fail_at, build, lambda sn: sn.pagerank_push(10)))
    assert len(results) > 15
    want = results[-1][0]
    for got, again in results:
        assert got is not None and max_rel_err(got, want) <= 1e-12
        assert max_rel_err(again, want) <= 1e-12


@pytest.mark.parametrize("K,ktile", [(32, 256), (64, 32), (96, 256), (160, 256), (256, 256)])
def test_ppr_runs_over_the_levels(fail_at, K, ktile):
    """Without the flat in-CSR; seeds with and without in-edges, some twice."""
    V = 4000
    s, d = _graph(V, 60_000, K)
    s, d = np.concatenate([s, np.arange(V)]), np.concatenate([d, np.full(V, 7)])  # a hub
    m = d % 9 != 4                                # vertices without in-edges
    k = np.unique(s[m] * V + d[m])
    s, d = k // V, k % V
    rng = np.random.default_rng(K)
    seeds = rng.integers(0, V, K)
    seeds[:8] = [4, 4, 13, 7, 7, 22, 31, 4]
    late = rng.random(len(k)) < 0.3
    dead = ~late & (rng.random(len(k)) < 0.1)

    def build():
        st = Store()
        st.build_level(V, s[~late], d[~late])
        st.build_level(V, s[late], d[late], None, s[dead], d[dead])
        return st
    tune_set(0, "ppr_ktile", ktile)
    try:
        results = list(_each_failure(fail_at, build, lambda sn: ppr([sn], seeds, iterations=6)))
    finally:
        tune_reset(0)
    want = results[-1][0]
    # the call's own allocations are eight at the most; the others, and there are
    # some, are the flat in-CSR's
    none = sum(got is None for got, _ in results)
    assert none <= 8 and len(results) - none >= 4
    for got, again in results:
        # rows of at most 4000 positive terms, six iterations
        assert got is None or max_rel_err(got, want) <= 6 * 2 * 4000 * 2.0 ** -53
        assert np.array_equal(again, want)


def test_triangles_sort_without_the_flat_copy(fail_at):
    V = 3000
    s, d = _graph(V, 90_000, 7)

    def build():
        st = Store(reverse_edges=False)
        st.build_level(V, s, d)
        return st
    results = list(_each_failure(fail_at, build, lambda sn: sn.triangle_count().triangles))
    want = results[-1][0]
    right = [got is not None for got, _ in results]
    assert all(got in (None, want) and again == want for got, again in results)
    # two of the sort's at the least: its second array of keys and its counts
    assert sum(right[:-1]) >= 2 and want > 0
