"""Cooperative launches where fewer CTAs fit than the device's properties say (a
share of the GPU): they take a smaller grid, down to one CTA; without any, the
forms with a launch per step."""
import numpy as np
import pytest

from llama_b200 import LgError, Store, _lib
from llama_b200.graph import tune_reset, tune_set
from tests._util import max_rel_err

pytestmark = pytest.mark.gpu


@pytest.fixture
def limit():
    f = _lib.lib.lg_test_limits
    f.argtypes, f.restype = [_lib.C.c_int64, _lib.C.c_int64], _lib.C.c_int64
    yield lambda ctas: f(-1, ctas)
    f(-1, -1)
    tune_reset(0)


def _results(st, sn, w, v):
    out = [sn.bfs(1)[0], sn.scc()[0], sn.pagerank_pull(9)]
    for levels in (0, 1):
        tune_set(0, "sssp_levels", levels)
        out.append(sn.sssp(1, 16)[0])
    tune_reset(0)
    x, tape, _ = sn.pagerank_fwd(w, v, tol=1e-13)
    out += [x, tape.backward(v)[0]]
    tape.close()
    return out


def test_smaller_grids(limit):
    V = 9000
    rng = np.random.default_rng(8)
    k = np.unique(np.concatenate([rng.integers(0, V * V, 60000), np.arange(V) * V]))
    s, d = k // V, k % V
    w = rng.uniform(0.5, 1.0, len(s)) / np.bincount(s, minlength=V)[s]
    v = rng.random(V) / V
    with Store() as st:
        st.build_level(V, s, d, rng.integers(1, 50, len(s)))
        with st.snapshot() as sn:
            sn.flatten(0).flatten(1)
            want = _results(st, sn, w, v)
            for ctas in (40, 3, 1):
                limit(ctas)
                for a, b in zip(_results(st, sn, w, v), want):
                    if a.dtype == np.float64:
                        # sums in another order; a fixed point to tol / (1 - 0.85)
                        assert np.abs(a - b).sum() <= 2e-12
                    else:
                        assert np.array_equal(a, b)


def test_without_cooperative_launches(limit):
    V = 9000
    rng = np.random.default_rng(9)
    k = np.unique(np.concatenate([rng.integers(0, V * V, 60000), np.arange(V) * V]))
    s, d = k // V, k % V
    with Store() as st:
        st.build_level(V, s, d, rng.integers(1, 50, len(s)))
        with st.snapshot() as sn:
            for flat in (False, True):
                if flat:
                    sn.flatten(0).flatten(1)
                limit(-1)
                want = sn.bfs(1)[0], sn.scc()[0], sn.sssp(1, 16)[0], sn.pagerank_pull(9)
                limit(0)
                got = sn.bfs(1)[0], sn.scc()[0], sn.sssp(1, 16)[0], sn.pagerank_pull(9)
                for a, b in zip(got[:3], want[:3]):
                    assert np.array_equal(a, b)
                assert max_rel_err(got[3], want[3]) <= 1e-12


def test_a_wait_that_runs_out_is_seen():
    """PageRank in one launch, its barriers giving up: the call or the next wait
    says so, and ranks in device memory are not mistaken for a result."""
    import torch
    fails = _lib.lib.lg_test_barrier
    fails.argtypes, fails.restype = [_lib.C.c_int], None
    V = 3000
    rng = np.random.default_rng(10)
    k = np.unique(rng.integers(0, V * V, 30000))
    with Store() as st:
        st.build_level(V, k // V, k % V)
        with st.snapshot() as sn:
            want = sn.pagerank_pull(5)
            dev = torch.zeros(V, dtype=torch.float64, device="cuda")
            try:
                fails(1)
                with pytest.raises(LgError) as e:
                    sn.pagerank_pull(5)
                assert e.value.status == _lib.LG_ETIMEOUT
                sn.pagerank_pull(5, out=dev)
            finally:
                fails(0)
            torch.cuda.synchronize()
            assert torch.isnan(dev).all()
            with pytest.raises(LgError) as e:
                st.sync()
            assert e.value.status == _lib.LG_ETIMEOUT
            st.sync()                                # said once
            sn.pagerank_pull(5, out=dev)
            st.sync()
            assert np.array_equal(dev.cpu().numpy(), want)
            assert np.array_equal(sn.pagerank_pull(5), want)
