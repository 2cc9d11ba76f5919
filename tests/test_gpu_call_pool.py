"""Temporaries of a call come from the store's memory pool: they are counted,
kept between calls up to a bound, and buffers that outlive the store (a tape)
are still freed in order."""
import gc

import numpy as np
import pytest

from llama_b200 import Store

pytestmark = pytest.mark.gpu


def _store():
    rng = np.random.default_rng(3)
    key = np.unique(rng.integers(0, 5000 * 5000, 40000))
    st = Store()
    st.build_level(5000, (key // 5000).astype(np.uint32), (key % 5000).astype(np.uint32))
    return st


def test_pool_does_not_grow_from_call_to_call():
    with _store() as st, st.snapshot() as sn:
        ref = sn.scc()[0]
        sn.triangle_count()
        held = st.device_bytes
        for _ in range(20):
            assert np.array_equal(sn.scc()[0], ref)
            sn.triangle_count()
        assert st.device_bytes == held


def test_temporaries_beyond_the_pool():
    """1.6 GB of temporaries: what the pool cannot hold is given back."""
    V, n = 40_000_003, 1000
    ring = (np.arange(n, dtype=np.int64) * 39_999) % V
    with Store() as st:
        st.build_level(V, ring.astype(np.uint32), np.roll(ring, -1).astype(np.uint32))
        with st.snapshot() as sn:
            before = st.device_bytes
            want = np.arange(V)
            want[ring] = ring.min()
            for _ in range(2):
                labels, r = sn.scc()
                assert r.components == V - n + 1
                assert np.array_equal(labels, want)
                assert st.device_bytes - before <= (1 << 30) + (64 << 20)


def test_tape_freed_after_its_store():
    st = _store()
    sn = st.snapshot()
    w = np.full(sn.num_edges, 0.01)
    v = np.full(sn.max_nodes, 1.0 / sn.max_nodes)
    x, tape, _ = sn.pagerank_fwd(w, v)
    dw, _, _ = tape.backward(v)
    sn.close()
    st.close()
    tape.close()
    gc.collect()
    with _store() as st2, st2.snapshot() as sn2:      # the device is still in order
        assert np.array_equal(sn2.pagerank_fwd(w, v, keep_tape=False)[0], x)
