"""Edge decisions of one labelling when the contraction's list of exact
decisions overflows (a small alpha sends most tables of a large dependent set
there; EDDY_GENERAL_QUEUE_CAP lowers the queue): decided by the popcount
kernel instead, with the same result."""
import numpy as np
import pytest

from test_gpu_units import factor

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("g,n,alpha,cap", [(200, 1000, 1e-9, None), (30, 60, 0.05, "1")])
def test_overflow_is_decided_another_way(g, n, alpha, cap, eddy_lib, monkeypatch):
    rng = np.random.default_rng(8)
    data = factor(rng, g, n, 0.7)
    lab = np.concatenate([np.zeros(n * 2 // 5, np.uint8), np.ones(n - n * 2 // 5, np.uint8)])
    ctx = eddy_lib.Context(max_parents=3, rng=eddy_lib.RNG_EXTERNAL, alpha_edge=alpha,
                           alpha_edge_prior=0.33)
    ctx.load_matrix(data, lab)
    sid = ctx.add_set(np.arange(g))
    monkeypatch.setenv("EDDY_PAIRS_KERNEL", "popc")
    want = ctx.debug_edges(sid, lab)
    monkeypatch.setenv("EDDY_PAIRS_KERNEL", "mma")
    if cap:
        monkeypatch.setenv("EDDY_GENERAL_QUEUE_CAP", cap)
    assert np.array_equal(ctx.debug_edges(sid, lab), want)
    js, U = ctx.run_labellings(sid, lab[None, :])  # the masks are clean again
    monkeypatch.setenv("EDDY_PAIRS_KERNEL", "popc")
    js1, U1 = ctx.run_labellings(sid, lab[None, :])
    assert np.array_equal(U, U1) and np.array_equal(js, js1, equal_nan=True)
    ctx.close()
