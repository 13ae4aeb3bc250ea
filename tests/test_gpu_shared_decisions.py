"""The popcount kernel shares out the decisions its packed forms leave over a
block, FP32 ones a lane per table and exact FP64 ones a lane per decision:
steps with a single such table, with all of a block's 512 (every decision in
FP64; an alpha outside (0, 1]), tables with empty cells (one decision for all
of them), and a small alpha, which sends part of the tables to FP64.  Edge
decisions, unique networks and the decision counters against the oracle and
the tensor-core path."""
import numpy as np
import pytest

from test_gpu_parity import js_close, make_labels
from test_gpu_units import factor

pytestmark = pytest.mark.gpu

CASES = [
    # g, n, nA, alpha, fp64, missing: tiles of a few genes to three rows of them
    (2, 12, 6, 0.05, True, 0.0),
    (8, 40, 16, 0.05, True, 0.0),
    (33, 60, 25, 0.05, True, 0.05),
    (65, 40, 20, 1.5, False, 0.0),
    (40, 24, 12, 0.3, False, 0.1),
    (66, 400, 160, 1e-9, False, 0.0),
    (70, 300, 150, 1e-6, False, 0.02),
]


@pytest.mark.parametrize("case", CASES, ids=[f"g{c[0]}n{c[1]}a{c[3]}" for c in CASES])
def test_decisions_shared_over_a_block(case, eddy_lib, oracle_lib, monkeypatch):
    g, n, nA, alpha, fp64, missing = case
    rng = np.random.default_rng(g * 31 + n)
    data = factor(rng, g, n, 0.8, missing)
    labels0 = np.concatenate([np.zeros(nA, np.uint8), np.ones(n - nA, np.uint8)])
    prm = oracle_lib.params(mp=3, alpha_edge=alpha, alpha_edge_prior=0.33)
    if fp64:
        monkeypatch.setenv("EDDY_DECISIONS", "fp64")
    monkeypatch.setenv("EDDY_PAIRS_KERNEL", "popc")
    ctx = eddy_lib.Context(max_parents=3, rng=eddy_lib.RNG_EXTERNAL, alpha_edge=alpha,
                           alpha_edge_prior=0.33)
    ctx.load_matrix(data, labels0)
    sid = ctx.add_set(np.arange(g))
    lab = make_labels(rng, n, nA)
    e, _, _ = oracle_lib.k1_edges(data[:, lab == 0], data[:, lab == 1], None, prm)
    assert np.array_equal(ctx.debug_edges(sid, lab), e)
    for units in (1, 30, 300):  # quarters, halves, whole tiles
        labs = np.stack([make_labels(rng, n, nA) for _ in range(units)])
        js, U = ctx.run_labellings(sid, labs)
        st = ctx.stats()
        assert st["tables"] == units * g * (g - 1)
        if fp64 or alpha > 1:
            assert st["exact_rechecks"] >= st["tables"]
        ojs, oU = oracle_lib.units(data, labs[:2], None, prm)
        assert np.array_equal(U[:2], oU) and js_close(js[:2], ojs)
        if not fp64 and alpha <= 1:
            monkeypatch.setenv("EDDY_PAIRS_KERNEL", "mma")
            ja, Ua = ctx.run_labellings(sid, labs)
            monkeypatch.setenv("EDDY_PAIRS_KERNEL", "popc")
            assert np.array_equal(U, Ua) and np.array_equal(js, ja, equal_nan=True)
    ctx.close()
