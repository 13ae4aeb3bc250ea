"""The popcount kernel's tiles (32 x 32 pairs, four rows a warp, 16 plane
words a pass; four counted cells for sets without missing values, nine
otherwise) against the oracle's edge decisions at the edges of tiles and
word passes, and against the tensor-core path on the units of a batch."""
import numpy as np
import pytest

from test_gpu_parity import js_close, make_labels
from test_gpu_units import factor

pytestmark = pytest.mark.gpu

CASES = [
    # g, n, nA, missing: tiles of 1 to 3 rows of genes, 1 to 18 plane words
    (2, 64, 32, 0.0),
    (31, 65, 30, 0.03),
    (32, 127, 60, 0.0),
    (33, 300, 140, 0.0),
    (64, 1024, 400, 0.02),
    (65, 1088, 500, 0.0),
]


@pytest.mark.parametrize("case", CASES, ids=[f"g{c[0]}n{c[1]}" for c in CASES])
def test_popcount_tiles(case, eddy_lib, oracle_lib, monkeypatch):
    g, n, nA, missing = case
    rng = np.random.default_rng(17 * g + n)
    data = factor(rng, g, n, min(1.0, 8.0 / np.sqrt(n)), missing)
    labels0 = np.concatenate([np.zeros(nA, np.uint8), np.ones(n - nA, np.uint8)])
    pr = np.zeros((g, g), np.uint8)
    pr[0, 1] = pr[1, 0] = 1
    ctx = eddy_lib.Context(max_parents=3, rng=eddy_lib.RNG_EXTERNAL)
    ctx.load_matrix(data, labels0)
    sid = ctx.add_set(np.arange(g), pr)
    monkeypatch.setenv("EDDY_PAIRS_KERNEL", "popc")
    for _ in range(2):
        lab = make_labels(rng, n, nA)
        e, _, _ = oracle_lib.k1_edges(data[:, lab == 0], data[:, lab == 1], pr, oracle_lib.params())
        assert np.array_equal(ctx.debug_edges(sid, lab), e)
    labs = np.stack([make_labels(rng, n, nA) for _ in range(40)])
    a = ctx.run_labellings(sid, labs)
    monkeypatch.setenv("EDDY_PAIRS_KERNEL", "mma")
    b = ctx.run_labellings(sid, labs)
    assert np.array_equal(a[1], b[1]) and np.array_equal(a[0], b[0], equal_nan=True)
    monkeypatch.delenv("EDDY_PAIRS_KERNEL")
    c = ctx.run_labellings(sid, labs[:2])
    ojs, oU = oracle_lib.units(data, labs[:2], pr, oracle_lib.params())
    assert np.array_equal(c[1], oU) and js_close(c[0], ojs)
