"""Sets of mixed sizes and layouts (with and without missing values) in one
run: iteration 0 of all of them is one batch, largest set first, the others'
permutations follow by contingency kernel.  Every set's JS and unique networks
against the oracle on its own labellings, whatever the order of the sets; JS
as in test_gpu_parity."""
import numpy as np
import pytest

from test_gpu_parity import js_close

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("sizes", [(3, 70, 5, 110, 2, 33), (110, 33, 2), (6,)])
@pytest.mark.parametrize("mode", ["counter", "glibc"])
def test_mixed_sets(sizes, mode, eddy_lib, oracle_lib):
    rng = np.random.default_rng(sum(sizes))
    n, nA, R, seed = 150, 70, 9, 5
    z = rng.standard_normal(n)
    raw = 0.9 * z[None, :] + rng.standard_normal((130, n))
    data = np.digitize(raw, [-0.6, 0.6]).astype(np.int8) - 1
    data[120:][rng.random((10, n)) < 0.1] = 2  # genes with missing values
    labels0 = np.concatenate([np.zeros(nA, np.uint8), np.ones(n - nA, np.uint8)])
    ctx = eddy_lib.Context(max_parents=3, permutations=R, seed=seed,
                           rng=eddy_lib.RNG_COUNTER if mode == "counter" else eddy_lib.RNG_GLIBC)
    ctx.load_matrix(data, labels0)
    genes = [np.sort(rng.choice(130 if k % 2 else 120, g, replace=False)) for k, g in enumerate(sizes)]
    ids = [ctx.add_set(g) for g in genes]
    ctx.run()
    for k, g in zip(ids, genes):
        js, U = ctx.js(k)
        count = len(js) if mode == "counter" else 1  # (glibc: one stream over the sets)
        lab = oracle_lib.counter_labels(seed, k, labels0, R)[:count]
        ojs, oU = oracle_lib.units(data[g], lab, None, oracle_lib.params(mp=3))
        assert np.array_equal(U[:count], oU)
        assert js_close(js[:count], ojs)
    ctx.close()
