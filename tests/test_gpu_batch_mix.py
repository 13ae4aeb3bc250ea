"""Results of a set do not depend on the sets it shares a batch with.  A set
of 250 genes on its own takes unit blocks of 384 threads, beside many small
ones blocks of 256 (both choices are made for the whole batch): its JS values
and likelihoods are the same bits either way, and the oracle's.  A batch of
mixed sizes that takes 384 threads is compared with the oracle, too."""
import numpy as np
import pytest

from test_gpu_parity import js_close
from test_gpu_units import factor

pytestmark = pytest.mark.gpu

N, NA, SEED, R = 420, 200, 13, 4


def _run(eddy_lib, data, labels0, sets):
    ctx = eddy_lib.Context(max_parents=3, permutations=R, rng=eddy_lib.RNG_COUNTER, seed=SEED)
    ctx.load_matrix(data, labels0)
    ids = [ctx.add_set(g) for g in sets]
    ctx.run()
    out = [(ctx.js(k), ctx.networks(k), ctx.edge_list(k)) for k in ids]
    ctx.close()
    return out


@pytest.mark.parametrize("large,small", [((250,), 120), ((290, 250), 2), ((250, 251, 249), 60)])
def test_large_sets_alone_and_among_small_ones(large, small, eddy_lib, oracle_lib):
    rng = np.random.default_rng(len(large) * 100 + small)
    G = 300
    data = factor(rng, G, N, 0.62)
    labels0 = np.concatenate([np.zeros(NA, np.uint8), np.ones(N - NA, np.uint8)])
    big = [np.sort(rng.choice(G, g, replace=False)) for g in large]
    tiny = [rng.choice(G, 6, replace=False) for _ in range(small)]
    mixed = _run(eddy_lib, data, labels0, big + tiny)[:len(big)]
    alone = _run(eddy_lib, data, labels0, big)
    for k, genes in enumerate(big):
        (ja, na, ea), (jm, nm, em) = alone[k], mixed[k]
        assert na["U"] > 128  # more networks than one pass of a block's lanes
        assert np.array_equal(ja[1], jm[1])
        assert np.array_equal(ja[0], jm[0], equal_nan=True)
        for a, b in ((na, nm), (ea, em)):
            for f in a:
                assert np.array_equal(a[f], b[f]), f
        lab = oracle_lib.counter_labels(SEED, k, labels0, R)[:2]
        ojs, oU = oracle_lib.units(data[genes], lab, None, oracle_lib.params(mp=3))
        assert np.array_equal(ja[1][:2], oU)
        assert js_close(ja[0][:2], ojs)
