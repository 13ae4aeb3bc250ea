"""Counter-stream labellings drawn on the device (a warp per unit, four units
a block): sample counts around the words' edges, one sample or all but one in
class 1, and unit counts that leave warps of the last block idle, against the
oracle on its own labellings.  Unique networks exact; JS as in
test_gpu_parity."""
import numpy as np
import pytest

from test_gpu_parity import js_close

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,nA,R", [(33, 1, 5), (64, 63, 9), (65, 32, 4), (127, 126, 6),
                                    (129, 64, 11), (700, 345, 7), (2049, 1000, 3)])
def test_labellings_on_the_device(n, nA, R, eddy_lib, oracle_lib):
    rng = np.random.default_rng(n * 31 + nA)
    z = rng.standard_normal(n)
    raw = 1.2 * z[None, :] + rng.standard_normal((7, n))
    data = np.digitize(raw, [-0.6, 0.6]).astype(np.int8) - 1
    labels0 = np.concatenate([np.zeros(nA, np.uint8), np.ones(n - nA, np.uint8)])
    ctx = eddy_lib.Context(max_parents=3, permutations=R, rng=eddy_lib.RNG_COUNTER, seed=n)
    ctx.load_matrix(data, labels0)
    sid = ctx.add_set(np.arange(7))
    js, U = ctx.run_permutations(sid, 0, R)
    ctx.close()
    ojs, oU = oracle_lib.units(data, oracle_lib.counter_labels(n, sid, labels0, R), None,
                               oracle_lib.params(mp=3))
    assert np.array_equal(U, oU)
    assert js_close(js, ojs)


@pytest.mark.parametrize("units", [32768, 32771])
def test_largest_batches(units, eddy_lib):
    """One batch of 32768 units (the queue's largest unit index is used) and
    one more than a batch holds, against the same labellings in batches of
    8192."""
    rng = np.random.default_rng(9)
    g, n, nA = 40, 96, 40
    z = rng.standard_normal(n)
    data = np.digitize(z[None, :] + rng.standard_normal((g, n)), [-0.6, 0.6]).astype(np.int8) - 1
    labels0 = np.concatenate([np.zeros(nA, np.uint8), np.ones(n - nA, np.uint8)])
    ctx = eddy_lib.Context(max_parents=2, permutations=units, rng=eddy_lib.RNG_COUNTER, seed=3)
    ctx.load_matrix(data, labels0)
    sid = ctx.add_set(np.arange(g))
    js, U = ctx.run_permutations(sid, 0, units)
    parts = [ctx.run_permutations(sid, k, min(8192, units - k)) for k in range(0, units, 8192)]
    ctx.close()
    assert np.array_equal(U, np.concatenate([p[1] for p in parts]))
    assert np.array_equal(js, np.concatenate([p[0] for p in parts]), equal_nan=True)
