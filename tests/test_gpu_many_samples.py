"""Many samples and few genes.  The unit kernel's class planes are then packed
by several warps a row of genes, which share the sample words (from 1024
samples on): labellings in which whole stretches of samples belong to one
class, and classes of a few samples, leave some of them without a word.  The
popcount kernel takes parts of its tiles in batches of few units, and a set
with a class above 32767 samples (decided in FP64 throughout) goes to the
contraction as far as its list holds: every route gives the same."""
import numpy as np
import pytest

from test_gpu_parity import js_close, make_labels
from test_gpu_units import factor

pytestmark = pytest.mark.gpu


def _sorted(n, nA):
    return np.concatenate([np.zeros(nA, np.uint8), np.ones(n - nA, np.uint8)])


@pytest.mark.parametrize("g,n,nA", [(5, 4097, 7), (33, 1500, 1493), (70, 1100, 20), (40, 2048, 1024),
                                    (9, 1024, 500), (12, 1023, 500)])
def test_class_planes_of_several_warps(g, n, nA, eddy_lib, oracle_lib):
    rng = np.random.default_rng(g * n)
    data = factor(rng, g, n, 0.5, 0.01)
    lab0 = _sorted(n, nA)
    # the class in front, behind, and in the middle, then at random
    labs = np.stack([lab0, lab0[::-1], np.roll(lab0, n // 3), make_labels(rng, n, nA)])
    ctx = eddy_lib.Context(max_parents=3, rng=eddy_lib.RNG_EXTERNAL)
    ctx.load_matrix(data, lab0)
    js, U = ctx.run_labellings(ctx.add_set(np.arange(g)), labs)
    ctx.close()
    ojs, oU = oracle_lib.units(data, labs, None, oracle_lib.params(mp=3))
    assert np.array_equal(U, oU)
    assert js_close(js, ojs)


@pytest.mark.parametrize("units", [1, 3, 40])
@pytest.mark.parametrize("g", [3, 40, 100])
@pytest.mark.parametrize("nB", [32767, 32768])
def test_classes_above_the_fp32_limit(nB, g, units, eddy_lib, oracle_lib, monkeypatch):
    n = 36000
    nA = n - nB
    rng = np.random.default_rng(nB + g)
    data = factor(rng, g, n, 0.06)
    lab0 = _sorted(n, nA)
    labs = np.stack([make_labels(rng, n, nA) for _ in range(units)])
    ctx = eddy_lib.Context(max_parents=3, rng=eddy_lib.RNG_EXTERNAL)
    ctx.load_matrix(data, lab0)
    sid = ctx.add_set(np.arange(g))
    out = []
    for kernel in (None, "popc", "mma"):
        if kernel:
            monkeypatch.setenv("EDDY_PAIRS_KERNEL", kernel)
        out.append(ctx.run_labellings(sid, labs))
    ctx.close()
    for js, U in out[1:]:
        assert np.array_equal(U, out[0][1])
        assert np.array_equal(js, out[0][0], equal_nan=True)
    if g == 3:
        ojs, oU = oracle_lib.units(data, labs[:1], None, oracle_lib.params(mp=3))
        assert np.array_equal(out[0][1][:1], oU)
        assert js_close(out[0][0][:1], ojs)
