"""The tensor-core decision path at the ends of its ranges, pinned with
EDDY_PAIRS_KERNEL=mma (batches of few units take the popcount kernel unless
pinned), with the popcount kernel beside it, against the oracle: 512 genes (the
largest pair indices of the queue and the group table), classes of up to 4096
samples and more (the epilogue decides up to 4096, the general path past it),
and sets with and without missing values.  Also the two ways of forming the
unit kernel's lists at the precision-stress shape."""
import numpy as np
import pytest

from test_gpu_parity import js_close, make_labels, planted
from test_gpu_units import factor

pytestmark = pytest.mark.gpu


def _labels0(n, nA):
    return np.concatenate([np.zeros(nA, np.uint8), np.ones(n - nA, np.uint8)])


def _check(eddy_lib, oracle_lib, data, labs, nA, checked, mp=3):
    n = data.shape[1]
    ctx = eddy_lib.Context(max_parents=mp, rng=eddy_lib.RNG_EXTERNAL)
    ctx.load_matrix(data, _labels0(n, nA))
    sid = ctx.add_set(np.arange(len(data)))
    js, U = ctx.run_labellings(sid, labs)
    variant = ctx.stats()["variant"]
    ctx.close()
    ojs, oU = oracle_lib.units(data, labs[checked], None, oracle_lib.params(mp=mp))
    assert np.array_equal(U[checked], oU)
    assert js_close(js[checked], ojs)
    return js, U, variant


@pytest.mark.parametrize("kernel", ["mma", "popc"])
@pytest.mark.parametrize("n,nA,units", [(60, 30, 3), (150, 70, 130)])
def test_largest_set(n, nA, units, kernel, eddy_lib, oracle_lib, monkeypatch):
    rng = np.random.default_rng(n)
    data = planted(rng, 512, n, nA=nA, planted=40)
    data[256:384] = factor(rng, 128, n, 0.9)  # dense rows as well
    labs = np.stack([_labels0(n, nA)] + [make_labels(rng, n, nA) for _ in range(units - 1)])
    monkeypatch.setenv("EDDY_PAIRS_KERNEL", kernel)
    _, _, variant = _check(eddy_lib, oracle_lib, data, labs, nA, [0, units - 1])
    assert (variant >= 0) == (kernel == "mma")


@pytest.mark.parametrize("kernel", ["mma", "popc"])
@pytest.mark.parametrize("n,nA", [(4500, 2000), (8195, 4096), (8195, 4097), (4128, 32)])
def test_largest_classes(n, nA, kernel, eddy_lib, oracle_lib, monkeypatch):
    rng = np.random.default_rng(n + nA)
    data = np.concatenate([planted(rng, 6, n, nA=nA, planted=3), factor(rng, 6, n, 0.2)])
    labs = np.stack([_labels0(n, nA)] + [make_labels(rng, n, nA) for _ in range(2)])
    monkeypatch.setenv("EDDY_PAIRS_KERNEL", kernel)
    _check(eddy_lib, oracle_lib, data, labs, nA, [0, 1, 2])


@pytest.mark.parametrize("missing", [False, True])
@pytest.mark.parametrize("g", [12, 131])
def test_layouts_against_the_popcount_kernel(g, missing, eddy_lib, oracle_lib, monkeypatch):
    rng = np.random.default_rng(g)
    n, nA = 200, 90
    data = factor(rng, g, n, 0.6)
    if missing:
        data[g // 2, 17] = 2
        data[3][rng.random(n) < 0.05] = 2
    labs = np.stack([make_labels(rng, n, nA) for _ in range(40)])
    out = []
    for kernel in ("mma", "popc"):
        monkeypatch.setenv("EDDY_PAIRS_KERNEL", kernel)
        out.append(_check(eddy_lib, oracle_lib, data, labs, nA, [0, 39]))
    assert out[0][2] >= (5 if g == 131 and not missing else 0)
    assert np.array_equal(out[0][1], out[1][1])
    assert np.array_equal(out[0][0], out[1][0], equal_nan=True)


def test_lists_per_subset_and_per_sample(eddy_lib, oracle_lib, monkeypatch):
    """Rows whose lists are formed once per subset of their entries, and every
    row per left-out sample (EDDY_MEMO_MAX=0), at the precision-stress shape."""
    from eddy_gpu import synth
    w = synth.make(4, seed=1)
    genes, mp, pw = w.sets[0][1], w.flags["mp"], w.flags["pw"]
    out = []
    for memo in ("8", "0"):
        monkeypatch.setenv("EDDY_MEMO_MAX", memo)
        ctx = eddy_lib.Context(max_parents=mp, prior_weight=pw, permutations=65,
                               rng=eddy_lib.RNG_COUNTER, seed=9, keep_networks=False)
        ctx.load_matrix(w.data, w.labels)
        sid = ctx.add_set(genes)
        out.append(ctx.run_permutations(sid, 1, 64))
        ctx.close()
    assert np.array_equal(out[0][1], out[1][1])
    assert np.array_equal(out[0][0], out[1][0], equal_nan=True)
    labs = oracle_lib.counter_labels(9, sid, w.labels, 65)
    ojs, oU = oracle_lib.units(w.data[genes], labs[[1, 64]], None, oracle_lib.params(mp=mp, pw=pw))
    assert np.array_equal(out[0][1][[0, 63]], oU)
    assert js_close(out[0][0][[0, 63]], ojs)
