"""The unit kernel's ways of forming the capped lists of left-out samples,
against the oracle: rows whose lists are formed per subset of their flip
entries (memo rows, the default up to eight entries), rows formed per sample
(EDDY_MEMO_MAX=0 makes every row one; dense decisions without Bonferroni
make long rows), entries past the shared-memory cache, and units whose
networks differ from the full ones nowhere.  Unique networks, their ids and
lists exact; JS as in test_gpu_parity."""
import numpy as np
import pytest

from test_gpu_parity import js_close, make_labels

pytestmark = pytest.mark.gpu


def factor(rng, g, n, loading, missing=0.0):
    """Genes that share one latent factor: pair tests near the threshold."""
    from eddy_gpu import synth
    z = rng.standard_normal(n)
    d = synth.tertiles(loading * z[None, :] + rng.standard_normal((g, n)))
    if missing:
        d[rng.random(d.shape) < missing] = 2
    return d


CASES = [
    # g, n, nA, mp, bonf, loading, missing
    (2, 65, 31, 1, True, 1.2, 0.0),
    (9, 64, 32, 3, False, 0.9, 0.05),
    (33, 129, 60, 2, False, 0.7, 0.0),
    (64, 300, 130, 4, True, 0.7, 0.02),
    (130, 257, 128, 3, False, 0.6, 0.0),
    (40, 300, 150, 3, True, 0.0, 0.0),
]


@pytest.mark.parametrize("memo", [0, 2, 8])
@pytest.mark.parametrize("case", CASES, ids=[f"g{c[0]}n{c[1]}mp{c[3]}" for c in CASES])
def test_lists_of_left_out_samples(case, memo, eddy_lib, oracle_lib, monkeypatch):
    g, n, nA, mp, bonf, loading, missing = case
    rng = np.random.default_rng(g * 1009 + n)
    data = factor(rng, g, n, loading, missing)
    labels0 = np.concatenate([np.zeros(nA, np.uint8), np.ones(n - nA, np.uint8)])
    labs = np.stack([labels0] + [make_labels(rng, n, nA) for _ in range(3)])
    prm = oracle_lib.params(mp=mp, bonferroni=bonf)
    monkeypatch.setenv("EDDY_MEMO_MAX", str(memo))
    ctx = eddy_lib.Context(max_parents=mp, bonferroni=bonf, rng=eddy_lib.RNG_EXTERNAL)
    ctx.load_matrix(data, labels0)
    sid = ctx.add_set(np.arange(g))
    js, U = ctx.run_labellings(sid, labs)
    ojs, oU = oracle_lib.units(data, labs, None, prm)
    assert np.array_equal(U, oU)
    assert js_close(js, ojs)
    mpk = max(1, min(mp, g - 1))
    d, o = ctx.debug_unit(sid, labs[1], mpk), oracle_lib.unit(data, labs[1], None, prm)
    assert np.array_equal(d["ids"], o["unique_ids"])
    for u in range(o["U"]):
        ed = o["uni_edges"][o["uni_epn"][u]:o["uni_epn"][u + 1]]
        got = [d["parents"][u, t, :d["counts"][u, t]] for t in range(g)]
        assert np.array_equal(np.concatenate(got), ed), u
    np.testing.assert_allclose(d["dist"], o["out5"].sum(axis=2), rtol=1e-9, atol=1e-7)
    ctx.close()


def test_entries_past_the_shared_memory_cache(eddy_lib, oracle_lib, monkeypatch):
    """387 genes x 600 samples near the threshold keep ~1700 entries per unit
    (1280 are held in shared memory), rows of up to ~12 of them, and more
    distinct lists than one round of scores; formed per sample, they also
    overfill the table of such lists.  Both ways agree with each other and the
    oracle."""
    rng = np.random.default_rng(38)
    g, n, nA = 387, 600, 300
    data = factor(rng, g, n, 0.7)
    labels0 = np.concatenate([np.zeros(nA, np.uint8), np.ones(n - nA, np.uint8)])
    labs = np.stack([make_labels(rng, n, nA) for _ in range(4)])
    out = []
    for memo in (8, 0):
        monkeypatch.setenv("EDDY_MEMO_MAX", str(memo))
        ctx = eddy_lib.Context(max_parents=3, rng=eddy_lib.RNG_EXTERNAL)
        ctx.load_matrix(data, labels0)
        out.append(ctx.run_labellings(ctx.add_set(np.arange(g)), labs))
        ctx.close()
    assert np.array_equal(out[0][1], out[1][1])
    assert np.array_equal(out[0][0], out[1][0], equal_nan=True)
    ojs, oU = oracle_lib.units(data, labs[:1], None, oracle_lib.params(mp=3))
    assert np.array_equal(out[0][1][:1], oU)
    assert js_close(out[0][0][:1], ojs)


# classes of one word of samples to more than 32, of one side only, and units
# of a few variants (summed by a lane per sample) to several blocks of them
# (summed on the matrix units)
WALKS = [
    # g, n, nA, mp, bonf, loading
    (8, 40, 3, 3, True, 1.0),
    (12, 2100, 1056, 3, True, 0.5),
    (24, 1061, 1029, 3, True, 0.6),
    (90, 520, 257, 3, True, 0.7),
    (110, 290, 33, 4, True, 0.8),
]


@pytest.mark.parametrize("case", WALKS, ids=[f"g{c[0]}n{c[1]}a{c[2]}" for c in WALKS])
def test_sums_over_left_out_samples(case, eddy_lib, oracle_lib):
    g, n, nA, mp, bonf, loading = case
    rng = np.random.default_rng(g * 7919 + n)
    data = factor(rng, g, n, loading, 0.01)
    labels0 = np.concatenate([np.zeros(nA, np.uint8), np.ones(n - nA, np.uint8)])
    labs = np.stack([labels0] + [make_labels(rng, n, nA) for _ in range(3)])
    ctx = eddy_lib.Context(max_parents=mp, bonferroni=bonf, rng=eddy_lib.RNG_EXTERNAL)
    ctx.load_matrix(data, labels0)
    js, U = ctx.run_labellings(ctx.add_set(np.arange(g)), labs)
    ojs, oU = oracle_lib.units(data, labs, None, oracle_lib.params(mp=mp, bonferroni=bonf))
    assert np.array_equal(U, oU)
    assert js_close(js, ojs)
