"""Kept outputs (networks, likelihoods, edge lists) that do not fit the room a
batch has for them at first (EDDY_KEEP_CAP lowers it): the units that found
none run again in a larger one.  Everything a set reports, its decision
counters too, is what a run with room for all gives."""
import numpy as np
import pytest

from test_gpu_units import factor

pytestmark = pytest.mark.gpu


def _sweep(eddy_lib, rng_mode):
    rng = np.random.default_rng(61)
    G, n, nA = 160, 240, 110
    data = factor(rng, G, n, 0.7)
    labels0 = np.concatenate([np.zeros(nA, np.uint8), np.ones(n - nA, np.uint8)])
    ctx = eddy_lib.Context(max_parents=3, permutations=4, rng=rng_mode, seed=2)
    ctx.load_matrix(data, labels0)
    ids = [ctx.add_set(rng.choice(G, g, replace=False)) for g in (40, 3, 90, 25, 60, 12)]
    ctx.run()
    out = []
    for s in ids:
        su = ctx.summary(s)
        assert su["tables"] == 2 * su["iterations"] * su["genes"] * (su["genes"] - 1) // 2
        out.append((su, ctx.js(s), ctx.networks(s), ctx.edge_list(s)))
    st = ctx.stats()
    st.pop("variant")
    ctx.close()
    return out, st


@pytest.mark.parametrize("room", [8, 20000])
@pytest.mark.parametrize("mode", ["counter", "glibc"])
def test_kept_units_without_room_run_again(mode, room, eddy_lib, monkeypatch):
    rng_mode = eddy_lib.RNG_COUNTER if mode == "counter" else eddy_lib.RNG_GLIBC
    want, stats = _sweep(eddy_lib, rng_mode)
    monkeypatch.setenv("EDDY_KEEP_CAP", str(room))
    got, again = _sweep(eddy_lib, rng_mode)
    assert again == stats
    for (sa, ja, na, ea), (sb, jb, nb, eb) in zip(want, got):
        for k in sa:
            assert sa[k] == sb[k] or (np.isnan(sa[k]) and np.isnan(sb[k])), k
        assert all(np.array_equal(x, y, equal_nan=True) for x, y in zip(ja, jb))
        for a, b in ((na, nb), (ea, eb)):
            for k in a:
                assert np.array_equal(a[k], b[k], equal_nan=a is na and k == "lval"), k
