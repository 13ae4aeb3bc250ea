"""Labellings whose class sizes differ from the matrix's are refused by every
entry point that takes labellings from the caller (the kernels' arrays are laid
out for the matrix's class sizes), before anything is launched; the context
goes on as before."""
import numpy as np
import pytest

from test_gpu_parity import js_close, planted

pytestmark = pytest.mark.gpu

G, N, NA = 7, 70, 30


def _labels(first):
    return np.concatenate([np.zeros(first, np.uint8), np.ones(N - first, np.uint8)])


@pytest.mark.parametrize("first", [1, NA - 1, NA + 1, N - 1])
def test_other_class_sizes_are_refused(first, eddy_lib, oracle_lib):
    rng = np.random.default_rng(3)
    data, good, bad = planted(rng, G, N, nA=NA, planted=3), _labels(NA), _labels(first)

    def context():
        ctx = eddy_lib.Context(max_parents=3, rng=eddy_lib.RNG_EXTERNAL)
        ctx.load_matrix(data, good)
        return ctx, ctx.add_set(np.arange(G))

    ctx, sid = context()
    calls = [lambda: ctx.run_labellings(sid, np.stack([good, bad])),
             lambda: ctx.debug_unit(sid, bad, 3), lambda: ctx.debug_edges(sid, bad)]
    for call in calls:
        with pytest.raises(eddy_lib.EddyError, match="ERR_ARG"):
            call()
    js, U = ctx.run_labellings(sid, good[None, :])
    ojs, oU = oracle_lib.units(data, good[None, :], None, oracle_lib.params(mp=3))
    assert np.array_equal(U, oU) and js_close(js, ojs)
    # the labellings of a set: the unpermuted one, a later one
    for rows in ([bad, good], [good, bad]):
        ctx, sid = context()
        ctx.set_labellings(sid, np.stack(rows))
        with pytest.raises(eddy_lib.EddyError, match="ERR_ARG"):
            ctx.run()
        with pytest.raises(eddy_lib.EddyError, match="ERR_ARG"):
            ctx.run_permutations(sid, 0, 2)
        k = 0 if rows[0] is good else 1
        js, U = ctx.run_permutations(sid, k, 1)
        assert np.array_equal(U, oU) and js_close(js, ojs)
        ctx.close()
