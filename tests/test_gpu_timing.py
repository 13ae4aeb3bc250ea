"""Device time by kernel (eddy_last_stage_timing): the parts are all positive
where their work exists and add up to eddy_last_timing's, whether a batch is
launched directly or replayed."""
import numpy as np
import pytest

from test_gpu_units import factor

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("g,n,units", [(20, 200, 1), (120, 400, 700)])
def test_stages_add_up(g, n, units, eddy_lib):
    rng = np.random.default_rng(g)
    labels0 = np.concatenate([np.zeros(n // 2, np.uint8), np.ones(n - n // 2, np.uint8)])
    ctx = eddy_lib.Context(max_parents=3, permutations=units + 1, rng=eddy_lib.RNG_COUNTER, seed=1)
    ctx.load_matrix(factor(rng, g, n, 0.8), labels0)
    sid = ctx.add_set(np.arange(g))
    for _ in range(4):  # first batch, direct launches, captured, replayed
        _, U = ctx.run_permutations(sid, 1, units)
        assert U.max() > 2  # some unit has a JS to compute
        t = ctx.timing()
        assert min(t["ms_gemm"], t["ms_networks"], t["ms_js"]) > 0.0, t
        assert t["ms_js"] < t["ms_networks"], t
        assert abs(t["ms_gemm"] + t["ms_decide"] - t["ms_pairs"]) < 1e-3 * t["ms_pairs"] + 1e-3
        assert abs(t["ms_networks"] + t["ms_js"] - t["ms_units"]) < 1e-3 * t["ms_units"] + 1e-3
    ctx.close()
