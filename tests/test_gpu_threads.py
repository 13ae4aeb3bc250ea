"""Contexts of several threads at once, whose launches need different amounts
of dynamic shared memory: a kernel's limit belongs to the process, so a launch
must not depend on which thread set it last.  Every call succeeds and gives
what the same context gives alone."""
import threading

import numpy as np
import pytest

from test_gpu_units import factor

pytestmark = pytest.mark.gpu

# genes, samples, class-1 samples: labellings drawn on the device take 16 bytes
# of shared memory a sample (more than the default 48 KB from 2816 samples on),
# the unit kernel's grow with the genes
SHAPES = [(6, 4096, 1500), (8, 2900, 1400), (60, 3400, 1700)]


def test_launches_of_several_threads(eddy_lib):
    ctxs = []
    for g, n, nA in SHAPES:
        rng = np.random.default_rng(g + n)
        ctx = eddy_lib.Context(max_parents=3, permutations=4, rng=eddy_lib.RNG_COUNTER, seed=g)
        ctx.load_matrix(factor(rng, g, n, 0.3),
                        np.concatenate([np.zeros(nA, np.uint8), np.ones(n - nA, np.uint8)]))
        ctxs.append((ctx, ctx.add_set(np.arange(g))))
    want = [c.run_permutations(s, 1, 3) for c, s in ctxs]
    errors = []

    def work(k):
        ctx, sid = ctxs[k]
        try:
            for _ in range(400):
                js, U = ctx.run_permutations(sid, 1, 3)
                assert np.array_equal(U, want[k][1])
                assert np.array_equal(js, want[k][0], equal_nan=True)
        except Exception as e:  # noqa: BLE001  (reported by the test's own thread)
            errors.append(f"{SHAPES[k]}: {e}")

    threads = [threading.Thread(target=work, args=(k,)) for k in range(len(ctxs))]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    for c, _ in ctxs:
        c.close()
    assert not errors, errors
