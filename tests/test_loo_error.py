"""The FP32 error of the ten-decision form (loo_f2 in eddy_device.cuh): its
Q' of every one-sample-less table, restated in numpy float32 with a
reciprocal off by up to 2^-23, against 64 bits over random and strongly
dependent tables of 32 to 4096 samples: within 24 2^-24 Q', half of the
margin by which the thresholds are moved inward.  CPU only."""
import numpy as np

F = np.float32


def _rcp(x, rng):
    # rcp.approx.ftz.f32: at most one unit in the last place off
    r = F(1) / x
    return (r.view(np.int32) + rng.integers(-1, 2, r.shape, dtype=np.int32)).view(np.float32)


def _loo32(o, rng):
    R, C = o.sum(2), o.sum(1)
    eR, eC = _rcp(R * (R - F(1)), rng), _rcp(C * (C - F(1)), rng)
    iR, iR1, iC, iC1 = eR * (R - F(1)), eR * R, eC * (C - F(1)), eC * C
    p = o * o
    f = lambda a, b, c: (a.astype(np.float64) * b + c).astype(F)  # noqa: E731  one rounding
    S = f(p[:, :, 2], iC[:, None, 2], f(p[:, :, 1], iC[:, None, 1], p[:, :, 0] * iC[:, None, 0]))
    Q = f(S[:, 2], iR[:, 2], f(S[:, 1], iR[:, 1], S[:, 0] * iR[:, 0]))
    K = f(p[:, 2], iR[:, 2, None], f(p[:, 1], iR[:, 1, None], p[:, 0] * iR[:, 0, None]))
    Qb = f(eC, K, Q[:, None])
    Sab = f(p, eC[:, None, :], S[:, :, None])
    w = iC1[:, None, :] * iR1[:, :, None]
    return Q, f(f(o, F(-2), F(1)), w, f(eR[:, :, None], Sab, Qb[:, None, :]))


def _q64(o):
    R, C = o.sum(2), o.sum(1)
    return (o ** 2 / (R[:, :, None] * C[:, None, :])).sum((1, 2))


def test_error_of_the_ten_decision_form():
    rng = np.random.default_rng(4)
    worst, seen = 0.0, 0
    for n in (48, 64, 100, 187, 400, 601, 1500, 2777, 4096):
        prob = rng.dirichlet(np.full(9, 3.0), 4000)
        prob[::2] = np.outer([0.33, 0.33, 0.34], [0.3, 0.3, 0.4]).ravel()
        # diagonal tables: chi-square near its largest, 2 N
        prob[1::4] = 0.9 * np.eye(3).ravel() / 3 + 0.1 * prob[1::4]
        t = np.stack([rng.multinomial(n, q) for q in prob]).reshape(-1, 3, 3)
        rm, cm = t.sum(2).min(1), t.sum(1).min(1)
        t = t[(rm >= 2) & (cm >= 2) & ((rm - 1) * (cm - 1) >= 5 * (n - 1))]
        if not len(t):
            continue  # the smallest sizes may leave no table the form applies to
        seen += len(t)
        Q, Q1 = _loo32(t.astype(F), rng)
        q64 = _q64(t.astype(np.float64))
        worst = max(worst, float(np.max(np.abs(Q - q64) / q64)))
        for a in range(3):
            for b in range(3):
                less = t.astype(np.float64)
                less[:, a, b] -= 1
                ok = t[:, a, b] > 0
                q = _q64(less[ok])
                worst = max(worst, float(np.max(np.abs(Q1[ok, a, b] - q) / q)))
    assert seen > 10000
    assert worst < 24 * 2.0 ** -24, worst
