"""The single-precision enclosures of the bundle bounds (csrc/cvl_curvelets.cuh), restated
step by step in numpy float32 and compared with the float64 bounds: every accepted cell's
bounds lie within e0 max(1, |k| / max_k) of them, or are past max_k on the same side."""
import numpy as np
import pytest

U = 2.0 ** -24
F = np.float32


def _r(x):
    return np.asarray(x, np.float64).astype(F).astype(np.float64)  # one rounding to single


def _rcp(x, rng):
    y = _r(1.0 / x)  # rcp.approx: within 2u of 1/x
    return _r(y * (1.0 + rng.choice([-1.0, 0.0, 1.0], y.shape) * U))


def _pairs(kind, n, rng, nrad, dx):
    """DX, DY, T2, T0 of n pairs."""
    r = np.sqrt(rng.uniform(4 * dx * dx, nrad * nrad, n))
    phi = rng.uniform(-np.pi, np.pi, n)
    T2 = rng.uniform(-np.pi, np.pi, n)
    T0 = rng.uniform(-np.pi, np.pi, n)
    if kind == "along":  # neighbours on a curve
        T0 = T2 + rng.normal(0, 0.1, n)
        phi = T2 + rng.normal(0, 0.1, n) + np.pi * rng.integers(0, 2, n)
    elif kind == "beside":  # parallel curves: denominators and sines that cancel
        T0 = T2 + rng.normal(0, 0.02, n) + rng.choice([0.0, 15 / 180 * np.pi, -15 / 180 * np.pi], n)
        phi = T2 + np.pi / 2 + rng.normal(0, 1, n) * 10.0 ** rng.uniform(-9, -1, n)
    elif kind == "touching":  # just past the close pairs' radius: e1 near 0
        r = 2 * dx + 10.0 ** rng.uniform(-9, -1, n)
        phi = T2 + np.pi / 2 + rng.normal(0, 1, n) * 10.0 ** rng.uniform(-9, -1, n)
    elif kind == "lattice":
        d = rng.integers(-3, 4, (n, 2)).astype(float)
        d[(d ** 2).sum(1) == 0] = [1.0, 0.0]
        T2 = rng.integers(-4, 5, n) * (np.pi / 4)
        return d[:, 0], d[:, 1], T2, T2 + rng.integers(-1, 2, n) * (np.pi / 4)
    return r * np.cos(phi), r * np.sin(phi), T2, T0


@pytest.mark.parametrize("kind", ["any", "along", "beside", "touching", "lattice"])
@pytest.mark.parametrize("dx,dt,sx,st,max_k,nrad", [(0.4, 15 / 180 * np.pi, 0.1, 0.08, 0.3, 3.5),
                                                    (0.8, 15 / 180 * np.pi, 0.2, 0.08, 0.05, 5.0),
                                                    (0.4, 0.2, 0.1, 0.08, 3.0, 3.0)])
def test_enclosures_hold(kind, dx, dt, sx, st, max_k, nrad):
    rng = np.random.default_rng(len(kind) * 1000 + int(max_k * 100))
    n = 60000
    DX, DY, T2, T0 = _pairs(kind, n, rng, nrad, dx)
    keep = DX * DX + DY * DY >= 4 * dx * dx
    DX, DY, T2, T0 = DX[keep], DY[keep], T2[keep], T0[keep]
    n = DX.size
    P, Q = 9, 2 * int(np.floor(dt / st + 0.5)) + 1
    assert 2 * int(np.floor(dx / sx + 0.5)) + 1 == P
    dm = sx * (P - 1) / 2
    e0 = 2.0 ** -14 * max_k
    den = e0 - 8 * U * max_k
    up = 1.02
    X, Y = _r(DX), _r(DY)
    Rb = np.abs(X) + np.abs(Y)
    ethr = up * U * (4 * dm + 16 * dx + max_k * (3 * dm * dm + 6 * dx * dx) + Rb * (10 + max_k * 12 * dm)
                     + Rb * Rb * max_k * 7) / den
    dthr = up * U * (4 + max_k * 6 * dm + Rb * max_k * 5) / den
    S1 = up * (2 * max_k * dthr + 8 * U)
    dtiny = 2 * U * (5 * nrad + 6 * dm)
    A = _r(X * X + _r(Y * Y - _r(dx * dx)))
    accepted = 0
    for j in range(Q):
        T2t = T2 + st * (j - (Q - 1) / 2)
        sT, cT = np.sin(T2t), np.cos(T2t)
        sTf, cTf = _r(sT), _r(cT)
        tt = sT * DX - cT * DY
        t2 = _r(sTf * (-2 * X) + _r(cTf * (2 * Y)))
        exact, single = [], []
        for sign in (-1.0, 1.0):
            t = T0 + sign * dt
            c, s = np.cos(t), np.sin(t)
            cf, sf = _r(c), _r(s)
            exact.append((np.sin(T2t - t), c * DX, s * DY))
            single.append((_r(sTf * cf + _r(cTf * -sf)), _r(cf * X + _r(sf * Y))))
        for i in range(P):
            d = sx * (i - (P - 1) / 2)
            with np.errstate(all="ignore"):
                e1 = (((DX * DX - 2 * d * tt) + DY * DY) - dx * dx) + d * d
                want = [2 * (tt - d - dx) / e1, 2 * (tt - d + dx) / e1] + \
                       [s / (-s * d + c + q) for s, c, q in exact]
                e1f = _r(_r(d) * t2 + _r(A + _r(d * d)))
                nre = -_rcp(e1f, rng)
                klo = _r(_r(t2 + _r(2 * d + 2 * dx)) * nre)
                got = [klo, _r(nre * _r(-4 * dx) + klo)]
                ok = [e1f >= ethr] * 2
                for s, cn in single:
                    D = _r(-s * _r(d) + cn)
                    got.append(_r(s * _rcp(D, rng)))
                    ok.append((np.abs(D) >= dthr) | ((np.abs(s) >= S1) & (np.abs(D) >= dtiny)))
            every = np.logical_and.reduce(ok)
            accepted += every.sum()
            for w, g in zip(want, got):
                w, g = w[every], g[every]
                past = (np.abs(w) > max_k) & (np.abs(g) > max_k * (1 + 2.0 ** -13)) & (np.sign(w) == np.sign(g))
                near = np.abs(g - w) <= e0 * np.maximum(1.0, np.abs(w) / max_k)
                assert np.all(past | near), (kind, i, j, np.abs(g - w)[~(past | near)][:3], w[~(past | near)][:3])
    assert accepted > 0.2 * n * P * Q
