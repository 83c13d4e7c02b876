"""The enclosures' thresholds as the engine makes them (make_fast, csrc/cvl_enclosures.h,
compiled here), against the kernels' single-precision operations restated in numpy and the
reference's FP64 bounds: every accepted cell's bounds lie within e0 max(1, |k| / max_k) of
them, or are past max_k on the same side, with the search radius apart from nrad."""
import ctypes as C
import os
import shutil
import subprocess

import numpy as np
import pytest

U = 2.0 ** -24
CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))),
                    "curvelet_construction_on_gpu_b200", "csrc")
SHIM = """
#include "cvl_enclosures.h"
struct M { double nrad, rad_sqr, dx, dx2, dt, sx, st, max_k; int P, Q, cells, max_cand, w; };
extern "C" void model(const M *m, cvl::FastModel *f) { *f = cvl::make_fast(*m); }
extern "C" double radius(const M *m) { return cvl::pair_radius(*m); }
extern "C" int size() { return (int)sizeof(cvl::FastModel); }
"""


class _M(C.Structure):
    _fields_ = [(k, C.c_double) for k in ("nrad", "rad_sqr", "dx", "dx2", "dt", "sx", "st", "max_k")] + \
               [(k, C.c_int) for k in ("P", "Q", "cells", "max_cand", "w")]


class _F(C.Structure):
    _fields_ = [("d", C.c_float * 9), ("d2", C.c_float * 9), ("c2", C.c_float * 9)] + \
               [(k, C.c_float) for k in ("mk", "h", "dx2", "dx_2", "ndx_4", "e0", "eR", "eRR", "d0", "dR", "s0", "sR",
                                         "dtiny", "fe", "fd", "fa")] + \
               [("ok", C.c_int), ("rank", C.c_ubyte * 64), ("cell_of", C.c_ubyte * 64)]


@pytest.fixture(scope="module")
def shim(tmp_path_factory):
    d = tmp_path_factory.mktemp("enclosures")
    (d / "shim.cpp").write_text(SHIM)
    cxx = "/usr/bin/g++" if os.path.exists("/usr/bin/g++") else shutil.which("g++")
    subprocess.run([cxx, "-O1", "-std=c++17", "-shared", "-fPIC", "-I", CSRC, "-o", str(d / "shim.so"),
                    str(d / "shim.cpp")], check=True)
    lib = C.CDLL(str(d / "shim.so"))
    lib.radius.restype = C.c_double
    assert lib.size() == C.sizeof(_F)
    return lib


def _model(shim, nrad=3.5, rad=None, w=3, dx=0.4, dt=15 / 180 * np.pi, sx=0.1, st=0.08, max_k=0.3):
    rad = nrad if rad is None else rad
    P, Q = (2 * int(np.floor(a / s + 0.5)) + 1 for a, s in ((dx, sx), (dt, st)))
    m = _M(nrad, rad * rad, dx, dx * dx, dt, sx, st, max_k, P, Q, P * Q, 128, w)
    f = _F()
    shim.model(C.byref(m), C.byref(f))
    return m, f, shim.radius(C.byref(m))


def _r(x):
    return np.asarray(x, np.float64).astype(np.float32).astype(np.float64)  # one rounding to single


def _rcp(x, rng):
    y = _r(1.0 / x)  # rcp.approx: within 2u of 1/x
    return _r(y * (1.0 + rng.choice([-1.0, 0.0, 1.0], y.shape) * U))


def _offset(s, k, n):
    return s * (k - (n - 1.0) / 2.0)


def _pairs(rng, m, R, n, turns):
    """DX, DY, T2, T0 and a cell (i, j) each, a fifth of them each (where it is not a close pair):
    at random; a k_dt denominator D of the cell near 0; its e1 near 0; D near 0 and s with it,
    so that k_dt is about max_k; e1 near 0 and a k_dx numerator with it. Orientations
    within `turns` turns."""
    def turn():
        return 2 * np.pi * rng.integers(-turns, turns + 1, n)

    def sign():
        return rng.choice([-1.0, 1.0], n)

    T2, T0 = rng.uniform(-np.pi, np.pi, n) + turn(), rng.uniform(-np.pi, np.pi, n) + turn()
    i, j = rng.integers(0, m.P, n), rng.integers(0, m.Q, n)
    d, T2t = _offset(m.sx, i, m.P), T2 + _offset(m.st, j, m.Q)
    sT, cT = np.sin(T2t), np.cos(T2t)
    r, phi = R * np.sqrt(rng.uniform(0, 1, n)), rng.uniform(-np.pi, np.pi, n)
    tt, v = r * np.cos(phi), r * np.sin(phi)  # DX, DY along (sT, -cT) and (cT, sT)
    kind = np.arange(n) % 5
    tiny, k = sign() * 10.0 ** rng.uniform(-11, -2, n), m.max_k * rng.uniform(-1.5, 1.5, n)
    # e1 = (tt - d)^2 + v^2 - dx^2, and D is v where s is 0
    side, e = sign(), np.abs(tiny)
    tt = np.where(kind == 2, d + (m.dx + tiny) * np.cos(phi), np.where(kind == 4, d + side * (m.dx + k * e / 2), tt))
    v = np.where(kind == 2, (m.dx + tiny) * np.sin(phi), np.where(kind == 3, tiny, np.where(
        kind == 4, sign() * np.sqrt(np.maximum(e * (1 - k * m.dx) - (k * e / 2) ** 2, 0)), v)))
    DX, DY = sT * tt + cT * v, sT * v - cT * tt
    # D = a cos t + b sin t, with t = T0 -+ dt, a = DX - d sin T2t, b = DY + d cos T2t
    a, b = DX - d * sT, DY + d * cT
    t = np.where(kind == 1, np.arctan2(b, a) + np.pi / 2 + tiny / np.maximum(np.hypot(a, b), 1e-9), T2t - k * tiny) + turn()
    T0 = np.where((kind == 1) | (kind == 3), t + sign() * m.dt, T0)
    keep = (DX * DX + DY * DY >= 4 * m.dx2) & (DX * DX + DY * DY <= R * R)
    return tuple(x[keep] for x in (DX, DY, T2, T0, i, j))


def _want(m, DX, DY, T2, T0, i, j):
    """The reference's bounds of the cell: lower and upper k_dx, then k_dt from T0 - dt, T0 + dt."""
    d, T2t = _offset(m.sx, i, m.P), T2 + _offset(m.st, j, m.Q)
    tt = np.sin(T2t) * DX - np.cos(T2t) * DY
    e1 = (((DX * DX - 2 * d * tt) + DY * DY) - m.dx2) + d * d
    out = [2 * (tt - d - m.dx) / e1, 2 * (tt - d + m.dx) / e1]
    for t in (T0 - m.dt, T0 + m.dt):
        s = np.sin(T2t - t)
        out.append(s / (-s * d + np.cos(t) * DX + np.sin(t) * DY))
    return out


@pytest.fixture(autouse=True)
def _quotients_by_zero():
    with np.errstate(divide="ignore", invalid="ignore"):
        yield


def _check(m, want, got, ok):
    e0 = 2.0 ** -14 * m.max_k
    for w, g in zip(want, got):
        w, g = w[ok], g[ok]
        past = (np.abs(w) > m.max_k) & (np.abs(g) > m.max_k * (1 + 2.0 ** -13)) & (np.sign(w) == np.sign(g))
        near = np.abs(g - w) <= e0 * np.maximum(1.0, np.abs(w) / m.max_k)
        assert np.all(past | near), (np.sum(~(past | near)), (np.abs(g - w) / e0)[~(past | near)][:3], w[~(past | near)][:3])


def _trig(m, T2, j):
    """sin, cos of T2t by the addition theorem, in FP64, as k_curvelets makes them."""
    o = _offset(m.st, j, m.Q)
    s, c, so, co = np.sin(T2), np.cos(T2), np.sin(o), np.cos(o)
    return s * co + c * so, c * co - s * so


SETS = [dict(), dict(max_k=3.0), dict(dx=0.36), dict(dx=0.8, sx=0.2, nrad=5.0, w=5),
        dict(nrad=0.5, rad=8.0, w=8), dict(nrad=3.5, rad=40.0, w=32), dict(nrad=0.5, rad=1e6, w=64),
        dict(nrad=3.5, rad=8.0, w=2), dict(nrad=3.5, rad=8.0, w=8, max_k=0.05)]


@pytest.mark.parametrize("turns", [0, 166_000])  # orientations up to 1.04e6 rad: FAST_ANGLE is 2^20
@pytest.mark.parametrize("over", SETS, ids=lambda o: "-".join(f"{k}{v}" for k, v in o.items()) or "default")
def test_columns(shim, over, turns):
    m, f, R = _model(shim, **over)
    assert f.ok
    rng = np.random.default_rng(17)
    DX, DY, T2, T0, i, j = _pairs(rng, m, R, 1_500_000 if turns == 0 else 300_000, turns)
    sT, cT = (_r(x) for x in _trig(m, T2, j))
    d = _r(_offset(m.sx, i, m.P))
    X, Y = _r(DX), _r(DY)
    Rb = _r(np.abs(X) + np.abs(Y))
    ethr = _r(Rb * _r(Rb * f.eRR + f.eR) + f.e0)
    dthr, S1 = _r(Rb * f.dR + f.d0), _r(Rb * f.sR + f.s0)
    t2 = _r(sT * (-2 * X) + _r(cT * (2 * Y)))
    A = _r(X * X + _r(Y * Y - f.dx2))
    e1 = _r(d * t2 + _r(A + _r(d * d)))
    nre = -_rcp(e1, rng)
    klo = _r(_r(t2 + _r(2 * _offset(m.sx, i, m.P) + 2 * m.dx)) * nre)
    got, ok = [klo, _r(nre * f.ndx_4 + klo)], e1 >= ethr
    for t in (T0 - m.dt, T0 + m.dt):
        c, s = _r(np.cos(t)), _r(np.sin(t))
        sn = _r(sT * c + _r(cT * -s))
        D = _r(-sn * d + _r(c * X + _r(s * Y)))
        got.append(_r(sn * _rcp(D, rng)))
        ok &= (np.abs(D) >= dthr) | ((np.abs(sn) >= S1) & (np.abs(D) >= f.dtiny))
    assert ok.sum() > 0.1 * ok.size
    _check(m, _want(m, DX, DY, T2, T0, i, j), got, ok)


@pytest.mark.parametrize("turns", [0, 1, 16, 160, 166_000])
@pytest.mark.parametrize("over", SETS + [dict(max_k=0.002), dict(max_k=2.0 ** -10), dict(max_k=1000.0),
                                         dict(rad=1e6, w=64, max_k=0.002), dict(dx=0.36, max_k=2.0 ** -10),
                                         dict(dx=7.2, sx=2.0, max_k=0.002, nrad=30.0, w=30)],
                         ids=lambda o: "-".join(f"{k}{v:g}" for k, v in o.items()) or "default")
def test_fine_columns(shim, over, turns):
    """fine_column: FP64 quantities rounded once, under the thresholds of the pair's angles."""
    m, f, R = _model(shim, **over)
    assert f.ok
    rng = np.random.default_rng(18 + turns)
    DX, DY, T2, T0, i, j = _pairs(rng, m, R, 300_000, turns)
    sT, cT = _trig(m, T2, j)
    d = _offset(m.sx, i, m.P)
    t2 = -2.0 * (sT * DX - cT * DY)
    N = t2 + 2.0 * d
    e1 = _r(d * (t2 + d) + (DX * DX + (DY * DY - m.dx2)))
    ang = _r(_r(_r(np.abs(T2)) + _r(np.abs(T0))) + f.fa)
    ethr, dthr = _r(f.fe * ang), _r(f.fd * ang)
    re = _rcp(e1, rng)
    got, ok = [-_r(_r(N + 2.0 * m.dx) * re), _r(_r(2.0 * m.dx - N) * re)], e1 >= ethr
    small = (e1 < 100 * ethr)
    for t in (T0 - m.dt, T0 + m.dt):
        c, s = np.cos(t), np.sin(t)
        sn = sT * c - cT * s
        D = _r(-sn * d + (c * DX + s * DY))
        got.append(_r(_r(sn) * _rcp(D, rng)))
        ok &= np.abs(D) >= dthr
        small |= np.abs(D) < 100 * dthr
    assert ok.sum() > 0.1 * ok.size
    assert (ok & small).sum() > 1000  # denominators near the thresholds were drawn
    _check(m, _want(m, DX, DY, T2, T0, i, j), got, ok)


def test_the_pairs_radius(shim):
    """The smaller of the search radius and the window's corner; nrad has no part in it, and the
    model is turned away only where that radius is out of range."""
    for nrad, rad, w, want in ((3.5, 3.5, 3, 3.5), (0.5, 8.0, 8, 8.0), (3.5, 40.0, 3, 4 * 2 ** 0.5), (1e9, 2.0, 1, 2.0),
                               (1e-9, 3.5, 3, 3.5), (3.5, 1e9, 64, 65 * 2 ** 0.5)):
        m, f, R = _model(shim, nrad=nrad, rad=rad, w=w)
        assert abs(R - want) < 1e-12 * want and f.ok == 1
        assert f.dtiny >= U * (5 * R + 6 * 0.4)
    assert _model(shim, rad=1e-9)[1].ok == 0
