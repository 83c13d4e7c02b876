"""Float mode's rewrites of the bundle transport, checked bit for bit on the CPU.

k_bundles (csrc/cvl_path.cuh), float instantiation:
  - a double quotient of two floats rounded to float (:714-715) is taken as their float
    quotient: 53 >= 2 * 24 + 2 bits, so rounding twice gives what rounding once gives;
  - branch 2's denominator (:774) is formed as branch 1's (:711), the terms' signs turned
    and the last sum halved: round-to-nearest is odd-symmetric and x - x is +0 either way."""
import numpy as np
import pytest

F, D = np.float32, np.float64


def _bits(a):
    return np.ascontiguousarray(a, F).view(np.int32)


def _same(a, b):
    nan = np.isnan(a) & np.isnan(b)
    assert np.array_equal(_bits(a)[~nan], _bits(b)[~nan])


@pytest.mark.parametrize("kind", ["path", "any bits", "close quotients"])
def test_float_quotients(kind):
    rng = np.random.default_rng(7)
    n = 2_000_000
    if kind == "path":
        x, y = rng.uniform(-8, 8, n).astype(F), rng.uniform(-50, 50, n).astype(F)
        x[::997], y[::1009] = 0, 0
    elif kind == "any bits":  # subnormals, infinities, overflow, NaN
        x, y = rng.integers(0, 2**32, (2, n), dtype=np.uint32).view(F)
        x = np.where(np.abs(x) > 1e38, F(1), x)  # (2 x is exact on the path: |x| is a few pixels)
    else:  # quotients next to a float or to half way between two
        y = rng.integers(2**23, 2**24, n).astype(F)
        q = rng.integers(2**23, 2**24, n).astype(D) + rng.choice([0.0, 0.5], n)
        x = (q * y.astype(D)).astype(F)
    with np.errstate(all="ignore"):
        _same((D(2.0) * x.astype(D) / y.astype(D)).astype(F), F(2) * x / y)


@pytest.mark.parametrize("scale", [0.5, 4.0, 60.0])
def test_signed_denominators(scale):
    rng = np.random.default_rng(11)
    n = 200_000
    DX, DY = rng.uniform(-scale, scale, (2, n)).astype(F)
    tt = rng.uniform(-scale, scale, n).astype(F)
    dx2 = F(0.4) * F(0.4)
    DX[::50], DY[::50], tt[::50] = F(0.4), F(0), F(0)  # sums that cancel
    for i in range(9):
        d = F(F(0.1) * F(i - 4.0))
        sq = d * d
        X2, Y2 = (DX * DX).astype(D), (DY * DY).astype(D)
        ref1 = ((((-2.0 * D(d)) * tt.astype(D) + X2) + Y2) - D(dx2) + D(sq)).astype(F)
        ref2 = (-(((((2.0 * D(d)) * tt.astype(D) - X2) - Y2) + D(dx2)) - D(sq)) / 2.0).astype(F)
        for ref, s, half in ((ref1, 1.0, 1.0), (ref2, -1.0, -0.5)):
            e = ((((-2.0 * D(d)) * (s * tt.astype(D)) + s * X2) + s * Y2) + -s * D(dx2)) + s * D(sq)
            _same(ref, (e * half).astype(F))
